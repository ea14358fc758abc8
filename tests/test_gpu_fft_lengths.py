"""The transforms of lengths with two factors up to 20 or 25 or three up to 16 (and 1250, which has
neither) against the oracle: every register class, odd lengths, equal and very unequal factors, x
tiles with one valid point and with one missing, both directions, both precisions, the divergence and
a given field."""
import numpy as np
import pytest

import afid_gpu as ag
from helpers import Case, bou_text, rel_l2, rel_l2_mod_mean
from oracle import afid_oracle as o

pytestmark = pytest.mark.gpu

# (nxm, nym, nzm): factors  y                      z
SHAPES = [(17, 6, 10),    # 2 x 3, 2 x 5           smallest
          (3, 20, 45),    # 4 x 5, 5 x 9 (odd)
          (16, 144, 50),  # 12 x 12, 5 x 10
          (33, 240, 27),  # 15 x 16, 3 x 9 (odd)
          (15, 81, 160),  # 9 x 9 (odd), 10 x 16
          (10, 300, 20),  # 15 x 20
          (9, 18, 400),   # 20 x 20
          (8, 625, 6),    # 25 x 25 (odd)
          (12, 10, 450),  # 2 x 5, 10 x 9 x 5
          (5, 900, 4),    # 10 x 10 x 9
          (4, 4, 810),    # 10 x 9 x 9
          (6, 972, 2),    # 12 x 9 x 9
          (3, 1250, 2),   # no such factors: the general kernels
          (33, 480, 1),   # 10 x 8 x 6, 2-D
          (47, 100, 1)]   # 2-D


@pytest.mark.parametrize("shape", SHAPES)
def test_step_with_these_lengths(shape):
    case = Case(*shape, rayt=1e5, dt=1e-3)
    s = case.oracle_state(random_velocity=0.1)
    with case.solver() as gpu:
        gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
        gpu.time_marcher(1e-3, 0)
        out = gpu.download()
    o.time_marcher(case.g, s, 1e-3)
    n = case.p.nxm
    # FP64 transforms and solves against LAPACK and pocketfft: the parity tests' bound
    for f in ("vx", "vy", "vz", "temp"):
        assert rel_l2(out[f][..., :n], getattr(s, f)[..., :n]) < 1e-10, f
    assert rel_l2_mod_mean(out["pr"][..., :n], s.pr[..., :n]) < 1e-10


@pytest.mark.parametrize("shape", [(17, 6, 10), (33, 240, 50), (20, 300, 20), (8, 625, 6), (5, 900, 4)])
def test_mixed_follows_fp64(shape):
    # dt inside the explicit diffusion's bound 0.63 dy^2 Re (2.4e-4 at 900 points, Re = 316): beyond
    # it every substep amplifies rounding by the factor it amplifies the finest modes with
    outs = []
    for prec in (ag.PREC_FP64, ag.PREC_MIXED):
        case = Case(*shape, precision=prec, rayt=1e5, dt=1e-4)
        s = case.oracle_state(random_velocity=0.1)
        with case.solver() as gpu:
            gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
            gpu.time_marcher(1e-4, 0)
            outs.append(gpu.download())
    for f in ("vx", "vy", "vz"):  # 32-bit transforms: as tests/test_gpu_mixed.py
        assert rel_l2(outs[1][f], outs[0][f]) < 2e-5, f


@pytest.mark.parametrize("shape", [(9, 45, 20), (18, 240, 6)])
def test_spectra_of_a_field(shape):
    case = Case(*shape, rayt=1e5, dt=1e-3)
    s = case.oracle_state(random_velocity=0.1)
    acc = {}
    o.spectra_update(case.g, s, 0.5, acc)
    with case.solver() as gpu:
        gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
        gpu.spectra_reset()
        gpu.spectra_update(0.5)
        got = gpu.spectra()
    for f in ("vx", "vy", "vz", "temp"):
        want = [v for k, v in acc.items() if k.startswith(f[:2])][0] / 0.5
        assert np.allclose(got[f].reshape(want.shape), want, rtol=1e-10, atol=1e-12 * np.abs(want).max()), f


def test_batch_slot_equals_domain_with_these_lengths():
    """A batch binds each instance's scalars in the transform kernels; slots of different aspect ratio."""
    kw = dict(rayt=1e6, idtv=1, dt=1e-3, cflmax=1.0, dtmax=5e-3)
    inps = [ag.parse_bou_in(bou_text(40, 90, 1, ylen=y, **kw)) for y in (1.0, 2.0)]
    with ag.Batch(inps[0], 2) as b:
        for k in range(2):
            b.configure(k, inps[k])
            b.seed(k, 5 + k)
        b.set_active([1, 1])
        b.step(3)
        got = [b.download(k) for k in range(2)]
    for k in range(2):
        with ag.Batch(inps[k], 1) as a:
            a.seed(0, 5 + k)
            a.set_active([1])
            a.step(3)
            want = a.download(0)
        for f in ag.Batch.FIELDS:
            assert np.array_equal(got[k][f], want[f]), (k, f)
