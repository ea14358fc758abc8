"""The CFL and divergence maxima leave their accumulators ready for the next launch: calls in any
order give the same values, and a divergence check between steps does not enter a batch's CFL."""
import numpy as np
import pytest

import afid_gpu as ag
from helpers import Case, bou_text
from oracle import afid_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 6, 1), (33, 10, 6), (64, 96, 90)])  # one block .. more than 1184 columns
def test_maxima_repeat_in_any_order(shape):
    case = Case(*shape, rayt=1e6, dt=1e-3)
    s = case.oracle_state(random_velocity=0.3)
    cfl, div = o.calc_max_cfl(case.g, s), o.check_divergence(case.g, s)
    with case.solver() as gpu:
        gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
        # sums of a few terms in either order: rounding of the largest term
        for call in (gpu.calc_max_cfl, gpu.check_divergence, gpu.check_divergence, gpu.calc_max_cfl, gpu.calc_max_cfl):
            want = cfl if call == gpu.calc_max_cfl else div
            assert call() == pytest.approx(want, rel=1e-14)
        s.vx *= 0.25  # a smaller state afterwards: nothing of the old maximum is left
        s.vy *= 0.25
        s.vz *= 0.25
        gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
        assert gpu.calc_max_cfl() == pytest.approx(0.25 * cfl, rel=1e-14)


@pytest.mark.parametrize("nym,nzm,nslots", [(16, 1, 3), (50, 1, 2), (24, 16, 1)])  # one, several chunks; 3-D
def test_divergence_check_between_batch_steps(nym, nzm, nslots):
    inp = ag.parse_bou_in(bou_text(40, nym, nzm, rayt=1e6, idtv=1, dt=1e-3, cflmax=0.5, dtmax=5e-2))
    rng = np.random.default_rng(3)

    def make():
        b = ag.Batch(inp, nslots)
        for k in range(nslots):
            f = [0.5 * rng_fields[q][k] for q in range(5)]
            b.upload(k, *f)
        b.set_active([1] * nslots)
        return b

    rng_fields = rng.standard_normal((5, nslots) + ((nzm, nym, 41) if nzm > 1 else (nym, 41)))
    rng_fields[0, ..., 0] = rng_fields[0, ..., -1] = 0.0
    with make() as a, make() as b:
        for n in range(4):
            a.step(1)
            b.step(1)
            if n != 2:
                b.divmax()
        sa, sb = a.stats(), b.stats()
        for key in ("cfl", "dt", "time", "nu_vol"):
            assert np.array_equal(sa[key], sb[key]), key
