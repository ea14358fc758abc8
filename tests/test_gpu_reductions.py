"""The CFL and divergence maxima leave their accumulators ready for the next launch: calls in any
order give the same values (the refined CFL's words lie beside theirs), and a divergence check
before a step does not enter a batch's CFL."""
import numpy as np
import pytest

import afid_gpu as ag
from helpers import Case
from oracle import afid_oracle as o
from oracle import afid_salinity as sa
from test_gpu_salinity import SalCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 6, 1), (33, 10, 6), (64, 96, 90), (12, 120, 80)])
# one block .. 1080 blocks of eight columns .. more columns than the largest grid's 1184 x 8 warps
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


def test_maxima_of_both_grids_in_any_order():
    c = SalCase((16, 16, 8), (24, 48, 32))  # 1536 refined columns for 1184 blocks
    want = {"cfl": o.calc_max_cfl(c.g, c.s), "div": o.check_divergence(c.g, c.s),
            "ref": sa.calc_max_cfl_refined(c.m, c.ss)}
    assert len({round(v, 6) for v in want.values()}) == 3
    with c.solver() as gpu:
        call = {"cfl": gpu.calc_max_cfl, "div": gpu.check_divergence, "ref": gpu.sal_cfl}
        for k in ("ref", "cfl", "ref", "ref", "div", "ref", "cfl", "div", "cfl", "ref"):
            # the refined velocities are interpolated: the bound of tests/test_gpu_salinity.py
            assert call[k]() == pytest.approx(want[k], rel=1e-12 if k == "ref" else 1e-14), k


@pytest.mark.parametrize("nym,nzm,nslots", [(16, 1, 3), (50, 1, 2), (24, 16, 1)])  # one, several chunks; 3-D
def test_divergence_check_before_a_batch_step(nym, nzm, nslots):
    """A field that alternates along y: its divergence is far above its CFL number, which averages
    neighbours, so either one left in the other's place shows."""
    dt = 1e-6
    case = Case(40, nym, nzm, rayt=1e6, idtv=0, dt=dt, cflmax=1e3)
    states = []
    for k in range(nslots):
        s = case.oracle_state(random_velocity=0.05, rng_seed=k)
        s.vy[..., :40] += (5.0 + k) * (-1.0) ** np.arange(nym)[:, None]
        states.append(s)
    cfl = [o.calc_max_cfl(case.g, s) for s in states]
    div = [o.check_divergence(case.g, s) for s in states]
    assert all(d > 5 * c for c, d in zip(cfl, div))
    with ag.Batch(case.inp, nslots) as b:
        for check in (False, True, True):
            for k, s in enumerate(states):
                b.upload(k, s.vx, s.vy, s.vz, s.temp, s.pr)
            b.set_active([1] * nslots)
            if check:
                # sums of a few terms in either order: rounding of the largest term
                np.testing.assert_allclose(b.divmax(), div, rtol=1e-14)
            b.step(1)
            np.testing.assert_allclose(b.stats()["cfl"], np.array(cfl) * dt, rtol=1e-14)
            assert b.divmax().max() < 1e-6 * min(div)  # projected
