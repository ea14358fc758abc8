"""A tuning run between two steps leaves the state and the RK3 histories as they were, whether the
histories of its launches find room in dead buffers or need scratch memory."""
import numpy as np
import pytest

import afid_gpu as ag
from helpers import Case

pytestmark = pytest.mark.gpu


# scratch for two or three histories (fewer columns than a sample), for one, for none
@pytest.mark.parametrize("shape,precision", [((40, 20, 12), ag.PREC_FP64), ((40, 20, 12), ag.PREC_MIXED),
                                             ((33, 128, 100), ag.PREC_MIXED), ((128, 200, 180), ag.PREC_FP64),
                                             ((112, 300, 240), ag.PREC_FP64)])
def test_tuning_between_steps_changes_nothing(shape, precision):
    case = Case(*shape, precision=precision, rayt=1e6, dt=1e-4)
    s = case.oracle_state(random_velocity=0.1)
    outs = []
    for tune in (False, True):
        with case.solver() as gpu:
            gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
            for n in range(4):
                gpu.time_marcher(1e-4, n)
                if tune:
                    info = gpu.autotune(force=True)
                    assert all(us > 0 for *_, us in info["shapes"])
            outs.append(gpu.download())
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k]), k
