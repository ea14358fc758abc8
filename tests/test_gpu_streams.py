"""Steps on a caller's stream, between kernels of the caller that change the resident fields: the
library's overlapping launches neither start on a field before the caller's kernel has written it
nor run into the next one.  The reference run waits for the device after every call."""
import numpy as np
import pytest
import torch

import afid_gpu as ag
from helpers import Case
from test_gpu_salinity import SalCase

pytestmark = pytest.mark.gpu


class _View:
    def __init__(self, solver, which, ncol):
        ptr, ld = solver.device_ptr(which)
        self.__cuda_array_interface__ = {"shape": (ncol * ld,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": None, "stream": None}


def _scale(solver, ncol):
    """The caller's kernels: one long enough that the library's next launches are queued behind it."""
    for which in (1, 2, 3):
        t = torch.as_tensor(_View(solver, which, ncol), device="cuda")
        for f in (2.0, 0.25, 1.875):
            t.mul_(f)  # exact but for the last


@pytest.mark.parametrize("shape,precision", [((64, 128, 1), ag.PREC_FP64), ((47, 60, 50), ag.PREC_FP64),
                                             ((96, 64, 32), ag.PREC_MIXED), ((150, 100, 90), ag.PREC_FP64)])
def test_steps_between_the_callers_kernels(shape, precision):
    case = Case(*shape, precision=precision, rayt=1e6, dt=1e-4)
    s = case.oracle_state(random_velocity=0.1)
    outs = []
    for wait in (True, False):
        stream = torch.cuda.Stream()
        with case.solver() as gpu, torch.cuda.stream(stream):
            gpu.set_k1_shape(0)
            gpu.set_stream(stream.cuda_stream)
            gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
            for n in range(4):
                _scale(gpu, shape[1] * shape[2])
                if wait:
                    torch.cuda.synchronize()
                gpu.time_marcher(1e-4, n)
                if wait:
                    torch.cuda.synchronize()
            outs.append(dict(gpu.download(), cfl=gpu.calc_max_cfl()))
    for k in outs[0]:
        assert np.isfinite(outs[0][k]).all() and np.array_equal(outs[0][k], outs[1][k]), k


def test_salinity_steps_between_the_callers_kernels():
    c = SalCase((40, 30, 20), (60, 48, 36), vel=0.02)
    outs = []
    for wait in (True, False):
        stream = torch.cuda.Stream()
        with c.solver() as gpu, torch.cuda.stream(stream):
            gpu.set_k1_shape(0)
            gpu.set_stream(stream.cuda_stream)
            for n in range(3):
                _scale(gpu, 30 * 20)
                if wait:
                    torch.cuda.synchronize()
                gpu.time_marcher(1e-4, n)
                if wait:
                    torch.cuda.synchronize()
            outs.append(dict(gpu.download(), sal=gpu.sal_download(), cflr=gpu.sal_cfl()))
    for k in outs[0]:
        assert np.isfinite(outs[0][k]).all() and np.array_equal(outs[0][k], outs[1][k]), k
