"""Contexts of different transform lengths stepped from different host threads: kernels that serve many
lengths keep a shared-memory limit that no other context lowers before a launch."""
import threading

import numpy as np
import pytest

import afid_gpu as ag
from helpers import Case

pytestmark = pytest.mark.gpu

# y and z lengths of three factors, of two above 48 KB, and without such factors (the general kernels)
PAIRS = [((5, 720, 4), (5, 480, 4)), ((5, 4, 900), (5, 6, 450)), ((4, 400, 2), (4, 625, 2)),
         ((3, 2, 1250), (3, 1250, 2)), ((4, 900, 2), (4, 1250, 2))]


@pytest.mark.parametrize("pair", PAIRS)
def test_contexts_of_different_lengths_on_two_threads(pair):
    cases = [Case(*shape, rayt=1e5, dt=1e-5) for shape in pair]
    states = [c.oracle_state(random_velocity=0.1) for c in cases]
    steps = 150

    def march(k, out):
        try:
            with cases[k].solver() as gpu:
                gpu.set_k1_shape(0)
                s = states[k]
                gpu.upload(s.vx, s.vy, s.vz, s.temp, s.pr)
                for n in range(steps):
                    gpu.time_marcher(1e-5, n)
                out[k] = gpu.download()
        except Exception as e:  # handed to the asserting thread
            out[k] = e

    alone, together = [None, None], [None, None]
    for k in range(2):
        march(k, alone)
    threads = [threading.Thread(target=march, args=(k, together)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert not isinstance(alone[k], Exception), alone[k]
        assert not isinstance(together[k], Exception), together[k]
        for f in ag.Solver.FIELDS:
            assert np.array_equal(alone[k][f], together[k][f]), (k, f)
