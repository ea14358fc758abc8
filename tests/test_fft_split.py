"""The factors that the general-length transforms choose (fft2_split, host code of the library)."""
import ctypes
import os
import re

import afid_gpu as ag

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afid-murphfi_b200", "csrc",
                   "afid_fft2.cu")


class Split(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("r1", "r2", "r3", "m")]


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


def test_splits_hold_and_every_built_transform_is_reached():
    split = getattr(ag.lib(), "_ZN4afid10fft2_splitEi")
    split.restype, split.argtypes = Split, [ctypes.c_int]
    built = {int(r) for r in re.findall(r"case (\d+): dft_r<\1,", open(SRC).read())}
    reached = set()
    # 2048: the longest transform whose tiles fit a block
    for n in (n for n in range(2, 2049) if _smooth(n)):
        f = split(n)
        if f.r1 == 0:
            continue
        assert f.r1 * f.r2 * f.r3 == n and f.m == f.r2 * f.r3, n
        factors = {f.r1, f.r2, f.r3} - {1}
        assert factors <= built, n
        assert max(factors) <= (16 if f.r3 > 1 else 25), n
        reached |= factors
    assert reached == built
