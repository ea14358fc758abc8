"""Kernels of a launch chain (``chain_begin``) are resident while the kernel before them still writes,
so their sources may not read what it writes through the read-only path, nor let the compiler move
such a read above the wait: no ``__restrict__`` on their parameters and no read-only load, except of
tables that nothing writes after their creation."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afid-murphfi_b200", "csrc")
SOURCES = {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}
CONSTANT = ("tw",)  # twiddles; metric and interpolation tables come in Tables t / SalTables st


def _kernels():
    """(file, name, parameters, body) of every kernel."""
    for f, src in SOURCES.items():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(", src):
            start = src.index("{", m.end())
            end = src.index("\n}\n", start)
            yield f, m.group(1), src[m.end():start], src[start:end]


KERNELS = list(_kernels())
CHAINED = [k for k in KERNELS if "chain_begin();" in k[3]]


def test_every_chained_launch_begins_with_the_wait():
    bodies = {n: b for _, n, _, b in KERNELS}
    launched = set()
    for src in SOURCES.values():
        for m in re.finditer(r"launch_chained\(\s*\w+,\s*(\w+)", src):
            name = m.group(1)
            if name.startswith("k_"):
                launched.add(name)
            else:  # `auto kern = k_name<..>` before it, the last one in either branch of a choice
                defs = re.findall(r"auto %s =([^;]*);" % name, src[:m.start()])
                launched.update(re.findall(r"\bk_\w+", defs[-1]) if defs else [])
    assert len(launched) > 20
    for name in launched:
        assert re.match(r"\{\s*chain_begin\(\);", bodies[name]), name


@pytest.mark.parametrize("kernel", CHAINED, ids=lambda k: k[1])
def test_reads_of_earlier_kernels_results_are_coherent(kernel):
    _, _, params, body = kernel
    restricted = re.findall(r"__restrict__\s+(\w+)", params)
    assert [p for p in restricted if p not in CONSTANT] == []
    for arg in re.findall(r"__ldg\((?:reinterpret_cast<const \w+ \*>\()?([\w.]+)", body):
        assert re.match(r"(t|st)\.", arg), arg
    for arg in re.findall(r"\btld<\w+>\(([\w.]+)", body):
        assert re.match(r"ts?\.", arg), arg
    assert ".nc" not in body


def test_device_functions_of_chained_kernels():
    """Helpers read their arguments coherently; only ``tld`` (metric tables) has a read-only form."""
    k1, sal = SOURCES["afid_k1.cuh"], SOURCES["afid_salinity.cu"]
    assert k1.count("ld.global.nc") == 1 and k1.index("double tld(") < k1.index("ld.global.nc") < k1.index("double cld(")
    for arg in re.findall(r"\btld<\w+>\(([\w.]+)", k1):
        assert re.match(r"ts?\.", arg), arg
    for fn in ("coarse_ext", "sal_ext", "scan_line"):
        body = sal[sal.index(" %s(" % fn):]
        body = body[:body.index("\n}\n")]
        assert "__restrict__" not in body, fn
        assert re.findall(r"__ldg\((?!bp|tp)", body) == [], fn
    for fn in ("double cld(", "double nld(", "double gld("):
        src = k1 if fn != "double gld(" else SOURCES["afid_device.cuh"]
        body = src[src.index(fn):]
        body = body[:body.index("\n}\n")]
        assert "asm volatile" in body and '"memory"' in body and ".nc" not in body and "__ldg" not in body, fn


def test_a_batch_runs_and_is_tuned_with_plain_launches():
    # its steps are captured, where programmatic edges cost more than plain ones
    src = SOURCES["afid_batch.cu"]
    assert "launch_chained(" not in src and "chain_begin()" not in src
    # switched off once, at creation and thus before the autotuner, and never on again
    assert src.count("L.chained") == 1 and "b->ctx->L.chained = false;" in src
    assert src.index("b->ctx->L.chained = false;") < src.index("int afid_batch_step(")
