"""The barriers of the prompt path's tcgen05 kernels (k_pf_attn, k_pfx1, k_pft, k_pfx2), without a GPU: all agents' operations, a pair's two
CTAs together, run with vector clocks (test_gemm3_barriers_cpu.check)."""
import ctypes as C

import pytest

from test_gemm3_barriers_cpu import check


def _run(pkg, kernel, form, fmt, units, nsl):
    L, traces = pkg.llb.lib(), []
    while True:
        n = L.llb_b200_pf_trace(kernel, form, fmt, units, nsl, len(traces), None, 0)
        if n < 0:
            break
        buf = (C.c_int * (3 * n))()
        assert L.llb_b200_pf_trace(kernel, form, fmt, units, nsl, len(traces), buf, 3 * n) == n
        traces.append([tuple(buf[3 * i:3 * i + 3]) for i in range(n)])
    assert len(traces) in {0: (14,), 1: (32, 40), 2: (32,)}[kernel]
    return check(traces, [L.llb_b200_pf_bar_count(kernel, form, fmt, b) for b in range(128)])


@pytest.mark.parametrize("hd", [128, 256])
def test_attention(pkg, hd):
    for n in range(1, 40):
        assert _run(pkg, 0, hd, 0, 1, n) is None, n


@pytest.mark.parametrize("rows", [32, 64, 128])
@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_exact_codes(pkg, packs, fmt, rows):
    for units, nsl in [(1, n) for n in range(1, 12)] + [(2, 1), (2, 3), (3, 2), (3, 5), (4, 7)]:
        assert _run(pkg, 1, rows, packs.FMT[fmt], units, nsl) is None, (units, nsl)


def test_exact_codes_of_two_units(pkg):
    for units, nsl in [(1, n) for n in range(1, 16)] + [(2, 1), (2, 3), (3, 2), (3, 5), (4, 7)]:
        assert _run(pkg, 2, 0, 0, units, nsl) is None, (units, nsl)
