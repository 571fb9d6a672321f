"""Work units of the unique-quartet K gradient (kxargs.cuh: xgrad_split, unit_of): every bra
meets every ket once, and classes of millions of pairs still fit the 32-bit unit queue."""
import ctypes

import numpy as np
import pytest

from host_code import CUDA_WORDS, compile_host, source_part

CODE = """
struct XGradArgs { int boff[2], bn[2], koff[2], kn[2], chunk; };
%s
extern "C" void split(long nb, long kn0, long kn1, long lo, long hi, long units, long* out)
{
    const XSplit s = xgrad_split(nb, kn0, kn1, lo, hi, units);
    out[0] = s.chunk;
    out[1] = s.nunit;
}
extern "C" void unit(const int* a, unsigned k, int* out)
{
    const XGradArgs A = {{a[0], a[1]}, {a[2], a[3]}, {a[4], a[5]}, {a[6], a[7]}, a[8]};
    const XUnit u = unit_of(A, k);
    out[0] = u.i; out[1] = u.j0; out[2] = u.j1;
}
"""
MAX_UNITS = 0xffff0000
UNITS = 16 * 148 * 4
LANE, WARP = (32, 2048), (4, 256)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    part = source_part("kxargs.cuh", "// Work unit -> bra index and ket range.", "template <int L1, int L2>\nvoid launch_xgrad_12(")
    return compile_host(tmp_path_factory.mktemp("split"), CUDA_WORDS + CODE % part)


def split(lib, nb, kn, limits):
    out = (ctypes.c_long * 2)()
    lib.split(ctypes.c_long(nb), ctypes.c_long(kn[0]), ctypes.c_long(kn[1]), ctypes.c_long(limits[0]),
              ctypes.c_long(limits[1]), ctypes.c_long(UNITS), out)
    return out[0], out[1]


def unit(lib, boff, bn, koff, kn, chunk, k):
    out = (ctypes.c_int * 3)()
    lib.unit((ctypes.c_int * 9)(*boff, *bn, *koff, *kn, chunk), ctypes.c_uint(k), out)
    return tuple(out)


@pytest.mark.parametrize("limits", [LANE, WARP])
@pytest.mark.parametrize("bn,kn", [((1, 0), (1, 0)), ((3, 2), (0, 41)), ((0, 7), (130, 1)), ((40, 0), (33, 64))])
def test_every_pair_of_pairs_once(lib, limits, bn, kn):
    boff, koff = (5, 100), (7, 1000)
    chunk, n = split(lib, sum(bn), kn, limits)
    assert limits[0] <= chunk <= limits[1]
    seen = np.zeros((2000, 2000), int)
    for k in range(n):
        i, j0, j1 = unit(lib, boff, bn, koff, kn, chunk, k)
        assert j0 < j1
        seen[i, j0:j1] += 1
    want = np.zeros_like(seen)
    for r in range(2):
        for q in range(2):
            want[boff[r]:boff[r] + bn[r], koff[q]:koff[q] + kn[q]] = 1
    assert np.array_equal(seen, want)


@pytest.mark.parametrize("limits", [LANE, WARP])
@pytest.mark.parametrize("bn,kn", [((800000, 0), (740000, 0)), ((2500000, 10), (10, 2500000)), ((5000000, 5000000), (9999999, 1)),
                                   ((2147450880, 0), (2147450880, 0)), ((1073725440, 1073725440),) * 2, ((1, 0), (2147450880, 0))])
def test_large_classes_fit_the_queue(lib, limits, bn, kn):
    chunk, n = split(lib, sum(bn), kn, limits)
    exact = [-(-k // chunk) for k in kn]
    assert n == sum(bn) * sum(exact) <= MAX_UNITS
    koff = (0, kn[0] if kn[0] + kn[1] < 2 ** 31 else 0)
    # first and last unit of each ket range
    for r in range(2):
        if not kn[r]:
            continue
        first, last = sum(exact[:r]), sum(exact[:r + 1]) - 1
        assert unit(lib, (0, bn[0]), bn, koff, kn, chunk, first * sum(bn))[1:] == (koff[r], koff[r] + min(chunk, kn[r]))
        i, j0, j1 = unit(lib, (0, bn[0]), bn, koff, kn, chunk, last * sum(bn) + sum(bn) - 1)
        assert (i, j1) == (sum(bn) - 1, koff[r] + kn[r]) and j0 == koff[r] + (exact[r] - 1) * chunk
