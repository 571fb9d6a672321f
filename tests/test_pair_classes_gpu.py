"""Pair lists over shells far above the kernels' f: the list itself holds any angular
momentum (J and K refuse it later), its classes in (L1, L2) order, bound descending."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (7 <= L1 + L2 <= 10 is refused by the list)
@pytest.mark.parametrize("shells1,shells2", [((0, 11, 0, 11), None), ((15, 15, 15), None), ((0, 20), (0, 1, 20))])
def test_list_over_high_shells(ls, shells1, shells2):
    lib = ctypes.CDLL(ls.LIB_PATH)
    lib.lsjk_last_error.restype = ctypes.c_char_p
    lib.lsjk_pairlist_size.restype = ctypes.c_long
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    ctx = ctypes.c_void_p()
    assert lib.lsjk_context_create(0, ctypes.byref(ctx)) == 0

    def basis(shells):
        n = len(shells)
        L = np.array(shells, np.int32)
        nc = (L + 1) * (L + 2) // 2
        start = np.concatenate([[0], np.cumsum(nc)[:-1]]).astype(np.int32)
        f = np.arange(n, dtype=np.float64)
        xyz = np.stack([0.3 * f, 0.1 * f * f, -0.2 * f], 1).copy()
        c, e, idx = 1.0 + 0.1 * f, 0.5 + 0.25 * f, np.arange(n, dtype=np.int32)
        h = ctypes.c_void_p()
        rc = lib.lsjk_basis_create(ctx, n, ptr(c), ptr(e), ptr(xyz), ptr(L), ptr(np.zeros(n, np.int32)), ptr(start),
                                   ptr(start), ptr(idx), ptr(idx), ptr(idx), ctypes.byref(h))
        assert rc == 0, lib.lsjk_last_error()
        return h, L

    b1, L1 = basis(shells1)
    b2, L2 = (b1, L1) if shells2 is None else basis(shells2)
    pl = ctypes.c_void_p()
    try:
        rc = lib.lsjk_pairlist_build_schwarz(ctx, b1, b2, int(shells2 is None), ctypes.c_float(0.0), ctypes.byref(pl))
        assert rc == 0, lib.lsjk_last_error()
        n = lib.lsjk_pairlist_size(pl)
        assert n == (len(L1) * (len(L1) + 1) // 2 if shells2 is None else len(L1) * len(L2))
        l1, l2, p1, p2 = (np.zeros(n, np.int32) for _ in range(4))
        bound = np.zeros(n, np.float32)
        assert lib.lsjk_pairlist_export(pl, ptr(l1), ptr(l2), ptr(p1), ptr(p2), ptr(bound)) == 0
        assert np.array_equal(l1, L1[p1]) and np.array_equal(l2, L2[p2])
        assert len({(i, j) for i, j in zip(p1, p2)}) == n
        order = list(zip(l1, l2, -bound.astype(np.float64), p1, p2))
        assert order == sorted(order)
        if max(max(L1), max(L2)) > 3:   # refused by the one-electron kernels as by J and K
            assert lib.lsjk_overlap(ctx, pl, ptr(np.zeros(1))) != 0
    finally:
        lib.lsjk_pairlist_destroy(pl)
        lib.lsjk_basis_destroy(b1)
        if shells2 is not None:
            lib.lsjk_basis_destroy(b2)
        lib.lsjk_context_destroy(ctx)
