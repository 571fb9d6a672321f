"""J and its gradient with f shells: the class pairs of the warp kernel (Hermite classes
up to (6|6), and (7|6) in the gradient) against the exchange kernels and against
derivatives of the engine's own energies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ndens,ewald", [(1, 1, ([1.0], [-1.0])), (1, 3, ([-0.7, 0.7], [0.3, -1.0])),
                                           (2, 1, ([1.0], [0.4]))])
def test_coulomb_f_classes_match_exchange(ls, n, ndens, ewald):
    """(x z|y w) from J (of y w^T) and from K (of z w^T): two sets of kernels, every class up to f."""
    from lightspeed_b200.geometry import water_cluster
    bas = ls.Basis.from_gbs_file(water_cluster(n, seed=6), "cc-pvtz")
    x, y, z, w = np.random.default_rng(8).standard_normal((4, ndens, bas.nao)) * 0.2
    thre = 1e-18
    pl = ls.PairList.build_schwarz(bas, bas, True, thre)
    res, ew = ls.ResourceList.build(), ls.Ewald(*ewald)
    try:
        ls.set_precision(ls.PREC_FP64)
        Js = ls.IntBox.coulombMulti(res, ew, pl, pl, [ls.Tensor.array(np.outer(a, b)) for a, b in zip(y, w)],
                                    thre, thre)
        Ks = ls.IntBox.exchangeMulti(res, ew, pl, pl, [ls.Tensor.array(np.outer(a, b)) for a, b in zip(z, w)], False,
                                     thre, thre)
    finally:
        ls.set_precision(ls.PREC_MIXED)
    for k in range(ndens):
        vj, vk = x[k] @ Js[k].np @ z[k], x[k] @ Ks[k].np @ y[k]
        scale = np.abs(x[k]) @ np.abs(Js[k].np) @ np.abs(z[k])
        assert abs(vj) > 1e-6 * scale
        assert abs(vj - vk) < 1e-12 * scale   # FP64 sums of the same integrals in two orders


def test_gradients_with_f_shells_are_the_energys_derivatives(ls):
    """Fourth-order central differences (step 1e-2 Bohr, error ~ h^4 = 1e-8 of the fifth derivative)."""
    from lightspeed_b200.geometry import water_cluster
    mol = water_cluster(1, seed=1)
    bas = ls.Basis.from_gbs_file(mol, "cc-pvtz")
    X = np.random.default_rng(2).standard_normal((bas.nao, 5)) * 0.2
    D = ls.Tensor.array(X @ X.T)
    res, ew = ls.ResourceList.build(), ls.Ewald.coulomb()
    thre = 1e-16

    def energies(xyz):
        b = ls.Basis.from_gbs_file(ls.Molecule.from_arrays([a.symbol for a in mol.atoms], xyz), "cc-pvtz")
        pl = ls.PairList.build_schwarz(b, b, True, thre)
        J = ls.IntBox.coulomb(res, ew, pl, pl, D, thre, thre).np
        K = ls.IntBox.exchange(res, ew, pl, pl, D, True, thre, thre).np
        return np.array([np.sum(D.np * J), np.sum(D.np * K)])

    try:
        ls.set_precision(ls.PREC_FP64)
        pl = ls.PairList.build_schwarz(bas, bas, True, thre)
        GJ = ls.IntBox.coulombGrad(res, ew, pl, D, D, thre, thre).np
        GK = ls.IntBox.exchangeGrad(res, ew, pl, D, D, True, True, True, thre, thre).np
        h = 1e-2
        for atom, d in ((0, 0), (1, 2)):
            E = []
            for k in (-2, -1, 1, 2):
                xyz = mol.xyz.copy()
                xyz[atom, d] += k * h
                E.append(energies(xyz))
            num = (E[0] - 8.0 * E[1] + 8.0 * E[2] - E[3]) / (12.0 * h)
            scale = max(np.max(np.abs(GJ)), 1.0)
            assert abs(num[0] - GJ[atom, d]) < 1e-5 * scale
            assert abs(num[1] - GK[atom, d]) < 1e-5 * scale
    finally:
        ls.set_precision(ls.PREC_MIXED)
