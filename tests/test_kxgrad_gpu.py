"""K gradient of one symmetric density over unique quartets (the fully symmetric call)
against the general routine over every ordered quartet, which the golden vectors pin:
every bra and ket class up to f, a quartet per lane and per warp, full and partial
batches, range-separated operators."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system,basis,ewald", [
    ("w1", "sto-3g", ([1.0], [-1.0])), ("w2", "6-31gs", ([1.0], [-1.0])), ("w2", "cc-pvdz", ([-0.7, 0.7], [0.3, -1.0])),
    ("c3", "cc-pvdz", ([1.0], [0.3])), ("w1", "cc-pvtz", ([1.0], [-1.0])), ("w2", "cc-pvtz", ([1.0], [-1.0]))])
def test_symmetric_matches_general(ls, system, basis, ewald):
    from lightspeed_b200.geometry import alkane, water_cluster
    n = int(system[1:])
    mol = water_cluster(n, seed=2) if system[0] == "w" else alkane(n)
    bas = ls.Basis.from_gbs_file(mol, basis)
    X = np.random.default_rng(3).standard_normal((bas.nao, 6)) * 0.3
    D = ls.Tensor.array(X @ X.T)
    # nothing screened: the two routines screen a quartet by different blocks of D, and a derivative
    # is up to 2 alpha r (1e4 for the tightest s) times its screened estimate, so at 1e-14 they differ
    # by 1e-14 * 1e4 * sqrt(quartets dropped) ~ 1e-10 (1.9e-10 seen)
    thre = 1e-24
    pl = ls.PairList.build_schwarz(bas, bas, True, thre)
    res, ew = ls.ResourceList.build(), ls.Ewald(*ewald)
    G = ls.IntBox.exchangeGrad(res, ew, pl, D, D, True, True, True, thre, thre).np
    R = ls.IntBox.exchangeGrad(res, ew, pl, D, D, True, True, False, thre, thre).np
    scale = np.max(np.abs(R))
    assert scale > 1e-3
    # FP64 sums in another order: terms up to 1e4 times the result, 2e-16 each
    assert np.max(np.abs(G - R)) < 1e-11 * scale
    assert np.max(np.abs(G.sum(axis=0))) < 1e-11 * scale


def test_screen_bites_and_accumulates(ls):
    """At a coarse threshold most batches are partial; the error against the fine one stays near it."""
    from lightspeed_b200.geometry import water_cluster
    mol = water_cluster(3, seed=5)
    bas = ls.Basis.from_gbs_file(mol, "6-31gs")
    X = np.random.default_rng(4).standard_normal((bas.nao, 6)) * 0.3
    D = ls.Tensor.array(X @ X.T)
    res, ew = ls.ResourceList.build(), ls.Ewald.coulomb()
    out = {}
    for thre in (1e-14, 1e-8):
        pl = ls.PairList.build_schwarz(bas, bas, True, 1e-14)
        G = ls.IntBox.exchangeGrad(res, ew, pl, D, D, True, True, True, thre, thre)
        out[thre] = G.np.copy()
        ls.IntBox.exchangeGrad(res, ew, pl, D, D, True, True, True, thre, thre, G)
        assert np.max(np.abs(G.np - 2.0 * out[thre])) < 1e-11 * np.max(np.abs(out[thre]))
    # ~1e5 primitive pairs' quartets dropped, each below 1e-8 times a derivative factor 2 alpha r
    assert 0.0 < np.max(np.abs(out[1e-8] - out[1e-14])) < 1e-3
