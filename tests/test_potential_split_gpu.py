"""The nuclear attraction kernel shares the charges out over the grid where a class has few
pairs (oneint.cu: launch_one): V of all charges against the sum of each charge's V, for
which the grid has one slice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis", [(1, "cc-pvtz"), (20, "cc-pvdz")])
@pytest.mark.parametrize("ewald", [([1.0], [-1.0]), ([-0.7, 0.7], [0.3, -1.0])])
def test_potential_is_the_sum_over_its_charges(ls, n, basis, ewald):
    from lightspeed_b200.geometry import alkane
    mol = alkane(n)
    bas = ls.Basis.from_gbs_file(mol, basis)
    pl = ls.PairList.build_schwarz(bas, bas, True, 1e-14)
    res, ew = ls.ResourceList.build(), ls.Ewald(*ewald)
    q = np.array(mol.xyzZ)
    q[1, 3] = 0.0   # no charge: skipped
    V = ls.IntBox.potential(res, ew, pl, ls.Tensor.array(q)).np.copy()
    total, size = np.zeros_like(V), np.zeros_like(V)
    for row in q:
        v = ls.IntBox.potential(res, ew, pl, ls.Tensor.array(row[None].copy())).np
        total += v
        size += np.abs(v)
    # FP64 sums of the same terms in another order, up to contraction length^2 * atoms of them
    assert np.max(np.abs(V - total)) < 1e-13 * np.max(size)
    assert np.max(np.abs(V)) > 1.0
