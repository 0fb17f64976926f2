"""A list of more than 2^31 entries: its total, and its entries behind the 2^31st (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
def test_more_than_2_31_entries(kind):
    """A simple cubic lattice of 64^3 atoms and a cutoff of 12.55 lattice constants, between
    two shells (157 and 158 squared): every row has as many entries as lattice
    points lie inside."""
    from examinimd_gb300 import Context
    m, cut = 64, 12.55
    x = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5
    n = len(x)
    g = np.stack(np.meshgrid(*[np.arange(-13, 14)] * 3, indexing="ij"), -1).reshape(-1, 3)
    row = int((np.sum(g * g, axis=1) <= cut * cut).sum()) - 1
    assert n * row > 2 ** 31
    c = Context(0)
    c.system_init([1.0], 1.0, 1.0, 0.005, [float(m)] * 3)
    c.set_local(x, np.zeros(n, np.int32), np.arange(1, n + 1, dtype=np.int32))
    c.comm_init(cut)
    c.neigh_init(kind, cut)
    c.comm_exchange_halo()
    c.binning_create(cut, cut, cut, 1, True, True, False)
    assert c.neigh_create(False) == n * row
    if kind == 1:
        c.close()
        return
    num, ent = c.neigh_get(n * row)
    np.testing.assert_array_equal(num, np.full(n, row))
    # the last rows, behind the 2^31st entry: their partners lie within the cutoff
    ng = c.info()[1]
    xa = c.get(0, n + ng, fields=("x",))["x"]
    for i in (0, n // 2, n - 2, n - 1):
        j = ent[i * row:(i + 1) * row]
        assert len(np.unique(j)) == row and i not in j
        assert np.sum((xa[j] - xa[i]) ** 2, axis=1).max() <= cut * cut
    c.close()
