"""SNAP systems of more than one chunk (131,072 atoms) and of tiles of 64 atoms (GPU).

A cell of 1,024 displaced atoms is repeated; lattice constant and displacements are
multiples of 2^-20, so every copy's distances are the cell's to the last bit.
Each copy's forces are compared with the cell's own: FP64 to the order of the sums
(some 100 terms of 2^-53 each), mixed with the FP64 cell's to the form's error.
"""
import numpy as np
import pytest

from tests import mdloop
from tests.test_gpu_snap_tables import _deck

pytestmark = pytest.mark.gpu

A, M = 3.1875, 8


def _systems(J, copies, nelem):
    st, cell = _deck(J, (M, M, M), A, nelem=nelem, seed=J)
    if nelem == 2:  # pairs of the second element end at 4.36 inside the common cutoff of 4.73
        st.elements[1]["radius"] = 0.46
    cell["x"] = np.mod(np.round(cell["x"] * 2.0 ** 20) / 2.0 ** 20, M * A)
    big, _ = _deck(J, [M * k for k in copies], A, nelem=nelem, seed=J)
    big.elements, big.type_map, big.masses = st.elements, st.type_map, st.masses
    g = np.stack(np.meshgrid(*[np.arange(k) for k in copies], indexing="ij"), -1).reshape(-1, 1, 3) * (M * A)
    n = len(g) * len(cell["x"])
    rep = dict(x=(cell["x"][None] + g).reshape(-1, 3), v=np.zeros((n, 3)), id=np.arange(1, n + 1, dtype=np.int32),
               type=np.tile(cell["type"], len(g)))
    return (st, cell), (big, rep)


def _context(st, state, precision):
    from examinimd_gb300 import Context
    c = Context(0)
    mdloop.init(c, st, state, precision=precision)
    return c


@pytest.mark.parametrize("J,precision,copies,nelem", [
    (2, 0, (6, 5, 5), 1), (4, 0, (13, 10, 1), 2), (2, 1, (6, 5, 5), 2), (8, 1, (6, 5, 5), 2),
    (8, 1, (5, 1, 1), 2), (9, 1, (5, 1, 1), 1), (10, 1, (5, 1, 1), 1)])
def test_copies_of_a_cell(J, precision, copies, nelem):
    small, large = _systems(J, copies, nelem)
    n, m = len(large[1]["x"]), len(small[1]["x"])
    c = _context(*small, 0)
    ref, e = mdloop.by_id(c.get(0, m))["f"], c.snap_energy()
    c.close()
    c = _context(*large, precision)
    f = mdloop.by_id(c.get(0, n))["f"].reshape(-1, m, 3)
    assert abs(c.snap_energy() - e * (n // m)) <= 1e-12 * max(abs(e) * (n // m), float(n))
    c.close()
    rms = np.sqrt(np.mean(ref * ref))
    if precision == 0:
        assert np.abs(f - ref).max() <= 1e-13 * rms
    else:
        assert np.sqrt(np.mean((f - ref) ** 2, axis=(1, 2))).max() <= 1e-6 * rms
        assert np.abs(f - ref).max() <= 1e-5 * rms


@pytest.mark.parametrize("keep", [False, True])
def test_adjoint_of_copies(keep):
    """The gradient of the copies is the cell's times their number, also from kept U and Z."""
    small, large = _systems(4, (6, 5, 5), 2)
    grad = []
    for st, state in (small, large):
        n, m = len(state["x"]), len(small[1]["x"])
        c = _context(st, state, 0)
        if keep:
            c.snap_keep_for_adjoint(True)
            c.snap_compute()
        g = np.tile(np.random.default_rng(3).standard_normal((m, 3)), (n // m, 1))
        grad.append(c.snap_adjoint(g[c.get(0, n)["id"] - 1], 0.7, 2, len(st.elements[0]["beta"])) / (n // m))
        c.close()
    assert np.abs(grad[1] - grad[0]).max() <= 1e-12 * np.abs(grad[0]).max()
