"""The SNAP kernels over their table sizes and tile edges, against the CPU oracle (GPU).

twojmax from 0 to 10 (tables, power registers and the number of j per (m, m')
change at 8, 9 and 10), atom counts around the tile and pooling sizes,
neighbour counts from none to more than two 32-lane rounds, both switch
flags, two elements.  Tolerance: as for the other SNAP parity tests 1e-12 of
the RMS force (up to twojmax 8), four times that above, where the sums over j
are longer; the energy is a sum of n such terms.  Threads with systems of
different size use the library at once.
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from tests import mdloop

pytestmark = pytest.mark.gpu


def _ncoeff(J):
    return sum(1 for a in range(J + 1) for b in range(a + 1) for c in range(a - b, min(J, a + b) + 1, 2) if c >= a)


def _deck(J, cells, a, nelem=1, switchflag=1, kind=0, seed=1):
    rng = np.random.default_rng(seed)
    elems = [dict(name=f"E{k}", radius=0.5, weight=1.0 - 0.15 * k,
                  beta=list(np.concatenate([[-1.0], rng.normal(0.0, 0.1, _ncoeff(J))]))) for k in range(nelem)]
    snap = dict(elements=elems, params={"rcutfac": "4.73442", "twojmax": str(J), "rfac0": "0.99363", "rmin0": "0",
                                        "switchflag": str(switchflag)})
    st = mdloop.SnapSetup(*cells, snap, a=a, lattice_style=2, kind=kind, masses=[183.84] * nelem,
                          type_elems=[f"E{k}" for k in range(nelem)])
    g = np.stack(np.meshgrid(*[np.arange(k) for k in cells], indexing="ij"), -1).reshape(-1, 3)
    x = ((g[:, None, :] + np.array([[0, 0, 0], [0.5, 0.5, 0.5]])[None]) * a).reshape(-1, 3)
    x = np.mod(x + rng.normal(0.0, 0.05, x.shape), st.domain)
    n = len(x)
    return st, dict(x=x, v=np.zeros((n, 3)), id=np.arange(1, n + 1, dtype=np.int32),
                    type=rng.integers(0, nelem, n).astype(np.int32))


def _compare(st, state, tol):
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    gpu, orc = Context(0), Oracle(4)
    n = len(state["x"])
    mdloop.init(gpu, st, state)
    mdloop.init(orc, st, state)
    a, b = gpu.get(0, n)["f"], orc.get(0, n)["f"]
    rms = np.sqrt(np.mean(np.sum(b * b, axis=1)))
    assert rms > 1e-6 and np.abs(a - b).max() <= tol * rms, (np.abs(a - b).max(), rms)
    eg, eo = gpu.snap_energy(), orc.snap_energy()
    assert abs(eg - eo) <= tol * max(abs(eo), float(n)), (eg, eo)
    gpu.close()


@pytest.mark.parametrize("J", [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
@pytest.mark.parametrize("kind", [0, 1])
def test_every_twojmax(J, kind):
    _compare(*_deck(J, (2, 2, 3), 3.1803, kind=kind, seed=J), 1e-12 if J <= 8 else 4e-12)


# cells and lattice constant: 16 to 1,296 atoms (tiles of 4, 8, 16 and 32 with
# full and partly filled last ones), 0, 8, 26 and about 73 neighbours
@pytest.mark.parametrize("cells,a", [((2, 2, 2), 3.1803), ((3, 3, 3), 2.3), ((5, 5, 7), 3.1803), ((6, 7, 8), 3.1803),
                                     ((8, 9, 9), 3.1803), ((3, 3, 3), 5.0), ((4, 4, 5), 4.0)])
@pytest.mark.parametrize("nelem,switchflag", [(1, 1), (2, 1), (1, 0)])
def test_tile_and_neighbour_counts(cells, a, nelem, switchflag):
    _compare(*_deck(6, cells, a, nelem=nelem, switchflag=switchflag, seed=sum(cells)), 1e-12)


def test_mixed_form_of_large_twojmax_and_full_tiles():
    """RMS force error of the mixed form, with tables beyond twojmax 8 and tiles of 32 atoms."""
    from examinimd_gb300 import EMD_PREC_MIXED, Context
    for J, cells in ((10, (3, 3, 3)), (8, (9, 9, 9))):
        st, state = _deck(J, cells, 3.1803, seed=J)
        n = len(state["x"])
        f = []
        for prec in (0, EMD_PREC_MIXED):
            c = Context(0)
            mdloop.init(c, st, state, precision=prec)
            f.append(c.get(0, n)["f"])
            c.close()
        assert np.sqrt(np.mean((f[1] - f[0]) ** 2)) <= 1e-5 * np.sqrt(np.mean(f[0] ** 2))


@pytest.mark.parametrize("J", [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_mixed_form_of_every_twojmax(J):
    """RMS force error of the mixed form; 54 atoms, about 73 neighbours (three 32-lane rounds) or 26."""
    from examinimd_gb300 import EMD_PREC_MIXED, Context
    for a in (2.3, 3.1803):
        st, state = _deck(J, (3, 3, 3), a, seed=J)
        n = len(state["x"])
        f = []
        for prec in (0, EMD_PREC_MIXED):
            c = Context(0)
            mdloop.init(c, st, state, precision=prec)
            f.append(c.get(0, n)["f"])
            c.close()
        assert np.sqrt(np.mean((f[1] - f[0]) ** 2)) <= 1e-5 * np.sqrt(np.mean(f[0] ** 2))


def test_threads_with_systems_of_different_size():
    """Contexts of different size on several host threads at once: every force
    equals the one computed alone, to the scatter's order of adds."""
    from examinimd_gb300 import Context
    decks = [_deck(6, (2 + k % 4, 2 + k % 3, 3), 3.1803, seed=k) for k in range(12)]

    def force(deck):
        st, state = deck
        c = Context(0)
        out = []
        mdloop.init(c, st, state)
        for _ in range(4):
            c.zero_forces()
            c.snap_compute()
            c.comm_update_force()
            out.append(c.get(0, len(state["x"]))["f"])
        c.close()
        return out

    alone = [force(d)[0] for d in decks]
    with ThreadPoolExecutor(6) as ex:
        for ref, got in zip(alone, ex.map(force, decks)):
            for f in got:
                assert np.abs(f - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("J,nelem", [(0, 1), (4, 3), (8, 2), (10, 1)])
@pytest.mark.parametrize("precision", [0, 1])
def test_new_coefficients_are_those_of_a_new_potential(J, nelem, precision):
    """emd_snap_set_beta against emd_snap_init with the same coefficients: the same
    forces to the scatter's order of adds, the same energy."""
    from examinimd_gb300 import Context
    st, state = _deck(J, (3, 3, 3), 3.1803, nelem=nelem, seed=J)
    n = len(state["x"])
    new = np.array([[b * (1.0 + 0.3 * k) + 0.01 for b in e["beta"]] for k, e in enumerate(st.elements)])
    a, b = Context(0), Context(0)
    mdloop.init(a, st, state, precision=precision)
    a.snap_set_beta(new)
    for e, row in zip(st.elements, new):
        e["beta"] = list(row)
    mdloop.init(b, st, state, precision=precision)
    a.zero_forces()
    a.snap_compute()
    a.comm_update_force()
    fa, fb = a.get(0, n)["f"], b.get(0, n)["f"]
    assert np.abs(fa - fb).max() <= 1e-13 * np.abs(fb).max()
    assert a.snap_energy() == b.snap_energy()
    a.close()
    b.close()
