"""Precision of the SNAP forms (GPU).

Mixed forces against the FP64 form's on jittered lattices of 128 (26 neighbours) and
54 (about 73) atoms.  The bounds, RMS error over RMS force of six systems each, are
the errors of a form whose U recursion and pair scalars are FP64 throughout and
whose Z, Y and pair forces are FP32: the mixed form's FP32 pairs are to be no worse.
"""
import numpy as np
import pytest

from tests import mdloop
from tests.test_gpu_snap_tables import _deck

pytestmark = pytest.mark.gpu


def _forces(st, state, precision):
    from examinimd_gb300 import Context
    c = Context(0)
    mdloop.init(c, st, state, precision=precision)
    f = mdloop.by_id(c.get(0, len(state["x"])))["f"]
    c.close()
    return f


@pytest.mark.parametrize("J,cells,a,bound", [
    (4, (4, 4, 4), 3.1803, 3.35e-7), (6, (4, 4, 4), 3.1803, 3.76e-7), (7, (4, 4, 4), 3.1803, 3.97e-7),
    (8, (4, 4, 4), 3.1803, 3.09e-7), (9, (4, 4, 4), 3.1803, 2.99e-7), (4, (3, 3, 3), 2.3, 1.70e-8),
    (6, (3, 3, 3), 2.3, 5.13e-8), (8, (3, 3, 3), 2.3, 8.20e-8), (9, (3, 3, 3), 2.3, 7.31e-8)])
def test_mixed_forces_are_as_good_as_with_fp64_recursions(J, cells, a, bound):
    from examinimd_gb300 import EMD_PREC_MIXED
    err = []
    for seed in range(6):
        deck = _deck(J, cells, a, seed=100 * J + seed)
        ref, got = _forces(*deck, 0), _forces(*deck, EMD_PREC_MIXED)
        err.append(np.mean((got - ref) ** 2) / np.mean(ref ** 2))
    assert np.sqrt(np.mean(err)) <= bound


@pytest.mark.parametrize("cells,a", [((4, 4, 4), 3.1803), ((3, 3, 3), 2.3)])
def test_mixed_repulsion_is_fp64(cells, a):
    """With zero coefficients only the r^-14 repulsion is left.  A pair's force takes
    ten FP64 roundings in either form and an atom adds up to 2 n of them, n neighbours'
    own and reactions, in another order."""
    from examinimd_gb300 import EMD_PREC_MIXED
    st, state = _deck(4, cells, a, seed=3)
    st.elements[0]["beta"] = list(np.zeros(len(st.elements[0]["beta"])))
    ref, got = _forces(st, state, 0), _forces(st, state, EMD_PREC_MIXED)
    L, x = np.asarray(st.domain), state["x"]
    shifts = np.stack(np.meshgrid(*[(-1, 0, 1)] * 3, indexing="ij"), -1).reshape(-1, 3) * L
    d = x[None, :, None, :] - x[:, None, None, :] + shifts
    r = np.linalg.norm(d, axis=-1).reshape(len(x), -1)
    near = (r > 0) & (r < st.cut)
    pair = np.where(near, 1.5e6 * np.where(near, r, 1.0) ** -13, 0.0).sum(axis=1)  # sum of |f_ij| of each atom
    n = near.sum(axis=1)
    tol = 2.0 ** -53 * (20 + 2 * n) * 2 * pair
    assert np.all(np.abs(got - ref).max(axis=1) <= tol)


@pytest.mark.parametrize("J", [10, 12, 14])
def test_bispectrum_of_large_twojmax(J):
    """The bispectrum summed over the atoms (the adjoint's energy part) against the
    oracle's layer recursion, whose own RMS relative error against long double is up to
    1.1e-15 on these systems; twice that is allowed between the two."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _deck(J, (3, 3, 3), 2.3, seed=J)
    n = len(state["x"])
    gpu, orc = Context(0), Oracle(4)
    mdloop.init(gpu, st, state)
    mdloop.init(orc, st, state)
    got = gpu.snap_adjoint(np.zeros((n, 3)), 1.0, 1, len(st.elements[0]["beta"])).ravel()[1:]
    ref = orc.snap_bispectrum().sum(axis=0)
    gpu.close()
    assert np.sqrt(np.mean((got / ref - 1.0) ** 2)) <= 2.2e-15


def test_mixed_forces_of_tungsten():
    """bcc tungsten, 2,000 atoms displaced by 0.05 A, coefficients of the benchmark: RMS
    error in eV/A below the 5.9e-6 of FP64 recursions."""
    from tests.golden.decks import snap_w_synthetic
    n = 10
    st = mdloop.SnapSetup(n, n, n, snap_w_synthetic(), lattice_style=2)
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = ((g[:, None, :] + np.array([[0, 0, 0], [0.5, 0.5, 0.5]])[None]) * st.a).reshape(-1, 3)
    x = np.mod(x + np.random.default_rng(8).normal(0.0, 0.05, x.shape), st.domain)
    state = dict(x=x, v=np.zeros_like(x), id=np.arange(1, len(x) + 1, dtype=np.int32), type=np.zeros(len(x), np.int32))
    from examinimd_gb300 import EMD_PREC_MIXED
    d = _forces(st, state, EMD_PREC_MIXED) - _forces(st, state, 0)
    assert np.sqrt(np.mean(np.sum(d * d, axis=1))) <= 5.9e-6


@pytest.mark.parametrize("J", [11, 12, 13, 14])
@pytest.mark.parametrize("a", [3.1803, 2.3])
def test_forces_of_the_largest_twojmax(J, a):
    """FP64 against the oracle (four times 1e-12, as for 9 and 10) and mixed against FP64."""
    from examinimd_gb300 import EMD_PREC_MIXED
    from oracle.orc import Oracle
    st, state = _deck(J, (3, 3, 3), a, seed=J)
    orc = Oracle(8)
    mdloop.init(orc, st, state)
    ref = mdloop.by_id(orc.get(0, len(state["x"])))["f"]
    got, mixed = _forces(st, state, 0), _forces(st, state, EMD_PREC_MIXED)
    rms = np.sqrt(np.mean(ref * ref))
    assert np.abs(got - ref).max() <= 4e-12 * rms
    assert np.sqrt(np.mean((mixed - got) ** 2)) <= 1e-5 * rms


@pytest.mark.parametrize("J", [1, 4, 7, 8, 9])
def test_mixed_pairs_past_their_own_cutoff(J):
    """Without switching a pair of the smaller element counts up to the larger one's cutoff,
    where theta0 exceeds pi; RMS force error of the mixed form."""
    from examinimd_gb300 import EMD_PREC_MIXED
    st, state = _deck(J, (3, 3, 3), 3.1803, nelem=2, switchflag=0, seed=J)
    st.elements[1]["radius"] = 0.38
    ref, got = _forces(st, state, 0), _forces(st, state, EMD_PREC_MIXED)
    assert np.sqrt(np.mean((got - ref) ** 2)) <= 1e-5 * np.sqrt(np.mean(ref ** 2))


@pytest.mark.parametrize("J", [2, 5, 8, 9])
def test_pairs_near_theta0_pi(J):
    """A pair of the smaller element where theta0 is within 1e-5 of pi (no switching): the
    reference's derivatives of (a, b) are differences of terms 1e5 times as large, off
    by some 1e-11 along (a, b), which the force does not depend on.  The force is smooth
    in the pair's distance, so over steps of 1e-9 of it second differences are
    roundings: four times 2^-53 of each of some 200 terms."""
    worst = 0.0
    for seed in range(4):
        rng = np.random.default_rng(100 * J + seed)
        st, _ = _deck(J, (6, 6, 6), 3.1803, nelem=2, switchflag=0, seed=J)
        st.elements[1]["radius"] = 0.46
        rcut = 2 * 0.46 * st.rcutfac
        u = rng.normal(size=3)
        pair = rcut / st.rfac0 * (1.0 + 1e-5 / np.pi * rng.choice([-1, 1])) * u / np.linalg.norm(u)
        x = [np.full(3, 9.0), 9.0 + pair]
        while len(x) < 14:
            y = rng.uniform(4.0, 15.0, 3)
            if min(np.linalg.norm(y - z) for z in x) > 2.4:
                x.append(y)
        n = len(x)
        types = np.where(np.arange(n) < 2, 1, rng.integers(0, 2, n)).astype(np.int32)
        f = []
        for k in range(-4, 5):
            x[1] = 9.0 + pair * (1.0 + 1e-9 * k)
            f.append(_forces(st, dict(x=np.array(x), v=np.zeros((n, 3)), id=np.arange(1, n + 1, dtype=np.int32),
                                      type=types), 0))
        f = np.array(f)
        worst = max(worst, np.abs(f[2:] - 2.0 * f[1:-1] + f[:-2]).max() / np.sqrt(np.mean(f[4] ** 2)))
    assert worst <= 1e-13
