"""Halo, binning and reverse forces at the sizes where their kernels change, against
the CPU oracle: one CTA (up to 1,024 owned, 4,096 binned particles) and tiles of
1,024 (the last block scans 256 of them at a time), one CTA for up to 8,192
ghosts' forces and a cluster beyond.  GPU.
"""
import numpy as np
import pytest

from tests import mdloop

pytestmark = pytest.mark.gpu


def _gas(n, box, seed, half=False):
    rng = np.random.default_rng(seed)
    st = mdloop.LJSetup(1, half=half, newton=half)
    st.nx = st.ny = st.nz = 1
    st.a = box
    x = rng.uniform(0.0, box, (n, 3))
    x[: min(n, 3)] = 0.0  # on the faces
    return st, dict(x=x, v=rng.normal(size=(n, 3)), id=np.arange(1, n + 1, dtype=np.int32),
                    type=np.zeros(n, np.int32))


# box 6: about 6 ghosts an atom; box 12: 2; box 70: 300,000 atoms are 293 tiles
@pytest.mark.parametrize("n,box", [(1, 6.0), (65, 6.0), (590, 6.0), (1023, 12.0), (1024, 12.0), (1025, 12.0),
                                   (1400, 12.0), (4096, 18.0), (9000, 25.0), (300000, 70.0)])
def test_halo_and_binning_match_the_oracle(n, box):
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(n, box, n)
    out = []
    for b in (Context(0), Oracle()):
        b.system_init(st.masses, st.boltz, st.mvv2e, st.dt, st.domain)
        b.set_local(state["x"], state["type"], state["id"], v=state["v"])
        b.comm_init(st.neigh_cut)
        c = st.neigh_cut
        r = []
        for _ in range(2):  # the second time with the room the first one made
            b.comm_exchange()
            b.binning_create(c, c, c, 1, True, False, True)
            b.comm_exchange_halo()
            nb = b.binning_create(c, c, c, 1, True, True, False)
            info = b.info()
            nt = info[0] + info[1]
            g = b.get(0, nt)
            r += [np.asarray(info[:2]), g["x"], g["v"], g["id"], g["type"]]
            r += list(b.binning_get(int(np.prod(nb)), nt))
        out.append(r)
    for p, q in zip(*out):
        np.testing.assert_array_equal(p, q)


@pytest.mark.parametrize("n,box", [(700, 9.0), (9000, 25.0), (20000, 30.0), (40000, 38.0)])
def test_reverse_forces(n, box):
    """Half list with newton: ghosts' forces return to their owners; the sums are
    in another order than the oracle's, a few hundred terms rounded to 2^-53 each."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(n, box, 7 * n, half=True)
    out = []
    for b in (Context(0), Oracle()):
        mdloop.init(b, st, state)
        out.append(mdloop.by_id(b.get(0, n))["f"])
    scale = np.abs(out[1]).max()
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * scale


@pytest.mark.parametrize("half,prec", [(False, 0), (True, 0), (False, 1)])
def test_rows_of_crowded_bins(half, prec):
    """90 atoms a bin: every chunk of 32 centre atoms stages some 900 candidates, 256 at a
    time, and finds its own atoms among those carried over."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(3000, 9.0, 21, half=half)
    gpu, orc = Context(0), Oracle(4)
    tg, to = mdloop.init(gpu, st, state, precision=prec), mdloop.init(orc, st, state)
    assert tg == to
    for p, q in zip(gpu.neigh_get(tg), orc.neigh_get(to)):
        np.testing.assert_array_equal(p, q)
    gpu.close()


@pytest.mark.parametrize("half,prec", [(False, 0), (True, 0), (False, 1)])
@pytest.mark.parametrize("n,box", [(1, 9.0), (300, 30.0), (2500, 30.0), (8000, 35.0)])
def test_rows_of_a_gas(n, box, half, prec):
    """Empty bins, and bins with up to eight, nine and 32 candidates (0.2, 1.7 and 4 atoms a bin)."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(n, box, 5 * n, half=half)
    gpu, orc = Context(0), Oracle(4)
    tg, to = mdloop.init(gpu, st, state, precision=prec), mdloop.init(orc, st, state)
    assert tg == to
    for p, q in zip(gpu.neigh_get(tg), orc.neigh_get(to)):
        np.testing.assert_array_equal(p, q)
    gpu.close()


@pytest.mark.parametrize("n,lo,hi", [(140000, 42000, 50000), (170000, 50001, 60000)])
def test_reverse_forces_on_either_side_of_the_cluster(n, lo, hi):
    """Up to 50,000 ghosts one cluster, beyond a launch per phase (tolerance as above)."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(n, (n / 0.8442) ** (1.0 / 3.0), n, half=True)
    out = []
    for b in (Context(0), Oracle(8)):
        mdloop.init(b, st, state)
        assert lo <= b.info()[1] <= hi
        out.append(mdloop.by_id(b.get(0, n))["f"])
    scale = np.abs(out[1]).max()
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * scale
