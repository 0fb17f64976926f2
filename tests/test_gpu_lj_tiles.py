"""The FP64 LJ tiles (lj_fp64.cuh) where they can go wrong, against the CPU oracle (GPU).

Random gases: fewer rows than a tile, partly filled last tiles, rows whose
neighbours overflow a warp's list (dense gas), overlapping pairs, one shared
parameter set and 13 types with a table per pair (more than 12 types keep
separate parameters).  Full lists: forces bit for bit.  Half lists and the
energy sum in another order than the serial oracle: the terms of one sum are
rounded to 2^-53 each, a few thousand of them at most, so 1e-12 of the sum of
magnitudes bounds the difference.
"""
import numpy as np
import pytest

from tests import mdloop

pytestmark = pytest.mark.gpu


def _gas(n, box, ntypes, seed, half, kind):
    rng = np.random.default_rng(seed)
    kw = {}
    if ntypes > 1:
        kw = dict(masses=[1.0 + 0.1 * t for t in range(ntypes)],
                  coeffs=[(a, b, 0.5 + 0.1 * a + 0.05 * b, 0.9 + 0.01 * (a + b), 1.8 + 0.05 * ((a + b) % 15))
                          for a in range(1, ntypes + 1) for b in range(a, ntypes + 1)])
    st = mdloop.LJSetup(1, half=half, kind=kind, newton=half, **kw)
    st.nx = st.ny = st.nz = 1
    st.a = box
    state = dict(x=rng.uniform(0.0, box, (n, 3)), v=np.zeros((n, 3)), id=np.arange(1, n + 1, dtype=np.int32),
                 type=rng.integers(0, ntypes, n).astype(np.int32))
    return st, state


# atoms, box edge: rows of 1 (n = 1), about 8, 78 (liquid density) and 430
# (dense) entries; 7 and 9 rows are the tile sizes, 608 the schedulers
SIZES = [(1, 6.0), (2, 6.0), (7, 6.0), (10, 6.0), (64, 6.0), (611, 9.0), (4257, 17.0), (2500, 8.5)]


@pytest.mark.parametrize("n,box", SIZES)
@pytest.mark.parametrize("ntypes", [1, 13])
@pytest.mark.parametrize("half,kind", [(False, 0), (False, 1), (True, 0), (True, 1)])
def test_forces_and_energy_of_random_gases(n, box, ntypes, half, kind):
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(n, box, ntypes, 100 * n + ntypes, half, kind)
    gpu, orc = Context(0), Oracle()
    mdloop.init(gpu, st, state)
    mdloop.init(orc, st, state)
    a, b = gpu.get(0, n), orc.get(0, n)
    assert np.array_equal(a["id"], b["id"])
    if half:
        scale = np.abs(b["f"]).max()
        assert np.abs(a["f"] - b["f"]).max() <= 1e-12 * scale
    else:
        assert np.array_equal(a["f"], b["f"])
    eg, eo = gpu.lj_energy(), orc.lj_energy()
    # each shifted pair energy is a difference of terms below eps_max (r^-12 + 1)
    assert abs(eg - eo) <= 1e-12 * max(abs(eo), float(n))
    gpu.close()


@pytest.mark.parametrize("shift", [0.0, 4096.0])
def test_filter_far_from_the_origin(shift):
    """The FP32 filter's threshold grows with the coordinates: a gas placed in
    a box whose far corner lies thousands of cutoffs away loses no pair."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    n, edge = 700, 9.0
    box = [max(edge, shift + edge), edge, edge]
    rng = np.random.default_rng(3)
    x = rng.uniform(0.0, edge, (n, 3))
    x[:, 0] += shift
    st = mdloop.LJSetup(1)
    f = []
    for b in (Context(0), Oracle()):
        b.system_init(st.masses, 1.0, 1.0, st.dt, box)
        b.set_local(x, np.zeros(n, np.int32), np.arange(1, n + 1, dtype=np.int32))
        st.force_init(b)
        b.comm_init(2.8)
        b.neigh_init(0, 2.8, False)
        b.comm_exchange()
        b.binning_create(2.8, 2.8, 2.8, 1, True, False, True)
        b.comm_exchange_halo()
        b.binning_create(2.8, 2.8, 2.8, 1, True, True, False)
        b.neigh_create(False)
        b.zero_forces()
        b.lj_compute()
        f.append(b.get(0, n)["f"])
    assert np.array_equal(f[0], f[1])


@pytest.mark.parametrize("n", [300, 16384, 16385, 30000])
@pytest.mark.parametrize("ntypes", [1, 13])
@pytest.mark.parametrize("half", [False, True])
def test_gas_with_short_rows(n, ntypes, half):
    """One entry a row on average, none above nine: a thread per row for the energy, and
    for the forces of more than 16,384 atoms."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    st, state = _gas(n, (n / 0.011) ** (1.0 / 3.0), ntypes, n, half, 0)
    gpu, orc = Context(0), Oracle()
    total = mdloop.init(gpu, st, state)
    mdloop.init(orc, st, state)
    assert 0 < gpu.neigh_get(total)[0].max() <= 9
    a, b = gpu.get(0, n), orc.get(0, n)
    for again in range(2):  # the second time on top of the first one's forces
        if half:
            assert np.abs(a["f"] - b["f"]).max() <= 1e-12 * np.abs(b["f"]).max()
        else:
            assert np.array_equal(a["f"], b["f"])
        gpu.lj_compute()
        orc.lj_compute()
        a, b = gpu.get(0, n), orc.get(0, n)
    eg, eo = gpu.lj_energy(), orc.lj_energy()
    assert abs(eg - eo) <= 1e-12 * max(abs(eo), float(n))
    assert gpu.lj_energy_noalloc() == eg
    gpu.close()


def test_intensity_dial_with_short_rows():
    """One evaluation per pair is the plain force, divided by one."""
    import ctypes
    from examinimd_gb300 import Context
    n = 20000
    st, state = _gas(n, (n / 0.011) ** (1.0 / 3.0), 1, 9, False, 0)
    gpu = Context(0)
    mdloop.init(gpu, st, state)
    f = gpu.get(0, n)["f"]
    one = np.ones(1)
    assert gpu.lib.emd_lj_set_intensity(gpu.h, one.ctypes.data_as(ctypes.c_void_p)) == 0
    gpu.zero_forces()
    gpu.lj_compute()
    assert np.array_equal(gpu.get(0, n)["f"], f) and np.abs(f).max() > 0.0
    gpu.close()


@pytest.mark.parametrize("n,cut,half,by_rows", [(20000, 5.0, False, False), (20004, 5.0, False, True),
                                                (12500, 6.0, False, True), (20004, 5.0, True, True), (12500, 6.6, True, True)])
def test_rows_of_hundreds_of_entries(n, cut, half, by_rows):
    """Either side of the rule for long rows (full lists: above 250 entries from 20,001
    atoms, above 350 from 12,001; half lists above 160 and 300)."""
    from examinimd_gb300 import Context
    from oracle.orc import Oracle
    rng = np.random.default_rng(n)
    st = mdloop.LJSetup(1, half=half, newton=half, cut=cut - 0.3)
    st.nx = st.ny = st.nz = 1
    m = int(np.ceil(n ** (1.0 / 3.0)))
    st.a = m * 1.18  # a simple cubic lattice at about 0.6 of the volume's atoms, displaced
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = np.mod((g + 0.5) * 1.18 + 0.05 * rng.standard_normal((n, 3)), st.a)
    state = dict(x=x, v=np.zeros((n, 3)), id=np.arange(1, n + 1, dtype=np.int32), type=np.zeros(n, np.int32))
    gpu, orc = Context(0), Oracle(8)
    total = mdloop.init(gpu, st, state)
    mdloop.init(orc, st, state)
    longest = gpu.neigh_get(total)[0].max()
    lo = (160 if half else 250) if n > 20000 else (300 if half else 350)
    assert (longest > lo) == by_rows
    a, b = gpu.get(0, n), orc.get(0, n)
    if half:
        assert np.abs(a["f"] - b["f"]).max() <= 1e-12 * np.abs(b["f"]).max()
    else:
        assert np.array_equal(a["f"], b["f"])
    eg, eo = gpu.lj_energy(), orc.lj_energy_compensated()  # ten million terms: a serial sum is off by 1e-10
    assert abs(eg - eo) <= 1e-12 * max(abs(eo), float(n))
    gpu.close()
