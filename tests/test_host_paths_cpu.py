"""Host paths of the library on a CUDA runtime without a GPU (fake_cudart.cpp): what
the calls do with devices, limits and failing allocations.  No kernel runs."""
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

PRELUDE = """
import ctypes, numpy as np
from examinimd_gb300 import Batch, Context, EmdError, EMD_PREC_MIXED
from tests import mdloop
fake = ctypes.CDLL({so!r})
fake.fake_set_budget.argtypes = [ctypes.c_size_t]
fake.fake_held.restype = ctypes.c_size_t
fake.fake_seen.restype = ctypes.c_ulonglong
def current():
    d = ctypes.c_int()
    fake.cudaGetDevice(ctypes.byref(d))
    return d.value
def batch(n=(40, 30), box=9.0, device=0, **kw):
    x = np.random.default_rng(1).uniform(0.0, box, (sum(n), 3))
    return Batch(list(n), np.full((len(n), 3), box), x, 0.0 * x, device=device, **kw)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """run(code): the code in a process of its own, on the fake runtime."""
    from examinimd_gb300 import build
    cuda = build._cuda_home(build._nvcc())
    build.build()
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp")], check=True)

    def go(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE.format(so=so) + code], cwd=ROOT, capture_output=True, text=True,
                           env=dict(os.environ, LD_PRELOAD=so), timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
    return go


def test_a_batch_keeps_its_shared_memory_limit(run):
    """24^3 bins take 55 KB; the limit belongs to the kernel, not to the batch."""
    run("""
big = batch(box=62.0)
small = batch(box=9.0)
big.set_shape(512, 0)
for b in (big, small, big):
    b.run(40)
""")


@pytest.mark.parametrize("spl", [0, 20])
def test_a_batch_works_on_its_own_device(run, spl):
    """Whatever the calling thread's current device is, which stays as it was."""
    run(f"""
b = batch(device=1)
b.set_shape(512, {spl})
fake.cudaSetDevice(0)
b.get(); b.run(45); b.thermo(); b.tune(20); b.run(3); b.get(); b.info()
assert current() == 0 and fake.fake_wrong_device() == 0
held = fake.fake_held()
b.run(5); b.get()
assert fake.fake_held() == held
b.close()
assert fake.fake_held() == 0 and current() == 0
""")


def test_a_list_is_read_from_its_own_device(run):
    """The row starts of a list built without its total are formed when it is read."""
    run("""
setup = mdloop.LJSetup(4)
c = Context(1)
mdloop.init(c, setup, mdloop.make_lattice(setup))
assert c.lib.emd_neigh_create(c.h, 0, None) == 0
fake.cudaSetDevice(0)
c.neigh_get()
assert current() == 0 and fake.fake_wrong_device() == 0
""")


@pytest.mark.parametrize("precision", [0, 1])
def test_snap_works_in_smaller_chunks_where_memory_is_short(run, precision):
    """Work arrays for all atoms at once do not fit what is left: a call takes fewer atoms
    at a time, and fails only when those of 32 do not fit."""
    run(f"""
from tests.test_gpu_snap_tables import _deck
st, state = _deck(8, (28, 28, 28), 3.1803)
n, ncoeffall = len(state["x"]), len(st.elements[0]["beta"])
def held(compute):
    if not compute:
        st.force_compute = lambda b: None
    c = Context(0)
    mdloop.init(c, st, state, precision={precision})
    return c, fake.fake_held()
c, full = held(True)
c.close()
assert fake.fake_held() == 0
c, bare = held(False)
work = full - bare
assert work > 2000 * n
whole = int(1.25 * n * 8 * (1 + 3 + 2 * 125 + 1)) + 10000   # energies, dL/dF and the adjoint's sums of every atom
launches = []
for part in (1.2, 0.3, 0.1, 0.02):
    fake.fake_set_budget(int(bare + whole + part * work))
    l = fake.fake_launches()
    c.snap_compute()
    launches.append(fake.fake_launches() - l)
    c.snap_energy()
    if {precision} == 0:
        c.snap_adjoint(np.zeros((n, 3)), 1.0, 1, ncoeffall)
assert launches == sorted(launches) and launches[-1] > launches[0]
c.close()
c, bare = held(False)
fake.fake_set_budget(bare)
try:
    c.snap_compute()
    raise SystemExit("ran without memory")
except EmdError as e:
    assert "device allocation failed" in str(e)
fake.fake_set_budget(full)
c.snap_compute()
c.close()
assert fake.fake_held() == 0
""")


def test_a_batch_run_that_could_not_be_captured_changes_nothing(run):
    """The phased form's buffers alternate while a run is captured: if that fails, the
    positions are still where they were."""
    run("""
b = batch()
b.set_shape(512, 0)
fake.fake_watch(b"k_batch_pack", 2)
def positions():
    b.lib.emd_batch_get(b.h, np.empty(3 * 70).ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None, None)
    return fake.fake_seen()
p = positions()
fake.fake_fail_end_capture(1)
try:
    b.run(2)
    raise SystemExit("captured")
except EmdError:
    pass
assert positions() == p and b.info()["steps_done"] == 0
b.run(2)
assert positions() != p and b.info()["steps_done"] == 2
""")


def test_a_batch_without_room_for_more(run):
    """The phased form's second set of buffers and the packed read-back are extra: without
    room for them a run takes the persistent form, which gives the same bits, and the
    read-back copies system by system."""
    run("""
b = batch(n=(300, 200))
ref = b.get()
b.close()
b = batch(n=(300, 200))
b.set_shape(512, 0)
fake.fake_set_budget(fake.fake_held())
b.run(25)
got = b.get()
assert b.info()["steps_done"] == 25 and b.info()["steps_per_launch"] == 0
x = np.random.default_rng(1).uniform(0.0, 9.0, (500, 3))
np.testing.assert_array_equal(got[0], x)   # no kernel ran: what was put in
np.testing.assert_array_equal(got[1], 0.0 * x)
fake.fake_set_budget(2 ** 40)
b.run(25)
assert b.info()["steps_done"] == 50
""")


def test_bin_centres_after_a_failed_launch(run):
    """A box binned as before keeps its table of bin centres, unless the table was being
    replaced when the call failed."""
    run("""
c = Context(0)
setup = mdloop.LJSetup(4)
mdloop.init(c, setup, mdloop.make_lattice(setup))
fake.fake_watch(b"k_bin_ctab", 0)
def bins(width):
    c.binning_create(width, width, width, 1, True, True, False)
    return fake.fake_count()
assert bins(2.8) == 0 and bins(2.0) == 1 and bins(2.8) == 2 and bins(2.8) == 2
fake.fake_fail_launch(b"k_bin_ctab")
try:
    bins(0.5)
    raise SystemExit("launched")
except EmdError:
    pass
assert bins(2.8) == 3
""")


@pytest.mark.parametrize("how", ["arguments", "memory"])
def test_a_failed_snap_init_leaves_no_potential(run, how):
    """emd_snap_init that fails half way: later calls say so."""
    run(f"""
from tests.test_gpu_snap_tables import _deck
st, state = _deck(4, (3, 3, 3), 3.1803)
c = Context(0)
mdloop.init(c, st, state)
if {how!r} == "memory":
    fake.fake_set_budget(0)
else:
    st.elements[0]["beta"] = st.elements[0]["beta"][:-1]
try:
    st.force_init(c)
    raise SystemExit("initialised")
except EmdError:
    pass
fake.fake_set_budget(2 ** 40)
calls = [c.snap_compute, c.snap_energy, lambda: c.snap_adjoint(np.zeros((54, 3)), 1.0, 1, 15), c.snap_info]
for call in calls:
    try:
        call()
        raise SystemExit("went on")
    except EmdError as e:
        assert "not initialised" in str(e), e
st, state = _deck(4, (3, 3, 3), 3.1803)
st.force_init(c)
c.snap_compute()
c.close()
assert fake.fake_held() == 0
""")


def test_no_list_from_bins_without_a_halo_layer(run):
    """Rows read the 27 bins around each interior bin: without a layer of halo bins those
    of the outer ones do not exist."""
    run("""
c = Context(0)
setup = mdloop.LJSetup(4)
mdloop.init(c, setup, mdloop.make_lattice(setup))
c.binning_create(2.8, 2.8, 2.8, 0, True, True, False)
try:
    c.neigh_create(False)
    raise SystemExit("built")
except EmdError as e:
    assert "halo" in str(e)
c.binning_create(2.8, 2.8, 2.8, 1, True, True, False)
c.neigh_create(False)
""")
