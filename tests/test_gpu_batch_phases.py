"""The batch's phased form (rows by bin masks, force and integration in one kernel,
two sets of position buffers) against its persistent form (rows and force an atom
per thread, in place), which does the same arithmetic: equal bits.  GPU.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A = (4.0 / 0.8442) ** (1.0 / 3.0)
BASIS = np.array([(0, 0, 0), (0.5, 0.5, 0), (0.5, 0, 0.5), (0, 0.5, 0.5)])


def _system(cells, rng):
    g = np.stack(np.meshgrid(*[np.arange(k) for k in cells], indexing="ij"), -1).reshape(-1, 3)
    x = ((g[:, None, :] + BASIS[None]) * A).reshape(-1, 3)
    box = A * np.asarray(cells, float)
    x = np.mod(x + 0.05 * rng.standard_normal(x.shape), box)
    # atoms on the faces: bins of the first and the last layer, wraps either way
    x[0] = 0.0
    x[1, 2] = np.nextafter(box[2], 0.0)
    x[2, 1] = np.nextafter(box[1], 0.0)
    x[3, 0] = 0.0
    v = 1.2 * rng.standard_normal(x.shape)
    return x, v, box


@pytest.mark.parametrize("systems", [[(4, 4, 4)], [(4, 5, 9), (5, 4, 4), (11, 6, 4)], [(14, 13, 12), (4, 4, 4)]])
@pytest.mark.parametrize("runs", [(41,), (1, 2, 17, 20, 5)])
def test_phased_equals_persistent(systems, runs):
    from examinimd_gb300 import Batch
    rng = np.random.default_rng(11)
    parts = [_system(c, rng) for c in systems]
    ns = [len(p[0]) for p in parts]
    boxes = np.array([p[2] for p in parts])
    x, v = np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    out = []
    for threads, spl in ((256, 7), (512, 0)):
        b = Batch(ns, boxes, x, v, dt=0.0005)
        b.set_shape(threads, spl)
        for k in runs:
            b.run(k)
        out.append([*b.get(), *b.thermo()])
        b.close()
    assert np.all(np.isfinite(out[0][0]))
    for p, q in zip(*out):
        np.testing.assert_array_equal(p, q)


@pytest.mark.parametrize("spl", [7, 0])
@pytest.mark.parametrize("what", ["one_nan", "all_nan", "far", "inf"])
def test_a_blown_up_system_leaves_the_others_alone(spl, what):
    """NaN, infinite and far positions stay in their bins and images' bounds: the run
    goes on, and the other systems' bits are those of a run beside a sound system."""
    from examinimd_gb300 import Batch
    rng = np.random.default_rng(12)
    parts = [_system(c, rng) for c in ((5, 4, 4), (5, 5, 4), (4, 4, 4))]
    ns, boxes = [len(p[0]) for p in parts], np.array([p[2] for p in parts])
    x = np.concatenate([p[0] for p in parts])
    o = np.concatenate([[0], np.cumsum(ns)])
    out = []
    for bad in (False, True):
        v = np.concatenate([p[1] for p in parts])
        if bad and what == "one_nan":
            v[o[1] + 7] = np.nan
        elif bad and what == "all_nan":
            v[o[1]:o[2]] = -np.nan if spl else np.nan
        elif bad:
            v[o[1] + 7] = [1e300, -1e300, 1e25] if what == "inf" else [1e6, -1e6, 1e12]
        b = Batch(ns, boxes, x, v, dt=0.0005)
        b.set_shape(256, spl)
        b.run(45)
        out.append(b.get())
        b.close()
    for p, q in zip(*out):
        np.testing.assert_array_equal(p[:o[1]], q[:o[1]])
        np.testing.assert_array_equal(p[o[2]:], q[o[2]:])
    if what == "all_nan":
        assert np.all(np.isnan(out[1][0][o[1]:o[2]]))


def test_a_small_batch_leaves_a_large_one_its_shared_memory():
    """24^3 bins take 55 KB of shared memory, more than a kernel gets unasked; a batch
    with few bins, created in between, does not lower the limit."""
    from examinimd_gb300 import Batch
    rng = np.random.default_rng(13)
    box, n = 62.0, 8000
    g = np.stack(np.meshgrid(*[np.arange(20)] * 3, indexing="ij"), -1).reshape(-1, 3) * (box / 20)
    x, v = np.mod(g + 0.1 * rng.standard_normal((n, 3)), box), rng.standard_normal((n, 3))
    out = []
    for between in (False, True):
        b = Batch([n], np.full((1, 3), box), x, v)
        b.set_shape(512, 0)
        if between:
            xs, vs, bs = _system((4, 4, 4), rng)
            small = Batch([len(xs)], bs[None], xs, vs)
        b.run(25)
        out.append(b.get())
        b.close()
    small.close()
    for p, q in zip(*out):
        np.testing.assert_array_equal(p, q)


def test_bins_of_more_than_64_particles():
    """Bins of about 90: put in ascending order by one lane, so that no sum depends on
    the order in which the particles arrived (other CTA sizes, either form)."""
    from examinimd_gb300 import Batch
    rng = np.random.default_rng(14)
    a = 1.0  # fcc, four atoms per unit volume
    g = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = ((g[:, None, :] + BASIS[None]) * a).reshape(-1, 3)
    x = np.mod(x + 0.02 * rng.standard_normal(x.shape), 9 * a)
    v = rng.standard_normal(x.shape)
    out = []
    for threads, spl in ((256, 0), (1024, 0), (256, 10), (1024, 10)):
        b = Batch([len(x)], np.full((1, 3), 9 * a), x, v, dt=1e-7, max_neigh=512, every=2)
        b.set_shape(threads, spl)
        b.run(9)
        out.append(b.get())
        b.close()
    assert np.all(np.isfinite(out[0][2]))
    for o in out[1:]:
        for p, q in zip(out[0], o):
            np.testing.assert_array_equal(p, q)
