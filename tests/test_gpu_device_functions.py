"""Arithmetic the kernels do themselves, against the operations it replaces (GPU):
the correctly rounded reciprocal of the LJ kernels against the divide, bit for bit,
and sine, cosine, reciprocal root and splitting of the 48-bit FP32 pairs against
NumPy's FP64 functions within the bounds they state."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    from examinimd_gb300 import build
    so = str(tmp_path_factory.mktemp("probe") / "libprobe.so")
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    "-o", so, os.path.join(ROOT, "tests", "kernels_probe.cu")], check=True)
    lib = ctypes.CDLL(so)

    def call(name, x):
        x = np.ascontiguousarray(x, np.float64)
        a, b = np.empty_like(x), np.empty_like(x)
        p = [v.ctypes.data_as(ctypes.c_void_p) for v in (x, a, b)]
        assert getattr(lib, "probe_" + name)(*p, len(x)) == 0
        return a, b
    return call


def test_reciprocal_is_the_divide(probe):
    rng = np.random.default_rng(1)
    m = rng.integers(0, 2 ** 52, 200000, dtype=np.uint64)
    m[:4000] = 2 ** 52 - 1 - np.arange(4000)   # significands at and near all ones
    m[4000:8000] = np.arange(4000)             # powers of two and just above
    parts = [((e + 1023).astype(np.uint64) << np.uint64(52) | m).view(np.float64) for e in (
        rng.integers(-96, 96, m.size), rng.integers(-6, 7, m.size), rng.integers(-1022, 1023, m.size))]
    # both sides of the quick path's ends, subnormals, zeros, infinities, NaN, negative values
    edge = [np.nextafter(2.0 ** e, s) for e in (-97, -96, -95, 95, 96, 97) for s in (0.0, np.inf)]
    edge += [2.0 ** e for e in (-1074, -1022, -97, -96, -95, 0, 95, 96, 97, 1023)]
    edge += [0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, -2.8, -2.0 ** 200, 5e-324, 1.7976931348623157e308]
    x = np.concatenate(parts + [np.array(edge)])
    y, ref = probe("recip", x)
    np.testing.assert_array_equal(np.isnan(y), np.isnan(ref))
    ok = ~np.isnan(ref)
    np.testing.assert_array_equal(y[ok].view(np.uint64), ref[ok].view(np.uint64))


def test_sine_and_cosine_of_pairs(probe):
    """Within 2^-44 of the values for angles up to a few hundred (angles the pair holds to
    2^-47 of themselves, which is allowed for)."""
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(0.0, 3.2, 200000), rng.uniform(-300.0, 300.0, 100000),
                        np.pi / 4 * np.arange(-40, 41), np.pi / 2 * np.arange(-40, 41) * (1 + 1e-9),
                        [0.0, -0.0, 1e-8, -1e-8, 1e-20]])
    s, c = probe("sincos", x)
    tol = 2.0 ** -44 + 2.0 ** -47 * np.abs(x)
    assert np.all(np.abs(s - np.sin(x)) <= tol) and np.all(np.abs(c - np.cos(x)) <= tol)


def test_reciprocal_root_and_splitting_of_pairs(probe):
    """The root within 2^-44 of itself (two 48-bit squares and one quadratic Newton step),
    the splitting within 2^-47."""
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(0.1, 50.0, 200000), 2.0 ** rng.uniform(-60.0, 100.0, 100000), 2.0 ** np.arange(-60.0, 101.0)])
    y, split = probe("rsqrt", x)
    assert np.abs(split / x - 1.0).max() <= 2.0 ** -47
    assert np.abs(y * np.sqrt(x) - 1.0).max() <= 2.0 ** -44
