"""The CCD's far limit (pamo_b200/csrc/distance.cuh, built for the host): the FP64
first step of a contact block that is skipped by its float axis gap is beyond 1, on
random blocks of all sizes and on slivers on both sides of the area at which the
classification turns to the nearest corner.  The classified float distance, which the
limit was held against before, skips some of those whose first step is not."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PT, EE = 3, 4
SLACK, THICK, EE_THRES = 0.7, 1e-6, 1e-3  # the projection's defaults


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ccd") / "libccd_harness.so")
    src = os.path.join(ROOT, "tests", "native", "ccd_harness.cpp")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-w", "-I", os.path.join(cuda, "include"), src,
                    "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.h_ccd_far.restype = ctypes.c_float
    return lib


def _run(lib, x, p, kind, slack, thick):
    n = len(x)
    x, p = (np.ascontiguousarray(a, np.float32) for a in (x, p))
    d, gap, first = np.zeros(n, np.float32), np.zeros(n, np.float32), np.zeros(n)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    # the float parameters as the library holds them
    lib.h_blocks(ptr(x), ptr(p), ctypes.c_longlong(n), kind, ctypes.c_float(EE_THRES),
                 ctypes.c_double(np.float32(slack)), ctypes.c_double(np.float32(thick)), ptr(d), ptr(gap), ptr(first))
    return d, gap, first


def _far(lib, step, slack, thick, iters=100):
    return lib.h_ccd_far(ctypes.c_float(step), ctypes.c_float(slack), ctypes.c_float(thick), iters)


def _random_blocks(rng, n):
    size = 10.0 ** rng.uniform(-4, 0, (n, 1, 1))
    x = rng.random((n, 1, 3)) + size * rng.normal(size=(n, 4, 3))
    x[:, 0] += 10.0 ** rng.uniform(-4, 0, (n, 1)) * rng.normal(size=(n, 3))
    return x


def _slivers(rng, n):
    """A point over the middle of a triangle whose sine at x[1] lies about 1e-3, where
    the classification changes, within some float roundings of it."""
    u, w = rng.normal(size=(2, n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w -= (w * u).sum(1, keepdims=True) * u
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    L = 10.0 ** rng.uniform(-2, -0.5, (n, 1))
    sine = 1e-3 * (1 + rng.choice([-1e-2, -1e-5, -1e-7, 0, 1e-7, 1e-5, 1e-2], (n, 1)) * rng.random((n, 1)))
    a = rng.random((n, 3))
    b, c = a + L * u, a + 0.97 * L * (u + sine * w)
    top = a + 0.5 * L * (u + 0.5 * sine * w) + 10.0 ** rng.uniform(-5, -2, (n, 1)) * np.cross(u, w)
    return np.stack([top, a, b, c], 1)


@pytest.mark.parametrize("kind", [PT, EE])
@pytest.mark.parametrize("step", [0.0, 1e-7, 1e-5, 1e-4, 1e-3, 1e-2])
def test_skipped_blocks_are_done_in_fp64(harness, kind, step):
    rng = np.random.default_rng(kind)
    n = 60_000
    x = np.concatenate([_random_blocks(rng, n), _slivers(rng, n)])
    p = rng.normal(size=x.shape)
    p *= step / np.linalg.norm(p, axis=2, keepdims=True)  # every vertex moves by the bound: the worst
    p = p.astype(np.float32)
    bound = float(np.linalg.norm(p, axis=2).max())
    for slack, thick in ((SLACK, THICK), (0.9, 1e-4), (0.1, 0.0)):
        d, gap, first = _run(harness, x, p, kind, slack, thick)
        skip = gap > np.float32(_far(harness, bound, slack, thick))
        assert (first[skip] > 1).all()
        if 1e-4 <= step <= 1e-3 and (slack, thick) == (SLACK, THICK):
            assert skip.any()
    if kind == PT and step == 1e-3:
        d, gap, first = _run(harness, x, p, kind, SLACK, THICK)
        far = 4 * bound * 1.00001 / SLACK + THICK + 1e-5
        assert ((d * 0.99999 > far) & (first <= 1)).any()


def test_limits_that_skip_nothing(harness):
    for slack, iters in ((0.7, 0), (0.0, 100), (-0.5, 100), (float("nan"), 100)):
        assert _far(harness, 1e-3, slack, 1e-6, iters) > 1e38
    assert not 1e30 > _far(harness, float("nan"), 0.7, 1e-6)
