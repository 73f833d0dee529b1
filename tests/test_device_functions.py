"""The library's own scalar functions on the device, against values in extended precision."""

import ctypes
import os
import re
import subprocess
import sys

import numpy as np
import pytest
import torch

from pytential_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "device_functions.cu")
LIB = os.path.join(HERE, "_build", "libdevice_functions.so")
HEADERS = [os.path.join(build.CSRC, f) for f in ("common.cuh", "helmholtz.cuh")]

sys.path.insert(0, os.path.join(HERE, "golden"))
import make_hankel_pq as hankel  # noqa: E402


def _library():
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(map(os.path.getmtime, [SRC, *HEADERS])):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        tmp = f"{LIB}.{os.getpid()}"
        subprocess.run([build.NVCC, *build.ARCH, *build.FLAGS, "-shared", SRC, "-o", tmp, "-lcudart"],
                       check=True)
        os.replace(tmp, LIB)
    return ctypes.CDLL(LIB)


def _call(name, x, nout):
    a = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = [torch.empty_like(a) for _ in range(nout)]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = getattr(_library(), name)(len(x), *[ctypes.c_void_p(t.data_ptr()) for t in (a, *out)], stream)
    assert rc == 0
    return [t.cpu().numpy() for t in out]


def test_library_builds():
    _library()


def test_hankel_coefficients():
    """The table in the header is the one that the recipe gives."""
    with open(HEADERS[1]) as f:
        body = re.search(r"c_hankel_pq\[4\]\[13\] = \{(.*?)\n\};", f.read(), re.S).group(1)
    rows = [[float(v) for v in re.findall(r"-?\d[\d.]*(?:e-?\d+)?(?=,)", r)]
            for r in re.findall(r"\{([^{}]*)\}", re.sub(r"//.*", "", body))]
    want = hankel.coefficients()
    for name, row in zip(("P0", "Q0", "P1", "Q1"), rows, strict=True):
        # extended-precision rounding of the interpolation, amplified by the change of basis
        assert np.allclose(row, want[name], rtol=0, atol=1e-16), name


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(8.0, 8.001), (8.0, 25.0), (25.0, 200.0), (200.0, 1e5)])
def test_y01(lo, hi):
    x = np.geomspace(lo, hi, 50001)
    y0, y1 = _call("device_y01", x, 2)
    xl = x.astype(np.longdouble)
    s, c = np.sin(xl), np.cos(xl)
    a = 1 / np.sqrt(hankel.PI * xl)
    (p0, q0), (p1, q1) = hankel.pq(0, x), hankel.pq(1, x)
    amp = np.sqrt(2 / (np.pi * x))
    eps = 2.0 ** -53
    # amp (P sin + Q cos) with |P| < 1.01, |Q| < 0.01: sine and cosine within 2 eps each (CUDA's
    # sincos), their difference or sum (1.5 eps of sqrt 2), the polynomial (1.5), two products,
    # the sum and amp (root, division, product): below 10 roundings of the amplitude
    assert np.all(np.abs(y0 - a * (p0 * (s - c) + q0 * (s + c))) <= 10 * eps * amp)
    assert np.all(np.abs(y1 - a * (q1 * (s - c) - p1 * (s + c))) <= 10 * eps * amp)


@pytest.mark.gpu
def test_y01_against_scipy():
    """Across the library's range and this one: against AMOS (scipy's yv) where it is good to
    1e-13 of the amplitude; CUDA's y0 and y1 below 8 are good to a few units in the last place
    away from their zeros and to 1e-14 near them."""
    from scipy.special import hankel1
    x = np.linspace(0.05, 200.0, 100001)
    y0, y1 = _call("device_y01", x, 2)
    for nu, y in ((0, y0), (1, y1)):
        ref = hankel1(nu, x)
        assert np.all(np.abs(y - ref.imag) <= 1e-13 * np.abs(ref)), nu


def _rsqrt_arguments():
    rng = np.random.default_rng(0)
    # every upper word of [1, 4) (the approximation reads no more of x), lower words at
    # random; then all binades of the normal range
    top = np.arange(2 << 20, dtype=np.uint64) + (np.uint64(1023) << np.uint64(20))
    dense = (top << np.uint64(32) | rng.integers(0, 1 << 32, top.size, dtype=np.uint64)).view(float)
    e = rng.integers(-1022, 1024, 1 << 20)
    return np.concatenate([dense, np.ldexp(rng.uniform(1, 2, e.size), e)])


@pytest.mark.gpu
def test_rsqrt():
    x = _rsqrt_arguments()
    seed, h, lib = _call("device_rsqrt", x, 3)
    xl = x.astype(np.longdouble)
    root = np.sqrt(xl)
    assert float(np.abs(seed * root - 1).max()) <= 2.0 ** -18.4
    # the third-order step leaves 2.5 |seed error|^3 < 2^-54; x y, 1 - (x y) y, y e and the
    # last sum are rounded: below 2 units in the last place, like the library's
    ulp = np.spacing((1 / root).astype(float))
    assert float(np.abs((h - 1 / root) / ulp).max()) <= 2.0
    assert float(np.abs((h - lib) / ulp).max()) <= 3.0
