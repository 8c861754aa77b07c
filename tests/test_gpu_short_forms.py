"""Short forms the kernels use in place of a library call or a division, against
extended precision over the ranges they serve.

u = 2^-53. powTemp08: two roundings in y^5 reach the result by a fifth, the product
x y and the last addition round once each, the series stops below 0.1 u: 3 u.
powTemp17: four roundings in y^10 by a tenth and one of the corrected root, thrice
in its cube, and four products: 9 u. radDecay: the table's entry and the last
addition: 2.2 u; from 40 on it is 0, and e^-40 < 5e-18. vDivBy: the IEEE quotient."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from photon_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53


@pytest.fixture(scope="module")
def lib():
    src, so = os.path.join(ROOT, "tests", "cuda", "short_forms.cu"), os.path.join(build.BUILD, "short_forms.so")
    os.makedirs(build.BUILD, exist_ok=True)
    subprocess.run([build.NVCC] + build.ARCH + build.COMMON + ["--fmad=false", "-shared", src, "-o", so], check=True)
    return ctypes.CDLL(so)


def ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def relative(a, exact):
    return float(np.max(np.abs((a.astype(np.longdouble) - exact) / exact)))


def test_powers_of_a_temperature_ratio(lib):
    rng = np.random.default_rng(1)
    edges = [np.nextafter(v, d) for v in (0.25, 1.0, 32.0) for d in (0.0, 100.0)] + [0.25, 1.0, 32.0, 0.1, 100.0]
    x = np.concatenate([np.exp(rng.uniform(np.log(0.25), np.log(32.0), 2_000_000)), rng.uniform(200, 2300, 1_000_000) / 293.15,
                        1.0 + rng.uniform(-1e-6, 1e-6, 100_000), np.array(edges)])
    a, b = np.empty_like(x), np.empty_like(x)
    assert lib.temps(ptr(x), ctypes.c_longlong(len(x)), ptr(a), ptr(b)) == 0
    e = x.astype(np.longdouble)
    assert relative(a, e ** (np.longdouble(8) / 10)) <= 3 * U
    assert relative(b, e ** (np.longdouble(17) / 10)) <= 9 * U


def test_decay(lib):
    rng = np.random.default_rng(2)
    x = np.concatenate([np.exp(rng.uniform(np.log(1e-3), np.log(40.0), 2_000_000)), rng.uniform(1e-3, 2.0, 1_000_000),
                        np.arange(1, 512 * 57) * (np.log(2.0) / 1024), [1e-3, np.nextafter(40.0, 0.0)]])
    x = x[(x >= 1e-3) & (x < 40.0)]
    a = np.empty_like(x)
    assert lib.decay(ptr(x), ctypes.c_longlong(len(x)), ptr(a)) == 0
    assert relative(a, np.exp(-x.astype(np.longdouble))) <= 2.2 * U
    past = np.array([40.0, np.nextafter(40.0, 50.0), 700.0, 1e300, np.inf, np.nan])
    out = np.empty_like(past)
    assert lib.decay(ptr(past), ctypes.c_longlong(len(past)), ptr(out)) == 0
    assert (out[:5] == 0).all() and np.isnan(out[5])


def test_division_by_the_box(lib):
    rng = np.random.default_rng(3)
    n = 4_000_000
    d = np.exp(rng.uniform(np.log(1e-3), np.log(1e5), n)).astype(np.float32)
    x = (rng.choice([-1.0, 1.0], n) * np.exp(rng.uniform(np.log(1e-6), np.log(1e7), n))).astype(np.float32)
    k = n // 4   # products next to a rounding midpoint of the quotient
    q = rng.uniform(0.01, 100.0, k).astype(np.float32)
    x[:k] = ((q.astype(np.float64) + np.spacing(q) * 0.5) * d[:k]).astype(np.float32)
    x[k:k + 4] = [0.0, -0.0, 1.0, -1.0]
    f, r = np.empty_like(x), np.empty_like(x)
    assert lib.div_by(ptr(x), ptr(d), ctypes.c_longlong(n), ptr(f), ptr(r)) == 0
    assert np.array_equal(f, r)
