"""Lane sums of double-float accumulators (csrc/pi_float.cuh), compiled for the CPU: the tree of 32 lanes
that the FP32 multi-dot uses.

Triple-float keeps hi and mid exact and rounds lo, which is at most 2^-48 of the sum of magnitudes, in
some 3 x 31 additions: below 2^-64 of that sum, plus two FP64 roundings of the result."""
import ctypes
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "permutationalinvariantdynamics.jl_gb300" / "csrc"

WRAPPER = """
#include "pi_float.cuh"
using namespace picuda;
extern "C" void accumulate(int n, const float* a, const float* b, float* out) {
  DF s{0.f, 0.f};
  for (int i = 0; i < n; ++i) df_add_prod(s, a[i], b[i]);
  out[0] = s.hi, out[1] = s.lo;
}
extern "C" double lane_sum(const float* v) {
  TF t[16];
  for (int i = 0; i < 16; ++i) t[i] = tf_pair(DF{v[2 * i], v[2 * i + 1]}, DF{v[2 * i + 32], v[2 * i + 33]});
  for (int off = 8; off >= 1; off /= 2)
    for (int i = 0; i < off; ++i) t[i] = tf_sum(t[i], t[i + off]);
  return tf_value(t[0]);
}
extern "C" double serial_sum(int n, const float* x) {
  TF s{0.f, 0.f, 0.f};
  for (int i = 0; i < n; ++i) tf_add(s, x[i]);
  return tf_value(s);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("floats")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "libfloats.so"
    # contraction of a product and a sum would change the exact error terms
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{CSRC}",
                    str(d / "w.cpp"), "-o", str(so)], check=True)
    out = ctypes.CDLL(str(so))
    out.lane_sum.restype = out.serial_sum.restype = ctypes.c_double
    return out


def fptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def vectors(kind, n, rng):
    x, y = rng.standard_normal((2, n)).astype(np.float32)
    if kind == "orthogonal":
        xd = x.astype(float)
        y = (y - (xd @ y) / (xd @ xd) * xd).astype(np.float32)
    elif kind == "decades":
        x = (x * 10.0 ** rng.uniform(-12, 0, n)).astype(np.float32)
    return x, y


@pytest.mark.parametrize("kind", ["normal", "orthogonal", "decades"])
@pytest.mark.parametrize("per_lane", [1, 4, 40])
def test_lane_sums_of_products(lib, kind, per_lane):
    rng = np.random.default_rng(per_lane)
    for _ in range(50):
        x, y = vectors(kind, 32 * per_lane, rng)
        v = np.zeros((32, 2), dtype=np.float32)
        for lane in range(32):
            a, b = np.ascontiguousarray(x[lane::32]), np.ascontiguousarray(y[lane::32])
            lib.accumulate(per_lane, fptr(a), fptr(b), fptr(v[lane]))
        got = lib.lane_sum(fptr(v))
        exact = math.fsum(v.astype(float).ravel())
        tol = 2.0**-52 * abs(exact) + 2.0**-64 * float(np.abs(v[:, 0].astype(float)).sum())
        assert abs(got - exact) <= tol


@pytest.mark.parametrize("kind", ["normal", "decades"])
def test_serial_sums(lib, kind):
    rng = np.random.default_rng(5)
    for n in (1, 7, 107, 1000):
        x, _ = vectors(kind, n, rng)
        exact = math.fsum(x.astype(float))
        tol = 2.0**-52 * abs(exact) + n * 2.0**-70 * float(np.abs(x.astype(float)).sum())
        assert abs(lib.serial_sum(n, fptr(x)) - exact) <= tol
