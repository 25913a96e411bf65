"""First column of the small dense exponential (csrc/pi_dense.cpp) against scipy, on the CPU."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest
import scipy.linalg

CSRC = Path(__file__).resolve().parent.parent / "permutationalinvariantdynamics.jl_gb300" / "csrc"

WRAPPER = """
#include "pi_dense.hpp"
extern "C" void column(int n, const double* a, double* out) {
  picuda::CMat A(n);
  for (int i = 0; i < n * n; ++i) A.a[i] = picuda::cd(a[2 * i], a[2 * i + 1]);
  const auto c = picuda::expm_column(A);
  for (int i = 0; i < n; ++i) out[2 * i] = c[i].real(), out[2 * i + 1] = c[i].imag();
}
"""


@pytest.fixture(scope="module")
def column(tmp_path_factory):
    d = tmp_path_factory.mktemp("expm")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "libexpm.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}", str(d / "w.cpp"),
                    str(CSRC / "pi_dense.cpp"), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).column

    def call(A):
        A = np.ascontiguousarray(A, dtype=np.complex128)
        out = np.zeros(len(A), dtype=np.complex128)
        fn(len(A), A.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p))
        return out

    return call


# one case per Pade degree, with repeated application (s <= 6) and with squaring before it
@pytest.mark.parametrize("norm", [1e-3, 0.1, 0.6, 1.7, 4.0, 20.0, 300.0, 2000.0])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 31, 122])
def test_first_column_matches_scipy(column, n, norm):
    rng = np.random.default_rng(n)
    A = np.triu(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), -1)  # upper Hessenberg
    A -= 1.5 * np.linalg.norm(A, 2) * np.eye(n)  # a decaying flow, as a projected Liouvillian's
    A *= norm / np.abs(A).sum(axis=0).max()
    ref = scipy.linalg.expm(A)[:, 0]
    # a few rounding errors of an n-term product for each unit of the norm, on both sides; below
    # the normal range (exp(-731) at norm 2000) rounding is absolute
    tol = 16 * n * np.finfo(float).eps * (1 + norm) * max(np.abs(ref).max(), np.exp(-norm)) + np.finfo(float).tiny
    assert np.abs(column(A) - ref).max() <= tol


def test_matrix_that_is_not_finite_gives_no_number(column):
    A = np.eye(4, dtype=np.complex128)
    A[1, 2] = np.inf
    assert np.isnan(column(A)).all()
