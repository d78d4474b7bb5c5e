"""The integer-pipe sine and cosine polynomials (simplediffeq.jl_gb300/csrc/
intpoly.h) against the Horner steps of fused multiply-adds they stand for: the
header compiled with g++ against fma(), over the reduced arguments' whole
range, short fractions (exact sums and ties) and both ends of the window."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "simplediffeq.jl_gb300", "csrc")

SHIM = r'''
#include <cmath>
#include "intpoly.h"
extern "C" void polys(const double* z, long n, double* ps, double* cr, double* ws, double* wc, unsigned char* decided) {
  const double S[] = {GBODE_SIN_C0, GBODE_SIN_C1, GBODE_SIN_C2, GBODE_SIN_C3, GBODE_SIN_C4, GBODE_SIN_C5};
  const double C[] = {GBODE_COS_C0, GBODE_COS_C1, GBODE_COS_C2, GBODE_COS_C3, GBODE_COS_C4, GBODE_COS_C5};
  for (long i = 0; i < n; ++i) {
    double s = S[0], c = C[0];
    for (int j = 1; j < 6; ++j) { s = std::fma(s, z[i], S[j]); c = std::fma(c, z[i], C[j]); }
    ws[i] = s;
    wc[i] = std::fma(z[i], c, 1.0);
    decided[i] = gbode::ip_sincos(z[i], ps + i, cr + i);
  }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("intpoly")
    src, so = d / "shim.cpp", d / "libshim.so"
    src.write_text(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    L = ctypes.CDLL(str(so))
    L.polys.argtypes = [ctypes.c_void_p, ctypes.c_long] + [ctypes.c_void_p] * 5
    return L


def run(lib, z):
    z = np.ascontiguousarray(z)
    out = [np.empty(z.size) for _ in range(4)] + [np.empty(z.size, dtype=np.uint8)]
    lib.polys(z.ctypes.data, z.size, *[o.ctypes.data for o in out])
    ps, cr, ws, wc, ok = out
    ok = ok.astype(bool)
    assert np.array_equal(ps[ok].view(np.uint64), ws[ok].view(np.uint64))
    assert np.array_equal(cr[ok].view(np.uint64), wc[ok].view(np.uint64))
    return ok


@pytest.mark.parametrize("kind", ["uniform", "small", "short", "single"])
def test_decided_arguments_are_the_fma_steps(lib, kind):
    rng = np.random.default_rng(len(kind))
    r = rng.uniform(-0.7854, 0.7854, 2000000)
    if kind == "small":
        r = np.ldexp(r, -rng.integers(0, 13, r.size))
    elif kind == "short":
        r = np.ldexp(1.0 + rng.integers(0, 8, r.size), -rng.integers(4, 16, r.size))
    elif kind == "single":
        r = r.astype(np.float32).astype(np.float64)
    ok = run(lib, r * r)
    if kind == "uniform":
        assert ok.mean() > 0.999


@pytest.mark.parametrize("z", [0.0, 5e-324, 2.0 ** -27, np.nextafter(2.0 ** -26, 0), 1.0, 4.0, np.inf, np.nan])
def test_arguments_outside_the_window_are_left_undecided(lib, z):
    assert not run(lib, np.full(3, z)).any()


def test_window_edges(lib):
    lo, hi = 2.0 ** -26, 0.6169
    z = np.concatenate([np.nextafter(lo, 1) + lo * np.linspace(0, 1, 100001), hi * (1 - np.ldexp(np.arange(100001.0), -53))])
    assert run(lib, z).mean() > 0.999
