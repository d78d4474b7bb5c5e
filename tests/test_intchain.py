"""The integer-pipe linear combinations (simplediffeq.jl_gb300/csrc/intchain.h,
introws.h) against the chain of fused multiply-adds they stand for: on the
host, the header compiled with g++ against fma(), over every row of the
tableau, stages of one scale and of scales up to the window's edge, sums that
cancel, exact ties, and zero, subnormal, infinite and NaN stages; on the GPU,
the kernels that use them against the oracle's device rounding, bit for bit."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "simplediffeq.jl_gb300", "csrc")

SHIM = r'''
#include <cmath>
#include "introws.h"
using namespace gbode;
static const auto T5 = ic_make_table<ic_count(kSpecT5)>(kSpecT5, kValT5);
static const auto V7 = ic_make_table<ic_count(kSpecV7)>(kSpecV7, kValV7);
static const auto V7X = ic_make_table<ic_count(kSpecV7X)>(kSpecV7X, kValV7X);
struct Row { const IcRow* row; const IcTerm* term; const double* coef; };
template <class T> static Row at(const T& t, int r) { return {&t.row[r], t.term + t.row[r].first, t.coef + t.row[r].first}; }
/* rows of Tsit5, Verner 7 and Verner 7's extra stages, one after another */
enum { N5 = sizeof(kSpecT5) / sizeof(kSpecT5[0]), N7 = sizeof(kSpecV7) / sizeof(kSpecV7[0]),
       N7X = sizeof(kSpecV7X) / sizeof(kSpecV7X[0]) };
static Row row_of(int r) { return r < N5 ? at(T5, r) : r < N5 + N7 ? at(V7, r - N5) : at(V7X, r - N5 - N7); }
extern "C" {
int nrows() { return N5 + N7 + N7X; }
int nterms(int r) { return row_of(r).row->n; }
double coef(int r, int j) { return row_of(r).coef[j]; }
/* k[n][m]: the chain of row r for each column, as the integer pipe and as fma; undecided columns flagged */
void chain(int r, const double* k, long m, double* got, double* want, unsigned char* decided) {
  const Row R = row_of(r);
  const IcRow& row = *R.row;
  for (long i = 0; i < m; ++i) {
    IcSpan E = ic_span(k[i]);
    for (int j = 1; j < row.n; ++j) ic_widen(E, k[(long)j * m + i]);
    IcSum S = {0u, 0u, 0u, false};
    double s = 0.0;
    for (int j = 0; j < row.n; ++j) {
      const double kv = k[(long)j * m + i], c = R.coef[j];
      ic_add_product(S, ic_product(R.term[j], kv, E));
      s = j ? std::fma(c, kv, s) : c * kv;
    }
    decided[i] = !S.bad && ic_in_window(E, row.shift);
    got[i] = ic_result(S, E, row.emax);
    want[i] = s;
  }
}
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("intchain")
    src, so = d / "shim.cpp", d / "libshim.so"
    src.write_text(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    L = ctypes.CDLL(str(so))
    L.coef.restype = ctypes.c_double
    L.chain.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_long] + [ctypes.c_void_p] * 3
    return L


def run(lib, r, k):
    k = np.ascontiguousarray(k)
    m = k.shape[1]
    got, want, ok = np.empty(m), np.empty(m), np.empty(m, dtype=np.uint8)
    lib.chain(r, k.ctypes.data, m, got.ctypes.data, want.ctypes.data, ok.ctypes.data)
    return got, want, ok.astype(bool)


def stages(rng, n, m, spread, bits=52):
    """n x m doubles, exponents within `spread` of one another, signs mixed, the low 52 - bits fraction bits zero."""
    e = rng.integers(1023 - spread, 1024, (n, m)).astype(np.uint64) + rng.integers(-200, 200, m).astype(np.uint64)
    f = rng.integers(0, 1 << 52, (n, m), dtype=np.uint64) & np.uint64((1 << 52) - (1 << (52 - bits)))
    return ((rng.integers(0, 2, (n, m)).astype(np.uint64) << np.uint64(63)) | (e << np.uint64(52)) | f).view(np.float64)


@pytest.mark.parametrize("spread", [0, 1, 5, 15, 31, 40])
@pytest.mark.parametrize("row", range(22))
def test_decided_rows_are_the_fma_chain(lib, row, spread):
    rng = np.random.default_rng(100 * row + spread)
    assert lib.nrows() == 22
    n = lib.nterms(row)
    got, want, ok = run(lib, row, stages(rng, n, 60000, spread))
    assert np.array_equal(got[ok].view(np.uint64), want[ok].view(np.uint64))
    if spread <= 5 and n > 1:
        assert ok.mean() > 0.99  # a sum of random terms rarely cancels 16 bits
    # nearly cancelling sums: the last stage makes the sum small, by 0 to 60 bits
    k = stages(rng, n, 60000, min(spread, 15))
    part = sum((lib.coef(row, j) * k[j] for j in range(n - 1)), np.zeros(k.shape[1]))
    k[n - 1] = -part / lib.coef(row, n - 1) * (1 + np.ldexp(rng.uniform(-1, 1, k.shape[1]), -rng.integers(0, 60, k.shape[1])))
    got, want, ok = run(lib, row, k)
    assert np.array_equal(got[ok].view(np.uint64), want[ok].view(np.uint64))
    # short fractions: exact sums and ties
    got, want, ok = run(lib, row, stages(rng, n, 60000, spread, bits=2))
    assert np.array_equal(got[ok].view(np.uint64), want[ok].view(np.uint64))


@pytest.mark.parametrize("value", [0.0, -0.0, 5e-324, 1e-310, np.inf, -np.inf, np.nan])
def test_special_stages_are_left_undecided(lib, value):
    rng = np.random.default_rng(7)
    for row in range(lib.nrows()):
        n = lib.nterms(row)
        for j in range(n):
            k = stages(rng, n, 64, 2)
            k[j] = value
            assert not run(lib, row, k)[2].any()
    assert not run(lib, 1, np.ldexp(rng.uniform(1, 2, (2, 64)), -850))[2].any()  # near the subnormals


def big_enough(pkg):
    """An odd ensemble size just past where the integer-pipe kernels are chosen (crowded() in ode_capi.cu)."""
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 256 + 37


@pytest.mark.gpu
@pytest.mark.parametrize("rhs,dim", [("lorenz", 3), ("linear", 2), ("linear", 4), ("linear", 5), ("resting", 3)])
@pytest.mark.parametrize("schedule,nsave", [("persistent", 0), ("persistent", 9), ("plain", 5)])
def test_kernels_are_bit_identical(pkg, po, rhs, dim, schedule, nsave):
    n = big_enough(pkg)
    rng = np.random.default_rng(dim + nsave)
    if rhs == "lorenz":
        u0 = rng.uniform(-1, 1, (3, n)) + np.array([[0], [0], [20.0]])
        p = np.stack([np.full(n, 10.0), rng.uniform(0, 30, n), np.full(n, 8 / 3)])
    else:
        u0 = rng.uniform(-1, 1, (dim, n))
        p = rng.normal(0, 1, (dim * dim, n)) - np.eye(dim).reshape(-1, 1)
        if rhs == "resting":
            p[:dim] = 0.0  # a component whose stages are all zero, in every other trajectory's warp or in all
            p[:dim, : n // 2] = rng.normal(0, 1, (dim, n // 2))
            u0[1, ::3] = 0.0
    name = "lorenz" if rhs == "lorenz" else "linear"
    sv = np.linspace(0, 2, nsave) if nsave else None
    kw = dict(abstol=1e-8, reltol=1e-6, saveat=sv)
    ep = pkg.EnsembleProblem(pkg.ODEProblem(name, u0[:, 0], (0.0, 2.0), p[:, 0]), u0s=u0, ps=p)
    a = pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=n, dt=0.1, schedule=schedule, **kw)
    b = po.solve("ATsit5", name, u0, p, (0.0, 2.0), 0.1, rounding="device", nthreads=os.cpu_count(), **kw)
    assert np.array_equal(a.naccept, b["naccept"]) and np.array_equal(a.nreject, b["nreject"])
    assert np.array_equal(a.u_final, b["u_final"])
    if nsave:
        assert np.array_equal(a.us, b["us"], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("rhs,dim,nsave", [("vanderpol", 2, 0), ("vanderpol", 2, 40), ("linear", 3, 0), ("linear", 3, 3)])
def test_verner7_kernels_are_bit_identical(pkg, po, rhs, dim, nsave):
    n = big_enough(pkg) * (3 if nsave else 1)
    rng = np.random.default_rng(dim + nsave)
    u0 = rng.uniform(-2, 2, (dim, n))
    p = np.exp(rng.uniform(np.log(0.1), np.log(10.0), (1, n)))
    if rhs == "linear":
        p = rng.normal(0, 1, (dim * dim, n)) - np.eye(dim).reshape(-1, 1)
        u0[:, ::5] = 0.0  # trajectories at rest: every stage zero
    sv = np.linspace(0, 1, nsave) if nsave else None
    kw = dict(abstol=1e-10, reltol=1e-8, saveat=sv)
    ep = pkg.EnsembleProblem(pkg.ODEProblem(rhs, u0[:, 0], (0.0, 1.0), p[:, 0]), u0s=u0, ps=p)
    a = pkg.solve(ep, pkg.GPUSimpleAVern7(), trajectories=n, dt=0.1, **kw)
    b = po.solve("AVern7", rhs, u0, p, (0.0, 1.0), 0.1, rounding="device", nthreads=os.cpu_count(), **kw)
    assert np.array_equal(a.naccept, b["naccept"]) and np.array_equal(a.nreject, b["nreject"])
    assert np.array_equal(a.u_final, b["u_final"])
    if nsave:
        assert np.array_equal(a.us, b["us"], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("controller", ["fp64", "fp32"])
def test_kernels_with_other_controllers(pkg, po, controller):
    n = big_enough(pkg)
    rng = np.random.default_rng(11)
    u0 = rng.uniform(-1, 1, (3, n)) + np.array([[0], [0], [20.0]])
    p = np.stack([np.full(n, 10.0), rng.uniform(0, 30, n), np.full(n, 8 / 3)])
    ep = pkg.EnsembleProblem(pkg.ODEProblem("lorenz", u0[:, 0], (0.0, 1.0), p[:, 0]), u0s=u0, ps=p)
    a = pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=n, dt=0.1, abstol=1e-8, reltol=1e-6, controller=controller)
    b = po.solve("ATsit5", "lorenz", u0, p, (0.0, 1.0), 0.1, rounding="device", controller=controller, abstol=1e-8,
                 reltol=1e-6, nthreads=os.cpu_count())
    assert np.array_equal(a.naccept, b["naccept"]) and np.array_equal(a.u_final, b["u_final"])
