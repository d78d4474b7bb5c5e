"""Save points denser than a warp's staging ring holds: an iteration's points go
through it in several rounds (in single precision the lanes interpolate what
does not fit).  Against the oracle's device rounding, bit for bit: rings of the
crowded kernels, of one-warp blocks and of the prebuilt shapes, up to dozens of
points a step, and in bounds-check mode."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def inputs(rhs, dim, n):
    rng = np.random.default_rng(dim + n)
    if rhs == "lorenz":
        return rng.uniform(-1, 1, (3, n)) + 10, np.stack([np.full(n, 10.0), rng.uniform(0, 30, n), np.full(n, 8 / 3)])
    if rhs == "vanderpol":
        return rng.uniform(-2, 2, (2, n)), np.exp(rng.uniform(np.log(0.1), np.log(10.0), (1, n)))
    return rng.uniform(-1, 1, (dim, n)), rng.normal(0, 0.5, (dim * dim, n)) - np.eye(dim).reshape(-1, 1)


def check(pkg, po, alg, rhs, dim, n, nsave, precision="fp64", tf=1.0):
    u0, p = inputs(rhs, dim, n)
    sv = np.linspace(0, tf, nsave)
    kw = dict(abstol=1e-6, reltol=1e-5, saveat=sv, precision=precision)
    ep = pkg.EnsembleProblem(pkg.ODEProblem(rhs, u0[:, 0], (0.0, tf), p[:, 0]), u0s=u0, ps=p)
    a = pkg.solve(ep, getattr(pkg, "GPUSimple" + alg)(), trajectories=n, dt=0.1, **kw)
    assert pkg._lib.KERNEL[a.stats.kernel] == "staged" and a.stats.saves == n * (nsave - 1)
    b = po.solve(alg, rhs, u0, p, (0.0, tf), 0.1, rounding="device", nthreads=os.cpu_count(), **kw)
    assert np.array_equal(a.naccept, b["naccept"]) and np.array_equal(a.u_final, b["u_final"])
    assert np.array_equal(a.us, b["us"])


@pytest.mark.parametrize("alg,rhs,dim,nsave", [("ATsit5", "vanderpol", 2, 101), ("ATsit5", "lorenz", 3, 301),
                                               ("ATsit5", "linear", 4, 61), ("AVern7", "vanderpol", 2, 151)])
def test_crowded(pkg, po, alg, rhs, dim, nsave):
    import torch
    n = torch.cuda.get_device_properties(0).multi_processor_count * (256 if alg == "ATsit5" else 640) + 21
    check(pkg, po, alg, rhs, dim, n, nsave)


@pytest.mark.parametrize("nsave", [33, 400, 1501])
@pytest.mark.parametrize("alg,rhs,dim", [("ATsit5", "linear", 5), ("AVern7", "linear", 5), ("AVern9", "vanderpol", 2),
                                         ("AVern9", "linear", 4)])
def test_rings_of_about_a_round(pkg, po, alg, rhs, dim, nsave):
    check(pkg, po, alg, rhs, dim, 5003, nsave)


@pytest.mark.parametrize("precision", ["fp32", "fp32_kahan"])
@pytest.mark.parametrize("alg", ["ATsit5", "AVern7", "AVern9"])
def test_single_precision(pkg, po, alg, precision):
    check(pkg, po, alg, "vanderpol", 2, 1003, 900, precision)


@pytest.mark.parametrize("alg,rhs,dim", [("ATsit5", "linear", 6), ("AVern7", "linear", 5)])
def test_bounds_check_mode(pkg, alg, rhs, dim):
    L = pkg._lib
    n, nsave = 700, 400
    u0, p = inputs(rhs, dim, n)
    sv = np.linspace(0, 1.0, nsave)
    a = pkg.make_args(getattr(pkg, "GPUSimple" + alg)(), L.RHS[rhs], u0, p, (0.0, 1.0), 0.1, 1e-6, 1e-5, sv, False,
                      "fp64", "persistent", 0)
    res = []
    for check_mode in (True, False):
        h = L.Handle(0)
        h.set_bounds_check(check_mode)
        us = np.empty((nsave, dim, n))
        o = L.SolveOut()
        o.us = us.ctypes.data
        h.check(h.solve_raw(a, o))
        res.append(us)
        h.close()
    assert np.array_equal(*res)
