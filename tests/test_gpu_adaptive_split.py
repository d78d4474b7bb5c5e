"""Adaptive Tsit5 with a trajectory's components over the warps of a block
(run_adaptive_split) against the oracle's device rounding, bit for bit: sizes
around a block's 32 trajectories and the rule's last one, dimensions 2 to 8,
save points (none, the start among them, more than one a step, never reached),
both layouts, every controller, every step, early stops."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def inputs(rhs, dim, n):
    rng = np.random.default_rng(1000 * dim + n)
    u0 = rng.uniform(-1, 1, (dim, n))
    if rhs == "lorenz":
        return u0 + np.array([[0], [0], [20.0]]), np.stack([np.full(n, 10.0), rng.uniform(0, 30, n), np.full(n, 8 / 3)])
    if rhs == "vanderpol":
        return u0, np.exp(rng.uniform(np.log(0.1), np.log(10.0), (1, n)))
    return u0, rng.normal(0, 1, (dim * dim, n)) - np.eye(dim).reshape(-1, 1)


def both(pkg, po, rhs, dim, n, tf=2.0, expect="adaptivesplit", **kw):
    u0, p = inputs(rhs, dim, n)
    ep = pkg.EnsembleProblem(pkg.ODEProblem(rhs, u0[:, 0], (0.0, tf), p[:, 0]), u0s=u0, ps=p)
    tol = dict(abstol=1e-8, reltol=1e-6)
    a = pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=n, dt=0.1, throw=False, **tol, **kw)
    assert pkg._lib.KERNEL[a.stats.kernel] == expect
    kw.pop("layout", None)
    b = po.solve("ATsit5", rhs, u0, p, (0.0, tf), 0.1, rounding="device", **tol, **kw)
    for k in ("u_final", "t_final", "retcode", "naccept", "nreject"):
        assert np.array_equal(getattr(a, k), b[k]), k
    assert a.stats.attempts == int((b["naccept"] + b["nreject"]).sum())
    if kw.get("saveat") is not None:
        assert np.array_equal(a.us, b["us"], equal_nan=True)


@pytest.mark.parametrize("nsave", [0, 2, 60])
@pytest.mark.parametrize("n", [1, 31, 33, 500])
@pytest.mark.parametrize("rhs,dim", [("lorenz", 3), ("vanderpol", 2), ("linear", 5)])
def test_bit_identical(pkg, po, rhs, dim, n, nsave):
    both(pkg, po, rhs, dim, n, saveat=np.linspace(0, 2.0, nsave) if nsave else None)


@pytest.mark.parametrize("past", [0, 1])
def test_last_size(pkg, po, past):
    import torch
    n = torch.cuda.get_device_properties(0).multi_processor_count * 32 + past
    both(pkg, po, "lorenz", 3, n, saveat=np.array([0.5, 3.0]), layout="traj",
         expect="staged" if past else "adaptivesplit")


@pytest.mark.parametrize("controller", ["fp64", "fp32"])
def test_controllers(pkg, po, controller):
    both(pkg, po, "lorenz", 3, 77, saveat=np.linspace(0, 2, 5), controller=controller)


@pytest.mark.parametrize("maxiters,tf", [(1, 2.0), (20, 2.0), (0, 0.0)])
def test_early_ends(pkg, po, maxiters, tf):
    both(pkg, po, "lorenz", 3, 100, tf=tf, maxiters=maxiters)


def test_every_step(pkg):
    u0, p = inputs("lorenz", 3, 70)
    ep = pkg.EnsembleProblem(pkg.ODEProblem("lorenz", u0[:, 0], (0.0, 1.0), p[:, 0]), u0s=u0, ps=p)
    a, b = [pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=70, dt=0.1, abstol=1e-8, reltol=1e-6, schedule=s,
                      save_everystep=True) for s in ("plain", "persistent")]
    assert np.array_equal(a.offsets, b.offsets)
    assert np.array_equal(a.ts_rows, b.ts_rows) and np.array_equal(a.us_rows, b.us_rows)
