"""The persistent schedules' warps merge when the ensemble runs out (Feed in
csrc/ode_solver.cuh): results of ensembles large enough for it against the
plain schedule, which keeps every trajectory on its thread, bit for bit:
controllers, drivers (unstaged, staged), stages in shared memory and in
registers, trajectories of very different lengths, early stops, and ensembles
that finish at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 41003  # odd, and more than two warps on each SM sub-partition


def inputs(rhs, n, rng):
    if rhs == "lorenz":
        u0 = rng.uniform(-1, 1, (3, n)) + np.array([[0], [0], [20.0]])
        return u0, np.stack([np.full(n, 10.0), rng.uniform(0, 30, n), np.full(n, 8 / 3)])
    if rhs == "vanderpol":
        return rng.uniform(-2, 2, (2, n)), np.exp(rng.uniform(np.log(0.1), np.log(20.0), (1, n)))
    return rng.uniform(0, 2 * np.pi, (5, n)), np.vstack([rng.normal(0, 1, (5, n)), rng.uniform(0, 4, (1, n))])


CASES = [("lorenz", "ds", 0, 3.0), ("lorenz", "ds", 11, 3.0), ("lorenz", "fp64", 7, 2.0), ("lorenz", "fp32", 0, 2.0),
         ("vanderpol", "ds", 9, 4.0), ("kuramoto", "ds", 6, 4.0), ("kuramoto", "ds", 0, 4.0), ("kuramoto", "fp64", 3, 2.0)]


@pytest.mark.parametrize("rhs,controller,nsave,tf", CASES)
def test_merged_warps_keep_results(pkg, rhs, controller, nsave, tf):
    rng = np.random.default_rng(len(rhs) + nsave)
    u0, p = inputs(rhs, N, rng)
    sv = np.linspace(0, tf, nsave) if nsave else None
    ep = pkg.EnsembleProblem(pkg.ODEProblem(rhs, u0[:, 0], (0.0, tf), p[:, 0]), u0s=u0, ps=p)
    sols = [pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=N, dt=0.1, saveat=sv, controller=controller,
                      schedule=s, throw=False, abstol=1e-8, reltol=1e-6) for s in ("plain", "persistent", "persistent")]
    a = sols[0]
    for b in sols[1:]:
        for k in ("u_final", "t_final", "retcode", "naccept", "nreject", "dt_first"):
            assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=k in ("u_final", "dt_first")), k
        if nsave:
            assert np.array_equal(a.us, b.us, equal_nan=True)
        assert a.stats.attempts == b.stats.attempts and a.stats.saves == b.stats.saves


@pytest.mark.parametrize("tf,maxiters", [(0.0, 0), (3.0, 40), (3.0, 1)])
def test_early_ends(pkg, tf, maxiters):
    """Every trajectory done at the start, and attempt caps that stop most or all of them."""
    u0, p = inputs("lorenz", N, np.random.default_rng(3))
    ep = pkg.EnsembleProblem(pkg.ODEProblem("lorenz", u0[:, 0], (0.0, tf), p[:, 0]), u0s=u0, ps=p)
    a, b = [pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=N, dt=0.1, abstol=1e-8, reltol=1e-6, schedule=s,
                      maxiters=maxiters, throw=False) for s in ("plain", "persistent")]
    for k in ("u_final", "t_final", "retcode", "naccept", "nreject"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert a.stats.attempts == b.stats.attempts


def test_every_step_output(pkg):
    u0, p = inputs("lorenz", N, np.random.default_rng(5))
    ep = pkg.EnsembleProblem(pkg.ODEProblem("lorenz", u0[:, 0], (0.0, 1.0), p[:, 0]), u0s=u0, ps=p)
    a, b = [pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=N, dt=0.1, abstol=1e-8, reltol=1e-6, schedule=s,
                      save_everystep=True) for s in ("plain", "persistent")]
    assert np.array_equal(a.offsets, b.offsets)
    assert np.array_equal(a.ts_rows, b.ts_rows) and np.array_equal(a.us_rows, b.us_rows)


@pytest.mark.parametrize("nsave", [0, 5])
@pytest.mark.parametrize("warps", [1.0, 1.001, 1.2, 1.4, 1.41, 2.0, 2.01])
def test_sizes_around_the_launch_rules(pkg, warps, nsave):
    """Ensembles of a given number of warps per SM sub-partition: where the persistent launch takes fewer warps than
    the trajectories fill, and where the crowded kernels begin."""
    import torch
    n = int(torch.cuda.get_device_properties(0).multi_processor_count * 128 * warps)
    u0, p = inputs("vanderpol", n, np.random.default_rng(9))
    sv = np.linspace(0, 2.0, nsave) if nsave else None
    ep = pkg.EnsembleProblem(pkg.ODEProblem("vanderpol", u0[:, 0], (0.0, 2.0), p[:, 0]), u0s=u0, ps=p)
    a, b = [pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=n, dt=0.1, abstol=1e-8, reltol=1e-6, saveat=sv, schedule=s)
            for s in ("plain", "persistent")]
    assert np.array_equal(a.u_final, b.u_final) and np.array_equal(a.naccept, b.naccept)
    if nsave:
        assert np.array_equal(a.us, b.us)
