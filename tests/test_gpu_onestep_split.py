"""RK4 and Euler with a trajectory's components over the warps of a block
(run_onestep_split) against the oracle's device rounding, bit for bit: sizes
around a block's 32 trajectories and the last one the rule takes, dimensions
2 to 8, final states and every step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [False, True])
@pytest.mark.parametrize("rhs,dim", [("lorenz", 3), ("vanderpol", 2), ("linear", 5), ("linear", 4)])
@pytest.mark.parametrize("n", [1, 31, 33, 1000, "last"])
@pytest.mark.parametrize("alg", ["RK4", "Euler"])
def test_bit_identical(pkg, po, alg, n, rhs, dim, every):
    if n == "last":
        import torch
        n = torch.cuda.get_device_properties(0).multi_processor_count * 2 * 32
    rng = np.random.default_rng(n + dim)
    u0 = rng.uniform(-1, 1, (dim, n))
    p = {"lorenz": rng.uniform(1, 20, (3, n)), "vanderpol": rng.uniform(0.1, 3, (1, n))}.get(
        rhs, rng.normal(0, 1, (dim * dim, n)))
    ep = pkg.EnsembleProblem(pkg.ODEProblem(rhs, u0[:, 0], (0.0, 0.3), p[:, 0]), u0s=u0, ps=p)
    a = pkg.solve(ep, getattr(pkg, "GPUSimple" + alg)(), trajectories=n, dt=0.01, save_everystep=every)
    b = po.solve(alg, rhs, u0, p, (0.0, 0.3), 0.01, rounding="device", save_everystep=every)
    assert np.array_equal(a.u_final, b["u_final"]) and np.array_equal(a.t_final, b["t_final"])
    if every:
        assert np.array_equal(a.us, b["us"])
