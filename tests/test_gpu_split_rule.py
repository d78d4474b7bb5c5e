"""Which small adaptive ensembles take the component split (use_adaptive_split in
csrc/ode_capi.cu): each side of every line of the rule, with the results of the
plain schedule bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kernel(pkg, rhs, dim, n, nsave):
    rng = np.random.default_rng(dim * 100 + n + nsave)
    u0 = rng.uniform(-1, 1, (dim, n))
    p = rng.uniform(0.5, 2.0, (1, n)) if rhs == "vanderpol" else (
        rng.normal(0, 0.5, (dim * dim, n)) - np.eye(dim).reshape(-1, 1))
    sv = np.linspace(0, 1, nsave) if nsave else None
    ep = pkg.EnsembleProblem(pkg.ODEProblem(rhs, u0[:, 0], (0.0, 1.0), p[:, 0]), u0s=u0, ps=p)
    a, b = [pkg.solve(ep, pkg.GPUSimpleATsit5(), trajectories=n, dt=0.1, saveat=sv, schedule=s)
            for s in ("persistent", "plain")]
    assert np.array_equal(a.u_final, b.u_final)
    assert not nsave or np.array_equal(a.us, b.us)
    return pkg._lib.KERNEL[a.stats.kernel]


@pytest.mark.parametrize("rhs,dim,n,nsave,split", [
    ("linear", 2, 40, 32, True), ("linear", 2, 40, 33, False), ("vanderpol", 2, 40, 64, True),
    ("vanderpol", 2, 40, 65, False), ("linear", 3, 31, 100, True), ("linear", 3, 31, 101, False),
    ("linear", 3, 32, 101, True), ("linear", 8, 5, 101, False)])
def test_save_points(pkg, rhs, dim, n, nsave, split):
    assert kernel(pkg, rhs, dim, n, nsave) == ("adaptivesplit" if split else "staged")


@pytest.mark.parametrize("dim,nsave,warps", [(2, 0, 4), (2, 5, 2), (3, 5, 4), (5, 5, 4), (6, 0, 4), (6, 5, 2), (8, 5, 2)])
def test_last_size(pkg, dim, nsave, warps):
    """`warps` of an SM's four sub-partitions to have a warp each."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    last = 32 * (sms * (warps // dim) if dim <= 4 else sms * warps // dim)
    assert kernel(pkg, "linear", dim, last, nsave) == "adaptivesplit"
    assert kernel(pkg, "linear", dim, last + 1, nsave) == ("staged" if nsave else "persistent")
