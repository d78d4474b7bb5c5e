"""Routes into the crowded kernels (crowded() in csrc/ode_capi.cu) at the sizes
where they begin: the plain schedule with Verner 7, whose lanes interpolate
from stages in shared memory, against the oracle's device rounding; and a
user's right-hand side and output function against the built-in ones.  Bit for
bit."""
import os

import numpy as np
import pytest

from conftest import lorenz_inputs
from test_learned import USER_LORENZ

pytestmark = pytest.mark.gpu


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("nsave", [0, 20, 21, 100])
def test_verner7_plain(pkg, po, nsave):
    """More than 20 save points take the register kernel."""
    n = sms() * 640 + 13
    rng = np.random.default_rng(nsave)
    u0, p = rng.uniform(-2, 2, (2, n)), np.exp(rng.uniform(np.log(0.1), np.log(10.0), (1, n)))
    sv = np.linspace(0, 1, nsave) if nsave else None
    kw = dict(abstol=1e-10, reltol=1e-8, saveat=sv)
    ep = pkg.EnsembleProblem(pkg.ODEProblem("vanderpol", u0[:, 0], (0.0, 1.0), p[:, 0]), u0s=u0, ps=p)
    a = pkg.solve(ep, pkg.GPUSimpleAVern7(), trajectories=n, dt=0.1, schedule="plain", **kw)
    b = po.solve("AVern7", "vanderpol", u0, p, (0.0, 1.0), 0.1, rounding="device", nthreads=os.cpu_count(), **kw)
    assert np.array_equal(a.naccept, b["naccept"]) and np.array_equal(a.nreject, b["nreject"])
    assert np.array_equal(a.u_final, b["u_final"])
    if nsave:
        assert np.array_equal(a.us, b["us"], equal_nan=True)


@pytest.mark.parametrize("alg,warps", [("ATsit5", 2.01), ("AVern7", 5.02)])
@pytest.mark.parametrize("schedule", ["plain", "persistent"])
def test_user_code(pkg, alg, warps, schedule):
    n = int(sms() * 128 * warps)
    u0, p = lorenz_inputs(n, seed=17)
    alg = getattr(pkg, "GPUSimple" + alg)()
    kw = dict(trajectories=n, dt=0.1, abstol=1e-8, reltol=1e-6, schedule=schedule)
    user, builtin = [pkg.EnsembleProblem(pkg.ODEProblem(f, u0[:, 0], (0.0, 2.0), p[:, 0]), u0s=u0, ps=p)
                     for f in (pkg.UserRHS(USER_LORENZ, 3, 3), "lorenz")]
    sv = np.linspace(0, 2, 9)
    a, b = [pkg.solve(e, alg, saveat=sv, **kw) for e in (user, builtin)]
    assert a.stats.jit == 1
    assert np.array_equal(a.u_final, b.u_final) and np.array_equal(a.us, b.us) and np.array_equal(a.naccept, b.naccept)
    c = pkg.solve(user, alg, saveat=sv, output=pkg.UserOutput("out[0] = u[0] * u[1]; out[1] = t;", width=2), **kw)
    assert np.array_equal(c.us[:, 0], b.us[:, 0] * b.us[:, 1]) and (c.us[:, 1] == sv[:, None]).all()
    d, e = [pkg.solve(x, alg, **kw) for x in (user, builtin)]
    assert np.array_equal(d.u_final, e.u_final) and np.array_equal(d.u_final, b.u_final)
