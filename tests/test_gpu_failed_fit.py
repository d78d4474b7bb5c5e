"""A fit of the cost model that fails leaves the handle as it was: the model
fitted before stays in use for its problem, and none is in use for the other."""
import numpy as np
import pytest

from conftest import lorenz_inputs
from test_learned import USER_LORENZ

pytestmark = pytest.mark.gpu


def args_of(pkg, rhs, u0, p, schedule, maxiters=0):
    return pkg.make_args(pkg.GPUSimpleATsit5(), rhs, u0, p, (0.0, 10.0), 0.1, 1e-8, 1e-6, None, False, "fp64", schedule,
                         maxiters)


def test_the_fitted_model_stays(pkg):
    L = pkg._lib
    h = L.Handle(0)
    u0, p = lorenz_inputs(4096, seed=7)
    args = args_of(pkg, L.RHS["lorenz"], u0, p, "learned")
    h.learn_fit(args, {"epochs": 2})
    before = h.learn_predict(args, 4096)
    user = h.compile_rhs(USER_LORENZ, 3, 3)
    # one attempt a trajectory: none finishes, so there is nothing to fit
    for opts in ({"seed_dt0": 1}, {"hidden": 24}):
        with pytest.raises(pkg.GB300ODEError) as e:
            h.learn_fit(args_of(pkg, user, u0, p, "plain", maxiters=1), opts)
        assert e.value.code == L.EINVAL
        after = h.learn_predict(args, 4096)
        assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
        with pytest.raises(pkg.GB300ODEError) as e:
            h.learn_predict(args_of(pkg, user, u0, p, "plain"), 4096)
        assert e.value.code == L.ENOMODEL
    uf = np.empty((3, 4096))
    o = L.SolveOut()
    o.u_final = uf.ctypes.data
    h.check(h.solve_raw(args, o))
    h.close()
