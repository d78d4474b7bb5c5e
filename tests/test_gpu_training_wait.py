"""An exchange between the training kernel's thread blocks that runs out of time
ends the kernel with an error the host reads; the fitted model stays as it was
and the context usable."""
import numpy as np
import pytest

from conftest import lorenz_inputs
from test_mlp import params_for

pytestmark = pytest.mark.gpu


def test_the_wait_runs_out(pkg):
    L = pkg._lib
    h = L.Handle(0)
    u0, p = lorenz_inputs(4096, seed=7)
    args = pkg.make_args(pkg.GPUSimpleATsit5(), 0, u0, p, (0.0, 10.0), 0.1, 1e-8, 1e-6, None, False, "fp64", "learned", 0)
    rng = np.random.default_rng(1)
    x, y = rng.normal(size=(3000, 6)).astype(np.float32), rng.normal(size=(3000, 2)).astype(np.float32)
    prm = params_for(6, 64, 11)
    h.learn_fit(args, {"epochs": 2})
    fitted = h.learn_predict(args, 4096)
    grad = h.learn_gradcheck(6, 64, prm, x, y)
    h.learn_hold_exchanges(True)
    for call in (lambda: h.learn_fit(args, {"epochs": 2, "seed": 5}), lambda: h.learn_gradcheck(6, 64, prm, x, y)):
        with pytest.raises(pkg.GB300ODEError, match="ran out of time") as e:
            call()
        assert e.value.code == L.ECUDA
    kept = h.learn_predict(args, 4096)
    h.learn_hold_exchanges(False)
    again = h.learn_gradcheck(6, 64, prm, x, y)
    h.learn_fit(args, {"epochs": 2})
    refitted = h.learn_predict(args, 4096)
    for k in (0, 1):
        assert np.array_equal(fitted[k], kept[k]) and np.array_equal(fitted[k], refitted[k])
    assert np.array_equal(grad[0], again[0])
    h.close()
