"""Bounds-check mode on the kernels of both ends of the size range: ensembles
small enough for the component split, and large enough for the crowded
kernels, whose warps merge through the parking place.  No violation, every
trajectory started once, and the results of the unchecked kernels, which are
the same kind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def checked(pkg):
    h = pkg._lib.Handle(0)
    h.set_bounds_check(True)
    yield h
    h.close()


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def both(pkg, checked, alg, rhs, n, nsave, schedule, layout, expect):
    L = pkg._lib
    rng = np.random.default_rng(n + nsave)
    tf = 2.0
    if rhs == "lorenz":
        u0 = rng.uniform(-1, 1, (3, n)) + np.array([[0], [0], [20.0]])
        p = np.stack([np.full(n, 10.0), rng.uniform(0, 30, n), np.full(n, 8 / 3)])
    else:
        u0, p = rng.uniform(-2, 2, (2, n)), np.exp(rng.uniform(np.log(0.1), np.log(20.0), (1, n)))
    sv = np.linspace(0, tf, nsave) if nsave else None
    res = []
    for h in (checked, pkg._handle(0)):
        a = pkg.make_args(getattr(pkg, "GPUSimple" + alg)(), L.RHS[rhs], u0, p, (0.0, tf), 0.1, 1e-8, 1e-6, sv, False,
                          "fp64", schedule, 0, layout=layout)
        out = {"u_final": np.empty(u0.shape), "naccept": np.empty(n, dtype=np.int32)}
        if nsave:
            out["us"] = np.empty((n, nsave, len(u0)) if layout == "traj" else (nsave, len(u0), n))
        o, st = L.SolveOut(), L.SolveStats()
        for k, v in out.items():
            setattr(o, k, v.ctypes.data)
        assert h.solve_raw(a, o, st) == L.OK, h.error()
        assert L.KERNEL[st.kernel] == expect
        res.append(out)
    for k in res[0]:
        assert np.array_equal(res[0][k], res[1][k], equal_nan=True), k


@pytest.mark.parametrize("layout", ["soa", "traj"])
@pytest.mark.parametrize("rhs,n,nsave", [("lorenz", 1, 0), ("lorenz", 500, 17), ("vanderpol", 33, 9)])
def test_component_split(pkg, checked, rhs, n, nsave, layout):
    both(pkg, checked, "ATsit5", rhs, n, nsave, "persistent", layout, "adaptivesplit")


@pytest.mark.parametrize("alg,rhs,warps,nsave,schedule,layout,expect", [
    ("ATsit5", "lorenz", 2.05, 0, "persistent", "soa", "persistent"),
    ("ATsit5", "vanderpol", 2.7, 11, "persistent", "traj", "staged"),
    ("ATsit5", "lorenz", 2.05, 5, "plain", "soa", "plain"),
    ("AVern7", "vanderpol", 2.7, 0, "persistent", "soa", "persistent"),
    ("AVern7", "vanderpol", 5.3, 7, "persistent", "soa", "staged"),
    ("AVern7", "vanderpol", 5.3, 7, "plain", "soa", "plain")])
def test_crowded(pkg, checked, alg, rhs, warps, nsave, schedule, layout, expect):
    """`warps` trajectories' warps for every SM sub-partition: just past where the crowded kernels begin."""
    both(pkg, checked, alg, rhs, int(sms() * 128 * warps) + 5, nsave, schedule, layout, expect)
