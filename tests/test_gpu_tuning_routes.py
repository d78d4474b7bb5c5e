"""The autotuner at both ends of the size range: the component split, whose block
size is fixed and which has no staging ring, and the crowded kernels, which are
tuned, saved and loaded under keys of their own.  Results never change."""
import numpy as np
import pytest

from conftest import lorenz_inputs

pytestmark = pytest.mark.gpu


def solve(pkg, h, args, nsave, n):
    L = pkg._lib
    us, uf = np.empty((nsave, 3, n)), np.empty((3, n))
    o, st = L.SolveOut(), L.SolveStats()
    o.us, o.u_final = us.ctypes.data, uf.ctypes.data
    h.check(h.solve_raw(args, o, st))
    return us, uf, st


def round_trip(pkg, n, path):
    L = pkg._lib
    u0, p = lorenz_inputs(n, seed=5)
    sv = np.linspace(0, 2, 11)
    args = pkg.make_args(pkg.GPUSimpleATsit5(), 0, u0, p, (0.0, 2.0), 0.1, 1e-8, 1e-6, sv, False, "fp64", "persistent", 0)
    h1, h2, h3 = (L.Handle(0) for _ in range(3))
    rep = h1.autotune(args, sample=8192)
    h1.tune_save(path)
    assert h2.tune_load(path) == L.OK
    runs = [solve(pkg, h, args, len(sv), n) for h in (h1, h2, h3)]
    for us, uf, st in runs[:2]:
        assert np.array_equal(us, runs[2][0]) and np.array_equal(uf, runs[2][1])
        if rep.best_ms < rep.default_ms:
            assert st.jit == 1  # the chosen shape, compiled at run time
    for h in (h1, h2, h3):
        h.close()
    return rep, path.read_text().splitlines()[1:], runs[0][2]


def test_component_split(pkg, tmp_path):
    rep, keys, st = round_trip(pkg, 500, tmp_path / "split.txt")
    assert pkg._lib.KERNEL[st.kernel] == "adaptivesplit"
    assert rep.block == 96 and rep.stage_bytes == 0
    rows = rep.rows()
    assert len(rows) == rep.variants and {(b, s) for b, _, s, _ in rows} == {(96, 0)}
    assert [k.split()[0].split("|")[1] for k in keys] == ["adaptivesplit"]


def test_crowded(pkg, tmp_path):
    import torch
    n = torch.cuda.get_device_properties(0).multi_processor_count * 256 + 37
    rep, keys, st = round_trip(pkg, n, tmp_path / "crowded.txt")
    assert pkg._lib.KERNEL[st.kernel] == "staged" and rep.sample == 8192
    assert len(keys) == 1 and keys[0].split()[0].endswith("|crowded")
