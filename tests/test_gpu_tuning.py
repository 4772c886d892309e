"""The variables that pin the level-0 kernels' launch shapes hold for every handle, also on a grid whose shapes an earlier handle
of the process has tuned."""
import numpy as np
import pytest

from comech_b200 import _lib, engine
from comech_b200.grid import Grid, lame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair,variable,shape", [("1", "FEB_PAIR_CONFIG", (8, 3)), ("0", "FEB_KU_CONFIG", (12, 5))])
def test_pinned_shape_after_a_tuned_handle(monkeypatch, pair, variable, shape):
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    monkeypatch.setenv("FEB_KU_PAIR", pair)
    g = Grid(*(np.arange(n + 1.0) for n in (23, 11, 9)))
    lam, mu = lame(np.full(g.ncell, 10.0), np.full(g.ncell, 0.3))
    base = np.arange((g.nx + 1) * (g.ny + 1))

    def solved_shape():
        with engine.Problem(g, _lib.MAT_ISO_SRI, np.concatenate([lam, mu]), np.ones(g.ncell, bool), pen_node=base,
                            pen_k=np.full((len(base), 3), 10.0)) as P:
            info = P.solve(torch.ones(3 * P.ntotal, dtype=torch.float64, device="cuda"))[1]
        return list(info.ku_shape)

    solved_shape()                               # tunes the grid
    monkeypatch.setenv(variable, "%d,%d" % shape)
    assert solved_shape() == [*shape, *shape]


def test_benchmark_step_has_the_plans_form(monkeypatch):
    """feb_benchmark_smooth_set times the form that the handle's smoothing steps have, fused (one launch) or split (two), and both
    leave the same r, x and d' (sums of a few hundred FP32 products: 1e-5 relative L2)."""
    import ctypes as C
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    g = Grid(*(np.arange(n + 1.0) for n in (23, 19, 17)))
    lam, mu = lame(np.full(g.ncell, 10.0), np.full(g.ncell, 0.3))
    base = np.arange((g.nx + 1) * (g.ny + 1))
    rng = np.random.default_rng(0)
    start = [torch.from_numpy(rng.standard_normal(3 * g.nnode).astype(np.float32)).cuda() for _ in range(3)]
    lib, ms, out = _lib.load(), C.c_float(), {}
    for split in (0, 1):
        monkeypatch.setenv("FEB_PAIR_CONFIG", f"8,5,5,{split}")
        with engine.Problem(g, _lib.MAT_ISO_SRI, np.concatenate([lam, mu]), np.ones(g.ncell, bool), pen_node=base,
                            pen_k=np.full((len(base), 3), 10.0), precision="mixed", options=dict(min_dofs=500)) as P:
            d, r, x = (v.clone() for v in start)
            e = torch.zeros_like(d)
            before = lib.feb_launch_count()
            _lib.check(lib.feb_benchmark_smooth_set(P.h, 1, *((C.c_void_p * 1)(v.data_ptr()) for v in (d, r, x, e)), 2,
                                                    C.byref(ms)))
            assert lib.feb_launch_count() - before == 3 * (1 + split)       # two timed steps after an untimed one
            out[split] = [v.cpu().numpy() for v in (r, x, e)]
    for a, b in zip(out[0], out[1]):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
