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
