"""The dense coarsest level (csrc/dense.cu): on a grid small enough to be its own coarsest level the preconditioner
is the explicit inverse of K, so K (M r) = r.

Sizes: one tile, one dof triple below and above a 64-wide tile edge, whole tiles, two rows per warp in the solve
(above 2368 dofs), and a right-hand side longer than the solve's 4096-value chunk.  Tolerance: the residual of an
explicit FP64 inverse is about cond(K) eps; with unit cells, E = 1 and springs of order 1 on the base cond(K) stays
below 1e6 here, so 1e-9 leaves a factor of 4."""
import numpy as np
import pytest

from comech_b200 import _lib, engine
from comech_b200.grid import Grid, face_node_areas, lame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nodes", [(2, 2, 2), (7, 3, 2), (11, 2, 2), (4, 4, 4), (9, 5, 3), (10, 10, 8), (14, 14, 7)])
def test_explicit_inverse_solves(nodes, precision):
    import torch
    nx, ny, nz = (n - 1 for n in nodes)
    g = Grid(*(np.arange(n + 1.0) for n in (nx, ny, nz)))
    rng = np.random.default_rng(nx * ny * nz)
    lam, mu = lame(rng.uniform(0.5, 2.0, g.ncell), np.full(g.ncell, 0.3))
    base, _ = face_node_areas(g, g.cell_nodes, np.flatnonzero(g.cK == 0), "z-")
    base = np.unique(base)
    P = engine.Problem(g, _lib.MAT_ISO_SRI, np.concatenate([lam, mu]), np.ones(g.ncell, bool), pen_node=base,
                       pen_k=np.ones((len(base), 3)), precision=precision)
    try:
        r = torch.from_numpy(rng.standard_normal(3 * g.nnode)).cuda()
        e = P.apply(P.precondition(r)) - r
        tol = 1e-9 if precision == "fp64" else 1e-2      # mixed: z is rounded to FP32, so the residual is cond eps32
        assert float(e.norm() / r.norm()) < tol
    finally:
        P.close()
