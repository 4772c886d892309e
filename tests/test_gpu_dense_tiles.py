"""The product with the inverse of the dense coarsest level (csrc/dense.cu, k_dense_solve: a CTA a lower 64 x 64 tile, partial
vectors summed by the last CTA of a block row) on a grid that is its own coarsest level and whose blocks of inactive cells leave
nodes without dofs: repeated calls on a handle agree in every bit (the arrival counters are at zero again, sums have a fixed
order), nodes without dofs get zeros, and K (M r) = r.

Sizes: within one tile, one dof triple past a tile's edge, several tiles with a partial one.  Tolerance: the residual of an
explicit FP64 inverse is about cond(K) eps; with unit cells, moduli of order 1 and springs of order 1 on the base cond(K) stays
below 1e6, so 1e-9 leaves a factor of 4."""
import numpy as np
import pytest

from comech_b200 import _lib, engine
from comech_b200.grid import Grid, lame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(3, 2, 2), (5, 3, 2), (9, 7, 5), (12, 11, 8)])
def test_repeated_products(cells):
    import torch
    g = Grid(*(np.arange(n + 1.0) for n in cells))
    rng = np.random.default_rng(sum(cells))
    lam, mu = lame(rng.uniform(0.5, 2.0, g.ncell), np.full(g.ncell, 0.3))
    active = np.ones(cells, bool)
    active[-1:, -1:, -1:] = False                # cells are numbered z fastest
    active[:1, -1:, -1:] = False
    base = np.arange((g.nx + 1) * (g.ny + 1))
    with engine.Problem(g, _lib.MAT_ISO_SRI, np.concatenate([lam, mu]), active.ravel(), pen_node=base,
                        pen_k=np.ones((len(base), 3)), precision="fp64") as P:
        used = P.used_mask()[0].bool().repeat_interleave(3)
        assert int((~used).sum()) == 6           # the two corners
        r = torch.from_numpy(rng.standard_normal(3 * g.nnode)).cuda() * used
        z = P.precondition(r)
        for _ in range(3):
            assert torch.equal(P.precondition(r), z)
        assert float(z[~used].abs().max()) == 0.0
        assert float((P.apply(z) - r).norm()) <= 1e-9 * float(r.norm())
