"""Grid transfers of the V-cycle (csrc/coarse.cu, k_restrict and k_prolong): with equal smoothing before and after, restriction
the transpose of prolongation and Galerkin coarse levels, the preconditioner is symmetric.  A weight, node or split copy that one
of the two transfers treats otherwise than the other breaks this in the third digit at least; FP64 rounding, amplified by the
soft modes that the coarse levels resolve, stays below 1e-9 of |M r| |s|.

Grids: even cell counts on every axis (weights 1 and 1/2), odd ones on one or all (tables), both with split copies, and
unequal spacing."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth
from comech_b200.grid import Grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,stretch", [((24, 18, 16), False), ((25, 18, 16), False), ((29, 21, 17), False),
                                          ((24, 18, 16), True)])
def test_preconditioner_is_symmetric(dims, stretch):
    import torch
    F = synth.hindfoot_problem(*dims, h=2.0, seed=6)
    g = F["grid"]
    if stretch:
        rng = np.random.default_rng(1)
        g = Grid(*(np.r_[0.0, np.cumsum(rng.uniform(1.5, 2.5, n))] for n in dims))
    fn, fa = F["fixed"]
    nr, cr, nc, cc, v = F["extra"].node_coo()
    with engine.Problem(g, _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"], precision="fp64",
                        cn=F["cn"], orig=F["orig"], pen_node=fn, pen_k=np.repeat((fa * 1e6)[:, None], 3, 1),
                        extra_coo=(3 * nr + cr, 3 * nc + cc, v), options=dict(min_dofs=300)) as P:
        used = P.used_mask()[0].cpu().numpy().astype(bool)
        r, s = (torch.from_numpy((np.random.default_rng(k).standard_normal((P.ntotal, 3)) * used[:, None]).ravel()).cuda()
                for k in (2, 3))
        mr, ms = P.precondition(r), P.precondition(s)
        assert float((mr @ s - r @ ms).abs()) <= 1e-9 * float(mr.norm() * s.norm())
