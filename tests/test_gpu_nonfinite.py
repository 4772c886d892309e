"""A handle that refused a non-finite right-hand side solves the next one: nothing of the refused solve is left in the vectors
that the next one starts from.  Both solves stop at 1e-10 of the right-hand side; solutions within 1e-8 relative L2."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,graphs,batch", [("fp64", 2, False), ("fp64", 0, False), ("mixed", 2, False),
                                                    ("refine", 2, False), ("fp64", 2, True), ("mixed", 2, True)])
def test_solve_after_a_refused_one(precision, graphs, batch):
    import torch
    F = synth.hindfoot_problem(20, 15, 13, h=2.0, seed=3)
    fn, fa = F["fixed"]
    nr, cr, nc, cc, v = F["extra"].node_coo()
    with engine.Problem(F["grid"], _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"], cn=F["cn"],
                        orig=F["orig"], pen_node=fn, pen_k=np.repeat((fa * 1e6)[:, None], 3, 1),
                        extra_coo=(3 * nr + cr, 3 * nc + cc, v), precision=precision, tol=1e-10,
                        options=dict(use_graphs=graphs)) as P:
        solve = (lambda f: engine.solve_batch_device([P], [f])[0][0]) if batch else (lambda f: P.solve(f)[0])
        f = P.rhs(F["loads"])
        ref = solve(f).clone()
        for bad in (float("nan"), float("inf")):
            g = f.clone()
            g[torch.nonzero(f)[0]] = bad
            with pytest.raises(RuntimeError):
                solve(g)
            x = solve(f)
            assert float((x - ref).norm()) <= 1e-8 * float(ref.norm())
