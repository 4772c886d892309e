"""feb_precondition with its result in the right-hand side's place, against the same call with a vector of its own: with and
without rigid groups (whose coefficients are formed beside the V-cycle), the paired and the per-cell level-0 kernels, and a grid
that is its own coarsest level.

Tolerances: FP64 1e-10 (the order of a few atomic sums, amplified by soft modes); mixed 2e-3 (the same in FP32).  A right-hand
side that is overwritten is an error of the size of the result."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 2e-3)])
@pytest.mark.parametrize("pair", ["1", "0"])
@pytest.mark.parametrize("dims,groups", [((22, 16, 14), True), ((22, 16, 14), False), ((8, 6, 6), True)])
def test_result_in_place(monkeypatch, dims, groups, pair, precision, tol):
    import torch
    monkeypatch.setenv("FEB_KU_PAIR", pair)
    monkeypatch.setenv("FEB_PAIR_CONFIG", "8,5,5,1")
    F = synth.hindfoot_problem(*dims, h=80.0 / dims[0], seed=4)
    fn, fa = F["fixed"]
    nr, cr, nc, cc, v = F["extra"].node_coo()
    with engine.Problem(F["grid"], _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"], cn=F["cn"],
                        orig=F["orig"], pen_node=fn, pen_k=np.repeat((fa * 1e6)[:, None], 3, 1),
                        extra_coo=(3 * nr + cr, 3 * nc + cc, v), precision=precision) as P:
        if groups:
            P.set_rigid_groups(F["node_groups"])
        used = P.used_mask()[0].cpu().numpy().astype(bool)
        r = torch.from_numpy((np.random.default_rng(2).standard_normal((P.ntotal, 3)) * used[:, None]).ravel()).cuda()
        z = P.precondition(r)
        p = r.clone()
        for _ in range(2):                       # the second call takes the first one's result
            _lib.check(_lib.load().feb_precondition(P.h, p.data_ptr(), p.data_ptr()))
            assert float((p - z).norm()) <= tol * float(z.norm())
            z = P.precondition(z)
