"""Chebyshev degrees 6 to 9 of the paired level-0 smoother (csrc/solver.cu, vcycle0_pair): further patterns in which directions
join the iterate late, fused and split, against the separate kernels of FEB_KU_PAIR=0.

Tolerances as for the lower degrees: a direction that is lost or added twice is an error of the size of the result; FP64 1e-10 and
FP32 2e-3 hold rounding, amplified by soft modes."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 2e-3)])
@pytest.mark.parametrize("degree", [6, 7, 8, 9])
def test_high_degrees(monkeypatch, degree, precision, tol):
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    F = synth.hindfoot_problem(24, 18, 16, h=2.0, seed=4)
    fn, fa = F["fixed"]
    nr, cr, nc, cc, v = F["extra"].node_coo()
    z, r = {}, None
    for name, pair, cfg in (("unfused", "0", ""), ("fused", "1", "8,5,5,0"), ("split", "1", "8,5,5,1")):
        monkeypatch.setenv("FEB_KU_PAIR", pair)
        monkeypatch.setenv("FEB_PAIR_CONFIG", cfg)
        with engine.Problem(F["grid"], _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"], cn=F["cn"],
                            orig=F["orig"], pen_node=fn, pen_k=np.repeat((fa * 1e6)[:, None], 3, 1),
                            extra_coo=(3 * nr + cr, 3 * nc + cc, v), precision=precision,
                            options=dict(cheb_degree=degree)) as P:
            if r is None:
                used = P.used_mask()[0].cpu().numpy().astype(bool)
                r = (np.random.default_rng(degree).standard_normal((P.ntotal, 3)) * used[:, None]).ravel()
            z[name] = P.precondition(torch.from_numpy(r).cuda()).cpu().numpy()
    for name in ("fused", "split"):
        assert np.linalg.norm(z[name] - z["unfused"]) <= tol * np.linalg.norm(z["unfused"]), name
