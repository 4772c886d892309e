"""The row list of the paired-row operator (csrc/fine_pair.cu, finish_row): nodes that irregular cells or extra entries
reach, finished cell by cell, against the per-cell kernel.  Cases: split connectivity on box-shaped voxels and with full
integration and orthotropic coefficients (general geometry in the rows), springs with far columns and repeated penalties,
an operator without any cell (every node a row, more rows than one pass of the CTAs takes), and copies no cell uses.

Tolerances: FP64 products 1e-12 of the largest entry (sums of at most a few hundred products in another order, 1e-14
relative to their size); FP32 products 2e-6 relative L2 against the FP64 product."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth
from comech_b200.grid import Grid

pytestmark = pytest.mark.gpu


def _cases():
    P = synth.hindfoot_problem(26, 19, 17, h=(1.0, 1.3, 0.8), seed=3)
    g = P["grid"]
    fn, fa = P["fixed"]
    rng = np.random.default_rng(0)
    nr, cr, nc, cc, v = P["extra"].node_coo()
    far = rng.integers(0, len(P["orig"]), (60, 2))          # symmetric pairs of far dofs, some on unused nodes
    er = np.concatenate([3 * nr + cr, 3 * far[:, 0] + 1, 3 * far[:, 1] + 2])
    ec = np.concatenate([3 * nc + cc, 3 * far[:, 1] + 2, 3 * far[:, 0] + 1])
    w = rng.uniform(1, 50, 60)
    kw = dict(cn=P["cn"], orig=P["orig"], pen_node=np.r_[fn, fn[:40]], extra_coo=(er, ec, np.concatenate([v, w, w])),
              pen_k=np.r_[np.repeat((fa * 1e6)[:, None], 3, 1), rng.uniform(1, 9, (40, 3))])
    lam, mu = P["lam"], P["mu"]
    yield "box voxels", (g, _lib.MAT_ISO_SRI, np.concatenate([lam, mu]), P["active"]), kw
    yield "full integration", (g, _lib.MAT_ISO_FULL, np.concatenate([lam, mu]), P["active"]), kw
    c = np.stack([lam + 2 * mu, lam, lam, lam + 2 * mu, mu, 0.7 * mu], 1)
    yield "orthotropic", (g, _lib.MAT_ORTHO, np.ascontiguousarray(c).ravel(), P["active"]), kw
    kw2 = dict(kw, orig=np.r_[P["orig"], P["orig"][:5]])    # five copies that no cell uses
    yield "unused copies", (g, _lib.MAT_ISO_SRI, np.concatenate([lam, mu]), P["active"]), kw2
    g2 = Grid(*(np.arange(n + 1.0) for n in (40, 33, 29)))
    n = 3 * g2.nnode
    d = np.arange(n)
    o = d[:-7]
    yield "no cells", (g2, _lib.MAT_ISO_SRI, np.zeros(2 * g2.ncell), np.zeros(g2.ncell, bool)), dict(
        extra_coo=(np.r_[d, o, o + 7], np.r_[d, o + 7, o], np.r_[4 + rng.random(n), np.full(2 * len(o), -1.0)]),
        mark_used=np.arange(g2.nnode))


@pytest.mark.parametrize("shape", ["8,1", "8,64"])
def test_rows_match_cell_kernel(monkeypatch, shape):
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    monkeypatch.setenv("FEB_PAIR_CONFIG", shape)
    for name, args, kw in _cases():
        out, u = {}, None
        for pair in ("1", "0"):
            monkeypatch.setenv("FEB_KU_PAIR", pair)
            with engine.Problem(*args, options=dict(max_levels=0), **kw) as P:
                if u is None:
                    used = P.used_mask()[0].cpu().numpy().astype(bool)
                    u = np.random.default_rng(1).standard_normal((P.ntotal, 3)) * used[:, None]
                out[pair] = [P.apply(torch.from_numpy(u.ravel().astype(t)).cuda()).cpu().numpy()
                             for t in (np.float64, np.float32)]
        (y64, y32), (c64, _) = out["1"], out["0"]
        assert np.abs(y64 - c64).max() <= 1e-12 * np.abs(c64).max(), name
        assert np.linalg.norm(y32 - c64) / np.linalg.norm(c64) < 2e-6, name


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 2e-3)])
def test_split_and_fused_steps_match_unfused(monkeypatch, precision, tol):
    """One V-cycle with the smoothing steps fused into the product and split into product and update, for every pattern in
    which directions join the iterate late (degrees 1 to 5), against the separate kernels of FEB_KU_PAIR=0.  A direction that
    is lost or added twice is an error of the size of the result; FP32 rounding, amplified by soft modes, is far below 2e-3."""
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    F = synth.hindfoot_problem(28, 21, 18, h=2.0, seed=4)
    fn, fa = F["fixed"]
    nr, cr, nc, cc, v = F["extra"].node_coo()
    kw = dict(cn=F["cn"], orig=F["orig"], pen_node=fn, pen_k=np.repeat((fa * 1e6)[:, None], 3, 1),
              extra_coo=(3 * nr + cr, 3 * nc + cc, v))
    for degree in (1, 2, 3, 4, 5):
        z, r = {}, None
        for name, pair, cfg in (("unfused", "0", ""), ("fused", "1", "8,5,5,0"), ("split", "1", "8,5,5,1")):
            monkeypatch.setenv("FEB_KU_PAIR", pair)
            monkeypatch.setenv("FEB_PAIR_CONFIG", cfg)
            with engine.Problem(F["grid"], _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"],
                                precision=precision, options=dict(cheb_degree=degree), **kw) as P:
                if r is None:
                    used = P.used_mask()[0].cpu().numpy().astype(bool)
                    r = (np.random.default_rng(degree).standard_normal((P.ntotal, 3)) * used[:, None]).ravel()
                z[name] = P.precondition(torch.from_numpy(r).cuda()).cpu().numpy()
                if name != "unfused":                    # the same with the result in r's place
                    p = torch.from_numpy(r).cuda()
                    _lib.check(_lib.load().feb_precondition(P.h, p.data_ptr(), p.data_ptr()))
                    z[name + ", in place"] = p.cpu().numpy()
        for name in set(z) - {"unfused"}:
            assert np.linalg.norm(z[name] - z["unfused"]) <= tol * np.linalg.norm(z["unfused"]), (degree, name)
