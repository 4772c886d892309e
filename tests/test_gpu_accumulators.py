"""The paired-row operator with its sparse part through accumulators (csrc/fine_pair.cu, add_sparse), which it
takes where the row list would be long: many irregular cells with their copies, entries on every node, a few long rows.  Products
(twice: the accumulators are clear again) and one V-cycle with fused and split smoothing steps, against the per-cell kernels.

Tolerances: FP64 products 1e-12 of the largest entry (sums of at most a few hundred products in another order, 1e-14
relative to their size); FP32 products 2e-6 relative L2 against the FP64 product; V-cycles 1e-10 (FP64) and 2e-3 (FP32 rounding,
amplified by soft modes): a node that is lost or added twice is an error of the size of the result."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


def _springs(a, b, k):
    """COO of springs between node pairs, all three components."""
    A, B = (3 * np.repeat(n, 3) + np.tile(np.arange(3), len(n)) for n in (a, b))
    k = np.full(len(A), k)
    return np.r_[A, B, A, B], np.r_[A, B, B, A], np.r_[k, k, -k, -k]


def _case(kind):
    F = synth.hindfoot_problem(26, 19, 17, h=2.0, seed=4)
    cn, orig, act = F["cn"].copy(), F["orig"], np.flatnonzero(F["active"])
    used = np.unique(cn[act])
    rng = np.random.default_rng(7)
    nr, cr, nc, cc, v = F["extra"].node_coo()
    er, ec, ev = 3 * nr + cr, 3 * nc + cc, v
    if kind == "irregular cells":                # a third of the cells on four nodes of their own, tied to the old ones
        sel = act[rng.random(len(act)) < 0.3]
        old = cn[sel][:, [0, 2, 5, 7]].ravel()
        own = len(orig) + np.arange(len(old))
        cn[sel[:, None], [0, 2, 5, 7]] = own.reshape(-1, 4)
        orig = np.r_[orig, orig[old]]
        add = _springs(own, old, 50.0)
    elif kind == "every node":
        add = _springs(used, np.roll(used, 1), 5.0)
    else:                                        # rank-1 rows of 70 entries on few nodes
        d = 3 * rng.choice(used, 70, replace=False) + 1
        add = np.repeat(d, 70), np.tile(d, 70), np.full(4900, 0.3)
    fn, fa = F["fixed"]
    kw = dict(cn=cn, orig=orig, pen_node=fn, pen_k=np.repeat((fa * 1e6)[:, None], 3, 1),
              extra_coo=tuple(np.concatenate(p) for p in zip((er, ec, ev), add)))
    return (F["grid"], _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"]), kw


def _vector(P, seed):
    used = P.used_mask()[0].cpu().numpy().astype(bool)
    return (np.random.default_rng(seed).standard_normal((P.ntotal, 3)) * used[:, None]).ravel()


@pytest.mark.parametrize("kind", ["irregular cells", "every node", "long rows"])
def test_products(monkeypatch, kind):
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    monkeypatch.setenv("FEB_PAIR_CONFIG", "8,5")
    args, kw = _case(kind)
    out, u = {}, None
    for pair in ("1", "0"):
        monkeypatch.setenv("FEB_KU_PAIR", pair)
        with engine.Problem(*args, options=dict(max_levels=0), **kw) as P:
            u = _vector(P, 1) if u is None else u
            before = _lib.load().feb_launch_count()
            out[pair] = [P.apply(torch.from_numpy(u.astype(t)).cuda()).cpu().numpy()
                         for t in (np.float64, np.float32, np.float64, np.float32)]
            if pair == "1":                      # k_fine_sparse and the tiles
                assert _lib.load().feb_launch_count() - before == 4 * 2
    ref = out["0"][0]
    for q in (0, 2):
        assert np.abs(out["1"][q] - ref).max() <= 1e-12 * np.abs(ref).max()
        assert np.linalg.norm(out["1"][q + 1] - ref) <= 2e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 2e-3)])
@pytest.mark.parametrize("kind", ["irregular cells", "every node", "long rows"])
def test_smoothing_steps(monkeypatch, kind, precision, tol):
    import torch
    monkeypatch.setenv("FEB_KU_TC", "0")
    args, kw = _case(kind)
    for degree in (1, 3):
        z, r = {}, None
        for name, pair, cfg in (("unfused", "0", ""), ("fused", "1", "8,5,5,0"), ("split", "1", "8,5,5,1")):
            monkeypatch.setenv("FEB_KU_PAIR", pair)
            monkeypatch.setenv("FEB_PAIR_CONFIG", cfg)
            with engine.Problem(*args, precision=precision, options=dict(cheb_degree=degree), **kw) as P:
                r = _vector(P, degree) if r is None else r
                z[name] = P.precondition(torch.from_numpy(r).cuda()).cpu().numpy()
        for name in ("fused", "split"):
            assert np.linalg.norm(z[name] - z["unfused"]) <= tol * np.linalg.norm(z["unfused"]), (degree, name)
