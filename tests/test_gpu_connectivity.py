"""Connectivity whose corners are not the grid node there or a copy of it: the level-0 operator sums every cell's force at the
nodes that the connectivity names, whatever their position, against the oracle's assembled matrix.

Tolerances: FP64 products 1e-12 of the largest entry (sums of at most a few hundred products in another order, 1e-14 relative
to their size); FP32 products 2e-6 relative L2."""
import numpy as np
import pytest

from comech_b200 import _lib, engine, synth
from oracle import fe_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["grid node elsewhere", "copy of a node elsewhere", "one node at two corners"])
def test_every_corner_counts(kind):
    import torch
    F = synth.hindfoot_problem(20, 15, 13, h=2.0, seed=3)
    g, cn, orig = F["grid"], F["cn"].copy(), F["orig"]
    act = np.flatnonzero(F["active"])
    if kind == "grid node elsewhere":
        cn[act[100], 3] = cn[act[2000], 0]
    elif kind == "copy of a node elsewhere":
        orig = np.r_[orig, 5]
        cn[act[300], 2] = len(orig) - 1
    else:
        cn[act[500], 7] = cn[act[500], 0]
    og = O.OGrid(g.xe, g.ye, g.ze)
    K, _, used = O.assemble(og, F["lam"], F["mu"], act, cn, O.kl_sri(og))
    with engine.Problem(g, _lib.MAT_ISO_SRI, np.concatenate([F["lam"], F["mu"]]), F["active"], cn=cn, orig=orig,
                        options=dict(max_levels=0)) as P:
        u = np.zeros((P.ntotal, 3))
        u[used] = np.random.default_rng(1).standard_normal((len(used), 3))
        ref = K @ u[used].ravel()
        y64, y32 = (P.apply(torch.from_numpy(u.ravel().astype(t)).cuda()).cpu().numpy().reshape(-1, 3)[used].ravel()
                    for t in (np.float64, np.float32))
    assert np.abs(y64 - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.linalg.norm(y32 - ref) <= 2e-6 * np.linalg.norm(ref)
