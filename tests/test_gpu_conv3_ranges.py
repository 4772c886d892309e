"""3x3x3 layers (csrc/net.cu: k_conv3, k_wgrad3) on channel ranges of wider rows (in_c0, out_c0, mask_c0, p_c0, q_c0) and with
accumulation, against the float64 oracle; the channels beside the output's stay as they were.

Tolerances: outputs 4e-3 relative L2 (rounding to BF16, 2^-9 a value, with a factor of 2; an accumulating layer rounds its sum
once); weight gradients 1e-5 (FP32 sums of exact products)."""
import numpy as np
import pytest

from comech_b200 import _lib
from oracle import net_oracle as O

from test_gpu_warm import bf16, conv, dev_rows, from_rows, host, rel, tables, wgrad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ci,co,c0,o0,m0", [(32, 32, 8, 40, 16), (64, 32, 24, 0, 8), (64, 64, 64, 8, 0), (96, 32, 8, 32, 24)])
@pytest.mark.parametrize("dims", [(6, 5, 7), (40, 28, 22)])
def test_channel_ranges(ci, co, c0, o0, m0, dims):
    rng = np.random.default_rng(ci + co + dims[0])
    wide = bf16(rng.normal(size=dims + (ci + c0 + 16,)))
    X = wide[..., c0:c0 + ci]
    W = bf16(rng.normal(0, np.sqrt(2 / (27 * ci)), (27, co, ci)))
    before = bf16(rng.normal(size=dims + (co + o0 + 8,)))
    gate = bf16(rng.normal(size=dims + (co + m0,)))
    f, _ = tables(W, flip=1)
    src, out, mask = dev_rows(wide), dev_rows(before), dev_rows(gate)
    conv(_lib.GATHER_SHIFT, dims, None, src, ci, f, co, out, relu=0, mask=mask, accumulate=1, src_c0=c0, out_c0=o0, mask_c0=m0)
    got = from_rows(host(out), dims)
    ref = (before[..., o0:o0 + co] + O.conv3(X, W)) * (gate[..., m0:m0 + co] > 0)
    assert rel(got[..., o0:o0 + co], ref) < 4e-3
    kept = np.r_[0:o0, o0 + co:co + o0 + 8]
    assert (got[..., kept] == before[..., kept]).all()
    # weight gradient of the same ranges: P the output's gradient, Q the layer's input
    dw = wgrad(_lib.GATHER_SHIFT, dims, None, out, co, src, ci, 27, p_c0=o0, q_c0=c0)
    G, Xp = got[..., o0:o0 + co].reshape(-1, co), O._pad(X)
    assert rel(dw, np.stack([G.T @ O._shift(Xp, d, dims).reshape(-1, ci) for d in O.TAPS3])) < 1e-5
