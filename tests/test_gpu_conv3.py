"""3x3x3 convolution kernels (csrc/net.cu: k_conv3, k_wgrad3) at the sizes where its tiling can go wrong, against the float64
oracle: 126-row tiles (one wave) and 252-row tiles (more tiles than SMs), rows that end just before, at and after a
tile, several tiles per CTA, windows longer than the whole grid, and a z extent whose window does not fit shared memory
(one (x, y) offset per step).  Operands are exact in BF16 and sums are FP32, so the output's own rounding to BF16
bounds the error: 2^-9 per value, 4e-3 relative L2 with a factor of 2.  Weight and bias gradients are FP32 sums of exact
products over at most 41,000 rows: 1e-5 relative L2 (sqrt(rows) eps is 1.2e-5 for one sum in sequence; the sums are split)."""
import numpy as np
import pytest

from comech_b200 import _lib
from comech_b200.engine import _ptr, _stream
from oracle import net_oracle as O

from test_gpu_warm import bf16, conv, dev_rows, empty_rows, from_rows, host, rel, tables, wgrad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ci,co,dims", [
    (32, 32, (1, 1, 1)),          # 27 rows: one partial tile
    (32, 32, (5, 4, 1)),          # 126 rows: exactly one tile
    (32, 64, (5, 1, 4)),          # 126 rows, two channel tiles
    (64, 32, (2, 2, 6)),          # 128 rows: two rows past a tile
    (96, 32, (12, 16, 8)),        # 2520 rows: whole tiles, three slices
    (32, 64, (40, 28, 22)),       # 252-row tiles, more than one per CTA
    (64, 32, (30, 31, 50)),       # 252-row tiles of 18 steps through the ring
    (32, 32, (2, 3, 700)),        # the window of three y offsets does not fit: one offset per step
    (256, 256, (4, 3, 2)),        # many slices, eight channel tiles
])
def test_conv3_tiles(ci, co, dims):
    import torch
    rng = np.random.default_rng(ci + co + sum(dims))
    X = bf16(np.maximum(rng.normal(size=dims + (ci,)), 0))
    W = bf16(rng.normal(0, np.sqrt(2 / (27 * ci)), (27, co, ci)))
    b = rng.normal(0, 0.1, co).astype(np.float32)
    f, bw = tables(W, flip=1)
    Xd, out = dev_rows(X), empty_rows(dims, co)
    out.fill_(7.0)
    conv(_lib.GATHER_SHIFT, dims, None, Xd, ci, f, co, out, bias=torch.as_tensor(b).cuda())
    assert rel(from_rows(host(out), dims), O.relu(O.conv3(X, W, b.astype(np.float64)))) < 4e-3
    shell = np.ones([d + 2 for d in dims], bool)
    shell[1:-1, 1:-1, 1:-1] = False
    assert (host(out).reshape(*shell.shape, co)[shell] == 0).all()
    # data gradient: the flipped table, masked by the input's ReLU, without bias
    G = bf16(rng.normal(size=dims + (co,)))
    gx, Gd = empty_rows(dims, ci), dev_rows(G)
    conv(_lib.GATHER_SHIFT, dims, None, Gd, co, bw, ci, gx, relu=0, mask=Xd)
    rX, rW, rb = O.conv3_back(X, W, G)
    assert rel(from_rows(host(gx), dims), rX * (X > 0)) < 4e-3
    # weight gradient (row steps of 128 split over the SMs, 32 x 32 channel tiles) and bias gradient
    assert rel(wgrad(_lib.GATHER_SHIFT, dims, None, Gd, co, Xd, ci, 27), rW) < 1e-5
    db = torch.zeros(co, dtype=torch.float32, device="cuda")
    _lib.check(_lib.load().feb_net_colsum(_ptr(Gd), Gd.shape[0], co, 0, co, _ptr(db), _stream()))
    assert rel(host(db), rb) < 1e-5


@pytest.mark.parametrize("rows,ld,c0,nc", [(1, 8, 0, 8), (255, 40, 8, 24), (70001, 32, 0, 32), (513, 256, 0, 256), (300, 36, 4, 30)])
def test_column_sums(rows, ld, c0, nc):
    """feb_net_colsum: 8-channel groups (one thread per group, uneven groups per block) and the general form."""
    import torch
    rng = np.random.default_rng(rows)
    G = bf16(rng.uniform(0.5, 1.5, (rows, ld)))
    Gd = torch.as_tensor(G.astype(np.float32)).to(torch.bfloat16).cuda()
    out = torch.full((nc,), 2.0, dtype=torch.float32, device="cuda")
    _lib.check(_lib.load().feb_net_colsum(_ptr(Gd), rows, ld, c0, nc, _ptr(out), _stream()))
    assert rel(host(out), 2.0 + G[:, c0:c0 + nc].sum(0)) < 1e-5
