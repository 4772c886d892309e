"""FP32 error of the 3x3x3 weight gradients (csrc/net.cu, k_wgrad3) against the float64 oracle: an accumulator takes at most
512 rows in sequence on grids of up to 200,000 rows and 128 on those of up to 20,000, so its error does not grow with the size.

Tolerance: every step of 16 rows adds to the accumulator and cuts off at most 2^-23 of it, half of that on average, and over a
sum of k steps of random signs the accumulator is two thirds of its end on average: k 2^-24 2/3 of the sum, in one direction.
The few additions between the sums are rounded to nearest and stay far below."""
import numpy as np
import pytest

from comech_b200 import _lib
from oracle import net_oracle as O

from test_gpu_warm import bf16, dev_rows, rel, wgrad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,dims,rows", [(32, (12, 8, 6), 128), (128, (24, 16, 12), 128), (64, (33, 21, 17), 128),
                                         (32, (2, 3, 700), 128), (96, (40, 30, 20), 512)])
def test_error_of_the_sums(c, dims, rows):
    rng = np.random.default_rng(c + sum(dims))
    X, G = bf16(rng.normal(size=dims + (c,))), bf16(rng.normal(size=dims + (c,)))
    Xp = O._pad(X)
    ref = np.stack([G.reshape(-1, c).T @ O._shift(Xp, d, dims).reshape(-1, c) for d in O.TAPS3])
    dw = wgrad(_lib.GATHER_SHIFT, dims, None, dev_rows(G), c, dev_rows(X), c, 27)
    assert rel(dw, ref) <= rows / 16 * 2.0 ** -24 * 2 / 3
