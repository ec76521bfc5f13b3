"""Accuracy of the network's weight gradients as sums over the cells: parameters under
which every other quantity of the pass is exact, so that the gradient of a mixing
matrix is a plain sum over the cells, known in 64 bits."""
import numpy as np
import pytest

from cugmres_b200 import learned
from oracle import fno_oracle as FO

pytestmark = pytest.mark.gpu

# The sums are FP32 additions in chains of at most 173 (a few hundred blocks share the
# cells, eight cells an addition), the blocks' sums are added in FP64 and rounded once.
# A chain's rounding errors average out over the blocks: 4 standard deviations of that
# (6e-8) and the last rounding (6e-8).
BOUND = 2.0 ** -23


@pytest.mark.parametrize("shape", [(16, 160, 160), (16, 64, 64), (3, 33, 35), (1, 32, 32)])
def test_weight_gradients_are_exact_sums(cuda_device, shape):
    B, H, W = shape
    p = np.zeros(FO.NPARAM, np.float32)
    p[FO.OFF_PB:FO.OFF_PB + FO.C] = 8.0  # v = 8 through the first three layers (GELU(8) = 8 in FP32)
    for layer in range(FO.LAYERS):
        b = FO.off_r(layer) + FO.RSZ + FO.C * FO.C
        p[b:b + FO.C] = 8.0 if layer < FO.LAYERS - 1 else 1.0
    sign = np.where(np.arange(FO.C) % 2 == 0, 1.0, -1.0)
    p[FO.OFF_Q1:FO.OFF_Q1 + FO.C] = sign  # hidden unit 0 sees 0: GELU' = 1/2; the others too
    p[FO.OFF_Q2:FO.OFF_Q2 + FO.HID] = 1.0
    rng = np.random.default_rng(7)
    chi, k0h = rng.random(shape).astype(np.float32), np.full(B, 0.3, np.float32)
    # cotangents: eight significant bits, all positive, over a range of 2^12, so that a
    # chain's sums do not fit 24 bits; residuals of modulus one leave them unscaled
    d = np.ldexp(rng.integers(128, 256, shape) / 128.0, -rng.integers(0, 13, shape)).astype(np.float32)
    net = learned.FNO(cuda_device, seed=0)
    net.set_params(p)
    net.forward_train(chi, k0h, np.ones(shape, np.complex64))
    g = net.backward(d.astype(np.complex64), want_grad=True).astype(np.float64)
    net.close()
    total = 0.5 * d.astype(np.float64).sum()
    w, b, last = FO.off_r(FO.LAYERS - 1) + FO.RSZ, FO.OFF_BQ1, FO.off_r(FO.LAYERS - 1) + FO.RSZ + FO.C * FO.C
    assert np.abs(g[FO.OFF_Q1:FO.OFF_Q1 + FO.HID * FO.C] / total - 1.0).max() <= BOUND
    assert np.abs(g[b:b + FO.HID] / total - 1.0).max() <= BOUND
    dw = g[w:w + FO.C * FO.C].reshape(FO.C, FO.C)
    assert np.abs(dw / (8.0 * total * sign[:, None]) - 1.0).max() <= BOUND
    assert np.abs(g[last:last + FO.C] / (total * sign) - 1.0).max() <= BOUND
