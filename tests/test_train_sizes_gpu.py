"""Training kernels at the edges of their tiles, against the FP64 oracle.

The convolutions compute 32 columns x 16 rows per block (8 for the stride-2
layer), four columns per thread, the 3-D ones up to 32 columns of every
disparity, the weight gradients 8 rows x 32 columns; dilations 1, 2 and 4 are
compiled in and others are read at run time.  So: quarter sizes below and above
one tile and no multiple of four, one disparity row per block up to the largest
D, dilations up to 8, the smallest crop, one image and several.

Tolerances are the training kernels' own (test_train_gpu.py): per block
max |g - g_ref| <= 2e-3 max |g_ref| + 1e-6 max over all blocks, cosine
>= 0.9999, losses within 1e-4 relative.  FP32 activations carry 1e-7 per layer
over a dozen layers and sums of up to 1e4 terms, well inside these."""

from importlib import import_module

import numpy as np
import pytest

from test_train_gpu import LOSS_REL, assert_grads_close

pytestmark = pytest.mark.gpu


def _net(svb, C, Cm, D, dil, seed):
    arch = svb.weights.NetArch(feat_C=C, cost_C=Cm, D=D, refine_C=8, refine_dil=dil)
    rng = np.random.default_rng(seed)
    sizes = arch.block_sizes()
    last = {len(sizes) - 2, len(sizes) - 2 - 2 * (len(dil) + 1)}     # residual layers: small
    blocks = []
    for i, n in enumerate(sizes):
        if i % 2 == 0:
            gain = 0.05 if i in last else 1.0
            blocks.append(gain * rng.normal(0.0, np.sqrt(2.0 * sizes[i + 1] / n), n))
        else:
            blocks.append(rng.normal(0.0, 0.02, n))
    return svb.weights.StereoNetWeights(arch, blocks)


@pytest.mark.parametrize("C,Cm,D,dil,W,H,B", [
    (12, 6, 12, (1, 2, 4), 52, 20, 3),          # 13 x 5 at a quarter
    (12, 6, 12, (1, 2, 4), 132, 36, 1),         # 33 columns: one past a tile
    (8, 4, 16, (1, 3, 8), 136, 40, 2),          # the largest D and dilation
    (12, 6, 5, (8, 1), 128, 64, 1),             # whole tiles, odd D
    (8, 4, 2, (5,), 8, 8, 5),                   # the smallest crop
])
def test_train_grads_at_tile_edges(svb, orc, C, Cm, D, dil, W, H, B):
    train = import_module(svb.__name__ + ".train")
    w = _net(svb, C, Cm, D, dil, seed=W + D)
    rng = np.random.default_rng(1000 * W + H)
    L, R = rng.random((2, B, H * W))
    disp = rng.random((B, H * W)) * min(4.0 * (D - 1), W / 2)
    valid = (rng.random((B, H * W)) < 0.9).astype(np.uint8)
    t = train.Trainer(w)
    loss = t.compute_grads(L.reshape(B, H, W), R.reshape(B, H, W), disp.reshape(B, H, W),
                           valid.reshape(B, H, W)).cpu().numpy()
    ref = []
    for k in range(B):
        lo, gr, _ = orc.train_grads(w, L[k], R[k], disp[k], valid[k], W, H)
        assert abs(loss[k] - lo) <= LOSS_REL * abs(lo), (k, loss[k], lo)
        ref.append(gr)
    assert_grads_close(w, t.grads(), np.mean(ref, axis=0))
