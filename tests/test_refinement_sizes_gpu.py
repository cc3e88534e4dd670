"""Refinement's 3x3 convolutions at the edges of their tiles and of the rule that
chooses them: 32 x 16 outputs per block from 40,000 pixels on, columns in fours or
one by one, dilations 1, 2 and 4 compiled in, up to 8 read, larger ones without a
tile (batched).  Against the FP64 oracle with the forward's own tolerance (FP32
sums of 72 products over a dozen layers; test_network_gpu.py), and a batch against
its pairs alone, bit for bit."""

import numpy as np
import pytest
import torch

from conftest import bits
from test_network_gpu import TOL_PX

pytestmark = pytest.mark.gpu


def _net(svb, dil, seed):
    arch = svb.weights.NetArch(feat_C=8, cost_C=4, D=8, refine_C=8, refine_dil=dil)
    rng = np.random.default_rng(seed)
    sizes = arch.block_sizes()
    blocks = [rng.normal(0.0, 0.5 * np.sqrt(2.0 * sizes[i + 1] / n), n) if i % 2 == 0 else
              rng.normal(0.0, 0.02, n) for i, n in enumerate(sizes)]
    return svb.weights.StereoNetWeights(arch, blocks)


@pytest.mark.parametrize("W,H,dil", [
    (200, 200, (1, 2, 4)),              # the first size of the rule, whole columns
    (199, 201, (1, 2, 4)),              # one pixel below it
    (257, 157, (1, 2, 4)),              # 40,349 pixels, ragged in both directions
    (260, 162, (2, 8, 3)),
    (226, 179, (4, 5)),
])
def test_forward_at_tile_edges(svb, orc, W, H, dil):
    w = _net(svb, dil, W)
    rng = np.random.default_rng(H)
    L, R = rng.random((2, H * W))
    gh, _, _ = orc.avgpool2(L, 1, H, W)
    got = svb.network.forward(w, L, R, H, W, gh, L)
    ref = orc.stereonet_forward(w, L, R, H, W, gh, L)
    for g, r in zip(got, ref):
        assert np.abs(np.asarray(g) - np.asarray(r)).max() <= TOL_PX


@pytest.mark.parametrize("dil", [(1, 2, 4), (3, 9), (1, 8)])
def test_batch_equals_pairs_alone(svb, dil):
    w = _net(svb, dil, 3)
    pairs = [svb.synth.make_pair(40 + k, W, H, 1.0, 20.0) for k, (W, H) in
             enumerate([(333, 201), (90, 61), (320, 240)])]
    nb = svb.batch.NetBatch([(p.W, p.H) for p in pairs], w, tol=2.0, R=10, P1=12.0, P2=150.0,
                            rx=4, ry=3)
    for i, p in enumerate(pairs):
        nb.left[i].copy_(torch.from_numpy(p.left.ravel()))
        nb.right[i].copy_(torch.from_numpy(p.right.ravel()))
    nb.predict()
    torch.cuda.synchronize()
    for i, p in enumerate(pairs):
        (df, _, _, _), _ = svb.network.predict_auto(w, p.left, p.right, p.W, p.H, verbose=False,
                                                    return_trace=True)
        assert np.array_equal(bits(nb.disparity(i).cpu().numpy()), bits(df)), i
