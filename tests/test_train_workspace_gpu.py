"""sv_train_grads with room for the widest layer's partial sums only: the gradients,
losses and prediction of the full workspace, bit for bit; a byte less is refused."""

import ctypes
from importlib import import_module

import numpy as np
import pytest
import torch

from test_train_sizes_gpu import _net

pytestmark = pytest.mark.gpu


def _partials(C, Cm, Rc, nd):
    """Partial sums of all layers and of the widest, in workspace bytes."""
    layers = [C * 10] + [C * (9 * C + 1)] * 3 + [Cm * (27 * C + 1), Cm * (27 * Cm + 1), 27 * Cm + 1]
    layers += 2 * ([Rc * 19] + [Rc * (9 * Rc + 1)] * (nd - 1) + [9 * Rc + 1])
    up = lambda n: (4 * 592 * n + 255) // 256 * 256
    return up(sum(layers)), up(max(layers))


@pytest.mark.parametrize("C,Cm,dil", [(12, 6, (1, 2, 4)), (8, 4, (1, 3, 8, 2, 1, 1, 1, 5)),
                                      (12, 6, (4,))])
def test_least_workspace_gives_the_same_bits(svb, C, Cm, dil):
    train = import_module(svb.__name__ + ".train")
    lib = svb._lib.load()
    B, W, H = 3, 64, 32
    t = train.Trainer(_net(svb, C, Cm, 8, dil, 5))
    g = torch.Generator(device="cuda").manual_seed(C)
    left, right, disp = (torch.rand(B * W * H, device="cuda", generator=g) for _ in range(3))
    disp = disp * 12
    valid = torch.ones(B * W * H, dtype=torch.uint8, device="cuda")
    need = lib.sv_train_workspace_size(t.handle, B, W, H)
    every, widest = _partials(C, Cm, 8, len(dil))
    p = lambda x: ctypes.c_void_p(x.data_ptr())
    got = []
    for size in (need, need - every + widest):
        ws = torch.zeros(size + 512, dtype=torch.uint8, device="cuda")
        loss = torch.empty(B, dtype=torch.float64, device="cuda")
        pred = torch.empty(B * W * H, device="cuda")
        args = (p(left), p(right), p(disp), p(valid), B, W, H, p(loss), p(pred), p(ws))
        svb._lib.check(lib.sv_train_grads(t.handle, *args, size, None), "grads")
        torch.cuda.synchronize()
        assert not ws[size:].any()                     # nothing past the given size
        got.append((loss.cpu().numpy(), pred.cpu().numpy(), t.grads()))
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    assert np.abs(got[0][2]).max() > 0
    rc = lib.sv_train_grads(t.handle, *args, need - every + widest - 1, None)
    assert rc == svb._lib.SV_ERR_WORKSPACE
