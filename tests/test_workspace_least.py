"""The smaller layout of the refinement's workspace.

It is never larger than slots of 24 or 48 bytes, two census maps and the rest of an
lr_refine side by side, which is what the library asked for before the rows grew to 32
bytes and 64 slots: a workspace of that size is taken, with the bits of the larger one
(the arithmetic is exact, only addresses differ)."""

import ctypes

import numpy as np
import pytest

from conftest import bits

WIDTHS = (8, 16, 24, 32, 48, 64, 96, 128, 192, 256)


def _earlier(W, H, p, views):
    up = lambda n: (n + 255) // 256 * 256
    N, K = W * H, 2 * p.R + 1
    Kp = next(w for w in WIDTHS if w >= K + 2 or w == 256)
    nbits = (2 * p.rx + 1) * (2 * p.ry + 1) - 1
    b = 2 if nbits + 4 + p.P2 > 255 else 1
    one = up(4 * N) + up(N * Kp)
    paths = up(views * (8 if p.paths == 8 else 4) * N * Kp * b)
    return 256 + views * one + 2 * up(8 * N) + paths + (3 * up(8 * N) if views == 2 else 0)


@pytest.mark.parametrize("paths", [4, 8])
@pytest.mark.parametrize("P2", [150.0, 200.0])
def test_least_is_no_more_than_before(svb, P2, paths):
    lib = svb._lib.load()
    for R in list(range(0, 127)):
        p = svb.refine._params(R=R, P1=12.0, P2=P2, rx=4, ry=3, paths=paths)
        for W, H in ((1, 1), (2, 3), (7, 5), (31, 33), (160, 120), (1397, 1101)):
            ref = ctypes.byref(p)
            for least, size, views in (
                    (lib.sv_refine_workspace_least, lib.sv_refine_workspace_size, 1),
                    (lib.sv_lr_refine_workspace_least, lib.sv_lr_refine_workspace_size, 2)):
                assert 0 < least(W, H, ref) <= _earlier(W, H, p, views), (R, W, H)
                assert least(W, H, ref) <= size(W, H, ref)


def test_bad_arguments_have_no_least(svb):
    lib = svb._lib.load()
    bad = svb.refine._params(R=127)
    assert lib.sv_refine_workspace_least(64, 8, ctypes.byref(bad)) == 0
    assert lib.sv_lr_refine_workspace_least(64, 8, ctypes.byref(bad)) == 0
    assert lib.sv_refine_disparity_workspace_least(64, 8, ctypes.byref(bad), 12) == 0
    assert lib.sv_batch_lr_refine_workspace_least(None, 0, ctypes.byref(bad)) == 0
    assert lib.sv_netbatch_workspace_least(None) == 0


def _short_of_memory(svb, monkeypatch):
    """The first allocation of each workspace fails; returns the sizes that were given."""
    import torch
    plain, given = svb.refine._workspace, []
    fail = [True]

    def tight(n):
        if fail[0]:
            fail[0] = False
            raise torch.OutOfMemoryError("no room")
        fail[0] = True
        given.append(int(n))
        return plain(n)
    monkeypatch.setattr(svb.refine, "_workspace", tight)
    return given


def _pair(svb, seed, W, H):
    q = svb.synth.make_pair(seed, W, H, 1.0, 20.0)
    d0 = q.disp.ravel() + np.random.default_rng(seed).uniform(-2.0, 2.0, W * H)
    return q.left.ravel(), q.right.ravel(), np.maximum(d0, 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("R,P2", [(3, 150.0), (7, 150.0), (10, 150.0), (10, 200.0), (15, 150.0),
                                  (22, 200.0), (23, 150.0), (78, 150.0)])
@pytest.mark.parametrize("W,H", [(97, 61), (1, 1), (3, 40)])
def test_same_bits_in_the_least_workspace(svb, monkeypatch, R, P2, W, H):
    L, Rt, d0 = _pair(svb, R, W, H)
    kw = dict(R=R, P1=12.0, P2=P2, rx=4, ry=3)
    want = svb.refine.lr_refine(L, Rt, d0, W, H, tol=2.0, **kw)
    full = svb.refine.refine_fullres(L, Rt, d0, W, H, return_conf=True, **kw)
    given = _short_of_memory(svb, monkeypatch)
    got = svb.refine.lr_refine(L, Rt, d0, W, H, tol=2.0, **kw)
    assert np.array_equal(bits(got[0]), bits(want[0])) and np.array_equal(got[1], want[1])
    one = svb.refine.refine_fullres(L, Rt, d0, W, H, return_conf=True, **kw)
    assert np.array_equal(bits(one[0]), bits(full[0])) and np.array_equal(bits(one[1]), bits(full[1]))
    p = svb.refine._params(**kw)
    assert given == [svb._lib.load().sv_lr_refine_workspace_least(W, H, ctypes.byref(p)),
                     svb._lib.load().sv_refine_workspace_least(W, H, ctypes.byref(p))]


@pytest.mark.gpu
def test_one_byte_less_is_refused(svb):
    import torch
    lib = svb._lib.load()
    W, H = 64, 48
    p = svb.refine._params(R=10, P1=12.0, P2=150.0, rx=4, ry=3)
    least = lib.sv_lr_refine_workspace_least(W, H, ctypes.byref(p))
    t = [torch.zeros(W * H * 8, dtype=torch.uint8, device="cuda") for _ in range(5)]
    ws = torch.zeros(least, dtype=torch.uint8, device="cuda")
    q = lambda x: ctypes.c_void_p(x.data_ptr())
    call = lambda n: lib.sv_lr_refine(q(t[0]), q(t[1]), 0, q(t[2]), W, H, 2.0, ctypes.byref(p),
                                      q(t[3]), q(t[4]), q(ws), n, None)
    assert call(least) == 0 and call(least - 1) == svb._lib.SV_ERR_WORKSPACE
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("R,P2", [(5, 150.0), (10, 150.0), (10, 200.0), (14, 150.0)])
def test_batches_in_the_least_workspace(svb, monkeypatch, R, P2):
    kw = dict(R=R, P1=12.0, P2=P2, rx=4, ry=3)
    pairs = [(*_pair(svb, 50 + k, W, H), W, H) for k, (W, H) in
             enumerate([(97, 61), (1, 1), (160, 45), (7, 90)])]
    want = svb.batch.lr_refine_batch(pairs, tol=2.0, **kw)
    given = _short_of_memory(svb, monkeypatch)
    got = svb.batch.lr_refine_batch(pairs, tol=2.0, **kw)
    assert len(given) == 1
    for a, b in zip(got, want):
        assert np.array_equal(bits(a[0]), bits(b[0])) and np.array_equal(a[1], b[1])


@pytest.mark.gpu
def test_network_batch_and_disparity_in_the_least_workspace(svb, net, monkeypatch):
    import torch
    sizes = [(160, 120), (200, 90)]
    outs = []
    for short in (False, True):
        if short:
            given = _short_of_memory(svb, monkeypatch)
        nb = svb.batch.NetBatch(sizes, net)
        for i, (W, H) in enumerate(sizes):
            L, Rt, _ = _pair(svb, 70 + i, W, H)
            nb.left[i].copy_(torch.from_numpy(L))
            nb.right[i].copy_(torch.from_numpy(Rt))
        nb.run()
        nb.run()                                             # the recorded graph too
        torch.cuda.synchronize()
        W, H = sizes[0]
        L, Rt, d0 = _pair(svb, 90, W, H)
        rgb = np.random.default_rng(3).random(3 * W * H)
        res = svb.post.refine_disparity(L, Rt, rgb, d0, W, H)
        outs.append([t.cpu().numpy() for t in nb.out + nb.status] + [np.asarray(r) for r in res])
    assert len(given) == 2
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
