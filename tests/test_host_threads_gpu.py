"""Calls of several host threads, each with its own stream, workspace and sizes.

A kernel's dynamic shared-memory limit belongs to the kernel, not to the call, so two
calls that need different amounts must not lower it for each other: every call returns
without an error, with the bits of the same call made alone.  The sizes are the ones
whose kernels ask for different amounts above the default 48 KB; most are small
images, so that the host's part of a call (where the threads meet) is most of it."""

import ctypes
import threading
from importlib import import_module

import pytest
import torch

from test_train_sizes_gpu import _net as _train_net
from test_refinement_sizes_gpu import _net as _forward_net

pytestmark = pytest.mark.gpu


def _together(jobs, n):
    """jobs: [(call(stream), outputs)]; each call once alone, then n times in a thread
    of its own beside the others."""
    streams = [torch.cuda.Stream() for _ in jobs]
    want = []
    torch.cuda.synchronize()
    for (call, outs), s in zip(jobs, streams):
        call(s.cuda_stream)
        s.synchronize()
        want.append([o.clone() for o in outs])
    torch.cuda.synchronize()
    errors = []
    gate = threading.Barrier(len(jobs))

    def work(call, stream):
        gate.wait()
        for _ in range(n):
            try:
                call(stream.cuda_stream)
            except Exception as e:                       # every refused call counts
                errors.append(str(e))
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(j[0], s)) for j, s in zip(jobs, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, (len(errors), errors[0])
    for (_, outs), w in zip(jobs, want):
        for a, b in zip(outs, w):
            assert torch.equal(a, b)


def _images(seed, W, H):
    g = torch.Generator(device="cuda").manual_seed(seed)
    left = torch.randint(0, 256, (H, W), dtype=torch.uint8, device="cuda", generator=g)
    right = torch.roll(left, -3, 1)
    d0 = 3.0 + torch.rand(H * W, dtype=torch.float64, device="cuda", generator=g)
    return left.ravel(), right.ravel().contiguous(), d0


def _refine_job(svb, W, H, **kw):
    refine = import_module(svb.__name__ + ".refine")
    r = refine.LRRefiner(W, H, **kw)
    left, right, d0 = _images(W, W, H)
    out = torch.empty(W * H, dtype=torch.float64, device="cuda")
    st = torch.empty(W * H, dtype=torch.uint8, device="cuda")
    return (lambda s: r.run(left, right, d0, out, st, stream=s)), [out, st]


@pytest.mark.parametrize("sizes,R,n", [
    (((1300, 4), (2000, 4)) * 2, 10, 3000),     # SGM rings of 7 and 8 warps
    (((720, 576), (1397, 1101)), 10, 200),
    (((450, 375), (640, 480)), 12, 200),
    (((600, 4), (2000, 4)) * 2, 40, 2000),
    (((4000, 2), (8000, 2)) * 2, 10, 2000),     # row kernels: a row in shared memory
])
def test_refiners_of_two_sizes(svb, sizes, R, n):
    _together([_refine_job(svb, W, H, R=R) for W, H in sizes], n)


def test_batches_of_two_widths(svb):
    jobs = []
    for W in (4000, 8000) * 2:
        b = svb.batch.BatchRefiner([(W, 2)] * 2)
        for i in range(2):
            for dst, src in zip((b.left[i], b.right[i], b.disp0[i]), _images(W + i, W, 2)):
                dst.copy_(src)
        jobs.append((lambda s, b=b: b.run(stream=s), b.out + b.status))
    _together(jobs, 1000)


def test_plane_snaps_of_two_steps(svb):
    lib = svb._lib.load()
    jobs = []
    for step in (21, 24) * 2:
        W, H = 96, 64
        g = torch.Generator(device="cuda").manual_seed(step)
        rgb = torch.rand(3 * W * H, dtype=torch.float64, device="cuda", generator=g)
        d = 5.0 + torch.rand(W * H, dtype=torch.float64, device="cuda", generator=g)
        out = torch.empty_like(d)
        need = lib.sv_postproc_workspace_size(W, H, step)
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")

        def call(s, d=d, rgb=rgb, out=out, ws=ws, need=need, step=step):
            p = lambda t: ctypes.c_void_p(t.data_ptr())
            svb._lib.check(lib.sv_plane_snap(p(d), p(rgb), 96, 64, None, step, 1.0, 0.3, 40,
                                             ctypes.c_uint32(7), p(out), p(ws), need, s), "snap")
        jobs.append((call, [out]))
    _together(jobs, 1000)


def test_forwards_of_two_dilations(svb):
    network = import_module(svb.__name__ + ".network")
    lib = svb._lib.load()
    jobs = []
    for dil in ((1, 7), (1, 8)) * 2:
        g = network.gpu_net(_forward_net(svb, dil, dil[1]))
        H = W = 200
        gen = torch.Generator(device="cuda").manual_seed(dil[1])
        new = lambda n: torch.rand(n, device="cuda", generator=gen)
        ins = [new(H * W), new(H * W), new(H * W // 4), new(H * W)]
        outs = [torch.empty(n, device="cuda") for n in (H * W // 16, H * W // 4, H * W)]
        need = lib.sv_forward_workspace_size(g.handle, H, W)
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")

        def call(s, g=g, ins=ins, outs=outs, ws=ws, need=need):
            p = lambda t: ctypes.c_void_p(t.data_ptr())
            svb._lib.check(lib.sv_stereonet_forward(
                g.handle, p(ins[0]), p(ins[1]), 200, 200, p(ins[2]), p(ins[3]), p(outs[0]),
                p(outs[1]), p(outs[2]), svb._lib.SV_FP32, p(ws), need, s), "forward")
        jobs.append((call, outs))
    _together(jobs, 1000)


def test_trainers_of_two_dilations(svb):
    train = import_module(svb.__name__ + ".train")
    lib = svb._lib.load()
    jobs = []
    for dil in ((6, 1), (8, 1)) * 2:
        t = train.Trainer(_train_net(svb, 8, 4, 4, dil, dil[0]))
        B, W, H = 1, 32, 32
        g = torch.Generator(device="cuda").manual_seed(dil[0])
        left, right, disp = (torch.rand(B * W * H, device="cuda", generator=g) for _ in range(3))
        valid = torch.ones(B * W * H, dtype=torch.uint8, device="cuda")
        loss = torch.empty(B, dtype=torch.float64, device="cuda")
        pred = torch.empty(B * W * H, device="cuda")
        need = lib.sv_train_workspace_size(t.handle, B, W, H)
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")

        def call(s, t=t, a=(left, right, disp, valid), loss=loss, pred=pred, ws=ws, need=need):
            p = lambda x: ctypes.c_void_p(x.data_ptr())
            svb._lib.check(lib.sv_train_grads(t.handle, p(a[0]), p(a[1]), p(a[2]), p(a[3]), 1, 32,
                                              32, p(loss), p(pred), p(ws), need, s), "grads")
        jobs.append((call, [loss, pred]))
    _together(jobs, 300)
