"""Kernels set up before the one ahead has ended: same results in chains, in a
captured graph replayed on new inputs, and beside another stream's chain.

Whole numbers and bytes throughout (the refined disparities are exact FP64
arithmetic), so results must be equal, not close."""

from importlib import import_module

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(svb, seed, W, H):
    p = svb.synth.make_pair(seed, W, H, 1.0, 20.0)
    rng = np.random.default_rng(seed)
    d0 = np.clip(p.disp.ravel() + rng.normal(0, 1.0, W * H), 0, None)
    u8 = lambda a: torch.as_tensor(a.astype(np.uint8).ravel(), device="cuda")
    return [u8(p.left), u8(p.right), torch.as_tensor(d0, device="cuda")]


@pytest.mark.parametrize("W,H", [(97, 61), (320, 200)])
def test_graph_and_streams_match_plain_runs(svb, W, H):
    refine = import_module(svb.__name__ + ".refine")
    sets = [_inputs(svb, s, W, H) for s in (1, 2, 3)]
    r = refine.LRRefiner(W, H)
    new = lambda: (torch.empty(W * H, dtype=torch.float64, device="cuda"),
                   torch.empty(W * H, dtype=torch.uint8, device="cuda"))
    want = []
    for s in sets:
        o, st = new()
        r.run(*s, o, st)
        torch.cuda.synchronize()
        want.append((o.clone(), st.clone()))
    # captured once, replayed on the other inputs
    cur = [t.clone() for t in sets[0]]
    o, st = new()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        r.run(*cur, o, st)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.run(*cur, o, st)
    for s, (wo, ws) in zip(sets, want):
        for a, b in zip(cur, s):
            a.copy_(b)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(o, wo) and torch.equal(st, ws)
    # two refiners on two streams, chains of runs without a host wait between
    r2 = refine.LRRefiner(W, H)
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[new() for _ in sets] for _ in streams]
    torch.cuda.synchronize()
    for k, s in enumerate(sets):
        for obj, stream, res in zip((r, r2), streams, outs):
            with torch.cuda.stream(stream):
                obj.run(*s, *res[k])
    torch.cuda.synchronize()
    for res in outs:
        for (a, b), (wo, ws) in zip(res, want):
            assert torch.equal(a, wo) and torch.equal(b, ws)
