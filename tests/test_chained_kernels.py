"""Kernels that start while the one before them still runs: what they may assume of their inputs, and that a chain of them gives what
the same chain gives with the device idle between any two."""
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "csrc"


def _kernels(text):
    """(name, parameters, body) of every kernel of a source file."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params, at = text[m.end():at - 1], text.index("{", at)
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), params, text[at:end]


def test_inputs_of_chained_kernels_are_not_promised_constant():
    """A const __restrict__ pointer may be read before the wait, by a path that does not see the writes of a running kernel."""
    seen = {}
    for src in sorted(CSRC.glob("*.cu")):
        for name, params, body in _kernels(src.read_text()):
            if "chain_wait()" in body:
                seen[name] = [p.strip() for p in params.split(",") if "const " in p and "__restrict__" in p]
    assert len(seen) >= 8, sorted(seen)      # the norm, rotary, SwiGLU, store and product kernels
    assert not any(seen.values()), seen


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("rows", [1, 40])
def test_chain_of_short_kernels_is_that_of_separate_ones(rows, fp8):
    """Layers of a decode step (norm, products with and without clusters, rotary, store, attention, SwiGLU) over one set of buffers
    that every pass writes again: eager and from a graph, many times, bit for bit the results with a synchronisation after each."""
    from b200fw import ops
    dev, H, Hq, Hkv, I, L = "cuda", 1024, 16, 8, 3072, 6
    g = torch.Generator(device=dev).manual_seed(1)
    rnd = lambda *s, by=1.0: torch.randn(*s, device=dev, generator=g).mul(by).to(torch.bfloat16)
    layers = [dict(n1=1 + rnd(H, by=0.1), n2=1 + rnd(H, by=0.1), nq=1 + rnd(128, by=0.1), nk=1 + rnd(128, by=0.1),
                   qkv=rnd((Hq + 2 * Hkv) * 128, H, by=0.03), o=rnd(H, Hq * 128, by=0.03), gu=rnd(2 * I, H, by=0.03),
                   down=rnd(H, I, by=0.03)) for _ in range(L)]
    cos, sin = ops.rope_tables(256, 128, 1e6, torch.device(dev))
    blocks, lens = rows * 4, torch.randint(1, 64, (rows,), generator=torch.Generator().manual_seed(2))
    kind = torch.uint8 if fp8 else torch.bfloat16
    table = torch.randperm(blocks, device=dev, generator=g).int().view(rows, 4)
    ctx = lens.int().to(dev)
    pos = ctx - 1
    page = table.gather(1, (pos // 16).long()[:, None])[:, 0]
    segs = torch.stack([page, torch.arange(rows, device=dev).int(), torch.ones_like(page), pos % 16], 1).int().contiguous()
    first, old_k, old_v = rnd(rows, H), rnd(blocks, 16, Hkv, 128), rnd(blocks, 16, Hkv, 128)
    if fp8:
        old_k, old_v = (t.to(torch.float8_e4m3fn).view(torch.uint8) for t in (old_k, old_v))
    kc, vc, h = torch.empty_like(old_k), torch.empty_like(old_v), torch.empty_like(first)
    ks, vs = (torch.empty(blocks, Hkv, device=dev) if fp8 else None for _ in range(2))

    def chain(between):
        h.copy_(first), kc.copy_(old_k), vc.copy_(old_v)
        if fp8:
            ks.fill_(1.0), vs.fill_(1.0)
        x = h
        for w in layers:
            def step(f, *a, **k):
                r = f(*a, **k)
                between()
                return r
            y = step(ops.rmsnorm, x, w["n1"])
            y = step(ops.linear, y, w["qkv"])
            q, k, v = step(ops.qknorm_rope, y, w["nq"], w["nk"], pos, cos, sin, Hq, Hkv, 128)
            step(ops.kv_store, k, v, kc, vc, segs, ks, vs)
            y = step(ops.paged_decode_attention, q, kc, vc, table, ctx, Hq, k_scale=ks, v_scale=vs)
            x = step(ops.linear, y, w["o"], x)
            y = step(ops.rmsnorm, x, w["n2"])
            y = step(ops.swiglu, step(ops.linear, y, w["gu"]))
            x = step(ops.linear, y, w["down"], x)
        return x

    with torch.no_grad():
        want = chain(torch.cuda.synchronize).clone()
        assert want.dtype == torch.bfloat16 and kc.dtype == kind and bool(torch.isfinite(want).all())
        for _ in range(20):
            assert torch.equal(chain(lambda: None), want)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            chain(lambda: None)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = chain(lambda: None)
        for _ in range(50):
            out.zero_()
            graph.replay()
            assert torch.equal(out, want)
