"""Decode attention and products with few rows against 64-bit references, at the sizes where their splits change."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _error(got, want):
    """Relative error in the 2-norm, and that of the 64-bit result rounded to bf16 (which no bf16 output can do without)."""
    want = want.double().cpu()
    d = lambda t: float((t.double().cpu() - want).norm() / want.norm().clamp(min=1e-30))
    return d(got), d(want.to(torch.bfloat16))


def _decode_reference(q, kc, vc, bt, lens, Hq, ks, vs):
    Hkv = kc.shape[2]
    K, V = (t.view(torch.float8_e4m3fn).double() * s.double()[:, None, :, None] if s is not None else t.double()
            for t, s in ((kc, ks), (vc, vs)))
    out = torch.zeros(q.shape, dtype=torch.float64, device=DEV)
    for b, n in enumerate(lens):
        if n:
            pos = torch.arange(n, device=DEV)
            at = bt[b, pos // 16].long() * 16 + pos % 16
            k, v = K.reshape(-1, Hkv, 128)[at], V.reshape(-1, Hkv, 128)[at]
            s = torch.einsum("hgd,nhd->hgn", q[b].double().reshape(Hkv, Hq // Hkv, 128), k) / math.sqrt(128)
            out[b] = torch.einsum("hgn,nhd->hgd", s.softmax(-1), v).reshape(-1)
    return out


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (4, 2), (6, 2), (8, 2), (5, 1), (8, 1)])     # 1, 2, 3, 4, 5 and 8 heads per kv head
@pytest.mark.parametrize("lens", [[1], [0, 5, 16, 17], [63, 64, 65, 130, 257], [2000, 1]])
def test_decode_attention_over_clusters(fp8, Hq, Hkv, lens):
    """Contexts of no token, of less than a page and of unequal parts; pages past the end hold NaN; scales differ per page."""
    from b200fw.ops import paged_decode_attention
    g = torch.Generator(device=DEV).manual_seed(1)
    need = [-(-n // 16) for n in lens]
    blocks = sum(need) + 1
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    kc, vc = rnd(blocks, 16, Hkv, 128), rnd(blocks, 16, Hkv, 128)
    perm = torch.randperm(blocks - 1, device=DEV, generator=g)
    bt = torch.full((len(lens), 160), -1, dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(need):
        bt[b, :n] = perm[at:at + n].int()
        if lens[b] % 16:      # rows past the end of the context
            kc[bt[b, n - 1].long(), lens[b] % 16:] = math.nan
            vc[bt[b, n - 1].long(), lens[b] % 16:] = math.nan
        at += n
    ks = vs = None
    if fp8:
        kc, vc = (t.to(torch.float8_e4m3fn).view(torch.uint8) for t in (kc, vc))
        ks, vs = (10.0 ** (-4 + 4 * torch.rand(blocks, Hkv, device=DEV, generator=g)) for _ in range(2))
    else:
        kc, vc = kc.to(torch.bfloat16), vc.to(torch.bfloat16)
    q = rnd(len(lens), Hq * 128).to(torch.bfloat16)
    cl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    want = _decode_reference(q, kc, vc, bt, lens, Hq, ks, vs)
    for part, nsplit in ((0, 1), (64, max(1, -(-max(lens) // 64)))):
        got, floor = _error(paged_decode_attention(q, kc, vc, bt, cl, Hq, k_scale=ks, v_scale=vs, partition=part, nsplit=nsplit), want)
        # rounding the output, plus 32-bit scores of up to about 30 and their exponentials
        assert got <= 1.02 * floor + 2e-5, (part, nsplit, got, floor)


@pytest.mark.parametrize("v_exp", [[None, None], [None, 0], [0, None], [-90, -90], [-60, -90], [100, -20], [118, 118]])
@pytest.mark.parametrize("q_exp", [-110, 0, 110])
def test_fp8_decode_over_the_range_of_scales(v_exp, q_exp):
    """Value scales of zero (None: an all-zero page as other writers leave it), tiny and large powers of two; queries whose scores
    are nearly all zero, ordinary, or so large that one key takes everything."""
    from b200fw.ops import paged_decode_attention
    g = torch.Generator(device=DEV).manual_seed(10)
    Hkv, n = 2, 300
    pages = -(-n // 16)
    kc, vc = (torch.randn(pages, 16, Hkv, 128, device=DEV, generator=g).to(torch.float8_e4m3fn).view(torch.uint8) for _ in range(2))
    ks = torch.full((pages, Hkv), 2.0 ** -8, device=DEV)
    vs = torch.zeros(pages, Hkv, device=DEV)
    for i, e in enumerate(v_exp):      # pages take turns
        vs[i::2] = 0.0 if e is None else 2.0 ** e
    q = (torch.randn(1, 4 * 128, device=DEV, generator=g) * 2.0 ** q_exp).to(torch.bfloat16)
    bt, cl = torch.arange(pages, device=DEV).int().view(1, -1), torch.tensor([n], device=DEV).int()
    want = _decode_reference(q, kc, vc, bt, [n], 4, ks, vs)
    for part, nsplit in ((0, 1), (64, 5)):
        out = paged_decode_attention(q, kc, vc, bt, cl, 4, k_scale=ks, v_scale=vs, partition=part, nsplit=nsplit)
        assert bool(torch.isfinite(out).all())
        if v_exp == [None, None]:
            assert not out.any()
            continue
        got, floor = _error(out, want)
        assert got <= 1.02 * floor + 2e-5, (part, got, floor)      # as in test_decode_attention_over_clusters


@pytest.mark.parametrize("G", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n,split", [(5, (0, 1)), (200, (0, 1)), (200, (64, 4))])
def test_decode_attention_with_infinite_values(G, n, split):
    """An infinity (or NaN) in one channel of one cached value reaches that channel of the output and nothing else."""
    from b200fw.ops import paged_decode_attention
    g = torch.Generator(device=DEV).manual_seed(11)
    pages, Hkv = -(-n // 16), 2
    kc, vc = (torch.randn(pages, 16, Hkv, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    flat = vc.view(-1, Hkv, 128)
    flat[1, 0, 3] = flat[n - 1, 0, 100] = math.inf
    flat[2, 0, 64] = flat[3, 1, 5] = -math.inf
    flat[4, 1, 127] = math.nan
    q = torch.randn(1, G * Hkv * 128, device=DEV, generator=g).mul(0.5).to(torch.bfloat16)
    bt, cl = torch.arange(pages, device=DEV).int().view(1, -1), torch.tensor([n], device=DEV).int()
    want = _decode_reference(q, kc, vc, bt, [n], G * Hkv, None, None)
    out = paged_decode_attention(q, kc, vc, bt, cl, G * Hkv, partition=split[0], nsplit=split[1]).double()
    odd = ~torch.isfinite(want)
    assert int(odd.sum()) == 5 * G and torch.equal(out[odd].nan_to_num(7.0), want[odd].nan_to_num(7.0))
    got, floor = _error(out[~odd], want[~odd])
    assert got <= 1.02 * floor + 2e-5, (got, floor)      # as in test_decode_attention_over_clusters


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("Hq,Hkv,lens", [
    (16, 8, [4999, 1, 2100, 2049, 4096, 15, 3000, 700]),              # 64 pairs: clusters of four
    (32, 8, [2561, 2560, 5000] + [130] * 13),                         # 128 pairs: clusters of two, over 32 pages a warp
    (8, 4, [2048, 2049, 2064, 2065, 4500, 4112] + [33] * 58),         # 256 pairs: four warps a context
    (12, 4, [1024, 1025, 1040, 1041, 2300, 2072] + [40] * 294),       # 1200 pairs: two warps a context
])
def test_decode_attention_of_long_contexts(fp8, Hq, Hkv, lens):
    """Every cluster size, and more than 32 pages a warp: page numbers and scales are then fetched again."""
    from b200fw.ops import paged_decode_attention
    g = torch.Generator(device=DEV).manual_seed(13)
    need = [-(-n // 16) for n in lens]
    blocks = sum(need)
    kc, vc = (torch.randn(blocks, 16, Hkv, 128, device=DEV, generator=g) for _ in range(2))
    kc, vc = (t.to(torch.float8_e4m3fn).view(torch.uint8) if fp8 else t.to(torch.bfloat16) for t in (kc, vc))
    ks, vs = (10.0 ** (-2 + 2 * torch.rand(blocks, Hkv, device=DEV, generator=g)) if fp8 else None for _ in range(2))
    perm = torch.randperm(blocks, device=DEV, generator=g).int()
    bt = torch.full((len(lens), max(need)), -1, dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(need):
        bt[b, :n] = perm[at:at + n]
        at += n
    q = torch.randn(len(lens), Hq * 128, device=DEV, generator=g).to(torch.bfloat16)
    cl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got, floor = _error(paged_decode_attention(q, kc, vc, bt, cl, Hq, k_scale=ks, v_scale=vs),
                        _decode_reference(q, kc, vc, bt, lens, Hq, ks, vs))
    assert got <= 1.02 * floor + 2e-5, (got, floor)      # as in test_decode_attention_over_clusters


def test_decode_attention_of_many_pairs_and_unaligned_queries():
    """So many (sequence, kv head) pairs that CTAs of two warps run; queries two bytes off a vector's alignment."""
    from b200fw.ops import paged_decode_attention
    g = torch.Generator(device=DEV).manual_seed(2)
    B, Hq, Hkv = 300, 8, 4
    lens = torch.randint(1, 70, (B,), generator=torch.Generator().manual_seed(3)).tolist()
    kc, vc = (torch.randn(B * 5, 16, Hkv, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    bt = torch.arange(B * 5, device=DEV, dtype=torch.int32).reshape(B, 5)
    flat = torch.randn(B * Hq * 128 + 1, device=DEV, generator=g).to(torch.bfloat16)
    q = flat[1:].view(B, Hq * 128)
    cl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got, floor = _error(paged_decode_attention(q, kc, vc, bt, cl, Hq), _decode_reference(q, kc, vc, bt, lens, Hq, None, None))
    assert got <= 1.02 * floor + 2e-5, (got, floor)


@pytest.mark.parametrize("b_mn", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1024, 1024), (7, 776, 1032), (128, 200, 2056), (300, 72, 1544)])
@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("cluster", [1, 2, 4, 8])
def test_cluster_products(b_mn, M, N, K, bn, cluster):
    """Every tile width and cluster size, whatever the shape would choose: bf16 and fp32 outputs, residual, accumulation."""
    from b200fw import _native as nv
    g = torch.Generator(device=DEV).manual_seed(4)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    a, b, r = rnd(M, K).to(torch.bfloat16), rnd(*((K, N) if b_mn else (N, K))).to(torch.bfloat16), rnd(M, N).to(torch.bfloat16)
    prod = a.double() @ (b.double() if b_mn else b.double().t())
    wide = torch.zeros(M, N + 8, device=DEV, dtype=torch.bfloat16)     # a strided output: nothing past its columns
    f32 = rnd(M, N)
    acc = r.clone()
    for out, res, flags, want in ((wide[:, :N], None, 0, prod), (torch.empty_like(r), r, 4, prod + r.double()),
                                  (acc, None, 2, prod + r.double()), (f32, None, 3, prod + f32.double())):
        nv.check(nv.lib().b2_gemm_bf16_cluster(nv.ptr(a), nv.ptr(b), nv.ptr(out), nv.ptr(res), M, N, K, a.stride(0), b.stride(0),
                                               out.stride(0), b_mn, flags, bn, cluster, 0, 0, nv.stream_ptr()), "cluster")
        got, floor = _error(out, want)
        # 32-bit sums of K terms in a fixed order: well below sqrt(K) * 2^-24 of the result, 1e-5 with room to spare
        assert got <= (1.02 * floor if flags != 3 else 0.0) + 1e-5, (flags, got, floor)
    assert float(wide[:, N:].abs().max()) == 0.0
    nv.assert_ok()


@pytest.mark.parametrize("bn", [0, 128, 256])      # 0: the dispatch's own choice (a cluster)
@pytest.mark.parametrize("M,N", [(5, 1028), (130, 36), (3, 20)])
def test_residual_beside_fp32_rows_of_four(bn, M, N):
    """Rows of 4 n elements: every other row of the bf16 addend starts 8 bytes off a vector of 16."""
    from b200fw.ops import gemm
    g = torch.Generator(device=DEV).manual_seed(8)
    a, b, r = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((M, 2048), (N, 2048), (M, N)))
    got, _ = _error(gemm(a, b, residual=r, out_dtype=torch.float32, bn=bn), a.double() @ b.double().t() + r.double())
    assert got <= 1e-5, got      # 32-bit sums, as in test_cluster_products


@pytest.mark.parametrize("bn", [0, 128, 256])      # 0: the dispatch's own choice (a cluster for the smaller two)
@pytest.mark.parametrize("M,N,K", [(5, 1024, 2048), (130, 72, 2048), (300, 776, 520), (3000, 1000, 256)])
def test_addend_and_accumulation_together(bn, M, N, K):
    """out += a b^T + residual, in both output types and by both kernels."""
    from b200fw.ops import gemm
    g = torch.Generator(device=DEV).manual_seed(9)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    a, b, r = rnd(M, K).to(torch.bfloat16), rnd(N, K).to(torch.bfloat16), rnd(M, N).to(torch.bfloat16)
    for old in (rnd(M, N).mul(20).to(torch.bfloat16), rnd(M, N).mul(20)):
        want = a.double() @ b.double().t() + old.double() + r.double()
        got, floor = _error(gemm(a, b, out=old, accumulate=True, residual=r, bn=bn), want)
        assert got <= (1.02 * floor if old.dtype == torch.bfloat16 else 0.0) + 1e-5, (got, floor)      # as in test_cluster_products


@pytest.mark.parametrize("act", ["silu", "relu2"])
@pytest.mark.parametrize("M", [1, 33, 256])
def test_products_with_few_rows_take_every_epilogue(act, M):
    """Through the public entry points, at a shape that the dispatch gives to clusters, against the persistent kernel too."""
    from b200fw.ops import gemm
    from b200fw.ops.gemm import linear_act
    g = torch.Generator(device=DEV).manual_seed(5)
    a, b = (torch.randn(*s, device=DEV, generator=g).mul(0.2).to(torch.bfloat16) for s in ((M, 3072), (1024, 3072)))
    prod = a.double() @ b.double().t()
    z = prod[:, :520]
    want = prod.clone()
    want[:, :520] = z * torch.sigmoid(z) if act == "silu" else z.clamp(min=0) ** 2
    got, floor = _error(linear_act(a, b, act, 520), want)
    assert got <= 1.05 * floor + 2e-5, (got, floor)
    got, floor = _error(gemm(a, b), prod)
    assert got <= 1.02 * floor + 1e-5
    got, floor = _error(gemm(a, b, bn=128), prod)       # a given width keeps the persistent kernel
    assert got <= 1.02 * floor + 1e-5
    assert torch.equal(gemm(a, b), gemm(a, b))


@pytest.mark.parametrize("M,H", [(1, 1024), (7, 256), (2500, 1000), (300, 2048), (2400, 2560), (33, 3072), (40, 3080), (50, 4096), (20, 5120)])
@pytest.mark.parametrize("frozen", [False, True])
def test_rmsnorm_backward_over_row_lengths(M, H, frozen):
    """Row lengths on either side of each register layout, whole and ragged warps, a frozen weight (no column sums)."""
    from b200fw.ops import rmsnorm
    g = torch.Generator(device=DEV).manual_seed(6)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x, w, dy = rnd(M, H).to(torch.bfloat16).requires_grad_(), (1 + 0.1 * rnd(H)).to(torch.bfloat16), rnd(M, H).to(torch.bfloat16)
    w.requires_grad_(not frozen)
    rmsnorm(x, w).backward(dy)
    xd, wd = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    (xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * wd).backward(dy.double())
    got, floor = _error(x.grad, xd.grad)
    assert got <= 1.02 * floor + 1e-5, (got, floor)       # 32-bit arithmetic on the way to a bf16 result
    if frozen:
        assert w.grad is None
    else:
        got, floor = _error(w.grad, wd.grad)
        assert got <= 1.02 * floor + 1e-5, (got, floor)


def test_attention_backward_of_ragged_rows():
    """231 rows of dO * O: the last warp of the row sums is not full."""
    from b200fw.ops import flash_attention
    g = torch.Generator(device=DEV).manual_seed(7)
    B, S, Hq, Hkv = 1, 77, 3, 1
    q, k, v = (torch.randn(B * S, h * 128, device=DEV, generator=g).to(torch.bfloat16).requires_grad_() for h in (Hq, Hkv, Hkv))
    dy = torch.randn(B * S, Hq * 128, device=DEV, generator=g).to(torch.bfloat16)
    flash_attention(q, k, v, B, S, Hq, Hkv).backward(dy)
    qd, kd, vd = (t.detach().double().requires_grad_() for t in (q, k, v))
    s = torch.einsum("qhd,kd->hqk", qd.reshape(S, Hq, 128), kd) / math.sqrt(128)
    s = s.masked_fill(torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1), -math.inf).softmax(-1)
    torch.einsum("hqk,kd->qhd", s, vd).reshape(S, -1).backward(dy.double())
    for a, b in ((q, qd), (k, kd), (v, vd)):
        # P and dS are bf16 operands of the gradient products: 2^-9 each, a few of them added up
        assert _error(a.grad, b.grad)[0] < 1e-2


@pytest.mark.parametrize("bn", [0, 128])      # cluster, persistent kernel
def test_failed_launch_is_reported_once(bn):
    """A product on a stream whose capture has been invalidated is refused by the runtime; the next operation is not."""
    import ctypes
    from b200fw.ops import gemm, rmsnorm
    a, b, w = (torch.ones(*s, device=DEV, dtype=torch.bfloat16) for s in ((5, 2048), (1024, 2048), (1024,)))
    out, want = gemm(a, b, bn=bn), rmsnorm(torch.ones(5, 1024, device=DEV, dtype=torch.bfloat16), w)
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream()
    raw, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    with torch.cuda.stream(stream):
        assert rt.cudaStreamBeginCapture(raw, 2) == 0
        assert rt.cudaStreamSynchronize(raw) != 0      # not allowed while capturing: the capture is invalid from here on
        with pytest.raises(RuntimeError, match="launch failed"):
            gemm(a, b, out=out, bn=bn)
        assert rt.cudaStreamEndCapture(raw, ctypes.byref(graph)) != 0
    rt.cudaGetLastError()
    assert torch.equal(rmsnorm(out.mul(0).add(1), w), want)


_SAME_IN_ANY_BATCH = """
import torch
from b200fw import ops
g = torch.Generator(device="cuda").manual_seed(12)
rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
for n, k in ((1024, 3072), (4096, 1024), (2560, 9728)):
    x, w, r = rnd(1100, k), rnd(n, k), rnd(1100, n)
    alone = ops.linear(x[:1], w, r[:1])
    for m in (2, 64, 130, 1100):
        assert torch.equal(ops.linear(x[:m], w, r[:m])[:1], alone), (n, k, m)
x, w, first = rnd(1100, 3072), rnd(4096, 3072), rnd(1100, 4096).float()      # 32-bit outputs, added to what is there or not
for add in (False, True):
    run = lambda m: ops.gemm(x[:m], w, out=first[:m].clone(), accumulate=add)
    alone = run(1)
    for m in (2, 64, 130, 1100):
        assert torch.equal(run(m)[:1], alone), (add, m)
B, Hq, Hkv, n = 300, 16, 8, 700
pages = -(-n // 16)
kc, vc, q = rnd(4 * pages, 16, Hkv, 128), rnd(4 * pages, 16, Hkv, 128), rnd(B, Hq * 128)
table = (torch.arange(pages)[None] + pages * (torch.arange(B) % 4)[:, None]).int().cuda()
lens = torch.full((B,), n, dtype=torch.int32, device="cuda")
for fp8 in (False, True):
    if fp8:
        kc, vc = (t.to(torch.float8_e4m3fn).view(torch.uint8) for t in (kc, vc))
    s = torch.rand(4 * pages, Hkv, device="cuda", generator=g) if fp8 else None
    run = lambda b: ops.paged_decode_attention(q[:b], kc, vc, table[:b].contiguous(), lens[:b], Hq, k_scale=s, v_scale=s)
    alone = run(1)
    for b in (3, 20, 70, B):
        assert torch.equal(run(b)[:1], alone), (fp8, b)
"""


def test_results_do_not_depend_on_the_batch_where_asked():
    """With B200FW_BATCH_INVARIANT=1 (read once, hence a process of its own) a row is the same alone and among others."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SAME_IN_ANY_BATCH], cwd=root, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "B200FW_BATCH_INVARIANT": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
