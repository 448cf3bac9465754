"""Numerics of every sm_100a kernel against the fp32 PyTorch restatement of the same op
(hcache_deepspeed_b200.ops.reference). Mirrors the reference's per-kernel tests
(tests/unit/inference/v2/kernels/{core_ops,ragged_ops}/*, tolerances inference_test_utils.py:14-22)."""
import math

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

from hcache_deepspeed_b200.ops import reference as ref  # noqa: E402

DTYPES = [torch.bfloat16, torch.float16]


def tol(dtype):
    # bf16 has 8 bits of mantissa: one rounding of the output is 2^-8 relative
    return dict(rtol=1.6e-2, atol=2e-2) if dtype == torch.bfloat16 else dict(rtol=4e-3, atol=4e-3)


def K():
    from hcache_deepspeed_b200.ops import kernels
    return kernels


def rand(*shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(dtype)


# ------------------------------------------------------------------------------------------------
# GEMM
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K_,bn", [
    (128, 256, 128, 0), (300, 520, 192, 0), (16, 4096, 4096, 0), (1, 1024, 512, 32), (77, 384, 320, 64),
    (2048, 1024, 1024, 256), (512, 768, 2048, 128), (9, 11008 // 8 * 2, 4096, 0),
])
def test_gemm_store(dtype, M, N, K_, bn):
    torch.manual_seed(0)
    a, w = rand(M, K_, dtype=dtype), rand(N, K_, dtype=dtype, scale=K_ ** -0.5)
    out = K().gemm(a, w, bn=bn)
    torch.cuda.synchronize()
    want = ref.gemm(a, w, out_dtype=torch.float32)
    torch.testing.assert_close(out.float(), want, **tol(dtype))


@pytest.mark.parametrize("M,N,K_,bn,splits,gated", [(16, 4096, 4096, 128, 4, False), (1, 12288, 4096, 0, 0, False),
                                                    (64, 2 * 1376, 2048, 64, 3, True), (100, 520, 1024, 128, 2, False),
                                                    (8, 22016, 4096, 0, 0, True)])
def test_gemm_store_splitk(M, N, K_, bn, splits, gated):
    torch.manual_seed(12)
    a, w, b = rand(M, K_), rand(N, K_, scale=K_ ** -0.5), rand(N)
    ws = torch.zeros(K().gemm_splitk_workspace_bytes(M, N), dtype=torch.uint8, device="cuda")
    want = ref.gemm(a, w, bias=b, act=3 if gated else 0, gated=gated, out_dtype=torch.float32)
    for _ in range(2):  # second call: scratch must have been left zeroed
        out = K().gemm(a, w, bias=b, act=3 if gated else 0, gated=gated, bn=bn, splits=splits, workspace=ws)
        torch.testing.assert_close(out.float(), want, **tol(torch.bfloat16))
    assert int(ws.view(torch.int32).abs().max()) == 0


@pytest.mark.parametrize("M,N,K_", [(8, 4096, 4096), (64, 1000, 520), (300, 2 * 688, 1024), (1, 96, 64)])
def test_gemm_tiled_weights(M, N, K_):
    """pre-tiled weight layout: same results as the row-major operand for store / gated / accum epilogues"""
    torch.manual_seed(13)
    k = K()
    a, w, b = rand(M, K_), rand(N, K_, scale=K_ ** -0.5), rand(N)
    wt = k.TiledWeight.from_dense(w)
    torch.testing.assert_close(wt.to_dense(), w, rtol=0, atol=0)
    want = ref.gemm(a, w, bias=b, out_dtype=torch.float32)
    torch.testing.assert_close(k.gemm(a, wt, bias=b).float(), want, **tol(torch.bfloat16))
    if N % 2 == 0:
        wantg = ref.gemm(a, w, act=3, gated=True, out_dtype=torch.float32)
        torch.testing.assert_close(k.gemm(a, wt, act=3, gated=True).float(), wantg, **tol(torch.bfloat16))
    acc = torch.zeros(M, N, device="cuda")
    k.gemm_accum(a, wt, acc, bias=b)
    torch.testing.assert_close(acc, want, rtol=2e-3, atol=2e-3)
    if N >= 64:
        sub = wt.rows_from(32)
        torch.testing.assert_close(k.gemm(a, sub).float(), ref.gemm(a, w[32:], out_dtype=torch.float32), **tol(torch.bfloat16))


@pytest.mark.parametrize("act", [1, 2, 3, 4])
def test_gemm_bias_act(act):
    torch.manual_seed(1)
    M, N, K_ = 200, 640, 256
    a, w, b = rand(M, K_), rand(N, K_, scale=K_ ** -0.5), rand(N)
    out = K().gemm(a, w, bias=b, act=act)
    want = ref.gemm(a, w, bias=b, act=act, out_dtype=torch.float32)
    torch.testing.assert_close(out.float(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("mode", ["store", "gated", "accum"])
@pytest.mark.parametrize("use_ws", [False, True])
def test_gemm_skinny(dtype, M, mode, use_ws):
    """Decode-size M takes the feature-major weight-streaming kernel (gemm_skinny.cuh): ragged N and K, every token
    tile (16/32/64; bn=-1 forces the kernel for every M <= 64), with and without split-K scratch; scratch must come back zeroed."""
    torch.manual_seed(M)
    N, K_ = (690 if mode == "gated" else 1000), 2120
    a, w, b = rand(M, K_, dtype=dtype), rand(N, K_, dtype=dtype, scale=K_ ** -0.5), rand(N, dtype=dtype)
    ws = torch.zeros(K().gemm_splitk_workspace_bytes(M, N), dtype=torch.uint8, device="cuda") if use_ws else None
    for rep in range(2):
        if mode == "accum":
            acc = torch.zeros(M, N, device="cuda", dtype=torch.float32)
            K().gemm_accum(a, w, acc, bias=b, bn=-1)
            want = ref.gemm(a, w, bias=b, out_dtype=torch.float32)
            torch.testing.assert_close(acc, want, rtol=2e-3, atol=2e-3)
        else:
            gated = mode == "gated"
            out = K().gemm(a, w, bias=b, act=3 if gated else 2, gated=gated, workspace=ws, bn=-1)
            want = ref.gemm(a, w, bias=b, act=3 if gated else 2, gated=gated, out_dtype=torch.float32)
            torch.testing.assert_close(out.float(), want, **tol(dtype))
    if ws is not None:
        assert int(ws.view(torch.int32).abs().max()) == 0


@pytest.mark.parametrize("M", [5, 128, 700])
def test_gemm_gated(M):
    torch.manual_seed(2)
    N, K_ = 2 * 688, 512
    a, w = rand(M, K_), rand(N, K_, scale=K_ ** -0.5)
    out = K().gemm(a, w, act=3, gated=True)
    assert out.shape == (M, N // 2)
    want = ref.gemm(a, w, act=3, gated=True, out_dtype=torch.float32)
    torch.testing.assert_close(out.float(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("M,N,K_,splits", [(8, 4096, 4096, 0), (64, 512, 11008, 4), (300, 1024, 1024, 2), (16, 256, 64, 0)])
def test_gemm_accum_splitk(M, N, K_, splits):
    torch.manual_seed(3)
    a, w, b = rand(M, K_), rand(N, K_, scale=K_ ** -0.5), rand(N)
    acc = torch.zeros(M, N, device="cuda", dtype=torch.float32)
    K().gemm_accum(a, w, acc, bias=b, splits=splits)
    want = ref.gemm(a, w, bias=b, out_dtype=torch.float32)
    torch.testing.assert_close(acc, want, rtol=2e-3, atol=2e-3)
    K().gemm_accum(a, w, acc, bias=b, splits=splits)  # accumulates on top
    torch.testing.assert_close(acc, 2 * want, rtol=2e-3, atol=4e-3)


# ------------------------------------------------------------------------------------------------
# norms
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("cols", [768, 4096, 5120, 8192])
@pytest.mark.parametrize("layer_norm", [False, True])
def test_norm_plain(dtype, cols, layer_norm):
    torch.manual_seed(4)
    x, g, b = rand(37, cols, dtype=dtype), rand(cols, dtype=dtype), rand(cols, dtype=dtype)
    out = torch.empty_like(x)
    K().norm(x, g, out, beta=b if layer_norm else None, eps=1e-5, layer_norm=layer_norm)
    want = ref.norm(x, g, b if layer_norm else None, 1e-5, layer_norm)
    torch.testing.assert_close(out.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("delta_f32", [False, True])
@pytest.mark.parametrize("layer_norm", [False, True])
def test_norm_residual(delta_f32, layer_norm):
    torch.manual_seed(5)
    rows, cols = 19, 4096
    x, g, b = rand(rows, cols), rand(cols), rand(cols)
    delta = torch.randn(rows, cols, device="cuda") if delta_f32 else rand(rows, cols)
    delta_in = delta.clone()
    res = torch.empty_like(x)
    out = torch.empty_like(x)
    K().norm(x, g, out, beta=b if layer_norm else None, delta=delta, zero_delta=True, res_out=res, eps=1e-6,
             layer_norm=layer_norm)
    want_res = (x.float() + delta_in.float()).to(torch.bfloat16)
    want = ref.norm(want_res, g, b if layer_norm else None, 1e-6, layer_norm)
    torch.testing.assert_close(res.float(), want_res.float(), rtol=0, atol=0)
    torch.testing.assert_close(out.float(), want.float(), **tol(torch.bfloat16))
    if delta_f32:
        assert float(delta.abs().max()) == 0.0  # consumed and zeroed


def test_norm_gather_rows():
    torch.manual_seed(6)
    x, g = rand(50, 2048), rand(2048)
    idx = torch.tensor([49, 0, 7, 7, 31], device="cuda", dtype=torch.int32)
    out = torch.empty(5, 2048, device="cuda", dtype=torch.bfloat16)
    K().norm(x, g, out, row_idx=idx, eps=1e-5)
    want = ref.norm(x[idx.long()], g, None, 1e-5, False)
    torch.testing.assert_close(out.float(), want.float(), **tol(torch.bfloat16))


# ------------------------------------------------------------------------------------------------
# ragged helpers
# ------------------------------------------------------------------------------------------------
def make_cache(n_blocks, n_kv, bs, d, dtype=torch.bfloat16):
    return torch.zeros(n_blocks, 2, n_kv, bs, d, device="cuda", dtype=dtype)


def make_slots(T, n_blocks, bs, seed=0):
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(n_blocks * bs, generator=g)[:T]
    return perm.to(torch.int32).cuda()


@pytest.mark.parametrize("max_pos", [5000, 200000])     # long contexts: the in-kernel range reduction must hold up
@pytest.mark.parametrize("d,rd,n_q,n_kv", [(128, 128, 4, 4), (128, 128, 8, 2), (64, 64, 12, 12), (80, 32, 4, 4), (96, 96, 2, 1)])
def test_rope_kv_append(d, rd, n_q, n_kv, max_pos):
    torch.manual_seed(7)
    T, bs, n_blocks = 45, 64, 6
    qkv = rand(T, (n_q + 2 * n_kv) * d)
    pos = torch.randint(max_pos // 2, max_pos, (T,), device="cuda", dtype=torch.int32)
    slot = make_slots(T, n_blocks, bs)
    slot[3] = -1
    inv = ref.default_inv_freq(rd, device="cuda")
    cache = make_cache(n_blocks, n_kv, bs, d)
    q_out = torch.empty(T, n_q * d, device="cuda", dtype=torch.bfloat16)
    K().rope_kv_append(qkv, q_out, cache, pos, slot, inv, n_q, n_kv, d, rd, bs)
    q, k, v = qkv.split([n_q * d, n_kv * d, n_kv * d], dim=1)
    want_q = ref.rope_rotate_half(q.view(T, n_q, d), pos, inv, rd)
    want_k = ref.rope_rotate_half(k.reshape(T, n_kv, d), pos, inv, rd)
    want_cache = make_cache(n_blocks, n_kv, bs, d)
    ref.kv_append(want_cache, want_k, v.reshape(T, n_kv, d), slot)
    torch.testing.assert_close(q_out.view(T, n_q, d).float(), want_q.float(), **tol(torch.bfloat16))
    torch.testing.assert_close(cache.float(), want_cache.float(), **tol(torch.bfloat16))


def test_embed_gather_argmax_cvt():
    torch.manual_seed(8)
    V, H, T = 1000, 768, 33
    W, P = rand(V, H), rand(64, H)
    ids = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    pos = torch.randint(0, 60, (T,), device="cuda", dtype=torch.int32)
    out = torch.empty(T, H, device="cuda", dtype=torch.bfloat16)
    K().embed(ids, W, out, pos_weight=P, tok_pos=pos, pos_offset=2)
    want = ref.embed(ids, W, P, pos, 2)
    torch.testing.assert_close(out.float(), want.float(), rtol=1e-2, atol=1e-2)
    K().embed(ids, W, out)
    torch.testing.assert_close(out, W[ids.long()], rtol=0, atol=0)

    idx = torch.tensor([5, 1, 32], device="cuda", dtype=torch.int32)
    g = torch.empty(3, H, device="cuda", dtype=torch.bfloat16)
    K().gather_rows(out, idx, g)
    torch.testing.assert_close(g, out[idx.long()], rtol=0, atol=0)

    logits = rand(7, 32000)
    got = K().argmax(logits)
    assert got.tolist() == logits.float().argmax(-1).tolist()
    lf = torch.randn(3, 50257, device="cuda")
    assert K().argmax(lf).tolist() == lf.argmax(-1).tolist()

    src = torch.randn(1000, device="cuda")
    dst = torch.empty(1000, device="cuda", dtype=torch.bfloat16)
    K().cvt_f32(src, dst, zero_src=True)
    assert float(src.abs().max()) == 0.0


def test_kv_blocks_copy_roundtrip():
    torch.manual_seed(9)
    L, nb, kvh, bs, d = 3, 10, 2, 64, 128
    cache = rand(L, nb, 2, kvh, bs, d)
    ids = torch.tensor([7, 2, 9], device="cuda", dtype=torch.int32)
    staging = torch.empty(3, L, 2, kvh, bs, d, device="cuda", dtype=torch.bfloat16)
    K().kv_blocks_copy(cache, staging, ids, to_staging=True)
    want = cache[:, ids.long()].permute(1, 0, 2, 3, 4, 5)
    torch.testing.assert_close(staging, want.contiguous(), rtol=0, atol=0)
    cache2 = torch.zeros_like(cache)
    K().kv_blocks_copy(cache2, staging, ids, to_staging=False)
    torch.testing.assert_close(cache2[:, ids.long()], cache[:, ids.long()], rtol=0, atol=0)


# ------------------------------------------------------------------------------------------------
# fused projections (restore kernel and forward QKV)
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,H,n_kv,d,rope", [(200, 512, 4, 128, True), (1000, 1024, 8, 128, True), (70, 768, 12, 64, False),
                                             (33, 256, 2, 64, True), (1100, 512, 32, 128, True),   # last two: CTA-pair kernel
                                             (700, 256, 40, 128, False)])
def test_restore_kv_proj(dtype, T, H, n_kv, d, rope):
    torch.manual_seed(10)
    bs = 64 if d == 128 else 128
    n_blocks = (T + bs - 1) // bs + 3
    lat = rand(T, H, dtype=dtype)
    w_kv = rand(2 * n_kv * d, H, dtype=dtype, scale=H ** -0.5)
    bias = None if rope else rand(2 * n_kv * d, dtype=dtype)
    pos = torch.arange(T, device="cuda", dtype=torch.int32) + 17
    slot = make_slots(T, n_blocks, bs, seed=1)
    inv = ref.default_inv_freq(d, device="cuda") if rope else None
    cache = make_cache(n_blocks, n_kv, bs, d, dtype)
    K().restore_kv_proj(lat, w_kv, cache, pos, slot, inv, n_kv, d, bs, bias_kv=bias)
    kv = ref.gemm(lat, w_kv, bias=bias, out_dtype=torch.float32)
    k, v = kv[:, :n_kv * d].view(T, n_kv, d), kv[:, n_kv * d:].view(T, n_kv, d)
    if rope:
        k = ref.rope_rotate_half(k, pos, inv, d)
    want = make_cache(n_blocks, n_kv, bs, d, torch.float32)
    ref.kv_append(want, k, v, slot)
    torch.testing.assert_close(cache.float(), want, **tol(dtype))


@pytest.mark.parametrize("T,n_q,n_kv", [(150, 4, 2), (1100, 32, 8)])   # the second shape takes the CTA-pair kernel
def test_qkv_rope_proj(T, n_q, n_kv):
    torch.manual_seed(11)
    H, d, bs = 512, 128, 64
    n_blocks = (T + bs - 1) // bs + 2
    x = rand(T, H)
    w = rand((n_q + 2 * n_kv) * d, H, scale=H ** -0.5)
    pos = torch.arange(T, device="cuda", dtype=torch.int32)
    slot = make_slots(T, n_blocks, bs, seed=2)
    inv = ref.default_inv_freq(d, device="cuda")
    cache = make_cache(n_blocks, n_kv, bs, d)
    q_out = torch.empty(T, n_q * d, device="cuda", dtype=torch.bfloat16)
    K().qkv_rope_proj(x, w, q_out, cache, pos, slot, inv, n_q, n_kv, d, bs)
    qkv = ref.gemm(x, w, out_dtype=torch.float32)
    q, k, v = qkv.split([n_q * d, n_kv * d, n_kv * d], dim=1)
    want_q = ref.rope_rotate_half(q.view(T, n_q, d), pos, inv, d)
    want_k = ref.rope_rotate_half(k.reshape(T, n_kv, d), pos, inv, d)
    want = make_cache(n_blocks, n_kv, bs, d, torch.float32)
    ref.kv_append(want, want_k, v.reshape(T, n_kv, d), slot)
    torch.testing.assert_close(q_out.view(T, n_q, d).float(), want_q, **tol(torch.bfloat16))
    torch.testing.assert_close(cache.float(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K_,splits,gated", [(1, 128, 4096, 8, False), (16, 200, 1024, 3, True), (17, 264, 640, 5, False), (33, 1000, 2048, 7, True), (64, 4096, 512, 2, False),
                                                 (5, 520, 192, 100, True)])
def test_gemm_cluster_splits(dtype, M, N, K_, splits, gated):
    """K splits of a decode GEMM that meet in a cluster: every token tile, more tokens than splits and fewer, ragged features, split counts
    past what K or a cluster holds; without scratch."""
    torch.manual_seed(M + N)
    a, w, b = rand(M, K_, dtype=dtype), rand(N, K_, dtype=dtype, scale=K_ ** -0.5), rand(N, dtype=dtype)
    out = K().gemm(a, w, bias=b, act=3 if gated else 0, gated=gated, bn=-1, splits=splits)
    want = ref.gemm(a, w, bias=b, act=3 if gated else 0, gated=gated, out_dtype=torch.float32)
    torch.testing.assert_close(out.float(), want, **tol(dtype))


@pytest.mark.parametrize("splits,kept", [(16, 0.0), (8, 16.0), (1, 16.0)])
def test_gemm_accum_explicit_splits(splits, kept):
    """As many K splits of an accumulating product as the caller asks for, past the 8 that a cluster holds: sixteen ones that come one by
    one are lost beside 2^24, in pairs or as one sum they are not."""
    a, w = torch.zeros(1, 1024, dtype=torch.bfloat16, device="cuda"), torch.ones(128, 1024, dtype=torch.bfloat16, device="cuda")
    a[0, ::64] = 1.0
    acc = torch.full((1, 128), 2.0**24, device="cuda")
    K().gemm_accum(a, w, acc, bn=-1, splits=splits)
    assert bool((acc - 2.0**24 == kept).all())


def kernels_of(calls):
    """The kernels that each of ``calls`` (expressions over this module as ``t``) launches, as a child process sees them."""
    import json
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    code = f"""
import json, sys, torch
sys.path[:0] = [{here!r}, {os.path.dirname(here)!r}]
import test_gpu_kernels as t
out = []
for c in json.loads({json.dumps(json.dumps(calls))}):
    eval(c); torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        eval(c); torch.cuda.synchronize()
    out.append(" ".join(e.key for e in p.key_averages()))
print(json.dumps(out))
"""
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    return json.loads(res.stdout.splitlines()[-1])


ACCUM_RULE = [(16, 64, 4096, "gemm_skinny"), (17, 16, 2048, "gemm_tn"), (32, 1016, 4096, "gemm_tn"), (32, 1024, 8192, "gemm_skinny"), (33, 2048, 4096, "gemm_skinny"),
              (33, 2040, 4096, "gemm_tn"), (64, 2048, 4104, "gemm_tn"), (64, 4096, 8192, "gemm_skinny")]


@pytest.mark.parametrize("M,N,K_,_", ACCUM_RULE)
def test_gemm_accum_around_the_rule(M, N, K_, _):
    torch.manual_seed(M + N)
    a, w, base = rand(M, K_), rand(N, K_, scale=K_ ** -0.5), torch.randn(M, N, device="cuda")
    acc = base.clone()
    K().gemm_accum(a, w, acc)
    torch.testing.assert_close(acc, base + ref.gemm(a, w, out_dtype=torch.float32), rtol=1e-4, atol=2e-4)     # fp32 sums of up to 8192 products


def test_gemm_accum_rule():
    """On both sides of each line of the rule: the kernel that runs."""
    ran = kernels_of([f"t.K().gemm_accum(t.rand({M}, {K_}), t.rand({N}, {K_}), torch.zeros({M}, {N}, device='cuda'))" for M, N, K_, _ in ACCUM_RULE])
    for names, case in zip(ran, ACCUM_RULE):
        assert case[3] in names, case


# ------------------------------------------------------------------------------------------------
# paged attention
# ------------------------------------------------------------------------------------------------
def build_paged_problem(seq_specs, n_q_heads, n_kv, d, bs, dtype=torch.bfloat16, seed=0):
    """seq_specs: list of (ctx_before, n_new). Returns q, cache, block_tables, items(list)."""
    g = torch.Generator().manual_seed(seed)
    total_blocks = sum((c + n + bs - 1) // bs for c, n in seq_specs) + 4
    perm = torch.randperm(total_blocks, generator=g).tolist()
    max_blocks = max((c + n + bs - 1) // bs for c, n in seq_specs)
    cache = (torch.randn(total_blocks, 2, n_kv, bs, d, generator=g) * 0.5).to(dtype).cuda()
    tables = torch.zeros(len(seq_specs), max_blocks, dtype=torch.int32)
    items, row = [], 0
    for s, (ctx, n_new) in enumerate(seq_specs):
        nb = (ctx + n_new + bs - 1) // bs
        tables[s, :nb] = torch.tensor([perm.pop() for _ in range(nb)], dtype=torch.int32)
        items.append((s, row, n_new, ctx))
        row += n_new
    q = (torch.randn(row, n_q_heads, d, generator=g)).to(dtype).cuda()
    return q, cache, tables.cuda(), items


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n_q_heads,n_kv,d,bs,n_splits", [(8, 8, 128, 64, 1), (8, 8, 128, 64, 4), (16, 2, 128, 64, 3),
                                                         (12, 12, 64, 128, 2), (4, 4, 128, 32, 5)])
def test_attention_splitkv_decode(dtype, n_q_heads, n_kv, d, bs, n_splits):
    specs = [(0, 1), (5, 1), (127, 1), (128, 1), (1000, 1), (4095, 1), (333, 1)]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    G = n_q_heads // n_kv
    out = torch.zeros_like(q)
    ws_bytes = K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, n_splits, G)
    ws = torch.zeros(max(ws_bytes, 16), dtype=torch.uint8, device="cuda")
    scale = 1.0 / math.sqrt(d)
    for _ in range(2):  # second call checks the scratch counters were left clean
        out.zero_()
        K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), G, n_q_heads, n_kv, d, bs, n_splits,
                                    scale, ws)
        want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale)
        torch.testing.assert_close(out.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n_q_heads,n_kv,d,bs,n_splits,many", [(8, 1, 128, 16, 1, False), (3, 3, 128, 64, 2, False), (12, 4, 128, 64, 16, False),
                                                               (2, 2, 64, 32, 9, False), (10, 2, 64, 128, 1, True), (21, 3, 128, 64, 2, True)])
def test_attention_group_strips(dtype, n_q_heads, n_kv, d, bs, n_splits, many):
    """Ends of the 16-key strips, fewer strips than warps or splits, every row count of a group, CTAs of eight warps and (``many``: more
    than 148 of them) of four. Rows behind a sequence's last key are not numbers. Weights in two 16-bit parts are off by 2^-16 of
    themselves at most, so that the outputs' own rounding to 16 bits is what separates them from 64 bits."""
    specs = [(c, 1) for c in (0, 14, 15, 16, 30, 31, 47, 63, 64, 127, 500)] * (16 if many else 1) + [(40, 8 // (n_q_heads // n_kv))]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=5)
    for (seq, _, n, pos0), t in zip(items, tables.tolist()):
        if (pos0 + n) % bs:
            cache[t[(pos0 + n) // bs], :, :, (pos0 + n) % bs:] = float("nan")
    G, items_t = n_q_heads // n_kv, torch.tensor(items, dtype=torch.int32, device="cuda")
    rows = max(it[2] for it in items) * G
    ws = torch.zeros(max(K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, n_splits, rows), 16), dtype=torch.uint8, device="cuda")
    want, scale = torch.empty_like(q, dtype=torch.float64), 1.0 / math.sqrt(d)
    for (seq, row, n, pos0), t in zip(items, tables.tolist()):
        pages = torch.cat([cache[b] for b in t[:(pos0 + n + bs - 1) // bs]], 2).double().repeat_interleave(G, 1)   # [2, heads, keys, d]
        for i in range(n):
            k, v = pages[0, :, :pos0 + i + 1], pages[1, :, :pos0 + i + 1]
            p = torch.softmax((q[row + i].double()[:, None] * k).sum(-1) * scale, -1)
            want[row + i] = (p[..., None] * v).sum(1)
    flat = torch.zeros(q.numel() + 1, dtype=dtype, device="cuda")
    flat[1:] = q.flatten()
    eps = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    for src in (q, flat[1:].view(q.shape)):     # queries on any boundary
        out = torch.zeros_like(q)
        K().paged_attention_splitkv(src, out, cache, tables, items_t, len(items), rows, n_q_heads, n_kv, d, bs, n_splits, scale, ws, grouped=True)
        torch.testing.assert_close(out.double(), want, rtol=eps, atol=2e-5)


@pytest.mark.parametrize("opts", ["alibi", "window", "keep", "sink", "sigmoid", "softcap"])
@pytest.mark.parametrize("n_q_heads,n_kv,d,bs,n_splits", [(16, 4, 128, 64, 1), (6, 2, 64, 128, 3), (8, 1, 128, 16, 12)])
def test_attention_group_options(opts, n_q_heads, n_kv, d, bs, n_splits):
    """What may ride on an attention launch, in the grouped kernel as in the one for single heads: windows that begin inside a strip, at
    its edge and before the first key, kept first tokens on both sides of a strip's end, and the rest with a gate and strided rows."""
    specs = [(0, 1), (16, 1), (48, 1), (79, 1), (80, 1), (333, 1), (700, 8 // (n_q_heads // n_kv))]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, seed=6)
    T, items_t = q.shape[0], torch.tensor(items, dtype=torch.int32, device="cuda")
    vec, gate = torch.linspace(-2.0, 2.0, n_q_heads, device="cuda"), rand(T, n_q_heads * d)
    kw = {"alibi": dict(alibi=2.0**vec), "window": dict(window=64), "keep": dict(window=33, keep_first=17), "sink": dict(sink=vec, gate=gate, window=200),
          "sigmoid": dict(sigmoid_bias=vec - 4.0, gate=gate), "softcap": dict(softcap=4.0, sink=vec)}[opts]
    ws = torch.zeros(K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, n_splits, 8), dtype=torch.uint8, device="cuda")
    got, want = (torch.zeros(T, n_q_heads * d + 8, dtype=q.dtype, device="cuda")[:, :n_q_heads * d] for _ in range(2))
    for out, grouped in ((got, True), (want, False)):
        K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), 8, n_q_heads, n_kv, d, bs, n_splits, 1 / math.sqrt(d), ws, grouped=grouped, **kw)
    torch.testing.assert_close(got.float(), want.float(), rtol=2.0**-7, atol=1e-3)     # each rounds its own outputs to bf16


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bias", [-9.0, -12.0, -14.0])
@pytest.mark.parametrize("n_q_heads,n_kv,d,n_splits", [(8, 2, 128, 1), (8, 1, 128, 5), (6, 2, 64, 1)])
def test_attention_group_small_weights(dtype, bias, n_q_heads, n_kv, d, n_splits):
    """Sigmoid weights down to 1e-7 keep their precision in the grouped kernel: large values times small weights against 64 bits. Besides
    the output's own rounding, a weight is off by 2^-16 (bf16, two parts of 8 bits) or 2^-21 (fp16), and by what the fp32 score under
    it is off (1e-5)."""
    specs = [(0, 1), (15, 1), (333, 1), (900, 1)]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, 64, dtype, seed=10)
    cache[:, 1] *= 256.0
    items_t, G = torch.tensor(items, dtype=torch.int32, device="cuda"), n_q_heads // n_kv
    vec = torch.linspace(bias - 1.0, bias + 1.0, n_q_heads, device="cuda")
    ws = torch.zeros(max(K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, n_splits, G), 16), dtype=torch.uint8, device="cuda")
    out = torch.zeros_like(q)
    K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), G, n_q_heads, n_kv, d, 64, n_splits, 1 / math.sqrt(d), ws, sigmoid_bias=vec,
                                grouped=True)
    eps, per_weight = (2.0**-8, 2.0**-16) if dtype == torch.bfloat16 else (2.0**-11, 2.0**-21)
    for (seq, row, n, pos0), t in zip(items, tables.tolist()):
        pages = torch.cat([cache[b] for b in t[:(pos0 + n + 63) // 64]], 2).double().repeat_interleave(G, 1)
        k, v = pages[0, :, :pos0 + 1], pages[1, :, :pos0 + 1]
        p = torch.sigmoid((q[row].double()[:, None] * k).sum(-1) / math.sqrt(d) + vec.double()[:, None])[..., None]
        want, size = (p * v).sum(1), (p * v.abs()).sum(1)
        assert ((out[row].double() - want).abs() <= eps * want.abs() + (per_weight + 1e-5) * size + 2.0**-25).all()


@pytest.mark.parametrize("n_q_heads,n_kv,d", [(8, 2, 128), (6, 2, 128), (4, 2, 64)])
def test_attention_of_a_batch_for_smaller_groups(n_q_heads, n_kv, d):
    """Items of up to 8 tokens, as a batch built for heads of their own has them, under grouped attention: every row is computed."""
    import types
    from hcache_deepspeed_b200.ops.backend import CudaOps
    q, cache, tables, items = build_paged_problem([(40, 8), (300, 3), (17, 1)], n_q_heads, n_kv, d, 64, seed=9)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    batch = types.SimpleNamespace(block_size=64, group=1, n_items_small=3, n_items_large=0, rows_per_small_item=8, max_kv_len_small=303,
                                  block_tables=lambda: tables, items_small=lambda: items_t)
    out = torch.full_like(q, float("nan"))
    CudaOps().attention(q.view(q.shape[0], -1), out.view(q.shape[0], -1), cache, batch, n_q_heads, n_kv, d, 1 / math.sqrt(d))
    want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, 1 / math.sqrt(d))
    torch.testing.assert_close(out.float(), want.float(), **tol(torch.bfloat16))


def test_attention_splitkv_multirow():
    # short continuations: several query tokens per item (MHA: rows = tokens)
    n_q_heads = n_kv = 4
    d, bs = 128, 64
    specs = [(300, 8), (0, 5), (64, 8), (2000, 3)]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    out = torch.zeros_like(q)
    ws = torch.zeros(K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, 2, 8), dtype=torch.uint8, device="cuda")
    scale = 1.0 / math.sqrt(d)
    K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), 8, n_q_heads, n_kv, d, bs, 2, scale, ws)
    want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale)
    torch.testing.assert_close(out.float(), want.float(), **tol(torch.bfloat16))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n_q_heads,n_kv,d,bs", [(4, 4, 128, 64), (8, 2, 128, 64), (6, 6, 64, 128), (4, 4, 128, 16)])
def test_attention_prefill(dtype, n_q_heads, n_kv, d, bs):
    specs = [(0, 128), (0, 17), (100, 64), (1000, 128), (4000, 96), (63, 1), (128, 128)]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=3)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    out = torch.zeros_like(q)
    scale = 1.0 / math.sqrt(d)
    K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale)
    want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale)
    torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
    # split-KV variant (partials merged through scratch); twice to check the tickets were reset
    for n_splits in (3, 8):
        ws = torch.zeros(K().prefill_workspace_bytes(len(items), n_q_heads, d, n_splits), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            out.zero_()
            K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale,
                                        n_splits=n_splits, workspace=ws)
            torch.testing.assert_close(out.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n_q_heads,n_kv,bs", [(8, 1, 64), (32, 4, 64), (16, 4, 32), (64, 8, 64), (8, 2, 128)])
def test_attention_packed_gqa_decode(dtype, n_q_heads, n_kv, bs):
    """Head-packed grouped-query decode on the tensor cores (one CTA per (item, KV head), MMA rows = (token, head of the
    group)): decode items of 1 token — and as many tokens as 128 / G allows — against the fp32 paged-attention oracle,
    unsplit and split-KV (tickets must come back zeroed: every launch runs twice)."""
    d = 128
    G = n_q_heads // n_kv
    specs = [(0, 1), (100, 1), (1000, 1), (4000, 1), (63, 1), (127, 1), (128, 1), (5, min(3, 128 // G)), (700, min(128 // G, 6))]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=5)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    scale = 1.0 / math.sqrt(d)
    want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale)
    out = torch.zeros_like(q)
    K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale, packed=True)
    torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
    for n_splits in (2, 5):
        ws = torch.zeros(K().prefill_workspace_bytes(len(items), n_kv, d, n_splits), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            out.zero_()
            K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale,
                                        n_splits=n_splits, workspace=ws, packed=True)
            torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
        assert int(ws[:len(items) * n_kv * 32].view(torch.int32).abs().max()) == 0


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_alibi_all_kernels(dtype):
    """ALiBi (``hds_attention_next_alibi``): score += slope[head] * (key - query position) in the split-KV decode kernel
    (1 and several rows per item, split and unsplit), the tensor-core prefill kernel (unsplit / split-KV) and the
    head-packed GQA kernel, against the fp32 oracle; the setting is consumed by ONE launch (the next one is plain)."""
    scale_of = lambda d: 1.0 / math.sqrt(d)
    # split-KV decode, MHA (Bloom-like: 6 heads = interleaved slope sequence) and GQA rows
    for n_q_heads, n_kv, d, bs, rows in ((6, 6, 64, 128, 1), (8, 8, 128, 64, 1), (16, 4, 128, 64, 1), (4, 4, 128, 64, 8)):
        specs = [(0, rows), (5, rows), (127, 1), (1000, rows), (4095, 1), (333, 1)]
        q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=11)
        items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
        slopes = ref.alibi_slopes(n_q_heads).cuda()
        G = n_q_heads // n_kv
        R = rows * G
        want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale_of(d), alibi=slopes)
        plain = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale_of(d))
        assert (want.float() - plain.float()).abs().max() > 0.05          # the bias matters in this problem
        for n_splits in (1, 3):
            ws = torch.zeros(max(K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, n_splits, R), 16), dtype=torch.uint8,
                             device="cuda")
            out = torch.zeros_like(q)
            K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), R, n_q_heads, n_kv, d, bs, n_splits,
                                        scale_of(d), ws, alibi=slopes)
            torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
            out.zero_()
            K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), R, n_q_heads, n_kv, d, bs, n_splits,
                                        scale_of(d), ws)
            torch.testing.assert_close(out.float(), plain.float(), **tol(dtype))
    # tensor-core prefill
    # (32 heads: the steepest slope moves the row maximum by > 126 log2 units from one key tile to the next, so the rescale
    # factor of the accumulator underflows to exactly 0 — stale contributions must still be wiped)
    for n_q_heads, n_kv, d, bs in ((4, 4, 128, 64), (6, 6, 64, 128), (8, 2, 128, 16), (32, 8, 128, 64)):
        specs = [(0, 128), (0, 17), (100, 64), (1000, 128), (4000, 96), (63, 1)]
        q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=12)
        items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
        slopes = ref.alibi_slopes(n_q_heads).cuda()
        want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale_of(d), alibi=slopes)
        out = torch.zeros_like(q)
        K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale_of(d), alibi=slopes)
        torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
        ws = torch.zeros(K().prefill_workspace_bytes(len(items), n_q_heads, d, 3), dtype=torch.uint8, device="cuda")
        out.zero_()
        K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale_of(d), n_splits=3,
                                    workspace=ws, alibi=slopes)
        torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
    # head-packed grouped-query decode: every row of the tile has its own head's slope
    n_q_heads, n_kv, d, bs = 32, 4, 128, 64
    specs = [(0, 1), (100, 1), (1000, 1), (4000, 1), (5, 3), (700, 6)]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=13)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    slopes = ref.alibi_slopes(n_q_heads).cuda()
    want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, scale_of(d), alibi=slopes)
    out = torch.zeros_like(q)
    K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, scale_of(d), packed=True,
                                alibi=slopes)
    torch.testing.assert_close(out.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [1, 100, 128, 1000])
def test_attention_sliding_window_all_kernels(dtype, window):
    """Sliding-window attention (``hds_attention_next_window``): keys (p - window, p] only, key tiles before the window
    skipped, in the split-KV decode kernel (split and unsplit, one and several rows), the tensor-core prefill kernel and the
    head-packed GQA kernel; combined with ALiBi once; consumed by ONE launch."""
    sc = lambda d: 1.0 / math.sqrt(d)
    for n_q_heads, n_kv, d, bs, rows in ((8, 8, 128, 64, 1), (12, 12, 64, 128, 1), (16, 4, 128, 64, 1), (4, 4, 128, 64, 8)):
        specs = [(0, rows), (5, rows), (127, 1), (1000, rows), (4095, 1), (333, 1)]
        q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=21)
        items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
        R = rows * (n_q_heads // n_kv)
        want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, sc(d), window=window)
        plain = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, sc(d))
        for n_splits in (1, 3):
            ws = torch.zeros(max(K().splitkv_workspace_bytes(len(items), n_q_heads, n_kv, d, n_splits, R), 16), dtype=torch.uint8,
                             device="cuda")
            out = torch.zeros_like(q)
            for _ in range(2):
                out.zero_()
                K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), R, n_q_heads, n_kv, d, bs, n_splits, sc(d),
                                            ws, window=window)
                torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
            out.zero_()
            K().paged_attention_splitkv(q, out, cache, tables, items_t, len(items), R, n_q_heads, n_kv, d, bs, n_splits, sc(d), ws)
            torch.testing.assert_close(out.float(), plain.float(), **tol(dtype))
    for n_q_heads, n_kv, d, bs in ((4, 4, 128, 64), (6, 6, 64, 128), (8, 2, 128, 16)):
        specs = [(0, 128), (0, 17), (100, 64), (1000, 128), (4000, 96), (63, 1), (300, 128)]
        q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=22)
        items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
        want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, sc(d), window=window)
        out = torch.zeros_like(q)
        K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, sc(d), window=window)
        torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
        ws = torch.zeros(K().prefill_workspace_bytes(len(items), n_q_heads, d, 3), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            out.zero_()
            K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, sc(d), n_splits=3,
                                        workspace=ws, window=window)
            torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
        slopes = ref.alibi_slopes(n_q_heads).cuda()
        want_a = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, sc(d), window=window, alibi=slopes)
        out.zero_()
        K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, sc(d), window=window,
                                    alibi=slopes)
        torch.testing.assert_close(out.float(), want_a.float(), **tol(dtype))
    n_q_heads, n_kv, d, bs = 32, 4, 128, 64
    specs = [(0, 1), (100, 1), (1000, 1), (4000, 1), (5, 3), (700, 6)]
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=23)
    items_t = torch.tensor(items, dtype=torch.int32, device="cuda")
    want = ref.paged_attention(q, cache, tables, items_t.cpu(), n_q_heads, n_kv, sc(d), window=window)
    out = torch.zeros_like(q)
    K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, sc(d), packed=True, window=window)
    torch.testing.assert_close(out.float(), want.float(), **tol(dtype))
    ws = torch.zeros(K().prefill_workspace_bytes(len(items), n_kv, d, 4), dtype=torch.uint8, device="cuda")
    out.zero_()
    K().paged_attention_prefill(q, out, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, sc(d), packed=True, n_splits=4,
                                workspace=ws, window=window)
    torch.testing.assert_close(out.float(), want.float(), **tol(dtype))


def test_attention_prefill_64_key_tiles_subprocess():
    """The opt-in 64-key-tile / two-CTAs-per-SM shape of the tensor-core attention kernel (HDS_PREFILL_TILE=64, read once per
    process): the prefill attention tests of this file are re-run in a child process with the variable set."""
    import os
    import subprocess
    import sys
    env = dict(os.environ, HDS_PREFILL_TILE="64")
    res = subprocess.run([sys.executable, "-m", "pytest", __file__, "-q", "-m", "gpu", "-k", "test_attention_prefill and not subprocess",
                          "--timeout", "120", "-p", "no:cacheprovider"], env=env, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-1000:]
    assert " passed" in res.stdout


_SWITCH_PROBES = {
    "attention": """
q, cache, tables, items = t.build_paged_problem([(0, 128)] * 20, 16, 4, 128, 64)
it = torch.tensor(items, dtype=torch.int32, device="cuda")
call = lambda: t.K().paged_attention_prefill(q, torch.empty_like(q), cache, tables, it, len(items), 16, 4, 128, 64, 0.09)
""",
    "experts": """
x, w, pad = torch.zeros(256, 128, dtype=torch.bfloat16, device="cuda"), t.rand(256, 128), torch.tensor([0, 128, 256], dtype=torch.int32, device="cuda")
call = lambda: t.K().moe_gemm(x, w, pad, 2, torch.empty(256, 128, dtype=torch.bfloat16, device="cuda"), choices=8)
""",
}


@pytest.mark.parametrize("probe,var,value,kernel", [("attention", "HDS_PREFILL_TILE", "64", "paged_attn_prefill64_kernel"),
                                                    ("attention", "HDS_PREFILL_TILE", "128", "paged_attn_pair_kernel"),
                                                    ("experts", "HDS_GEMM_SKINNY", "0", "gemm_tn_kernel"), ("experts", "HDS_GEMM_SKINNY", "1", "gemm_skinny_kernel")])
def test_switches_read_once_per_process(probe, var, value, kernel):
    """Environment switches that choose a kernel: the kernel that a child process with the variable set really runs."""
    import os
    import subprocess
    import sys
    code = f"""
import sys, torch
sys.path.insert(0, {os.path.dirname(os.path.abspath(__file__))!r}); sys.path.insert(0, {os.path.dirname(os.path.dirname(os.path.abspath(__file__)))!r})
import test_gpu_kernels as t
{_SWITCH_PROBES[probe]}
call(); torch.cuda.synchronize()
with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
    call(); torch.cuda.synchronize()
print([e.key for e in p.key_averages()])
"""
    res = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **{var: value}), capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    assert kernel in res.stdout


STORE_RULE = [(16, 57344, 512, "gemm_skinny"), (17, 14336, 2048, "gemm_tn"), (17, 14336, 2056, "gemm_skinny"), (33, 14336, 8192, "gemm_tn"), (33, 13312, 2048, "gemm_tn"),
              (64, 12288, 2048, "gemm_tn"), (64, 11264, 2048, "gemm_skinny"), (33, 12288, 2056, "gemm_skinny"), (64, 18944, 2048, "gemm_tn"), (64, 18952, 2048, "gemm_skinny"),
              (33, 37888, 2048, "gemm_skinny"), (33, 37896, 2048, "gemm_tn"), (32, 37896, 2048, "gemm_skinny"), (64, 37896, 4096, "gemm_skinny")]


def test_gemm_store_rule():
    """Plain stores of decode sizes on both sides of each line of the rule: the kernel that runs."""
    ran = kernels_of([f"t.K().gemm(t.rand({M}, {K_}), t.rand({N}, {K_}), out=t.rand({M}, {N}))" for M, N, K_, _ in STORE_RULE])
    for names, case in zip(ran, STORE_RULE):
        assert case[3] in names, case


@pytest.mark.parametrize("M,N,K_,gated", [(33, 37896, 256, False), (64, 37896, 256, True), (17, 43008, 8192, False), (64, 13320, 512, False), (40, 57344, 4096, True)])
def test_gemm_past_a_wave(M, N, K_, gated):
    """More feature tiles than run at once, split and unsplit, and widths around the rule: against the product in fp32."""
    torch.manual_seed(M + N)
    a, w, b = rand(M, K_), rand(N, K_, scale=K_ ** -0.5), rand(N)
    out = K().gemm(a, w, bias=b, act=3 if gated else 0, gated=gated)
    want = ref.gemm(a, w, bias=b, act=3 if gated else 0, gated=gated, out_dtype=torch.float32)
    torch.testing.assert_close(out.float(), want, **tol(torch.bfloat16))


def prefill_of(items, **kw):
    q, cache, tables, its = build_paged_problem([(64, 64)] * items, 16, 4, 128, 64)
    if "sigmoid" in kw:
        kw = dict(sigmoid_bias=torch.full((16, ), -3.0, device="cuda"))
    K().paged_attention_prefill(q, torch.empty_like(q), cache, tables, torch.tensor(its, dtype=torch.int32, device="cuda"), items, 16, 4, 128, 64, 0.09, **kw)


def experts_of(choices, K_, gated):
    x, w, pad = torch.zeros(256, K_, dtype=torch.bfloat16, device="cuda"), rand(256, K_), torch.tensor([0, 128, 256], dtype=torch.int32, device="cuda")
    K().moe_gemm(x, w, pad, 2, torch.empty(256, 64 if gated else 128, dtype=torch.bfloat16, device="cuda"), gated=gated, choices=choices)


def test_experts_rule():
    """Expert products of a decode step: the kernel by choices, inner size and form."""
    cases = [("0, 128, False", "gemm_tn"), ("64, 128, False", "gemm_skinny"), ("65, 128, False", "gemm_tn"), ("32, 128, True", "gemm_skinny"), ("33, 4088, True", "gemm_tn"),
             ("64, 4096, True", "gemm_skinny")]
    for names, (args, kernel) in zip(kernels_of([f"t.experts_of({a})" for a, _ in cases]), cases):
        assert kernel in names, args


def test_attention_pair_rule():
    """Pairs of heads from one per SM on, weights with quotients from three for two SMs on: the kernel that runs, at 8 pairs an item."""
    cases = [("18", "prefill"), ("19", "pair"), ("27, softcap=4.0", "prefill"), ("28, softcap=4.0", "pair"), ("27, sigmoid=1", "prefill"), ("28, sigmoid=1", "pair")]
    for names, (args, kernel) in zip(kernels_of([f"t.prefill_of({a})" for a, _ in cases]), cases):
        assert f"paged_attn_{kernel}_kernel" in names, args


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("opts", ["plain", "window", "keep", "sink", "sigmoid", "softcap"])
@pytest.mark.parametrize("n_q_heads,n_kv,bs", [(16, 4, 64), (12, 2, 16), (32, 1, 128)])
def test_attention_pair(dtype, opts, n_q_heads, n_kv, bs):
    """Two heads of a group per CTA (from 148 such pairs on): one key tile and many (more than the ring's slots), ragged last tiles, items of
    one token and of 128, quadrants without rows, windows and kept tokens; against the kernel with one head per CTA, which takes the
    same items a few at a time."""
    d = 128
    specs = [(0, 1), (0, 128), (0, 127), (1, 128), (100, 33), (127, 1), (128, 128), (255, 65), (300, 128), (640, 96), (1000, 128), (1407, 17)] * 3
    q, cache, tables, items = build_paged_problem(specs, n_q_heads, n_kv, d, bs, dtype, seed=8)
    T, items_t = q.shape[0], torch.tensor(items, dtype=torch.int32, device="cuda")
    vec, gate = torch.linspace(-2.0, 2.0, n_q_heads, device="cuda"), rand(T, n_q_heads * d, dtype=dtype)
    kw = {"plain": {}, "window": dict(window=200), "keep": dict(window=129, keep_first=130), "sink": dict(sink=vec, gate=gate, window=300),
          "sigmoid": dict(sigmoid_bias=vec - 4.0), "softcap": dict(softcap=4.0, sink=vec)}[opts]
    got, want = (torch.zeros(T, n_q_heads * d + 8, dtype=dtype, device="cuda")[:, :n_q_heads * d] for _ in range(2))
    assert len(items) * n_q_heads // 2 >= 148
    few = max(1, 147 // (n_q_heads // 2))
    K().paged_attention_prefill(q, got, cache, tables, items_t, len(items), n_q_heads, n_kv, d, bs, 1 / math.sqrt(d), **kw)
    for i in range(0, len(items), few):
        part = items_t[i:i + few].contiguous()
        K().paged_attention_prefill(q, want, cache, tables, part, part.shape[0], n_q_heads, n_kv, d, bs, 1 / math.sqrt(d), **kw)
    # both round weights to 16 bits, against maxima that may differ by 2^8, and their outputs: the errors of two roundings
    eps = 2.0**-7 if dtype == torch.bfloat16 else 2.0**-10
    torch.testing.assert_close(got.float(), want.float(), rtol=2 * eps, atol=eps)


# ------------------------------------------------------------------------------------------------
# mixture of experts
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("T,E,k,norm", [(1, 8, 2, True), (37, 8, 2, False), (300, 60, 4, True), (5, 3, 1, False)])
def test_moe_pipeline(T, E, k, norm):
    """top-k gating -> scatter -> grouped gated GEMM -> grouped GEMM -> weighted gather vs a per-token fp32 loop."""
    torch.manual_seed(T + E)
    H, I = 256, 384
    kern = K()
    x = rand(T, H)
    w_router = rand(E, H, scale=H ** -0.5)
    w_up = rand(E * 2 * I, H, scale=H ** -0.5)     # stacked, gate/up interleaved per expert
    w_down = rand(E * H, I, scale=I ** -0.5)
    logits = kern.gemm(x, w_router)
    scores = torch.empty(T, k, dtype=torch.float32, device="cuda")
    ids = torch.empty(T, k, dtype=torch.int32, device="cuda")
    offs = torch.empty(T, k, dtype=torch.int32, device="cuda")
    slots = torch.empty(T, k, dtype=torch.int32, device="cuda")
    counts = torch.zeros(E, dtype=torch.int32, device="cuda")
    pad_off = torch.zeros(E + 1, dtype=torch.int32, device="cuda")
    rows = kern.moe_padded_rows(T, E, k)
    xs = torch.zeros(rows, H, dtype=x.dtype, device="cuda")
    hs = torch.zeros(rows, I, dtype=x.dtype, device="cuda")
    ys = torch.zeros(rows, H, dtype=x.dtype, device="cuda")
    out = torch.zeros(T, H, dtype=torch.float32, device="cuda")
    for rep in range(2):  # the counters must come back zeroed
        kern.moe_topk_gating(logits, k, norm, scores, ids, offs, counts)
        kern.moe_scatter(x, xs, ids, offs, counts, pad_off, slots, k)
        kern.moe_gemm(xs, w_up, pad_off, E, hs, act=3, gated=True)
        kern.moe_gemm(hs, w_down, pad_off, E, ys)
        out.zero_()
        kern.moe_gather(ys, slots, scores, out)
    torch.cuda.synchronize()
    assert int(counts.abs().max()) == 0 and int(pad_off[-1]) % 128 == 0
    # oracle
    probs = torch.softmax(logits.float(), -1)
    topv, topi = torch.topk(probs, k, dim=-1)
    assert torch.equal(topi.int().sort(-1).values, ids.sort(-1).values)
    if norm:
        topv = topv / topv.sum(-1, keepdim=True)
    torch.testing.assert_close(scores.sort(-1).values, topv.sort(-1).values, rtol=1e-4, atol=1e-5)
    want = torch.zeros(T, H, device="cuda")
    for t in range(T):
        for j in range(k):
            e = int(ids[t, j])
            h = ref.gemm(x[t:t + 1], w_up[e * 2 * I:(e + 1) * 2 * I], act=3, gated=True, out_dtype=torch.float32).to(x.dtype)
            y = ref.gemm(h, w_down[e * H:(e + 1) * H], out_dtype=torch.float32).to(x.dtype)
            want[t] += float(scores[t, j]) * y[0].float()
    torch.testing.assert_close(out, want, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,E,k,N,K_,gated", [(1, 3, 1, 128, 64, False), (8, 16, 2, 2688, 2048, False), (16, 5, 1, 200, 328, True), (11, 40, 3, 264, 136, True),
                                              (16, 70, 4, 136, 512, False)])
def test_moe_gemm_few(dtype, T, E, k, N, K_, gated):
    """Experts of a decode step, streamed feature-major: 1..64 choices (token tiles of 16, 32 and 64 rows), experts without rows, more than 32
    experts, ragged feature tiles and K, against the token-major kernel's own oracle row by row."""
    torch.manual_seed(T + N)
    kern = K()
    x, w = rand(T, K_, dtype=dtype), rand(E * N, K_, dtype=dtype, scale=K_ ** -0.5)
    ids = torch.stack([torch.randperm(E, device="cuda")[:k] for _ in range(T)]).int()
    counts = torch.bincount(ids.flatten().long(), minlength=E)
    offs = torch.empty_like(ids)
    seen = [0] * E
    for t in range(T):
        for j in range(k):
            offs[t, j] = seen[int(ids[t, j])]
            seen[int(ids[t, j])] += 1
    rows = kern.moe_padded_rows(T, E, k)
    xs = torch.zeros(rows, K_, dtype=dtype, device="cuda")
    pad_off, slots = torch.zeros(E + 1, dtype=torch.int32, device="cuda"), torch.empty_like(ids)
    kern.moe_scatter(x, xs, ids, offs, counts.int(), pad_off, slots, k)
    out = torch.full((rows, N // 2 if gated else N), 7.0, dtype=dtype, device="cuda")
    kern.moe_gemm(xs, w, pad_off, E, out, act=3 if gated else 0, gated=gated, choices=T * k)
    for e in range(E):
        lo = int(pad_off[e])
        if counts[e] == 0:
            continue
        want = ref.gemm(xs[lo:lo + int(counts[e])], w[e * N:(e + 1) * N], act=3 if gated else 0, gated=gated, out_dtype=torch.float32)
        torch.testing.assert_close(out[lo:lo + int(counts[e])].float(), want, **tol(dtype))
    assert bool((out[int(pad_off[E]):] == 7.0).all())      # nothing past the last expert's range


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,cols,layer", [(1, 8, False), (3, 2056, True), (16, 4096, False), (5, 16384, False)])
def test_norm_fp8(dtype, rows, cols, layer):
    """The norm's own 8-bit codes are those of the quantiser, bit for bit, and its 16-bit output is what it is without them; rows of zeros
    and past the quantiser's registers among them."""
    torch.manual_seed(rows + cols)
    x, g, d32 = rand(rows, cols, dtype=dtype), rand(cols, dtype=dtype), torch.randn(rows, cols, device="cuda")
    x[0], d32[0] = 0.0, 0.0
    kw = dict(beta=rand(cols, dtype=dtype), layer_norm=True) if layer else {}
    outs = []
    for fp8 in (None, (torch.zeros(rows, cols, dtype=torch.uint8, device="cuda"), torch.zeros(rows, device="cuda"))):
        res, out, delta = torch.empty_like(x), torch.empty_like(x), d32.clone()
        K().norm(x, g, out, delta=delta, zero_delta=True, res_out=res, fp8=fp8, **kw)
        outs.append((out, res))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    q, s = K().quantize_fp8_rows(outs[0][0])
    assert torch.equal(q, fp8[0]) and torch.equal(s, fp8[1])
    wide = rand(2, 20000, dtype=dtype)      # longer than a row that stays in registers
    q, s = K().quantize_fp8_rows(wide)
    want = (wide.double().abs().amax(1) / 448.0).float()       # (quotients as fp32 rounds them)
    inv = (1.0 / want.double()).float()
    assert torch.equal(s, want) and torch.equal(q, (wide.float() * inv[:, None]).to(torch.float8_e4m3fn).view(torch.uint8))


@pytest.mark.parametrize("K_", [768, 2048, 4096, 8184, 8192, 16384])
def test_quantize_fp8_many_rows(K_):
    """More rows than SMs take other numbers of threads: a row's codes and scale are the same, bit for bit, as in a launch of a few."""
    x = rand(300, K_) * torch.linspace(0.0, 3.0, 300, device="cuda")[:, None].bfloat16()
    q, s = K().quantize_fp8_rows(x)
    for r in range(0, 300, 100):
        q1, s1 = K().quantize_fp8_rows(x[r:r + 100])
        assert torch.equal(q[r:r + 100], q1) and torch.equal(s[r:r + 100], s1)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (5, 2, 2056), (33, 4, 4096)])
def test_moe_gather_shared(dtype, T, k, H):
    torch.manual_seed(T + H)
    x, y, ys, wg = rand(T, H, dtype=dtype), rand(128, H, dtype=dtype), rand(T, H, dtype=dtype), rand(1, H, dtype=dtype, scale=2 * H ** -0.5)
    slots, scores = torch.randint(0, 128, (T, k), device="cuda", dtype=torch.int32), torch.rand(T, k, device="cuda")
    out = torch.randn(T, H, device="cuda")
    want = out.double() + (y.double()[slots.long()] * scores.double()[..., None]).sum(1) + torch.sigmoid(x.double() @ wg.double().T) * ys.double()
    K().moe_gather_shared(y, slots, scores, x, wg, ys, out)
    torch.testing.assert_close(out.double(), want, rtol=1e-5, atol=2e-5)      # fp32 sums of up to 4096 products in the gate


@pytest.mark.parametrize("dtype", DTYPES)
def test_moe_gather_shared_boundaries(dtype):
    """The gate's weights on any boundary, as a slice of a flat buffer: the same bits; rows that are not on 16 bytes are refused."""
    T, k, H = 5, 2, 264
    x, y, ys, flat = rand(T, H, dtype=dtype), rand(64, H, dtype=dtype), rand(T, H, dtype=dtype), rand(H + 8, dtype=dtype)
    slots, scores = torch.randint(0, 64, (T, k), device="cuda", dtype=torch.int32), torch.rand(T, k, device="cuda")
    for off in (1, 3, 4):
        outs = []
        for gate in (flat[off:off + H], flat[off:off + H].clone()):
            outs.append(torch.zeros(T, H, device="cuda"))
            K().moe_gather_shared(y, slots, scores, x, gate.view(1, H), ys, outs[-1])
        assert torch.equal(*outs)
    with pytest.raises(RuntimeError, match="16-byte"):
        K().moe_gather_shared(y, slots, scores, rand(T * H + 1, dtype=dtype)[1:].view(T, H), flat[:H].view(1, H), ys, outs[0])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K_", [(130, 512, 64), (256, 256, 128), (300, 1000, 2096), (1024, 4096, 1024), (4100, 1376, 512)])
@pytest.mark.parametrize("bn", [0, 128, 256])
@pytest.mark.parametrize("mode", ["store", "gated"])
def test_gemm_2sm(dtype, M, N, K_, bn, mode):
    """CTA-pair kernel (tcgen05 cta_group::2, 256 x bn tiles): ragged M / N / K, both tile widths, both epilogues."""
    torch.manual_seed(M)
    a, w, b = rand(M, K_, dtype=dtype), rand(N, K_, dtype=dtype, scale=K_ ** -0.5), rand(N, dtype=dtype)
    gated = mode == "gated"
    out = K().gemm_2sm(a, w, bias=b, act=3 if gated else 2, gated=gated, bn=bn)
    want = ref.gemm(a, w, bias=b, act=3 if gated else 2, gated=gated, out_dtype=torch.float32)
    torch.testing.assert_close(out.float(), want, **tol(dtype))


def test_v2_kernel_wrapper_objects_cuda_vs_host():
    """inference.v2.kernels wrapper classes: the CUDA path (native kernels) against their own host formulation."""
    from hcache_deepspeed_b200.inference.v2.kernels import (BlasLibLinear, CUDAFPPreLN, CUDARMSNorm, MoEGather, MoEGEMM,
                                                            MoEScatter, RaggedLogitsGather, RaggedTopKGating)
    torch.manual_seed(5)
    T, H, I, E, k = 70, 256, 384, 8, 2
    x = rand(T, H)
    gate_w = rand(E, H, scale=H ** -0.5)
    w1, w2 = rand(E, 2 * I, H, scale=H ** -0.5), rand(E, H, I, scale=I ** -0.5)

    lg = torch.empty(T, E, dtype=x.dtype, device="cuda")
    BlasLibLinear(x.dtype)(lg, x, gate_w)
    torch.testing.assert_close(lg.float(), x.float() @ gate_w.float().t(), rtol=2e-2, atol=2e-2)
    # one set of fp32 logits for both devices, ties broken, so both route identically
    shared_logits = lg.float() + torch.arange(E, device="cuda") * 1e-4

    def run(dev):
        xd, a, b = x.to(dev), w1.to(dev), w2.to(dev)
        logits = shared_logits.to(dev)
        counts = torch.zeros(E, dtype=torch.int32, device=dev)
        scores = torch.empty(T, k, dtype=torch.float32, device=dev)
        ids, offs, slots = (torch.empty(T, k, dtype=torch.int32, device=dev) for _ in range(3))
        RaggedTopKGating(xd.dtype)(counts, scores, ids, offs, logits)
        rows = int(((counts + 127) // 128 * 128).sum())
        xs = torch.zeros(rows, H, dtype=xd.dtype, device=dev)
        cum = torch.zeros(E + 1, dtype=torch.int32, device=dev)
        MoEScatter(xd.dtype)(xs, cum, slots, xd, counts, ids, offs)
        hs = torch.zeros(rows, I, dtype=xd.dtype, device=dev)
        ys = torch.zeros(rows, H, dtype=xd.dtype, device=dev)
        MoEGEMM(xd.dtype, "silu", gated=True)(hs, xs, a, cum)
        MoEGEMM(xd.dtype)(ys, hs, b, cum)
        out = torch.zeros(T, H, dtype=torch.float32, device=dev)
        MoEGather(xd.dtype)(out, ys, scores, slots)
        gamma, beta = torch.ones(H, dtype=xd.dtype, device=dev), torch.zeros(H, dtype=xd.dtype, device=dev)
        n1 = torch.empty_like(xd)
        CUDARMSNorm(H, xd.dtype, 1e-6)(n1, xd, gamma)
        zr, zh = torch.empty_like(xd), torch.empty_like(xd)
        CUDAFPPreLN(H, xd.dtype, 1e-5)(zr, zh, xd, n1, gamma, beta)
        last = torch.empty(3, H, dtype=xd.dtype, device=dev)
        RaggedLogitsGather(H, xd.dtype)(last, zh, torch.tensor([0, 9, T - 1], dtype=torch.int32, device=dev))
        return out.cpu(), n1.float().cpu(), zh.float().cpu(), last.float().cpu()

    got, want = run("cuda"), run("cpu")
    torch.testing.assert_close(got[0], want[0], rtol=4e-2, atol=4e-2)
    for g_, w_ in zip(got[1:], want[1:]):
        torch.testing.assert_close(g_, w_, rtol=2e-2, atol=2e-2)
