"""Per-op parity of the CUDA kernels (called through the C ABI) against the oracle's plain-torch
restatement evaluated on the same GPU in bf16 (same rounding points as the HF eager graph)."""
import math

import pytest
import torch

from livecc_b200 import _cabi as A
from oracle import restated as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rand(shape, seed, scale=1.0, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(shape, device=DEV, generator=g) * scale).to(dtype)


def _attn_ref_fp32(q, k, v, mask, scale):
    """softmax(q k^T * scale + mask) v with fp32 scores/probabilities (what a flash kernel computes;
    the HF eager path rounds the scores to bf16 first, which is *less* accurate, mq2vl.py:366-371)."""
    w = torch.matmul(q.float(), k.float().transpose(1, 2)) * scale
    if mask is not None:
        w = w + mask.float()
    w = torch.softmax(w, dim=-1)
    return torch.matmul(w, v.float())


def _attn_close(out, ref, what=""):
    out, ref = out.float(), ref.float()
    err = (out - ref).abs()
    tol = 6e-3 + 1.5e-2 * ref.abs()  # P is rounded to bf16 before P.V (2^-9 relative) + bf16 output rounding
    bad = (err > tol).float().mean().item()
    assert bad < 1e-4, f"{what}: {bad:.2e} of elements outside tolerance, max abs err {err.max().item():.3e}"


def _mismatch(out, ref, ulps=1.0, floor=1e-3):
    """fraction of elements further than `ulps` bf16 ulps (relative 2^-8) from ref."""
    out, ref = out.float(), ref.float()
    tol = ulps * 2.0 ** -8 * ref.abs().clamp_min(floor)
    return ((out - ref).abs() > tol).float().mean().item()


@pytest.mark.parametrize("rows,dim", [(1024, 1280), (77, 320), (3, 3584)])
def test_layernorm(ctx, rows, dim):
    x = _rand((rows, dim), 1, 2.0)
    w = (1 + 0.1 * torch.randn(dim, device=DEV)).to(torch.bfloat16)
    b = (0.02 * torch.randn(dim, device=DEV)).to(torch.bfloat16)
    y = ctx.layernorm(x, w, b, 1e-6)
    ref = R.layer_norm(x, w, b, 1e-6)
    assert _mismatch(y, ref, 1.0) < 2e-3 and _mismatch(y, ref, 2.0) == 0


@pytest.mark.parametrize("rows,dim", [(281, 3584), (1, 3584), (50, 1792)])
def test_rmsnorm(ctx, rows, dim):
    x = _rand((rows, dim), 2, 3.0)
    w = (1 + 0.1 * torch.randn(dim, device=DEV)).to(torch.bfloat16)
    y = ctx.rmsnorm(x, w, 1e-6)
    ref = R.rms_norm(x, w, 1e-6)
    assert _mismatch(y, ref, 1.0) < 2e-3 and _mismatch(y, ref, 2.0) == 0


@pytest.mark.parametrize("rows,dim", [(1, 8), (2400, 8), (5, 512), (2368, 520), (2367, 1536), (2369, 1536), (9, 1544), (700, 4096), (500, 4104), (3, 16392)])
def test_norms_at_the_edges_of_their_forms(ctx, rows, dim):
    """teams of 64, 192 and 256 threads, a warp per row, columns beyond the registers; strided rows; a row's result does not depend on
    how many rows there are"""
    x = _rand((rows, dim + 8), 3, 2.0)[:, :dim] + 0.5
    x = torch.cat([x, x[:, :8]], 1)[:, :dim]
    w, b = 1 + _rand((dim,), 4, 0.1), _rand((dim,), 5, 0.1)
    x64 = x.double()
    d = x64 - x64.mean(1, keepdim=True)
    ln, rms = ctx.layernorm(x, w, b, 1e-6), ctx.rmsnorm(x, w, 1e-6)
    want = d / (d.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double() + b.double()
    # rounding to bf16 (8 significant bits: 2^-8 of the value at most), plus fp32 arithmetic on terms of up to 2^3 (a few ulps of 2^-21)
    assert ((ln.double() - want).abs() <= 2 ** -7.95 * want.abs() + 2 ** -17).all()
    want = x64 / (x64.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
    assert ((rms.double() - want).abs() <= 2 ** -6.95 * want.abs()).all()     # two roundings to bf16
    n = max(1, rows // 3)
    assert torch.equal(ctx.layernorm(x[:n], w, b, 1e-6), ln[:n]) and torch.equal(ctx.rmsnorm(x[:n], w, 1e-6), rms[:n])


def test_cast(ctx):
    x = torch.randn((1024, 1176), device=DEV)
    assert torch.equal(ctx.cast_f32_bf16(x), x.to(torch.bfloat16))
    x = torch.randn((13,), device=DEV)
    assert torch.equal(ctx.cast_f32_bf16(x), x.to(torch.bfloat16))


@pytest.mark.parametrize("grid", [(1, 32, 32), (3, 8, 10), (2, 26, 46)])
def test_vit_rope(ctx, grid):
    t, h, w = grid
    heads, hd = 4, 80
    N = t * h * w
    g = torch.tensor([[t, h, w]])
    cos_ref, sin_ref = R.vit_rotary_cos_sin(g, hd, DEV)  # [N, 80] fp32 (cos of host-built angles, on GPU)
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, hd // 2, 2, dtype=torch.float) / (hd // 2)))).to(DEV)
    cos, sin = ctx.vit_rope_table(t, h, w, hd, inv_freq)
    torch.cuda.synchronize()
    assert torch.allclose(cos, cos_ref[:, : hd // 2], atol=2e-7, rtol=0)
    assert torch.allclose(sin, sin_ref[:, : hd // 2], atol=2e-7, rtol=0)
    qkv = _rand((N, 3 * heads * hd), 3)
    q, k, v = qkv.reshape(N, 3, heads, hd).permute(1, 0, 2, 3).unbind(0)
    qr, kr = R.vit_apply_rotary(q, k, cos_ref, sin_ref)
    out = ctx.vit_rope_apply(qkv.clone(), cos, sin, heads, hd).reshape(N, 3, heads, hd)
    assert _mismatch(out[:, 0], qr, 1.0) < 1e-3 and _mismatch(out[:, 1], kr, 1.0) < 1e-3
    assert torch.equal(out[:, 2], v)


@pytest.mark.parametrize("seglens,heads", [([1024], 4), ([256, 256, 256], 4), ([1196, 1196], 4), ([64, 80], 4),
                                           ([1024] * 5, 16), ([1196] * 4, 16), ([200, 1024, 328], 16)])
@pytest.mark.parametrize("impl", [2, 1])
def test_vit_attention(ctx, seglens, heads, impl):
    """impl 2 = tcgen05/TMEM kernel (default; 128-key tiles up to one wave of CTAs, 64-key tiles beyond),
    impl 1 = mma.sync kernels (the last three cases are large enough to take their 128-row variant)"""
    hd = 80
    N = sum(seglens)
    qkv = _rand((N, 3 * heads * hd), 4)
    cu = [0]
    for n in seglens:
        cu.append(cu[-1] + n)
    # reference: eager attention per segment (no rotary here: identity cos/sin)
    out = ctx.vit_attention(qkv, torch.tensor(cu, dtype=torch.int32, device=DEV), max(seglens), heads, hd, impl=impl)
    q, k, v = qkv.reshape(N, 3, heads, hd).permute(1, 2, 0, 3).unbind(0)  # [heads, N, hd]
    refs = [_attn_ref_fp32(q[:, s:e], k[:, s:e], v[:, s:e], None, hd ** -0.5) for s, e in zip(cu[:-1], cu[1:])]
    ref = torch.cat(refs, dim=1).transpose(0, 1).reshape(N, heads * hd)
    _attn_close(out, ref, "vit_attention")
    # and within bf16-eager noise of the HF eager formulation
    cos = torch.ones((N, hd), device=DEV)
    sin = torch.zeros((N, hd), device=DEV)
    eager = R.vit_attention(qkv, cu, heads, cos, sin)
    assert (out.float() - eager.float()).abs().max().item() < 5e-2


def test_embed_gather(ctx):
    V, H, S = 5000, 1792, 700
    table = _rand((V, H), 5)
    ids = torch.randint(0, V, (S,), device=DEV)
    vid_id = 4987
    ids[ids == vid_id] = 0  # random ids must not collide with the placeholder id
    ids[40:296] = vid_id
    ids[500:564] = vid_id
    video = _rand((320, H), 6)
    out, rank = ctx.embed_gather(ids, table, video, vid_id)
    ref = table[ids].clone()
    ref[ids == vid_id] = video
    assert torch.equal(out, ref)
    assert int(rank[S].item()) == 320
    out2, _ = ctx.embed_gather(ids[:30], table, None, vid_id)
    assert torch.equal(out2, table[ids[:30]])


class PagedCache:
    def __init__(self, layers, Hkv, max_tokens, seed=0):
        self.pages = (max_tokens + 63) // 64 + 3
        g = torch.Generator().manual_seed(seed)
        self.page_table = torch.randperm(self.pages, generator=g).to(torch.int32).to(DEV)
        self.k = torch.zeros((layers, self.pages, Hkv, 64, 128), dtype=torch.bfloat16, device=DEV)
        self.v = torch.zeros_like(self.k)

    def gather(self, layer, T):
        """logical [Hkv, T, 128] views of the cache."""
        pt = self.page_table.long()[: (T + 63) // 64]
        k = self.k[layer][pt].permute(1, 0, 2, 3).reshape(self.k.shape[2], -1, 128)[:, :T]
        v = self.v[layer][pt].permute(1, 0, 2, 3).reshape(self.v.shape[2], -1, 128)[:, :T]
        return k, v


def _text_inv_freq():
    return (1.0 / (1e6 ** (torch.arange(0, 128, 2, dtype=torch.int64).to(torch.float) / 128))).to(DEV)


@pytest.mark.parametrize("impl,split", [(2, False), (2, True), (1, False), (1, True)])
@pytest.mark.parametrize("S,past", [(281, 0), (300, 1000), (1, 64), (70, 3), (281, 4100)])
def test_mrope_kv_write_and_prefill_attention(ctx, S, past, impl, split):
    """impl 2 = tcgen05/TMEM kernel (default), impl 1 = mma.sync kernel; split = with split-KV scratch (the split
    count is the kernel's choice: > 1 only for the long-past cases). The cache pages start as NaN bit patterns, as a
    recycled pool page may: nothing behind the newest token may leak into the result."""
    Hq, Hkv = 14, 2
    cache = PagedCache(1, Hkv, past + S)
    cache.k.fill_(float("nan"))
    cache.v.fill_(float("nan"))
    inv = _text_inv_freq()
    # pre-fill the past part of the cache with random (already rotated) keys/values
    if past:
        pk, pv = _rand((Hkv, past, 128), 7), _rand((Hkv, past, 128), 8)
        for t0 in range(0, past, 64):
            n = min(64, past - t0)
            pg = int(cache.page_table[t0 // 64])
            cache.k[0, pg, :, :n] = pk[:, t0:t0 + n]
            cache.v[0, pg, :, :n] = pv[:, t0:t0 + n]
    qkv = _rand((S, (Hq + 2 * Hkv) * 128), 9)
    g = torch.Generator().manual_seed(10)
    pos3 = torch.stack([torch.arange(past, past + S) + int(torch.randint(0, 50, (1,), generator=g)) for _ in range(3)])
    pos3[1, S // 3:] += 7
    pos3[2, S // 2:] += 11
    q = qkv[:, : Hq * 128].view(S, Hq, 128).transpose(0, 1)
    k = qkv[:, Hq * 128:(Hq + Hkv) * 128].view(S, Hkv, 128).transpose(0, 1)
    v = qkv[:, (Hq + Hkv) * 128:].view(S, Hkv, 128).transpose(0, 1)
    cos, sin = R.mrope_cos_sin(pos3.to(DEV), 128, 1e6, torch.bfloat16, (16, 24, 24))
    q_ref, k_ref = R.apply_mrope(q, k, cos, sin)
    work = qkv.clone()
    ctx.mrope_kv_write(work, pos3.to(torch.int32).to(DEV).contiguous(), inv, 16, 24, Hq, Hkv, cache.k[0], cache.v[0],
                       cache.page_table, past)
    q_out = work[:, : Hq * 128].view(S, Hq, 128).transpose(0, 1)
    assert _mismatch(q_out, q_ref, 1.0) < 2e-3 and _mismatch(q_out, q_ref, 2.0) < 1e-5
    kc, vc = cache.gather(0, past + S)
    assert _mismatch(kc[:, past:], k_ref, 1.0) < 2e-3
    assert torch.equal(vc[:, past:], v)
    if past:
        assert torch.equal(kc[:, :past], pk) and torch.equal(vc[:, :past], pv)
    # attention of the S new rows over past+S
    out = ctx.attn_prefill(work, cache.k[0], cache.v[0], cache.page_table, Hq, Hkv, past, impl=impl, split=split)
    T = past + S
    rep = Hq // Hkv
    kr = kc[:, None].expand(Hkv, rep, T, 128).reshape(Hq, T, 128)
    vr = vc[:, None].expand(Hkv, rep, T, 128).reshape(Hq, T, 128)
    iq = torch.arange(past, T, device=DEV)[:, None]
    ik = torch.arange(T, device=DEV)[None, :]
    mask = torch.zeros((S, T), dtype=torch.bfloat16, device=DEV).masked_fill_(ik > iq, torch.finfo(torch.bfloat16).min)
    ref = _attn_ref_fp32(q_out.contiguous(), kr, vr, mask, 128 ** -0.5).transpose(0, 1).reshape(S, Hq * 128)
    _attn_close(out, ref, "attn_prefill")
    eager = R.eager_attention(q_out.contiguous(), kr, vr, mask, 128 ** -0.5).transpose(0, 1).reshape(S, Hq * 128)
    assert (out.float() - eager.float()).abs().max().item() < 5e-2


@pytest.mark.parametrize("S,past,rows", [(1, 16384, 32), (24, 17000, 32), (24, 17000, 5), (19, 1100, 32), (300, 9000, 3), (40, 511, 32), (2, 126, 32)])
def test_prefill_attention_split_counts(ctx, S, past, rows):
    """few new rows over a long past: as many splits as there are places for, at least 8 tiles each, and as fit into the scratch (`rows`
    splits' worth); splits of 1, 2 and more tiles, a last one cut short"""
    Hq, Hkv = 14, 2
    T = past + S
    cache = PagedCache(1, Hkv, T)
    k, v = _rand((Hkv, T, 128), 31), _rand((Hkv, T, 128), 32)
    cache.k.zero_(), cache.v.zero_()
    for t0 in range(0, T, 64):
        n, pg = min(64, T - t0), int(cache.page_table[t0 // 64])
        cache.k[0, pg, :, :n], cache.v[0, pg, :, :n] = k[:, t0:t0 + n], v[:, t0:t0 + n]
    q = _rand((S, Hq * 128), 33)
    out = torch.empty_like(q)
    part_o = torch.empty((rows * S * Hq, 128), device=DEV)
    part_ml = torch.empty((rows * S * Hq, 2), device=DEV)
    ctx.call("lcc_attn_prefill", A._ptr(q), A._i(q.stride(0)), A._ptr(cache.k[0]), A._ptr(cache.v[0]), A._ptr(cache.page_table), A._i(Hq), A._i(Hkv),
             A._i(S), A._i(past), A._ptr(out), A._i(out.stride(0)), A._ptr(part_o), A._ptr(part_ml), A.C.c_int64(part_o.shape[0]), A._i(2),
             ctx.stream_ptr())
    rep = Hq // Hkv
    mask = torch.zeros((S, T), device=DEV).masked_fill_(torch.arange(T, device=DEV)[None, :] > torch.arange(past, T, device=DEV)[:, None], float("-inf"))
    ref = _attn_ref_fp32(q.view(S, Hq, 128).transpose(0, 1), k.repeat_interleave(rep, 0), v.repeat_interleave(rep, 0), mask, 128 ** -0.5)
    _attn_close(out, ref.transpose(0, 1).reshape(S, Hq * 128), "attn_prefill")


@pytest.mark.parametrize("kv_len", [0, 1, 63, 64, 65, 1000, 5000])
@pytest.mark.parametrize("nsplit", [1, 8, 37])
def test_attn_decode(ctx, kv_len, nsplit):
    Hq, Hkv = 14, 2
    cache = PagedCache(1, Hkv, kv_len + 1, seed=kv_len)
    inv = _text_inv_freq()
    if kv_len:
        pk, pv = _rand((Hkv, kv_len, 128), 11), _rand((Hkv, kv_len, 128), 12)
        for t0 in range(0, kv_len, 64):
            n = min(64, kv_len - t0)
            pg = int(cache.page_table[t0 // 64])
            cache.k[0, pg, :, :n] = pk[:, t0:t0 + n]
            cache.v[0, pg, :, :n] = pv[:, t0:t0 + n]
    qkv = _rand(((Hq + 2 * Hkv) * 128,), 13)
    pos = kv_len - 37 if kv_len > 100 else kv_len + 5
    sc = torch.zeros(A.SC_COUNT, dtype=torch.int32, device=DEV)
    sc[A.SC_KV_LEN] = kv_len
    sc[A.SC_ROPE_POS] = pos
    out = ctx.attn_decode(qkv.clone(), cache.k[0], cache.v[0], cache.page_table, sc, inv, Hq, Hkv, nsplit)
    q = qkv[: Hq * 128].view(1, Hq, 128).transpose(0, 1)
    k = qkv[Hq * 128:(Hq + Hkv) * 128].view(1, Hkv, 128).transpose(0, 1)
    v = qkv[(Hq + Hkv) * 128:].view(1, Hkv, 128).transpose(0, 1)
    pos3 = torch.full((3, 1), pos, dtype=torch.long, device=DEV)
    cos, sin = R.mrope_cos_sin(pos3, 128, 1e6, torch.bfloat16, (16, 24, 24))
    q_ref, k_ref = R.apply_mrope(q, k, cos, sin)
    T = kv_len + 1
    kc, vc = cache.gather(0, T)
    assert _mismatch(kc[:, kv_len:], k_ref, 1.0) < 5e-3 and torch.equal(vc[:, kv_len:], v)
    rep = Hq // Hkv
    kr = kc[:, None].expand(Hkv, rep, T, 128).reshape(Hq, T, 128)
    vr = vc[:, None].expand(Hkv, rep, T, 128).reshape(Hq, T, 128)
    q_used = q_ref  # the kernel rotates q itself; rotated-q parity is covered by the k check above
    ref = _attn_ref_fp32(q_used, kr, vr, None, 128 ** -0.5).transpose(0, 1).reshape(Hq * 128)
    _attn_close(out, ref, "attn_decode")


@pytest.mark.parametrize("H,Hq,Hkv,I", [(3584, 28, 4, 18944), (1792, 14, 2, 4864)])
def test_decode_gemvs(ctx, H, Hq, Hkv, I):
    from livecc_b200.checkpoint import interleave_gate_up

    x = _rand((H,), 20, 2.0)
    nw = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16)
    xn = R.rms_norm(x[None], nw, 1e-6)[0]
    Nq = (Hq + 2 * Hkv) * 128
    W = _rand((Nq, H), 21, 0.02)
    b = _rand((Nq,), 22, 0.02)
    out = ctx.gemv_norm_bias(W, x, nw, 1e-6, b)
    ref = (W.float() @ xn.float() + b.float()).to(torch.bfloat16)
    assert _mismatch(out, ref, 2.0, floor=1e-2) < 1e-3
    # o_proj + residual
    Wo = _rand((H, Hq * 128), 23, 0.02)
    a = _rand((Hq * 128,), 24)
    h = x.clone()
    ctx.gemv_residual(Wo, a, h)
    ref = (Wo.float() @ a.float()).to(torch.bfloat16) + x
    assert _mismatch(h, ref, 2.0, floor=1e-2) < 1e-3
    # gate/up + swiglu
    Wg, Wu = _rand((I, H), 25, 0.02), _rand((I, H), 26, 0.02)
    act = ctx.gemv_norm_swiglu(interleave_gate_up(Wg, Wu), x, nw, 1e-6)
    gt = (Wg.float() @ xn.float()).to(torch.bfloat16)
    up = (Wu.float() @ xn.float()).to(torch.bfloat16)
    ref = torch.nn.functional.silu(gt) * up
    assert _mismatch(act, ref, 3.0, floor=1e-2) < 2e-3
    # down + residual (split-K kernel when I > 8192)
    Wd = _rand((H, I), 27, 0.01)
    h2 = x.clone()
    ctx.gemv_residual(Wd, ref, h2)
    ref2 = (Wd.float() @ ref.float()).to(torch.bfloat16) + x
    assert _mismatch(h2, ref2, 2.0, floor=1e-2) < 1e-3
    # logits
    V = 16384 + 40
    Wl = _rand((V, H), 28, 0.02)
    lg, lg2 = ctx.gemv_norm_logits(Wl, x, nw, 1e-6)
    refl = (Wl.float() @ xn.float()).to(torch.bfloat16).float()
    assert torch.equal(lg, lg2)
    assert _mismatch(lg, refl, 2.0, floor=1e-2) < 1e-3


def test_sample_greedy(ctx):
    V, H = 152064, 3584
    g = torch.Generator(device=DEV).manual_seed(30)
    raw = torch.randn(V, device=DEV, generator=g) * 3
    embed = _rand((V, H), 31)
    hist = torch.randint(0, V, (5000,), device=DEV, generator=g)
    top = int(raw.argmax())
    hist[17] = top
    hist[900] = top  # duplicates must be penalised once
    seq = torch.zeros(6000, dtype=torch.int64, device=DEV)
    seq[:5000] = hist
    sc = torch.zeros(A.SC_COUNT, dtype=torch.int32, device=DEV)
    sc[A.SC_KV_LEN], sc[A.SC_ROPE_POS], sc[A.SC_SEQ_LEN] = 5000, 4000, 5000
    sp = A.Sampling(1.05, -1, 0.0, 0.0, 7, 16, 1.0 / 1.05, -1)
    proc = raw.clone()
    h = torch.empty(H, dtype=torch.bfloat16, device=DEV)
    ctx.sample_greedy(raw, proc, seq, sc, sp, 1, embed, h)
    ref = raw.clone()
    s = ref[hist]
    ref[hist] = torch.where(s < 0, s * 1.05, s / 1.05)
    tok = int(ref.argmax())
    if not torch.equal(proc, ref):  # diagnostic: which rounding variant does torch use on this build?
        ref_div = raw.clone()
        ref_div[hist] = torch.where(s < 0, s * 1.05, (s.double() / 1.05).float())
        bad = (proc != ref).nonzero().flatten()
        print("penalty mismatches vs torch:", bad.numel(), "vs true division:", int((proc != ref_div).sum()),
              [(int(i), float(raw[i]), float(proc[i]), float(ref[i])) for i in bad[:4]])
    assert torch.equal(proc, ref)  # bit-exact with torch's CUDA semantics
    assert int(seq[5000]) == tok and torch.equal(h, embed[tok])
    assert sc.tolist()[:6] == [5001, 4001, 0, 1, 5001, tok]
    # threshold processor: force -inf on the would-be argmax token
    sc2 = torch.zeros(A.SC_COUNT, dtype=torch.int32, device=DEV)
    sc2[A.SC_SEQ_LEN] = 5000
    proc2 = raw.clone()
    sp2 = A.Sampling(1.0, tok, 1.1, 0.0, 7, 1, 1.0, -1)
    ctx.sample_greedy(raw, proc2, seq, sc2, sp2, 0, embed, h)
    ref2 = raw.clone()
    ref2[tok] = -float("inf")
    assert int(seq[5000]) == int(ref2.argmax())
    assert sc2.tolist()[:5] == [0, 0, 1, 1, 5001]  # finished by max_new_tokens = 1, no kv advance
    # finished flag => no-op
    before = seq.clone()
    ctx.sample_greedy(raw, proc2, seq, sc2, sp2, 0, embed, h)
    assert torch.equal(seq, before)


def test_threshold_processor_matches_reference_golden(ctx):
    """ThresholdLogitsProcessor inside the sampling kernel vs the reference's own class (REF/demo/infer.py:10-23)
    executed verbatim by tests/golden/make_threshold_golden.py: the `<=` boundary, a threshold that rises with
    `count` (= tokens generated so far in this generate(), a new processor is built per chunk: infer.py:161-162) and
    the canonical caller's base 0.0 / step 0 (REF/demo/cli.py:16-19)."""
    import json
    import os

    gold = json.load(open(os.path.join(os.path.dirname(__file__), "golden", "threshold_golden.json")))
    V, H = gold["V"], 64
    embed = _rand((V, H), 41)
    for c in gold["cases"]:
        raw = torch.tensor(c["scores"], dtype=torch.float32, device=DEV)
        for k in range(c["n_calls"]):
            seq = torch.zeros(64, dtype=torch.int64, device=DEV)
            sc = torch.zeros(A.SC_COUNT, dtype=torch.int32, device=DEV)
            sc[A.SC_N_GENERATED] = k          # == the reference processor's `count` at this call
            sp = A.Sampling(1.0, c["token"], c["base"], c["step"], V + 7, 64, 1.0, -1)
            proc = raw.clone()
            h = torch.empty(H, dtype=torch.bfloat16, device=DEV)
            ctx.sample_greedy(raw, proc, seq, sc, sp, 0, embed, h)
            torch.cuda.synchronize()
            masked = bool(torch.isinf(proc[c["token"]]) and proc[c["token"]] < 0)
            assert masked == c["masked"][k], (c["name"], k, masked, c["prob"], c["base"] + c["step"] * k)
            assert int(seq[0]) == c["argmax"][k], (c["name"], k, int(seq[0]), c["argmax"][k])
            assert sc.tolist()[A.SC_N_GENERATED] == k + 1


def test_embed_gather_never_reads_past_the_video_rows(ctx):
    """More <|video_pad|> ids than ViT rows (the mismatch the engine raises on, mq2vl.py:1169-1175): placeholders
    beyond the last feature row keep their text embedding instead of reading past the end of `video_embeds`."""
    H, V, vid = 256, 1000, 999
    table = _rand((V, H), 51)
    # the feature buffer is the tail of an allocation whose neighbour is poisoned with NaN
    buf = torch.full((8, H), float("nan"), dtype=torch.bfloat16, device=DEV)
    buf[:3] = _rand((3, H), 52)
    feats = buf[:3]
    ids = torch.tensor([5, vid, vid, 6, vid, vid, vid, 7], dtype=torch.int64, device=DEV)  # 5 placeholders, 3 rows
    out, rank = ctx.embed_gather(ids, table, feats, vid)
    torch.cuda.synchronize()
    assert int(rank[ids.numel()]) == 5                       # the count the host compares with the feature rows
    assert torch.equal(out[1], feats[0]) and torch.equal(out[2], feats[1]) and torch.equal(out[4], feats[2])
    assert torch.equal(out[5], table[vid]) and torch.equal(out[6], table[vid])
    assert torch.equal(out[0], table[5]) and not torch.isnan(out.float()).any()
    # no features at all: placeholders are plain text ids, as in the reference when pixel values are absent
    out2, rank2 = ctx.embed_gather(ids, table, None, vid)
    torch.cuda.synchronize()
    assert torch.equal(out2, table[ids]) and int(rank2[ids.numel()]) == 0


@pytest.mark.parametrize("V", [1, 7, 8191, 32768 + 5, 152064])
@pytest.mark.parametrize("hist", [0, 1, 8193, 70001])
def test_sample_greedy_sizes(ctx, V, hist):
    """The selection is shared out over the CTAs of a cluster: vocabularies smaller than a CTA, remainders behind the 4-wide part,
    histories from none to several passes, ties whose copies lie in different CTAs (the lowest index wins), the threshold's sum."""
    g = torch.Generator(device=DEV).manual_seed(V + hist)
    raw = torch.randn(V, device=DEV, generator=g)
    ties = torch.randint(0, V, (4,), device=DEV, generator=g)
    raw[ties] = 9.0
    ids = torch.randint(0, V, (hist,), device=DEV, generator=g)
    ids[ids == ties.min()] = (int(ties.min()) + 1) % V if V > 1 else 0
    seq = torch.zeros(hist + 2, dtype=torch.int64, device=DEV)
    seq[:hist] = ids
    ref = raw.clone()
    s = ref[ids]
    ref[ids] = torch.where(s < 0, s * 1.25, s * 0.8)
    for thr in (-1, int(ref.argmax())):
        sc = torch.zeros(A.SC_COUNT, dtype=torch.int32, device=DEV)
        sc[A.SC_SEQ_LEN] = hist
        want = ref.clone()
        if thr >= 0:      # the share of the best token lies between the two bases
            share = float(torch.softmax(ref.double(), 0)[thr])
            for base, masked in ((share * 0.999, False), (share * 1.001, True)):
                proc, sc2 = raw.clone(), sc.clone()
                ctx.sample_greedy(raw, proc, seq, sc2, A.Sampling(1.25, thr, base, 0.0, -1, 16, 0.8, -1), 0, torch.zeros((V, 8), dtype=torch.bfloat16, device=DEV),
                                  torch.zeros(8, dtype=torch.bfloat16, device=DEV))
                assert bool(torch.isinf(proc[thr])) == masked
            continue
        proc = raw.clone()
        ctx.sample_greedy(raw, proc, seq, sc, A.Sampling(1.25, -1, 0.0, 0.0, -1, 16, 0.8, -1), 1, torch.zeros((V, 8), dtype=torch.bfloat16, device=DEV),
                          torch.zeros(8, dtype=torch.bfloat16, device=DEV))
        assert torch.equal(proc, want)
        assert int(seq[hist]) == int((want == want.max()).nonzero()[0])
        assert sc.tolist()[:6] == [1, 1, 0, 1, hist + 1, int(seq[hist])]


@pytest.mark.parametrize("Hq,Hkv", [(28, 4), (8, 1), (3, 3)])
@pytest.mark.parametrize("nsplit", [8, 16, 24, 64])
@pytest.mark.parametrize("kv_len", [0, 63, 64, 511, 4095, 9001])
def test_attn_decode_splits_merged_in_clusters(ctx, kv_len, nsplit, Hq, Hkv):
    """Multiples of 8 splits merge inside clusters, one query head per CTA: one to eight clusters, empty splits, groups of 1 to 8 heads,
    the new token alone in its tile; launched twice, since the arrival counts of a launch have to be back at zero."""
    cache = PagedCache(1, Hkv, kv_len + 1, seed=kv_len)
    cache.k.fill_(float("nan"))     # (a recycled page may hold anything behind the newest token)
    cache.v.fill_(float("nan"))
    pk, pv = _rand((Hkv, max(kv_len, 1), 128), 61), _rand((Hkv, max(kv_len, 1), 128), 62)
    for t0 in range(0, kv_len, 64):
        n = min(64, kv_len - t0)
        pg = int(cache.page_table[t0 // 64])
        cache.k[0, pg, :, :n], cache.v[0, pg, :, :n] = pk[:, t0:t0 + n], pv[:, t0:t0 + n]
    qkv = _rand(((Hq + 2 * Hkv) * 128,), 63)
    sc = torch.zeros(A.SC_COUNT, dtype=torch.int32, device=DEV)
    sc[A.SC_KV_LEN], sc[A.SC_ROPE_POS] = kv_len, kv_len + 3
    outs = [ctx.attn_decode(qkv.clone(), cache.k[0], cache.v[0], cache.page_table, sc, _text_inv_freq(), Hq, Hkv, nsplit) for _ in range(2)]
    assert torch.equal(outs[0], outs[1]) and not ctx._attn_counters.any()
    q = qkv[: Hq * 128].view(1, Hq, 128).transpose(0, 1)
    k = qkv[Hq * 128:(Hq + Hkv) * 128].view(1, Hkv, 128).transpose(0, 1)
    cos, sin = R.mrope_cos_sin(torch.full((3, 1), kv_len + 3, dtype=torch.long, device=DEV), 128, 1e6, torch.bfloat16, (16, 24, 24))
    q_ref, _ = R.apply_mrope(q, k, cos, sin)
    kc, vc = cache.gather(0, kv_len + 1)
    rep = Hq // Hkv
    kr, vr = (x[:, None].expand(Hkv, rep, kv_len + 1, 128).reshape(Hq, kv_len + 1, 128) for x in (kc, vc))
    _attn_close(outs[0], _attn_ref_fp32(q_ref, kr, vr, None, 128 ** -0.5).transpose(0, 1).reshape(Hq * 128), "attn_decode")


def test_a_context_does_not_wait_for_the_gpu():
    """A context beside running work: nothing of its creation or its end synchronises (some 300 ms of products lie in front)."""
    import time

    A.Context(0)          # (the first one of a process may)
    x = torch.randn((8192, 8192), device="cuda")
    x @ x
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    for _ in range(20):
        x = torch.tanh(x @ x)
    done.record()
    for _ in range(3):
        A.Context(0)
    assert not done.query()
    torch.cuda.synchronize()
