"""ORACLE (test infrastructure — never imported by the product path).

Plain-torch restatement of the arithmetic on LiveCC's encode -> prefill -> decode path, one function per
stage, each citing the lines of the third-party implementation the reference runs
(`mq2vl.py` = transformers 5.5.0 models/qwen2_vl/modeling_qwen2_vl.py; `gen/utils.py` =
transformers/generation/utils.py). It imports no HF modeling code. Two uses:

  * CPU fp32: must reproduce the installed HF model's greedy ids *exactly* and its logits to fp32
    round-off (tests/test_oracle_cpu.py pins this, and tests/golden/ holds HF-generated vectors);
  * GPU bf16: per-op reference for the CUDA kernels — the ops are issued in the same order as the HF
    eager graph so every bf16 rounding point coincides.

Parity status: the reference repo has no tests or golden vectors for this path, so the
restatement is pinned against outputs of the installed HF implementation, generated by
tests/golden/make_golden.py (committed with its outputs).
"""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import Dict, List, Optional, Tuple

import torch
import torch.nn.functional as F


# ------------------------------------------------------------------------------------------------
# elementwise pieces
# ------------------------------------------------------------------------------------------------
def rms_norm(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    """Qwen2VLRMSNorm.forward, mq2vl.py:126-131 (fp32 statistics, cast back *before* the weight multiply)."""
    dt = x.dtype
    h = x.to(torch.float32)
    var = h.pow(2).mean(-1, keepdim=True)
    h = h * torch.rsqrt(var + eps)
    return w * h.to(dt)


def layer_norm(x: torch.Tensor, w: torch.Tensor, b: torch.Tensor, eps: float = 1e-6) -> torch.Tensor:
    """nn.LayerNorm(embed_dim, eps=1e-6), mq2vl.py:464-465,317."""
    return F.layer_norm(x, (x.shape[-1],), w, b, eps)


def quick_gelu(x: torch.Tensor) -> torch.Tensor:
    """ACT2FN['quick_gelu'], SP/transformers/activations.py:117-123."""
    return x * torch.sigmoid(1.702 * x)


def rotate_half(x: torch.Tensor) -> torch.Tensor:
    """mq2vl.py:205-209."""
    x1 = x[..., : x.shape[-1] // 2]
    x2 = x[..., x.shape[-1] // 2:]
    return torch.cat((-x2, x1), dim=-1)


# ------------------------------------------------------------------------------------------------
# ViT
# ------------------------------------------------------------------------------------------------
def vit_pos_ids(grid_thw: torch.Tensor, merge: int = 2) -> torch.Tensor:
    """rot_pos_emb index part, mq2vl.py:725-748: (h, w) id of every patch in merge-window order -> [N, 2]."""
    out = []
    for t, h, w in grid_thw.tolist():
        hpos = torch.arange(h).unsqueeze(1).expand(-1, w)
        hpos = hpos.reshape(h // merge, merge, w // merge, merge).permute(0, 2, 1, 3).flatten()
        wpos = torch.arange(w).unsqueeze(0).expand(h, -1)
        wpos = wpos.reshape(h // merge, merge, w // merge, merge).permute(0, 2, 1, 3).flatten()
        out.append(torch.stack([hpos, wpos], dim=-1).repeat(t, 1))
    return torch.cat(out, dim=0)


def vit_rotary_cos_sin(grid_thw: torch.Tensor, head_dim: int, device, theta: float = 10000.0):
    """mq2vl.py:271-284,749-752,773-775: fp32 cos/sin of shape [N, head_dim]."""
    dim = head_dim // 2
    inv_freq = 1.0 / (theta ** (torch.arange(0, dim, 2, dtype=torch.float) / dim))
    pos = vit_pos_ids(grid_thw)
    max_grid = int(grid_thw[:, 1:].max())
    seq = torch.arange(max_grid, dtype=torch.float)
    freqs_full = torch.outer(seq, inv_freq)
    rot = freqs_full[pos].flatten(1).to(device)          # [N, dim]
    emb = torch.cat((rot, rot), dim=-1)                  # [N, head_dim]
    return emb.cos(), emb.sin()


def vit_apply_rotary(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """apply_rotary_pos_emb_vision, mq2vl.py:257-268 (fp32 math, cast back). q,k: [N, heads, d]."""
    dq, dk = q.dtype, k.dtype
    q, k = q.float(), k.float()
    cos, sin = cos.unsqueeze(-2).float(), sin.unsqueeze(-2).float()
    qe = (q * cos) + (rotate_half(q) * sin)
    ke = (k * cos) + (rotate_half(k) * sin)
    return qe.to(dq), ke.to(dk)


def eager_attention(q, k, v, mask, scaling):
    """eager_attention_forward, mq2vl.py:353-375 with KV heads already repeated. q:[H,S,d] k,v:[H,T,d]."""
    w = torch.matmul(q, k.transpose(1, 2)) * scaling
    if mask is not None:
        w = w + mask
    w = F.softmax(w, dim=-1, dtype=torch.float32).to(q.dtype)
    return torch.matmul(w, v)  # [H,S,d]


def vit_attention(qkv: torch.Tensor, cu_seqlens: List[int], heads: int, cos, sin) -> torch.Tensor:
    """VisionAttention.forward minus the projections, mq2vl.py:392-454 (non-flash branch: each
    cu_seqlens segment attends only to itself). qkv: [N, 3*heads*d] -> [N, heads*d]."""
    N = qkv.shape[0]
    q, k, v = qkv.reshape(N, 3, heads, -1).permute(1, 0, 2, 3).unbind(0)
    q, k = vit_apply_rotary(q, k, cos, sin)
    d = q.shape[-1]
    outs = []
    for s, e in zip(cu_seqlens[:-1], cu_seqlens[1:]):
        o = eager_attention(q[s:e].transpose(0, 1), k[s:e].transpose(0, 1), v[s:e].transpose(0, 1), None, d ** -0.5)
        outs.append(o.transpose(0, 1))  # [n, heads, d]
    return torch.cat(outs, dim=0).reshape(N, -1)


# ------------------------------------------------------------------------------------------------
# decoder pieces
# ------------------------------------------------------------------------------------------------
def mrope_cos_sin(pos3: torch.Tensor, head_dim: int, theta: float, dtype, mrope_section) -> Tuple[torch.Tensor, torch.Tensor]:
    """Qwen2VLRotaryEmbedding.forward (mq2vl.py:188-201) + the section gather of
    apply_multimodal_rotary_pos_emb (mq2vl.py:244-250). pos3: [3,S] int -> cos,sin [S, head_dim] in `dtype`."""
    inv_freq = 1.0 / (theta ** (torch.arange(0, head_dim, 2, dtype=torch.int64).to(dtype=torch.float) / head_dim))
    inv_freq = inv_freq.to(pos3.device)
    freqs = pos3[:, :, None].float() * inv_freq[None, None, :]       # [3,S,d/2]  (== inv_freq @ pos, K=1 matmul)
    emb = torch.cat((freqs, freqs), dim=-1)                           # [3,S,d]
    cos, sin = emb.cos().to(dtype), emb.sin().to(dtype)
    sec = list(mrope_section) * 2
    cos = torch.cat([m[i % 3] for i, m in enumerate(cos.split(sec, dim=-1))], dim=-1)
    sin = torch.cat([m[i % 3] for i, m in enumerate(sin.split(sec, dim=-1))], dim=-1)
    return cos, sin


def apply_mrope(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """mq2vl.py:252-254. q: [Hq,S,d], k: [Hkv,S,d], cos/sin: [S,d] (already section-gathered)."""
    c, s = cos.unsqueeze(0), sin.unsqueeze(0)
    return (q * c) + (rotate_half(q) * s), (k * c) + (rotate_half(k) * s)


def get_vision_position_ids(start: int, grid, merge: int = 2) -> torch.Tensor:
    """mq2vl.py:934-988 (transformers 5.5.0 semantics: constant temporal index)."""
    t, h, w = int(grid[0]), int(grid[1]) // merge, int(grid[2]) // merge
    n = t * h * w
    pw = torch.arange(start, start + w).repeat(h * t)
    ph = torch.arange(start, start + h).repeat_interleave(w * t)
    pt = torch.full((n,), start, dtype=torch.long)
    return torch.stack([pt, ph, pw], dim=0)


def get_rope_index(input_ids: List[int], video_token_id: int, image_token_id: int, grids: List[List[int]],
                   merge: int = 2) -> Tuple[torch.Tensor, int]:
    """Qwen2VLModel.get_rope_index for one un-padded sequence, mq2vl.py:1053-1090.
    Returns (pos [3,L], rope_delta = max_pos + 1 - L)."""
    types = [2 if t == video_token_id else (1 if t == image_token_id else 0) for t in input_ids]
    groups = []
    start = 0
    for i in range(1, len(types) + 1):
        if i == len(types) or types[i] != types[start]:
            groups.append((types[start], start, i))
            start = i
    cur = 0
    gi = iter(grids)
    parts = []
    for typ, s, e in groups:
        if typ == 0:
            n = e - s
            parts.append(torch.arange(n).view(1, -1).expand(3, -1) + cur)
            cur += n
        else:
            g = next(gi)
            parts.append(get_vision_position_ids(cur, g, merge))
            cur += max(int(g[1]), int(g[2])) // merge
    pos = torch.cat(parts, dim=1).reshape(3, -1)
    return pos, int(pos.max()) + 1 - len(input_ids)


# ------------------------------------------------------------------------------------------------
# the model
# ------------------------------------------------------------------------------------------------
@dataclass
class RestatedCache:
    """DynamicCache equivalent (cache_utils.py:102-121): per layer K,V [Hkv, T, d], grown by cat."""
    k: List[Optional[torch.Tensor]] = field(default_factory=list)
    v: List[Optional[torch.Tensor]] = field(default_factory=list)
    rope_delta: Optional[int] = None  # the reference keeps this on the *model* (mq2vl.py:923,1207,1518)

    def get_seq_length(self) -> int:
        return 0 if not self.k or self.k[0] is None else self.k[0].shape[1]


class RestatedLiveCC:
    """Weights are the HF-named tensors of livecc_b200.checkpoint (any dtype/device)."""

    def __init__(self, cfg, sd: Dict[str, torch.Tensor]):
        self.cfg, self.sd = cfg, sd
        self.dtype = sd["lm_head.weight"].dtype
        self.device = sd["lm_head.weight"].device

    # -- ViT --------------------------------------------------------------------------------
    def vit_forward(self, pixel_values: torch.Tensor, grid_thw: torch.Tensor, return_blocks: bool = False):
        """Qwen2VisionTransformerPretrainedModel.forward, mq2vl.py:757-795."""
        v, sd = self.cfg.vision_config, self.sd
        V = "model.visual."
        # PatchEmbed: Conv3d with kernel == stride is a GEMM over flattened patches (mq2vl.py:304-310)
        w = sd[V + "patch_embed.proj.weight"].reshape(v.embed_dim, -1)
        h = F.linear(pixel_values.to(self.dtype), w)
        cos, sin = vit_rotary_cos_sin(grid_thw, v.head_dim, self.device)
        lens = torch.repeat_interleave(grid_thw[:, 1] * grid_thw[:, 2], grid_thw[:, 0]).tolist()
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + int(n))
        blocks = []
        for i in range(v.depth):
            B = f"{V}blocks.{i}."
            x = layer_norm(h, sd[B + "norm1.weight"], sd[B + "norm1.bias"])
            qkv = F.linear(x, sd[B + "attn.qkv.weight"], sd[B + "attn.qkv.bias"])
            a = vit_attention(qkv, cu, v.num_heads, cos, sin)
            h = h + F.linear(a, sd[B + "attn.proj.weight"], sd[B + "attn.proj.bias"])
            x = layer_norm(h, sd[B + "norm2.weight"], sd[B + "norm2.bias"])
            x = quick_gelu(F.linear(x, sd[B + "mlp.fc1.weight"], sd[B + "mlp.fc1.bias"]))
            h = h + F.linear(x, sd[B + "mlp.fc2.weight"], sd[B + "mlp.fc2.bias"])
            if return_blocks:
                blocks.append(h)
        # PatchMerger, mq2vl.py:313-326
        x = layer_norm(h, sd[V + "merger.ln_q.weight"], sd[V + "merger.ln_q.bias"])
        x = x.view(-1, v.embed_dim * v.spatial_merge_size ** 2)
        x = F.gelu(F.linear(x, sd[V + "merger.mlp.0.weight"], sd[V + "merger.mlp.0.bias"]))
        out = F.linear(x, sd[V + "merger.mlp.2.weight"], sd[V + "merger.mlp.2.bias"])
        return (out, blocks) if return_blocks else out

    # -- decoder ----------------------------------------------------------------------------
    def decoder_forward(self, embeds: torch.Tensor, pos3: torch.Tensor, cache: RestatedCache,
                        return_layers: bool = False):
        """Qwen2VLTextModel.forward over S new tokens with a KV cache, mq2vl.py:828-910,613-662,546-594.
        embeds [S,H]; pos3 [3,S]. Returns final-normed hidden [S,H]."""
        t, sd = self.cfg.text_config, self.sd
        L = "model.language_model."
        S = embeds.shape[0]
        Hq, Hkv, d = t.num_attention_heads, t.num_key_value_heads, t.head_dim
        cos, sin = mrope_cos_sin(pos3.to(self.device), d, t.rope_theta, self.dtype, t.mrope_section)
        past = cache.get_seq_length()
        T = past + S
        # causal mask over past+new (bottom-right aligned), as create_causal_mask yields for eager attention
        idx_q = torch.arange(past, T, device=self.device)[:, None]
        idx_k = torch.arange(T, device=self.device)[None, :]
        mask = torch.zeros((S, T), dtype=self.dtype, device=self.device)
        mask.masked_fill_(idx_k > idx_q, torch.finfo(self.dtype).min)
        while len(cache.k) < t.num_hidden_layers:
            cache.k.append(None)
            cache.v.append(None)
        h = embeds
        layers_out = []
        for i in range(t.num_hidden_layers):
            B = f"{L}layers.{i}."
            x = rms_norm(h, sd[B + "input_layernorm.weight"], t.rms_norm_eps)
            q = F.linear(x, sd[B + "self_attn.q_proj.weight"], sd[B + "self_attn.q_proj.bias"])
            k = F.linear(x, sd[B + "self_attn.k_proj.weight"], sd[B + "self_attn.k_proj.bias"])
            v = F.linear(x, sd[B + "self_attn.v_proj.weight"], sd[B + "self_attn.v_proj.bias"])
            q = q.view(S, Hq, d).transpose(0, 1)
            k = k.view(S, Hkv, d).transpose(0, 1)
            v = v.view(S, Hkv, d).transpose(0, 1)
            q, k = apply_mrope(q, k, cos, sin)
            if cache.k[i] is not None:
                k = torch.cat([cache.k[i], k], dim=1)
                v = torch.cat([cache.v[i], v], dim=1)
            cache.k[i], cache.v[i] = k, v
            rep = Hq // Hkv
            kr = k[:, None].expand(Hkv, rep, T, d).reshape(Hq, T, d)
            vr = v[:, None].expand(Hkv, rep, T, d).reshape(Hq, T, d)
            a = eager_attention(q, kr, vr, mask, d ** -0.5)        # [Hq,S,d]
            a = a.transpose(0, 1).reshape(S, Hq * d)
            h = h + F.linear(a, sd[B + "self_attn.o_proj.weight"])
            x = rms_norm(h, sd[B + "post_attention_layernorm.weight"], t.rms_norm_eps)
            g = F.silu(F.linear(x, sd[B + "mlp.gate_proj.weight"])) * F.linear(x, sd[B + "mlp.up_proj.weight"])
            h = h + F.linear(g, sd[B + "mlp.down_proj.weight"])
            if return_layers:
                layers_out.append(h)
        out = rms_norm(h, sd[L + "norm.weight"], t.rms_norm_eps)
        return (out, layers_out) if return_layers else out

    def embed(self, ids: torch.Tensor, video_embeds: Optional[torch.Tensor]) -> torch.Tensor:
        """embed_tokens + masked_scatter of the video features, mq2vl.py:1255-1272. ids: [S]."""
        e = F.embedding(ids, self.sd["model.language_model.embed_tokens.weight"])
        if video_embeds is not None:
            m = ids == self.cfg.video_token_id
            assert int(m.sum()) == video_embeds.shape[0], "video tokens / features mismatch (mq2vl.py:1169-1175)"
            e = e.clone()
            e[m] = video_embeds.to(e.dtype)
        return e

    def logits(self, hidden_last: torch.Tensor) -> torch.Tensor:
        """lm_head on the last position then the fp32 cast of _sample (mq2vl.py:1437-1438, gen/utils.py:2762)."""
        return F.linear(hidden_last, self.sd["lm_head.weight"]).to(torch.float32)

    # -- generate ---------------------------------------------------------------------------
    @torch.inference_mode()
    def generate(self, input_ids: torch.Tensor, pixel_values_videos: Optional[torch.Tensor],
                 video_grid_thw: Optional[torch.Tensor], cache: Optional[RestatedCache] = None,
                 max_new_tokens: int = 16, repetition_penalty: float = 1.05, forced_ids: Optional[List[int]] = None,
                 return_logits: bool = False):
        """GenerationMixin.generate/_sample for the kwargs live_cc uses (REF/demo/infer.py:165-172):
        greedy, repetition penalty over the full history (logits_process.py:407-410), EOS stop,
        multi-turn KV reuse with turn-0 rope_delta (mq2vl.py:1493-1529, 1179-1226).
        input_ids: [1, L] full history. forced_ids: teacher forcing (use these instead of the argmax)."""
        cfg = self.cfg
        cache = cache if cache is not None else RestatedCache()
        ids_all = input_ids[0].tolist()
        past = cache.get_seq_length()
        new = ids_all[past:]
        S = len(new)
        if past == 0 or cache.rope_delta is None:
            pos3, delta = get_rope_index(new, cfg.video_token_id, cfg.image_token_id,
                                         video_grid_thw.tolist() if video_grid_thw is not None else [])
            cache.rope_delta = delta
        else:
            p = torch.arange(past, past + S) + cache.rope_delta
            pos3 = p.view(1, -1).expand(3, -1)
        new_t = torch.tensor(new, dtype=torch.long, device=self.device)
        vid = None
        if pixel_values_videos is not None and (new_t == cfg.video_token_id).any():
            vid = self.vit_forward(pixel_values_videos.to(self.device), video_grid_thw)
        h = self.decoder_forward(self.embed(new_t, vid), pos3, cache)
        logits_list, out_ids = [], []
        seq = list(ids_all)
        cur = h[-1:]
        for step in range(max_new_tokens):
            lg = self.logits(cur)[0]
            if return_logits:
                logits_list.append(lg.clone())
            if repetition_penalty != 1.0:
                idx = torch.tensor(seq, dtype=torch.long, device=self.device)
                sc = lg[idx]
                lg[idx] = torch.where(sc < 0, sc * repetition_penalty, sc / repetition_penalty)
            tok = int(torch.argmax(lg))
            if forced_ids is not None:
                tok = int(forced_ids[step])
            seq.append(tok)
            out_ids.append(tok)
            if tok == cfg.eos_token_id or step == max_new_tokens - 1:
                break
            p = cache.get_seq_length() + cache.rope_delta
            pos3 = torch.full((3, 1), p, dtype=torch.long)
            e = self.embed(torch.tensor([tok], dtype=torch.long, device=self.device), None)
            cur = self.decoder_forward(e, pos3, cache)
        sequences = torch.tensor([seq], dtype=torch.long, device=self.device)
        if return_logits:
            return sequences, cache, logits_list
        return sequences, cache
