"""Workloads this framework is timed on, each through the calls a program makes: frame ingest, the vision tower, turns of the
streaming loop (`generate`, one stream and several), and prompts and generation of the hybrid sequence models.

Every model has the widths of a served one and fewer layers, so that a pass shows its layers and not the number of them; weights
are random, with one trait of a trained model: the output head prefers one successor per token, so that greedy ids do not hang on the last
bit of a logit. `exact` restates each path in float64 torch."""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

F64 = torch.float64
TEXT = dict(hidden=3584, inter=18944, q_heads=28, kv_heads=4, vocab=152064, theta=1e6, eps=1e-6)
VIT = dict(dim=1280, heads=16, mlp=5120)
IDS = 150000          # text ids the workloads draw from (special ids lie above)
VIDEO_ID = 151656
SUCC, SUCC_ADD = 48271, 12345   # the successor the head prefers: i -> (i * SUCC + SUCC_ADD) mod ids
SEQ = dict(width=2048, vocab=32768, ff=5632, chunk=1024)
MEAN = (0.48145466, 0.4578275, 0.40821073)
STD = (0.26862954, 0.26130258, 0.27577711)


def listed():
    turn = dict(kind="turn", depth=2, layers=4, streams=1)
    return [
        # one 2-fps chunk of a 1080p source, brought to the size the model sees
        dict(name="ingest_1080p", kind="ingest", frames=2, h=1080, w=1920, H=448, W=796),
        # the vision tower on one streaming chunk (1024 patches; replayed as a whole)
        dict(name="vision_chunk", kind="vision", frames=2, H=448, W=448, depth=4),
        # the vision tower on a clip of a question about a video (8192 patches)
        dict(name="vision_clip", kind="vision", frames=16, H=448, W=448, depth=2),
        # one turn of live commentary: a chunk's frames, 281 new tokens behind a running stream, 16 tokens out
        dict(turn, name="turn_chunk", frames=2, H=448, W=448, text=25, past=8000, new=16),
        # a question typed late in a long stream: few tokens in, 16 out over a long cache
        dict(turn, name="turn_long", frames=0, H=0, W=0, text=24, past=65536, new=16),
        # a turn that is only read (scored): 281 tokens behind a long past, one token out
        dict(turn, name="turn_read", frames=0, H=0, W=0, text=281, past=17001, new=1),
        # the opening of a question about a clip: 16 frames and the question, one token out
        dict(turn, name="turn_open", frames=16, H=448, W=448, text=42, past=0, new=1),
        # eight streams answered together
        dict(turn, name="turn_8_streams", frames=0, H=0, W=0, text=24, past=8000, new=16, streams=8),
        # hybrid models: a prompt whose rows are scored, and a short prompt with generation, of two designs
        dict(name="recurrent_prompt", kind="prompt", design="Bimopel", layers=4, tokens=2048),
        dict(name="recurrent_generate", kind="gen", design="Bimopel", layers=4, tokens=128, new=32),
        dict(name="routed_prompt", kind="prompt", design="Dibedra", layers=2, tokens=1024),
        dict(name="routed_generate", kind="gen", design="Dibedra", layers=2, tokens=128, new=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ingest", "vision", "turn", "turn", "turn", "streams", "prompt", "prompt", "gen"])
    if kind == "ingest":
        h, w = rng.choice([(360, 640), (480, 854), (720, 1280), (1080, 1920), (rng.randrange(300, 1081), rng.randrange(400, 1921))])
        return dict(kind="ingest", frames=rng.randrange(1, 7), h=h, w=w, H=28 * rng.randrange(5, 21), W=28 * rng.randrange(5, 29))
    if kind == "vision":
        H, W = 28 * rng.randrange(5, 19), 28 * rng.randrange(5, 29)
        most = max(1, 8192 * 196 // (H * W))    # no more patches than the largest listed case has
        return dict(kind="vision", frames=min(2 * most, _log(rng, 1, 16)), H=H, W=W, depth=2)
    if kind == "turn":
        frames = rng.choice([0, 2, 2, 6])
        H, W = (28 * rng.randrange(8, 17), 28 * rng.randrange(8, 17)) if frames else (0, 0)
        past = rng.choice([0, _log(rng, 1, 65536), _log(rng, 1000, 32768)])
        return dict(kind="turn", depth=2, layers=4, streams=1, frames=frames, H=H, W=W, text=_log(rng, 2, 1200), past=past, new=_log(rng, 1, 16))
    if kind == "streams":
        return dict(kind="turn", depth=2, layers=4, streams=rng.randrange(2, 9), frames=0, H=0, W=0, text=_log(rng, 2, 64),
                    past=_log(rng, 100, 16384), new=rng.randrange(4, 17))
    design = rng.choice(["Bimopel", "Dibedra"])
    layers = 4 if design == "Bimopel" else 2
    if kind == "prompt":
        return dict(kind="prompt", design=design, layers=layers, tokens=_log(rng, 16, 2048))
    return dict(kind="gen", design=design, layers=layers, tokens=_log(rng, 1, 2048), new=_log(rng, 2, 32))


# ------------------------------------------------------------------------------------------------ inputs made from the seed
class _Fill:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)

    def u(self, *shape, width=1.0, at=0.0):
        """uniform in at +- width / 2, in the checkpoint's bf16"""
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        return t.uniform_(at - width / 2, at + width / 2, generator=self.g)

    def w(self, rows, cols, shape=None, most=1.0):
        """matrix whose rows have unit norm (or entries of +- most)"""
        return self.u(*(shape or (rows, cols)), width=min(2 * most, 3.4641 / cols ** 0.5))

    def ids(self, n, below):
        return torch.randint(0, below, (n,), generator=self.g, device="cuda")


def _head(f, embed, ids, scale):
    """Output rows: row succ(i) points along embedding i; rows without a predecessor are random."""
    head = f.w(embed.shape[0], embed.shape[1])
    i = torch.arange(ids, device="cuda")
    head[(i * SUCC + SUCC_ADD) % ids] = embed[:ids] * scale
    return head


def _chain(last, n, ids):
    out = []
    for _ in range(n):
        last = (last * SUCC + SUCC_ADD) % ids
        out.append(last)
    return out


def _livecc(seed, depth, layers, vocab=TEXT["vocab"], inter=TEXT["inter"]):
    """Checkpoint tensors by their published names."""
    f, t, H, D = _Fill(seed), {}, TEXT["hidden"], VIT["dim"]
    V, L = "model.visual.", "model.language_model."

    def lin(name, rows, cols, bias=True):
        t[name + ".weight"] = f.w(rows, cols, most=0.0346)
        if bias:
            t[name + ".bias"] = f.u(rows, width=0.04)

    def norm(name, n, bias=True):
        t[name + ".weight"] = f.u(n, width=0.2, at=1.0)
        if bias:
            t[name + ".bias"] = f.u(n, width=0.04)

    t[V + "patch_embed.proj.weight"] = f.w(D, 1176, shape=(D, 3, 2, 14, 14), most=0.0346)
    for i in range(depth):
        b = f"{V}blocks.{i}."
        norm(b + "norm1", D), norm(b + "norm2", D)
        lin(b + "attn.qkv", 3 * D, D), lin(b + "attn.proj", D, D), lin(b + "mlp.fc1", VIT["mlp"], D), lin(b + "mlp.fc2", D, VIT["mlp"])
    norm(V + "merger.ln_q", D)
    lin(V + "merger.mlp.0", 4 * D, 4 * D), lin(V + "merger.mlp.2", H, 4 * D)
    kv = TEXT["kv_heads"] * 128
    for i in range(layers):
        b = f"{L}layers.{i}."
        norm(b + "input_layernorm", H, False), norm(b + "post_attention_layernorm", H, False)
        lin(b + "self_attn.q_proj", H, H), lin(b + "self_attn.k_proj", kv, H), lin(b + "self_attn.v_proj", kv, H)
        lin(b + "self_attn.o_proj", H, H, False)
        lin(b + "mlp.gate_proj", inter, H, False), lin(b + "mlp.up_proj", inter, H, False), lin(b + "mlp.down_proj", H, inter, False)
    embed = f.w(vocab, H)
    t[L + "embed_tokens.weight"] = embed * 32
    t["lm_head.weight"] = _head(f, embed, IDS, 1.0) if vocab > IDS else f.w(vocab, H)
    norm(L + "norm", H, False)
    return t, f


def _turn_inputs(case, f):
    """Per stream: history ids, new ids, cached K/V, position offset; frames of the (one) stream that has some."""
    out = []
    for _ in range(case["streams"]):
        frames = torch.randint(0, 256, (case["frames"], 3, case["H"], case["W"]), generator=f.g, device="cuda", dtype=torch.uint8) if case["frames"] else None
        text = f.ids(case["text"], IDS)
        half = case["text"] // 2
        vid = torch.full((_video_tokens(case),), VIDEO_ID, device="cuda")
        new = torch.cat([text[:half], vid, text[half:]])
        past = case["past"]
        kv = [torch.randn((2, case["layers"], TEXT["kv_heads"], past, 128), generator=f.g, device="cuda").mul_(0.6).to(torch.bfloat16)]
        out.append(dict(frames=frames, old=f.ids(past, IDS), new=new, kv=kv[0], delta=-(past // 3)))
    return out


def _video_tokens(case):
    return (case["frames"] + 1) // 2 * (case["H"] // 28) * (case["W"] // 28) if case["frames"] else 0


def _seq_json(case):
    """config.json of a hybrid model at the sizes of the repository's own benchmark."""
    W, ff, chunk = SEQ["width"], SEQ["ff"], SEQ["chunk"]
    heads, layers = W // 128, []
    base = {"architecture": case["design"], "vocab": SEQ["vocab"], "width": W, "layers": layers}
    for i in range(case["layers"]):
        if case["design"] == "Bimopel":
            if i % 4 < 3:
                layers.append({"type": "mamba2", "mlp": None, "mixer": dict(heads=2 * W // 64, vdim=64, state=128, groups=8, conv=4, norm_groups=8)})
            else:
                layers.append({"type": "parallel", "mlp": {"ff": ff, "kind": "dense"}, "mixer": {
                    "left": dict(heads=heads, kv_heads=heads // 8, dim=128, vdim=128, mask={"size": chunk}, scale=128 ** -0.5),
                    "right": dict(heads=W // 256, dim=128, vdim=256, tau=8.0)}})
        else:
            mlp = {"kind": "dense", "ff": 3 * ff // 2 // 8 * 8} if i % 2 else {
                "kind": "moe", "expert": {"ff": ff // 4 // 8 * 8, "limit": 7.0},
                "router": {"experts": 16, "identity": 2, "top": 4, "groups": {"count": 9, "keep": 6}}}
            layers.append({"type": "attention", "mlp": mlp, "mixer": dict(
                heads=heads, kv_heads=heads // 8, dim=128, vdim=128, mask={"size": chunk}, rot={"dims": 64, "base": 250000.0}, scale=128 ** -0.5)})
    if case["design"] == "Bimopel":
        base.update(norm={"eps": 1e-5}, postln_alpha=2.0, embedding={"scale": W ** 0.5}, logit_softcap=50.0)
    else:
        base.update(norm={"eps": 1e-6}, logit_scale=0.5)
    return base


def _seq_weights(case, seed):
    f, t, cfg = _Fill(seed), {}, _seq_json(case)
    W, V = cfg["width"], cfg["vocab"]
    dyt = case["design"] == "Dibedra"

    def norm(name, n=W):
        t[name] = f.u(n, width=0.5, at=1.0)
        if dyt and n == W:
            t[name + ".b"], t[name + ".alpha"] = f.u(W, width=0.5), torch.tensor(0.75, dtype=torch.bfloat16, device="cuda")

    def mats(pre, **sizes):
        for k, (rows, cols) in sizes.items():
            t[pre + k] = f.w(rows, cols)

    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.", L["mixer"]
        norm(p + "norm1")
        if L["type"] == "mamba2":
            inner, ch = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
            mats(p + "mix.", **{"in": (inner + ch + m["heads"], W), "o": (W, inner)})
            t[p + "mix.conv"], t[p + "mix.conv.b"] = f.u(ch, m["conv"], width=1.5), f.u(ch, width=0.5)
            t[p + "mix.dt_bias"], t[p + "mix.A_log"] = f.u(m["heads"], width=4.0, at=-2.0), f.u(m["heads"], width=3.0)
            t[p + "mix.D"], t[p + "mix.norm"] = f.u(m["heads"], width=1.0, at=1.0), f.u(inner, width=0.5, at=1.0)
        elif L["type"] == "parallel":
            l, r = m["left"], m["right"]
            a, b = p + "mix.left.", p + "mix.right."
            nq, nk, rq, rv = l["heads"] * l["dim"], l["kv_heads"] * l["dim"], r["heads"] * r["dim"], r["heads"] * r["vdim"]
            mats(a, q=(nq, W), k=(nk, W), v=(nk, W), g=(l["heads"], W), o=(W, nq))
            t[a + "q.b"], t[a + "k.b"], t[a + "v.b"] = f.u(nq, width=0.5), f.u(nk, width=0.5), f.u(nk, width=0.5)
            t[a + "q.norm"], t[a + "k.norm"] = f.u(nq, width=0.5, at=1.0), f.u(nk, width=0.5, at=1.0)
            mats(b, q=(rq, W), k=(rq, W), v=(rv, W), g=(rv, W), o=(W, rv), a1=(64, W), a2=(rq, 64))
            t[b + "a2.b"], t[b + "norm"] = f.u(rq, width=4.0, at=2.0), f.u(r["vdim"], width=0.5, at=1.0)
            t[a + "out"], t[b + "out"] = f.u(W, width=0.5, at=1.0), f.u(W, width=0.5, at=1.0)
        else:
            nq, nk = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
            mats(p + "mix.", q=(nq, W), k=(nk, W), g=(nq, W), o=(W, nq))
            t[p + "mix.q.norm"], t[p + "mix.k.norm"] = f.u(m["dim"], width=0.5, at=1.0), f.u(m["dim"], width=0.5, at=1.0)
        mlp = L["mlp"]
        if mlp is None:
            continue
        if not dyt:
            norm(p + "norm2")
            mats(p + "mlp.", gate=(mlp["ff"], W), up=(mlp["ff"], W), down=(W, mlp["ff"]))
        elif mlp["kind"] == "dense":
            mats(p + "mlp.", up=(mlp["ff"], W), down=(W, mlp["ff"]))
        else:
            n, ff = 16, mlp["expert"]["ff"]
            for j in range(n):
                mats(f"{p}mlp.e{j}.", gate=(ff, W), up=(ff, W), down=(W, ff))
            mats(p + "mlp.", router=(n + 2, W))
            t[p + "mlp.correction"] = f.u(n + 2, width=0.1)
    norm("final.norm")
    embed = f.u(V, W, width=3.4641)
    t["embed"] = embed * 4 if dyt else embed
    t["head"] = _head(f, embed, V, W ** -0.5)
    return cfg, t, f


# ------------------------------------------------------------------------------------------------ what a program holds, and one pass
def _livecc_model(case, seed, **text):
    from livecc_b200.config import LiveCCConfig, TextConfig, VisionConfig
    from livecc_b200.engine import LiveCCB200ForConditionalGeneration

    t, f = _livecc(seed, case["depth"], case.get("layers", 1), **text)
    names = {"vocab": "vocab_size", "inter": "intermediate_size"}
    cfg = LiveCCConfig(text_config=TextConfig(num_hidden_layers=case.get("layers", 1), **{names[k]: v for k, v in text.items()}),
                       vision_config=VisionConfig(depth=case["depth"]))
    m = LiveCCB200ForConditionalGeneration.from_state_dict(cfg, t)
    m.generation_config.eos_token_id = -1      # random weights: no turn ends early
    return m, f


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ingest":
        from livecc_b200._cabi import Context

        ctx = Context(0)
        ctx.resize_plan(case["h"], case["w"], case["H"], case["W"])
        return dict(case=case, ctx=ctx, clip=_clip(case, seed))
    if kind == "vision":
        m, f = _livecc_model(case, seed, vocab=2048, inter=4864)
        return dict(case=case, model=m, frames=_frames(case, f))
    if kind == "turn":
        m, f = _livecc_model(case, seed)
        streams = []
        for s in _turn_inputs(case, f):
            c = m.new_cache()
            c.ensure_tokens(case["past"] + s["new"].numel() + case["new"])
            streams.append((c, s))
        m.pool.k.zero_(), m.pool.v.zero_()
        for c, s in streams:
            n = case["past"]
            if n:
                full = len(c.pages) * 64
                kv = torch.zeros((2, case["layers"], TEXT["kv_heads"], full, 128), dtype=torch.bfloat16, device="cuda")
                kv[:, :, :, :n] = s.pop("kv")
                kv = kv.view(2, case["layers"], TEXT["kv_heads"], len(c.pages), 64, 128).transpose(2, 3)
                at = torch.tensor(c.pages, device="cuda")
                m.pool.k[:, at], m.pool.v[:, at] = kv[0], kv[1]
                c.rope_delta = s["delta"]
            s["ids"] = torch.cat([s["old"], s["new"]]).view(1, -1)
        return dict(case=case, model=m, streams=streams)
    from livecc_b200.config import SeqModelConfig
    from livecc_b200.seq_engine import SeqLMForCausalLM

    cfg, t, f = _seq_weights(case, seed)
    m = SeqLMForCausalLM.from_state_dict(SeqModelConfig.from_json(cfg), t, "bfloat16", max_tokens=case["tokens"] + case.get("new", 0) + 64)
    ids = f.ids(case["tokens"], SEQ["vocab"]).cpu()
    return dict(case=case, model=m, ids=ids.view(1, -1) if case["kind"] == "gen" else ids.tolist())


def _clip(case, seed):
    f = _Fill(seed)      # a smooth picture with noise on it
    low = torch.rand((case["frames"], 3, 12, 20), generator=f.g, device="cuda") * 255
    big = F.interpolate(low, size=(case["h"], case["w"]), mode="bilinear")
    return (big + torch.randn(big.shape, generator=f.g, device="cuda") * 12).clamp(0, 255).to(torch.uint8)


def _frames(case, f):
    return torch.randint(0, 256, (case["frames"], 3, case["H"], case["W"]), generator=f.g, device="cuda", dtype=torch.uint8)


def _want(case):
    return list(range(case["tokens"] - 1, -1, -16))[::-1]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ingest":
        return state["ctx"].resize_bicubic_aa_u8(state["clip"], (case["H"], case["W"]))
    m = state["model"]
    if kind == "vision":
        return m.get_video_features_from_frames(state["frames"])
    if kind == "prompt":     # teacher-forced scoring of chosen places
        cache = m.new_cache()
        logits = m.forward_step([(cache, state["ids"])], [_want(case)])
        cache.release()
        return logits
    if kind == "gen":
        out = m.generate(state["ids"], max_new_tokens=case["new"], eos_token_id=-1, output_logits=True)
        out.past_key_values.release()
        return {"ids": out.sequences[:, case["tokens"]:], "logits": out.logits}
    past, how = case["past"], dict(repetition_penalty=1.05, max_new_tokens=case["new"], output_logits=True)
    for c, s in state["streams"]:
        c.seq_len = past                    # the turn is taken again from the same place
        c.rope_delta = s["delta"] if past else None
    rq = [dict(input_ids=s["ids"], past_key_values=c, **({"video_frames": s["frames"]} if s["frames"] is not None else {})) for c, s in state["streams"]]
    outs = m.generate_batch(rq, **how) if case["streams"] > 1 else [m.generate(**rq[0], **how)]
    n = state["streams"][0][1]["ids"].shape[1]
    res = []
    for o, (c, s) in zip(outs, state["streams"]):
        a, b = c.pages[past // 64], c.pages[len(c.pages) - 1] + 1     # a stream's pages lie behind one another in this pool
        res.append({"ids": o.sequences[:, n:], "logits": torch.stack(o.logits) if case["streams"] > 1 else o.logits,
                    "k": m.pool.k[:, a:b], "v": m.pool.v[:, a:b]})
    return res


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "ingest":
        src, dst = 3 * case["frames"] * case["h"] * case["w"], 3 * case["frames"] * case["H"] * case["W"]
        taps = lambda a, b: 4 * max(1.0, a / b)
        return {"bytes": src + dst, "flops": 2 * 3 * case["frames"] * (case["h"] * case["W"] * taps(case["w"], case["W"]) + case["H"] * case["W"] * taps(case["h"], case["H"]))}
    if kind == "vision":
        b, fl = _vision_work(case)
        return {"bytes": b, "flops": fl}
    if kind == "turn":
        H, I, B = TEXT["hidden"], TEXT["inter"], case["streams"]
        per_layer = H * (H + 2 * TEXT["kv_heads"] * 128) + H * H + 3 * H * I
        head = H * TEXT["vocab"]
        S, past, steps = case["text"] + _video_tokens(case), case["past"], case["new"] - 1
        kv_tok = 2 * TEXT["kv_heads"] * 128 * 2 * case["layers"]
        att = lambda rows, keys: 4 * rows * keys * TEXT["q_heads"] * 128 * case["layers"]
        by, fl = _vision_work(case) if case["frames"] else (0, 0)
        weights = 2 * (per_layer * case["layers"] + head)
        by += (1 + steps) * weights                       # every stream's new tokens could share one pass, and each step does
        by += B * (kv_tok * (past + S) + 4 * TEXT["vocab"]) + B * steps * (kv_tok * (past + S + steps / 2) + 4 * TEXT["vocab"])
        fl += 2 * B * (S * per_layer * case["layers"] + head) + B * att(S, past + S / 2)
        fl += B * steps * (2 * (per_layer * case["layers"] + head) + att(1, past + S + steps / 2))
        return {"bytes": by, "flops": fl}
    W, V, ff = SEQ["width"], SEQ["vocab"], SEQ["ff"]
    n, T, steps = case["layers"], case["tokens"], max(case.get("new", 1) - 1, 0)
    rows = len(_want(case)) if kind == "prompt" else 1
    if case["design"] == "Bimopel":
        inner, st = 2 * W, 2 * W // 64 * 64 * 128
        ssd, par = W * (3 * inner + 2 * 8 * 128 + 2 * W // 64), W * (W * 2 + W // 4 + W // 128 + W + W + 64 + W) + 64 * W // 2 + 3 * W * ff
        params = sum(ssd if i % 4 < 3 else par for i in range(n))
        active, mix = params, sum(6 * st if i % 4 < 3 else 4 * min(T, 1024) / 2 * W + 6 * W * 128 for i in range(n))
        state = 4 * sum(st if i % 4 < 3 else W * 128 for i in range(n))
    else:
        att, dense, moe = W * (3 * W + W // 8), 2 * W * (3 * ff // 2), 3 * W * (ff // 4 // 8 * 8)
        params = sum(att + (dense if i % 2 else 16 * moe) for i in range(n))
        active = sum(att + (dense if i % 2 else 4 * moe) for i in range(n))
        mix, state = 4 * min(T, 1024) * W * n, 0
    read = lambda t: 2 * (min(params, active * t) + V * W)      # a routed step reads the experts its rows chose
    by = read(T) + 4 * rows * V + steps * (read(1) + 2 * state + 4 * V)
    fl = 2 * (T * active + rows * V * W) + T * mix + steps * (2 * (active + V * W) + mix)
    return {"bytes": by, "flops": fl}


def _vision_work(case):
    t, D = (case["frames"] + 1) // 2, VIT["dim"]
    per = (case["H"] // 14) * (case["W"] // 14)
    N = t * per
    block, ends = D * 3 * D + D * D + 2 * D * VIT["mlp"], (4 * D) ** 2 + 4 * D * TEXT["hidden"]
    fl = 2 * N * (1176 * D + block * case["depth"]) + 2 * N / 4 * ends + 4 * N * per * D * case["depth"]
    by = 2 * (1176 * D + block * case["depth"] + ends) + 3 * case["frames"] * case["H"] * case["W"] + 2 * N / 4 * TEXT["hidden"]
    return by, fl


def tolerance(case):
    """About four times what the path was measured off `exact` by (2-norm): 0.007 in the vision tower, 0.011 in a turn's logits, 0.005
    and 0.002 in the two hybrid designs; a turn's is held at 0.03."""
    kind = case["kind"]
    if kind == "ingest":
        return "exact"
    return {"rel": {"vision": 0.025, "turn": 0.03}.get(kind) or (0.02 if case["design"] == "Bimopel" else 0.01), "max": 0.4}


# ------------------------------------------------------------------------------------------------ the same in float64
def _rms(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _turn_half(x, c, s):
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _exact_vision(t, frames, depth):
    w = lambda n: t["model.visual." + n].to(F64)
    D, heads, hd = VIT["dim"], VIT["heads"], VIT["dim"] // VIT["heads"]
    x = frames.to(F64) / 255
    x = (x - torch.tensor(MEAN, dtype=F64, device="cuda").view(1, 3, 1, 1)) / torch.tensor(STD, dtype=F64, device="cuda").view(1, 3, 1, 1)
    if x.shape[0] % 2:
        x = torch.cat([x, x[-1:]])
    T, h, wd = x.shape[0] // 2, x.shape[2] // 14, x.shape[3] // 14
    # rows in windows of 2 x 2 patches, a row = [channel, frame of the pair, y, x]
    x = x.view(T, 2, 3, h // 2, 2, 14, wd // 2, 2, 14).permute(0, 3, 6, 4, 7, 2, 1, 5, 8).reshape(T * h * wd, 1176)
    x = x @ w("patch_embed.proj.weight").view(D, 1176).T
    win = lambda g: g.view(h // 2, 2, wd // 2, 2).permute(0, 2, 1, 3).flatten()
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(wd, device="cuda"), indexing="ij")
    freq = 10000.0 ** (-torch.arange(0, hd // 2, 2, dtype=F64, device="cuda") / (hd // 2))
    ang = torch.cat([win(yy)[:, None] * freq, win(xx)[:, None] * freq], -1).repeat(T, 1)[:, None]
    c, s = ang.cos(), ang.sin()
    ln = lambda v, n: F.layer_norm(v, (D,), w(n + ".weight"), w(n + ".bias"), 1e-6)
    lin = lambda v, n: v @ w(n + ".weight").T + w(n + ".bias")
    for i in range(depth):
        b = f"blocks.{i}."
        q, k, v = lin(ln(x, b + "norm1"), b + "attn.qkv").view(-1, 3, heads, hd).unbind(1)
        q, k = _turn_half(q, c, s), _turn_half(k, c, s)
        out = []
        for j in range(T):        # a frame pair attends to itself
            r = slice(j * h * wd, (j + 1) * h * wd)
            p = torch.softmax(q[r].transpose(0, 1) @ k[r].permute(1, 2, 0) * hd ** -0.5, -1)
            out.append((p @ v[r].transpose(0, 1)).transpose(0, 1).reshape(-1, D))
        x = x + lin(torch.cat(out), b + "attn.proj")
        z = lin(ln(x, b + "norm2"), b + "mlp.fc1")
        x = x + lin(z * torch.sigmoid(1.702 * z), b + "mlp.fc2")
    x = ln(x, "merger.ln_q").view(-1, 4 * D)
    return lin(F.gelu(lin(x, "merger.mlp.0")), "merger.mlp.2")


def _positions(case, n, past, delta):
    """[3, n] positions of the new tokens: behind a past all three run on; an opening turn's video rows span its grid."""
    if past:
        return (torch.arange(n) + past + delta).expand(3, -1)
    if not case["frames"]:
        return torch.arange(n).expand(3, -1)
    a, vt = case["text"] // 2, _video_tokens(case)
    h, w = case["H"] // 28, case["W"] // 28
    y, x = torch.arange(h).repeat_interleave(w).repeat(vt // (h * w)), torch.arange(w).repeat(vt // w)
    after = a + max(h, w) + torch.arange(case["text"] - a)
    head = torch.arange(a)
    pos = torch.stack([torch.cat([head, torch.full((vt,), a), after]), torch.cat([head, a + y, after]), torch.cat([head, a + x, after])])
    more = int(pos.max()) + 1 + torch.arange(n - pos.shape[1])
    return torch.cat([pos, more.expand(3, -1)], 1)


def _exact_turn(case, t, s, weights):
    """Logits of the last prompt token and of every generated one but the last (the ids follow the head's preference)."""
    L, H, G, Q = "model.language_model.", TEXT["hidden"], TEXT["kv_heads"], TEXT["q_heads"]
    ids = s["new"].tolist()
    chain = _chain(ids[-1], case["new"], IDS)
    seq = torch.tensor(ids + chain[:-1], device="cuda")
    x = t[L + "embed_tokens.weight"][seq].to(F64)
    if s["frames"] is not None:
        x[seq == VIDEO_ID] = _exact_vision(t, s["frames"], case["depth"])
    n, past = seq.numel(), case["past"]
    pos = _positions(case, n, past, s["delta"]).to("cuda", F64)
    freq = TEXT["theta"] ** (-torch.arange(0, 128, 2, dtype=F64, device="cuda") / 128)
    part = torch.repeat_interleave(torch.arange(3, device="cuda"), torch.tensor([16, 24, 24], device="cuda"))
    ang = pos[part].T * freq
    c, si = ang.cos(), ang.sin()
    see = torch.arange(past + n, device="cuda")[None, :] <= past + torch.arange(n, device="cuda")[:, None]
    for i in range(case["layers"]):
        b = f"{L}layers.{i}."
        w = lambda name: weights(b + name)
        h = _rms(x, TEXT["eps"]) * w("input_layernorm.weight")
        q, k, v = ((h @ w(f"self_attn.{p}_proj.weight").T + w(f"self_attn.{p}_proj.bias")).view(n, -1, 128).transpose(0, 1) for p in "qkv")
        q, k = _turn_half(q, c, si), _turn_half(k, c, si)
        k, v = torch.cat([s["kv"][0, i].to(F64), k], 1), torch.cat([s["kv"][1, i].to(F64), v], 1)
        o = torch.empty((Q, n, 128), dtype=F64, device="cuda")
        for j in range(Q):
            p = (q[j] @ k[j // (Q // G)].T * 128 ** -0.5).masked_fill_(~see, -math.inf)
            o[j] = torch.softmax(p, -1) @ v[j // (Q // G)]
        x = x + o.transpose(0, 1).reshape(n, H) @ w("self_attn.o_proj.weight").T
        h = _rms(x, TEXT["eps"]) * w("post_attention_layernorm.weight")
        x = x + (F.silu(h @ w("mlp.gate_proj.weight").T) * (h @ w("mlp.up_proj.weight").T)) @ w("mlp.down_proj.weight").T
    x = _rms(x[len(ids) - 1:], TEXT["eps"]) * weights(L + "norm.weight")
    head = t["lm_head.weight"]
    logits = torch.cat([x @ head[r:r + 16384].to(F64).T for r in range(0, head.shape[0], 16384)], 1)
    return chain, logits


def exact(case, seed):
    kind = case["kind"]
    with torch.inference_mode():
        if kind == "ingest":
            return F.interpolate(_clip(case, seed).to(F64), size=(case["H"], case["W"]), mode="bicubic", antialias=True).clamp(0, 255).round().to(torch.uint8)
        if kind == "vision":
            t, f = _livecc(seed, case["depth"], 1, vocab=2048, inter=4864)
            return _exact_vision(t, _frames(case, f), case["depth"])
        if kind == "turn":
            t, f = _livecc(seed, case["depth"], case["layers"])
            streams, kept = _turn_inputs(case, f), {}

            def weights(name):
                if name not in kept:
                    kept[name] = t[name].to(F64)
                return kept[name]

            out = []
            for s in streams:
                chain, logits = _exact_turn(case, t, s, weights)
                out.append({"ids": torch.tensor([chain]), "logits": logits if case["streams"] > 1 else list(logits), "k": None, "v": None})
            return out
        cfg, t, f = _seq_weights(case, seed)
        ids = f.ids(case["tokens"], SEQ["vocab"]).tolist()
        if kind == "prompt":
            return _exact_seq(cfg, t, ids, _want(case))
        chain = _chain(ids[-1], case["new"], SEQ["vocab"])
        seq = ids + chain[:-1]
        logits = _exact_seq(cfg, t, seq, list(range(len(ids) - 1, len(seq))))
        return {"ids": torch.tensor([chain]), "logits": list(logits)}


def _exact_seq(cfg, t, ids, want):
    w = lambda n: t[n].to(F64)
    T, W, eps = len(ids), cfg["width"], cfg["norm"]["eps"]
    x = w("embed")[torch.tensor(ids, device="cuda")]
    pos = torch.arange(T, dtype=F64, device="cuda")
    gelu = lambda z: F.gelu(z, approximate="tanh")
    if cfg["architecture"] == "Bimopel":
        ang = pos[:, None] * 10000.0 ** (-torch.arange(0, W, 2, dtype=F64, device="cuda") / W)
        x = x * cfg["embedding"]["scale"] + torch.stack([ang.sin(), ang.cos()], -1).reshape(T, W)
        for i, L in enumerate(cfg["layers"]):
            p = f"l{i}."
            y = _exact_ssd(x, w, p + "mix.", L["mixer"], eps) if L["type"] == "mamba2" else _exact_parallel(x, w, p + "mix.", L["mixer"], eps)
            x = _rms(cfg["postln_alpha"] * x + y, eps) * w(p + "norm1")
            if L["mlp"]:
                y = (gelu(x @ w(p + "mlp.gate").T) * (x @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
                x = _rms(cfg["postln_alpha"] * x + y, eps) * w(p + "norm2")
        x = _rms(x, eps) * w("final.norm")
        cap = cfg["logit_softcap"]
        return cap * torch.tanh(x[want] @ w("head").T / cap)
    dyt = lambda v, n: torch.tanh(w(n + ".alpha") * v) * w(n) + w(n + ".b")
    for i, L in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", L["mixer"], L["mlp"]
        h = dyt(x, p + "norm1")
        y = _exact_window(h, w, p + "mix.", m, eps, pos)
        if mlp["kind"] == "dense":
            y = y + gelu(h @ w(p + "mlp.up").T) @ w(p + "mlp.down").T
        else:
            score = torch.softmax(h @ w(p + "mlp.router").T, -1)
            choice = score + w(p + "mlp.correction")
            gr, n = mlp["router"]["groups"], score.shape[1]
            best = choice.view(T, gr["count"], -1).amax(-1).topk(gr["keep"], -1).indices
            open_ = torch.zeros((T, gr["count"]), dtype=torch.bool, device="cuda").scatter_(1, best, True)
            choice = choice.masked_fill(~open_.repeat_interleave(n // gr["count"], 1), -math.inf)
            top = choice.topk(mlp["router"]["top"], -1).indices
            share = torch.zeros_like(score).scatter_(1, top, score.gather(1, top))
            lim = mlp["expert"]["limit"]
            for j in range(16):
                rows = share[:, j].nonzero().flatten()
                g = (h[rows] @ w(f"{p}mlp.e{j}.gate").T).clamp(max=lim)
                u = (h[rows] @ w(f"{p}mlp.e{j}.up").T).clamp(-lim, lim)
                y[rows] += share[rows, j:j + 1] * ((g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(f"{p}mlp.e{j}.down").T)
            y = y + share[:, 16:].sum(1, keepdim=True) * h
        x = x + y
    return dyt(x, "final.norm")[want] @ w("head").T * cfg["logit_scale"]


def _attend(q, k, v, scale, see, sink):
    """q [T, H, d], k and v [T, G, d]: softmax over the keys that `see` [T, T] leaves, with a zero-logit sink where asked."""
    out = torch.empty_like(q)
    per = q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        e = (q[:, h] @ k[:, h // per].T * scale).masked_fill_(~see, -math.inf)
        if sink:
            e = torch.cat([e, torch.zeros_like(e[:, :1])], 1)
        p = torch.softmax(e, -1)
        out[:, h] = (p[:, :-1] if sink else p) @ v[:, h // per]
    return out


def _exact_window(h, w, p, m, eps, pos):
    T, d, dims = h.shape[0], m["dim"], m["rot"]["dims"]
    q, k = (h @ w(p + "q").T).view(T, -1, d), (h @ w(p + "k").T).view(T, -1, d)
    v = k
    ang = (pos[:, None] * m["rot"]["base"] ** (-torch.arange(0, dims, 2, dtype=F64, device="cuda") / dims))[:, None]
    c, s = ang.cos(), ang.sin()

    def turn(x, n):
        x = _rms(x, eps) * w(n)
        a, b = x[..., 0:dims:2], x[..., 1:dims:2]
        return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), x[..., dims:]], -1)

    back = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    o = _attend(turn(q, p + "q.norm"), turn(k, p + "k.norm"), v, m["scale"], (back >= 0) & (back < m["mask"]["size"]), False)
    return (o.reshape(T, -1) * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T


def _exact_ssd(x, w, p, m, eps):
    T, H, P, G, N = x.shape[0], m["heads"], m["vdim"], m["groups"], m["state"]
    inner = H * P
    proj = x @ w(p + "in").T
    z, xbc, dt = proj[:, :inner], proj[:, inner:-H], F.softplus(proj[:, -H:] + w(p + "dt_bias"), threshold=1e9)
    xbc = F.conv1d(F.pad(xbc.T[None], (m["conv"] - 1, 0)), w(p + "conv")[:, None], w(p + "conv.b"), groups=xbc.shape[1])[0].T
    xs, B, C = torch.split(F.silu(xbc), [inner, G * N, G * N], -1)
    xs = xs.reshape(T, H, P)
    B, C = (u.reshape(T, G, N).repeat_interleave(H // G, 1) for u in (B, C))
    keep, S, y = torch.exp(-torch.exp(w(p + "A_log")) * dt), torch.zeros((H, N, P), dtype=F64, device="cuda"), torch.empty_like(xs)
    for i in range(T):
        S = keep[i, :, None, None] * S + (dt[i, :, None] * B[i])[:, :, None] * xs[i][:, None]
        y[i] = (C[i][:, None] @ S)[:, 0]
    y = (y + w(p + "D")[:, None] * xs).reshape(T, inner) * F.silu(z)
    return (_rms(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * w(p + "norm")) @ w(p + "o").T


def _exact_parallel(x, w, p, m, eps):
    T, l, r = x.shape[0], m["left"], m["right"]
    a, b = p + "left.", p + "right."
    q, k, v = (x @ w(a + n).T + w(a + n + ".b") for n in "qkv")
    q, k = _rms(q, eps) * w(a + "q.norm"), _rms(k, eps) * w(a + "k.norm")
    i = torch.arange(T, device="cuda")
    see = (i[None] <= i[:, None]) & (i[None] // l["mask"]["size"] == i[:, None] // l["mask"]["size"])
    o = _attend(*(u.reshape(T, -1, l["dim"]) for u in (q, k, v)), l["scale"], see, True) * torch.sigmoid(x @ w(a + "g").T)[:, :, None]
    left = o.reshape(T, -1) @ w(a + "o").T
    H, d, dv = r["heads"], r["dim"], r["vdim"]
    q, k, v = (x @ w(b + "q").T).view(T, H, d) * d ** -0.5, (x @ w(b + "k").T).view(T, H, d), (x @ w(b + "v").T).view(T, H, dv)
    keep = torch.sigmoid((x @ w(b + "a1").T) @ w(b + "a2").T + w(b + "a2.b")).pow(1 / r["tau"]).view(T, H, d)
    S, y = torch.zeros((H, d, dv), dtype=F64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        S = keep[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
        y[t] = (q[t][:, None] @ S)[:, 0]
    right = ((_rms(y, eps) * w(b + "norm")).reshape(T, -1) * F.silu(x @ w(b + "g").T)) @ w(b + "o").T
    return 0.5 * (_rms(left, eps) * w(a + "out") + _rms(right, eps) * w(b + "out"))
