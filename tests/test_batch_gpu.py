"""Several streams in one pass (prefill, decode steps, lm_head of each stream's last row): prompts have the bits of a pass of their own (cache and
first logits), decode steps have the same bits whoever the neighbours are and in whichever place a stream stands; against the one-stream
decode kernels logits and caches agree within the rounding of the storage type. Ids are the selection that each stream's own logits and history
give. Streams that end early leave the others alone."""
import pytest
import torch

from livecc_b200.checkpoint import synthetic_state_dict
from livecc_b200.config import LiveCCConfig, TextConfig, VisionConfig

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def engines():
    from livecc_b200.engine import LiveCCB200ForConditionalGeneration

    cfgs = {"small": LiveCCConfig.small(),
            "wide": LiveCCConfig(text_config=TextConfig(num_hidden_layers=2), vision_config=VisionConfig(depth=1), name="wide-l2")}
    out = {}
    for name, cfg in cfgs.items():
        sd = synthetic_state_dict(cfg, dtype=torch.bfloat16, device=DEV, gen_device=DEV)
        out[name] = LiveCCB200ForConditionalGeneration.from_state_dict(cfg, sd, DEV)
        out[name].generation_config.eos_token_id = -1
    return out


def _requests(eng, spec, seed):
    """spec: per stream (past tokens, new text ids, frames). The past is prefilled by a call of its own, alike for both arms."""
    g = torch.Generator().manual_seed(seed)
    below = min(eng.config.text_config.vocab_size, eng.config.video_token_id) - 16
    reqs = []
    for past, new, frames in spec:
        ids = torch.randint(0, below, (1, past + new), generator=g)
        vid = None
        if frames:
            vid = torch.randint(0, 256, (frames, 3, 56, 84), generator=g, dtype=torch.uint8).to(DEV)
            pads = torch.full((1, (frames + 1) // 2 * 2 * 3), eng.config.video_token_id)
            ids = torch.cat([ids[:, :past + 1], pads, ids[:, past + 1:]], 1)
        reqs.append((ids, past, vid))
    return reqs


def _caches(eng, reqs):
    res = []
    for ids, past, _ in reqs:
        res.append(eng.generate(input_ids=ids[:, :past].to(DEV), max_new_tokens=1).past_key_values if past else None)
    return res


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


# Each arm is the float64 result plus 0.4 % (small) to 1 % (wide) of rounding in bf16 activations: two independent ones differ by sqrt(2) of that.
TOL = 0.02


def _check_ids(out, n, penalty):
    """Every id is the best of its own logits, those of ids that the stream has seen divided (or multiplied, if negative) by the penalty."""
    ids = out.sequences[0]
    for i, lg in enumerate(out.logits):
        seen = ids[:n + i].unique()
        lg = lg.clone()
        lg[seen] = torch.where(lg[seen] < 0, lg[seen] * penalty, lg[seen] / penalty)
        best = lg.max()
        assert lg[ids[n + i]] >= best - 1e-6 * best.abs(), (i, int(ids[n + i]), int(lg.argmax()))


@pytest.mark.parametrize("which,spec", [
    ("small", [(0, 1, 0), (0, 2, 0)]),                                                       # single new rows
    ("small", [(63, 5, 0), (64, 1, 0), (65, 17, 2)]),                                        # edges of a page, one stream with frames
    ("small", [(0, 9, 2), (130, 3, 0), (1, 1, 0), (64, 64, 0), (200, 2, 2), (0, 300, 0), (40, 18, 6), (7, 11, 0)]),
    ("wide", [(700, 24, 0), (0, 40, 2)]),
    ("wide", [(300, 24, 0), (512, 1, 0), (0, 33, 0), (90, 19, 2), (1000, 5, 0)]),
    ("small", [(30, 1200, 0), (0, 900, 2), (5, 30, 0)]),                                     # more rows than one pass takes
    ("wide", [(300, 281, 0), (0, 281, 0), (40, 200, 0), (0, 330, 0), (10, 150, 0)]),         # K cut alike, more rows than a wave of clusters takes
    ("wide", [(16384, 64, 0)] * 7 + [(12932, 50, 0)]),     # attention in two groups that share the partials' scratch; the second has an empty key range
])
def test_streams_together_match_streams_alone(engines, which, spec):
    eng, new = engines[which], 5
    reqs = _requests(eng, spec, seed=len(spec))
    how = dict(repetition_penalty=1.05, max_new_tokens=new, output_logits=True)
    alone = [eng.generate(input_ids=ids.to(DEV), past_key_values=c, **({"video_frames": v} if v is not None else {}), **how)
             for (ids, _, v), c in zip(reqs, _caches(eng, reqs))]
    kv_alone = [[tuple(x.clone() for x in o.past_key_values.gather(l)) for l in range(eng.config.text_config.num_hidden_layers)] for o in alone]
    together = eng.generate_batch([dict(input_ids=ids.to(DEV), past_key_values=c, **({"video_frames": v} if v is not None else {}))
                                   for (ids, _, v), c in zip(reqs, _caches(eng, reqs))], **how)
    for b, (a, t, (ids, _, _)) in enumerate(zip(alone, together, reqs)):
        n = ids.shape[1]
        assert t.past_key_values.get_seq_length() == a.past_key_values.get_seq_length() == n + new - 1
        _check_ids(a, n, 1.05)
        _check_ids(t, n, 1.05)
        assert torch.equal(t.logits[0], a.logits[0]), b            # the prompt's pass: the bits of the stream alone
        same = new
        for i in range(new):
            assert _rel(t.logits[i], a.logits[i]) < TOL, (b, i)
            if t.sequences[0, n + i] != a.sequences[0, n + i]:     # (each arm has selected by its own logits: from here on they go apart)
                same = i
                break
        m = n + min(same, new - 1)
        for l, (k, v) in enumerate(kv_alone[b]):
            tk, tv = t.past_key_values.gather(l)
            assert torch.equal(tk[..., :n, :], k[..., :n, :]) and torch.equal(tv[..., :n, :], v[..., :n, :]), (b, l)
            assert _rel(tk[..., :m, :], k[..., :m, :]) < TOL and _rel(tv[..., :m, :], v[..., :m, :]) < TOL, (b, l)
        a.past_key_values.release()
        t.past_key_values.release()


@pytest.mark.parametrize("which,spec,penalty", [
    ("small", [(0, 9, 2), (130, 3, 0), (1, 1, 0), (64, 64, 0), (200, 2, 2), (0, 300, 0), (40, 18, 6), (7, 11, 0)], 1.6),
    ("wide", [(4200, 40, 0), (90, 19, 2), (16500, 7, 0), (700, 400, 0), (16300, 90, 0)], 1.05),    # 1, 2 and more key ranges; both sides of the bound
])
def test_a_streams_bits_do_not_depend_on_its_neighbours(engines, which, spec, penalty):
    eng, new = engines[which], 6
    reqs = _requests(eng, spec, seed=len(spec))
    def together(of):
        outs = eng.generate_batch([dict(input_ids=reqs[b][0].to(DEV), past_key_values=c, **({"video_frames": reqs[b][2]} if reqs[b][2] is not None else {}))
                                   for b, c in zip(of, _caches(eng, [reqs[b] for b in of]))], repetition_penalty=penalty, max_new_tokens=new, output_logits=True)
        res = {}
        for b, o in zip(of, outs):
            _check_ids(o, reqs[b][0].shape[1], penalty)
            res[b] = (o.sequences.clone(), torch.stack(o.logits), [tuple(x.clone() for x in o.past_key_values.gather(l)) for l in range(eng.config.text_config.num_hidden_layers)])
            o.past_key_values.release()
        return res

    every = list(range(len(spec)))
    full = together(every)
    for of in ([0, 1], every[::-1], [4, 2, 3], [3, 4]):
        for b, (seq, logits, kv) in together(of).items():
            assert torch.equal(seq, full[b][0]) and torch.equal(logits, full[b][1]), (of, b)
            for l, (k, v) in enumerate(kv):
                assert torch.equal(k, full[b][2][l][0]) and torch.equal(v, full[b][2][l][1]), (of, b, l)


def test_a_stream_that_ends_leaves_the_others_alone(engines):
    eng = engines["small"]
    reqs = _requests(eng, [(20, 4, 0), (70, 3, 0), (0, 12, 0)], seed=5)
    call = lambda: eng.generate_batch([dict(input_ids=ids.to(DEV), past_key_values=c) for (ids, _, _), c in zip(reqs, _caches(eng, reqs))],
                                      max_new_tokens=8, output_logits=True)
    full = call()
    n = reqs[1][0].shape[1]
    eos = int(full[1].sequences[0, n + 2])
    eng.generation_config.eos_token_id = eos
    try:
        cut = call()
    finally:
        eng.generation_config.eos_token_id = -1
    for b, (f, c, (ids, _, _)) in enumerate(zip(full, cut, reqs)):
        gen = f.sequences[0, ids.shape[1]:].tolist()
        want = gen[:gen.index(eos) + 1] if eos in gen else gen
        assert c.sequences[0, ids.shape[1]:].tolist() == want
        assert c.past_key_values.get_seq_length() == ids.shape[1] + len(want) - 1
        for x, y in zip(c.logits, f.logits):
            assert torch.equal(x, y)
        k0, k1 = f.past_key_values.gather(0)[0], c.past_key_values.gather(0)[0]
        assert torch.equal(k1, k0[..., :k1.shape[-2], :])
        f.past_key_values.release()
        c.past_key_values.release()


def test_one_token_each_of_a_model_that_batched_decoding_refuses():
    """Prefill of several streams asks for no more than prefill of one; decode steps of several streams need widths of 256."""
    from livecc_b200._cabi import LiveCCNativeError
    from livecc_b200.engine import LiveCCB200ForConditionalGeneration

    cfg = LiveCCConfig(text_config=TextConfig(hidden_size=384, intermediate_size=1056, num_hidden_layers=2, num_attention_heads=3, num_key_value_heads=1),
                       vision_config=VisionConfig(depth=1, embed_dim=320, hidden_size=384, num_heads=4), name="odd").with_vocab(4104)
    sd = synthetic_state_dict(cfg, dtype=torch.bfloat16, device=DEV, gen_device=DEV)
    eng = LiveCCB200ForConditionalGeneration.from_state_dict(cfg, sd, DEV)
    reqs = _requests(eng, [(0, 9, 2), (70, 3, 0), (0, 140, 0)], seed=3)
    call = lambda new: eng.generate_batch([dict(input_ids=ids.to(DEV), **({"video_frames": v} if v is not None else {})) for ids, _, v in reqs],
                                          max_new_tokens=new, output_logits=True)
    for t, (ids, _, v) in zip(call(1), reqs):
        a = eng.generate(input_ids=ids.to(DEV), max_new_tokens=1, output_logits=True, **({"video_frames": v} if v is not None else {}))
        assert torch.equal(t.logits[0], a.logits[0]) and torch.equal(t.sequences, a.sequences)
    with pytest.raises(LiveCCNativeError, match="batched decoding"):
        call(2)


def test_prompts_of_several_streams_through_the_mma_attention(engines, monkeypatch):
    """LIVECC_B200_PREFILL_ATTN=mma: the mma.sync kernel takes each stream of a joint pass by itself, with the bits of the stream alone."""
    monkeypatch.setenv("LIVECC_B200_PREFILL_ATTN", "mma")
    for which, spec in (("small", [(130, 3, 0), (0, 40, 2), (200, 17, 0)]), ("wide", [(2100, 40, 0), (64, 1, 0), (0, 200, 0)])):
        eng = engines[which]
        reqs = _requests(eng, spec, seed=8)
        kw = [dict(input_ids=ids.to(DEV), **({"video_frames": v} if v is not None else {})) for ids, _, v in reqs]
        alone = [eng.generate(past_key_values=c, max_new_tokens=1, output_logits=True, **k) for k, c in zip(kw, _caches(eng, reqs))]
        together = eng.generate_batch([dict(k, past_key_values=c) for k, c in zip(kw, _caches(eng, reqs))], max_new_tokens=1, output_logits=True)
        for a, t in zip(alone, together):
            assert torch.equal(t.logits[0], a.logits[0]) and torch.equal(t.sequences, a.sequences)
            a.past_key_values.release()
            t.past_key_values.release()
