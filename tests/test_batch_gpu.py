"""Several streams in one pass (prefill, decode steps, lm_head of each stream's last row) against the same streams taken one by one through
the one-stream kernels: logits within the rounding of the storage type, ids the same unless the best two logits are that close, caches equal
in length and content within the same rounding; streams that end early leave the others alone."""
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


@pytest.mark.parametrize("which,spec", [
    ("small", [(0, 1, 0), (0, 2, 0)]),                                                       # single new rows
    ("small", [(63, 5, 0), (64, 1, 0), (65, 17, 2)]),                                        # edges of a page, one stream with frames
    ("small", [(0, 9, 2), (130, 3, 0), (1, 1, 0), (64, 64, 0), (200, 2, 2), (0, 300, 0), (40, 18, 6), (7, 11, 0)]),
    ("wide", [(700, 24, 0), (0, 40, 2)]),
    ("wide", [(300, 24, 0), (512, 1, 0), (0, 33, 0), (90, 19, 2), (1000, 5, 0)]),
    ("small", [(30, 1200, 0), (0, 900, 2), (5, 30, 0)]),                                     # more rows than one pass takes
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
        same = True
        for i in range(new):
            if not same:
                break
            assert _rel(t.logits[i], a.logits[i]) < TOL, (b, i)
            x, y = int(t.sequences[0, n + i]), int(a.sequences[0, n + i])
            if x != y:   # only where the best two are within both arms' rounding
                same = False
                assert abs(a.logits[i][x] - a.logits[i][y]) < 0.06 * max(1.0, a.logits[i].abs().max().item()), (b, i)
        m = n if not same else n + new - 1
        for l, (k, v) in enumerate(kv_alone[b]):
            tk, tv = t.past_key_values.gather(l)
            assert _rel(tk[..., :m, :], k[..., :m, :]) < TOL and _rel(tv[..., :m, :], v[..., :m, :]) < TOL, (b, l)
        a.past_key_values.release()
        t.past_key_values.release()


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
