"""What a turn brings to the device in one launch, and the device times that are read behind the call."""
import pytest
import torch

from livecc_b200 import _cabi
from livecc_b200.config import LiveCCConfig
from livecc_b200.engine import LiveCCB200ForConditionalGeneration

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,S", [(1, 1), (8, 3), (255, 255), (257, 1000), (80001, 24), (9, 0)])
def test_ids_positions_and_scalars(L, S):
    ctx = _cabi.Context(0)
    ids = torch.randint(0, 1 << 40, (L + 1,), device="cuda")[1:]          # (8-byte, not 16-byte alignment)
    seq = torch.full((L + 7,), -1, dtype=torch.int64, device="cuda")
    pos3 = torch.full((3, S), -1, dtype=torch.int32, device="cuda") if S else None
    scalars = torch.full((9,), -1, dtype=torch.int32, device="cuda")
    values = [7, -3, 0, 1 << 30, L, 0, 5, 9]
    other = torch.zeros(20, dtype=torch.int64, device="cuda")             # a second stream's turn beside it
    sc2 = torch.zeros(8, dtype=torch.int32, device="cuda")
    ctx.turn_setup([(ids, seq, pos3, 1234, scalars, values), (torch.arange(20, device="cuda"), other, None, 0, sc2, range(8))])
    assert other.tolist() == list(range(20)) and sc2.tolist() == list(range(8))
    with pytest.raises(_cabi.LiveCCNativeError):
        ctx.turn_setup([(ids, seq, pos3, 1, scalars, values)] * 9)
    assert torch.equal(seq[:L], ids) and bool((seq[L:] == -1).all())
    assert scalars.tolist() == values + [-1]
    if S:
        assert torch.equal(pos3, (torch.arange(S, dtype=torch.int32, device="cuda") + 1234).expand(3, -1))
    ctx.close()


def test_ids_of_other_types_and_strides_and_the_times_of_a_call():
    m = LiveCCB200ForConditionalGeneration.from_synthetic(LiveCCConfig.small())
    ids = torch.randint(5, 900, (1, 20))
    want = m.generate(ids, max_new_tokens=4).sequences
    assert m.last_stats["prefill_tokens"] == 20 and m.last_stats["prefill_ms"] > 0
    before = dict(m.phase_ms_total)
    wide = torch.stack([ids[0], ids[0] + 1], 1).view(1, -1).cuda()
    for form in (ids.to(torch.int32), ids.cuda().to(torch.int32), wide[:, ::2], wide.cpu()[:, ::2]):
        c = m.new_cache()
        first = m.generate(form[:, :12], past_key_values=c, max_new_tokens=1).sequences
        assert torch.equal(first[:, :12].cpu(), ids[:, :12])
        assert torch.equal(m.generate(form, max_new_tokens=4).sequences, want)
        c.seq_len = 12
        two = m.generate(form, past_key_values=c, max_new_tokens=4).sequences      # a second turn: positions run on
        assert torch.equal(two[:, :20].cpu(), ids)
    assert m.phase_ms_total["calls"] == before["calls"] + 12 and m.phase_ms_total["prefill"] > before["prefill"]
    for _ in range(3):       # calls that end in an error leave the times of the last one that did not
        m.generate(ids, max_new_tokens=1)
        with pytest.raises(ValueError):
            m.generate(torch.cat([ids, torch.full((1, 2), m.config.video_token_id)], 1), max_new_tokens=1, video_frames=torch.zeros((2, 3, 56, 56), dtype=torch.uint8))
        assert m.generate(ids, max_new_tokens=1) is not None and m.last_stats["prefill_ms"] > 0
    m.phase_ms_total["calls"] = 0
    assert m.phase_ms_total["calls"] == 0


def test_the_times_of_a_call_are_there_when_it_returns_and_can_be_replaced():
    m = LiveCCB200ForConditionalGeneration.from_synthetic(LiveCCConfig.small())
    ids = torch.randint(5, 900, (1, 20))
    held = m.phase_ms_total
    for n in (1, 2):
        m.generate(ids, max_new_tokens=3)
        assert held["calls"] == n and held["decode_steps"] == 2 * n and held["prefill"] > 0
    m.phase_ms_total, m.last_stats = {k: 0 for k in held}, {}
    m.generate(ids, max_new_tokens=3)
    assert m.phase_ms_total["calls"] == 1 and m.last_stats["generated"] == 3 and held["calls"] == 2
