"""The gated linear recurrence by itself (bf16 rows, fp32 state and output), in blocks of 64 rows on the tensor cores: infinite entries give what the
fp32 kernels give for the same values."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(S, H, G, N, P, seed, sign=True):
    g = torch.Generator().manual_seed(seed)
    draw = lambda *s: (torch.randn(s, generator=g) if sign else torch.rand(s, generator=g) + 0.25).to(torch.bfloat16).to(DEV)
    return dict(k=draw(S, G, N), c=draw(S, G, N), u=draw(S, H, P), log_decay=-torch.rand((S, H), generator=g).to(DEV) * 0.05,
                state=draw(H, P, N).float(), sc=(torch.rand((S, H), generator=g) + 0.5).to(DEV), skip=torch.rand(H, generator=g).to(DEV))


def _scan(ctx, t, dt):
    a = {n: v.clone().to(dt) if n in ("k", "c", "u") else v.clone() for n, v in t.items()}
    y = ctx.gated_scan(**a, cs=0.5)
    return y, a["state"]


@pytest.mark.parametrize("name,row", [("u", 0), ("u", 64), ("u", 128), ("k", 0), ("k", 64), ("c", 3), ("c", 70), ("c", 129), ("state", 0)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf")])
def test_infinite_entries(ctx, name, row, value):
    t = _inputs(130, 4, 2, 72, 72, seed=row, sign=False)    # positive operands: no infinities of two signs meet
    t[name][row, 1, 5] = value
    y, state = _scan(ctx, t, torch.bfloat16)
    y32, state32 = _scan(ctx, t, torch.float32)
    assert bool(torch.isinf(y32).any())
    for got, want in ((y, y32), (state, state32)):
        at = torch.isinf(want)
        assert torch.equal(got[at], want[at])
        at = torch.isfinite(want)
        # 64 + 72 terms a sum, whatever its order: fp32 rounding of each, all terms of one sign
        assert bool(((got[at] - want[at]).abs() <= want[at].abs() * 2.0 ** -24 * 300).all())
