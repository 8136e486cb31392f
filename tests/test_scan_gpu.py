"""The gated linear recurrence by itself (bf16 rows, fp32 state and output), in blocks of 64 rows on the tensor cores: the error of fp32
sums against float64, and infinite entries give what the fp32 kernels give for the same values."""
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


def _exact(t, cs):
    """Outputs and final state token by token in float64, and the magnitudes that are summed for each."""
    k, c, u, la, st, sc, skip = (t[n].double() for n in ("k", "c", "u", "log_decay", "state", "sc", "skip"))
    k, c = (x.repeat_interleave(u.shape[1] // k.shape[1], 1) for x in (k, c))
    s, sa, y, ya = st.clone(), st.abs(), [], []
    for i in range(k.shape[0]):
        d = (sc[i][:, None] * u[i])[:, :, None] * k[i][:, None, :]
        s, sa = la[i].exp()[:, None, None] * s + d, la[i].exp()[:, None, None] * sa + d.abs()
        q = (cs * c[i])[:, None, :]
        y.append((s * q).sum(-1) + skip[:, None] * u[i])
        ya.append((sa * q.abs()).sum(-1) + (skip[:, None] * u[i]).abs())
    return torch.stack(y), torch.stack(ya), s, sa


@pytest.mark.parametrize("sign,state,decay", [(True, 1.0, 0.05), (False, 1.0, 0.05), (True, 1e4, 0.05), (True, 1.0, 3.0), (False, 1.0, 0.002)])
@pytest.mark.parametrize("S,H,G,N,P", [(200, 4, 2, 136, 72), (64, 2, 1, 64, 64), (129, 2, 2, 16, 8)])
def test_error_of_the_sums(ctx, S, H, G, N, P, sign, state, decay):
    """Against float64, relative to the magnitudes summed: some ten fp32 roundings (a block's sums of up to nine groups of 16 terms, decays, the state).
    Values cut in two instead of three are 1e-5 off, running sums in the tensor cores' accumulators 2e-6. Single values may also be off by what the
    difference of two running sums of log decays carries, each up to 64 decays and rounded at 2^-24 of that."""
    t = _inputs(S, H, G, N, P, seed=S, sign=sign)
    t["state"] *= state
    t["log_decay"] *= decay / 0.05
    y, st = _scan(ctx, t, torch.bfloat16)
    y64, ya, s64, sa = _exact(t, 0.5)
    for got, want, size in ((y, y64, ya), (st, s64, sa)):
        err = (got.double() - want).abs()
        assert float(err.norm() / size.norm()) < 8 * 2.0 ** -24 and float((err / size).max()) < (32 + 64 * decay) * 2.0 ** -24


def _vec(t, decay, seed):
    S, H, N = t["u"].shape[0], t["u"].shape[1], t["k"].shape[2]
    t["log_decay"] = -torch.rand((S, H, N), generator=torch.Generator().manual_seed(seed)).to(DEV) * decay
    return t


def _exact_vec(t, cs):
    """_exact for a log decay per key channel."""
    k, c, u, la, st, sc, skip = (t[n].double() for n in ("k", "c", "u", "log_decay", "state", "sc", "skip"))
    k, c = (x.repeat_interleave(u.shape[1] // k.shape[1], 1) for x in (k, c))
    s, sa, y, ya = st.clone(), st.abs(), [], []
    for i in range(k.shape[0]):
        d, f = (sc[i][:, None] * u[i])[:, :, None] * k[i][:, None, :], la[i].exp()[:, None, :]
        s, sa = f * s + d, f * sa + d.abs()
        q = (cs * c[i])[:, None, :]
        y.append((s * q).sum(-1) + skip[:, None] * u[i])
        ya.append((sa * q.abs()).sum(-1) + (skip[:, None] * u[i]).abs())
    return torch.stack(y), torch.stack(ya), s, sa


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("sign,decay", [(True, 0.05), (False, 0.002), (True, 3.0), (True, 60.0)])
@pytest.mark.parametrize("S,H,G,N,P", [(32, 1, 1, 8, 8), (200, 4, 2, 136, 72), (64, 2, 1, 64, 128), (130, 2, 2, 40, 136), (97, 2, 1, 13, 21), (65, 1, 1, 20, 64)])
def test_error_of_the_sums_with_a_decay_per_key_channel(ctx, S, H, G, N, P, sign, decay, dt):
    """The bounds of test_error_of_the_sums: a weight's decay is now the product of two (two more roundings of its some ten), and each of their exponents carries
    what the difference of two running sums does: rounded at up to 32 x decay on average, so that much of 2^-24 is added to the norm's bound too. Sizes: both sides of 64 rows, 64 and 128 channels, slabs of 16 and 32 key channels, rows that are not aligned."""
    t = _vec(_inputs(S, H, G, N, P, seed=S, sign=sign), decay, S)
    y, st = _scan(ctx, t, dt)
    y64, ya, s64, sa = _exact_vec(t, 0.5)
    for got, want, size in ((y, y64, ya), (st, s64, sa)):
        err = (got.double() - want).abs()
        assert float(err.norm() / size.norm()) < (8 + 32 * decay) * 2.0 ** -24 and float((err / size).max()) < (32 + 64 * decay) * 2.0 ** -24


@pytest.mark.parametrize("name,row", [("u", 0), ("u", 64), ("u", 128), ("k", 0), ("k", 40), ("c", 3), ("c", 129), ("state", 0)])
def test_infinite_entries_with_a_decay_per_key_channel(ctx, name, row):
    t = _vec(_inputs(130, 4, 2, 72, 136, seed=row, sign=False), 0.05, row)
    t[name][row, 1, 5] = float("inf")
    y, state = _scan(ctx, t, torch.bfloat16)
    y32, state32 = _scan(ctx, t, torch.float32)
    assert bool(torch.isinf(y32).any())
    for got, want in ((y, y32), (state, state32)):
        at = torch.isinf(want)
        assert torch.equal(got[at], want[at]) and torch.equal(torch.isnan(got), torch.isnan(want))
        at = torch.isfinite(want)
        assert bool(((got[at] - want[at]).abs() <= want[at].abs() * 2.0 ** -24 * 300).all())
