"""The projections of a decode step of several streams (gemv_batch.cu) by themselves: whole-number operands whose products and sums are exact in
fp32, so that every order of summation gives the same bits; every number of streams, short and long K, finished streams. With real-valued operands, a stream's row has the same bits whoever its neighbours are."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BIAS, RESIDUAL, SWIGLU, LOGITS = range(4)


def _case(B, N, K, whole, seed):
    g = torch.Generator().manual_seed(seed)
    draw = lambda *s: (torch.randint(-3, 4, s, generator=g).float() if whole else torch.randn(s, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    return draw(N, K), draw(B, K), draw(N), draw(B, N), [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(B)]


def _run(ctx, W, x, bias, h, sc):
    return {BIAS: ctx.gemv_batch(BIAS, W, x, sc, bias=bias), RESIDUAL: ctx.gemv_batch(RESIDUAL, W, x, sc, out=h.clone()),
            SWIGLU: ctx.gemv_batch(SWIGLU, W, x, sc), LOGITS: ctx.gemv_batch(LOGITS, W, x, sc)}


# (|x| |W| <= 9: sums stay below 2^24 up to K = 2^20)
@pytest.mark.parametrize("B", range(1, 9))
@pytest.mark.parametrize("N,K", [(32, 64), (96, 576), (64, 1088), (2400, 512), (160, 8128), (160, 8192), (160, 8256), (4800, 8256), (32, 18944)])
def test_batched_projections_are_exact_on_whole_numbers(ctx, B, N, K):
    W, x, bias, h, sc = _case(B, N, K, True, B * 1000 + K)
    y = (x.double() @ W.double().t()).float()
    got = _run(ctx, W, x, bias, h, sc)
    assert torch.equal(got[BIAS], (y + bias.float()).bfloat16())
    assert torch.equal(got[RESIDUAL], (y.bfloat16().float() + h.float()).bfloat16())
    for logits in got[LOGITS]:
        assert torch.equal(logits, y.bfloat16().float())
    gu = y.bfloat16().float().view(B, N // 32, 2, 16)
    gate, up = gu[:, :, 0].reshape(B, -1).double(), gu[:, :, 1].reshape(B, -1)
    want = (gate / (1 + torch.exp(-gate))).float().bfloat16().double() * up.double()
    # silu's own rounding may fall to the next bf16 value, and the product's with it: 2^-8 each
    assert bool(((got[SWIGLU].double() - want).abs() <= want.abs() * 2.0 ** -7 + 1e-30).all())


@pytest.mark.parametrize("N,K", [(96, 576), (160, 8256)])
def test_finished_streams_keep_their_rows(ctx, N, K):
    W, x, bias, h, sc = _case(5, N, K, True, 7)
    sc[1][2] = sc[4][2] = 1   # LCC_SC_FINISHED
    for kind, cols in ((BIAS, N), (RESIDUAL, N), (SWIGLU, N // 2)):
        old = torch.full((5, cols), 3.0, dtype=torch.bfloat16, device=DEV)
        open_ = ctx.gemv_batch(kind, W, x, [torch.zeros_like(s) for s in sc], bias=bias, out=old.clone())
        got = ctx.gemv_batch(kind, W, x, sc, bias=bias, out=old.clone())
        for b in range(5):
            assert torch.equal(got[b], old[b] if b in (1, 4) else open_[b]), (kind, b)


@pytest.mark.parametrize("N,K", [(96, 576), (512, 3584), (160, 8256), (160, 18944)])
def test_a_row_has_the_same_bits_whoever_its_neighbours_are(ctx, N, K):
    W, x, bias, h, sc = _case(8, N, K, False, K)
    full = _run(ctx, W, x, bias, h, sc)
    for rows in ([0], [7], [3, 5], [6, 2, 0, 1, 4], [7, 6, 5, 4, 3, 2, 1, 0]):
        part = _run(ctx, W, x[rows], bias, h[rows], [sc[r] for r in rows])
        for kind in full:
            a, b = (full[kind][0], part[kind][0]) if kind == LOGITS else (full[kind], part[kind])
            assert torch.equal(b, a[rows]), (kind, rows)


def test_nothing_is_read_once_every_stream_has_ended(ctx):
    """Steps behind the end of every stream (a replayed graph) cost launches, not the weights' bytes: 272 MB take some 45 us."""
    W, x, bias, h, sc = _case(8, 38016, 3584, False, 1)

    def us():
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(11)]
        torch.cuda.synchronize()
        ev[0].record()
        for e in ev[1:]:
            ctx.gemv_batch(SWIGLU, W, x, sc)
            e.record()
        torch.cuda.synchronize()
        return min(a.elapsed_time(b) for a, b in zip(ev, ev[1:])) * 1e3

    us()
    open_ = us()
    for s in sc[:-1]:
        s[2] = 1
    some = us()
    sc[-1][2] = 1
    ended = us()
    assert ended < 0.6 * open_ and some > 0.8 * open_, (ended, some, open_)
