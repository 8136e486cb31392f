"""tcgen05 GEMM core vs torch on the GPU: bit-exact on integer-valued operands (fp32 accumulation is
exact there, so any descriptor/swizzle/tile bug shows as a hard mismatch), tolerance on random ones."""
import math

import pytest
import torch

from livecc_b200 import _cabi as A

pytestmark = pytest.mark.gpu

SHAPES = [
    (128, 128, 64), (128, 256, 128), (256, 512, 256), (100, 136, 72), (281, 4608, 3584),
    (1024, 1280, 1176), (1024, 3840, 1280), (3072, 5120, 1280), (33, 64, 3584), (130, 264, 200),
]


def _ints(shape, lo, hi, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(lo, hi + 1, shape, device="cuda", generator=g).to(torch.bfloat16)


@pytest.mark.parametrize("block_n", [0, 32, 48, 64, 80, 112, 128, 144, 176, 208, 224, 240, 256, -64, -96, -128, -160, -224, -256])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_exact_integer_operands(ctx, M, N, K, block_n):
    a = _ints((M, K), -2, 2, 1)
    b = _ints((N, K), -2, 2, 2)
    ref = (a.float() @ b.float().T).to(torch.bfloat16)
    out = ctx.gemm(a, b, block_n=block_n)
    torch.cuda.synchronize()
    assert torch.equal(out, ref), f"mismatch: {(out.float() - ref.float()).abs().max().item()}"


@pytest.mark.parametrize("M,N,K", [(281, 4608, 3584), (1024, 1280, 5120), (200, 136, 72)])
def test_gemm_bias_residual_exact(ctx, M, N, K):
    a = _ints((M, K), -2, 2, 3)
    b = _ints((N, K), -1, 1, 4)
    bias = _ints((N,), -8, 8, 5)
    res = _ints((M, N), -8, 8, 6)
    acc = a.float() @ b.float().T
    out = ctx.gemm(a, b, bias=bias, epilogue=A.EPI_BIAS)
    assert torch.equal(out, (acc + bias.float()).to(torch.bfloat16))
    out = ctx.gemm(a, b, residual=res, epilogue=A.EPI_RESIDUAL)
    assert torch.equal(out, acc.to(torch.bfloat16) + res)
    out = ctx.gemm(a, b, bias=bias, residual=res, epilogue=A.EPI_BIAS_RESIDUAL)
    assert torch.equal(out, (acc + bias.float()).to(torch.bfloat16) + res)
    # in-place residual (out aliases residual), the way the engine uses it
    res2 = res.clone()
    ctx.gemm(a, b, out=res2, residual=res2, epilogue=A.EPI_RESIDUAL)
    assert torch.equal(res2, acc.to(torch.bfloat16) + res)


def _close(out, ref, ulps=2):
    out, ref = out.float(), ref.float()
    tol = ulps * 2.0 ** -8 * ref.abs().clamp_min(1e-2)
    bad = (out - ref).abs() > tol
    return bad.float().mean().item()


@pytest.mark.parametrize("M,N,K", [(1024, 5120, 1280), (256, 3584, 5120), (77, 320, 136)])
def test_gemm_activation_epilogues(ctx, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(7)
    a = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    b = (torch.randn((N, K), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    bias = (torch.randn((N,), device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    lin = (a.float() @ b.float().T + bias.float()).to(torch.bfloat16)
    out = ctx.gemm(a, b, bias=bias, epilogue=A.EPI_BIAS_QUICKGELU)
    ref = lin * torch.sigmoid(1.702 * lin)
    assert _close(out, ref) < 1e-3
    out = ctx.gemm(a, b, bias=bias, epilogue=A.EPI_BIAS_GELU)
    assert _close(out, torch.nn.functional.gelu(lin)) < 1e-3
    out = ctx.gemm(a, b, bias=bias, epilogue=A.EPI_BIAS)
    assert _close(out, lin, ulps=1) < 5e-3  # accumulation-order flips at the bf16 rounding boundary
    assert _close(out, lin, ulps=2) == 0


@pytest.mark.parametrize("M,I,K", [(281, 18944, 3584), (64, 2432, 896), (300, 96, 64)])
def test_gemm_swiglu(ctx, M, I, K):
    from livecc_b200.checkpoint import interleave_gate_up

    g = torch.Generator(device="cuda").manual_seed(8)
    a = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    wg = (torch.randn((I, K), device="cuda", generator=g) * 0.03).to(torch.bfloat16)
    wu = (torch.randn((I, K), device="cuda", generator=g) * 0.03).to(torch.bfloat16)
    gate = (a.float() @ wg.float().T).to(torch.bfloat16)
    up = (a.float() @ wu.float().T).to(torch.bfloat16)
    ref = torch.nn.functional.silu(gate) * up
    out = ctx.gemm(a, interleave_gate_up(wg, wu), epilogue=A.EPI_SWIGLU)
    assert out.shape == (M, I)
    assert _close(out, ref) < 1e-3


@pytest.mark.parametrize("block_n", [32, 96, 160, 224, -64, -160, -256])
def test_gemm_swiglu_every_tile_width(ctx, block_n):
    """The N tile is a run-time value (multiples of 32 for the SwiGLU epilogue): every width gives the same bits as 256.
    Negative widths select the CTA-pair kernel (cta_group::2, 256 x |block_n| tiles)."""
    from livecc_b200.checkpoint import interleave_gate_up

    g = torch.Generator(device="cuda").manual_seed(18)
    M, I, K = 281, 1184, 512
    a = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    w = interleave_gate_up((torch.randn((I, K), device="cuda", generator=g) * 0.03).to(torch.bfloat16),
                           (torch.randn((I, K), device="cuda", generator=g) * 0.03).to(torch.bfloat16))
    assert torch.equal(ctx.gemm(a, w, epilogue=A.EPI_SWIGLU, block_n=block_n), ctx.gemm(a, w, epilogue=A.EPI_SWIGLU, block_n=256))


@pytest.mark.parametrize("block_n", [48, 80, 144, 240, -96, -192, -256])
def test_gemm_epilogues_every_tile_width(ctx, block_n):
    """Bias / activation / residual epilogues with a half-used last 32-column chunk (block_n % 32 == 16) and a ragged N."""
    g = torch.Generator(device="cuda").manual_seed(19)
    M, N, K = 300, 1096, 320
    a = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    b = (torch.randn((N, K), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    bias = (torch.randn((N,), device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    res = torch.randn((M, N), device="cuda", generator=g).to(torch.bfloat16)
    for epi, kw in [(A.EPI_BIAS, dict(bias=bias)), (A.EPI_BIAS_QUICKGELU, dict(bias=bias)), (A.EPI_BIAS_GELU, dict(bias=bias)),
                    (A.EPI_RESIDUAL, dict(residual=res)), (A.EPI_BIAS_RESIDUAL, dict(bias=bias, residual=res))]:
        assert torch.equal(ctx.gemm(a, b, epilogue=epi, block_n=block_n, **kw), ctx.gemm(a, b, epilogue=epi, block_n=256, **kw)), epi


@pytest.mark.parametrize("M,N,K,epi", [(2048, 10304, 1160, 8), (2049, 10304, 1096, 9), (2303, 5120, 1224, 11), (1281, 4640, 1096, A.EPI_SWIGLU),
                                       (2090, 4616, 1088, A.EPI_NONE), (513, 10312, 1344, A.EPI_NONE)])   # 8, 9, 11: relu^2, tanh gelu, erf gelu
def test_gemm_default_kernel_equals_one_cta(ctx, M, N, K, epi):
    """Large products run on CTA pairs by default: the same sums in the same order as the one-CTA kernel, every epilogue."""
    a, b = _ints((M, K), -2, 2, 21), _ints((N, K), -2, 2, 22)
    a, b = (a * 0.11).to(torch.bfloat16), (b * 0.07).to(torch.bfloat16)
    assert torch.equal(ctx.gemm(a, b, epilogue=epi), ctx.gemm(a, b, epilogue=epi, block_n=256))


@pytest.mark.parametrize("epi", [A.EPI_NONE, A.EPI_BIAS, A.EPI_BIAS_QUICKGELU, A.EPI_BIAS_GELU, A.EPI_RESIDUAL, A.EPI_BIAS_RESIDUAL, A.EPI_SWIGLU, 8, 9, 11])
@pytest.mark.parametrize("M,N,K", [(1, 3584, 3584), (24, 4608, 3584), (33, 2080, 4104), (281, 3584, 3592), (288, 3584, 18944), (300, 37888, 512), (1000, 1280, 5120),
                                   (513, 3584, 4096)])
def test_gemm_few_rows_every_epilogue(ctx, M, N, K, epi):
    """Few rows, most of them with the operands swapped, K split inside a cluster: equal to the one-CTA kernel on sums that fp32 holds
    exactly (so the order of the splits cannot show); ragged rows, columns and k. (The shapes that must take the swapped kernel, and its
    forms one by one, are in the two tests behind this one.)"""
    a, b = _ints((M, K), -1, 1, 31), _ints((N, K), -1, 1, 32)
    kw = {}
    if epi in (A.EPI_BIAS, A.EPI_BIAS_QUICKGELU, A.EPI_BIAS_GELU, A.EPI_BIAS_RESIDUAL):
        kw["bias"] = _ints((N,), -8, 8, 33)
    if epi in (A.EPI_RESIDUAL, A.EPI_BIAS_RESIDUAL):
        kw["residual"] = _ints((M, N), -8, 8, 34)
    # (activations: integers are exact before them; the fp32 math after the sum is the same code)
    assert torch.equal(ctx.gemm(a, b, epilogue=epi, **kw), ctx.gemm(a, b, epilogue=epi, block_n=128, **kw))


@pytest.mark.parametrize("M,N,K", [(24, 4608, 3584), (281, 3584, 3584), (281, 3584, 18944), (256, 5120, 5120), (281, 37888, 3584)])
def test_gemm_plan_takes_the_swapped_kernel(ctx, M, N, K):
    """The shapes the rule was measured on take the swapped form, the last one with more tiles than clusters; sums held exactly."""
    assert ctx.gemm_plan(M, N, K)[0] == 2
    a, b = _ints((M, K), -1, 1, 41), _ints((N, K), -1, 1, 42)
    assert torch.equal(ctx.gemm(a, b), ctx.gemm_form(a, b, 0, 128))


# M, N, K, width, splits: one and two column groups (width up to and above 256), ragged rows, columns and k, more tiles than clusters (one
# tile of rows and several), every split, the whole tile range of rows
SWAP_FORMS = [(1, 288, 72, 32, 1), (33, 544, 200, 64, 1), (33, 544, 328, 64, 2), (97, 320, 1224, 128, 3), (128, 288, 520, 128, 4),
              (250, 1056, 328, 256, 1), (281, 1312, 1224, 288, 2), (500, 544, 136, 512, 1), (300, 544, 392, 160, 2), (40, 20512, 200, 64, 1),
              (281, 7712, 136, 96, 1), (290, 19232, 328, 320, 1)]


@pytest.mark.parametrize("epi,limit", [(A.EPI_NONE, 0), (A.EPI_BIAS, 0), (A.EPI_BIAS_QUICKGELU, 0), (A.EPI_BIAS_GELU, 0), (A.EPI_RESIDUAL, 0), (A.EPI_BIAS_RESIDUAL, 0),
                                       (A.EPI_SWIGLU, 0), (8, 0), (9, 0), (11, 0), (A.EPI_CLAMP_GLU, 7.0), (A.EPI_CLAMP_GLU, math.inf)])
@pytest.mark.parametrize("M,N,K,width,splits", SWAP_FORMS)
def test_gemm_swapped_form(ctx, M, N, K, width, splits, epi, limit):
    """Every form of the swapped kernel equals the one-CTA kernel on sums that fp32 holds exactly, whatever the rule would choose."""
    a, b = _ints((M, K), -1, 1, 43), _ints((N, K), -1, 1, 44)
    kw = dict(epilogue=epi)
    if epi in (A.EPI_BIAS, A.EPI_BIAS_QUICKGELU, A.EPI_BIAS_GELU, A.EPI_BIAS_RESIDUAL):
        kw["bias"] = _ints((N,), -8, 8, 45)
    if epi in (A.EPI_RESIDUAL, A.EPI_BIAS_RESIDUAL):
        kw["residual"] = _ints((M, N), -8, 8, 46)
    if epi == A.EPI_CLAMP_GLU:
        kw.update(limit=limit, alpha=1.702 if limit < 8 else 1.0, up_bias=1.0 if limit < 8 else 0.0)
    assert torch.equal(ctx.gemm_form(a, b, 2, width, splits, **kw), ctx.gemm_form(a, b, 0, 128, **kw))


@pytest.mark.parametrize("N,K,splits", [(544, 65536, 1), (544, 65536, 2), (544, 65536, 3), (20512, 8192, 1)])
@pytest.mark.parametrize("epi", [A.EPI_NONE, A.EPI_RESIDUAL, A.EPI_SWIGLU, 8, A.EPI_CLAMP_GLU])
def test_gemm_swapped_wait_that_runs_out(epi, N, K, splits):
    """A limit of 1 us on waits for sums that take 50 us and more: the kernel ends, every value it stores is NaN (also where the activation would
    turn a NaN into a number, and in a cluster's second tile), the context says so from then on, and others go on."""
    ctx = A.Context(0)
    M = 97
    a, b = _ints((M, K), -1, 1, 48), _ints((N, K), -1, 1, 49)
    out = torch.zeros((M, N // 2 if epi in (A.EPI_SWIGLU, A.EPI_CLAMP_GLU) else N), dtype=torch.bfloat16, device="cuda")
    res = _ints((M, N), -8, 8, 50) if epi == A.EPI_RESIDUAL else None
    ctx.check_fault()
    try:      # (the launch itself may find the word set already)
        ctx.gemm_form(a, b, 2, 128, splits, epilogue=epi, residual=res, limit=7.0, wait_ns=1000, out=out)
    except A.LiveCCNativeError:
        pass
    torch.cuda.synchronize()
    assert bool(torch.isnan(out).all())
    with pytest.raises(A.LiveCCNativeError, match="gave up"):
        ctx.check_fault()
    with pytest.raises(A.LiveCCNativeError, match="gave up"):
        ctx.gemm(a, b)
    del ctx
    other = A.Context(0)
    other.check_fault()
    assert torch.equal(other.gemm_form(a, b, 2, 128, splits), other.gemm_form(a, b, 0, 128))
    other.check_fault()


@pytest.mark.parametrize("form,width,splits", [(0, 96, 1), (1, 128, 1), (1, 224, 1), (2, 96, 2)])
@pytest.mark.parametrize("limit", [7.0, math.inf])
def test_gemm_clamped_glu(ctx, form, width, splits, limit):
    """Epilogue 10 of each kernel against float64: gate and up rows interleaved by 16; one rounding to bf16 (2^-9) and fp32 sums before it."""
    from livecc_b200.checkpoint import interleave_gate_up

    g = torch.Generator(device="cuda").manual_seed(47)
    M, F, K = 281, 656, 520
    a = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    wg, wu = ((torch.randn((F, K), device="cuda", generator=g) * 0.2).to(torch.bfloat16) for _ in range(2))
    gate, up = (a.double() @ w.double().T for w in (wg, wu))
    gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
    ref = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    out = ctx.gemm_form(a, interleave_gate_up(wg, wu), form, width, splits, epilogue=A.EPI_CLAMP_GLU, limit=limit)
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2.0 ** -9


def test_gemm_strided_views(ctx):
    """A and C may be column slices of wider buffers (leading dimension > width)."""
    M, N, K = 256, 384, 320
    big_a = _ints((M, K + 64), -2, 2, 9)
    a = big_a[:, 32:32 + K]
    if a.data_ptr() % 16:  # TMA needs a 16-byte aligned base
        pytest.skip("unaligned view")
    b = _ints((N, K), -2, 2, 10)
    big_c = torch.zeros((M, N + 128), dtype=torch.bfloat16, device="cuda")
    ctx.gemm(a, b, out=big_c[:, 64:64 + N])
    ref = (a.float() @ b.float().T).to(torch.bfloat16)
    assert torch.equal(big_c[:, 64:64 + N], ref)
    assert big_c[:, :64].abs().sum().item() == 0 and big_c[:, 64 + N:].abs().sum().item() == 0


@pytest.mark.parametrize("M,N,K", [(281, 3584, 18944), (281, 3584, 3584), (281, 4608, 3584), (64, 256, 2048), (384, 136, 4096)])
def test_gemm_splitk_exact_integer_operands(ctx, M, N, K):
    """split-K (fp32 partial tiles + reduce kernel with the fused epilogue): integer operands keep every partial sum
    exact, so the result must be bit-identical to the unsplit reference for all four supported epilogues. By default
    the dispatch splits only K >= 8192 (the first shape); LIVECC_B200_GEMM_SPLITK=1 forces it for all of them (both
    modes were run on B200)."""
    a = _ints((M, K), -2, 2, 11)
    b = _ints((N, K), -1, 1, 12)
    bias = _ints((N,), -8, 8, 13)
    res = _ints((M, N), -8, 8, 14)
    ws = torch.empty((8 * M * N,), dtype=torch.float32, device="cuda")
    acc = a.float() @ b.float().T
    assert torch.equal(ctx.gemm(a, b, splitk_ws=ws), acc.to(torch.bfloat16))
    assert torch.equal(ctx.gemm(a, b, bias=bias, epilogue=A.EPI_BIAS, splitk_ws=ws), (acc + bias.float()).to(torch.bfloat16))
    out = res.clone()  # in place: residual aliases the output, as in the decoder
    ctx.gemm(a, b, out=out, residual=out, epilogue=A.EPI_RESIDUAL, splitk_ws=ws)
    assert torch.equal(out, (acc.to(torch.bfloat16).float() + res.float()).to(torch.bfloat16))
    out = ctx.gemm(a, b, bias=bias, residual=res, epilogue=A.EPI_BIAS_RESIDUAL, splitk_ws=ws)
    assert torch.equal(out, ((acc + bias.float()).to(torch.bfloat16).float() + res.float()).to(torch.bfloat16))


@pytest.mark.parametrize("M,N,K,width", [(1024, 1280, 1176, 96), (1000, 5112, 1280, 160), (2090, 4600, 3584, 192), (1020, 3832, 1288, 224)])
@pytest.mark.parametrize("epi", [A.EPI_NONE, A.EPI_BIAS, A.EPI_BIAS_RESIDUAL])
def test_gemm_widths_between_128_and_256(ctx, M, N, K, width, epi):
    """Products whose last wave only a width in between fills take one CTA per tile of that width, with ragged rows, columns and k; sums of
    integers are exact, so they equal the 128-column kernel's bit for bit."""
    assert ctx.gemm_plan(M, N, K)[:2] == (0, width)
    a, b = _ints((M, K), -1, 1, 51), _ints((N, K), -1, 1, 52)
    kw = {}
    if epi != A.EPI_NONE:
        kw["bias"] = _ints((N,), -8, 8, 53)
    if epi == A.EPI_BIAS_RESIDUAL:
        kw["residual"] = _ints((M, N), -8, 8, 54)
    assert torch.equal(ctx.gemm(a, b, epilogue=epi, **kw), ctx.gemm(a, b, epilogue=epi, block_n=128, **kw))


@pytest.mark.parametrize("M,N,K,form", [(328, 3584, 3584, 0), (344, 3584, 3584, 0), (328, 4608, 3584, 0), (1288, 1280, 5120, 0), (1400, 1280, 5120, 0),
                                        (24, 4608, 3584, 2), (281, 3584, 18944, 2), (281, 37888, 3584, 2)])
def test_plan_weighs_the_exchange_of_a_split(ctx, M, N, K, form):
    """The swapped form with K split over a cluster where it measured faster (form 2), one CTA per tile where the exchange of many rows costs more
    than the split gives (328 x 3584 x 3584: 20.3 us, 23.9 split in four)."""
    assert ctx.gemm_plan(M, N, K)[0] == form


@pytest.mark.parametrize("epi", [A.EPI_SWIGLU, A.EPI_CLAMP_GLU])
@pytest.mark.parametrize("form,width", [(0, 96), (0, 160), (0, 224), (1, 160), (1, 224)])
@pytest.mark.parametrize("M,N,K", [(130, 224, 192), (1, 96, 64), (700, 1056, 320)])
def test_gated_epilogues_at_widths_in_between(ctx, epi, form, width, M, N, K):
    """Two lanes exchange the halves of a row's 16 outputs: every width, ragged rows and columns, the bits of the 128-column kernel."""
    a, b = _ints((M, K), -1, 1, 61) * 0.25, _ints((N, K), -1, 1, 62) * 0.25
    kw = dict(epilogue=epi, limit=1.5)
    want = ctx.gemm_form(a, b, 0, 128, **kw)
    out = torch.full((M + 2, N // 2), 7.0, dtype=torch.bfloat16, device="cuda")
    ctx.gemm_form(a, b, form, width, out=out[:M], **kw)
    assert torch.equal(out[:M], want) and bool((out[M:] == 7.0).all())
    g, u = (a.double() @ b.double().T).view(M, N // 32, 2, 16).unbind(2)
    if epi == A.EPI_SWIGLU:
        y = (g / (1 + (-g).exp())) * u
    else:
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        y = g / (1 + (-1.702 * g).exp()) * (u + 1.0)
    # bf16 roundings of gate, up, their product (and silu): 2^-9 relative each, 4 of them
    assert bool(((out[:M].double() - y.reshape(M, -1)).abs() <= y.reshape(M, -1).abs() * 2.0 ** -7 + 1e-6).all())
