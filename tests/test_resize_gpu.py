"""GPU frame ingest: lcc_resize_bicubic_aa_u8 through the C ABI against the oracle, the golden
digests of the reference's torchvision call, and live torchvision. Bar: bit-exact (uint8)."""
import json
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.dirname(__file__))
from resize_cases import CASES, digest, make_clip, torchvision_resize  # noqa: E402

pytestmark = pytest.mark.gpu
GOLDEN = json.load(open(os.path.join(os.path.dirname(__file__), "golden", "resize_aa_golden.json")))


@pytest.fixture(scope="module")
def ctx():
    from livecc_b200 import _cabi

    c = _cabi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_kernel_matches_golden_and_oracle(ctx, case):
    from oracle import resize_aa

    name, T, h, w, H, W = case
    clip = make_clip(name, T, h, w)
    out = ctx.resize_bicubic_aa_u8(clip.cuda(), (H, W))
    torch.cuda.synchronize()
    assert out.shape == (T, 3, H, W) and out.dtype == torch.uint8
    assert digest(out) == GOLDEN["cases"][name]["sha256"]
    if T * h * w <= 2 * 720 * 1280:
        assert np.array_equal(out.cpu().numpy(), resize_aa.resize_bicubic_aa_u8(clip.numpy(), (H, W)))


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_kernel_matches_live_torchvision(ctx, case):
    """The reference's own call on this box's CPU. Bit-exact on the ATen build the rounding order was pinned on; another
    build of the reference's dependency may move a handful of pixels by one level (oracle/resize_aa.py)."""
    name, T, h, w, H, W = case
    clip = make_clip(name, T, h, w)
    ref = torchvision_resize(clip, (H, W))
    out = ctx.resize_bicubic_aa_u8(clip.cuda(), (H, W)).cpu()
    if torch.backends.cpu.get_cpu_capability() == GOLDEN["cpu_capability"] and torch.__version__ == GOLDEN["torch"]:
        assert torch.equal(out, ref)
    else:
        d = (out.to(torch.int16) - ref.to(torch.int16)).abs()
        assert int(d.max()) <= 1 and float((d != 0).float().mean()) < 1e-3


def test_rows_per_cta_and_alignment_do_not_change_the_result(ctx):
    """Every tiling (rows per CTA) and every 16-byte phase of the source rows gives the same bytes; W % 4 != 0 takes the
    scalar store path."""
    from oracle import resize_aa

    for (h, w, H, W) in [(211, 173, 56, 84), (120, 90, 173, 201), (64, 257, 30, 61)]:
        clip = make_clip(f"t{h}x{w}", 2, h, w)
        want = torch.from_numpy(resize_aa.resize_bicubic_aa_u8(clip.numpy(), (H, W)))
        for th in (0, 1, 2, 4, 8, 16):
            assert torch.equal(ctx.resize_bicubic_aa_u8(clip.cuda(), (H, W), rows_per_cta=th).cpu(), want), (h, w, th)
        # shift the whole clip by 1..15 bytes inside a larger buffer
        flat = clip.flatten()
        for shift in (1, 3, 8, 15):
            buf = torch.zeros(flat.numel() + 32, dtype=torch.uint8, device="cuda")
            buf[shift:shift + flat.numel()] = flat.cuda()
            view = buf[shift:shift + flat.numel()].view(clip.shape)
            assert torch.equal(ctx.resize_bicubic_aa_u8(view, (H, W)).cpu(), want), (h, w, shift)


def test_full_size_properties(ctx):
    """1080p -> 448x796 (the ingest shape of a 16:9 source): constant frames stay constant (weights sum to 1 within
    rounding -> exact after rounding to uint8), a horizontal flip commutes with the resize up to the window asymmetry
    (<= 1 level), and planes are independent (a batched call equals per-plane calls)."""
    h, w, H, W = 1080, 1920, 448, 796
    for v in (0, 1, 127, 255):
        c = torch.full((1, 3, h, w), v, dtype=torch.uint8, device="cuda")
        assert bool((ctx.resize_bicubic_aa_u8(c, (H, W)) == v).all())
    clip = make_clip("full", 2, h, w).cuda()
    out = ctx.resize_bicubic_aa_u8(clip, (H, W))
    for t in range(2):
        for ch in range(3):
            one = ctx.resize_bicubic_aa_u8(clip[t, ch].contiguous(), (H, W))
            assert torch.equal(one, out[t, ch])
    flipped = ctx.resize_bicubic_aa_u8(clip.flip(-1).contiguous(), (H, W)).flip(-1)
    assert int((flipped.to(torch.int16) - out.to(torch.int16)).abs().max()) <= 1
    assert digest(out.cpu()) == digest(torchvision_resize(clip.cpu(), (H, W))) or \
        torch.backends.cpu.get_cpu_capability() != GOLDEN["cpu_capability"]


def test_mirror_routes_cuda_clips_through_the_kernel(ctx):
    """livecc_utils.get_smart_resized_clip(device=cuda) == the host path, and _spatial_resize_video on a CUDA clip."""
    from livecc_b200 import _cabi
    from livecc_b200.livecc_utils import video_process_patch as vpp

    reader = vpp.SyntheticVideoReader("synthetic://40x360x640@30?seed=3")
    reader.get_frame_timestamp(0)
    pts = reader._frame_pts[:, 1]
    stamps = torch.arange(0.0, 3.0, 0.5)
    host, ts_h, idx_h = vpp.get_smart_resized_clip(reader, 252, 448, stamps, pts)
    before = _cabi.launch_count()
    dev, ts_d, idx_d = vpp.get_smart_resized_clip(reader, 252, 448, stamps, pts, device="cuda")
    assert _cabi.launch_count() == before + 1
    assert dev.is_cuda and idx_h == idx_d and torch.equal(ts_h, ts_d)
    if torch.backends.cpu.get_cpu_capability() == GOLDEN["cpu_capability"]:
        assert torch.equal(dev.cpu(), host)
    else:
        assert int((dev.cpu().to(torch.int16) - host.to(torch.int16)).abs().max()) <= 1


def test_plan_rejects_windows_larger_than_shared_memory(ctx):
    from livecc_b200 import _cabi

    with pytest.raises(_cabi.LiveCCNativeError):
        ctx.resize_plan(30000, 30000, 28, 28)
    with pytest.raises(_cabi.LiveCCNativeError):  # output width 1 with a height change: outside the oracle's domain
        ctx.resize_plan(60, 20, 30, 1)
    ctx.resize_plan(60, 20, 60, 1)  # width only: fine


@pytest.mark.parametrize("h,w,H,W", [(40, 52, 60, 84), (61, 157, 28, 70), (64, 160, 33, 66), (120, 400, 30, 100), (97, 401, 30, 97), (90, 550, 28, 100),
                                     (300, 520, 20, 40), (301, 523, 21, 37), (47, 8, 31, 9), (5, 3, 40, 24)])
def test_every_form_of_the_width_products(ctx, h, w, H, W):
    """1 to 4 k-steps and more per window, rows on and off word boundaries, planes that leave a tile ragged; noise (few pixels need the stated order),
    a checkerboard (half and even sizes: every tile is summed again) and steps of full height (clamped values)."""
    from oracle import resize_aa

    g = torch.Generator().manual_seed(h * w)
    noise = torch.randint(0, 256, (3, 1, h, w), generator=g, dtype=torch.uint8)
    check = ((torch.arange(h)[:, None] + torch.arange(w)[None]) % 2 * 255).to(torch.uint8).expand(2, 1, h, w)
    steps = ((torch.arange(w) // 7 % 2) * 255).to(torch.uint8).expand(1, 1, h, w)
    clip = torch.cat([noise, check, steps]).contiguous()
    want = torch.from_numpy(resize_aa.resize_bicubic_aa_u8(clip.numpy(), (H, W)))
    assert torch.equal(ctx.resize_bicubic_aa_u8(clip.cuda(), (H, W)).cpu(), want)
    half = torch.from_numpy(resize_aa.resize_bicubic_aa_u8(check.contiguous().numpy(), (max(h // 2, 2), max(w // 2, 2))))
    assert torch.equal(ctx.resize_bicubic_aa_u8(check.contiguous().cuda(), (max(h // 2, 2), max(w // 2, 2))).cpu(), half)


@pytest.mark.parametrize("h,w,H,W", [(1080, 1920, 448, 796), (2160, 3840, 448, 796)])
def test_a_plan_costs_little_more_than_its_weight_tables(ctx, h, w, H, W):
    """A size that is met once pays for its plan. Bound: twice the two weight tables for the operands and the error bound, and 150 us for memory and upload.
    (With an exponent and a power of two by library calls for every tap it took five times the tables.)"""
    import ctypes as C
    import time

    lib = ctx.lib

    def least(f):
        best = 1e9
        for _ in range(15):
            t = time.perf_counter()
            made = f()
            best = min(best, time.perf_counter() - t)
            if made:
                lib.lcc_resize_plan_destroy(C.c_void_p(made))
        return best * 1e6

    def tables():
        for n, m in ((w, W), (h, H)):
            buf = np.empty(m * lib.lcc_resize_aa_taps(n, m), np.float32)
            at = np.empty((2, m), np.int32)
            assert lib.lcc_resize_aa_table(n, m, at[0].ctypes.data_as(C.c_void_p), at[1].ctypes.data_as(C.c_void_p), buf.ctypes.data_as(C.c_void_p)) == 0

    def plan():
        return lib.lcc_resize_plan_create(C.c_void_p(ctx.handle), h, w, H, W, 0)

    kept = plan()      # (its block of device memory serves the others: a fresh one costs the driver some 400 us)
    assert least(plan) < 3 * least(tables) + 150
    lib.lcc_resize_plan_destroy(C.c_void_p(kept))


@pytest.mark.parametrize("h,w,H,W,frames", [(360, 640, 448, 796, (1, 2, 3)), (97, 61, 112, 140, (1, 49, 50)), (28, 28, 28, 28, (1,)), (64, 200, 65, 140, (1, 60))])
def test_both_sides_of_the_rule_for_enlarged_pictures_of_one_wave(ctx, h, w, H, W, frames):
    """Enlarged pictures whose CTAs are one wave take the stated order throughout, larger calls (and an axis made smaller) the products: the same bytes."""
    from oracle import resize_aa

    clip = make_clip("one_wave", max(frames), h, w)
    clip[:, :, ::2] = 255 * (clip[:, :, ::2] > 127)          # also values on the edge of the range
    for n in frames:
        out = ctx.resize_bicubic_aa_u8(clip[:n].cuda(), (H, W)).cpu()
        for t in {0, n - 1}:
            assert np.array_equal(out[t].numpy(), resize_aa.resize_bicubic_aa_u8(clip[t:t + 1].numpy(), (H, W))[0]), (n, t)
