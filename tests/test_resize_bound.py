"""The error of one tensor-core step of the resize's width pass: 16 exact products of bytes minus 128 and fp16 weights, and an fp32 addend. The plan counts
(n + 4) units in the last place of S per step, n the products that are not zero and S the sum of all magnitudes (resize.cu). Here: the forms that the
instruction's contract leaves open stay within that (CPU), and so does the device."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest


def _steps(n, seed):
    """Bytes minus 128, weights and an addend: bands of a filter, one large product beside tiny ones of one sign, large products that cancel."""
    rng = np.random.default_rng(seed)
    a = rng.integers(-128, 128, (n, 16)).astype(np.float64)
    taps = rng.integers(1, 17, n)
    w = rng.standard_normal((n, 16)) * 2.0 ** rng.integers(-12, 1, (n, 1)) * (np.arange(16) < taps[:, None])
    c = rng.standard_normal(n) * 2.0 ** rng.integers(-14, 9, n)
    third = n // 3
    a[:third] = np.abs(a[:third]) + 1
    w[:third] = np.abs(w[:third]) * 2.0 ** -rng.integers(8, 14, (third, 1))        # tiny, one sign ...
    w[:third, 0] = rng.uniform(0.5, 1, third)                                      # ... behind a large one
    a[third:2 * third, 1] = -a[third:2 * third, 0]                                 # two that cancel
    w[third:2 * third, :2] = rng.uniform(0.5, 1, (third, 1))
    w = (np.clip(w, -2, 2) * 2.0 ** 14).astype(np.float16).astype(np.float64)
    w[np.abs(w) < 2.0 ** -14] = 0                                                  # (no subnormal operands)
    return a, w, np.float32(c * 2.0 ** 14).astype(np.float64)


def _bound(a, w, c):
    """(n + 4) units in the last of 24 bits of S."""
    s = (np.abs(a * w).sum(1) + np.abs(c)) * 1.0001
    return (np.count_nonzero(w, axis=1) + 4) * np.exp2(np.floor(np.log2(s)) - 23)


def _exact(a, w, c):
    """Exact in float64: products of 19 bits, magnitudes 2^-14 .. 2^29."""
    return (a * w).sum(1) + c


def _cut(x, unit):
    return np.trunc(x / unit) * unit


def _ulp(x):
    return np.exp2(np.floor(np.log2(np.maximum(np.abs(x), 2.0 ** -60))) - 23)


def _aligned(terms):
    """Addends cut behind 24 bits of the largest one, summed, the sum cut to 24 bits."""
    s = _cut(terms, _ulp(np.abs(terms).max(1))[:, None]).sum(1)
    return _cut(s, _ulp(s))


def _one_by_one(terms, order):
    s = terms[:, order[0]]
    for i in order[1:]:
        s = s + terms[:, i]
        s = _cut(s, _ulp(s))
    return s


@pytest.mark.parametrize("form", ["together", "halves", "forward", "backward", "shuffled"])
def test_every_form_of_a_step_stays_within_what_the_plan_counts(form):
    a, w, c = _steps(30000, 1)
    p = a * w
    if form == "together":
        d = _aligned(np.concatenate([p, c[:, None]], 1))
    elif form == "halves":
        d = _aligned(np.concatenate([p[:, 8:], _aligned(np.concatenate([p[:, :8], c[:, None]], 1))[:, None]], 1))
    else:
        order = {"forward": np.arange(17), "backward": np.arange(17)[::-1], "shuffled": np.random.default_rng(2).permutation(17)}[form]
        d = _one_by_one(np.concatenate([c[:, None], p], 1), order)
    err, most = np.abs(d - _exact(a, w, c)), _bound(a, w, c)
    assert (err <= most).all()
    # 17 units of the largest addend and one of the sum, counted for one alignment, do not cover every form
    lone = 17 * _ulp(np.maximum(np.abs(p).max(1), np.abs(c))) + _ulp(np.abs(_exact(a, w, c)))
    assert form != "forward" or (err > lone).any()


SOURCE = r"""
#include <cstdint>
__global__ void steps(const uint32_t* a, const uint32_t* b, const float* c, float* d) {   // a warp: 16 rows x 8 columns; [step][lane][regs]
    const size_t at = (size_t)blockIdx.x * 32 + threadIdx.x;
    const uint32_t *x = a + at * 4, *y = b + at * 2;
    const float* z = c + at * 4;
    float* o = d + at * 4;
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3])
                 : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "f"(z[0]), "f"(z[1]), "f"(z[2]), "f"(z[3]));
}
extern "C" int run(int n, const void* a, const void* b, const void* c, void* d) {
    steps<<<n, 32>>>((const uint32_t*)a, (const uint32_t*)b, (const float*)c, (float*)d);
    return cudaDeviceSynchronize();
}
"""


@pytest.mark.gpu
def test_the_device_stays_within_it(tmp_path):
    import torch

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "steps.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC", "-o", str(tmp_path / "steps.so"),
                    str(tmp_path / "steps.cu")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "steps.so"))
    tiles = 4000
    a, w, c = (x.reshape(tiles, 8, *x.shape[1:]) for x in _steps(tiles * 8, 3))      # a tile's column g: weights w[g]; row g and row g + 8: a[g], a[7 - g]
    rows = np.concatenate([a, a[:, ::-1]], 1)                                        # [tile, 16, 16]
    add = np.broadcast_to(c[:, None, :], (tiles, 16, 8))
    lane = np.arange(32)
    g, t = lane >> 2, lane & 3
    k = np.stack([2 * t, 2 * t + 1, 2 * t + 8, 2 * t + 9], 1)                        # the columns of A (rows of B) of a lane's register halves
    half = lambda x: np.ascontiguousarray(x.astype(np.float16))
    ra = half(np.stack([rows[:, g[:, None], k[:, :2]], rows[:, g[:, None] + 8, k[:, :2]], rows[:, g[:, None], k[:, 2:]], rows[:, g[:, None] + 8, k[:, 2:]]], 2))
    rb = half(np.stack([w[:, g[:, None], k[:, :2]], w[:, g[:, None], k[:, 2:]]], 2))
    at = [(g, 2 * t), (g, 2 * t + 1), (g + 8, 2 * t), (g + 8, 2 * t + 1)]
    rc = np.ascontiguousarray(np.stack([add[:, r, n] for r, n in at], 2).astype(np.float32))
    dev = [torch.from_numpy(x).cuda() for x in (ra.view(np.int16), rb.view(np.int16), rc)]
    out = torch.empty((tiles, 32, 4), device="cuda")
    assert lib.run(tiles, *(ctypes.c_void_p(x.data_ptr()) for x in dev), ctypes.c_void_p(out.data_ptr())) == 0
    got = out.cpu().numpy().astype(np.float64)
    for i, (r, n) in enumerate(at):
        A, B, C = rows[:, r].reshape(-1, 16), w[:, n].reshape(-1, 16), add[:, r, n].reshape(-1)
        err = np.abs(got[:, :, i].reshape(-1) - _exact(A, B, C))
        assert (err <= _bound(A, B, C)).all(), float((err / _bound(A, B, C)).max())
