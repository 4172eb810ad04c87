"""The block quantizer's two arithmetics (f32 with a tie check, double).

Codes, scales and sums are the oracle's bit for bit wherever the f32 arithmetic hands over to the double one: a
maximum of zero, tiny, huge; elements on and next to every k + 0.5.  The GEMM's pre-pass quantizes by the same rule:
its result is, bit for bit, that of the float mode on code * scale from the quantizer kernel's arrays.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from raster_b200 import Context
from raster_b200 import _lib as L
from raster_b200.quant import cpu_quant as cq

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(("cuda:0",))
    yield c
    c.close()


def hard_blocks():
    """Blocks of 32: maxima over the whole range, elements at and around the ties of their scale."""
    rng = np.random.default_rng(7)
    blocks = [np.zeros(32, np.float32)]
    for top in (1e-38, 9.9e-31, 1.1e-30, 1e-5, 1.0, 3.0, 127.0, 9e36, 1.1e37, 3.3e38):
        for _ in range(4):
            k = rng.integers(-127, 127, 32).astype(np.float64) + 0.5
            x = (k * (np.float64(np.float32(top)) / 127.0)).astype(np.float32)
            if rng.integers(0, 2):
                x = np.nextafter(x, np.where(rng.integers(0, 2, 32) == 1, np.inf, -np.inf).astype(np.float32))
            x = np.clip(x, -np.float32(top), np.float32(top)).astype(np.float32)
            x[rng.integers(0, 32)] = np.float32(top) * rng.choice([-1, 1])
            blocks.append(x)
    blocks += [rng.standard_normal(32).astype(np.float32) for _ in range(2007)]
    return np.stack(blocks)


def test_codes_scales_sums_bit_for_bit(ctx):
    x = hard_blocks()
    n = x.size
    bx = ctx.array_to_buffer(x.ravel())
    q, s, z = ctx.make_buffer(n, np.int8), ctx.make_buffer(n // 32, np.float32), ctx.make_buffer(n // 32, np.int32)
    ctx.quant_act_i8(bx, q, s, z, 1, n)
    ctx.sync()
    oq, os_, oz = orc.quantize_act_i8(x.ravel(), 1, n)
    assert np.array_equal(q.download(), oq)
    assert np.array_equal(s.download().view(np.uint32), os_.view(np.uint32))
    assert np.array_equal(z.download(), oz)
    for b in (bx, q, s, z):
        b.free()


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("in_,M", [(32, 64), (288, 65), (4128, 100), (8192, 64), (8224, 70), (12288, 66)])
def test_pre_pass_quantizes_like_the_quantizer(ctx, act, in_, M):
    """Rows in one pass of registers (<= 8192) and longer, whole and partial warps of 8-element pieces."""
    out = 136
    rng = np.random.default_rng(in_ + M)
    wq, ws = orc.quantize_weight(rng.standard_normal(out * in_).astype(np.float32), 4)
    w = ctx.bind_weight(wq, ws, out, in_, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
    blocks = hard_blocks()
    blocks = blocks[np.abs(blocks).max(1) <= 1e6]
    x = torch.from_numpy(blocks[rng.integers(0, len(blocks), M * in_ // 32)].ravel()).to(act).cuda()
    xf = x.to(torch.float32)
    torch.cuda.synchronize()
    n = M * in_
    bx = ctx.wrap_buffer(x.data_ptr(), n, np.float32 if act == torch.float32 else np.uint16)
    by = ctx.make_buffer(M * out, np.float32)
    ctx.qmatmul(w, bx, by, M, L.F32 if act == torch.float32 else L.BF16, L.F32, L.MODE_A8)
    ctx.sync()
    got = by.download()
    bxf, q, s = ctx.wrap_buffer(xf.data_ptr(), n, np.float32), ctx.make_buffer(n, np.int8), ctx.make_buffer(n // 32, np.float32)
    z = ctx.make_buffer(n // 32, np.int32)
    ctx.quant_act_i8(bxf, q, s, z, M, in_)
    ctx.sync()
    v = (q.download().reshape(-1, 32).astype(np.float32) * s.download()[:, None]).ravel()
    bv = ctx.array_to_buffer(v)
    ctx.qmatmul(w, bv, by, M, L.F32, L.F32, L.MODE_F)
    ctx.sync()
    assert np.isfinite(got).all()
    assert np.array_equal(got.view(np.uint32), by.download().view(np.uint32))
    for b in (bx, by, bxf, q, s, z, bv, w):
        b.free()


@pytest.mark.parametrize("fmt", ["q4_0", "q8_0", "q4k", "q6k"])
@pytest.mark.parametrize("nan", [slice(5, 6), slice(64, 96), slice(256, 512), slice(300, 1000, 3)])   # an element, a block, a super-block, every third
def test_elements_that_are_no_number_get_the_same_code_on_every_route(ctx, fmt, nan):
    """One token: the quantizer inside the decode kernel (x from a buffer, x among the launch's parameters) and the
    quantizer kernel in front of it give the same results, bit for bit, and as many of them are NaN."""
    out, in_ = 2048, 2048
    rng = np.random.default_rng(3)
    W = (rng.standard_normal(out * in_) * 0.02).astype(np.float32)
    if fmt == "q4k":
        w = ctx.bind_weight_q4k(cq.quantize_weight_q4k(W), out, in_)
    elif fmt == "q6k":
        w = ctx.bind_weight_q6k(cq.quantize_weight_q6k(W), out, in_)
    else:
        q = cq.quantize_weight(W, cq.q4_0 if fmt == "q4_0" else cq.q8_0)
        w = ctx.bind_weight(q["wq"], q["ws"], out, in_, L.FMT_Q4_0 if fmt == "q4_0" else L.FMT_Q8_0, L.LAYOUT_ROWMAJOR)
    x = rng.standard_normal(in_).astype(np.float32)
    x[nan] = np.nan
    bx, by, got = ctx.array_to_buffer(x), ctx.make_buffer(out, np.float32), {}
    try:
        for fused in (0, 1):
            ctx.tune(L.TUNE_FUSE_QUANT, fused)
            ctx.qmatmul(w, bx, by, 1)
            ctx.sync()
            got[fused] = by.download()
    finally:
        ctx.tune(L.TUNE_FUSE_QUANT, 1)
    # a scale is a NaN, and with it every result, only where all elements under it are
    whole = (nan.stop - nan.start) // (nan.step or 1) >= (256 if fmt in ("q4k", "q6k") else 32) and not nan.step
    assert np.isnan(got[0]).all() if whole else np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1], equal_nan=True)
    assert np.array_equal(got[0], ctx.qmatmul_host(w, x)[0], equal_nan=True)
    for b in (bx, by, w):
        b.free()


@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 5, 7, 8, 9, 31, 33, 300])   # parts of a warp, of a thread block, several
@pytest.mark.parametrize("act", [L.F32, L.BF16])
def test_numbers_of_blocks_that_fill_no_warp(ctx, act, blocks):
    """Eight lanes quantize a block, a thread block 64 / 8 of them: codes, scales and sums (f32), and through a product of two
    to four tokens the image of odd and even numbers of tokens (both types), against the oracle."""
    all_ = hard_blocks()
    all_ = all_[np.abs(all_).max(1) <= 1e6]
    rng = np.random.default_rng(blocks)
    x = all_[rng.integers(0, len(all_), blocks)].ravel()
    n = x.size
    if act == L.F32:
        bx = ctx.array_to_buffer(x)
        q, s, z = ctx.make_buffer(n + 64, np.int8), ctx.make_buffer(blocks + 8, np.float32), ctx.make_buffer(blocks + 8, np.int32)
        for b in (q, s, z):
            b.fill_bytes(0x5A)
        ctx.quant_act_i8(bx, q, s, z, 1, n)
        ctx.sync()
        oq, os_, oz = orc.quantize_act_i8(x, 1, n)
        assert np.array_equal(q.download()[:n], oq) and (q.download()[n:] == 0x5A).all()
        assert np.array_equal(s.download().view(np.uint32)[:blocks], os_.view(np.uint32)) and (s.download().view(np.uint32)[blocks:] == 0x5A5A5A5A).all()
        assert np.array_equal(z.download()[:blocks], oz) and (z.download()[blocks:] == 0x5A5A5A5A).all()
        for b in (bx, q, s, z):
            b.free()
    out = 40
    wq, ws = orc.quantize_weight(rng.standard_normal(out * n).astype(np.float32), 4)
    w = ctx.bind_weight(wq, ws, out, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
    for M in (2, 3, 4):
        xm = all_[rng.integers(0, len(all_), M * blocks)].ravel()
        bits = (xm.view(np.uint32) >> 16).astype(np.uint16)
        if act == L.BF16:
            xm = (bits.astype(np.uint32) << 16).view(np.float32)
        bx, by = ctx.array_to_buffer(bits if act == L.BF16 else xm), ctx.make_buffer(M * out, np.float32)
        ctx.qmatmul(w, bx, by, M, act, L.F32, L.MODE_A8)
        ctx.sync()
        ref = orc.matmul_a8_f64(wq, ws, 0, *orc.quantize_act_i8(xm, M, n), M, n, out).reshape(M, out)
        got = by.download().reshape(M, out)
        assert (np.abs(got - ref).max(1) <= 2e-6 * np.abs(ref).max(1)).all()
        bx.free(), by.free()
    w.free()
