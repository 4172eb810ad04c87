"""Prefill GEMM over equal ranges of K-steps: tiles cut between thread blocks at any step.

A range that begins inside a tile hands its f32 sums to the thread block with the tile's first step.  Forced here
(selector 4) at sizes where that can go wrong: one step per range, tiles cut many times, rows whose last K-step is
partial, one and two accumulators, a ragged number of tokens.  The result is the whole-tile one up to the order of
f32 additions: at most 260 partial sums of a row, each rounded to 2^-23 of a running value that stays below
about 4 max|y|, as a random walk sqrt(260) * 4 * 2^-23 = 8e-6 of max|y|; the bound against f64 is the GEMM's own.
"""
import numpy as np
import pytest

from oracle import oracle as orc
from raster_b200 import _lib as L
from raster_b200 import synth

pytestmark = pytest.mark.gpu
TUNE_GEMM_WIDE = 13


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("out,in_,M", [(200, 160, 33), (300, 4128, 100), (2500, 1056, 60), (19000, 1056, 20),
                                       (3000, 2080, 300), (1032, 8192, 515)])
def test_ranges_against_whole_tiles(ctx, bits, out, in_, M):
    w = synth.normal(out + in_ + bits, out * in_, 0.02)
    wq, ws = orc.quantize_weight(w, bits)
    x = synth.normal(out + in_ + M, M * in_)
    bw = ctx.bind_weight(wq, ws, out, in_, L.FMT_Q4_0 if bits == 4 else L.FMT_Q8_0, L.LAYOUT_ROWMAJOR)
    y = {}
    try:
        for how in (3, 4):
            ctx.tune(TUNE_GEMM_WIDE, how)
            y[how] = ctx.qmatmul_host(bw, x, M, L.F32, L.MODE_F).reshape(M, out).astype(np.float64)
        again = ctx.qmatmul_host(bw, x, M, L.F32, L.MODE_F).reshape(M, out)
    finally:
        ctx.tune(TUNE_GEMM_WIDE, 0)
    assert np.array_equal(again.astype(np.float64), y[4])          # sums in a fixed order
    top = np.abs(y[3]).max()
    assert np.abs(y[4] - y[3]).max() <= 4 * 8e-6 * top
    rows = np.unique(np.concatenate([np.arange(0, out, max(1, out // 64)), [out - 1]]))
    c = np.ascontiguousarray(wq.reshape(out, -1)[rows]).ravel()
    s = np.ascontiguousarray(ws.reshape(out, -1)[rows]).ravel()
    ref = orc.matmul_dq_f64(c, s, 0 if bits == 4 else 1, x, M, in_, rows.size).reshape(M, rows.size)
    assert np.abs(y[4][:, rows] - ref).max() <= 1e-3 * np.abs(ref).max()
    bw.free()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("out,in_,M", [(100, 160, 129), (300, 4128, 300), (2500, 1056, 200), (1000, 2080, 256), (1032, 8192, 515),
                                       (256, 32, 257), (300, 2048, 6000), (700, 1056, 176), (300, 2080, 240), (256, 160, 161)])
def test_tiles_on_pairs_of_sms_against_tiles_on_one(ctx, bits, out, in_, M):
    """256-token tiles on pairs of SMs: an odd number of 128-feature tiles (one of a pair has none), tokens in the first SM's
    half alone, widths (of 160, 192 and 256 columns) that the tokens do not fill, tiles shared by two pairs, cut at any step, partial last K-steps, rows of one K-step.  Same products, same
    sums as a 256-token tile on one SM; cut tiles differ as above.  300 x 2048 at M = 6000: 72 tiles, cut in two on single SMs,
    would be 96 pairs so, more than there are places or scratch for, and stay whole on pairs."""
    w = synth.normal(out + in_ + bits, out * in_, 0.02)
    wq, ws = orc.quantize_weight(w, bits)
    x = synth.normal(out + in_ + M, M * in_)
    bw = ctx.bind_weight(wq, ws, out, in_, L.FMT_Q4_0 if bits == 4 else L.FMT_Q8_0, L.LAYOUT_ROWMAJOR)
    y = {}
    try:
        for how in (2, 5, 6, 5):
            ctx.tune(TUNE_GEMM_WIDE, how)
            got = ctx.qmatmul_host(bw, x, M, L.F32, L.MODE_F).reshape(M, out).astype(np.float64)
            assert how not in y or np.array_equal(got, y[how])
            y[how] = got
    finally:
        ctx.tune(TUNE_GEMM_WIDE, 0)
    top = np.abs(y[2]).max()
    assert np.abs(y[5] - y[2]).max() <= 4 * 8e-6 * top and np.abs(y[6] - y[2]).max() <= 4 * 8e-6 * top
    rows = np.unique(np.concatenate([np.arange(0, out, max(1, out // 64)), [out - 1]]))
    c = np.ascontiguousarray(wq.reshape(out, -1)[rows]).ravel()
    s = np.ascontiguousarray(ws.reshape(out, -1)[rows]).ravel()
    ref = orc.matmul_dq_f64(c, s, 0 if bits == 4 else 1, x, M, in_, rows.size).reshape(M, rows.size)
    assert np.abs(y[5][:, rows] - ref).max() <= 1e-3 * np.abs(ref).max()
    bw.free()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("out,in_,M", [(100, 2080, 20), (40, 20000, 17), (40, 65536, 17), (300, 4128, 40), (1000, 16384, 30), (2500, 4128, 100),
                                       (130, 8192, 128), (250, 2048, 64), (600, 8224, 200)])
def test_few_tiles_cut_over_many_thread_blocks(ctx, bits, out, in_, M):
    """A call of few tiles: each cut over as many thread blocks as its K-steps are worth (2 .. 43 here), tiles of 32, 64 and
    128 tokens, parts of unequal length, a partial last K-step.  As whole tiles up to the order of the additions; three calls
    in a row (each finds the flags of the one before taken down) give the same bits."""
    w = synth.normal(out + in_ + bits, out * in_, 0.02)
    wq, ws = orc.quantize_weight(w, bits)
    x = synth.normal(out + in_ + M, M * in_)
    bw = ctx.bind_weight(wq, ws, out, in_, L.FMT_Q4_0 if bits == 4 else L.FMT_Q8_0, L.LAYOUT_ROWMAJOR)
    try:
        y = [ctx.qmatmul_host(bw, x, M, L.F32, L.MODE_F).reshape(M, out).astype(np.float64) for _ in range(3)]
        ctx.tune(TUNE_GEMM_WIDE, 3)
        whole = ctx.qmatmul_host(bw, x, M, L.F32, L.MODE_F).reshape(M, out).astype(np.float64)
    finally:
        ctx.tune(TUNE_GEMM_WIDE, 0)
    assert np.array_equal(y[0], y[1]) and np.array_equal(y[0], y[2])
    assert not np.array_equal(y[0], whole)                         # (it was cut)
    # (rows of 65536, 4096 additions of 16 products, no random walk of 260: each off by 2^-23 of a running value, about max|y| at most)
    bound = 4 * 8e-6 if in_ <= 32768 else in_ / 16 * 2.0 ** -23
    assert np.abs(y[0] - whole).max() <= bound * np.abs(whole).max()
    rows = np.unique(np.concatenate([np.arange(0, out, max(1, out // 64)), [out - 1]]))
    c = np.ascontiguousarray(wq.reshape(out, -1)[rows]).ravel()
    s = np.ascontiguousarray(ws.reshape(out, -1)[rows]).ravel()
    ref = orc.matmul_dq_f64(c, s, 0 if bits == 4 else 1, x, M, in_, rows.size).reshape(M, rows.size)
    assert np.abs(y[0][:, rows] - ref).max() <= 1e-3 * np.abs(ref).max()
    bw.free()
