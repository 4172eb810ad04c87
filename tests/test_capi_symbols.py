"""The C-ABI library loads without a GPU and exports every symbol rstq.h declares."""
import ctypes as C
import os
import re

import pytest

from raster_b200 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    names = set()
    for f in os.listdir(os.path.join(ROOT, "include")):
        if f.endswith(".h"):
            text = open(os.path.join(ROOT, "include", f)).read()
            names |= set(re.findall(r"RSTQ_API\s+[\w\s\*]+?\b(rstq_\w+)\s*\(", text))
    return names


def test_library_exports_every_declared_symbol():
    lib = L.load()
    names = declared_symbols()
    assert len(names) >= 30
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/ but not exported"
    assert names == set(L.SIGNATURES), names ^ set(L.SIGNATURES)


def test_version_and_error_string():
    lib = L.load()
    assert lib.rstq_version() >= 100
    assert isinstance(lib.rstq_last_error(), bytes)


def test_null_and_bad_handles_are_status_codes_not_crashes():
    lib = L.load()
    assert lib.rstq_shutdown(None) == L.OK
    assert lib.rstq_free(None) == L.OK
    assert lib.rstq_weight_free(None) == L.OK
    assert lib.rstq_graph_destroy(None) == L.OK
    assert lib.rstq_event_destroy(None) == L.OK
    assert lib.rstq_sync(None, 0) == L.E_INVALID
    assert lib.rstq_init(None, None, 1) == L.E_INVALID
    h = C.c_void_p()
    assert lib.rstq_init(None, C.byref(h), 0) == L.E_INVALID
    assert lib.rstq_alloc(None, C.byref(h), 0, 16) == L.E_INVALID
    assert b"context" in lib.rstq_last_error()


@pytest.mark.skipif(os.path.exists("/dev/nvidia0"), reason="a GPU is present")
def test_init_without_gpu_fails_loudly():
    lib = L.load()
    devs = (C.c_int32 * 1)(0)
    h = C.c_void_p()
    assert lib.rstq_init(devs, C.byref(h), 1) == L.E_NODEV
    assert not h.value
    assert b"no CPU path" in lib.rstq_last_error()
    from raster_b200 import Context
    with pytest.raises(L.RstqError):
        Context()


def test_gemm_plan_is_host_arithmetic_and_follows_the_wave_model():
    """rstq_gemm_plan needs no device: tile width and thread blocks per tile of the prefill GEMM on a
    148-SM part.  4096 features: up to 256 tokens the grid fills at most half the SMs and K = 4096 is
    long enough, so two thread blocks share a tile; 512 tokens are one wave of 128 tiles of 128; from
    768 on the tiles are 256 wide (one wave of 96 instead of two of 192)."""
    import ctypes as C
    from raster_b200 import _lib as L
    lib = L.load()
    plan = (C.c_int32 * 2)()

    def of(out, in_, m, sm=148):
        L.check(lib.rstq_gemm_plan(plan, out, in_, m, sm))
        return plan[0], plan[1]
    assert of(4096, 4096, 17) == (32, 2)
    assert of(4096, 4096, 64) == (64, 2)
    assert of(4096, 4096, 256) == (128, 2)
    assert of(4096, 4096, 512) == (128, 1)
    assert of(4096, 4096, 768) == (256, 1)
    assert of(4096, 4096, 2048) == (256, 1)
    assert of(28672, 8192, 256) == (256, 1)          # 224 wide tiles, run as ranges of their K-steps (below)
    assert of(28672, 8192, 16) == (32, 1)            # 224 tiles: more than half the SMs, no split
    assert of(4096, 256, 64) == (64, 1)              # K too short to cut
    assert of(4096, 4096, 512, sm=296) == (128, 2)   # a part twice as wide would split
    assert lib.rstq_gemm_plan(plan, 4096, 100, 64, 148) == L.E_SHAPE
    assert lib.rstq_gemm_plan(None, 4096, 4096, 64, 148) == L.E_INVALID


def test_gemm_ranges_where_whole_tiles_leave_sms_idle():
    """rstq_gemm_ranges: one range per SM where whole tiles would leave SMs idle for much of the last wave, whole tiles
    (or pairs) on the other side of the line.  Whatever is chosen, the parts of ranges fit the scratch they go to
    (160 parts of 128 x 256 sums) and there are no more than 256 of them."""
    from raster_b200 import runtime as R
    for out, in_, m in [(28672, 8192, 32), (28672, 8192, 256), (11008, 4096, 512)]:
        assert R.gemm_ranges(out, in_, m) == 148
    for out, in_, m in [(20000, 2048, 200), (14336, 4096, 512), (5120, 5120, 1024), (22016, 4096, 32), (24576, 3072, 20),
                        (24576, 3072, 64), (28672, 4096, 64), (8192, 28672, 256)]:
        assert R.gemm_ranges(out, in_, m) == 148
    # one wave, too little saved, too many tiles per range, rows of one or two K-steps
    for out, in_, m in [(8192, 8192, 512), (12288, 4096, 300), (4096, 4096, 768), (4096, 4096, 512), (4096, 4096, 64),
                        (4096, 4096, 2048), (4096, 11008, 2048), (27648, 1024, 256), (6144, 8192, 1024), (9000, 6144, 900),
                        (5120, 13824, 300), (26000, 2048, 32), (11008, 4096, 1024), (11008, 4096, 2048), (28672, 256, 2048), (28672, 128, 2048)]:
        assert R.gemm_ranges(out, in_, m) == 0
    for sm in (1, 20, 74, 132, 148, 160, 200, 296):
        for out in (32, 1000, 4096, 11008, 28672, 131072):
            for in_ in (32, 160, 1024, 4128, 28672):
                for m in (17, 33, 64, 100, 129, 300, 512, 2048):
                    n = R.gemm_ranges(out, in_, m, sm)
                    p = R.gemm_plan(out, in_, m, sm)
                    assert 0 <= n <= min(sm, 256) and n * p["tile_tokens"] <= 160 * 256
                    assert n == 0 or p["blocks_per_tile"] == 1
    with pytest.raises(Exception):
        R.gemm_ranges(4096, 100, 64)
    assert L.load().rstq_gemm_ranges(None, 4096, 4096, 64, 148) == L.E_INVALID


@pytest.mark.parametrize("wide", range(7))
def test_thread_blocks_that_share_gemm_tiles_have_a_slot_each(wide):
    """The scratch of shared tiles holds 160 slots of 128 x 256 sums and there are 256 flags, whatever the selector; pairs of SMs
    round an odd number of feature tiles up, which counts: 300 x 4096 at M = 6000 is 72 tiles of 256 tokens, and 48 pairs of
    feature tiles with a slot for each of their 96 thread blocks and part."""
    from raster_b200 import runtime as R
    shapes = [(300, 4096, 6000), (384, 2048, 6144), (128, 2048, 18944), (1032, 4096, 2048), (1100, 8192, 2048), (100, 4096, 37000)]
    shapes += [(out, in_, m) for out in (1, 32, 129, 300, 1000, 1152, 4096, 11008, 28672) for in_ in (32, 160, 2048, 4128, 28672)
               for m in (17, 33, 64, 100, 129, 161, 176, 240, 300, 512, 2048, 6000, 20000)]
    for sm in (20, 74, 132, 148, 160, 296):
        for out, in_, m in shapes:
            v = R.gemm_layout(out, in_, m, sm, wide)
            ft, tt, cs = -(-out // 128), -(-m // v["tile_tokens"]), 2 if v["pairs"] else 1
            assert v["blocks"] == cs * (v["ranges"] or -(-ft // cs) * tt * v["per_tile"])
            if v["per_tile"] > 1 or v["ranges"]:
                assert v["blocks"] <= min(sm, 256) and v["blocks"] * v["tile_tokens"] <= 160 * 256
            assert v["pairs"] <= (v["tile_tokens"] == 256)
            # an MMA of cta_group::2 with M = 256 takes N in thirty-twos
            assert v["columns"] == (min(-(-m // 32) * 32, 256) if v["pairs"] else v["tile_tokens"])
            if wide >= 5 and m > 128:
                assert v["pairs"]
    assert R.gemm_layout(28672, 8192, 256) == {"tile_tokens": 256, "per_tile": 1, "ranges": 74, "pairs": True, "blocks": 148, "columns": 256}
    # the calls of few tiles that the GPU tests run, on both sides of the lines
    for out, in_, m, parts in [(100, 2080, 20, 9), (40, 20000, 17, 23), (40, 65536, 17, 43), (300, 4128, 40, 7), (1000, 16384, 30, 16),
                               (2500, 4128, 100, 5), (130, 8192, 128, 6), (250, 2048, 64, 2), (600, 8224, 200, 6), (2048, 2048, 128, 2),
                               (4096, 4096, 256, 2), (512, 1024, 32, 1)]:
        assert R.gemm_layout(out, in_, m, 148)["per_tile"] == parts or wide, (out, in_, m)
    lib = L.load()
    assert lib.rstq_gemm_layout(None, 4096, 4096, 64, 148, 0) == L.E_INVALID
    v = (C.c_int64 * 6)()
    assert lib.rstq_gemm_layout(v, 4096, 100, 64, 148, 0) == L.E_SHAPE
    assert lib.rstq_gemm_layout(v, 4096, 4096, 64, 148, 7) == L.E_INVALID


def test_pairs_of_sms_take_no_more_waves_than_single_ones():
    """Whole 256-token tiles run on pairs only where their number, feature tiles rounded up to two, needs no wave more."""
    from raster_b200 import runtime as R
    for out, in_, m in [(6272, 11008, 768), (6145, 10752, 600), (2688, 10752, 1792), (3712, 11008, 1280), (4736, 10752, 1024),
                        (4736, 5120, 2048), (6272, 5632, 1536), (28672, 1056, 2048), (28280, 2112, 1177)]:
        v = R.gemm_layout(out, in_, m)
        assert v["tile_tokens"] == 256 and not v["pairs"]
    for out, in_, m in [(28672, 8192, 256), (8192, 28672, 256), (4096, 8192, 2048), (7168, 16384, 512), (5968, 5824, 1500), (2400, 14464, 1410)]:
        assert R.gemm_layout(out, in_, m)["pairs"]
    for out in range(1100, 28672, 331):
        for in_ in (1056, 4096, 8192, 16384):
            for m in (200, 256, 512, 700, 1024, 1500, 2048):
                v = R.gemm_layout(out, in_, m)
                if v["pairs"] and not v["ranges"]:
                    ft, tt = -(-out // 128), -(-m // 256)
                    assert -(-(-(-ft // 2) * tt) // 74) <= -(-ft * tt // 148)


def test_decode_plan_is_host_arithmetic_and_always_fits_shared_memory():
    """rstq_decode_plan needs no device: what the first decode launch of a call would be.  One token keeps its
    activations resident; several tokens of MODE_A8 ride the weight ring in one launch whatever K is (three
    stages up to 8 tokens, two at 9 .. 16); MODE_F rides the ring where the staged terms do not fit (up to 16
    columns of terms), else takes fewer tokens.  Over a sweep of shapes and token counts the plan never asks
    for more than the 227 KB of dynamic shared memory a thread block can have, nor for fewer than two stages."""
    import ctypes as C
    from raster_b200 import _lib as L
    lib = L.load()
    plan = (C.c_int32 * 6)()

    def of(mode, bits, out, in_, m, act=L.F32, sm=148):
        L.check(lib.rstq_decode_plan(plan, mode, bits, out, in_, m, act, sm))
        return {"tokens": plan[0], "stages": plan[1], "chunk": plan[2], "ring": plan[3], "smem": plan[4], "blocks": plan[5]}
    p = of(L.MODE_A8, 4, 11008, 4096, 1)
    assert (p["tokens"], p["ring"], p["chunk"], p["blocks"]) == (1, 0, 64, 115) and p["stages"] >= 4
    p = of(L.MODE_A8, 4, 8192, 28672, 8)
    assert (p["tokens"], p["ring"], p["stages"], p["chunk"], p["blocks"]) == (8, 1, 3, 64, 128)
    p = of(L.MODE_A8, 4, 28672, 8192, 16)
    assert (p["tokens"], p["ring"], p["stages"]) == (16, 1, 2)
    p = of(L.MODE_A8, 8, 4096, 4096, 4)
    assert (p["tokens"], p["ring"], p["chunk"]) == (4, 1, 32)
    p = of(L.MODE_F, 4, 4096, 11008, 4, L.F32)          # 4 f32 tokens = 8 columns of terms: one launch on the ring
    assert (p["tokens"], p["ring"]) == (4, 1)
    p = of(L.MODE_F, 4, 4096, 11008, 8, L.BF16)
    assert (p["tokens"], p["ring"]) == (8, 1)
    p = of(L.MODE_F, 4, 4096, 4096, 4, L.BF16)          # fits beside the ring: resident
    assert (p["tokens"], p["ring"]) == (4, 0)
    p = of(L.MODE_F, 4, 4096, 11008, 16, L.F32)         # 32 columns of terms: the 8 tokens (16 columns) that ride the ring
    assert (p["tokens"], p["ring"], p["chunk"]) == (8, 1, 32)
    p = of(L.MODE_A8, 4, 4096, 65536, 1)                # one token of a row too long to stay resident: the ring serves it
    assert (p["tokens"], p["ring"]) == (1, 1)
    for mode in (L.MODE_A8, L.MODE_F):
        for bits in (4, 8):
            for in_ in (32, 256, 4096, 8192, 11008, 16384, 28672, 65536):
                for m in (1, 2, 3, 5, 8, 9, 12, 16, 40):
                    for act in (L.F32, L.BF16):
                        p = of(mode, bits, 4096, in_, m, act)
                        assert 1 <= p["tokens"] <= min(m, 16)
                        assert p["stages"] >= 2 and 16 <= p["chunk"] <= 64
                        assert 0 < p["smem"] <= 231424, (mode, bits, in_, m, act, p)
                        assert 1 <= p["blocks"] <= 148
                        if mode == L.MODE_A8 and m > 1:
                            assert p["ring"] == 1 and p["tokens"] == min(m, 16)
    assert lib.rstq_decode_plan(plan, L.MODE_A8, 4, 4096, 100, 1, L.F32, 148) == L.E_SHAPE
    assert lib.rstq_decode_plan(plan, 7, 4, 4096, 4096, 1, L.F32, 148) == L.E_INVALID
    assert lib.rstq_decode_plan(None, L.MODE_A8, 4, 4096, 4096, 1, L.F32, 148) == L.E_INVALID
