"""One token of a Q4_K / Q6_K matrix with the activation quantizer inside the decode kernel: bit-identical to the
quantizer kernel followed by the decode kernel."""
import numpy as np
import pytest

from raster_b200 import Context
from raster_b200 import _lib as L
from raster_b200.quant import cpu_quant as cq

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(("cuda:0",))
    yield c
    c.close()


@pytest.mark.parametrize("fmt", ["q4k", "q6k"])
@pytest.mark.parametrize("out,in_", [(8000, 256), (4096, 4096), (1000, 11008), (520, 12288), (520, 12544)])   # 12288: the longest row it takes
def test_fused_quantizer_of_kquants(ctx, fmt, out, in_):
    rng = np.random.default_rng(out)
    W = (rng.standard_normal(out * in_) * 0.02).astype(np.float32)
    w = ctx.bind_weight_q4k(cq.quantize_weight_q4k(W), out, in_) if fmt == "q4k" else \
        ctx.bind_weight_q6k(cq.quantize_weight_q6k(W), out, in_)
    by = ctx.make_buffer(out, np.float32)
    for kind in range(4):
        x = rng.standard_normal(in_).astype(np.float32)
        if kind == 1:
            x[:256] = 0                                            # a super-block of zeros
            x[256:] = np.round(x[256:] * 4) / 8                    # ties
        elif kind == 2:
            x *= np.float32(1e-32)                                 # below the f32 shortcut
        elif kind == 3:
            x[::7] *= np.float32(1e30)
        bx, got = ctx.array_to_buffer(x), {}
        try:
            for fused in (0, 1):
                ctx.tune(L.TUNE_FUSE_QUANT, fused)
                by.fill_bytes(0xFF)
                n0 = ctx.launch_count()
                ctx.qmatmul(w, bx, by, 1)
                ctx.sync()
                assert ctx.launch_count() - n0 == (1 if fused and in_ <= 12288 else 2)
                got[fused] = by.download(np.uint32)
        finally:
            ctx.tune(L.TUNE_FUSE_QUANT, 1)
        assert np.array_equal(got[0], got[1])
        bx.free()
    w.free(), by.free()
