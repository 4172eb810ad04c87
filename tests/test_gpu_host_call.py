"""One-token calls on host arrays: rows whose activations travel as launch parameters (up to 7936) and longer
ones, results below and above what is waited for word by word, against the oracle's operator."""
import numpy as np
import pytest

from oracle import oracle as orc
from raster_b200 import Context
from raster_b200 import _lib as L
from raster_b200.quant import op

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(("cuda:0",))
    yield c
    c.close()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("out,in_", [(8, 32), (40, 4096), (64, 4128), (24, 7936), (24, 7968), (16384, 64), (16392, 64)])
def test_host_call(ctx, bits, out, in_):
    rng = np.random.default_rng(out + in_)
    wq, ws = orc.quantize_weight(rng.standard_normal(out * in_).astype(np.float32), bits)
    wqi, wsi = orc.repack_stream(wq, ws, out, in_, bits, 8)
    fn = op.qlinear_i8 if bits == 4 else op.qlinear_i8_q8
    for _ in range(3):       # the same staging memory, other results
        x = rng.standard_normal(in_).astype(np.float32)
        ref = orc.qlinear_i8(x, wqi, wsi, in_, out, bits)
        # integer dots are exact; each of the in / 32 scaled sums is rounded a few times at 2^-24
        assert np.abs(fn(x, wqi, wsi, in_, out, ctx) - ref).max() <= 4e-6 * np.abs(ref).max()


def test_nan_results_are_returned(ctx):
    """A scale of infinity makes every result a NaN (another one than the pattern that is waited for to go: the wait for
    that is tested in test_host_wait.py)."""
    out, in_ = 64, 256
    codes = np.full(out * in_, 200, np.uint8)
    scales = np.full(out * in_ // 32, np.float32(np.inf))
    w = ctx.bind_weight(codes, scales, out, in_, L.FMT_Q8_0, L.LAYOUT_ROWMAJOR)
    x = np.zeros(in_, np.float32)
    assert np.isnan(ctx.qmatmul_host(w, x)).all()
    w.free()
