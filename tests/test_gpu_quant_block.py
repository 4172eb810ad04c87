"""The block quantizer's two arithmetics (f32 with a tie check, double).

Codes, scales and sums are the oracle's bit for bit wherever the f32 arithmetic hands over to the double one: a
maximum of zero, tiny, huge; elements on and next to every k + 0.5.
"""
import numpy as np
import pytest

from oracle import oracle as orc
from raster_b200 import Context

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
