"""The backward-data GEMM at the edges of its tiles, stages and clusters, against the f64 product."""
import numpy as np
import pytest

from raster_b200 import Context

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(("cuda:0",))
    yield c
    c.close()


def run(ctx, m, in_, out, dy, codes, scales):
    bufs = [ctx.array_to_buffer(a) for a in (dy, codes, scales)] + [ctx.make_buffer(m * in_, np.float32)]
    bufs[3].fill_bytes(0xFF)
    ctx.qlinear_q8_dx_device(*bufs, m, in_, out)
    ctx.sync()
    dx = bufs[3].download().reshape(m, in_).astype(np.float64)
    for b in bufs:
        b.free()
    return dx


def check(ctx, m, in_, out, dy, codes, scales):
    dx = run(ctx, m, in_, out, dy, codes, scales)
    w = codes.reshape(out, in_).astype(np.float64) * np.repeat(scales.reshape(out, in_ // 32).astype(np.float64), 32, axis=1)
    d = dy.reshape(m, out).astype(np.float64)
    # Per product: code * scale is rounded to f32 (2^-24), both factors are then held whole, and what the six products of
    # their terms leave out is at most 2 * 2^-8 * 2^-17 of it.  Per sum: 16 products at a time are added to an f32, twice
    # (first and second terms), each addition off by at most 2^-23 of the sum of magnitudes; up to 8 partial sums and
    # two scalings follow.
    bound = (2 * 2.0 ** -24 + (out / 8 + 12) * 2.0 ** -23) * (np.abs(d) @ np.abs(w))
    assert np.all(np.abs(dx - d @ w) <= bound)
    assert np.abs(dx - d @ w).max() <= 2e-5 * np.abs(d @ w).max() + 1e-300


# m: around the 32 / 64 / 128-token tiles; in: one block, a ragged tile of 128 columns; out: one row, ragged
# groups of 16 and 64 rows, split over 1, 2, 4 and 8 blocks of a cluster
@pytest.mark.parametrize("m,in_,out", [(1, 32, 1), (3, 96, 15), (15, 160, 65), (32, 128, 64), (33, 128, 200), (64, 288, 1024),
                                       (65, 256, 1000), (128, 512, 513), (129, 4096, 640), (300, 1056, 2048), (257, 2048, 129),
                                       (16, 4096, 4096), (20, 96, 9001)])
def test_dx_at_the_edges(ctx, m, in_, out):
    rng = np.random.default_rng(m * in_ + out)
    check(ctx, m, in_, out, rng.standard_normal(m * out).astype(np.float32),
          rng.integers(-128, 128, out * in_).astype(np.int8),
          (rng.standard_normal(out * in_ // 32) * 0.01).astype(np.float32))


@pytest.mark.parametrize("m,in_,out", [(40, 256, 320), (20, 256, 2048)])   # whole tiles, tiles shared by a cluster
@pytest.mark.parametrize("row,col", [(1e-41, 1.0), (1e30, 1e-30), (1e-20, 1e15), (1e34, 1e-36), (1e-36, 1e34), (1e-30, 1e30),
                                     (1e-41, 1e34), (1e34, 1e-41)])
def test_dx_keeps_rows_and_column_blocks_of_any_magnitude(ctx, row, col, m, in_, out):
    """A token row and a column block far above or below the rest keep their own relative precision."""
    rng = np.random.default_rng(5)
    dy = (rng.uniform(0.5, 1, (m, out)) * rng.choice([-1, 1], (m, out))).astype(np.float32)
    dy[7] *= np.float32(row)
    scales = rng.uniform(0.5, 1, (out, in_ // 32)).astype(np.float32)
    scales[:, 3] *= np.float32(col)
    codes = rng.integers(-127, 128, (out, in_)).astype(np.int8)
    dx = run(ctx, m, in_, out, dy.ravel(), codes.ravel(), scales.ravel())
    w = codes.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, axis=1)
    want = dy.astype(np.float64) @ w
    for rows in (slice(7, 8), slice(8, None)):
        for cols in (slice(96, 128), slice(128, None)):
            a, b = dx[rows, cols], want[rows, cols]
            # 2e-5 as above, and half a step of the subnormal grid of the result
            assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max() + 1.5e-45 * (1 if np.abs(b).max() < 1e-37 else 0)


@pytest.mark.parametrize("m,in_,out", [(8, 96, 320), (40, 256, 320), (130, 128, 70)])
@pytest.mark.parametrize("below", [12, 24, 40, 90])
@pytest.mark.parametrize("what", ["dy", "scales"])
def test_dx_holds_all_bits_of_small_elements(ctx, what, below, m, in_, out):
    """Elements 2^-below of the largest of their row (scales: of their column block), which meets zeros: what
    remains is the sum of the small ones, with the precision that f32 gives it."""
    rng = np.random.default_rng(below)
    dy = (rng.uniform(0.5, 1, (m, out)) * rng.choice([-1, 1], (m, out))).astype(np.float32)
    scales = rng.uniform(0.5, 1, (out, in_ // 32)).astype(np.float32)
    codes = rng.integers(-127, 128, (out, in_)).astype(np.int8)
    if what == "dy":
        dy[:, 1:] *= np.float32(2.0 ** -below)
        codes[0] = 0
    else:
        scales[1:] *= np.float32(2.0 ** -below)
        dy[:, 0] = 0
    dx = run(ctx, m, in_, out, dy.ravel(), codes.ravel(), scales.ravel())
    w = codes.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, axis=1)
    d = dy.astype(np.float64)
    assert np.all(np.abs(dx - d @ w) <= (2 * 2.0 ** -24 + (out / 8 + 12) * 2.0 ** -23) * (np.abs(d) @ np.abs(w)))


@pytest.mark.parametrize("m", [3, 40])
def test_dx_of_infinities_and_nans(ctx, m):
    """What f32 arithmetic makes of them: an infinity times a code of zero is a NaN, else an infinity of its sign; other
    rows and other column blocks do not notice."""
    in_, out = 128, 200
    rng = np.random.default_rng(1)
    dy = rng.standard_normal((m, out)).astype(np.float32)
    dy[0, 7], dy[1, 9], dy[2, 70] = np.inf, np.nan, -np.inf
    codes = rng.integers(-127, 128, (out, in_)).astype(np.int8)
    codes[7, ::5] = 0
    scales = rng.uniform(0.25, 0.5, (out, in_ // 32)).astype(np.float32)
    scales[13, 2] = np.inf
    with np.errstate(all="ignore"):
        w = codes.astype(np.float32) * np.repeat(scales, 32, axis=1)
        want = np.stack([(dy[i][:, None] * w).sum(0) for i in range(m)])
    dx = run(ctx, m, in_, out, dy.ravel(), codes.ravel(), scales.ravel())
    assert np.array_equal(np.isnan(dx), np.isnan(want))
    assert np.array_equal(dx[np.isinf(want)], want[np.isinf(want)]) and np.isfinite(dx[np.isfinite(want)]).all()


def test_dx_recorded_without_a_first_call(ctx):
    m, in_, out = 700, 640, 2560      # more scratch than any call before it
    rng = np.random.default_rng(9)
    dy, codes = rng.standard_normal(m * out).astype(np.float32), rng.integers(-127, 128, out * in_).astype(np.int8)
    scales = np.full(out * in_ // 32, 0.01, np.float32)
    bufs = [ctx.array_to_buffer(a) for a in (dy, codes, scales)] + [ctx.make_buffer(m * in_, np.float32)]
    ctx.graph_begin()
    ctx.qlinear_q8_dx_device(*bufs, m, in_, out)
    g = ctx.graph_end()
    g.replay()
    ctx.sync()
    got = bufs[3].download()
    ctx.qlinear_q8_dx_device(*bufs, m, in_, out)
    ctx.sync()
    assert np.array_equal(got, bufs[3].download())
    g.destroy()
    for b in bufs:
        b.free()


@pytest.mark.parametrize("m,in_,out", [(5, 96, 64), (40, 160, 128), (64, 256, 200),              # short sums: triples in any case
                                       (300, 256, 320), (300, 160, 64), (5, 96, 256), (40, 160, 320), (64, 256, 300)])
@pytest.mark.parametrize("what,below", [("dy", 26), ("dy", 27), ("dy", 28), ("scales", 19), ("scales", 20), ("scales", 21)])
def test_dx_pairs_and_triples_on_both_sides_of_the_line(ctx, what, below, m, in_, out):
    """Rows whose smallest element, blocks whose smallest scale lies about where pairs of fp16 stop holding it whole, in
    one token tile beside tiles of plain rows; the small ones alone decide some of the results."""
    rng = np.random.default_rng(below + m)
    dy = (rng.uniform(0.5, 1, (m, out)) * rng.choice([-1, 1], (m, out))).astype(np.float32)
    scales = rng.uniform(0.5, 1, (out, in_ // 32)).astype(np.float32)
    codes = rng.integers(-128, 128, (out, in_)).astype(np.int8)
    if what == "dy":
        dy[m // 2, 1:] *= np.float32(2.0 ** -below)
        codes[0, ::3] = 0
    else:
        scales[1:, -1] *= np.float32(2.0 ** -below)
        dy[::4, 0] = 0
    dx = run(ctx, m, in_, out, dy.ravel(), codes.ravel(), scales.ravel())
    w = codes.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, axis=1)
    d = dy.astype(np.float64)
    # A product of pairs: 6 * 2^-24 for the weight (4 for the rounding of its second term, which may be a little more than
    # half a step of the first, 2 for that of the scale's), 2 * 2^-24 for dy, 6 * 2^-24 for the product of the second terms, left out.
    assert np.all(np.abs(dx - d @ w) <= (14 * 2.0 ** -24 + (out / 8 + 12) * 2.0 ** -23) * (np.abs(d) @ np.abs(w)))


@pytest.mark.parametrize("m,out,units", [(64, 512, 6), (40, 260, 6), (200, 512, 6), (64, 255, 1), (5, 64, 1), (200, 63, 1)])
def test_dx_holds_weights_and_elements_of_dy(ctx, m, out, units):
    """Sums of one term, which round nothing: dy with one 1 per row gives the weights, codes of 1 and scales of 1 in one row
    give the elements of dy back.  A weight as a pair of fp16 is off by 6 * 2^-24 of itself at most (see above), an element of dy by 2;
    short sums are triples, and only the f32 product of code and scale rounds: 1 * 2^-24."""
    in_ = 4096
    rng = np.random.default_rng(out)
    codes = rng.integers(-128, 128, (out, in_)).astype(np.int8)
    scales = np.exp2(rng.uniform(-6, 0, (out, in_ // 32))).astype(np.float32)
    rows = rng.integers(0, out, m)
    dy = np.zeros((m, out), np.float32)
    dy[np.arange(m), rows] = 1
    dx = run(ctx, m, in_, out, dy.ravel(), codes.ravel(), scales.ravel())
    w = (codes.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, axis=1))[rows]
    assert np.all(np.abs(dx - w) <= (units * (1 + 2.0 ** -10) * 2.0 ** -24) * np.abs(w))
    dy = (rng.uniform(0.01, 1, (m, out)) * rng.choice([-1, 1], (m, out))).astype(np.float32)
    codes[:], scales[:] = 0, 1
    codes[rows[0]] = 1
    dx = run(ctx, m, in_, out, dy.ravel(), codes.ravel(), scales.ravel())
    d = dy[:, rows[:1]].astype(np.float64)
    assert np.all(np.abs(dx - d) <= (2 * (1 + 2.0 ** -10) * 2.0 ** -24 if units > 1 else 0) * np.abs(d))
