"""Device memory that outlives a call: what is kept, what is given back, and what a recorded graph may still name."""
import threading

import numpy as np
import pytest
import torch

from raster_b200 import Context
from raster_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    c = Context(("cuda:0",))
    yield c
    c.close()


def test_binding_while_a_graph_is_alive_holds_no_outgrown_staging_blocks(ctx):
    """Matrices in turn below and above the size whose staging block is kept (64 MB): the block that the larger one
    outgrows goes back at once, for no graph names it."""
    rng = np.random.default_rng(0)
    arrays = {n: (rng.integers(0, 256, n * n, dtype=np.uint8), np.full(n * n // 32, 0.01, np.float32)) for n in (7168, 9216)}
    small = ctx.bind_weight(arrays[7168][0][:64 * 64], arrays[7168][1][:128], 64, 64, L.FMT_Q8_0, L.LAYOUT_ROWMAJOR)
    bx, by = ctx.make_buffer(64, np.float32), ctx.make_buffer(64, np.float32)
    bx.fill_bytes(0)
    ctx.qmatmul(small, bx, by, 1)
    ctx.graph_begin()
    ctx.qmatmul(small, bx, by, 1)
    g = ctx.graph_end()
    free = []
    for _ in range(4):
        for n in (7168, 9216):
            ctx.bind_weight(*arrays[n], n, n, L.FMT_Q8_0, L.LAYOUT_ROWMAJOR).free()
        ctx.sync()
        free.append(torch.cuda.mem_get_info()[0])
    g.destroy()
    for b in (small, bx, by):
        b.free()
    assert free[0] - free[-1] < 32 << 20, free


def dx_case(ctx, seed, m, in_, out):
    rng = np.random.default_rng(seed)
    a = (rng.standard_normal(m * out).astype(np.float32), rng.integers(-127, 128, out * in_).astype(np.int8),
         rng.uniform(0.01, 0.02, out * in_ // 32).astype(np.float32))
    bufs = [ctx.array_to_buffer(x) for x in a] + [ctx.make_buffer(m * in_, np.float32)]
    d = a[0].reshape(m, out).astype(np.float64)
    return bufs, d @ (a[1].reshape(out, in_) * np.repeat(a[2].reshape(out, -1).astype(np.float64), 32, axis=1))


def test_backward_recorded_in_a_graph_of_the_caller(ctx):
    """On a lent stream, without a call before it, and replayed after the scratch has grown and its old place (were it
    free) been scribbled on."""
    m, in_, out = 100, 256, 640
    bufs, want = dx_case(ctx, 1, m, in_, out)
    big, _ = dx_case(ctx, 2, 700, in_, out)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    ctx.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.graph(graph, stream=stream):
            ctx.qlinear_q8_dx_device(*bufs, m, in_, out)
        ctx.qlinear_q8_dx_device(*big, 700, in_, out)
        ctx.sync()
        other = [ctx.make_buffer(1 << 20, np.uint8) for _ in range(4)]
        for b in other:
            b.fill_bytes(0x7F)
        for _ in range(2):
            bufs[3].fill_bytes(0xFF)
            ctx.sync()
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            got = bufs[3].download().reshape(m, in_)
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    finally:
        torch.cuda.synchronize()
        del graph
        ctx.set_stream(None)
    for b in bufs + big + other:
        b.free()


def quant_arrays(n, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, 256, n * n // 2, dtype=np.uint8), (rng.standard_normal(n * n // 32) * 0.01).astype(np.float32)


def dense(codes, scales, n):
    b = codes.reshape(-1, 16)
    return (np.concatenate([b & 15, b >> 4], 1).astype(np.float64) - 8) * scales[:, None].astype(np.float64)


def test_an_array_that_serves_the_next_weight_of_its_size_holds_that_weight(ctx):
    """A weight takes the place of one that is gone, with a product of the old one still under way when that is freed; one of
    another size does not, and two alive at once have an array each."""
    n = 2048
    x = np.random.default_rng(1).standard_normal(n).astype(np.float32)
    bx = ctx.array_to_buffer(x)
    w, ys = None, []
    for seed in range(6):
        a = quant_arrays(n, seed)
        if w is not None:
            ctx.qmatmul(w, bx, ys[-1][1], 1, L.F32, L.F32, L.MODE_F)
            w.free()                                  # waits for the product
        w = ctx.bind_weight(*a, n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
        ys.append((a, ctx.make_buffer(n, np.float32)))
    other = ctx.bind_weight(*quant_arrays(1024, 9), 1024, 1024, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
    twin = ctx.bind_weight(*ys[0][0], n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
    ctx.qmatmul(w, bx, ys[-1][1], 1, L.F32, L.F32, L.MODE_F)
    ctx.sync()
    for a, by in ys:
        ref = dense(*a, n).reshape(n, n) @ x.astype(np.float64)
        assert np.abs(by.download() - ref).max() <= 2e-5 * np.abs(ref).max()
    for b in (w, other, twin, bx, *(y for _, y in ys)):
        b.free()


def test_arrays_of_weights_that_are_gone_are_bounded_and_go_with_the_context():
    torch.cuda.synchronize()
    c = Context(("cuda:0",))
    try:
        c.bind_weight(*quant_arrays(512, 0), 512, 512, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR).free()
        start = torch.cuda.mem_get_info()[0]
        for n in (4096, 4224, 4352, 4480, 4608, 4736, 4864, 4992, 5120, 8192, 14336):   # 10 .. 129 MB
            c.bind_weight(*quant_arrays(n, n), n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR).free()
        # at most 64 MB of arrays and 64 MB of staging stay, in allocations of 2 MB
        assert start - torch.cuda.mem_get_info()[0] <= (64 + 64 + 32) << 20
    finally:
        before = torch.cuda.mem_get_info()[0]
        c.close()
    assert torch.cuda.mem_get_info()[0] - before >= 40 << 20


@pytest.mark.parametrize("where", ["this thread", "another thread"])
def test_a_weight_is_freed_while_the_caller_captures_elsewhere(where):
    """The caller records a graph of their own (relaxed mode) on a stream that the context knows nothing of; freeing a weight and
    binding the next one meanwhile leaves it intact."""
    c = Context(("cuda:0",))
    try:
        w = c.bind_weight(*quant_arrays(512, 0), 512, 512, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
        x = c.array_to_buffer(np.ones(512, np.float32))
        y = c.make_buffer(512, np.float32)
        a = torch.zeros(64, device="cuda")
        graph, done = torch.cuda.CUDAGraph(), []

        def swap():
            c.qmatmul(w, x, y, 1, L.F32, L.F32, L.MODE_F)
            w.free()
            done.append(1)

        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            graph.capture_begin(capture_error_mode="relaxed")
            a.add_(1)
            if where == "this thread":
                swap()
            else:
                t = threading.Thread(target=swap)
                t.start()
                t.join()
            a.add_(1)
            graph.capture_end()
        graph.replay()
        torch.cuda.synchronize()
        assert done == [1] and a.eq(2).all()
        ref = dense(*quant_arrays(512, 0), 512).reshape(512, 512).sum(1)
        assert np.abs(y.download() - ref).max() <= 2e-5 * np.abs(ref).max()
    finally:
        c.close()


def test_arrays_are_not_kept_once_a_stream_was_lent():
    """On a stream of the caller's a graph that names the weight may be in flight: its array goes to cudaFree, which waits."""
    c = Context(("cuda:0",))
    try:
        n = 4096
        c.bind_weight(*quant_arrays(n, 0), n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR).free()
        with torch.cuda.stream(torch.cuda.Stream()):
            c.set_stream(torch.cuda.current_stream().cuda_stream)
            w = c.bind_weight(*quant_arrays(n, 1), n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
            before = torch.cuda.mem_get_info()[0]
            w.free()
            assert torch.cuda.mem_get_info()[0] - before >= 8 << 20
            c.set_stream(None)
    finally:
        c.close()


@pytest.mark.parametrize("who", ["buffer", "backward"])
def test_kept_arrays_are_given_back_before_an_allocation_fails(who):
    """An allocation that the device cannot hold is an error, not before the arrays kept for weights to come are free again; the
    backward call fails on its scratch (10 bytes per element of dy), ahead of any launch."""
    c = Context(("cuda:0",))
    try:
        n = 8192
        a = c.make_buffer(1 << 20, np.float32)
        c.bind_weight(*quant_arrays(n, 0), n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR).free()     # 42 MB
        before = torch.cuda.mem_get_info()[0]
        if who == "buffer":
            with pytest.raises(L.RstqError):
                c.make_buffer(1 << 40, np.uint8)
        else:
            m, out = 1 << 20, 1 << 15
            dy = c.wrap_buffer(a.device_ptr, m * out, np.float32)
            codes, scales = c.wrap_buffer(a.device_ptr, out * 32, np.int8), c.wrap_buffer(a.device_ptr, out, np.float32)
            dx = c.wrap_buffer(a.device_ptr, m * 32, np.float32)
            with pytest.raises(L.RstqError):
                c.qlinear_q8_dx_device(dy, codes, scales, dx, m, 32, out)
        assert torch.cuda.mem_get_info()[0] - before >= 40 << 20
    finally:
        c.close()


def test_arrays_of_sizes_that_do_not_come_back_make_room():
    """64 MB of other sizes are held; a size that comes again is kept and serves the next one all the same."""
    c = Context(("cuda:0",))
    try:
        def bind(n):
            return c.bind_weight(*quant_arrays(n, n), n, n, L.FMT_Q4_0, L.LAYOUT_ROWMAJOR)
        bind(8192).free()                                          # 42 MB, and the staging
        bind(5632).free()                                          # 20 MB: 62 of 64 MB are held
        bind(4096).free()                                          # 10 MB
        before = torch.cuda.mem_get_info()[0]
        w = bind(4096)
        assert torch.cuda.mem_get_info()[0] == before              # (it took the array that was kept)
        w.free()
        assert torch.cuda.mem_get_info()[0] == before              # (and gave it back to be kept)
    finally:
        c.close()
