"""Device memory that outlives a call: what is kept, what is given back, and what a recorded graph may still name."""
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
