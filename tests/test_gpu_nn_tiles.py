"""The dense layers' row pipelines at their edges against the FP32 reference of test_gpu_nn: one row, the
64-row stage of the weight gradients, and rings that wrap with a ragged last tile; and a gradient call
whose waits run out."""
import pytest
import torch

from cabanadem_b200 import _lib, api, nn
from test_gpu_nn import _check_layer, _sources

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kin,nout", nn.SHAPES)
@pytest.mark.parametrize("rows", [1, 64, 65, 128, 129, 3 * 148 * 128 + 70])
def test_layer_at_tile_edges(kin, nout, rows):
    _check_layer(kin, nout, rows, resid_src0=False)


@pytest.mark.parametrize("kin,nout", [(128, 128), (256, 128), (128, 16)])
def test_gradient_wait_that_runs_out_is_reported(kin, nout):
    dev = torch.device("cuda:0")
    ctx = api.Context(0)
    gen = torch.Generator().manual_seed(5)
    rows = 2 * 148 * 128 + 9
    L = _lib.lib()
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream_ptr())):
        m = nn.Mlp(kin, nout, dev, gen)
        srcs = _sources(kin, rows, gen, dev)
        h1 = torch.empty(rows, 128, device=dev, dtype=torch.bfloat16)
        m.forward(ctx, rows, srcs, h1=h1)
        dy = torch.randn(rows, nout, generator=gen).to(dev, torch.bfloat16)
        dz1 = torch.empty(rows, 128, device=dev, dtype=torch.bfloat16)
        dx = torch.empty(rows, kin, device=dev, dtype=torch.float32)
        m.zero_grad()
        m.backward(ctx, rows, srcs, dy, h1, dz1, dx=dx)
        want = [g.clone() for g in m.grads] + [dx.clone()]
        assert nn.status(ctx) == 0
        assert L.dem_nn_debug_waits(ctx.h, 1000, 1) == 0
        try:
            m.backward(ctx, rows, srcs, dy, h1, dz1, dx=dx)
            assert nn.status(ctx) == 0x020           # DEM_ERR_TIMEOUT
        finally:
            assert L.dem_nn_debug_waits(ctx.h, 0, 0) == 0
        m.zero_grad()
        m.backward(ctx, rows, srcs, dy, h1, dz1, dx=dx)
        assert nn.status(ctx) == 0
        for g, w in zip(list(m.grads) + [dx], want):
            assert torch.equal(g, w)
    ctx.close()
