"""Calls launched one directly behind the other, each reading what the one before has just written into a buffer that the
call before that has read: programmatic launches overlap their predecessors, and no stale activation may answer."""
import pytest
import torch

from bitween_b200.kernels import _lib
from bitween_b200.kernels.cuda_loader import quantized_matmul_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layers(n, N, K, bits, g, gen):
    made = []
    for _ in range(n):
        q = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), generator=gen, device=DEV, dtype=torch.int32)
        s = ((torch.rand(N, K // g, generator=gen, device=DEV) * 0.02 + 0.001) * 12 / K ** 0.5).half()     # (values keep their size)
        made.append((q, s, torch.randint(0, 2 ** bits, (N, K // g), generator=gen, device=DEV).half()))
    return made


@pytest.mark.parametrize("tokens,K,g,dt,kernel", [
    (3, 2048, 128, torch.float16, "qmm_rows_kernel"), (8, 1024, 64, torch.bfloat16, "qmm_rows_kernel"),
    (12, 2048, 128, torch.float16, "qmm_panel_kernel"), (30, 1408, 128, torch.float32, "qmm_panel_kernel"),
    (5, 512, 16, torch.bfloat16, "qmm_smallm_kernel"),
    (48, 2048, 128, torch.float16, "qmm_tc_kernel"), (48, 2048, 128, torch.bfloat16, "qmm_tc_kernel"), (200, 1024, 128, torch.float32, "qmm_tc_kernel"),
    # casts before 45 clusters of 3 and 26 of 5
    (100, 5760, 128, torch.bfloat16, "qmm_tc_kernel"), (100, 3328, 128, torch.float32, "qmm_tc_kernel"),
])
@pytest.mark.parametrize("residual", [False, True])
def test_two_buffers_in_turn(tokens, K, g, dt, kernel, residual):
    gen = torch.Generator(device=DEV).manual_seed(tokens + K)
    layers = _layers(6, K, K, 4, g, gen) * 4
    x0 = torch.randn(tokens, K, generator=gen, device=DEV).to(dt)
    r0 = torch.randn(tokens, K, generator=gen, device=DEV).half()
    fused = residual and dt == torch.float16

    # with an fp16 residual, each call adds to what its output buffer holds from two calls before
    def run(bufs):
        for i, layer in enumerate(layers):
            out = bufs[(i + 1) % 2]
            quantized_matmul_cuda(bufs[i % 2], *layer, None, 4, g, out_dtype=dt, out=out, residual=out if fused else r0 if residual else None)
            assert _lib.last_kernel() == kernel
        return bufs[len(layers) % 2]

    bufs = [x0, (r0 if fused else torch.zeros_like(x0))]
    for i, layer in enumerate(layers):
        torch.cuda.synchronize()
        bufs[(i + 1) % 2] = quantized_matmul_cuda(bufs[i % 2].clone(), *layer, None, 4, g, out_dtype=dt,
                                                  residual=bufs[(i + 1) % 2].clone() if fused else r0 if residual else None)
    want = bufs[len(layers) % 2]
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 1e-3

    own = [torch.empty_like(x0), torch.empty_like(x0)]
    start = [x0, (r0.to(dt) if fused else torch.zeros_like(x0))]

    def reset():
        for o, s in zip(own, start):
            o.copy_(s)

    for _ in range(5):
        reset()
        assert torch.equal(run(own), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run(own)
    for _ in range(20):
        reset()
        graph.replay()
        assert torch.equal(got, want)
    assert _lib.lib().bw_device_status() == 0
