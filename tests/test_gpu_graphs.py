"""Captured calls: every CUDA graph owns the scratch and the row-block counters of its calls, so graphs may be replayed
beside each other although torch captures all of them on one stream."""
import time

import pytest
import torch

from bitween_b200.kernels import _lib
from bitween_b200.kernels.cuda_loader import quantized_matmul_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(N, K, bits, g, seed=1):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    q = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), generator=gen, device=DEV, dtype=torch.int32)
    s = (torch.rand(N, K // g, generator=gen, device=DEV) * 0.02 + 0.001).half()
    z = torch.randint(0, 2 ** bits, (N, K // g), generator=gen, device=DEV).half()
    return q, s, z


@pytest.mark.parametrize("kernel,M,N,K,bits,g,xdt", [
    ("qmm_decode_kernel", 3, 19200, 2048, 4, 128, torch.float16),      # shares in the scratch, arrival counters
    ("qmm_decode_kernel", 24, 28672, 1024, 4, 128, torch.bfloat16),
    ("qmm_smallm_kernel", 5, 2048, 1408, 4, 128, torch.float16),       # prepared activations in the scratch
    ("qmm_tc_kernel", 48, 2048, 4096, 4, 128, torch.bfloat16),         # cast activations in the scratch
])
def test_graphs_replayed_beside_each_other(kernel, M, N, K, bits, g, xdt):
    layer = _layer(N, K, bits, g)
    gen = torch.Generator(device=DEV).manual_seed(2)
    xs = [torch.randn(M, K, generator=gen, device=DEV).to(xdt) for _ in range(2)]
    want = [quantized_matmul_cuda(x, *layer, None, bits, g) for x in xs]
    assert _lib.last_qmatmul_kernel() == kernel
    graphs, outs = [], []
    for x in xs:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs.append([quantized_matmul_cuda(x, *layer, None, bits, g) for _ in range(12)])
        assert _lib.last_qmatmul_kernel() == kernel
        graphs.append(graph)
    streams = [torch.cuda.Stream() for _ in graphs]
    torch.cuda.synchronize()
    for _ in range(10):
        for out in outs:
            for y in out:
                y.zero_()
        torch.cuda.synchronize()
        for _ in range(3):
            for graph, st in zip(graphs, streams):
                with torch.cuda.stream(st):
                    graph.replay()
        # and calls outside of graphs on a third stream
        eager = [quantized_matmul_cuda(x, *layer, None, bits, g) for x in xs]
        torch.cuda.synchronize()
        for out, y, ref in zip(outs, eager, want):
            assert torch.equal(y, ref)
            assert all(torch.equal(o, ref) for o in out)
    assert _lib.lib().bw_device_status() == 0


def test_counter_slices_are_given_back_with_their_graphs():
    # a layer with more row blocks than SMs (149), a row block shared by two CTAs; 448 slices for captured calls
    bits, g, M, N, K = 4, 64, 2, 149 * 128, 512
    q, s, z = _layer(N, K, bits, g)
    x = torch.randn(M, K, device=DEV).half()
    want = quantized_matmul_cuda(x, q, s, z, None, bits, g)
    gated = quantized_matmul_cuda(x, q, s, z, None, bits, g, activation="silu_mul")
    out, out_gated = torch.empty_like(want), torch.empty_like(gated)
    pool, stream = torch.cuda.graph_pool_handle(), torch.cuda.Stream()

    def capture(activation=None):
        graph = torch.cuda.CUDAGraph()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            graph.capture_begin(pool=pool)
            quantized_matmul_cuda(x, q, s, z, None, bits, g, out=out if activation is None else out_gated, activation=activation)
            quantized_matmul_cuda(x, q, s, z, None, bits, g, out=out if activation is None else out_gated, activation=activation)
            graph.capture_end()
        torch.cuda.current_stream().wait_stream(stream)
        return graph, _lib.last_qmatmul_kernel()

    anchor = capture()                                 # (keeps the pool)
    for _ in range(600):                               # one after the other, each gone before the next
        graph, kernel = capture()
        assert kernel == "qmm_decode_kernel"
        graph.reset()
    live = []
    for _ in range(600):
        live.append(capture())
        if live[-1][1] != "qmm_decode_kernel":
            break
    assert live[-1][1] == "qmm_smallm_kernel" and len(live) > 400      # slices are finite: another kernel takes over
    for graph, _ in (live[0], live[-2], live[-1]):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.allclose(out.float(), want.float(), rtol=2.0 ** -9, atol=1e-5 * float(want.float().abs().max()))
    graph, kernel = capture("silu_mul")                # no other kernel has the gated output stage
    graph.replay()
    torch.cuda.synchronize()
    assert kernel == "qmm_decode_kernel"
    assert torch.allclose(out_gated.float(), gated.float(), rtol=2.0 ** -8, atol=1e-4 * float(gated.float().abs().max()))
    del live, graph
    deadline = time.monotonic() + 20                   # the driver runs the graphs' destructors on a thread of its own
    while True:
        graph, kernel = capture()
        if kernel == "qmm_decode_kernel" or time.monotonic() > deadline:
            break
        time.sleep(0.05)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert kernel == anchor[1] == "qmm_decode_kernel" and torch.equal(out, want)
    assert _lib.lib().bw_device_status() == 0


def test_scratch_of_the_decode_kernel_only_where_row_blocks_are_shared():
    L = _lib.lib()
    for N, K, rc in ((1024, 4096, 0), (148 * 128, 512, 0), (149 * 128, 512, _lib.ERR_WORKSPACE)):
        q, s, z = _layer(N, K, 4, 64)
        x = torch.randn(5, K, device=DEV).half()
        out = torch.zeros(5, N, dtype=torch.float16, device=DEV)
        want = quantized_matmul_cuda(x, q, s, z, None, 4, 64)
        assert _lib.last_qmatmul_kernel() == "qmm_decode_kernel"
        got = L.bw_qmatmul(x.data_ptr(), _lib.F16, 5, N, K, q.data_ptr(), s.data_ptr(), z.data_ptr(), None, out.data_ptr(), _lib.F16,
                           4, 64, None, 0, _lib.raw_stream(x.device))
        assert got == rc and torch.equal(out, want if rc == 0 else torch.zeros_like(want))
    # a layout that runs on the cluster split-K kernel asks for its own scratch
    q, s, z = _layer(64, 1408, 4, 128)
    x = torch.randn(5, 1408, device=DEV).half()
    assert L.bw_qmatmul_workspace_bytes_for(5, 64, 1408, 4, 128, _lib.F16, 16) >= 5 * 1408 * 2
    quantized_matmul_cuda(x, q, s, z, None, 4, 128)
    assert _lib.last_qmatmul_kernel() == "qmm_smallm_kernel"
