"""Calls of at most 32 tokens that the row and panel kernels leave to the ring and the cluster kernel, against float64, by
the name of the kernel that ran; and graphs side by side for each kernel that keeps something in the scratch."""
import pytest
import torch

from bitween_b200 import dequantize_rtn
from bitween_b200.kernels import _lib
from bitween_b200.kernels.cuda_loader import quantized_matmul_cuda, quantized_matmul_noalloc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(N, K, bits, g, gen):
    q = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), generator=gen, device=DEV, dtype=torch.int32)
    s = (torch.rand(N, K // g, generator=gen, device=DEV) * 0.02 + 0.001).half()
    return q, s, torch.randint(0, 2 ** bits, (N, K // g), generator=gen, device=DEV).half()


def _without_scratch(x, q, s, z, b, bits, g, out):
    rc = _lib.lib().bw_qmatmul(x.data_ptr(), _lib.dtype_code(x.dtype), x.shape[0], q.shape[0], x.shape[1], q.data_ptr(), s.data_ptr(), z.data_ptr(),
                               b.data_ptr(), out.data_ptr(), _lib.dtype_code(out.dtype), bits, g, None, 0, _lib.raw_stream(x.device))
    assert rc == 0
    return out


@pytest.mark.parametrize("how,kernel,bits,g,N,K,tokens", [
    # ring kernel, at most 8 tokens: 2^25 weights, shared row blocks, rows too long for the row kernel
    ("scratch", "qmm_decode_kernel", 4, 128, 8200, 4096, (7, 8)), ("scratch", "qmm_decode_kernel", 2, 64, 19300, 1024, (1, 2, 8)),
    ("scratch", "qmm_decode_kernel", 4, 128, 19003, 1024, (5, 6, 8)), ("scratch", "qmm_decode_kernel", 4, 64, 19200, 512, (1, 3, 4)),
    ("scratch", "qmm_decode_kernel", 8, 32, 20000, 512, (3, 6)), ("scratch", "qmm_decode_kernel", 4, 128, 70, 32768, (5, 8)),
    # 9 tokens and more: shared row blocks, 2^26 weights of 2 bits, more than 9472 rows
    ("scratch", "qmm_decode_kernel", 4, 128, 19003, 1024, (9, 16, 32)), ("scratch", "qmm_decode_kernel", 2, 128, 8300, 8192, (9, 16)),
    ("scratch", "qmm_decode_kernel", 8, 64, 9600, 1024, (17, 32)),
    # without scratch; scales loaded directly: clusters of 8 and 4, whole row blocks
    ("none", "qmm_decode_kernel", 4, 128, 300, 2048, (9, 32)), ("none", "qmm_decode_kernel", 4, 128, 256, 16512, (9, 32)),
    ("none", "qmm_decode_kernel", 8, 128, 3330, 4480, (9, 32)), ("none", "qmm_decode_kernel", 2, 128, 3330, 10368, (9, 16)),
    ("none", "qmm_decode_kernel", 4, 128, 13400, 1152, (16, 17)),
    # cluster kernel: groups of half a lane's codes
    ("scratch", "qmm_smallm_kernel", 4, 16, 1000, 1312, (1, 8, 9, 16, 17, 32)), ("scratch", "qmm_smallm_kernel", 8, 8, 130, 4112, (1, 8, 12, 32)),
    # short rows of many row blocks, to either kernel; few rows of many activations; above 16 tokens more than 9472 rows, long
    # rows of 56 row blocks
    ("scratch", "qmm_smallm_kernel", 2, 64, 5530, 320, (1, 8)), ("scratch", "qmm_smallm_kernel", 4, 64, 19500, 704, (1, 3)),
    ("scratch", "qmm_smallm_kernel", 8, 32, 14300, 480, (2, 5)), ("scratch", "qmm_decode_kernel", 4, 32, 12222, 256, (1, 8)),
    ("scratch", "qmm_smallm_kernel", 2, 64, 12100, 2432, (7, 8)), ("scratch", "qmm_smallm_kernel", 4, 128, 937, 9600, (7, 8)),
    ("scratch", "qmm_decode_kernel", 4, 128, 9473, 1408, (17, 32)), ("scratch", "qmm_smallm_kernel", 4, 128, 19100, 1408, (17, 32)), ("scratch", "qmm_smallm_kernel", 2, 128, 20100, 384, (9, 16, 24)),
    ("scratch", "qmm_decode_kernel", 4, 128, 7200, 6144, (17, 32)), ("scratch", "qmm_decode_kernel", 4, 32, 4800, 3584, (24,)),
    # and with the scratch that is part of the library
    ("noalloc", "qmm_smallm_kernel", 2, 32, 1100, 2112, (1, 8, 9, 32)), ("noalloc", "qmm_smallm_kernel", 4, 128, 4737, 1408, (3, 16, 24)),
    ("noalloc", "qmm_smallm_kernel", 8, 64, 60, 9280, (2, 13, 30)),
])
def test_ring_and_cluster_kernels_match_float64(how, kernel, bits, g, N, K, tokens):
    gen = torch.Generator(device=DEV).manual_seed(N + K + bits)
    q, s, z = _layer(N, K, bits, g, gen)
    b = torch.randn(N, generator=gen, device=DEV).half()
    w = dequantize_rtn(q, s, z, g, bits=bits).half().double()
    for M in tokens:
        for xdt in (torch.float16, torch.bfloat16):
            x = torch.randn(M, K, generator=gen, device=DEV).to(xdt)
            if how == "scratch":
                y = quantized_matmul_cuda(x, q, s, z, b, bits, g, out_dtype=torch.float32)
            else:
                y = torch.empty(M, N, dtype=torch.float32, device=DEV)
                (_without_scratch if how == "none" else quantized_matmul_noalloc)(x, q, s, z, b, bits, g, y)
            assert _lib.last_kernel() == kernel, (M, xdt, _lib.last_kernel())
            xh = x.half().double()
            ref = xh @ w.T + b.double()
            # fp32 sums: a few roundings of partial sums of the order of |x| . |W|
            slack = 2.0 ** -23 * (K / 16 + 16) * (xh.abs() @ w.abs().T) + 1e-6
            assert bool(((y.double() - ref).abs() <= slack).all()), (M, xdt, float((y.double() - ref).abs().max()))
    assert _lib.lib().bw_device_status() == 0


@pytest.mark.parametrize("kernel,M,N,K,g,xdt", [
    ("qmm_panel_kernel", 16, 2048, 4096, 128, torch.float16), ("qmm_panel_kernel", 27, 4800, 1408, 128, torch.bfloat16),
    ("qmm_decode_kernel", 5, 19200, 1024, 128, torch.float16),          # shares in the scratch, arrival counters
    ("qmm_smallm_kernel", 5, 2048, 1312, 16, torch.float16),            # prepared activations
    ("qmm_rows_kernel", 3, 19200, 2048, 128, torch.float16),
])
def test_graphs_side_by_side(kernel, M, N, K, g, xdt):
    gen = torch.Generator(device=DEV).manual_seed(M)
    layer = _layer(N, K, 4, g, gen)
    xs = [torch.randn(M, K, generator=gen, device=DEV).to(xdt) for _ in range(2)]
    want = [quantized_matmul_cuda(x, *layer, None, 4, g) for x in xs]
    graphs, outs = [], []
    for x in xs:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs.append([quantized_matmul_cuda(x, *layer, None, 4, g) for _ in range(12)])
        assert _lib.last_kernel() == kernel
        graphs.append(graph)
    streams = [torch.cuda.Stream() for _ in graphs]
    torch.cuda.synchronize()
    for _ in range(10):
        for y in outs[0] + outs[1]:
            y.zero_()
        torch.cuda.synchronize()
        for _ in range(3):
            for graph, st in zip(graphs, streams):
                with torch.cuda.stream(st):
                    graph.replay()
        eager = [quantized_matmul_cuda(x, *layer, None, 4, g) for x in xs]
        torch.cuda.synchronize()
        for out, y, ref in zip(outs, eager, want):
            assert torch.equal(y, ref) and all(torch.equal(o, ref) for o in out)
    assert _lib.lib().bw_device_status() == 0
