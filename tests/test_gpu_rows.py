"""The kernels for at most 8 and for 9 to 32 tokens: edges of their row tiles, k-chunks, warps' k ranges and constant
tables, against float64."""
import pytest
import torch

from bitween_b200 import dequantize_rtn
from bitween_b200.kernels import _lib
from bitween_b200.kernels.cuda_loader import quantized_matmul_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(N, K, bits, g, gen, offset=0):
    q = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), generator=gen, device=DEV, dtype=torch.int32)
    flat = torch.empty(2, N * (K // g) + offset, dtype=torch.float16, device=DEV)
    s, z = (t[offset:].view(N, K // g) for t in flat)
    s.copy_(torch.rand(N, K // g, generator=gen, device=DEV) * 0.02 + 0.001)
    z.copy_(torch.randint(0, 2 ** bits, (N, K // g), generator=gen, device=DEV))
    return q, s, z


@pytest.mark.parametrize("bits,g,N,K,offset", [
    # one vector of codes; a chunk and a vector; odd numbers of groups; fewer chunks than warps
    (4, 32, 1, 32, 0), (4, 32, 15, 160, 0), (8, 16, 17, 16, 0), (8, 16, 33, 80, 0), (2, 64, 16, 64, 0), (2, 64, 31, 320, 0),
    # several row tiles a CTA with a ragged last one (more than 2 * 148 * 16 rows), ragged last k range
    (4, 128, 4737, 1408, 0), (8, 32, 4750, 608, 0), (2, 128, 9490, 1152, 0), (4, 64, 14208, 512, 0), (4, 64, 14209, 576, 0),
    # groups wider and narrower than a chunk; 2 bits with two groups in a lane's vector; many groups a warp
    (4, 512, 100, 2048, 0), (8, 256, 70, 2304, 0), (2, 32, 50, 1088, 0), (2, 32, 4800, 2112, 0), (2, 512, 48, 5632, 0), (4, 32, 200, 11008, 0),
    # more row blocks than SMs
    (4, 128, 19203, 1024, 0), (8, 64, 24576, 1024, 0),
    # scales and zero points off a 4-byte boundary
    (4, 128, 300, 2048, 1), (8, 64, 90, 1216, 3),
    # long rows: 16 warps, the longest that fit
    (4, 128, 64, 14336, 0), (8, 128, 40, 28672, 0), (2, 128, 24, 65536, 0),
])
def test_rows_kernel_matches_float64(bits, g, N, K, offset):
    gen = torch.Generator(device=DEV).manual_seed(N + K + bits)
    q, s, z = _layer(N, K, bits, g, gen, offset)
    b = torch.randn(N, generator=gen, device=DEV).half()
    w = dequantize_rtn(q, s.contiguous(), z.contiguous(), g, bits=bits).half().double()
    ran = 0
    for M in (1, 2, 3, 5, 8):
        for xdt in (torch.float16, torch.bfloat16, torch.float32):
            x = torch.randn(M, K, generator=gen, device=DEV).to(xdt)
            y = quantized_matmul_cuda(x, q, s, z, b if M % 2 else None, bits, g, out_dtype=torch.float32)
            ran += _lib.last_kernel() == "qmm_rows_kernel"
            assert _lib.last_kernel() == "qmm_rows_kernel" or M * K > 80000 or (M > 4 and N > 148 * 128), (M, xdt, _lib.last_kernel())
            xh = x.half().double()
            ref = xh @ w.T + (b.double() if M % 2 else 0.0)
            # fp32 sums: a few roundings of partial sums of the order of |x| . |W|
            slack = 2.0 ** -23 * (K / 16 + 16) * (xh.abs() @ w.abs().T) + 1e-6
            assert bool(((y.double() - ref).abs() <= slack).all()), (M, xdt, float((y.double() - ref).abs().max()))
            assert torch.equal(y, quantized_matmul_cuda(x, q, s, z, b if M % 2 else None, bits, g, out_dtype=torch.float32))
    assert ran >= 3


@pytest.mark.parametrize("bits,g,N,K,offset", [
    # 16 rows a CTA, 16 warps: less than a chunk, ragged chunks, odd groups, groups wider and narrower than a chunk
    (4, 32, 1, 32, 0), (8, 16, 33, 80, 0), (2, 64, 31, 320, 0), (4, 128, 2368, 1408, 0), (2, 32, 50, 1088, 0), (8, 256, 70, 2304, 0), (4, 32, 200, 11008, 0),
    # 16 rows and 8 warps or 32 rows; 32 or 64 rows, long rows; 64 or 32 rows: ragged last tiles
    (4, 128, 2369, 1408, 0), (8, 32, 2400, 608, 0), (2, 32, 4736, 1152, 0), (4, 64, 4737, 576, 0), (8, 128, 4750, 1280, 0), (2, 128, 4800, 9344, 0),
    (4, 128, 9472, 1408, 0), (4, 32, 9473, 672, 0), (8, 64, 9500, 448, 0), (2, 64, 19000, 448, 0),
    # 96 rows a CTA
    (4, 512, 9490, 1536, 0), (8, 64, 9505, 1600, 0), (2, 32, 14208, 448, 0),
    # scales and zero points off a 4-byte boundary
    (4, 128, 300, 2048, 1), (8, 64, 4790, 1216, 3),
])
def test_panel_kernel_matches_float64(bits, g, N, K, offset):
    gen = torch.Generator(device=DEV).manual_seed(N + K + bits)
    q, s, z = _layer(N, K, bits, g, gen, offset)
    b = torch.randn(N, generator=gen, device=DEV).half()
    w = dequantize_rtn(q, s.contiguous(), z.contiguous(), g, bits=bits).half().double()
    ran = 0
    for M, xdt in ((9, torch.float16), (16, torch.bfloat16), (13, torch.float32), (17, torch.float16), (32, torch.float32), (25, torch.bfloat16)):
        x = torch.randn(M, K, generator=gen, device=DEV).to(xdt)
        y = quantized_matmul_cuda(x, q, s, z, b if M % 2 else None, bits, g, out_dtype=torch.float32)
        ran += _lib.last_kernel() == "qmm_panel_kernel"
        xh = x.half().double()
        ref = xh @ w.T + (b.double() if M % 2 else 0.0)
        slack = 2.0 ** -23 * (K / 16 + 16) * (xh.abs() @ w.abs().T) + 1e-6
        assert bool(((y.double() - ref).abs() <= slack).all()), (M, xdt, float((y.double() - ref).abs().max()))
        assert torch.equal(y, quantized_matmul_cuda(x, q, s, z, b if M % 2 else None, bits, g, out_dtype=torch.float32))
    # (above 16 tokens the ring kernel keeps the wide layers of its layouts)
    assert ran == 6 or (ran == 3 and N > 9472)


def test_panel_kernel_without_scratch_leaves_the_call_to_the_ring_kernel():
    gen = torch.Generator(device=DEV).manual_seed(3)
    L = _lib.lib()
    for K, rc in ((1024, 0), (1408, _lib.ERR_WORKSPACE)):
        q, s, z = _layer(256, K, 4, 128, gen)
        x = torch.randn(12, K, generator=gen, device=DEV).half()
        want = quantized_matmul_cuda(x, q, s, z, None, 4, 128)
        assert _lib.last_kernel() == "qmm_panel_kernel"
        out = torch.zeros_like(want)
        got = L.bw_qmatmul(x.data_ptr(), _lib.F16, 12, 256, K, q.data_ptr(), s.data_ptr(), z.data_ptr(), None, out.data_ptr(), _lib.F16,
                           4, 128, None, 0, _lib.raw_stream(x.device))
        assert got == rc
        if rc == 0:
            assert _lib.last_kernel() == "qmm_decode_kernel"
            assert float((out.float() - want.float()).abs().max()) <= 2.0 ** -10 * float(want.float().abs().max())


@pytest.mark.parametrize("tokens,kernel", [(3, "qmm_rows_kernel"), (12, "qmm_panel_kernel"), (30, "qmm_panel_kernel")])
def test_calls_that_feed_each_other(tokens, kernel):
    # each call reads what the one before has just written, in place and in a graph: weights are requested before the
    # wait for the preceding kernel, activations and the residual after it
    gen = torch.Generator(device=DEV).manual_seed(7)
    layers = [_layer(1024, 1024, 4, 128, gen) for _ in range(6)]
    layers = [(q, s * 0.2, z) for q, s, z in layers]
    h0 = torch.randn(tokens, 1024, generator=gen, device=DEV).half()

    def run(h):
        for q, s, z in layers:
            quantized_matmul_cuda(h, q, s, z, None, 4, 128, residual=h.clone(), out=h)
            assert _lib.last_kernel() == kernel
        return h

    want = h0.clone()
    for q, s, z in layers:
        torch.cuda.synchronize()
        want = want + quantized_matmul_cuda(want, q, s, z, None, 4, 128)
    h = h0.clone()
    assert torch.equal(run(h), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(h)
    for _ in range(20):
        h.copy_(h0)
        graph.replay()
        assert torch.equal(h, want)
