"""Outputs that overlap the activations they are computed from."""
import pytest
import torch

from bitween_b200.kernels import _lib
from bitween_b200.kernels.cuda_loader import quantized_matmul_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(N, K, bits, g, gen):
    q = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), generator=gen, device=DEV, dtype=torch.int32)
    s = (torch.rand(N, K // g, generator=gen, device=DEV) * 0.02 + 0.001).half()
    return q, s, torch.randint(0, 2 ** bits, (N, K // g), generator=gen, device=DEV).half()


@pytest.mark.parametrize("tokens", [1, 3, 8, 12, 30, 48, 200])
@pytest.mark.parametrize("N,K,g", [(1024, 1024, 128), (1408, 1408, 128), (28672, 512, 64), (300, 4096, 16), (96, 120, 30)])
def test_out_may_overlap_x(tokens, N, K, g):
    gen = torch.Generator(device=DEV).manual_seed(tokens + N + K)
    layer = _layer(N, K, 4, g, gen)
    for shift in (0, K, 3):                            # the same start, a row further, off a 16-byte boundary
        buf = torch.zeros(tokens * max(N, K) + shift, dtype=torch.float16, device=DEV)
        x, out = buf[:tokens * K].view(tokens, K), buf[shift:shift + tokens * N].view(tokens, N)
        x0 = torch.randn(tokens, K, generator=gen, device=DEV).half()
        want = quantized_matmul_cuda(x0, *layer, None, 4, g)
        for _ in range(5):
            x.copy_(x0)
            got = quantized_matmul_cuda(x, *layer, None, 4, g, out=out)
            assert got.data_ptr() == out.data_ptr() and torch.equal(got, want)


@pytest.mark.parametrize("tokens", [1, 3, 8])
def test_layouts_of_the_cluster_kernel_in_place_through_the_c_entry(tokens):
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    K = 1408                                           # 11 groups a row
    layer = _layer(K, K, 4, 128, gen)
    x0 = torch.randn(tokens, K, generator=gen, device=DEV).half()
    want = quantized_matmul_cuda(x0, *layer, None, 4, 128)
    assert _lib.last_kernel() == "qmm_rows_kernel"
    L, x = _lib.lib(), x0.clone()
    ws = torch.empty(L.bw_qmatmul_workspace_bytes(tokens, K, K, 4, 128), dtype=torch.uint8, device=DEV)
    rc = L.bw_qmatmul(x.data_ptr(), _lib.F16, tokens, K, K, *(t.data_ptr() for t in layer), None, x.data_ptr(), _lib.F16, 4, 128,
                      ws.data_ptr(), ws.numel(), _lib.raw_stream(x.device))
    assert rc == 0 and _lib.last_kernel() == "qmm_smallm_kernel"
    # (sums in another order: one rounding to fp16, and a few of partial sums in fp32)
    slack = 2.0 ** -10 * want.float().abs() + 1e-4 * float(want.float().abs().max())
    assert bool(((x.float() - want.float()).abs() <= slack).all())
