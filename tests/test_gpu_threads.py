"""Threads that call on one stream share the stream's scratch: each call reads the activations that it prepared itself."""
import threading

import pytest
import torch

from bitween_b200.kernels import _lib
from bitween_b200.kernels.cuda_loader import quantized_matmul_cuda, quantized_matmul_noalloc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tokens,K,g,xdt,kernel,noalloc", [
    (16, 1024, 128, torch.float16, "qmm_panel_kernel", False),
    (12, 1408, 128, torch.bfloat16, "qmm_panel_kernel", False),
    (8, 512, 16, torch.float16, "qmm_smallm_kernel", False),       # groups of half a lane's codes: the cluster kernel
    (48, 1024, 128, torch.bfloat16, "qmm_tc_kernel", False),       # cast, then GEMM
    (16, 1024, 128, torch.float16, "qmm_smallm_kernel", True),     # the scratch that is part of the library
])
def test_two_threads_on_one_stream(tokens, K, g, xdt, kernel, noalloc):
    N, calls, rounds = 512, 100, 20
    gen = torch.Generator(device=DEV).manual_seed(tokens + K)
    q = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K // 8), generator=gen, device=DEV, dtype=torch.int32)
    s = (torch.rand(N, K // g, generator=gen, device=DEV) * 0.02 + 0.001).half()
    z = torch.randint(0, 16, (N, K // g), generator=gen, device=DEV).half()
    xs = [torch.randn(tokens, K, generator=gen, device=DEV).to(xdt) for _ in range(2)]

    def call(x):
        if noalloc:
            return quantized_matmul_noalloc(x, q, s, z, None, 4, g, torch.empty(tokens, N, dtype=torch.float16, device=DEV))
        return quantized_matmul_cuda(x, q, s, z, None, 4, g)

    want = [call(x) for x in xs]
    assert _lib.last_kernel() == kernel
    torch.cuda.synchronize()
    assert not torch.equal(*want)
    wrong, errors = [0, 0], []
    start = threading.Barrier(2)

    def work(i):
        try:
            for _ in range(rounds):
                start.wait(timeout=60)
                outs = [call(xs[i]) for _ in range(calls)]
                wrong[i] += sum(not torch.equal(y, want[i]) for y in outs)
        except Exception as e:      # noqa: BLE001 -- reported by the main thread
            errors.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and wrong == [0, 0]
    assert _lib.lib().bw_device_status() == 0
