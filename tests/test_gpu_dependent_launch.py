"""Launches that start early (programmatic dependent launch): without the promise of constant weights a projection reads what the
launch before it wrote, weights' scales included, in a chain that nobody waits for in between."""
import ctypes as C

import pytest

from vyre_b200 import ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def p(t):
    return C.c_void_p(t.data_ptr())


# the half-SM kernel (whole rows of 4096 and 2048, k blocks), eight rows of f16, the tensor-memory kernel, the bulk-copy kernel
@pytest.mark.parametrize("m,n,k", [(1, 14336, 4096), (2, 4096, 2048), (1, 4096, 14336), (5, 14336, 4096), (8, 4096, 6144), (3, 8192, 5120), (1, 2048, 1024)])
def test_scales_written_by_the_launch_before(m, n, k):
    L, g = ffi.lib(), torch.Generator(device="cuda").manual_seed(m * n + k)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    parts = [(torch.rand(n, k // 128, generator=g, device="cuda") * 0.02).to(torch.bfloat16) for _ in range(7)]
    scale, s = torch.zeros_like(parts[0]), torch.cuda.Stream()
    torch.cuda.synchronize()

    def step(i, y):
        ffi.check(L.vyb_k_residual_add(p(parts[i]), p(parts[i + 1]), p(scale), scale.numel(), ffi.DT_BF16, C.c_void_p(s.cuda_stream)))
        ffi.check(L.vyb_k_int4_gemv_ex(p(x), p(w), p(scale), p(y), m, n, k, 128, ffi.DT_BF16, 0, C.c_void_p(s.cuda_stream), None))

    want = [torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(6)]
    for i, y in enumerate(want):
        step(i, y)
        s.synchronize()
    assert not torch.equal(want[0], want[1])
    for _ in range(3):
        got = [torch.zeros_like(y) for y in want]
        torch.cuda.synchronize()
        for i, y in enumerate(got):
            step(i, y)
        s.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
