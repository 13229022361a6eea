"""The prefill GEMM takes any number of rows: one past what a grid's y dimension holds in tiles of 128 rows, and a few more."""
import ctypes as C

import pytest

from vyre_b200 import ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def gemm(x, w, scale, y, m, n, k):
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    ffi.check(ffi.lib().vyb_k_int4_prefill_gemm(x.data_ptr(), w.data_ptr(), scale.data_ptr(), y.data_ptr(), m, n, k, 64, ffi.DT_BF16,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_void_p(status.data_ptr())))
    torch.cuda.synchronize()
    assert status.tolist() == [0] * 4


@pytest.mark.parametrize("over", [1, 200])
def test_rows_beyond_a_grid_dimension(over):
    m, n, k, part = 65535 * 128 + over, 8, 64, 400
    g = torch.Generator(device="cuda").manual_seed(over)
    x = torch.randint(-2**15, 2**15, (m, k), generator=g, device="cuda", dtype=torch.int16)
    x = (x & -0x4001 | 0x3000).view(torch.bfloat16)  # every bit pattern of ordinary size
    w = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    scale = (torch.rand(n, 1, generator=g, device="cuda") * 0.02 + 0.001).to(torch.bfloat16)
    y = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(x, w, scale, y, m, n, k)
    assert (y[m] == 7.0).all()
    for r0 in (0, m // 2, m - part):  # rows do not depend on where they stand
        want = torch.empty(part, n, device="cuda", dtype=torch.bfloat16)
        gemm(x[r0:], w, scale, want, part, n, k)
        assert torch.equal(y[r0 : r0 + part], want)
