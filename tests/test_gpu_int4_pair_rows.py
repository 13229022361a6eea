"""The CTA-pair GEMM at row lengths off its 256 k of a fetch, and at outputs whose rows start on no vector's boundary: f32 sums against the oracle, and
bf16 outputs, which pass through shared memory, as those sums rounded."""
import ctypes as C

import numpy as np
import pytest

import oracle
from vyre_b200 import ffi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# more tiles than SMs, so that pairs take them: one 64-k block, one pass and a bit, one fetch and a bit, three passes of four; groups of several blocks;
# rows of outputs that are multiples of eight, four, two and one; a last tile of one row
@pytest.mark.parametrize("m,n,k,group", [(1000, 2562, 64, 64), (700, 3332, 192, 192), (520, 5003, 320, 64), (300, 9600, 1088, 64), (641, 4100, 704, 64), (513, 4001, 256, 128),
                                         (257, 9606, 1344, 192), (700, 3336, 1600, 320),
                                         (384, 6200, 1536, 128), (385, 4700, 1536, 128)])  # 147 and 148 tiles of single CTAs, all of which run at once
def test_row_lengths_and_row_starts(m, n, k, group):
    x, w, s = synth.int4_linear_inputs(m, n, k, group=group, seed=m + n + k)
    want = oracle.int4_rowmajor_linear(x, w, s, m, n, k, group=group, out_dtype=oracle.DT_F32, mode=1).reshape(m, n).astype(np.float64)
    tx, tw, ts = (torch.from_numpy(a).cuda() for a in (x.view(np.int16), w, s.view(np.int16)))
    out = {}
    for dt, torch_dt in ((ffi.DT_F32, torch.float32), (ffi.DT_BF16, torch.bfloat16)):
        y = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch_dt)
        status = torch.zeros(4, dtype=torch.int32, device="cuda")
        ffi.check(ffi.lib().vyb_k_int4_prefill_gemm(tx.data_ptr(), tw.data_ptr(), ts.data_ptr(), y.data_ptr(), m, n, k, group, dt,
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_void_p(status.data_ptr())))
        torch.cuda.synchronize()
        assert status.tolist() == [0] * 4 and (y[m] == 7.0).all()
        out[dt] = y[:m]
    assert torch.equal(out[ffi.DT_BF16], out[ffi.DT_F32].to(torch.bfloat16))
    # a step of the running sum is 16 k and may drop 2^-23 of it; the sum's RMS over the steps is below the outputs'
    assert np.sqrt(np.mean((out[ffi.DT_F32].cpu().numpy() - want) ** 2) / np.mean(want**2)) <= max(k / 16, 4) * 2.0**-23
