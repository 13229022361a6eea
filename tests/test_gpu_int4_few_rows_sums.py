"""int4 linears of few rows: what the partial sums keep. Up to eight rows, sums in the tensor core are no longer than 64 k, then they are added
in f32, rounded to nearest; a running sum there loses what lies below its 24 bits."""
import ctypes as C

import numpy as np
import pytest

import oracle
import vyre_b200 as vb
from vyre_b200 import ffi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def bits(v):
    b = np.ascontiguousarray(v, np.float32).view(np.uint32)
    assert not (b & 0xFFFF).any()
    return (b >> 16).astype(np.uint16)


# A sum of 2^24 - 1 over the first half of a group of 128; then 2 more and 2 less: over all 128 k the last bit would be gone. The next group
# takes 2^24 - 2 away. The row in one CTA, and split over a cluster.
@pytest.mark.parametrize("m,n,k", [(1, 300, 1152), (8, 300, 1152), (8, 19200, 384)])
def test_the_last_bit_of_a_group(m, n, k):
    one = np.zeros(k, np.float32)
    one[[0, 16, 32, 64, 80]] = 255 * 65536, 255 * 256, 255, 2, -2
    one[[128, 144, 160]] = -255 * 65536, -255 * 256, -254
    x = one[None, :] * 2.0 ** np.arange(m, dtype=np.float32)[:, None]
    w = np.full((n, k // 2), 0x99, np.uint8)  # q - 8 = 1
    w[1::2] = 0x77                            # -1
    s = bits(np.ones((n, k // 128), np.float32))
    d = vb.Device.acquire(0)
    sess = vb.ArtifactSession.compile(vb.linear_int4_grouped_rowmajor("x", "w", "s", "o", m, k, n, 128, ffi.DT_BF16), d)
    out = sess.run_host([bits(x), w.reshape(-1).view(np.uint32), s])[0]
    got = synth.bf16_bits_to_f32(np.frombuffer(out, np.uint16)).reshape(m, n)
    del sess
    d.release()
    want = 2.0 ** np.arange(m)[:, None] * np.where(np.arange(n) % 2, -1.0, 1.0)[None, :]
    assert (got == want).all()


# Rounded weights: a step of the running sum is 16 k and may drop 2^-23 of it; the sum's RMS over the steps is below the outputs'
@pytest.mark.parametrize("m,n,k,group", [(33, 1000, 4096, 128), (17, 9600, 4352, 64), (66, 9600, 4352, 64), (129, 300, 3072, 128)])
def test_rms_error_of_rounded_weights(m, n, k, group):
    x, w, s = synth.int4_linear_inputs(m, n, k, group=group, seed=m + n + k)
    want = oracle.int4_rowmajor_linear(x, w, s, m, n, k, group=group, out_dtype=oracle.DT_F32, mode=1).reshape(m, n).astype(np.float64)
    tx, tw, ts = (torch.from_numpy(a).cuda() for a in (x.view(np.int16), w, s.view(np.int16)))
    y = torch.empty(m, n, device="cuda")
    ffi.check(ffi.lib().vyb_k_int4_prefill_gemm(tx.data_ptr(), tw.data_ptr(), ts.data_ptr(), y.data_ptr(), m, n, k, group, ffi.DT_F32,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream), None))
    torch.cuda.synchronize()
    assert np.sqrt(np.mean((y.cpu().numpy() - want) ** 2) / np.mean(want**2)) <= k / 16 * 2.0**-23
