"""int4 linears on the kernel with weights in tensor memory: groups of 64 and row lengths that are no multiple of 256 (exact weights), and the
same pipeline with the prefill kernels' rounded weights, at the edges of its tiles."""
import ctypes as C

import numpy as np
import pytest

import oracle
import vyre_b200 as vb
from vyre_b200 import ffi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rel(got, want, floor_frac):
    want = want.astype(np.float64)
    floor = floor_frac * float(np.sqrt(np.mean(want**2))) + 1e-30
    return float(np.max(np.abs(got.astype(np.float64) - want) / np.maximum(np.abs(want), floor)))


# one to eight rows: first and last of a tile, a row of one stage and a bit, one 64-k block, k split over a cluster and not, 17 stages in one CTA
@pytest.mark.parametrize("m,n,k,group", [(1, 4096, 1088, 64), (2, 129, 1600, 64), (8, 127, 64, 64), (5, 2050, 320, 64), (8, 300, 6400, 64), (3, 128, 1152, 128),
                                         (7, 19200, 192, 64), (1, 9700, 4352, 64)])
def test_few_rows_of_other_groups(m, n, k, group):
    x, w, s = synth.int4_linear_inputs(m, n, k, group=group, seed=m + n + k)
    for dt, bits, tol in ((ffi.DT_BF16, oracle.DT_BF16, 1e-2), (ffi.DT_F32, oracle.DT_F32, 1e-4)):
        d = vb.Device.acquire(0)
        sess = vb.ArtifactSession.compile(vb.linear_int4_grouped_rowmajor("x", "w", "s", "o", m, k, n, group, dt), d)
        assert sess.kernel_variant() == 0
        out = sess.run_host([x, w.reshape(-1).view(np.uint32), s])[0]
        want = oracle.int4_rowmajor_linear(x, w, s, m, n, k, group=group, out_dtype=bits, mode=0).ravel()
        if dt == ffi.DT_F32:
            assert rel(np.frombuffer(out, np.float32), want, 0.1) <= tol
        else:
            assert rel(synth.bf16_bits_to_f32(np.frombuffer(out, np.uint16)), synth.bf16_bits_to_f32(want), 0.1) <= tol
        del sess
        d.release()


# rounded weights: every tile width, one row past it, several tiles of rows, long rows beyond 128 rows, groups that are no power of two, 16 and
# 17 stages in one CTA; CTA pairs: two passes a tile for four sets of warps, six, a last tile of few rows, ragged outputs
@pytest.mark.parametrize("m,n,k,group", [(16, 129, 448, 64), (17, 128, 1344, 192), (33, 1000, 4096, 128), (65, 260, 1024, 512), (128, 127, 64, 64),
                                         (129, 300, 3072, 128), (300, 257, 512, 256), (33, 9601, 4096, 128), (17, 9600, 4352, 64), (66, 9600, 4352, 64),
                                         (129, 9700, 256, 64), (260, 9601, 768, 128), (385, 5000, 512, 256)])
def test_rounded_weights(m, n, k, group):
    x, w, s = synth.int4_linear_inputs(m, n, k, group=group, seed=m + n + k)
    want = oracle.int4_rowmajor_linear(x, w, s, m, n, k, group=group, out_dtype=oracle.DT_F32, mode=1)
    tx, tw, ts = (torch.from_numpy(a).cuda() for a in (x.view(np.int16), w, s.view(np.int16)))
    y = torch.full((m + 1, n), 7.0, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    ffi.check(ffi.lib().vyb_k_int4_prefill_gemm(tx.data_ptr(), tw.data_ptr(), ts.data_ptr(), y.data_ptr(), m, n, k, group, ffi.DT_F32,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_void_p(status.data_ptr())))
    torch.cuda.synchronize()
    assert status.tolist() == [0] * 4 and (y[m] == 7.0).all()
    # Each of the k / 16 additions to a running sum may drop what lies below its f32 mantissa: at most 2^-23 of it, and running sums reach five
    # times the outputs' RMS, of which the window's floor is a tenth (the prefill kernels before had the same sums).
    assert rel(y[:m].cpu().numpy(), want.reshape(m, n), 0.1) <= max(1e-4, k / 16 * 2.0**-23 * 5 / 0.1)
