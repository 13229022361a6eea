"""linear_rows at size: the tensor-core form (16-bit [out, in] weights) against the oracle, the tiled form bit for bit."""
import numpy as np
import pytest

import oracle
import vyre_b200 as vb
from vyre_b200 import api, ffi

pytestmark = pytest.mark.gpu

BF16, F16, F32 = ffi.DT_BF16, ffi.DT_F16, ffi.DT_F32
ODT = {BF16: oracle.DT_BF16, F16: oracle.DT_F16, F32: oracle.DT_F32}


@pytest.fixture(scope="module")
def dev():
    d = vb.Device.acquire(0)
    yield d
    d.release()


def to_bits(a, dtype):
    return oracle.f32_to_bf16_bits(a) if dtype == BF16 else a.astype(np.float16).view(np.uint16) if dtype == F16 else a


def to_f32(b, dtype):
    return oracle.bf16_bits_to_f32(b) if dtype == BF16 else b.view(np.float16).astype(np.float32) if dtype == F16 else b


# split clusters (1, 2, 7, 8 parts), tails in outputs, rows and k, one and two row tiles, every tile width class
@pytest.mark.parametrize("rows,k,n,dtype", [(1, 4096, 520, BF16), (16, 8192, 4096, BF16), (3, 1032, 1000, F16), (17, 520, 8200, BF16), (33, 1800, 300, F16),
                                            (130, 256, 20000, BF16), (257, 72, 257, F16), (300, 2048, 129, BF16)])
def test_sixteen_bit_rows_on_the_tensor_cores(dev, rows, k, n, dtype):
    rng = np.random.default_rng(rows * 7 + k)
    x = to_bits(rng.standard_normal((rows, k)).astype(np.float32), dtype)
    w = to_bits((rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32), dtype)
    sess = vb.ArtifactSession.compile(api.linear_rows_no_bias_out_in_typed("x", "w", "out", rows, k, n, dtype), dev)
    assert sess.kernel_variant() == 10
    got = to_f32(np.frombuffer(sess.run_host([x, w])[0], np.uint16), dtype).reshape(rows, n)
    want = to_f32(x, dtype).astype(np.float64) @ to_f32(w, dtype).astype(np.float64).T
    # one rounding to the storage type (half an ulp) plus the f32 sums in another order (k 2^-24 of the summed magnitudes)
    half_ulp = 2.0 ** (-9 if dtype == BF16 else -12)
    mags = np.abs(to_f32(x, dtype)).astype(np.float64) @ np.abs(to_f32(w, dtype)).astype(np.float64).T
    assert np.all(np.abs(got - want) <= 2 * half_ulp * np.abs(want) + k * 2.0 ** -24 * mags + 1e-7)


def test_a_payload_that_names_the_reference_order_keeps_it(dev):
    """Payloads written before the tensor-core form existed say variant 0: they are admitted and give the reference's bits."""
    rows, k, n = 16, 256, 520
    rng = np.random.default_rng(1)
    x, w = (to_bits(rng.standard_normal(c).astype(np.float32), BF16) for c in (rows * k, n * k))
    prog = api.linear_rows_no_bias_out_in_typed("x", "w", "out", rows, k, n, BF16)
    sealed = vb.target_compile(vb.compile(prog)).to_bytes()
    for at in range(len(sealed) - 36):
        if sealed[at:at + 4] != (10).to_bytes(4, "little"):
            continue
        body = sealed[:at] + bytes(4) + sealed[at + 4:-32]
        try:
            old = api.TargetPayload.from_bytes(body + vb.blake3(body))
        except vb.BackendError:
            continue
        if old.kernel_variant() == 0:
            break
    else:
        raise AssertionError("no variant word found")
    sess = api.ArtifactSession(prog, dev, old.to_bytes())
    assert sess.kernel_variant() == 0
    got = np.frombuffer(sess.run_host([x, w])[0], np.uint16)
    assert np.array_equal(got, oracle.linear_rows(x, w, None, rows, k, n, dtype=oracle.DT_BF16, weight_out_in=True))


@pytest.mark.parametrize("rows,k,n,dtype,out_in", [(1, 1030, 321, F32, True), (5, 517, 129, F32, True), (16, 256, 65, F32, False), (19, 100, 300, BF16, False),
                                                   (4, 1001, 77, F16, True), (33, 31, 640, F32, True)])
def test_tiled_rows_keep_the_reference_order_bits(dev, rows, k, n, dtype, out_in):
    rng = np.random.default_rng(rows + k)
    x = to_bits(rng.standard_normal((rows, k)).astype(np.float32), dtype)
    w = to_bits(rng.standard_normal((n, k) if out_in else (k, n)).astype(np.float32), dtype)
    make = api.linear_rows_no_bias_out_in_typed if out_in else api.linear_rows_no_bias_typed
    got = np.frombuffer(vb.ArtifactSession.compile(make("x", "w", "out", rows, k, n, dtype), dev).run_host([x, w])[0], x.dtype)
    want = oracle.linear_rows(x, w, None, rows, k, n, dtype=ODT[dtype], weight_out_in=out_in)
    assert np.array_equal(got.view(np.uint8), np.ascontiguousarray(want).reshape(-1).view(np.uint8))


# the tiled kernel's range: f32 from 2^14 outputs ([out, in]) and 2^18 ([in, out]) or from 2^22 and 2^23 weights, 16 bits [out, in] from 5 x 2^15
# outputs and [in, out] from 2^21, one and four rows a warp, with and without a bias, tails in rows, outputs and k
@pytest.mark.parametrize("rows,k,n,dtype,out_in,bias", [(5, 33, 3300, F32, True, False), (4, 35, 4100, F32, True, False), (4, 5, 65600, F32, False, True),
                                                        (43, 100, 3900, BF16, True, False), (66, 9, 4100, F32, False, True), (42, 33, 3910, F16, True, False), (513, 5, 4100, F16, False, False),
                                                        (1, 2055, 2049, F32, True, False), (3, 4099, 2050, F32, False, True),
                                                        (70, 37, 3800, F32, False, False)])
def test_tiled_rows_where_they_are_chosen(dev, rows, k, n, dtype, out_in, bias):
    rng = np.random.default_rng(rows + k)
    x = to_bits(rng.standard_normal((rows, k)).astype(np.float32), dtype)
    w = to_bits(rng.standard_normal((n, k) if out_in else (k, n)).astype(np.float32), dtype)
    b = to_bits(rng.standard_normal(n).astype(np.float32), dtype) if bias else None
    make = api.linear_rows_no_bias_out_in_typed if out_in else api.linear_rows_no_bias_typed
    prog = api.linear_rows("x", "w", "b", "out", rows, k, n) if bias else make("x", "w", "out", rows, k, n, dtype)
    got = np.frombuffer(vb.ArtifactSession.compile(prog, dev).run_host([x, w] + ([b] if bias else []))[0], x.dtype)
    want = oracle.linear_rows(x, w, b, rows, k, n, dtype=ODT[dtype], weight_out_in=out_in)
    assert np.array_equal(got.view(np.uint8), np.ascontiguousarray(want).reshape(-1).view(np.uint8))


@pytest.mark.parametrize("m,k", [(2, 512), (1184, 512), (1185, 512), (1185, 520), (4097, 896), (4097, 904), (1, 16), (3, 2048), (5, 2064), (2, 8192), (3, 16384), (2, 16400)])
def test_wide_quantiser_equals_the_rule(m, k):
    import torch
    rng = np.random.default_rng(k)
    x = oracle.f32_to_bf16_bits((rng.standard_normal((m, k)) * rng.choice([1e-3, 1.0, 300.0], size=(m, 1))).astype(np.float32))
    x[0, :] = 0 if m > 1 else x[0, :]
    want_q, want_s = oracle.quantize_per_token_int8(x, m, k)
    xt = torch.from_numpy(x.view(np.int16)).cuda()
    q, s = torch.empty(m, k, dtype=torch.int8, device="cuda"), torch.empty(m, device="cuda")
    ffi.check(ffi.lib().vyb_k_quantize_per_token_int8(xt.data_ptr(), q.data_ptr(), s.data_ptr(), m, k, torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(q.cpu().numpy(), want_q.reshape(m, k)) and np.array_equal(s.cpu().numpy(), want_s)


# the register forms (16 and 32 elements a thread) and the loop: one summation order, restated here
@pytest.mark.parametrize("rows,hidden,dtype", [(3, 2048, BF16), (2, 4100, F32), (1, 4096, F16), (5, 8192, BF16), (2, 8200, F32),
                                               (592, 2052, BF16), (593, 2052, BF16), (297, 4100, BF16)])
def test_long_row_norm_in_registers_has_the_tree_bits(dev, rows, hidden, dtype):
    rng = np.random.default_rng(hidden)
    x = to_bits(rng.standard_normal((rows, hidden)).astype(np.float32), dtype)
    w = to_bits((1.0 + 0.1 * rng.standard_normal(hidden)).astype(np.float32), dtype)
    got = np.frombuffer(vb.ArtifactSession.compile(api.learned_rms_norm("x", "w", "o", rows, hidden, 1e-5, dtype), dev).run_host([x, w])[0], x.dtype)
    v = to_f32(x, dtype).reshape(rows, hidden)
    part = np.zeros((rows, 256), np.float32)
    for c in range(0, hidden, 256):  # thread t adds the squares of elements t, t + 256, ...
        blk = v[:, c:c + 256]
        part[:, :blk.shape[1]] = part[:, :blk.shape[1]] + blk * blk
    part = part.reshape(rows, 8, 32)
    for o in (16, 8, 4, 2, 1):
        part = part + part[:, :, np.arange(32) ^ o]
    total = np.zeros(rows, np.float32)
    for i in range(8):
        total = total + part[:, i, 0]
    inv = np.float32(1.0) / np.sqrt(total / np.float32(hidden) + np.float32(1e-5))
    n = v * inv[:, None]
    n = to_f32(to_bits(n, dtype), dtype) if dtype != F32 else n
    want = to_bits(n * to_f32(w, dtype), dtype)
    assert np.array_equal(got.reshape(rows, hidden), want)
