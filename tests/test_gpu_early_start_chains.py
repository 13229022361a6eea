"""Chains that nobody waits for: every launch reads what the launch before it wrote, which it starts beside, and rewrites what the one before
that reads. The outputs are those of the same chain waited for launch by launch."""
import ctypes as C

import numpy as np
import pytest

import vyre_b200 as vb
from vyre_b200 import ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STEPS = 10


def bf16(v):
    return torch.from_numpy(np.ascontiguousarray(v, np.float32)).to(torch.bfloat16).view(torch.int16).numpy().view(np.uint16)


# name -> (program of x [m, k] -> out [m, k], operands of one step, element size of x). Gains keep the values near their first size.
def affine(m, k, group):
    prog = (vb.linear_4bit_affine_grouped("x", "w", "s", "z", "b", "out", k, k, group) if m == 1
            else vb.linear_4bit_affine_grouped_batched("x", "w", "s", "z", "b", "out", k, k, group, m))
    return prog, lambda r: {"w": r.integers(0, 2**32, k // 8 * k, dtype=np.uint32), "s": r.uniform(0.1, 0.3, k // group * k).astype(np.float32) / np.float32(k**0.5),
                            "z": r.integers(6, 10, k // group * k, dtype=np.uint32), "b": r.standard_normal(k).astype(np.float32)}, 4


def k_quant(bits, k):
    make, block = (vb.q4_k_linear, 32) if bits == 4 else (vb.q2_k_linear, 16)
    return make("x", "w", "s", "mn", "b", "out", k, k), lambda r: {
        "w": r.integers(0, 2**32, k * k * bits // 32, dtype=np.uint32), "s": r.uniform(0.1, 0.2, k * k // block).astype(np.float32) / np.float32(k**0.5),
        "mn": (r.uniform(-1.5, -0.5, k * k // block) * 0.15 * (2**bits - 1) / 2).astype(np.float32) / np.float32(k**0.5), "b": r.standard_normal(k).astype(np.float32)}, 4


def int8(m, k):
    return vb.linear_int8_weight_only("x", "w", "s", "out", m, k, k), lambda r: {
        "w": r.integers(-127, 128, k * k, dtype=np.int8), "s": r.uniform(0.01, 0.02, k).astype(np.float32) / np.float32(k**0.5)}, 4


def dense(m, k, out_in=False):
    prog = vb.linear_rows_no_bias_out_in_typed("x", "w", "out", m, k, k, ffi.DT_F32) if out_in else vb.linear_rows_no_bias("x", "w", "out", m, k, k)
    return prog, lambda r: {"w": (r.standard_normal(k * k) / k**0.5).astype(np.float32)}, 4


def matvec(m, k):
    return vb.i4x8_batched_matvec_f32_scaled("w", "x", "s", "out", m, k, k), lambda r: {
        "w": r.integers(0, 2**32, k * k // 8, dtype=np.uint32), "s": r.uniform(0.15, 0.25, k).astype(np.float32) / np.float32(k**0.5)}, 4


def int4(m, k, group):
    return vb.linear_int4_grouped_rowmajor("x", "w", "s", "out", m, k, k, group, ffi.DT_BF16), lambda r: {
        "w": r.integers(0, 2**32, k * k // 8, dtype=np.uint32), "s": bf16(r.uniform(0.15, 0.25, k * k // group) / k**0.5)}, 2


CONTRACT = [affine(1, 4096, 128), affine(1, 512, 8), affine(3, 512, 64), affine(16, 1024, 32), affine(20, 512, 8), k_quant(4, 1024), k_quant(2, 4096), int8(1, 1001),
            int8(16, 1024), dense(4, 512), dense(64, 1024), dense(33, 1024, True), matvec(3, 512), int4(1, 4096, 128), int4(2, 512, 128), int4(3, 3072, 128),
            int4(5, 1600, 64), int4(6, 2048, 128), int4(8, 1152, 128), int4(12, 1600, 64), int4(16, 1024, 128), int4(40, 2048, 128), int4(70, 1600, 64)]


@pytest.mark.parametrize("i", range(len(CONTRACT)))
def test_submissions_of_one_instance(i):
    prog, operands, size = CONTRACT[i]
    d, rng = vb.Device.acquire(0), np.random.default_rng(i)
    sess = vb.ArtifactSession.compile(prog, d)
    slots = {b["name"]: b for b in prog.buffers()}
    count = slots["x"]["count"]
    x = rng.standard_normal(count)
    x = x.astype(np.float32) if size == 4 else bf16(x)
    held, steps = [], []
    bufs = [d.resident_from(x)] + [d.allocate_resident(count * size) for _ in range(STEPS)]
    for at in range(STEPS):
        bs = vb.BindingSet(sess.artifact.digest())
        for name, v in operands(rng).items():
            held.append(d.resident_from(v))
            bs.insert_resident(slots[name]["binding"], held[-1])
        bs.insert_resident(slots["x"]["binding"], bufs[at])
        bs.insert_resident(slots["out"]["binding"], bufs[at + 1])
        steps.append(bs)
    want = []
    for bs, out in zip(steps, bufs[1:]):
        sess.submit(bs, leave_resident=True).wait()
        want.append(d.download_resident(out, count * size).tobytes())
    assert len(set(want)) == STEPS
    final = np.frombuffer(want[-1], np.float32) if size == 4 else torch.from_numpy(np.frombuffer(want[-1], np.int16).copy()).view(torch.bfloat16).float().numpy()
    assert np.isfinite(final).all() and np.unique(final).size > 50
    for _ in range(3):
        d.upload_resident(bufs[0], np.zeros_like(x))
        for sub in [sess.submit(bs, leave_resident=True) for bs in steps]:  # other values in every buffer that a step could read too early
            sub.wait()
        d.upload_resident(bufs[0], x)
        for sub in [sess.submit(bs, leave_resident=True) for bs in steps]:
            sub.wait()
        assert [d.download_resident(out, count * size).tobytes() for out in bufs[1:]] == want
    del sess
    for h in held + bufs:
        d.free_resident(h)
    d.release()


def p(t):
    return C.c_void_p(t.data_ptr())


def unwaited(step, outputs):
    """step(i, stream) launches the i-th link; outputs(i) are the tensors that it leaves behind."""
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    want = []
    for i in range(STEPS):
        step(i, C.c_void_p(s.cuda_stream))
        s.synchronize()
        want.append([t.clone() for t in outputs(i)])
    torch.cuda.synchronize()
    assert not torch.equal(want[0][0], want[1][0])
    for _ in range(3):
        for i in range(STEPS):
            for t in outputs(i):
                t.zero_()
        torch.cuda.synchronize()
        for i in range(STEPS):
            step(i, C.c_void_p(s.cuda_stream))
        s.synchronize()
        assert all(torch.equal(a, b) for i in range(STEPS) for a, b in zip(outputs(i), want[i]))


@pytest.mark.parametrize("m,k", [(37, 4096), (300, 2048), (5, 1000), (600, 8192)])  # both quantiser kernels behind both norm kernels
def test_norm_then_quantiser(m, k):
    L, g = ffi.lib(), torch.Generator(device="cuda").manual_seed(m)
    xs = [torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16) for _ in range(STEPS)]
    w, normed = torch.rand(k, generator=g, device="cuda").to(torch.bfloat16), torch.empty(m, k, dtype=torch.bfloat16, device="cuda")
    q = [torch.empty(m, k, dtype=torch.int8, device="cuda") for _ in range(STEPS)]
    sc = [torch.empty(m, device="cuda") for _ in range(STEPS)]

    def step(i, s):
        ffi.check(L.vyb_k_rms_norm(p(xs[i]), p(w), p(normed), m, k, 1e-5, ffi.DT_BF16, s))
        ffi.check(L.vyb_k_quantize_per_token_int8(p(normed), p(q[i]), p(sc[i]), m, k, s))

    unwaited(step, lambda i: [q[i], sc[i]])


@pytest.mark.parametrize("tokens", [5, 70, 700])  # the form for few rows at two widths, and the pair GEMM
def test_norm_then_moe_layer(tokens):
    h, inter, experts, topk = 1024, 512, 8, 2
    L, g = ffi.lib(), torch.Generator(device="cuda").manual_seed(tokens)
    bf = lambda *sh, gain=1.0: (torch.randn(*sh, generator=g, device="cuda") * gain).to(torch.bfloat16)  # noqa: E731
    xs, norm, normed, wr = [bf(tokens, h) for _ in range(STEPS)], bf(h), torch.empty(tokens, h, dtype=torch.bfloat16, device="cuda"), bf(experts, h, gain=h**-0.5)
    w13 = torch.randint(0, 256, (experts, 2, inter, h // 2), generator=g, device="cuda", dtype=torch.uint8)
    w2 = torch.randint(0, 256, (experts, h, inter // 2), generator=g, device="cuda", dtype=torch.uint8)
    s13 = torch.full((experts, 2, inter, h // 128), 0.2 * h**-0.5, device="cuda").to(torch.bfloat16)
    s2 = torch.full((experts, h, inter // 128), 0.2 * inter**-0.5, device="cuda").to(torch.bfloat16)
    need = C.c_uint64(0)
    ffi.check(L.vyb_k_moe_ffn_int4_scratch_bytes(tokens, h, inter, experts, topk, C.byref(need)))
    scratch = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out = [torch.empty(tokens, h, dtype=torch.bfloat16, device="cuda") for _ in range(STEPS)]
    idx = [torch.empty(tokens, topk, dtype=torch.int32, device="cuda") for _ in range(STEPS)]
    wts = [torch.empty(tokens, topk, device="cuda") for _ in range(STEPS)]

    def step(i, s):
        ffi.check(L.vyb_k_rms_norm(p(xs[i]), p(norm), p(normed), tokens, h, 1e-5, ffi.DT_BF16, s))
        ffi.check(L.vyb_k_moe_ffn_int4(p(normed), p(wr), p(w13), p(s13), p(w2), p(s2), p(out[i]), p(idx[i]), p(wts[i]), p(scratch), need.value, tokens, h, inter,
                                       experts, topk, 128, s, None))

    unwaited(step, lambda i: [out[i], idx[i], wts[i]])


@pytest.mark.parametrize("m,n,k", [(12, 1000, 1600), (40, 2048, 4096), (100, 300, 1024), (300, 9600, 1024)])
def test_sums_then_prefill_gemm(m, n, k):
    """Activations and scales are written by the launch before."""
    L, g = ffi.lib(), torch.Generator(device="cuda").manual_seed(m)
    parts = [torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16) for _ in range(STEPS + 1)]
    sparts = [(torch.rand(n, k // 64, generator=g, device="cuda") * 0.02).to(torch.bfloat16) for _ in range(STEPS + 1)]
    x, scale = torch.empty_like(parts[0]), torch.empty_like(sparts[0])
    w = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    y = [torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(STEPS)]

    def step(i, s):
        ffi.check(L.vyb_k_residual_add(p(parts[i]), p(parts[i + 1]), p(x), x.numel(), ffi.DT_BF16, s))
        ffi.check(L.vyb_k_residual_add(p(sparts[i]), p(sparts[i + 1]), p(scale), scale.numel(), ffi.DT_BF16, s))
        ffi.check(L.vyb_k_int4_prefill_gemm(p(x), p(w), p(scale), p(y[i]), m, n, k, 64, ffi.DT_BF16, s, None))

    unwaited(step, lambda i: [y[i]])


def test_captured_with_forks_and_copies():
    """Early launches in a graph whose nodes also wait for copies, memsets and a second stream."""
    m, k = 64, 4096
    L, g = ffi.lib(), torch.Generator(device="cuda").manual_seed(8)
    bf = lambda *sh: torch.randn(*sh, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    a, b, w, x, n1, n2 = bf(m, k), bf(m, k), bf(k), bf(m, k), bf(m, k), bf(m, k)
    q, sc, kept = torch.empty(2, m, k, dtype=torch.int8, device="cuda"), torch.empty(2, m, device="cuda"), torch.empty(2, m, k, dtype=torch.int8, device="cuda")
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    cs, ct = C.c_void_p(s.cuda_stream), C.c_void_p(t.cuda_stream)

    def work():
        with torch.cuda.stream(s):
            ffi.check(L.vyb_k_residual_add(p(a), p(b), p(x), m * k, ffi.DT_BF16, cs))
            t.wait_stream(s)
            with torch.cuda.stream(t):
                ffi.check(L.vyb_k_rms_norm(p(x), p(w), p(n1), m, k, 1e-5, ffi.DT_BF16, ct))
                n2.copy_(n1)                                                             # a copy behind an early kernel
                ffi.check(L.vyb_k_swiglu(p(n2), p(n1), p(n1), m * k, ffi.DT_BF16, ct))   # and an early kernel behind a copy
            q.zero_()
            ffi.check(L.vyb_k_quantize_per_token_int8(p(x), p(q[0]), p(sc[0]), m, k, cs))
            s.wait_stream(t)
            ffi.check(L.vyb_k_quantize_per_token_int8(p(n1), p(q[1]), p(sc[1]), m, k, cs))  # behind kernels of two streams
            kept.copy_(q)

    torch.cuda.synchronize()
    work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        work()
    for _ in range(4):
        a.copy_(bf(m, k))
        torch.cuda.synchronize()
        work()
        torch.cuda.synchronize()
        want = [v.clone() for v in (kept, sc, n1)]
        for v in (x, n1, n2, q, sc, kept):
            v.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(u, v) for u, v in zip((kept, sc, n1), want)) and kept.any()
