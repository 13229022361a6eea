"""The int4 linear at 1 to 64 rows around the kernel that unpacks weights into tensor memory (bf16 outputs) and the ones that keep f32 outputs."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
import vyre_b200 as vb
from vyre_b200 import api, ffi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = vb.Device.acquire(0)
    yield d
    d.release()


def reference(x, w, s, m, n, k):
    q = np.stack((w & 15, w >> 4), axis=-1).reshape(n, k).astype(np.float64) - 8.0
    wf = q * np.repeat(synth.bf16_bits_to_f32(s).astype(np.float64), 128, axis=1)
    xf = synth.bf16_bits_to_f32(x).astype(np.float64)
    return xf @ wf.T, np.abs(xf) @ np.abs(wf).T


def check(got, want, mags, k, f32):
    # f32 sums in any order: k 2^-24 of the summed magnitudes at most; bf16 outputs add one rounding
    assert np.all(np.abs(got - want) <= k * 2.0 ** -24 * mags + (0.0 if f32 else 2.0 ** -8) * np.abs(want))


# every column class (16, 48, 64) at its edges, one to eight k parts, tails in n, fewer k blocks than pipeline stages
@pytest.mark.parametrize("m,n,k,f32", [(9, 200, 1024, True), (16, 4096, 2048, False), (17, 130, 1024, True), (48, 1000, 3072, False), (49, 260, 4096, True),
                                       (64, 128, 7168, False), (12, 14336, 1024, True), (33, 20000, 1024, False)])
def test_batched_decode_through_the_contract(dev, m, n, k, f32):
    x, w, s = synth.int4_linear_inputs(m, n, k, seed=m + n)
    x[0, :128] = oracle.f32_to_bf16_bits(oracle.bf16_bits_to_f32(x[0, :128]) * np.float32(2.0 ** 14))  # a group of outliers
    prog = api.linear_int4_grouped_rowmajor("x", "w", "s", "o", m, k, n, 128, ffi.DT_F32 if f32 else ffi.DT_BF16)
    out = vb.ArtifactSession.compile(prog, dev).run_host([x, w.view(np.uint32), s])[0]
    got = (np.frombuffer(out, np.float32) if f32 else oracle.bf16_bits_to_f32(np.frombuffer(out, np.uint16))).reshape(m, n).astype(np.float64)
    check(got, *reference(x, w, s, m, n, k), k, f32)


@pytest.mark.parametrize("m,n,k,f32", [(5, 300, 6144, False), (8, 4096, 14336, False), (2, 140, 8192, True), (8, 64, 6144, True), (1, 200, 1024, False),
                                       (3, 72, 3072, True), (8, 1000, 5120, False)])
def test_long_rows_beyond_four_at_kernel_level_in_a_chain(m, n, k, f32):
    x, w, s = synth.int4_linear_inputs(m, n, k, seed=k)
    t = [torch.from_numpy(v).cuda() for v in (x.view(np.int16), w, s.view(np.int16))]
    ys = [torch.zeros(m, n, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda") for _ in range(3)]
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for y in ys:  # consecutive launches overlap (constant weights)
        ffi.check(ffi.lib().vyb_k_int4_gemv_ex(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), y.data_ptr(), m, n, k, 128,
                                               ffi.DT_F32 if f32 else ffi.DT_BF16, 1, C.c_void_p(torch.cuda.current_stream().cuda_stream), status.data_ptr()))
    torch.cuda.synchronize()
    assert status.tolist() == [0] * 4
    for y in ys:
        assert torch.equal(y, ys[0])
    check(ys[0].double().cpu().numpy(), *reference(x, w, s, m, n, k), k, f32)


# f32 outputs: the sum of a 128-k group is exact, so large activations that cancel inside their group leave no trace in its small ones.
# (Whole rows of 2048 and 4096 beyond one row run on the tensor cores, whose group sums are f32.)
@pytest.mark.parametrize("m,n,k", [(1, 300, 1024), (3, 64, 3072), (8, 200, 5120), (2, 140, 6144), (5, 72, 14336), (12, 96, 3072), (33, 40, 8192)])
def test_f32_outputs_have_exact_group_sums(dev, m, n, k):
    rng = np.random.default_rng(m + k)
    xs = rng.integers(-100, 101, size=(m, k // 128, 128)).astype(np.float32)  # exact in bf16
    big = (rng.integers(64, 256, size=(m, k // 128, 32)) * 4096).astype(np.float32)
    xs[:, :, 64:96], xs[:, :, 96:] = big, -big
    q = rng.integers(0, 16, size=(n, k // 128, 128), dtype=np.uint8)
    q[:, :, 96:] = q[:, :, 64:96]
    x = synth.f32_to_bf16_bits(xs.reshape(m, k))
    qf = q.reshape(n, k)
    w = (qf[:, 0::2] | (qf[:, 1::2] << 4)).astype(np.uint8)
    s = synth.f32_to_bf16_bits(rng.uniform(1e-3, 2e-2, size=(n, k // 128)).astype(np.float32))
    prog = api.linear_int4_grouped_rowmajor("x", "w", "s", "o", m, k, n, 128, ffi.DT_F32)
    got = np.frombuffer(vb.ArtifactSession.compile(prog, dev).run_host([x, w.view(np.uint32), s])[0], np.float32).reshape(m, n)
    sums = np.einsum("mgk,ngk->mng", xs.astype(np.float64), q.astype(np.float64) - 8.0)  # the groups' sums, exact
    terms = sums * synth.bf16_bits_to_f32(s).reshape(n, -1).astype(np.float64)
    # roundings: scale times sum, then one addition for each group and a handful for the parts of a row
    assert np.all(np.abs(got - terms.sum(axis=2)) <= (k // 128 + 24) * 2.0 ** -24 * np.abs(terms).sum(axis=2))


# bf16 rows of 1024 and 3072 on both sides of the line between the bulk-copy and the tensor-memory kernel
@pytest.mark.parametrize("m,n,k", [(1, 2368, 1024), (8, 2369, 1024), (2, 130, 3072), (3, 130, 3072), (1, 2400, 3072)])
def test_small_bf16_shapes_on_both_sides_of_the_line(m, n, k):
    x, w, s = synth.int4_linear_inputs(m, n, k, seed=k + n)
    t = [torch.from_numpy(v).cuda() for v in (x.view(np.int16), w, s.view(np.int16))]
    y = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    ffi.check(ffi.lib().vyb_k_int4_gemv(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), y.data_ptr(), m, n, k, 128, ffi.DT_BF16,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream), None))
    torch.cuda.synchronize()
    check(y.double().cpu().numpy(), *reference(x, w, s, m, n, k), k, False)


@pytest.mark.parametrize("m,n,k", [(8, 40000, 6144), (1, 40000, 5120), (3, 1000, 5120)])
def test_one_sm_is_left_free_on_request(m, n, k):
    """VYB_LAUNCH_LEAVE_ONE_SM: no launch has more blocks than the other SMs hold at once; the outputs are the same bits."""
    x, w, s = synth.int4_linear_inputs(m, n, k, seed=k)
    t = [torch.from_numpy(v).cuda() for v in (x.view(np.int16), w, s.view(np.int16))]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    stream = torch.cuda.Stream()

    def launch(y, flags):
        ffi.check(ffi.lib().vyb_k_int4_gemv_ex(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), y.data_ptr(), m, n, k, 128, ffi.DT_BF16, flags,
                                               C.c_void_p(stream.cuda_stream), None))

    ys = [torch.zeros(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    launch(ys[0], 0)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        launch(ys[1], ffi.LAUNCH_LEAVE_ONE_SM)
    cu = pytest.importorskip("cuda.bindings.driver")
    raw = cu.CUgraph(graph.raw_cuda_graph())
    err, _, count = cu.cuGraphGetNodes(raw, 0)
    err, nodes, count = cu.cuGraphGetNodes(raw, count)
    assert int(err) == 0 and count >= 1
    for node in nodes[:count]:
        err, params = cu.cuGraphKernelNodeGetParams(node)
        assert int(err) == 0 and params.gridDimX * params.gridDimY <= 2 * (sms - 1)
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))


@pytest.mark.parametrize("m", [1, 4, 8])
def test_dependent_launches_wait_for_their_activations(m):
    """Seven projections in a row, each reading what the one before it wrote, launched with overlapping weight prefetch: tensor-memory, bulk-copy,
    k-block and whole-row launches in turn. Replayed as a graph with new activations each time, the bits are those of the plain chain."""
    dims = [(5120, 5120), (5120, 3072), (3072, 6144), (6144, 5120), (5120, 1024), (1024, 2048), (2048, 4096)]  # (k, n) of each
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    ws = [torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8) for k, n in dims]
    ss = [(torch.rand(n, k // 128, generator=g, device="cuda") * 0.4 + 0.8).mul_(0.22 / k ** 0.5).to(torch.bfloat16) for k, n in dims]
    x = torch.empty(m, dims[0][0], dtype=torch.bfloat16, device="cuda")
    chains = [[torch.zeros(m, n, dtype=torch.bfloat16, device="cuda") for _, n in dims] for _ in range(2)]
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()

    def launch(ys, flags):
        src = x
        for (k, n), w, s, y in zip(dims, ws, ss, ys):
            ffi.check(ffi.lib().vyb_k_int4_gemv_ex(src.data_ptr(), w.data_ptr(), s.data_ptr(), y.data_ptr(), m, n, k, 128, ffi.DT_BF16, flags,
                                                   C.c_void_p(stream.cuda_stream), status.data_ptr()))
            src = y

    x.normal_(generator=g)
    torch.cuda.synchronize()
    launch(chains[0], ffi.LAUNCH_CONSTANT_WEIGHTS)  # first use of every kernel and workspace
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        launch(chains[0], ffi.LAUNCH_CONSTANT_WEIGHTS)
    for _ in range(8):
        x.normal_(generator=g)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        stream.synchronize()
        launch(chains[1], 0)
        stream.synchronize()
        assert status.tolist() == [0] * 4
        assert torch.isfinite(chains[1][-1].float()).all() and chains[1][-1].float().abs().mean() > 1e-3
        for a, b in zip(*chains):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))
