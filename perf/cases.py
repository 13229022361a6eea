"""The work a program hands to this framework, as measured cases.

Two kinds of entry are used, as programs use them: the contract (compile -> materialize -> submissions, prepared ones for
host inputs, or a GraphSession) with weights as resident buffers, and the kernel-level entries on the caller's own buffers and stream. A
case whose weights would stay in the L2 cache between passes runs several layers' worth of them in one pass.
"""
import ctypes as C
import math

import numpy as np
import torch

from vyre_b200 import api, ffi

BF16, F16, F32 = ffi.DT_BF16, ffi.DT_F16, ffi.DT_F32
TORCH = {BF16: torch.bfloat16, F16: torch.float16, F32: torch.float32}
NAMES = {"bf16": BF16, "f16": F16, "f32": F32}
EPS = 1e-5


def listed():
    return [
        # a service that calls one small int8 linear with host data and waits for the answer: latency of the contract
        {"name": "int8_linear_host_16", "kind": "int8_host", "rows": 16, "k": 1024, "n": 1024},
        # one generated token: the residual feed-forward block (norm, gate / up, SwiGLU, down, residual) of four layers
        {"name": "decode_block_m1", "kind": "decode", "m": 1, "hidden": 4096, "inter": 14336, "group": 128, "layers": 4},
        # eight sequences decoded together through the same block
        {"name": "decode_block_m8", "kind": "decode", "m": 8, "hidden": 4096, "inter": 14336, "group": 128, "layers": 4},
        # 48 sequences in one batch, the projection through the contract with resident activations
        {"name": "int4_linear_batch48", "kind": "int4_contract", "m": 48, "k": 4096, "n": 14336, "group": 128, "layers": 8},
        # prompt processing: 2048 tokens through one projection
        {"name": "int4_prefill_2048", "kind": "int4_prefill", "m": 2048, "k": 4096, "n": 14336, "group": 128, "out": "bf16"},
        # dynamic int8: activations quantised per token, then the wide projection with int32 sums
        {"name": "int8_dynamic_4096", "kind": "int8_dynamic", "m": 4096, "k": 8192, "n": 28672},
        # a mixture-of-experts layer on a prompt, and on 64 sequences being decoded
        {"name": "moe_4096_tokens", "kind": "moe", "tokens": 4096, "hidden": 4096, "inter": 14336, "experts": 8, "topk": 2, "group": 128},
        {"name": "moe_64_tokens", "kind": "moe", "tokens": 64, "hidden": 4096, "inter": 14336, "experts": 8, "topk": 2, "group": 128},
        # the operator set's own affine-grouped linear: the published benchmark row (batch 256), and a decode step
        {"name": "affine_grouped_1m", "kind": "affine", "batch": 256, "k": 256, "n": 4096, "group": 64, "layers": 8},
        {"name": "affine_grouped_decode", "kind": "affine", "batch": 1, "k": 4096, "n": 28672, "group": 128, "layers": 4},
        # a GGML checkpoint's Q4_K projection for one token
        {"name": "q4_k_linear", "kind": "k_quant", "bits": 4, "k": 4096, "n": 14336, "layers": 4},
        # the dense gated MLP template (unquantised checkpoint), a small batch, host in and host out
        {"name": "dense_mlp_bf16", "kind": "dense", "rows": 16, "hidden": 4096, "inter": 14336, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["int8_host", "decode", "decode", "int4_contract", "int4_contract", "int4_prefill", "int8_dynamic", "moe", "moe",
                       "affine", "affine", "k_quant", "dense"])
    if kind == "int8_host":
        return {"kind": kind, "rows": _log(rng, 1, 128), "k": _log(rng, 64, 1024) * 4, "n": _log(rng, 200, 4096)}
    if kind == "decode":
        return {"kind": kind, "m": rng.randint(1, 8), "hidden": 1024 * rng.randint(2, 5), "inter": 1024 * rng.randint(4, 14),
                "group": 128, "layers": 4}
    if kind == "int4_contract":
        return {"kind": kind, "m": _log(rng, 1, 128), "k": rng.choice([1024 * rng.randint(1, 8), 64 * rng.randint(16, 100)]),
                "n": 8 * _log(rng, 128, 1792), "group": rng.choice([64, 128, 128]), "layers": 4}
    if kind == "int4_prefill":
        return {"kind": kind, "m": _log(rng, 65, 2048), "k": 256 * rng.randint(4, 28), "n": 8 * _log(rng, 128, 1792) + rng.choice([0, 0, 2]),
                "group": rng.choice([64, 128, 128]), "out": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "int8_dynamic":
        return {"kind": kind, "m": _log(rng, 1, 4096), "k": 16 * _log(rng, 32, 512), "n": 4 * _log(rng, 200, 7168)}
    if kind == "moe":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "hidden": 256 * rng.randint(4, 16), "inter": 256 * rng.randint(4, 24),
                "experts": rng.choice([4, 8, 16]), "topk": rng.randint(1, 4), "group": 128}
    if kind == "affine":
        b = _log(rng, 1, 256)
        return {"kind": kind, "batch": b, "k": 256 * rng.randint(1, 16), "n": 4 * _log(rng, 256, 3584 if b <= 16 else 1024),
                "group": rng.choice([32, 64, 128]), "layers": 4}
    if kind == "k_quant":
        return {"kind": kind, "bits": rng.choice([4, 4, 2]), "k": 256 * rng.randint(2, 24), "n": 64 * _log(rng, 16, 224), "layers": 4}
    return {"kind": kind, "rows": _log(rng, 1, 64), "hidden": 8 * _log(rng, 64, 512), "inter": 8 * _log(rng, 128, 1024),
            "dtype": rng.choice(["bf16", "f16", "f32"])}


# ---- inputs: made on the GPU from the seed, the same values for `prepare` and `exact` ------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (seed + 1))
    return g


def _normal(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _uniform(g, lo, hi, *shape, dtype=torch.float32):
    return (torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo).to(dtype)


def _ints(g, lo, hi, *shape, dtype=torch.uint8):
    return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=dtype)


def _words(g, *shape):
    return torch.randint(-2**31, 2**31, shape, generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _int4_weight(g, n, k, group, gain=1.0):
    """Packed nibbles [n, k / 2] (zero point 8) and bf16 scales [n, k / group]."""
    return _ints(g, 0, 256, n, k // 2), _uniform(g, 1e-3 * gain, 2e-2 * gain, n, k // group, dtype=torch.bfloat16)


def _int4_dequant(w, s, group):
    q = torch.stack((w & 15, w >> 4), dim=-1).reshape(w.shape[0], -1)
    return ((q.double() - 8.0).reshape(w.shape[0], -1, group) * s.double()[..., None]).reshape(w.shape[0], -1)


def _inputs(case, seed):
    g, k = _gen(seed), case["kind"]
    if k == "int8_host":
        return {"x": _normal(g, case["rows"], case["k"]), "w": _ints(g, -127, 128, case["n"], case["k"], dtype=torch.int8),
                "s": _uniform(g, 1e-3, 1e-2, case["n"])}
    if k == "decode":
        m, h, i, grp = case["m"], case["hidden"], case["inter"], case["group"]
        d = {"x": _normal(g, m, h, dtype=torch.bfloat16), "layers": []}
        for _ in range(case["layers"]):
            d["layers"].append({"norm": (1.0 + _normal(g, h, scale=0.1)).to(torch.bfloat16), "gate": _int4_weight(g, i, h, grp, 0.5),
                                "up": _int4_weight(g, i, h, grp, 0.5), "down": _int4_weight(g, h, i, grp, 0.1)})
        return d
    if k in ("int4_contract", "int4_prefill"):
        return {"x": _normal(g, case["m"], case["k"], dtype=torch.bfloat16),
                "layers": [_int4_weight(g, case["n"], case["k"], case["group"]) for _ in range(case.get("layers", 1))]}
    if k == "int8_dynamic":
        return {"x": _normal(g, case["m"], case["k"], dtype=torch.bfloat16), "w": _ints(g, -127, 128, case["n"], case["k"], dtype=torch.int8)}
    if k == "moe":
        t, h, i, e, grp = case["tokens"], case["hidden"], case["inter"], case["experts"], case["group"]
        return {"x": _normal(g, t, h, dtype=torch.bfloat16), "wr": _normal(g, e, h, dtype=torch.bfloat16, scale=0.02),
                "w13": _ints(g, 0, 256, e, 2, i, h // 2), "s13": _uniform(g, 1e-3, 2e-2, e, 2, i, h // grp, dtype=torch.bfloat16),
                "w2": _ints(g, 0, 256, e, h, i // 2), "s2": _uniform(g, 1e-3, 2e-2, e, h, i // grp, dtype=torch.bfloat16)}
    if k == "affine":
        n, groups = case["n"], case["k"] // case["group"]
        return {"x": _normal(g, case["batch"], case["k"]),
                "layers": [{"w": _words(g, case["k"] // 8, n), "s": _uniform(g, 1e-3, 2e-2, groups, n),
                            "z": _ints(g, 0, 16, groups, n, dtype=torch.int32), "b": _normal(g, n)} for _ in range(case["layers"])]}
    if k == "k_quant":
        vpw, blocks = 32 // case["bits"], case["k"] * case["n"] // (32 if case["bits"] == 4 else 16)
        return {"x": _normal(g, case["k"]),
                "layers": [{"w": _words(g, case["k"] * case["n"] // vpw), "s": _uniform(g, 1e-3, 2e-2, blocks),
                            "mn": _uniform(g, -0.15, 0.0, blocks), "b": _normal(g, case["n"])} for _ in range(case["layers"])]}
    dt, r, h, i = TORCH[NAMES[case["dtype"]]], case["rows"], case["hidden"], case["inter"]
    return {"x": _normal(g, r, h, dtype=dt), "norm": (1.0 + _normal(g, h, scale=0.1)).to(dt), "gate": _normal(g, i, h, dtype=dt, scale=h ** -0.5),
            "up": _normal(g, i, h, dtype=dt, scale=h ** -0.5), "down": _normal(g, h, i, dtype=dt, scale=i ** -0.5)}


# ---- what a program keeps -----------------------------------------------------------------------------------------------------
_device = None


def _dev():
    global _device
    if _device is None:
        _device = api.Device.acquire(0)
    return _device


_TYPESTR = {torch.float32: "<f4", torch.int32: "<i4", torch.uint8: "|u1", torch.int8: "|i1", torch.bfloat16: "<i2", torch.float16: "<i2"}


class _Resident:
    """A resident buffer, given back when the last tensor that views it is gone (a view keeps this object alive)."""

    def __init__(self, shape, dtype):
        self.handle = _dev().allocate_resident(math.prod(shape) * torch.empty(0, dtype=dtype).element_size())
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": _TYPESTR[dtype],
                                         "data": (_dev().resident_ptr(self.handle)[0], False), "version": 3}

    def __del__(self):
        try:
            torch.cuda.synchronize()
            _dev().free_resident(self.handle)
        except Exception:
            pass


class _State:
    """What a program keeps between calls: resident buffers and the handles that use them."""

    def __init__(self, kind):
        self.kind, self.keep, self.close = kind, [], []

    def resident(self, tensor=None, shape=None, dtype=None):
        """The handle of a new resident buffer and its torch view, filled from `tensor` or zeroed."""
        shape, dtype = (tensor.shape, tensor.dtype) if tensor is not None else (shape, dtype)
        buf = _Resident(shape, dtype)
        view = torch.as_tensor(buf, device="cuda")
        view = view.view(dtype) if view.dtype != dtype else view
        if tensor is not None:
            view.copy_(tensor)
        else:
            view.zero_()
        self.keep.append((buf, view))
        return buf.handle, view

    def __del__(self):
        try:
            torch.cuda.synchronize()
            for c in self.close:  # handles go before the buffers that they are bound to
                c()
        except Exception:
            pass


def _p(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _contract_chain(st, program, per_layer, out_name, out_shape, out_dtype):
    """One materialised program, one binding set for each layer's resident buffers; results stay resident."""
    sess = api.ArtifactSession.compile(program, _dev())
    slots = {b["name"]: b["binding"] for b in program.buffers()}
    counts = {b["name"]: b["count"] for b in program.buffers()}
    st.session, st.chain, st.outputs = sess, [], []
    n_out = math.prod(out_shape)
    for bound in per_layer:
        bs = api.BindingSet(sess.artifact.digest())
        for name, h in bound.items():
            bs.insert_resident(slots[name], h)
        h, view = st.resident(shape=(max(counts[out_name], n_out),), dtype=out_dtype)
        bs.insert_resident(slots[out_name], h)
        st.chain.append(bs)
        st.outputs.append(view[:n_out].view(out_shape))
    torch.cuda.synchronize()
    return st


def _block_ok(m, k, norm):
    """The shapes vyb_k_int4_linear_block documents."""
    return (m <= 2 and k in (2048, 4096)) or (not norm and m <= 4 and k > 4096 and k % 2048 == 0)


def _decode_pass(st):
    L, s, c = ffi.lib(), _stream(), st.case
    m, h, i, g, W = c["m"], c["hidden"], c["inter"], c["group"], 1  # W: the weights are constants of the graph
    x = st.x
    for ly, out in zip(st.layers, st.hidden):
        gw, gs = ly["gate"]
        uw, us = ly["up"]
        dw, ds = ly["down"]
        if _block_ok(m, h, True):
            ffi.check(L.vyb_k_int4_linear_block(_p(x), _p(ly["norm"]), EPS, _p(gw), _p(gs), None, None, _p(st.gate), m, i, h, g, W, s, None))
            ffi.check(L.vyb_k_int4_linear_block(_p(x), _p(ly["norm"]), EPS, _p(uw), _p(us), _p(st.gate), None, _p(st.act), m, i, h, g, W, s, None))
        else:
            ffi.check(L.vyb_k_rms_norm(_p(x), _p(ly["norm"]), _p(st.normed), m, h, EPS, BF16, s))
            ffi.check(L.vyb_k_int4_gemv_ex(_p(st.normed), _p(gw), _p(gs), _p(st.gate), m, i, h, g, BF16, W, s, None))
            ffi.check(L.vyb_k_int4_gemv_ex(_p(st.normed), _p(uw), _p(us), _p(st.up), m, i, h, g, BF16, W, s, None))
            ffi.check(L.vyb_k_swiglu(_p(st.gate), _p(st.up), _p(st.act), m * i, BF16, s))
        if _block_ok(m, i, False):
            ffi.check(L.vyb_k_int4_linear_block(_p(st.act), None, EPS, _p(dw), _p(ds), None, _p(x), _p(out), m, h, i, g, W, s, None))
        else:
            ffi.check(L.vyb_k_int4_gemv_ex(_p(st.act), _p(dw), _p(ds), _p(st.down), m, h, i, g, BF16, W, s, None))
            ffi.check(L.vyb_k_residual_add(_p(x), _p(st.down), _p(out), m * h, BF16, s))
        x = out


def prepare(case, seed):
    st, d, kind = _State(case["kind"]), _inputs(case, seed), case["kind"]
    st.case = case
    if kind == "int8_host":
        prog = api.linear_int8_weight_only("x", "w", "scale", "out", case["rows"], case["k"], case["n"])
        sess = api.ArtifactSession.compile(prog, _dev())
        slots = {b["name"]: b["binding"] for b in prog.buffers()}
        bs = api.BindingSet(sess.artifact.digest())
        st.x = d["x"].cpu().numpy().reshape(-1)
        bs.insert_host(slots["x"], st.x)
        bs.insert_resident(slots["w"], st.resident(d["w"])[0])
        bs.insert_resident(slots["scale"], st.resident(d["s"])[0])
        torch.cuda.synchronize()
        st.session, st.prepared, st.x_slot, st.out_slot = sess, sess.prepare(bs), slots["x"], slots["out"]
        st.close.append(st.prepared.free)
    elif kind == "decode":
        m, h, i = case["m"], case["hidden"], case["inter"]
        st.x, st.layers = d["x"], d["layers"]
        bf = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")  # noqa: E731
        st.normed, st.gate, st.up, st.act, st.down = bf(m, h), bf(m, i), bf(m, i), bf(m, i), bf(m, h)
        st.hidden = [bf(m, h) for _ in st.layers]
        st.stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(st.stream):
            _decode_pass(st)
        st.stream.synchronize()
        st.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st.graph, stream=st.stream):
            _decode_pass(st)
    elif kind == "int4_contract":
        m, k, n = case["m"], case["k"] // case["group"] * case["group"], case["n"]
        prog = api.linear_int4_grouped_rowmajor("x", "w", "scale", "out", m, k, n, case["group"], BF16)
        d = _inputs({**case, "k": k}, seed)
        x = st.resident(d["x"])[0]
        _contract_chain(st, prog, [{"x": x, "w": st.resident(w)[0], "scale": st.resident(s)[0]} for w, s in d["layers"]], "out", (m, n),
                        torch.bfloat16)
    elif kind == "int4_prefill":
        st.x, (st.w, st.s) = d["x"], d["layers"][0]
        st.y = torch.empty(case["m"], case["n"], dtype=TORCH[NAMES[case["out"]]], device="cuda")
    elif kind == "int8_dynamic":
        st.x, st.w, m = d["x"], d["w"], case["m"]
        st.q = torch.empty(m, case["k"], dtype=torch.int8, device="cuda")
        st.xs = torch.empty(m, dtype=torch.float32, device="cuda")
        st.y = torch.empty(m, case["n"], dtype=torch.int32, device="cuda")
    elif kind == "moe":
        t, need = case["tokens"], C.c_uint64(0)
        ffi.check(ffi.lib().vyb_k_moe_ffn_int4_scratch_bytes(t, case["hidden"], case["inter"], case["experts"], case["topk"], C.byref(need)))
        st.d, st.scratch_bytes = d, need.value
        st.scratch = torch.empty(need.value, dtype=torch.uint8, device="cuda")
        st.out = torch.empty(t, case["hidden"], dtype=torch.bfloat16, device="cuda")
        st.idx = torch.empty(t, case["topk"], dtype=torch.int32, device="cuda")
        st.wts = torch.empty(t, case["topk"], dtype=torch.float32, device="cuda")
    elif kind == "affine":
        b, k, n, g = case["batch"], case["k"], case["n"], case["group"]
        prog = (api.linear_4bit_affine_grouped("x", "w", "scale", "zp", "b", "out", k, n, g) if b == 1
                else api.linear_4bit_affine_grouped_batched("x", "w", "scale", "zp", "b", "out", k, n, g, b))
        x = st.resident(d["x"])[0]
        _contract_chain(st, prog, [{"x": x, "w": st.resident(ly["w"])[0], "scale": st.resident(ly["s"])[0], "zp": st.resident(ly["z"])[0],
                                    "b": st.resident(ly["b"])[0]} for ly in d["layers"]], "out", (b, n), torch.float32)
    elif kind == "k_quant":
        make = api.q4_k_linear if case["bits"] == 4 else api.q2_k_linear
        prog = make("x", "w", "scales", "mins", "b", "out", case["k"], case["n"])
        x = st.resident(d["x"])[0]
        _contract_chain(st, prog, [{"x": x, "w": st.resident(ly["w"])[0], "scales": st.resident(ly["s"])[0], "mins": st.resident(ly["mn"])[0],
                                    "b": st.resident(ly["b"])[0]} for ly in d["layers"]], "out", (case["n"],), torch.float32)
    else:
        graph = api.dense_gated_mlp_graph(api.DenseGatedMlpSpec(1, case["rows"], case["hidden"], case["inter"], NAMES[case["dtype"]], EPS))
        st.session = api.GraphSession(graph, _dev())
        st.close.append(st.session.close)
        for name, key in (("post_attention_layernorm.weight", "norm"), ("mlp.gate_proj.weight", "gate"), ("mlp.up_proj.weight", "up"),
                          ("mlp.down_proj.weight", "down")):
            st.session.set_constant(name, handle=st.resident(d[key])[0])
        torch.cuda.synchronize()
        x = d["x"].cpu()
        st.x = x.numpy() if case["dtype"] == "f32" else x.view(torch.int16).numpy()
    return st


def run(st):
    L, c, kind = ffi.lib(), st.case, st.kind
    if kind == "int8_host":
        done = st.prepared.submit({st.x_slot: st.x}).wait()
        return np.frombuffer(done.output(st.out_slot), dtype=np.float32)
    if kind == "decode":
        st.graph.replay()
        return {"hidden": st.hidden[-1], "first": st.hidden[0]}
    if kind in ("int4_contract", "affine", "k_quant"):
        pending = [st.session.submit(bs, leave_resident=True) for bs in st.chain]  # an instance's submissions run in order
        for sub in pending:
            sub.wait()
        return st.outputs
    if kind == "int4_prefill":
        ffi.check(L.vyb_k_int4_prefill_gemm(_p(st.x), _p(st.w), _p(st.s), _p(st.y), c["m"], c["n"], c["k"], c["group"], NAMES[c["out"]],
                                            _stream(), None))
        return st.y
    if kind == "int8_dynamic":
        ffi.check(L.vyb_k_quantize_per_token_int8(_p(st.x), _p(st.q), _p(st.xs), c["m"], c["k"], _stream()))
        ffi.check(L.vyb_k_int8_gemm_i32(_p(st.q), _p(st.w), _p(st.y), c["m"], c["n"], c["k"], _stream(), None))
        return {"y": st.y, "x_scale": st.xs}
    if kind == "moe":
        d = st.d
        ffi.check(L.vyb_k_moe_ffn_int4(_p(d["x"]), _p(d["wr"]), _p(d["w13"]), _p(d["s13"]), _p(d["w2"]), _p(d["s2"]), _p(st.out), _p(st.idx),
                                       _p(st.wts), _p(st.scratch), st.scratch_bytes, c["tokens"], c["hidden"], c["inter"], c["experts"],
                                       c["topk"], c["group"], _stream(), None))
        return {"out": st.out, "weights": st.wts}
    out = st.session.run_chained({"residual": st.x})["mlp.block_output"]
    if c["dtype"] == "f32":
        return np.frombuffer(out, dtype=np.float32)
    return torch.frombuffer(bytearray(out), dtype=TORCH[NAMES[c["dtype"]]])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------
def work(case):
    k = case["kind"]
    if k == "int8_host":
        r, kk, n = case["rows"], case["k"], case["n"]
        return {"bytes": 4 * r * kk + n * kk + 4 * n + 4 * r * n, "flops": 2 * r * kk * n}
    if k == "decode":
        m, h, i, g = case["m"], case["hidden"], case["inter"], case["group"]
        per = 3 * (h * i // 2 + 2 * h * i // g) + 2 * h
        return {"bytes": case["layers"] * per + 4 * m * h, "flops": case["layers"] * 6 * m * h * i}
    if k in ("int4_contract", "int4_prefill"):
        m, n, layers = case["m"], case["n"], case.get("layers", 1)
        kk = case["k"] // case["group"] * case["group"]
        out = 4 if case.get("out") == "f32" else 2
        return {"bytes": 2 * m * kk + layers * (n * kk // 2 + 2 * n * kk // case["group"] + out * m * n), "flops": layers * 2 * m * n * kk}
    if k == "int8_dynamic":
        m, kk, n = case["m"], case["k"], case["n"]
        return {"bytes": 2 * m * kk + n * kk + 4 * m * n + 4 * m, "flops": 2 * m * n * kk}
    if k == "moe":
        t, h, i, e = case["tokens"], case["hidden"], case["inter"], case["experts"]
        pairs = t * case["topk"]
        touched = min(e, pairs)
        return {"bytes": 4 * t * h + 2 * e * h + touched * 3 * (h * i // 2 + 2 * h * i // case["group"]) + 8 * pairs, "flops": pairs * 6 * h * i + 2 * t * e * h}
    if k == "affine":
        b, kk, n, groups = case["batch"], case["k"], case["n"], case["k"] // case["group"]
        return {"bytes": 4 * b * kk + case["layers"] * (kk * n // 2 + 8 * groups * n + 4 * n + 4 * b * n), "flops": case["layers"] * 2 * b * kk * n}
    if k == "k_quant":
        kk, n, bits = case["k"], case["n"], case["bits"]
        return {"bytes": 4 * kk + case["layers"] * (kk * n * bits // 8 + 8 * kk * n // (32 if bits == 4 else 16) + 8 * n), "flops": case["layers"] * 2 * kk * n}
    size, r, h, i = 4 if case["dtype"] == "f32" else 2, case["rows"], case["hidden"], case["inter"]
    return {"bytes": size * (3 * h * i + h + 2 * r * h), "flops": 6 * r * h * i}


def tolerance(case):
    k = case["kind"]
    if k == "int8_dynamic":
        return "exact"
    if k in ("int8_host", "affine", "k_quant"):
        return {"rel": 1e-6, "max": 2e-5}  # f32 sums in any order: 1.2e-7 to 1.8e-7 from the sums in 64 bits
    if k == "decode":
        return {"rel": 1.2e-2, "max": 2e-1}  # bf16 between the operators of four layers
    if k == "moe":
        return {"rel": 1.2e-2, "max": 3e-1}  # bf16 intermediates, bf16 dequantised weights; the top experts' outputs cancel
    if k == "dense":
        return {"rel": 4e-6, "max": 1e-4} if case["dtype"] == "f32" else {"rel": 1.2e-2 if case["dtype"] == "bf16" else 2e-3, "max": 1e-1}
    return {"rel": 8e-3, "max": 4e-2}  # one bf16 rounding of f32 sums


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------
def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + float(np.float32(EPS))) * w.double()


def _silu(v):
    return v * torch.sigmoid(v)


def exact(case, seed):
    k = case["kind"]
    if k == "int4_contract":
        case = {**case, "k": case["k"] // case["group"] * case["group"]}
    d = _inputs(case, seed)
    if k == "int8_host":
        return (d["x"].double() @ (d["w"].double() * d["s"].double()[:, None]).T).reshape(-1)
    if k == "decode":
        x, first = d["x"].double(), None
        for ly in d["layers"]:
            a = _rms(x, ly["norm"])
            gate = a @ _int4_dequant(*ly["gate"], case["group"]).T
            up = a @ _int4_dequant(*ly["up"], case["group"]).T
            x = x + (_silu(gate) * up) @ _int4_dequant(*ly["down"], case["group"]).T
            first = x if first is None else first
        return {"hidden": x, "first": first}
    if k in ("int4_contract", "int4_prefill"):
        ys = [d["x"].double() @ _int4_dequant(w, s, case["group"]).T for w, s in d["layers"]]
        return ys if k == "int4_contract" else ys[0]
    if k == "int8_dynamic":
        return {"y": None, "x_scale": d["x"].double().abs().amax(dim=1) / 127.0}
    if k == "moe":
        # the router's logits are bf16 values of the layer's definition; the rest is not rounded
        logits = (d["x"].double() @ d["wr"].double().T).to(torch.bfloat16).double()
        idx = torch.sort(logits, dim=1, descending=True, stable=True)[1][:, :case["topk"]]
        wts = torch.softmax(logits, dim=1).gather(1, idx)  # over all experts, not renormalised
        out = torch.zeros(d["x"].shape, dtype=torch.float64, device="cuda")
        for e in range(case["experts"]):
            rows, slot = torch.nonzero(idx == e, as_tuple=True)
            if not len(rows):
                continue
            x = d["x"][rows].double()
            gate = x @ _int4_dequant(d["w13"][e, 0], d["s13"][e, 0], case["group"]).T
            up = x @ _int4_dequant(d["w13"][e, 1], d["s13"][e, 1], case["group"]).T
            y = (_silu(gate) * up) @ _int4_dequant(d["w2"][e], d["s2"][e], case["group"]).T
            out.index_add_(0, rows, y * wts[rows, slot][:, None])
        return {"out": out, "weights": wts}
    if k == "affine":
        ys, shifts = [], torch.arange(0, 32, 4, device="cuda")
        for ly in d["layers"]:
            q = ((ly["w"][:, None, :] >> shifts[None, :, None]) & 15).reshape(case["k"], case["n"]).double()
            rep = lambda v: v.double().repeat_interleave(case["group"], dim=0)  # noqa: E731
            ys.append(d["x"].double() @ ((q - rep(ly["z"])) * rep(ly["s"])) + ly["b"].double())
        return ys
    if k == "k_quant":
        ys, bits = [], case["bits"]
        shifts, block = torch.arange(0, 32, bits, device="cuda"), 32 if bits == 4 else 16
        for ly in d["layers"]:
            q = ((ly["w"][:, None] >> shifts) & (2 ** bits - 1)).reshape(-1, block).double()
            ys.append(d["x"].double() @ (q * ly["s"].double()[:, None] + ly["mn"].double()[:, None]).reshape(case["k"], case["n"]) + ly["b"].double())
        return ys
    x = d["x"].double()
    a = _rms(x, d["norm"])
    act = _silu(a @ d["gate"].double().T) * (a @ d["up"].double().T)
    return (x + act @ d["down"].double().T).reshape(-1)
