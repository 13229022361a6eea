"""Kernels that start before the launches before them are complete (dependent_launch.cuh) read operands that those may still be writing, until the
wait. So nothing may promise the compiler or the read-only cache path that the operands do not change while the kernel lives. What such a
promise leaves to chance cannot be provoked, so this reads the sources."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vyre_b200", "csrc", "kernels")
SOURCES = {f: open(os.path.join(KERNELS, f), encoding="utf-8").read() for f in sorted(os.listdir(KERNELS)) if f.endswith(".cu")}


def functions(source):
    """(name, signature, body) of the device functions of a file."""
    source = re.sub(r"//[^\n]*", "", source)
    for m in re.finditer(r"\b__(?:global|device)__\b", source):
        end = source.find("{", m.end())
        head = source[m.start() : end]
        if end < 0 or ";" in head:
            continue
        depth, i = 1, end + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(source[i], 0)
            i += 1
        names = [n for n in re.findall(r"(\w+)\s*\(", head) if n != "__launch_bounds__"]
        yield names[0], head, source[end:i]


FUNCTIONS = {f: list(functions(s)) for f, s in SOURCES.items()}
EARLY = [(f, name) for f, fs in FUNCTIONS.items() for name, head, body in fs
         if "__global__" in head and re.search(r"\b(waits_for_previous|dependent_start)\(\)", body)]


def test_the_early_kernels_are_found():
    assert len(EARLY) >= 28 and ("int4_prefill_tcgen05.cu", "int4_tmem_kernel") in EARLY and ("moe_ffn.cu", "moe_combine_kernel") in EARLY


@pytest.mark.parametrize("f,name", EARLY)
def test_no_operand_is_promised_read_only(f, name):
    known = {n: (head, body) for n, head, body in FUNCTIONS[f]}
    todo, seen = [name], set()
    while todo:  # the kernel and the functions of its file that it calls
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        head, body = known[n]
        assert "__restrict__" not in head + body and "__ldg(" not in body, f"{n} ({f})"
        todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", body)) if c in known]


WITH_TENSOR_MEMORY = [(f, name) for f, name in EARLY if any(n == name and "tmem_alloc" in body for n, _, body in FUNCTIONS[f])]


@pytest.mark.parametrize("f,name", WITH_TENSOR_MEMORY)
def test_tensor_memory_is_held_before_the_next_launch_may_start(f, name):
    """A block of the next launch on the same SM could otherwise allocate first and wait for this one, which waits for the allocation."""
    assert len(WITH_TENSOR_MEMORY) >= 3
    body = next(body for n, _, body in FUNCTIONS[f] if n == name)
    alloc, meet, start = body.index("tmem_alloc("), body.index("__syncthreads()", body.index("tmem_alloc(")), body.index("lets_next_start()")
    assert alloc < meet < start and body.count("lets_next_start()") == 1 and "dependent_start()" not in body


def roles(body):
    """The branches of a kernel's chain of roles: (condition, text)."""
    at = [m for m in re.finditer(r"\n    (?:\} else )?(?:if constexpr|if|else if)? ?\((warp[^\n]*|G == 0)\) \{|\n    \} else \{", body)]
    return [(m.group(1), body[m.end() : n.start() if n else len(body)]) for m, n in zip(at, at[1:] + [None])]


WITH_LIMITS = [(f, name) for f, name in EARLY if any(n == name and re.search(r"\bmbar_wait2?\(", body) for n, _, body in FUNCTIONS[f])]


@pytest.mark.parametrize("f,name", WITH_LIMITS)
def test_waits_with_a_limit_begin_behind_the_wait_for_earlier_launches(f, name):
    """The time that earlier launches still take (a peer that is late, a kernel of seconds) would count against the limit."""
    assert {x[0] for x in WITH_LIMITS} == {"int4_gemv_bulk.cu", "int4_prefill_tcgen05.cu", "int4_skinny_tcgen05.cu", "moe_skinny_tcgen05.cu"}
    body = next(body for n, _, body in FUNCTIONS[f] if n == name)
    if f == "int4_gemv_bulk.cu":  # consumers: before anything of theirs; the producer: before the first stage that it has to wait for
        assert "if (warp != WARPS || !p.constant) waits_for_previous();" in body
        assert re.search(r"if \(u == STAGES\) waits_for_previous\(\);\s*if \(u >= STAGES\) ok = mbar_wait\(", body)
        return
    chain = body.index("bool ok = true;")
    guard = re.search(r"\n    (if \(([^;]*)\) )?waits_for_previous\(\);", body[body.index("lets_next_start()") : chain])
    left_out = {None: (), "warp != 0 && !(p.constant && warp >= 12)": ("warp == 0", "warp >= 12")}[guard.group(2)] if guard else None
    found = roles(body[chain:])
    assert len(found) >= 4
    # without a wait of the whole block, or for the roles that it leaves out for what they may read or prefetch before: before their own first wait
    for role, text in found:
        limit = re.search(r"\b(mbar_wait2?|done_wait)\(", text)
        if limit and (left_out is None or role in left_out):
            assert "waits_for_previous();" in text[: limit.start()], role


@pytest.mark.parametrize("f", ["int4_gemv_batch8.cu", "int4_gemv_bulk.cu", "int4_gemv_halfsm.cu", "int4_prefill_tcgen05.cu", "int4_skinny_tcgen05.cu"])
def test_a_launch_that_leaves_an_sm_free_lets_nobody_start(f):
    """The kernels that take a number of SMs: what starts early behind one that leaves SMs free would sit on them until it ends."""
    s = SOURCES[f]
    starts = re.findall(r"([^\n;{}]*)\blets_next_start\(\);", s)
    assert [x.strip() for x in starts] == ["if (p.early)"]
    launches, early = re.findall(r"cfg\.numAttrs = ([^;]*);", s), re.findall(r"p\.early = ([^;]*);", s)
    assert launches and set(launches) <= {"p.early ? 1 : 0", "p.early ? 2 : 1"} and len(early) == len(launches)
    assert set(early) <= {"all_sms", "constant_weights || all_sms", "constant_weights || whole_device(dev, sm_count)"}


def test_kernels_that_read_twice_keep_l1():
    """A preferred split of shared memory is a property of a kernel, whatever its size: what reads a row again from L1 must not have it."""
    between = re.findall(r"launch_between<([^;()]*)>\(", SOURCES["ref_ops.cu"])
    assert set(between) == {"residual_add_kernel", "swiglu_kernel", "rms_norm_tree_regs_kernel<16>", "rms_norm_tree_regs_kernel<32>", "rms_norm_kernel<true>"}
    assert "if (rows <= 64) return launch_between<rms_norm_kernel<true>>(" in SOURCES["ref_ops.cu"]


def test_no_instance_without_a_caller():
    """f32 outputs of up to 16 rows: int4_few_rows and the integer kernels."""
    s = SOURCES["int4_skinny_tcgen05.cu"]
    assert "int4_skinny_kernel<BN, BN != 16>" in s and "if (m <= 16 && !out_f32) return launch_bn<16>" in s
