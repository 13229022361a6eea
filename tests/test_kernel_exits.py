"""Every kernel that starts bulk copies waits for them before its shared memory goes away, and a role that issues MMAs waits for those it
issued when it gives up. What a wait that ran out leaves behind cannot be provoked without a fault, so this reads the sources."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vyre_b200", "csrc", "kernels")
SOURCES = {f: open(os.path.join(KERNELS, f), encoding="utf-8").read() for f in sorted(os.listdir(KERNELS)) if f.endswith(".cu")}
COPIES = [f for f, s in SOURCES.items() if re.search(r"\btma_load_2d(_pair)?\(|\bbulk_g2s\(", s)]


def test_the_kernels_with_copies_are_the_known_ones():
    assert COPIES == ["dense_rows_tcgen05.cu", "int4_gemm_pair_tcgen05.cu", "int4_gemv_bulk.cu", "int4_prefill_tcgen05.cu", "int4_skinny_tcgen05.cu",
                      "int8_gemm_pair_tcgen05.cu", "int8_gemm_tcgen05.cu", "moe_skinny_tcgen05.cu"]


@pytest.mark.parametrize("f", COPIES)
def test_copies_and_mmas_are_settled(f):
    s = SOURCES[f]
    if f == "int4_gemv_bulk.cu":  # its own barriers; the producer warp, which no block barrier waits for, stays until its copies have landed
        tail = s[s.index("produce(u);"):s.index("return;", s.index("produce(u);"))]
        assert "mbar_try_wait(smem_u32(&ctrl->full[v % STAGES]), (v / STAGES) & 1)" in tail
        return
    rings = set(re.findall(r"settle_copies\(bars->(\w+),", s))
    barriers = set(re.findall(r"\b(\w*full)\[\w+\]", s[s.index("struct Bars"):s.index("};", s.index("struct Bars"))]))
    # the rings that copies complete on (the other full barriers belong to MMAs or unpacking warps)
    assert rings == barriers - {"acc_full", "b_full", "d_full"} - ({"a_full"} if "skinny" in f else set())
    assert re.search(r"if \(\*abort_flag != 0[^\n]*\)\s*(\{\s*tc_commit_pair\(smem_u32\(&bars->drained\)\)|settle_mma\(smem_u32\(&bars->drained\)\))", s)
    assert "mbar_init(smem_u32(&bars->drained), 1)" in s
    # when all roles have met, and with the counts that the TMA role left
    assert s.index("settle_copies(") > s.rindex("issued = ") and s.index("settle_copies(") > s.index("tmem_ld_wait()")
    assert len(re.findall(r"settle_copies\(bars->\w+, [\w.:]+, bars->\w*issued\);", s)) == len(rings)
