"""What a kernel does when a bounded wait runs out, read from its source (no GPU is made to wait here): csrc/gemm_tc.cu, whose warps
execute instructions for a whole warp or a whole cluster behind their waits, and whose CTAs are sent copies by other CTAs."""
import os
import re

import pytest

from kappai_b200.ops.build import CSRC_DIR

WAIT = re.compile(r"\bkp_mbar_wait_bounded\(")


def kernels(name):
    """The text of each kernel of a source file, comments taken out."""
    with open(os.path.join(CSRC_DIR, name), encoding="utf-8") as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    out = {}
    for m in re.finditer(r"\n(\w+)\((?:[^()]|\([^()]*\))*\) \{\n", text):
        if "__global__" in text[text.rfind("template", 0, m.start()):m.start()]:
            out[m.group(1)] = text[m.start():text.index("\n}\n", m.end())]
    return out


@pytest.mark.parametrize("kernel", ["gemm_tc_kernel", "gemm_tc_pair_kernel"])
def test_a_warp_gives_up_as_one(kernel):
    body = kernels("gemm_tc.cu")[kernel]
    lines = [l for l in body.splitlines() if WAIT.search(l)]
    assert len(lines) >= 4
    for l in lines:
        assert re.search(r"__all_sync\(0xffffffffu, .*kp_mbar_wait_bounded\(", l), l


def test_a_cta_that_gave_up_lingers_before_it_leaves():
    body = kernels("gemm_tc.cu")["gemm_tc_pair_kernel"]
    linger = body.index("if (*abort_flag) kp_linger_after_failure();")
    assert body.rindex("*abort_flag = 1") < linger < body.rindex("kp_cluster_sync()") < body.index("kp_tmem_dealloc")


def test_a_cluster_is_told_before_a_cta_that_gave_up_lingers():
    """Other CTAs copy into this one: those that have not sent yet are told not to, and the last barrier of the cluster, before which
    none leaves, is behind the linger."""
    with open(os.path.join(CSRC_DIR, "gemm_tc.cu"), encoding="utf-8") as f:
        text = f.read()
    gave_up = text[text.index("void tc_gave_up("):]
    gave_up = gave_up[:gave_up.index("\n}\n")]
    assert gave_up.index("*abort_flag = 1") < gave_up.index("kp_st_cluster(") < gave_up.index("kp_linger_after_failure()")
    body = kernels("gemm_tc.cu")["gemm_tc_kernel"]
    assert body.index("tc_gave_up(") < body.rindex("kp_cluster_arrive()") < body.rindex("kp_cluster_wait()") < body.index("kp_tmem_dealloc")
    # what a CTA looks at before it sends: in front of its sums' staging, and behind a wait for the other CTAs' rings
    assert "kp_mbar_wait_bounded(&acc_full[b2], set_ph) && !*abort_flag" in body and "kp_mbar_wait_bounded(rings_free, 0) && !*abort_flag" in body


@pytest.mark.parametrize("name,barriers", [("attention_tc.cu", ["s_full", "pv_full"]), ("latent.cu", ["&s_full[b]", "u_full", "o_full"]),
                                           ("moe.cu", ["acc_full"]), ("attention_mma.cu", ["bar", "&full[s]"]), ("gemm_stream.cu", ["&full[s]"])])
def test_warps_of_other_kernels_give_up_as_one(name, barriers):
    """The waits of whole warps behind which a warp leaves its loop if it gave up (elsewhere one lane waits, or the walk goes on)."""
    with open(os.path.join(CSRC_DIR, name), encoding="utf-8") as f:
        lines = f.read().splitlines()
    for b in barriers:
        waits = [l for l in lines if f"kp_mbar_wait_bounded({b}," in l]
        assert waits and all("__all_sync(0xffffffffu, " in l for l in waits), (b, waits)


def test_no_attention_cta_leaves_with_copies_under_way():
    for name, n in (("attention_tc.cu", 2), ("attention_mma.cu", 2)):
        with open(os.path.join(CSRC_DIR, name), encoding="utf-8") as f:
            assert f.read().count("kp_linger_after_failure()") == n
