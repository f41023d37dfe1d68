"""Waits of the kernels that copy ahead, read from the source: what no run on a GPU shows reliably.

A wait gives up after a limit.  In a warp that stays converged - it elects a thread, or runs `.sync.aligned` tensor-memory instructions -
giving up has to be one decision of the whole warp, and a warp whose lanes poll different barriers has to pass what each lane acquired on to
the others before any of them goes on."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "powerserve_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _body(text, head):
    at = text.index("{", text.index(head))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError(head)


def test_giving_up_is_a_decision_of_the_warp():
    for name in ("ps_tc.cuh", "ps_arch_tc.cuh"):
        for cond, then in re.findall(r"if \(([^;{]*ps_tc_wait\([^;{]*)\)\s*\{([^}]*)\}", _source(name)):
            # a lane's own wait may only end a loop that nothing but the exit follows: the copies in flight at the end
            assert re.fullmatch(r"\s*\*a\.err = 5;\s*break;\s*", then), (name, cond, then)
    assert "__all_sync" in _body(_source("ps_ptx.cuh"), "bool ps_tc_wait_warp")


def test_epilogue_warps_meet_before_they_leave():
    body = _body(_source("ps_tc.cuh"), "ps_k_tc_gemm(const PsTcArgs a)")
    waits = [m.start() for m in re.finditer(r"ps_bar_all\(1, ET, ok\)\) break;", body)]
    plain = [m.start() for m in re.finditer(r"ps_bar_sync\(1, ET\);", body)]
    assert len(waits) == 1 and len(plain) == 1 and waits[0] < plain[0]
    assert not re.search(r"if \(!ok\) break;\s*if \(nu > 1\)", body)


def test_lanes_share_what_they_acquired():
    body = _body(_source("ps_tc.cuh"), "bool ps_tc_wait_all")
    assert "ps_tc_poll" in body and re.search(r"__syncwarp\(\);\s*return ok;\s*\}$", body) and body.count("return") == 1


def test_copies_arrive_before_the_shared_memory_is_given_up():
    """ps_k_matmul_ob: a wait that gives up sets the flag and nothing else, so that the loop goes on to wait for every later piece"""
    body = _body(_source("ps_mv32.cuh"), "ps_k_matmul_ob(const PsMbArgs a)")
    assert re.search(r"if \(g % cg == 0 && !ps_tc_wait\(&bar\[warp\]\[g / cg\], 0\)\) \*a\.err = PS_ERR_COPY;", body)
    assert body.count("ps_tc_wait") == 1 and "return;" not in body[body.index("ps_tc_wait"):]
