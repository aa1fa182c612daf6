"""Ordering rules of the tcgen05 kernels that no run can be relied on to violate, checked on the source text.

A tcgen05 access (ld, st, mma) that follows a wait on an mbarrier is only ordered behind the tcgen05 work which that
barrier reports if a ``tcgen05.fence::after_thread_sync`` stands between the two.  The scan below walks a kernel source in
textual order: a wait or a probe of a barrier clears "fenced", a fence sets it, and an access needs it.  A fence inside a
block of braces counts for that block alone; an unfenced wait inside a block counts behind it too.  The branches of an
if / else start from the same state.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "longcat_video_b200", "csrc")
TOKEN = re.compile(r"[{}]|\b(?:mbar_wait_warp|mbar_wait_thread|mbar_test|mbar_try|tc_fence_after|tc_ld32|tc_ld64|tc_ld_half64|tc_st_half32|tc_st16|tc_st32|tc_mma|tc_mma_ts)(?=\()")


def _unfenced(text):
    """Line numbers of tcgen05 accesses without a fence behind the last wait."""
    text = re.sub(r"//[^\n]*", "", text)
    found, stack, fenced = [], [], True
    branch = True  # state at the end of the branches before this one, while an else is open
    for m in TOKEN.finditer(text):
        tok = m.group()
        if tok == "{":
            stack.append((fenced, branch))
            branch = True
        elif tok == "}":
            before, others = stack.pop()
            end = fenced and others
            if re.match(r"\s*else\b", text[m.end():]):
                fenced, branch = before, end
            else:
                fenced, branch = before and end, True
        elif tok.startswith("mbar"):
            fenced = False
        elif tok == "tc_fence_after":
            fenced = True
        elif not fenced:
            found.append(text.count("\n", 0, m.start()) + 1)
    assert not stack
    return found


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


@pytest.mark.parametrize("name", ["attn_tc.cu", "attn_tc128.cu", "attn_bwd_tc.cu"])
def test_every_tcgen05_access_behind_a_wait_is_fenced(name):
    assert _unfenced(_source(name)) == []


def test_the_scan_sees_a_missing_fence():
    ok = "{ mbar_wait_warp(b); tc_fence_after(); { tc_st32(x); } }"
    assert _unfenced(ok) == []
    assert _unfenced(ok.replace("tc_fence_after();", "")) == [1]
    assert _unfenced("{ mbar_test(b); if (r) { tc_fence_after(); tc_st32(x); } else {\n tc_st32(x); } }") == [2]
    assert _unfenced("{ tc_fence_after(); if (!pre) { mbar_wait_warp(b); }\n tc_mma(x); }") == [2]
    assert _unfenced("{ if (k) { mbar_wait_warp(b); } else { mbar_wait_warp(c); tc_fence_after(); tc_ld32(x); }\n tc_ld32(x); }") == [2]


def test_key_masks_are_handed_on_by_arrivals_of_threads():
    """Ragged grids: the key masks are plain stores of the K producer.  Its arrival on k_full releases them to the issuer of
    S; the arrival of a tcgen05.commit reports MMAs and nothing else, so the issuer has to arrive on s_full itself."""
    src = re.sub(r"//[^\n]*", "", _source("attn_tc.cu"))
    store, full = src.index("masks[(gk %"), src.index("request(j, &P.tm_k")
    assert store < full and "__syncwarp()" in src[store:full]
    issue = src[src.index("mbar_wait_warp(bar_k_full(slot)"):src.index("tc_commit(bar_s_full(wg))")]
    assert "if (kRagged) mbar_arrive_elect(bar_s_full(wg));" in issue
    assert "mbar_init(bar_s_full(b), kRagged ? 2 : 1);" in src


def _codes_of_waits(text):
    """code -> barriers whose waits report it when they run out; codes are expressions of kMode, wg and is_k."""
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for bar, code in re.findall(r"\bmbar_wait_warp\((\w+)[^;]*?, ctl, ([^,]+),", text):
        yes, no = re.fullmatch(r"(?:\w+ \? )?([^:]+?)(?: : (.+))?", code).groups()
        for expr in filter(None, (yes, no)):
            for mode in (0, 1):
                for wg in (0, 1):
                    out.setdefault(eval(expr, {"kMode": mode, "wg": wg}), set()).add(bar)
    return out


@pytest.mark.parametrize("name", ["attn_tc.cu", "attn_tc128.cu", "attn_bwd_tc.cu"])
def test_a_reported_code_names_one_barrier(name):
    """The status word of a wait that ran out is the wait's code: waits on different barriers have different ones."""
    codes = _codes_of_waits(_source(name))
    assert len(codes) > 15
    assert {c: b for c, b in codes.items() if len(b) > 1} == {}


def test_the_scan_knows_the_accesses_there_are():
    """Every wrapper of a tcgen05 load, store or MMA is scanned for and used."""
    wrappers = set(re.findall(r"void (tc_(?:ld|st|mma)\w*)\(", _source("tc_common.cuh")))
    used = "".join(_source(n) for n in ("attn_tc.cu", "attn_tc128.cu", "attn_bwd_tc.cu", "tc_common.cuh"))
    for w in wrappers:
        assert len(re.findall(rf"\b{w}\(", used)) > 1, f"nothing calls {w}"
        assert TOKEN.search(f" {w}("), f"the scan does not know {w}"
    for w in re.findall(r"tc_(?:ld|st|mma)\w*", TOKEN.pattern):
        assert w in wrappers, f"the scan looks for {w}, which does not exist"
