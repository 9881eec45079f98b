"""Every role of a GEMM kernel leaves its loop as a whole warp: the result of a bounded wait, and the reading of
the abort flag, go through a vote before a role acts on them.  Lanes poll for themselves, so without the vote a
wait that runs out while its barrier completes lets part of a warp into .sync.aligned instructions.
That cannot be provoked on a device without a hang, so it is read from the sources here; the vote itself runs
in the self-test kernel (test_bounded_wait_gpu.py)."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "halops_b200", "csrc")


def _functions(name):
    """(heading, body) of every function of a source file that starts in column 0, without comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    heads = [(m.start(), m.end()) for m in re.finditer(r"^(?:template|__global__|__device__|inline|int|bool|struct)\b[^;{]*\{", text, re.M)]
    return [(text[a:b], text[b:text.find("\n}", b)]) for a, b in heads]


@pytest.mark.parametrize("name", ["gemm.cu", "decode.cuh"])
def test_roles_wait_as_whole_warps(name):
    for head, body in _functions(name):
        if re.search(r"\bwait_(bar|bars|bar_cluster)\(", head):
            assert "__all_sync(0xffffffffu" in body
        elif "wait_bar_lane(" not in head and "wait_selftest_kernel" not in head:
            # one lane-wise wait is meant: the scale builder's, whose lanes copy and arrive for themselves
            builder = re.search(r"kPlain && warp == 12.*?\} else if", body, re.S)
            if builder:
                assert not re.search(r"elect_one|__(all|any|ballot)_sync|lane == 0", builder.group(0))
                assert builder.group(0).count("__syncwarp()") == 1
                body = body.replace(builder.group(0), "")
            assert not re.search(r"\bwait_bar_lane\b|\bmbar_try_wait", body), f"{name}: {head.strip()[:80]} waits per lane"


@pytest.mark.parametrize("name", ["gemm.cu", "decode.cuh"])
def test_roles_read_the_abort_flag_as_whole_warps(name):
    for head, body in _functions(name):
        if "wait_bar_lane(" in head:
            continue
        for m in re.finditer(r"[^\n]*\*abort\b[^\n]*", body):
            line = m.group(0).strip()
            # declarations, votes, and the grace period of the teardown, which every warp reaches
            assert "uint32_t" in line or "_sync(" in line or "__nanosleep" in body[m.end():m.end() + 400], line


def test_commits_that_arrive_in_both_ctas_are_waited_for():
    """A commit with a destination in each CTA of the pair is asynchronous: a CTA that left before it arrived would have
    its barriers written afterwards.  So whatever such a commit signals is waited for to the last phase: the accumulators
    by the epilogue of every tile, the stages by the loads that refill them and, the last ring of them, behind the loop."""
    pair = [body for head, body in _functions("gemm.cu") if "gemm_pair_kernel(" in head]
    assert len(pair) == 1
    barriers = set(re.findall(r"tc_commit_both\(ptx::smem_u32\(&bars->(\w+)\[", pair[0]))
    assert barriers == {"empty", "acc_full"} and pair[0].count("tc_commit_both(") == 2
    loader = re.search(r"if \(warp == 0\) \{.*?\} else if", pair[0], re.S).group(0)
    refill, drain = re.search(r"(.*)pdl_launch_dependents\(\);(.*)", loader, re.S).groups()
    assert re.search(r"wait_bar\(ptx::smem_u32\(&bars->empty\[s\]\), \(\(it / C::kStages\) & 1u\) \^ 1u", refill)
    assert re.search(r"for \(uint32_t d = it > uint32_t\(C::kStages\) \? it - C::kStages : 0u; ok && d < it; \+\+d\)", drain)
    assert re.search(r"wait_bar\(ptx::smem_u32\(&bars->empty\[d % C::kStages\]\), \(d / C::kStages\) & 1u", drain)
    # the k-tile whose release a refill waits for and the phase that the drain waits for are the same
    for stages in (3, 4, 6, 8):
        for it in range(stages, 5 * stages):
            d = it - stages
            assert (d % stages, (d // stages) & 1) == (it % stages, ((it // stages) & 1) ^ 1)
