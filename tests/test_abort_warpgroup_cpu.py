"""A wait that gave up ends a launch role by role, and the warps of a compute warpgroup look at the next
task one by one: an abort between two warps' looks must not leave one of them in a barrier of the task
(the epilogues' barriers wait for all four warps, without a limit) while another is on its way out.

Every interleaving of the four warps, the scheduler's posts and the abort, as a host model of the
kernel's rule: an abort does not end a compute warp's look, the scheduler's end does, behind which
nothing is posted.  That the kernel keeps to it is read off the source
(megaattention_b200/csrc/fused_prefill.cu).  No GPU is made to time out in the middle of a task."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "megaattention_b200", "csrc", "fused_prefill.cu")
WARPS = 4


def _outcomes(tasks, rule):
    """(states in which somebody waits for ever, states in which all have left): ``tasks`` is the number of
    barriers of each task; behind the last one everybody is told to leave.  The scheduler runs one task
    ahead of the slowest warp, and after an abort it may leave before, or after one more post."""
    last = len(tasks)
    start = (0, False, False, tuple((0, "look", 0) for _ in range(WARPS)))
    seen, todo, stuck, left = {start}, [start], 0, 0

    def looked(task, full):                      # what a warp does after its look at a task
        if not full or task == last:
            return (task, "out", 0)
        return (task, "bar", 0) if tasks[task] else (task + 1, "look", 0)

    while todo:
        posted, abort, ended, warps = todo.pop()
        nxt = []
        if not abort:
            nxt.append((posted, True, ended, warps))
        if not ended:
            if posted <= last and posted < min(t for t, _, _ in warps) + 2:
                nxt.append((posted + 1, abort, ended, warps))
            if abort or posted > last:
                nxt.append((posted, abort, True, warps))
        for i, (task, pc, n) in enumerate(warps):
            # a look that fails is followed by one at a flag, and only then is it known what it leads to
            w = None
            if pc == "look":
                w = looked(task, True) if posted > task else (task, "missed", 0)
            elif pc == "missed" and rule:
                w = looked(task, posted > task) if ended else (task, "look", 0)
            elif pc == "missed":
                w = looked(task, False) if abort else (task, "look", 0)
            if w:
                nxt.append((posted, abort, ended, warps[:i] + (w,) + warps[i + 1:]))
        if all(pc == "bar" for _, pc, _ in warps):
            assert len(set(warps)) == 1
            nxt.append((posted, abort, ended, tuple(
                (t, "bar", n + 1) if n + 1 < tasks[t] else (t + 1, "look", 0) for t, _, n in warps)))
        left += all(pc == "out" for _, pc, _ in warps)
        stuck += ended and abort and all(s[3] == warps for s in nxt) and any(pc != "out" for _, pc, _ in warps)
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return stuck, left


@pytest.mark.parametrize("tasks", [(2,), (0, 2), (4, 0, 1), (1, 2)])
def test_an_abort_between_two_warps_looks(tasks):
    stuck, left = _outcomes(tasks, rule=True)
    assert stuck == 0 and left > 0
    assert _outcomes(tasks, rule=False)[0] > 0           # (what the rule is for)


def test_the_kernel_keeps_to_the_rule():
    code = re.sub(r"//[^\n]*", "", open(SRC).read())
    # the compute warps' tasks come by looks that only the scheduler's end ends
    compute = code[code.index("reg_inc<208>();"):code.index("#undef MA_TASK_FULL")]
    assert re.findall(r"MA_NEXT_TASK\w*(?=\()", compute) == ["MA_NEXT_TASK_WARPGROUP"]
    macro = re.search(r"#define MA_NEXT_TASK_WARPGROUP\([^)]*\)\s*\\\n(.*)", code).group(1)
    assert "__all_sync(0xffffffffu, MA_TASK_FULL_OR_END)" in macro
    look = re.search(r"bool wait_task_or_end\(.*?\n\}", code, re.S).group()
    assert "abort" not in look and re.search(
        r"if \(\*posted_all\) \{\s*__threadfence_block\(\);\s*return mbar_test_wait\(bar, parity\);", look)
    # the scheduler posts nothing into a slot that it did not see empty, and says so when it leaves
    scheduler = code[code.index("while (true) {\n        if (occupied[k])"):code.index("else if (warp == 0 && lane == 0)")]
    assert re.search(r"if \(occupied\[k\]\) \{\s*if \(!wait_bar\([^;]*task_empty\[k\][^;]*\)\) break;", scheduler)
    assert re.search(r"k \^= 1;\s*\}\s*__threadfence_block\(\);\s*"
                     r"\*const_cast<volatile int\*>\(&s_posted_all\) = 1;\s*\}\s*$", scheduler)
    assert scheduler.count("task_full[") == 1 and scheduler.count("s_posted_all") == 1
    # barriers without a limit inside tasks are the compute warpgroups' alone
    kernel = code[code.index("fused_prefill_kernel(const"):]
    assert "named_bar_sync" not in kernel[:kernel.index("reg_inc<208>();")]
    assert set(re.findall(r"named_bar_sync\(([^)]*)\)", code)) == {"1 + wg, 128"}
