"""Order of the column-split inverse between the CTAs of a cluster (CPU).

Every CTA of a split factors panel K from the global columns X[:, K], which the
owner replaces by the panel's transform and, one panel later, nobody may read
before its owner has updated them. The test takes the order of these accesses
and of the cluster barriers from the kernel's panel loop and runs every
interleaving of the CTAs over two panels."""

import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "quatrex_b200" / "csrc" / "zinv.cu"
TOKENS = {
    r"gj_factor_panel<": ("load",),  # X[:, K] into registers, all of it before the first column step
    r"\.barrier_arrive\(\)": ("arrive",),
    r"\.barrier_wait\(\)": ("wait",),
    r"\bcluster_sync\(\);": ("arrive", "wait"),
    r"x\[r \* ldx \+ k0 \+ c\] = T\[": ("transform",),  # the owner's store to X[:, K]
    r"\bupdate\(": ("update",),  # stores to this CTA's other columns, the next panel's among them
}


def _panel_ops():
    """The accesses and barriers of one panel in program order."""
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    kernel = text[text.index("zinv3_kernel("):]
    start = kernel.index("{", kernel.index("for (int k0 = 0; k0 < n; k0 += NB)"))
    depth, end = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(kernel[end], 0)
        end += 1
        if depth == 0:
            break
    body = kernel[start:end]
    found = [(m.start(), ops) for pat, ops in TOKENS.items() for m in re.finditer(pat, body)]
    ops = [op for _, group in sorted(found) for op in group]
    assert {"load", "transform", "update"} <= set(ops)
    return ops


def _violations(ops, ctas, panels=2):
    """All interleavings of `ctas` CTAs (CTA k owns panel k), as the set of
    rules that some interleaving breaks."""
    program = [(op, k) for k in range(panels) for op in ops]
    broken, seen = set(), set()
    # per CTA: (program counter, arrivals so far)
    todo = [tuple((0, 0) for _ in range(ctas))]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        arrivals = [a for _, a in state]
        for c, (pc, arrived) in enumerate(state):
            if pc == len(program):
                continue
            op, k = program[pc]
            if op == "wait" and min(arrivals) < arrived:
                continue  # the phase that this CTA arrived at is not complete
            done = lambda cta, what, panel: any(  # noqa: E731
                program[i] == (what, panel) for i in range(state[cta][0]))
            left = lambda cta, what, panel: any(  # noqa: E731
                program[i] == (what, panel) for i in range(state[cta][0], len(program)))
            if op == "transform" and c == k and any(not done(o, "load", k) for o in range(ctas)):
                broken.add("a CTA reads the transform in place of the panel")
            if op == "load" and k > 0 and left(k, "update", k - 1):
                broken.add("a CTA reads a panel before its owner has updated it")
            nxt = list(state)
            nxt[c] = (pc + 1, arrived + (op == "arrive"))
            todo.append(tuple(nxt))
    return broken


@pytest.mark.parametrize("ctas", [2, 3])
def test_panel_is_loaded_by_all_before_its_transform_is_stored(ctas):
    assert not _violations(_panel_ops(), ctas)


def test_the_check_sees_missing_barriers():
    ops = _panel_ops()
    plain = [op for op in ops if op not in ("arrive", "wait")]
    assert len(_violations(plain, 2)) == 2
    assert _violations(plain + ["arrive", "wait"], 2) == {"a CTA reads the transform in place of the panel"}
