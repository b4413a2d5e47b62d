"""Kernels launched with programmatic dependent launch are resident while the
kernel before them still writes the sweep's state, so they must not read that
state through the read-only path (__ldg, const __restrict__ parameters), whose
loads the wait does not order.  What such a load returns cannot be provoked, so
the sources are checked."""
import os
import re

import pytest

from conftest import PKG_DIR

STATE = r"(?:st\.)?(?:comm|newc|size|S)\b"
HELPERS = {"insert_row": 3, "insert_row_piece": 3, "eval_slots": 4}   # template arguments up to CO


def _split_template(args):
    out, depth = [""], 0
    for ch in args:
        depth += (ch == "(") - (ch == ")")
        if ch == "," and depth == 0:
            out.append("")
        else:
            out[-1] += ch
    return [a.strip() for a in out]


def _kernels():
    for name in sorted(os.listdir(os.path.join(PKG_DIR, "csrc"))):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(PKG_DIR, "csrc", name)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", src):
            at = src.index("{", m.end())
            head, depth, end = src[m.end():at], 0, at
            while True:
                depth += (src[end] == "{") - (src[end] == "}")
                end += 1
                if depth == 0:
                    break
            body = src[at:end]
            if "pdl_wait(" in body:
                yield m.group(1), head, body


KERNELS = {k: (head, body) for k, head, body in _kernels()}


def test_kernels_found():
    assert {"move_group_kernel", "move_group_narrow_kernel", "collect_movers_kernel", "apply_movers_kernel",
            "s2_kernel", "sweep_end_kernel"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_state_is_read_behind_the_wait(name):
    head, body = KERNELS[name]
    assert not re.search(r"__ldg\(\s*" + STATE, body)
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__\s+(?:comm|newc|size|S)\b", head)
    assert not re.search(r"\bst\.(?:comm|newc|size|S)\b", body[:body.index("pdl_wait(")])
    for fn, n in HELPERS.items():
        for m in re.finditer(r"\b" + fn + r"<", body):
            depth, end = 1, m.end()
            while depth:   # the argument list ends at the '>' before '('
                nxt = body[end]
                depth += (nxt == "(") - (nxt == ")")
                if nxt == ">" and body[end + 1] == "(" and depth == 1:
                    break
                end += 1
            args = _split_template(body[m.end():end])
            assert len(args) == n and args[-1] == "true", f"{fn} without coherent loads"
