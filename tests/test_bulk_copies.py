"""Staging by bulk copies, read from the kernels' sources (no GPU).

A bulk copy writes shared memory through the asynchronous proxy, which a CTA barrier does not order
after ordinary accesses to the same memory: a kernel that stages again what its threads have used
(a loop over tiles or plans) has to fence in between."""
from __future__ import annotations

import re

import pytest

from conftest import ROOT

CSRC = ROOT / "drone-race_b200" / "csrc"


def kernels():
    """(file, kernel, body) of every kernel."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            start = text.index("{", m.end())
            depth, end = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
                end += 1
            name = re.findall(r"(\w+)\s*\(\s*const|(\w+)\s*\(", text[m.end() : start])
            yield path.name, [a or b for a, b in name if (a or b) != "__launch_bounds__"][-1], text[start : end + 1]


def staged_in_a_loop(body: str) -> bool:
    blocks, head = [], 0
    for i, c in enumerate(body):
        if c == "{":
            blocks.append(bool(re.search(r"(\bfor|\bwhile)\s*\(", body[head:i])))
        elif c == "}":
            blocks.pop()
        elif body.startswith("bulk_g2s", i) and any(blocks):
            return True
        if c in "{}":
            head = i + 1
        elif c == ";" and body[head:i].count("(") == body[head:i].count(")"):
            head = i + 1
    return False


LOOPS = [(f, k, b) for f, k, b in kernels() if staged_in_a_loop(b)]


def test_the_kernels_that_stage_again_are_found():
    assert {k for _, k, _ in LOOPS} >= {"mppi_rollout", "mppi_verify", "mppi_ego_table"}


@pytest.mark.parametrize("kernel", [k for _, k, _ in LOOPS])
def test_a_kernel_that_stages_again_fences_first(kernel):
    body = next(b for _, k, b in LOOPS if k == kernel)
    fence = body.find("fence_before_bulk()")
    assert fence >= 0 and "__syncthreads()" in body[fence:], f"{kernel}: bulk copies over used shared memory without a proxy fence"


WAITS = [(k, b) for _, k, b in kernels() if "mbar_wait" in b]


@pytest.mark.parametrize("kernel", sorted({k for k, _ in WAITS}))
def test_a_wait_that_runs_out_is_counted(kernel):
    """A bounded wait that gives up leaves its kernel without its inputs: the count is how the host
    learns of it (DR_ERR_TIMEOUT), so no kernel may go on without one."""
    for k, body in WAITS:
        if k == kernel:
            assert re.search(r"!__syncthreads_and\(mbar_wait\([^;{]*\)\)\s*\{[^}]*atomicAdd\(&D\.stats\[1\], 1\);\s*return;", body), k
