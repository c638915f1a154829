"""Kernels chained by programmatic dependent launch wait for the grid before them ahead of every
exit: only then does the completion of a grid imply that of all grids before it, on which a
kernel launched normally after the chain relies.  Read from the sources."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "hadamag.jl_b200", "csrc")
ALLOW = re.compile(r"\b(allow_next_grid|mana_allow_next)\(\)")
WAIT = re.compile(r"\b(wait_prior_grid|mana_wait_prior)\(\)")
# heads its chain: launched without the attribute, when all work before it has finished
HEADS = {"k_adj_fused"}


def chained_kernels():
    for f in sorted(os.listdir(CSRC)):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read()) if f.endswith((".cu", ".cuh")) else ""
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\([^;{]*?\)\s*\{", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            body = src[m.end():i - 1]
            if ALLOW.search(body) and m.group(1) not in HEADS:
                yield m.group(1), body


def blocks_around(body, at):
    """Starts of the braces that are open at a position (the body's own first)."""
    open_at = [0]
    for i in range(at):
        if body[i] == "{":
            open_at.append(i + 1)
        elif body[i] == "}":
            open_at.pop()
    return open_at


@pytest.mark.parametrize("name,body", list(chained_kernels()), ids=lambda v: v if v.startswith("k_") else "")
def test_every_exit_waits_for_the_grid_before(name, body):
    assert WAIT.search(body)
    waits = [w.start() for w in WAIT.finditer(body)]
    for r in re.finditer(r"\breturn\s*;", body):
        # a wait that runs before this return: in one of the blocks that hold it
        around = blocks_around(body, r.start())
        assert any(w < r.start() and blocks_around(body, w)[-1] in around for w in waits), body[:r.end()][-120:]


def test_chained_kernels_are_found():
    names = {n for n, _ in chained_kernels()}
    assert {"k_sre_stage", "k_sre_wide_stage", "k_sre_stage3", "k_adj_wide", "k_mana_p1", "k_mc_p1"} <= names
