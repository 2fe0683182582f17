"""A block's shared memory may be accessed by the other blocks of its cluster only once
that block runs: in the source of every kernel a cluster-wide barrier stands before the
first remote access. (A run cannot show this: it depends on when the blocks start.)
"""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "hifde3d_b200", "csrc", "hif_kernels.cu")


def kernels():
    """name -> body of the kernels that reach into other blocks, comments taken out"""
    with open(SRC) as fh:
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", fh.read(), flags=re.S)
    out = {}
    for part in text.split("__global__")[1:]:
        head = re.match(r"(?:\s|__launch_bounds__\((?:[^()]|\([^()]*\))*\)|void)*(\w+)\s*\(", part)
        start = part.index("{")
        depth, end = 0, start
        for end in range(start, len(part)):
            depth += {"{": 1, "}": -1}.get(part[end], 0)
            if depth == 0:
                break
        body = part[start:end]
        if "map_shared_rank" in body:
            out[head.group(1)] = body
    return out


def test_kernels_found():
    assert {"k_pchol_panel", "k_gemv1", "k_apply_mma", "k_qr_panel_cluster"} <= set(kernels())


@pytest.mark.parametrize("name", sorted(kernels()))
def test_barrier_before_first_remote_access(name):
    body = kernels()[name]
    assert "cl.sync()" in body[:body.index("map_shared_rank")]
