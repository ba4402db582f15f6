"""Kernels that come up while the launch before them runs read nothing of what it wrote through the read-only path: that path may be
used only for data no one writes while the kernel is alive, and its loads may be moved over the wait."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "calibquant_b200", "csrc")


def _kernels():
    """(file:name, parameters, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\(.*\)\s*)?(\w+)\s*\(", text):
            ends = []
            for opening, closing, start in (("(", ")", m.end() - 1), ("{", "}", None)):
                at = ends[-1] if start is None else start
                if start is None:
                    rest = re.match(r"\s*", text[at:]).end()
                    if text[at + rest] != "{":       # a declaration
                        break
                    at += rest
                depth, i = 0, at
                while True:
                    depth += {opening: 1, closing: -1}.get(text[i], 0)
                    i += 1
                    if depth == 0:
                        break
                ends.append(i)
            if len(ends) == 2:
                yield f"{os.path.basename(path)}:{m.group(1)}", text[m.end():ends[0] - 1], text[ends[0]:ends[1]]


WAITING = [k for k in _kernels() if "pdl_wait" in k[2]]


def test_the_kernels_are_found():
    assert {name.split(":")[1] for name, _, _ in WAITING} >= {
        "k1_scores", "k2_fp_tokens", "k2_attn_v", "k3_combine", "step_kernel", "u8_step_kernel", "prefill_tc_kernel",
        "quant_encode_kernel", "pack_k_per_channel_kernel", "pack_last_dim_group_kernel"}


@pytest.mark.parametrize("name,params,body", WAITING, ids=[k[0] for k in WAITING])
def test_inputs_are_not_read_only(name, params, body):
    assert "__ldg" not in body and "ld.global.nc" not in body
    for p in re.split(r",(?![^<]*>)", params):
        m = re.match(r"\s*const\b.*\*\s*__restrict__\s+(\w+)", p, re.S)
        # a pointer that comes out of the wait itself is another one than the parameter
        assert not m or re.search(rf"\b{m.group(1)} = ptx::pdl_wait_for\({m.group(1)}\)", body), f"{name}: {p.strip()}"


def test_the_live_count_is_a_plain_load():
    for path in glob.glob(os.path.join(CSRC, "cq_decode_mma.cu")):
        assert "__ldg" not in open(path).read()
