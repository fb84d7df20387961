"""Bulk copies to global memory go on beside the thread that issued them. A kernel
that issues one, itself or through a device function, waits for its copies to be
written (bulk_wait_all) after the last of them, before it ends. Checked on the
CUDA sources, without a GPU."""
import os
import re

from pipeline_gb300 import build as B


def _functions():
    """(name, is a kernel, body) of every function in the CUDA sources."""
    out = []
    for f in sorted(os.listdir(B.CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(B.CSRC, f)).read())
        for m in re.finditer(r"(__global__|__device__)[^;{}()]*(?:__launch_bounds__\([^)]*\))?"
                             r"[^;{}()]*?\b(\w+)\s*\([^;{}]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            out.append((m.group(2), m.group(1) == "__global__", text[m.end():i]))
    return out


def test_kernels_wait_for_their_bulk_stores():
    functions = _functions()
    issuers = {"bulk_store_s2g"}
    while True:  # device functions that issue one, through others too
        more = {name for name, kernel, body in functions if not kernel
                and any(re.search(rf"\b{i}\s*\(", body) for i in issuers)} - issuers
        if not more:
            break
        issuers |= more
    assert {"prefix_slots_tile", "store_node_block", "msd_item"} <= issuers
    checked = []
    for name, kernel, body in functions:
        at = [m.start() for i in issuers for m in re.finditer(rf"\b{i}\s*\(", body)]
        if kernel and at:
            assert body.rfind("bulk_wait_all()") > max(at), name
            checked.append(name)
    assert len(checked) >= 7, checked
