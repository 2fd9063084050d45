"""A kernel that is launched before the kernel ahead of it has finished (those
that call wait_for_previous) must read global memory by ordinary loads: the
read-only path promises that the data does not change while the kernel runs.
Checked in the source, over each such kernel and the functions it calls."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kami_b200", "csrc")
HEAD = re.compile(r"\b(\w+)\s*\(([^;{}]*)\)\s*(?:const\s*)?\{")


def _functions(path):
    """name -> [(signature, body)] of the functions defined in a CUDA source"""
    out = {}
    text = re.sub(r"//[^\n]*", "", open(path).read())
    text = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in HEAD.finditer(text):
        if m.group(1) in ("if", "for", "while", "switch"):
            continue
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out.setdefault(m.group(1), []).append((m.group(2), text[m.end():i]))
    return out


def test_ordinary_loads_only():
    shared = {}
    for path in glob.glob(os.path.join(CSRC, "*.cuh")):
        for name, defs in _functions(path).items():
            shared.setdefault(name, []).extend(defs)
    waiting, seen, bad = set(), set(), []
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        functions = {**shared, **_functions(path)}
        todo = [n for n, defs in functions.items()
                if n != "wait_for_previous" and any("wait_for_previous()" in body for _, body in defs)]
        waiting.update(todo)
        here = set()
        while todo:
            name = todo.pop()
            if name in here:
                continue
            here.add(name)
            for signature, body in functions[name]:
                if "__ldg" in body or "ld.global.nc" in body or "__restrict__" in signature:
                    bad.append((os.path.basename(path), name))
                todo += [c for c in re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\s*\(", body) if c in functions]
        seen |= here
    assert {"block_mma_kernel", "f64_ring_kernel", "h16_ring_kernel", "spgemm_count_kernel", "spgemm_scan_kernel",
            "spgemm_numeric_push_kernel", "tc05_stream_kernel", "tc05_bwd_kernel", "spmm_tc05_kernel",
            "split_f64_persistent"} <= waiting
    assert {"ld2", "gather2", "stage_tile", "build_row_bitmap"} <= seen
    assert not bad, bad
