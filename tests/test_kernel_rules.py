"""Rules of the stage kernels that a run shows only by chance, checked in their
source.  A kernel that raises an error or a halt changes the halt word while its
own blocks start, so the warps of one block may read different values.  Where
the block's threads then work together (barriers, shared memory), the block has
to take one decision: by a block-wide vote, or by going on with nothing to do."""
import os
import re

from lbibcell_b200 import build

# Kernels whose blocks may differ, because whatever a warp reads it ends alike:
ALIKE = {
    "remesh_apply_kernel": "raises the halt only where every thread returns",
    "cross_tie_kernel": "its barrier only counts the connections to split, for a pass that the error cancels",
}


def _functions(text):
    """{name: (is a kernel, body)} of the functions in a source text."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    out = {}
    for m in re.finditer(r"(__global__|__device__)[^;{}=]*?\b(\w+)\s*\([^;{}]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(2)] = (m.group(1) == "__global__", text[m.end():i])
    return out


def _sources():
    functions = {}
    for path in sorted(build.sources()):
        if path.endswith((".cu", ".cuh")):
            with open(path) as f:
                functions.update(_functions(f.read()))
    return functions


def _reaches(functions, pattern):
    """Names of the functions that contain `pattern`, or call one that does."""
    found = {n for n, (_, body) in functions.items() if re.search(pattern, body)}
    while True:
        more = {n for n, (_, body) in functions.items()
                if n not in found and any(re.search(r"\b%s\s*(<[^;()]*>)?\(" % f, body) for f in found)}
        if not more:
            return found
        found |= more


def test_blocks_of_raising_kernels_decide_as_one():
    functions = _sources()
    raising = _reaches(functions, r"&st->halt")
    meeting = _reaches(functions, r"__syncthreads")
    kernels = {n for n, (kernel, _) in functions.items() if kernel}
    assert {"crossings_kernel", "spread_kernel", "coarsen_cell_kernel"} <= kernels & raising & meeting
    alone = re.compile(r"if \(((?!__syncthreads_or)[^;{}])*\bhalt\b((?!__syncthreads_or)[^;{}])*\)\s*(\{[^{}]*)?return")
    # a thread that leaves on the halt word by itself, in the kernel or in a function it calls
    leaves = {n for n, (_, body) in functions.items() if alone.search(body)}
    leaving = {n for n in kernels & raising & meeting
               if n in leaves or any(re.search(r"\b%s\s*\(" % f, functions[n][1]) for f in leaves)}
    assert leaving - set(ALIKE) == set()
