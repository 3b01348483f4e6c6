"""CPU check of the kernels' source: programmatic launches overlap a kernel with the one before it in its stream, and "complete" stays
transitive along the stream only if every thread of every such kernel waits for the grid before it."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WAIT = re.compile(r"cudaGridDependencySynchronize\s*\(\s*\)|\bQ36_GDS\s*\(\s*\)")


def _kernels():
    for path in sorted(glob.glob(os.path.join(ROOT, "q36_b200", "csrc", "*.cu*"))):
        txt = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        txt = re.sub(r"//[^\n]*", "", txt)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", txt):
            i = txt.index("{", m.end())
            j, depth = i, 0
            while True:
                depth += {"{": 1, "}": -1}.get(txt[j], 0)
                j += 1
                if depth == 0:
                    break
            yield os.path.basename(path), m.group(1), txt[i:j]


KERNELS = list(_kernels())


def test_the_kernels_are_found():
    names = {n for _, n, _ in KERNELS}
    assert {"k_repack", "k_front_decode", "k_quant_rows", "k_gateup_wide", "k_ffn_fused_small", "k_ep_send"} <= names and len(names) >= 20


@pytest.mark.parametrize("path,name,body", KERNELS, ids=[n for _, n, _ in KERNELS])
def test_every_thread_waits_for_the_grid_before(path, name, body):
    waits = [m.start() for m in WAIT.finditer(body)]
    assert waits, f"{path}: {name} never waits for the grid before it"
    # (lambdas aside, a return ahead of the wait would let some threads leave without it)
    ahead = re.sub(r"\[&?\]\s*\([^)]*\)[^{;]*\{.*?\n\s*\};", "", body[:waits[0]], flags=re.S)
    assert not re.search(r"\breturn\b", ahead), f"{path}: {name} returns ahead of its wait"
