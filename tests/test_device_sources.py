"""Rules of the CUDA sources that no single run shows broken, checked by reading them."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "scale-track_b200", "csrc")


def kernels():
    """(file, name, parameter list, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"/\*.*?\*/|//[^\n]*", "", f.read(), flags=re.S)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)"
                             r"\s+)?(\w+)\s*\(", text):
            at, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            args = text[m.end():at - 1]
            start = text.index("{", at)
            at, depth = start + 1, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield os.path.basename(path), m.group(1), args, text[start:at]


def test_programmatically_launched_kernels_promise_no_read_only_data():
    """A kernel that waits for the kernels before it may be resident while they still write:
    const __restrict__ would let the compiler read their output by non-coherent loads, and
    before the wait."""
    waiting = [k for k in kernels() if "grid_dep_wait()" in k[3]]
    assert {"k_step", "k_step_ring", "k_step_tet", "k_step_tet_ring", "k_finalize", "k_zero_f64",
            "k_noalloc_finalize"} <= {name for _, name, _, _ in waiting}
    bad = [(path, name, a.strip()) for path, name, args, _ in waiting for a in args.split(",")
           if "const" in a and "__restrict__" in a]
    assert not bad
