"""Orders that device code must keep and no run can be relied on to show broken: read from the source.

* A block of a cluster may touch another block's shared memory only after a cluster barrier has shown
  that the other block runs.
* Kernels launched with programmatic stream serialization are resident while the one before still
  writes.  What an earlier kernel of the chain writes is not read by the non-coherent load, nor through
  a __restrict__ pointer, from which the compiler may load before the wait.
"""
import os
import re

import pytest

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dopamine_b200", "csrc", "cuda")


def _source(name):
    with open(os.path.join(CUDA, name)) as fh:
        s = fh.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", s, flags=re.S))


def _bodies(src, head):
    """(signature, body) of every function whose definition matches head, which ends at its name."""
    out = []
    for m in re.finditer(head + r"\s*\(", src):
        i = src.index("{", m.end())
        if ";" in src[m.end():i]:
            continue  # a declaration
        depth, j = 0, i
        while True:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            j += 1
            if depth == 0:
                break
        out.append((src[m.start():i], src[i:j]))
    return out


def test_cluster_blocks_meet_before_the_first_remote_access():
    (_, body), = _bodies(_source("pcg_cluster.cuh"), r"__global__[^;{]*?k_pcg_cluster")
    # code that runs: the lambdas' bodies run where they are called
    code = re.sub(r"auto (\w+) = \[&\]\([^)]*\) \{.*?\n  \};", "", body, flags=re.S)
    remote = min(code.index(f) for f in ("cl_allreduce(", "product(", "cl_barrier("))
    assert not re.search(r"cl_(ld|st)\(", code[:remote])
    arrive, wait = code.index("cl_arrive()"), code.index("cl_wait()")
    assert arrive < wait < remote
    # reached by every thread: outside any block of the kernel's body
    for at in (arrive, wait):
        assert code[:at].count("{") - code[:at].count("}") == 1


def test_chained_kernels_read_written_data_behind_the_wait():
    src = _source("mlkern.cuh")
    # arrays of the set-up, which no kernel of the chain writes (q: matrix entries, rows of the inverse)
    constant = {"L.col", "L.dinv", "L.diag", "L.g", "m.off", "m.ent", "om", "a.pinv", "q"}
    loads = re.findall(r"__ldg\(&([\w.]+)", src)
    assert src.count("__ldg(") == len(loads)
    assert set(loads) <= constant, set(loads) - constant
    kernels = [k for k in _bodies(src, r"__global__[^;{]*?k_mlk_\w+") if "mlk_enter();" in k[1]]
    assert len(kernels) >= 10
    for sig, body in kernels:
        assert "__restrict__" not in sig, sig
        assert body[1:].lstrip().startswith("mlk_enter();"), sig
    for sig, _ in _bodies(src, r"__device__[^;{]*?mlk_(?:rowsum|row0|step|start|totals)"):
        assert "__restrict__" not in sig, sig
