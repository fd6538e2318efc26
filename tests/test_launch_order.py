"""Rules that every kernel source keeps, read from the sources (no GPU)."""
import glob
import os
import re

import pytest

import maxibone_b200

CSRC = os.path.join(os.path.dirname(maxibone_b200.__file__), "csrc")


def _kernels(path):
    """(name, body) of every __global__ function of a source file, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__global__", text):
        head = re.compile(r"(\w+)\s*\((?:[^(){}]|\([^()]*\))*\)\s*\{").search(text, m.end())
        depth, i = 1, head.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield head.group(1), text[head.end():i]


# A block that lets the next pass's blocks come up before it holds its own tensor memory can find
# the columns taken by one of them, which waits for this pass to end.
@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "tc_*.cuh"))), ids=os.path.basename)
def test_dependents_come_up_after_the_tensor_memory(path):
    for name, body in _kernels(path):
        at = [body.find(s) for s in ("tmem_alloc(", "__syncthreads()", "pass_prepare(", "pass_wait(")]
        if at[0] < 0:
            continue
        at[1] = body.find("__syncthreads()", at[0])
        assert 0 <= at[0] < at[1] < at[2] < at[3], (name, at)
        assert body.count("pass_prepare(") == 1, name
