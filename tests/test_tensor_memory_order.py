"""Kernels that take tensor memory let the kernels behind them go only once they hold it (no GPU needed).

A block that waits for tensor memory must never wait for a block that waits for it.  The blocks of the next kernel start
once every block of this one has let them go; if that comes before the allocation, they can take the columns that a
block of this kernel still needs, and hold them while they wait for this kernel's end."""
import os
import re

import pytest

from nanoinfer_b200.kernels import build

FILES = [f for f in build.sources() if "tmem_alloc" in open(os.path.join(build.CSRC_DIR, f)).read()]


def _kernels(text):
    """The bodies of the file's __global__ functions."""
    for m in re.finditer(r"__global__", text):
        at = text.index("{", m.end())
        depth, i = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield text[at:i]


def test_the_files_are_found():
    assert {"attention_prefill_tc.cu", "attention_wide_tc.cu", "gemm_tcgen05.cu", "gemm_tcgen05_pair.cu"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_dependents_are_let_go_behind_the_allocation(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(build.CSRC_DIR, name)).read())
    bodies = [b for b in _kernels(text) if re.search(r"tmem_alloc(_pair)?\(", b)]
    assert bodies
    for b in bodies:
        taken = re.search(r"tmem_alloc(_pair)?\(", b).start()
        known = b.index("__syncthreads()", taken)          # from here on every thread's block holds its columns
        let_go = [m.start() for m in re.finditer(r"pdl_trigger\(\)", b)]
        assert let_go and min(let_go) > known
