"""Source checks of the kernels that are launched with programmatic dependence (launch_chain): what such a kernel must not
do cannot be provoked on a GPU in a controlled way, so it is looked for in the text."""
from __future__ import annotations

import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "race_attention_kernel_b200", "csrc")


def _functions():
    """(file, name, text) of every __global__ or __device__ function of the kernel sources, comments removed."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        starts = [m.start() for m in re.finditer(r"^(?:__global__|__device__|inline|static|template|cudaError_t)", text, flags=re.M)]
        for a, b in zip(starts, starts[1:] + [len(text)]):
            part = text[a:b]
            m = re.search(r"__global__.*?\n(\w+)\(", part, flags=re.S) or re.search(r"__device__.*?(\w+)\(", part)
            if m:
                yield os.path.basename(path), m.group(1), part


WAITING = [(f, n, t) for f, n, t in _functions() if "chain_wait();" in t and n != "chain_wait"]


def test_what_releases_its_successor_also_waits():
    assert len(WAITING) >= 15
    for f, n, t in _functions():
        if "chain_release();" in t and n != "chain_release":
            assert (f, n, t) in WAITING, n


@pytest.mark.parametrize("file,name", [(f, n) for f, n, _ in WAITING])
def test_nothing_is_read_before_the_wait(file, name):
    """Not the hyperplanes either: the kernel before may be a caller's, and what it wrote is visible after the wait only."""
    text = next(t for f, n, t in WAITING if (f, n) == (file, name))
    before = text[text.index("{"):text.index("chain_wait();")]
    assert not re.search(r"__ld(g|cg|cs)|ld_chain|build_plane_tab|load_plane_frags|fold_prefix|tma_load", before)
    pointers = set(re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*[,)]", text[:text.index("{")]))
    assert not [p for p in pointers if re.search(rf"(?<![\w.]){p}\[|\*\s*{p}\b(?!\s*[*+-])", before)]


CHAINED_FILES = ["causal_tc.cu", "causal_tc_bf16.cu", "causal_bwd_tc.cu", "causal_bwd_bf16_tc.cu", "bucket_probs_bwd.cu", "probs_frag.cuh"]


@pytest.mark.parametrize("file", CHAINED_FILES)
def test_helpers_of_chained_kernels_load_what_may_still_change(file):
    assert "__ldg(" not in re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())


@pytest.mark.parametrize("file,name", [(f, n) for f, n, t in WAITING if "__global__" in t])
def test_no_input_of_a_chained_kernel_is_declared_constant_for_its_life(file, name):
    text = next(t for f, n, t in WAITING if (f, n) == (file, name))
    assert "__ldg(" not in text
    assert not re.search(r"const \w+\s*\*\s*__restrict__", text)
