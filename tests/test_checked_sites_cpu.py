"""The checked build's index checks stand where an index that a kernel computed is used.

A bad index must become a status, never a fault, so it is not provoked on a GPU: the sources
are read as text.  Every place listed here is guarded by a GCA_INDEX_OK in the same statement
or just before it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda_3d_gb300", "csrc")

# file, the use of a computed index, what the check must name, how often the use occurs
SITES = [
    ("sort_scan.cu", r"kout\[g\] =", r"g", 1),  # the sort passes' scatter
    ("cluster_sort.cuh", r"s_words\[at\] =", r"at, cnt", 1),  # digit order within a block
    ("cluster_sort.cuh", r"map_shared_rank\(s_words, to\)\[at", r"at, n", 1),  # to its block
    ("cluster_sort.cuh", r"mk\.point\(0, (\(int\))?i\)", r"i, n", 2),  # a word's index read back
    ("cluster_sort.cuh", r"o\.d_starts\[at\] =", r"at, n", 1),  # run starts
    ("grid.cu", r"\(slots\)\[rk\] =", r"rk, 1ll << \(L\.total_bits - L\.zs\)", 1),  # row table entries
    ("grid_query.cuh", r"run_load\(g\.slots, i \+ b0\)", r"i \+ b1, 1ll << \(L\.total_bits - L\.zs\)", 1),
]


@pytest.mark.parametrize("name,use,check,count", SITES)
def test_computed_index_is_checked(name, use, check, count):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    found = [m.start() for m in re.finditer(use, text)]
    assert len(found) == count, f"{name}: the listed use has changed"
    for at in found:
        assert re.search(r"GCA_INDEX_OK\([^;]*" + check, text[max(0, at - 260):at]), f"{name}: {use} is not checked"
