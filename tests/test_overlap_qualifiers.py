"""Device code behind griddepcontrol.wait reads what the kernel in front has just written, so
none of the pointers it reads that through may be __restrict__ (which allows the read to be
moved, or taken through the read-only path).  Checked over the sources: the helpers that such
kernels call, and the parameters of the kernels themselves that earlier kernels of the same
call write."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "apbf_gb300" / "csrc"


def _parameters(source, name):
    """The parameter list of the definition of `name`."""
    m = re.search(r"\b" + name + r"\s*\(", source)
    assert m, name
    depth, i = 1, m.end()
    while depth:
        depth += {"(": 1, ")": -1}.get(source[i], 0)
        i += 1
    return source[m.end():i - 1]


@pytest.mark.parametrize("file,function,params", [
    ("solver.cu", "density_one", ["pos"]),
    ("solver.cu", "delta_row", ["pos", "row"]),
    ("solver.cu", "delta_corrections", ["pos"]),
    ("solver.cu", "delta_one", ["pos"]),
    ("solver.cu", "delta_skip_filter", ["pos"]),
    ("solver.cu", "lane_row", ["row"]),
    ("apbf_internal.cuh", "remap_transfers", ["inv_perm"]),
    ("neighborhood_bs.cu", "first_not", ["code"]),
    ("neighborhood.cu", "k_reorder", ["perm"]),
    ("neighborhood.cu", "k_cell_ranges", ["skeys", "inv_perm"]),
    ("neighborhood.cu", "k_clamp_rev", ["rcount"]),
    ("neighborhood_bs.cu", "k_sorted_codes", ["pos", "width", "inv_perm"]),
    ("sort.cu", "k_onesweep", ["kin", "vin"]),
    ("sort.cu", "k_digit_count", ["kin"]),
    ("sort.cu", "k_digit_scatter", ["tile_counts", "group_counts"]),
    ("sort.cu", "k_sort_small", ["kin", "vin"]),
    ("mlp.cu", "k_mlp_grad", ["P", "X", "T"]),
    ("mlp.cu", "k_mlp_adam", ["partials"]),
])
def test_overlapped_reads_are_not_restrict(file, function, params):
    text = _parameters((CSRC / file).read_text(), function)
    for p in params:
        m = re.search(r"([\w\s:]*\*[^,]*?)\b" + p + r"\s*(?:,|$)", text)
        assert m, (function, p)
        assert "__restrict__" not in m.group(0), (function, p)
