"""The launch-shape rules (apbf_gb300/csrc/launch_rules.cuh), compiled for the host."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "apbf_gb300" / "csrc"

SHIM = """
#include "launch_rules.cuh"
extern "C" void pass_shape(const unsigned *t, unsigned capacity, int features, unsigned *out) {
    const apbf::PassShape s = apbf::pass_shape_rule({t[0], t[1], t[2]}, capacity, features != 0);
    out[0] = s.lanes;
    out[1] = s.block;
    out[2] = s.per_sm;
}
// the places given to runs of m entries each, asked one after the other from `start` entries on
extern "C" unsigned long long pool_places(unsigned long long start, unsigned runs, unsigned m, unsigned size) {
    apbf::PoolCount used = start;
    unsigned long long given = 0;
    for (unsigned k = 0; k < runs; ++k) {
        if (apbf::pool_run(used, m, size) != apbf::kNoRun) ++given;
        used += m;
    }
    return given;
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))


def _shape(rules, tuned, capacity, features=False):
    out = (C.c_uint * 3)()
    rules.pass_shape((C.c_uint * 3)(*tuned), C.c_uint(capacity), int(features), out)
    return tuple(out)


@pytest.mark.parametrize("capacity,lanes", [(1, 4), (2197, 4), (32_768, 4), (32_769, 2), (98_304, 2), (98_305, 1),
                                            (1 << 27, 1)])
def test_shape_of_a_new_context_goes_by_capacity(rules, capacity, lanes):
    """Its tuning's fields (1, 256, 8) are no shape of their own: a tuning that sets the sort's
    digit width, or writes back what it read, keeps the threads per row."""
    got = _shape(rules, (1, 256, 8), capacity)
    assert got == ((lanes, 256, 32) if lanes > 1 else (1, 128, 8))
    assert _shape(rules, (1, 256, 8), capacity, features=True)[0] == 1


def test_given_shapes_are_taken(rules):
    for lanes in (1, 2, 4, 8):
        for block in (128, 256):
            for per_sm in (1, 2, 4, 8):
                if (lanes, block, per_sm) == (1, 256, 8):
                    continue
                for cap in (2197, 50_000, 1_000_000):
                    assert _shape(rules, (lanes, block, per_sm), cap) == (lanes, block, per_sm)
                    assert _shape(rules, (lanes, block, per_sm), cap, features=True) == (1, block, per_sm)


@pytest.mark.parametrize("m,size,runs", [(1000, 2_000_000, 5_000_000), (4_000_000, 1 << 29, 2000), (7, 0, 10), (1, 5, 9)])
def test_pool_places_are_given_once(rules, m, size, runs):
    """However many entries are asked for in all (here up to 8e9), the pool's own are given to
    the first that fit and to nobody else."""
    rules.pool_places.restype = C.c_ulonglong
    assert rules.pool_places(C.c_ulonglong(0), C.c_uint(runs), C.c_uint(m), C.c_uint(size)) == min(runs, size // m)
