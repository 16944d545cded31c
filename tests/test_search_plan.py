"""The searches' split over the grid: the scratch that a training run reserves covers
every batch it can have. The host header is compiled by itself; no GPU is needed."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "%s/e-means_b200/csrc/search_plan.hpp"
using namespace emb;
extern "C" unsigned long reserved(int sms, unsigned long m, unsigned long k, int tc) {
    return search_part_rows(sms, m, k, tc != 0);
}
// most partial rows of any batch of 1 .. m rows
extern "C" unsigned long needed(int sms, unsigned long m, unsigned long k, int tc) {
    unsigned long rows = 0;
    for (unsigned long b = 1; b <= m; b++)
        rows = std::max(rows, b * (unsigned long)(tc ? tc_nsplit(sms, b, k) : simt_plan(sms, b, k).nsplit));
    return rows;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE % ROOT)
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(d / "plan.so"), str(d / "plan.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "plan.so"))
    for f in (lib.reserved, lib.needed):
        f.restype = ctypes.c_ulong
        f.argtypes = [ctypes.c_int, ctypes.c_ulong, ctypes.c_ulong, ctypes.c_int]
    return lib


@pytest.mark.parametrize("tc", [0, 1])
@pytest.mark.parametrize("k", [1, 63, 64, 65, 200, 257, 700, 1573, 4096, 9000, 65536])
def test_reserved_partials_cover_every_batch(plan, k, tc):
    for sms in (1, 20, 148):
        for m in (1, 63, 64, 65, 127, 128, 129, 191, 700, 1425, 1605, 4096, 5001):
            assert plan.reserved(sms, m, k, tc) == plan.needed(sms, m, k, tc), (sms, m)


def test_a_shorter_batch_can_need_more(plan):
    # 1425 rows take 25 splits of 64 x 64 tiles where 1408 and 1536 rows take fewer
    assert plan.needed(148, 4096, 1573, 0) >= 25 * 1425
