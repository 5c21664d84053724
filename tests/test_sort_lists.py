"""The lists of a sort round hold every segment that its levels can send them:
the capacities (csrc/sort_lists.h) against a count of the finished segments that
keys of a few distinct values leave.  No GPU needed."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
COPY_SPLIT = 4096

SHIM = """
#include "sort_lists.h"
extern "C" void caps(uint64_t n, uint32_t local_max, uint32_t key_bits, uint64_t *out)
{
    const fmcs::SortListCaps c = fmcs::sort_list_caps(n, local_max, key_bits);
    out[0] = c.large; out[1] = c.copy; out[2] = c.copy_large;
}
"""


@pytest.fixture(scope="module")
def caps(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("lists") / "caps.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-x", "c++", "-", "-o", so,
                    "-I", os.path.join(ROOT, "fastmulticolsort_b200", "csrc")], input=SHIM.encode(), check=True)
    lib = ctypes.CDLL(so)

    def f(n, local_max, key_bits):
        out = (ctypes.c_uint64 * 3)()
        lib.caps(ctypes.c_uint64(n), local_max, key_bits, out)
        return dict(zip(("large", "copy", "copy_large"), out))
    return f


def _lists(codes, counts, local_max, key_bits):
    """Radix levels of 8 bits over one segment of these codes (ascending) and row
    counts: the most large segments of a level, and the finished ones by size."""
    segs, shift = [(0, len(codes))], key_bits
    most = copy = copy_large = 0
    while segs and shift:
        most = max(most, len(segs))
        shift -= min(8, shift)
        nxt = []
        for a, b in segs:
            cuts = np.flatnonzero(np.diff(codes[a:b] >> shift)) + a + 1
            for lo, hi in zip([a, *cuts], [*cuts, b]):
                rows = int(counts[lo:hi].sum())
                if rows == 1 or shift == 0:
                    copy_large += rows > COPY_SPLIT
                    copy += rows <= COPY_SPLIT
                elif rows > local_max:
                    nxt.append((lo, hi))
        segs = nxt
    return dict(large=most, copy=copy, copy_large=copy_large)


@pytest.mark.parametrize("local_max", [128, 2048, 4096, 8192])
@pytest.mark.parametrize("rows", [1, 2, 4096, 4097, 5000, 8192])
@pytest.mark.parametrize("key_bits,groups", [(8, 256), (12, 700), (12, 4096), (20, 600)])
def test_every_finished_segment_has_a_place(caps, key_bits, groups, rows, local_max):
    codes = np.sort(np.random.default_rng(groups).permutation(1 << min(key_bits, 12))[:groups].astype(np.int64))
    if key_bits == 20:   # two codes for each of their first 16 bits: finished at the third level
        codes = np.sort(np.concatenate([codes[:groups // 2] << 4, (codes[:groups // 2] << 4) + 9]))
    n = groups * rows
    need = _lists(codes, np.full(groups, rows), local_max, key_bits)
    have = caps(n, local_max, key_bits)
    for k in need:
        assert need[k] <= have[k], (k, need[k], have[k])
