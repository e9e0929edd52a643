"""The cut of a grouped design's cells into slices and pieces
(devil_b200/csrc/group_cut.h, host code): every cell once, in key order, and
slices cut at the clusters where their pieces would pass a limit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

WRAP = r"""
#include "group_cut.h"
using namespace devil;
extern "C" int cut(const int64_t* kst, int U, int C, int cells, int by, int limit, int* out, int* by_out) {
    SliceCut c = cut_slices_fitting(std::vector<int64_t>(kst, kst + (size_t)U * C + 1), U, C, cells, by != 0,
                                    [&](int pieces) { return pieces <= limit; });
    *by_out = c.by_cluster;
    for (auto* v : {&c.sl_start, &c.sl_key, &c.kslice, &c.f_key, &c.f_slice, &c.f_base, &c.f_loc, &c.f_kslice}) {
        *out++ = (int)v->size();
        for (int32_t x : *v) *out++ = x;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("cut")
    (d / "cut.cpp").write_text(WRAP)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "devil_b200", "csrc"),
                    str(d / "cut.cpp"), "-o", str(d / "cut.so")], check=True)
    lib = C.CDLL(str(d / "cut.so"))

    def run(sizes, cells, by=False, limit=1 << 30):
        U, K = sizes.shape
        kst = np.concatenate([[0], np.cumsum(sizes.reshape(-1))]).astype(np.int64)
        out, flag = np.zeros(64 + 16 * int(kst[-1]) + 16 * U * K, np.int32), C.c_int()
        lib.cut(kst.ctypes.data_as(C.c_void_p), U, K, cells, int(by), limit, out.ctypes.data_as(C.c_void_p),
                C.byref(flag))
        r, i = [], 0
        for _ in range(8):
            r.append(out[i + 1:i + 1 + out[i]])
            i += 1 + out[i]
        return kst, bool(flag.value), r

    return run


@pytest.mark.parametrize("U,K,cells,by", [(1, 1, 10, False), (3, 1, 7, False), (2, 5, 10, False), (2, 5, 10, True),
                                          (4, 9, 16, False), (3, 40, 4, False)])
def test_every_cell_once(cut, U, K, cells, by):
    rng = np.random.default_rng(U * K)
    sizes = rng.integers(0, 25, (U, K))
    sizes[0, 0] = 0
    kst, flag, (start, key, kslice, fk, fs, fb, fl, fks) = cut(sizes, cells, by)
    assert flag == (by or K == 1)
    size = np.diff(start)
    assert start[0] == 0 and start[-1] == kst[-1] and (size > 0).all() and (size <= cells).all()
    rows = np.repeat(np.arange(U), sizes.sum(1))  # design row of every cell
    assert all((rows[a:b] == u).all() for a, b, u in zip(start[:-1], start[1:], key))
    np.testing.assert_array_equal(kslice, [np.sum(key < u) for u in range(U + 1)])
    if K == 1:
        assert len(fk) == 0
        return
    first = np.append(fb + fl, kst[-1])
    keys = np.repeat(np.arange(U * K), sizes.reshape(-1))
    assert (np.diff(first) > 0).all() and first[0] == 0
    assert all((keys[a:b] == k).all() for a, b, k in zip(first[:-1], first[1:], fk))
    assert all(b <= start[s + 1] and a >= start[s] == c for a, b, s, c in zip(first[:-1], first[1:], fs, fb))
    np.testing.assert_array_equal(fks, [np.sum(fk < k) for k in range(U * K + 1)])
    if by:  # every piece is a slice
        np.testing.assert_array_equal(first, start)
        assert (fl == 0).all()


def test_cut_at_the_limit(cut):
    # 2 rows x 6 clusters of 30 cells, slices of 20: 9 slices a row; five cluster
    # ends inside a row, two of them at a slice's end: 12 pieces a row
    sizes = np.full((2, 6), 30)
    _, flag, r = cut(sizes, 20)
    pieces = len(r[3])
    assert not flag and len(r[1]) == 18 and pieces == 24
    for limit, by in ((pieces, False), (pieces - 1, True)):
        _, flag, r = cut(sizes, 20, limit=limit)
        assert flag == by
    assert len(r[1]) == len(r[3]) == 24  # two slices per cluster, each one piece
