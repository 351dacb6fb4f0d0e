"""The builder's level grids (csrc/split_grid.h), against a count of what is there: every
open segment of a level has a block for each of its tiles, and the blocks are not many
more than the tiles, whatever the jobs of a call look like."""
import ctypes as C
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MIN, TILE, HTILE = 4096, 2048, 8192

SRC = """
#include "split_grid.h"
extern "C" void grid(long long n, long long njobs, int level, long long* o) {
    const ikdg::SplitGrid g = ikdg::split_grid(n, njobs, level);
    o[0] = g.segs, o[1] = g.tiles, o[2] = g.htiles;
    o[3] = ikdg::split_segs_cap(n), o[4] = ikdg::split_tiles_cap(n), o[5] = ikdg::split_htiles_cap(n);
}
"""


@pytest.fixture(scope="module")
def grid(tmp_path_factory):
    d = tmp_path_factory.mktemp("split_grid")
    src, lib = str(d / "g.cpp"), str(d / "g.so")
    open(src, "w").write(SRC)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ikd-tree_gb300", "csrc"),
                    src, "-o", lib], check=True)
    f = C.CDLL(lib).grid
    f.argtypes = [C.c_longlong, C.c_longlong, C.c_int, C.POINTER(C.c_longlong)]

    def call(n, njobs, level):
        o = (C.c_longlong * 6)()
        f(n, njobs, level, o)
        return list(o)
    return call


def up(a, b):
    return -(-a // b)


def check(grid, jobs):
    n, njobs = sum(jobs), len(jobs)
    level, size = 0, max(jobs)
    open_ = {}
    for j in jobs:
        if j > MIN:
            open_[j] = open_.get(j, 0) + 1
    while size > MIN:
        segs = sum(open_.values())
        tiles = sum(c * up(s, TILE) for s, c in open_.items())
        htiles = sum(c * up(s, HTILE) for s, c in open_.items())
        g = grid(n, njobs, level)
        assert segs <= g[0] <= g[3] and tiles <= g[1] <= g[4] and htiles <= g[2] <= g[5]
        # the work: the points' tiles and one more per segment there can be
        assert g[1] <= n // TILE + n // MIN + 1 and g[1] < 2**31
        nxt = {}
        for s, c in open_.items():
            for h in (s // 2, s - s // 2):
                if h > MIN:
                    nxt[h] = nxt.get(h, 0) + c
        open_, size, level = nxt, size - size // 2, level + 1


def test_one_job(grid):
    for n in (4097, 8192, 8193, 8194, 140001, 2000000, 20000001, 2**30 - 1):
        check(grid, [n])


def test_one_large_job_beside_many_small_ones(grid):
    for big, small, each in ((8_000_000, 2000, 300), (2_500_000, 4000, 900), (100_000_000, 25000, 4096),
                             (150_000_000, 60000, 800), (500_000_000, 100000, 4097)):
        check(grid, [big] + [each] * small)


def test_any_jobs(grid):
    rng = random.Random(7)
    for _ in range(200):
        jobs = [int(2 ** rng.uniform(0, rng.choice((10, 13, 16, 22)))) for _ in range(rng.choice((1, 3, 50, 2000)))]
        check(grid, jobs)
