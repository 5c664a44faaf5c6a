"""Which binaries the blocks and warps of a launch take, on the host: the kernels'
own index arithmetic (gbx_index.h) compiled with the C++ compiler, at sizes that
no test can run."""

import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    (d / "p.cpp").write_text(r'''
#include <cstdio>
#include <cstdlib>
#include "gbx_index.h"
using namespace gbx;
int main(int, char **v)
{
    const int n = atoi(v[1]);
    const unsigned blocks = ll_blocks(n), end = kLlBlock - 1;
    // first binaries of the first and second warps, of the first block's last warp and
    // of the last block's first and last, and the next round of those two
    printf("%u %u %u %u %u %u %u %u\n", blocks, ll_first_binary(0, 0), ll_first_binary(0, 32),
           ll_first_binary(0, end), ll_first_binary(blocks - 1, 0), ll_first_binary(blocks - 1, end),
           ll_first_binary(0, 0) + ll_stride(blocks), ll_first_binary(blocks - 1, end) + ll_stride(blocks));
    // the row-major fill: its largest grid, and the walk of a warp of a smaller one
    const unsigned grid = 1216, full = (unsigned)bulk_blocks(n);
    long long walked = 0, b = bulk_first_binary(grid - 1, kBulkWarps - 1);
    for (; b < n && walked < 10; walked++) b += bulk_stride(grid) * (n / 4096 + 1);
    printf("%d %lld %lld %lld ", bulk_blocks(n), bulk_first_binary(full - 1, 0), bulk_stride(full), b);
    // clusters where 8 and 4, only 4, only 8 and neither can be resident
    for (int fit = 0; fit < 4; fit++)
        printf("%d ", cluster_log2(n, v[2] ? atoi(v[2]) : 256, 152,
                                   [&](int lc) { return lc == 3 ? fit == 0 || fit == 2 : fit < 2; }));
}
''')
    exe = str(d / "p")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "gbgpu_gb300", "csrc"),
                    str(d / "p.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 2 ** 28 - 1, 2 ** 28, 2 ** 28 + 1, 2 ** 31 - 1])
def test_ll_covers_every_binary_once(program, n):
    out = subprocess.run([program, str(n)], capture_output=True, text=True, check=True).stdout
    blocks, first, second, end0, last_block, last, again, last_again = map(int, out.split()[:8])
    # warp w takes binaries 2w and 2w + 1, four warps a block
    assert (first, second, end0) == (0, 2, 6)
    assert blocks == -(-n // 8) and blocks < 2 ** 31
    assert last_block == 8 * (blocks - 1) < n
    assert last == 8 * (blocks - 1) + 6
    assert n <= again == 8 * blocks and last_again == again + last      # and stops after it


@pytest.mark.parametrize("n", [1, 2, 3, 2 ** 28, 2 ** 31 - 2432, 2 ** 31 - 1])
def test_row_major_fill_covers_every_binary(program, n):
    out = subprocess.run([program, str(n)], capture_output=True, text=True, check=True).stdout
    blocks, last_first, stride, end = map(int, out.split()[8:12])
    assert blocks == -(-n // 2) and last_first == 2 * (blocks - 1) < n <= stride
    assert end >= n                  # a warp's walk ends past the last binary, not below zero


@pytest.mark.parametrize("n,N,want", [(1, 256, [3, 2, 3, 0]), (19, 4096, [3, 2, 3, 0]), (20, 512, [2, 2, 0, 0]),
                                      (57, 256, [2, 2, 0, 0]), (58, 256, [0] * 4), (1, 128, [0] * 4)])
def test_clusters_only_where_they_fit(program, n, N, want):
    out = subprocess.run([program, str(n), str(N)], capture_output=True, text=True, check=True).stdout
    assert list(map(int, out.split()[12:])) == want
