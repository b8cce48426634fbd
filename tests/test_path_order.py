"""The order of a wave's paths (pt_gb300/csrc/device/order.h), on the host:
every pixel and every sample of it exactly once, path_at the inverse of
path_place, at image sizes with whole, ragged and missing tiles and sample
counts below, at and around the group size."""
import subprocess

import pytest

from pt_gb300 import build as native

_SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "order.h"
int main(int argc, char** argv)
{
    const uint32_t w = std::atoi(argv[1]), h = std::atoi(argv[2]), n = w * h;
    std::vector<int> seen(n, 0);
    for (uint32_t q = 0; q < n; q++) {
        uint32_t x, y;
        pt::ordered_pixel(q, w, h, x, y);
        if (x >= w || y >= h || seen[y * w + x]++)
            return std::printf("place %u: pixel %u %u\n", q, x, y), 1;
    }
    for (uint32_t k : {1u, 2u, 7u, 8u, 9u, 16u, 23u}) {
        std::vector<int> used((size_t)n * k, 0);
        for (uint32_t p = 0; p < n * k; p++) {
            uint32_t q, j;
            pt::path_place(p, n, k, q, j);
            if (q >= n || j >= k || used[(size_t)q * k + j]++ || pt::path_at(q, j, n, k) != p)
                return std::printf("%u samples, path %u: place %u sample %u\n", k, p, q, j), 1;
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(_SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{native.CSRC / 'device'}", str(d / "order.cpp"), "-o", str(d / "order")], check=True)
    return d / "order"


@pytest.mark.parametrize("size", [(1, 1), (8, 4), (7, 3), (9, 5), (16, 8), (333, 217), (1, 40), (40, 1), (64, 6), (13, 48)])
def test_every_path_once(program, size):
    r = subprocess.run([str(program), str(size[0]), str(size[1])], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
