"""The instance of a warp in the kernel that takes a warp to an instance
(pt_gb300/csrc/device/warps.h), on the host: the item of every thread up to the
most instances that a scene may have (2^28 - 1, whose threads need 33 bits)."""
import subprocess

from pt_gb300 import build as native

_SRC = r"""
#include <cstdio>
#include <initializer_list>
#include "warps.h"
int main()
{
    const uint64_t items[] = {1, 7, 8, 9, 1000, (1u << 27) - 1, 1u << 27, (1u << 27) + 1, (1u << 27) + 12345, (1u << 28) - 1};
    for (uint64_t n : items)
        for (uint64_t i = n < 16 ? 0 : n - 16; i < n; i++)
            for (uint64_t lane : {0ull, 1ull, 31ull}) {
                const uint64_t thread = 32 * i + lane; // blocks of 256 threads
                const uint32_t got = pt::warp_item((uint32_t)(thread / 256), 256, (uint32_t)(thread % 256));
                if (got != i)
                    return std::printf("item %llu: %u\n", (unsigned long long)i, got), 1;
            }
    return 0;
}
"""


def test_every_item_up_to_the_most(tmp_path):
    (tmp_path / "items.cpp").write_text(_SRC)
    exe = tmp_path / "items"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{native.CSRC / 'device'}", str(tmp_path / "items.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
