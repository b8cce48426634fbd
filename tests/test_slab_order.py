"""The traversal's box test takes each slab's entry and exit distance from one
plane, chosen by the ray's direction sign (pt_gb300/csrc/device/slab.h).  On
the host, against the form that takes the minimum and maximum of both planes'
distances (NaN ignored): the same entry and exit for every sign, zero
components of either sign, subnormal directions whose inverse overflows,
origins on, inside and beside the slab, and both signs of zero planes."""
import subprocess

import pytest

from pt_gb300 import build as native

_SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "slab.h"
int main()
{
    const float planes[] = {-65504.0f, -3.0f, -1e-3f, -0.0f, 0.0f, 1e-3f, 2.0f, 65504.0f};
    const float origins[] = {-1e30f, -7.0f, -3.0f, -1.0f, -0.0f, 0.0f, 1e-3f, 2.0f, 5.0f, 1e30f};
    const float dirs[] = {0.0f, -0.0f, 1e-45f, -1e-45f, 1e-38f, -1e-38f, 1e-3f, -1e-3f, 0.6f, -0.6f, 1.0f, -1.0f,
                          1e30f, -1e30f, NAN};
    const float tmins[] = {0.0f, 0.1f}, tmaxs[] = {1.0f, 1000.0f, INFINITY};
    int bad = 0, n = 0;
    for (float lo : planes) for (float hi : planes) if (lo <= hi) for (float o : origins) for (float d : dirs)
        for (float tmin : tmins) for (float tmax : tmaxs) {
            const float inv = 1.0f / d, oinv = o * inv;
            const float x0 = std::fmaf(lo, inv, -oinv), x1 = std::fmaf(hi, inv, -oinv);
            const float enter = std::fmax(std::fmin(x0, x1), tmin), leave = std::fmin(std::fmax(x0, x1), tmax);
            uint32_t bits;
            std::memcpy(&bits, &inv, 4);
            const bool h = pt::slab_hi_first(bits);
            const float e = std::fmax(h ? x1 : x0, tmin), l = std::fmin(h ? x0 : x1, tmax);
            n++;
            if (!(e == enter && l == leave) && bad++ < 5)
                std::printf("lo %g hi %g o %g d %g: enter %g %g leave %g %g\n", lo, hi, o, d, enter, e, leave, l);
        }
    std::printf("%d of %d differ\n", bad, n);
    return bad != 0;
}
"""


@pytest.mark.parametrize("opt", ["-O0", "-O2"])
def test_one_plane_per_distance_equals_min_and_max(tmp_path, opt):
    src, exe = tmp_path / "slab.cpp", tmp_path / "slab"
    src.write_text(_SRC)
    subprocess.run(["g++", "-std=c++17", opt, "-ffp-contract=off", "-fno-fast-math", f"-I{native.CSRC / 'device'}", str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
