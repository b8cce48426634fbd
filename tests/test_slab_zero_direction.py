"""Box tests of rays with zero direction components (pt_gb300/csrc/device/slab.h).

On the host: a slab that holds the origin is never missed and one beside it is,
whatever side of coordinate 0 its planes are on, for both signs of zero and for
components so small that o / d overflows; every other component keeps 1 / d and
o / d as they are.  On the GPU: scenes lit along the axes, where every shadow
ray has two zero components, with occluders across the coordinate planes, equal
the oracle's image bit for bit.  No tolerance: whether a ray hits is exact."""
import subprocess

import numpy as np
import pytest

import oracle
import pt_gb300 as P
from pt_gb300 import abi, build as native, scenes

_SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "slab.h"
int main()
{
    const float at[] = {-3e38f, -1e30f, -65504.0f, -3.0f, -1.0f, -0.5f, -1e-3f, -1e-6f, -0.0f, 0.0f, 1e-6f, 1e-3f, 0.5f, 1.0f, 2.0f, 65504.0f, 1e30f, 3e38f};
    const float dirs[] = {0.0f, -0.0f, 1e-45f, -1e-45f, 1e-39f, -1e-39f, 1e-38f, -1e-38f, 1e-30f, -1e-30f, 1e-3f, -1e-3f, 0.6f, -0.6f, 1.0f, -1.0f, 1e30f};
    const float far = 1e15f; // no ray here is longer
    int bad = 0, n = 0;
    auto fail = [&](const char* what, float lo, float hi, float o, float d, float e, float l) {
        if (bad++ < 8)
            std::printf("%s: lo %g hi %g o %g d %g: enter %g leave %g\n", what, lo, hi, o, d, e, l);
    };
    for (float o : at) for (float d : dirs) {
        float inv = 1.0f / d, oinv = o * inv;
        pt::slab_finite(o, inv, oinv);
        if (!std::isfinite(inv) || !std::isfinite(oinv) || std::signbit(inv) != std::signbit(d))
            fail("inverse", 0, 0, o, d, inv, oinv);
        const bool plain = std::isfinite(1.0f / d) && std::isfinite(o * (1.0f / d));
        if (plain && (inv != 1.0f / d || oinv != o * (1.0f / d)))
            fail("changed", 0, 0, o, d, inv, oinv);
        if (std::fabs(d) > 1e-30f || plain)
            continue;
        uint32_t bits;
        std::memcpy(&bits, &inv, 4);
        const bool h = pt::slab_hi_first(bits);
        for (float lo : at) for (float hi : at) if (lo <= hi) {
            const float x0 = std::fmaf(lo, inv, -oinv), x1 = std::fmaf(hi, inv, -oinv);
            const float e = h ? x1 : x0, l = h ? x0 : x1;
            n++;
            if (lo < o && o < hi && !(e < 0.0f && l > far))
                fail("inside, missed", lo, hi, o, d, e, l);
            if (lo <= o && o <= hi && !(e <= 0.0f && l >= 0.0f))
                fail("on a plane, missed", lo, hi, o, d, e, l);
            if ((o < lo || hi < o) && !(e > far || l < 0.0f))
                fail("beside, entered", lo, hi, o, d, e, l);
        }
    }
    std::printf("%d of %d wrong\n", bad, n);
    return bad != 0;
}
"""


@pytest.mark.parametrize("opt", ["-O0", "-O2"])
def test_a_slab_that_holds_the_origin_is_entered(tmp_path, opt):
    src, exe = tmp_path / "slab.cpp", tmp_path / "slab"
    src.write_text(_SRC)
    subprocess.run(["g++", "-std=c++17", opt, "-ffp-contract=off", "-fno-fast-math", f"-I{native.CSRC / 'device'}", str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def axis_lit_scene(direction, instances):
    """Displaced grids (many small triangles, nodes on both sides of every
    coordinate plane) between a plane and a light along an axis: one
    mesh, or many instances of it around the origin."""
    ms = []
    rng = np.random.default_rng(5)
    for k in range(instances):
        M = np.eye(4)
        if instances > 1:
            M[:3, :3] *= 0.3
            M[:3, 3] = rng.uniform(-1.5, 1.5, 3)
        ms.append(M)
    p, n, uv, ix = scenes.displaced_grid(12, scenes.SceneRng(3))
    if abs(direction[2]) == 1:  # the light is on the side of the camera: stand the grid up
        p, n = p[:, [0, 2, 1]].copy(), n[:, [0, 2, 1]].copy()
    meshes = [((p, n, uv, ix), scenes.material_row((0.8, 0.5, 0.3), 0.6), ms)]
    wall = scenes.quad(8.0, -2.0, False)
    if abs(direction[2]) == 1:
        wp, wn, wuv, wix = wall
        wp, wn = wp[:, [0, 2, 1]].copy(), wn[:, [0, 2, 1]].copy()
        wp[:, 2], wn[:, 2] = -2.0, 1.0
        wall = (wp, wn, wuv, wix)
    meshes.append((wall, scenes.material_row((0.7, 0.7, 0.7), 0.8), [np.eye(4)]))
    raw = scenes.assemble_raw(meshes, (0.05, 0.05, 0.08))
    raw["directional_lights"] = np.array([[*direction, 3.0, 2.5, 2.0]], np.float32)
    cam = {"position": (0.5, -4.0, -6.0), "lookdir": (-0.5, 4.0, 6.0), "fov_degrees": 50.0}
    return P.HostScene.from_raw(raw, cam)


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [abi.PT_KERNEL_WAVEFRONT, abi.PT_KERNEL_MEGA], ids=["wavefront", "mega"])
@pytest.mark.parametrize("instances", [1, 40])
@pytest.mark.parametrize("direction", [(0.0, 1.0, 0.0), (0.0, 0.0, 1.0)], ids=["y", "z"])
def test_axis_parallel_light_bitexact(direction, instances, kernel):
    hs = axis_lit_scene(direction, instances)
    view = hs.pack()
    params = hs.render_params(96, 64, 2, 3, kernel=kernel)
    with P.Context(0) as ctx:
        ctx.upload(view)
        ctx.build_accel()
        ctx.render(params)
        img = ctx.read_image().copy()
    ref, _ = oracle.OracleScene(view).render(params)
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
