"""Traversal warps that fetch new rays while some of theirs go on (GPU): images
and traversal counts equal those of the megakernel, which traces every ray by
itself, for queues below, at and above the size from which warps do so, with and
without transparent instances.  Extend refills in one pass only, so the same
comparison also runs in a process without the step budget that the other tests
set.  No tolerance: every ray takes the same steps."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import pt_gb300 as P
from pt_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


def _render(ctx, hs, w, h, spp, kernel):
    st = ctx.render(hs.render_params(w, h, spp, 4, kernel=kernel))
    return ctx.read_image().copy(), (st.segments, st.shadow_rays, st.node_visits, st.tri_tests)


def _scene(alpha):
    rng = np.random.default_rng(7)
    meshes = []
    for k in range(5):
        p, nrm, uv, ix = scenes.displaced_grid(14, scenes.SceneRng(3 + k))
        ms = []
        for _ in range(6):
            M = np.eye(4)
            M[:3, :3] *= rng.uniform(0.2, 0.6)
            M[:3, 3] = rng.uniform(-2, 2, 3)
            ms.append(M)
        row = scenes.material_row(rng.uniform(0.2, 0.9, 3), 0.6, alpha=0.4 if alpha and k % 2 else 1.0)
        meshes.append(((p, nrm, uv, ix), row, ms))
    meshes.append((scenes.quad(2.0, 4.0, True), scenes.material_row((0, 0, 0), 1.0, 0.0, 8.0), [np.eye(4)]))
    cam = {"position": (0.0, -2.0, -6.0), "lookdir": (0.0, 2.0, 6.0), "fov_degrees": 55.0}
    return P.HostScene.from_raw(scenes.assemble_raw(meshes, (0.1, 0.15, 0.3)), cam)


def _check(w, h, spp, alpha):
    hs = _scene(alpha)
    with P.Context(0) as ctx:
        ctx.upload(hs.pack())
        ctx.build_accel()
        img, counts = _render(ctx, hs, w, h, spp, abi.PT_KERNEL_MEGA)
        got, got_counts = _render(ctx, hs, w, h, spp, abi.PT_KERNEL_WAVEFRONT)
    assert counts == got_counts
    assert np.array_equal(img.view(np.uint32), got.view(np.uint32))


# 152 x 32 resident warps, half of them counted, 32 rays each: warps are refilled from 75,393 rays on
SIZES = [(61, 37, 1), (304, 247, 1), (305, 248, 1), (509, 333, 3)]


@pytest.mark.parametrize("alpha", [False, True])
@pytest.mark.parametrize("w,h,spp", SIZES)
def test_wavefront_equals_megakernel(w, h, spp, alpha):
    _check(w, h, spp, alpha)


@pytest.mark.parametrize("alpha", [False, True])
def test_one_pass_equals_megakernel(alpha):
    root = Path(__file__).resolve().parent.parent
    code = f"import sys; sys.path[:0] = ['tests', '.']; import test_gpu_refill as t; [t._check(w, h, s, {alpha}) for w, h, s in t.SIZES]"
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, PT_EXTEND_BUDGET="0"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
