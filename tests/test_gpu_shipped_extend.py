"""Closest hits as a program gets them: one pass, warps that fetch new rays
while some of theirs go on.  The other tests set a step budget for every wave
(conftest.py), so these run in processes without it: a batch whose waves hold
several scenes, where the lanes of a warp come from different jobs, and the
bounds-checked library, single renders and a batch, all on more rays than the
75,393 from which warps are refilled.  Images and counts equal the megakernel's,
which traces every ray by itself; no tolerance."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import pt_gb300 as P
from pt_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

# (scene, width, height, samples, bounces): transparent, refractive and textured jobs beside plain ones
JOBS = [(("batch", 11, 2000), 211, 173, 4, 4), (("textured",), 160, 120, 3, 5), (("batch", 13, 9000), 307, 201, 2, 6),
        (("glass",), 128, 96, 5, 8), (("batch", 12, 800), 97, 260, 3, 3), (("batch", 14, 1500), 333, 217, 1, 5)]


def _scene(spec):
    raw, cam = {"batch": scenes.batch_scene, "textured": scenes.textured_raw, "glass": scenes.glass_raw}[spec[0]](*spec[1:])
    return P.HostScene.from_raw(raw, cam)


def check(plain_only):
    """Single renders and the batch of the jobs (of the plain ones: other shading kernels) against the megakernel."""
    assert not [k for k in os.environ if k.startswith("PT_EXTEND")]
    keep, jobs, want = [], [], []
    counts = np.zeros(4, np.int64)
    for spec, w, h, spp, bounces in JOBS:
        if plain_only and spec[0] != "batch":
            continue
        hs = _scene(spec)
        view = hs.pack()
        c = P.Context(0)
        c.upload(view)
        c.build_accel()
        st = c.render(hs.render_params(w, h, spp, bounces, kernel=abi.PT_KERNEL_MEGA))
        img, one = c.read_image().copy(), np.array((st.segments, st.shadow_rays, st.node_visits, st.tri_tests))
        params = hs.render_params(w, h, spp, bounces, kernel=abi.PT_KERNEL_WAVEFRONT)
        st = c.render(params)
        assert st.error_word == 0 and (one == (st.segments, st.shadow_rays, st.node_visits, st.tri_tests)).all()
        assert np.array_equal(img.view(np.uint32), c.read_image().view(np.uint32))
        keep.append((hs, view))
        jobs.append((c, params))
        want.append(img)
        counts += one
    assert sum(w * h * s for _, w, h, s, _ in JOBS) > 4 * 75393
    with P.Context(0) as ctx:
        for flags in (abi.PT_BATCH_NO_TUNE, abi.PT_BATCH_NO_TUNE | abi.PT_BATCH_NO_GRAPH | abi.PT_BATCH_CAPACITY_LOG2(18)):
            st = ctx.render_batch(jobs, flags)
            assert st.error_word == 0 and (st.segments, st.shadow_rays) == tuple(counts[:2])
            for j, img in enumerate(want):
                assert np.array_equal(ctx.read_batch_image(j).view(np.uint32), img.view(np.uint32)), j
    for c, _ in jobs:
        c.close()


@pytest.mark.parametrize("plain_only", [False, True])
@pytest.mark.parametrize("checked", [False, True])
def test_one_pass_equals_megakernel(checked, plain_only):
    env = {k: v for k, v in os.environ.items() if not k.startswith("PT_EXTEND")}
    if checked:
        env["PT_CHECKED"] = "1"
    name = "libptgpu_checked.so" if checked else "libptgpu.so"
    code = (f"import sys; sys.path[:0] = ['tests', '.']; import test_gpu_shipped_extend as t; "
            f"assert t.abi.LIB_PATH.name == '{name}'; t.check({plain_only})")
    r = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
