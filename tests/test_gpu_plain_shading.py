"""Scenes without maps and refraction are shaded by kernels without that code.
The same scene with an all-zero material_ior array (zero = the usual BSDF) takes
the general kernels: same image bit for bit, in single renders and in a batch
that mixes both kinds."""
import numpy as np
import pytest

import pt_gb300 as P
from pt_gb300 import scenes

pytestmark = pytest.mark.gpu


def _raws(kind):
    if kind == "batch":
        raw, cam = scenes.batch_scene(5, 900)
    elif kind == "clutter":
        raw, cam = scenes.heavy_scene(seed=2, instances=60, grids=3, spheres=3, grid_n=8, sphere_subdiv=2, emitters=6)
    else:
        raw, cam = scenes.tiny_raw("two_tris")
    return raw, dict(raw, material_ior=np.zeros(len(raw["materials"]), np.float32)), cam


def _context(raw, cam):
    hs = P.HostScene.from_raw(raw, cam)
    ctx = P.Context(0)
    ctx.upload(hs.pack())
    ctx.build_accel()
    return hs, ctx


@pytest.mark.parametrize("kind", ["tiny", "batch", "clutter"])
def test_plain_equals_general(kind):
    plain, general, cam = _raws(kind)
    images, jobs = [], []
    for raw in (plain, general):
        hs, ctx = _context(raw, cam)
        p = hs.render_params(61, 43, 3, 6)
        ctx.render(p)
        images.append(ctx.read_image().copy())
        jobs.append((ctx, p))
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
    with P.Context(0) as batch:
        for use in (jobs, jobs[:1]):
            batch.render_batch(use)
            for j in range(len(use)):
                assert np.array_equal(batch.read_batch_image(j).view(np.uint32), images[0].view(np.uint32))
