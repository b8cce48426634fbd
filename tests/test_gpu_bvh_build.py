"""The acceleration-structure build at the sizes where it changes over: a
segment's clusters are finished by a small block (at most 512), a large block
(at most 4,096) or after rounds over all segments (more).  Every tree is
checked on the host for structure (PT_VALIDATE_BVH, set by conftest), the image
equals the oracle's bit for bit, and a second build gives the same tree."""
import numpy as np
import pytest

import oracle
import pt_gb300 as P
from pt_gb300 import scenes

pytestmark = pytest.mark.gpu


def _mesh(tris: int, seed: int):
    """A displaced grid cut to exactly `tris` triangles."""
    n = max(2, int(np.ceil(np.sqrt(tris / 2))))
    p, nrm, uv, ix = scenes.displaced_grid(n, scenes.SceneRng(seed))
    return p, nrm, uv, ix[:tris]


def _scene(tri_counts, instances):
    rng = np.random.default_rng(sum(tri_counts) + instances)
    meshes = []
    for k, t in enumerate(tri_counts):
        ms = []
        for _ in range(instances):
            M = np.eye(4)
            M[:3, :3] *= rng.uniform(0.3, 0.8)
            M[:3, 3] = rng.uniform(-2, 2, 3)
            ms.append(M)
        meshes.append((_mesh(t, 3 + k), scenes.material_row(rng.uniform(0.2, 0.9, 3), 0.6), ms))
    meshes.append((scenes.quad(2.0, 4.0, True), scenes.material_row((0, 0, 0), 1.0, 0.0, 8.0), [np.eye(4)]))
    cam = {"position": (0.0, -2.0, -6.0), "lookdir": (0.0, 2.0, 6.0), "fov_degrees": 55.0}
    return scenes.assemble_raw(meshes, (0.1, 0.15, 0.3)), cam


@pytest.mark.parametrize("tri_counts,instances", [((1, 2, 3), 1), ((255, 256, 257), 1), ((511, 512, 513), 1), ((4095, 4096), 2), ((4097, 1, 256), 1),
                                                  ((9001, 300), 1), ((2,), 300), ((5, 40), 2100)],
                         ids=["tiny", "around_256", "around_512", "up_to_4096", "past_4096", "9001", "300_instances", "4200_instances"])
def test_tree_is_valid_and_image_equals_oracle(tri_counts, instances):
    raw, cam = _scene(tri_counts, instances)
    hs = P.HostScene.from_raw(raw, cam)
    view = hs.pack()
    params = hs.render_params(48, 32, 1, 3)
    with P.Context(0) as ctx:
        ctx.upload(view)
        ctx.build_accel()  # PT_VALIDATE_BVH: fails on a malformed tree
        a = ctx.render(params)
        img = ctx.read_image().copy()
        ctx.build_accel()
        b = ctx.render(params)
        again = ctx.read_image()
    assert (a.node_visits, a.tri_tests) == (b.node_visits, b.tri_tests)
    assert np.array_equal(img.view(np.uint32), again.view(np.uint32))
    ref, _ = oracle.OracleScene(view).render(params)
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
