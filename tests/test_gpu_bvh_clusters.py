"""The acceleration-structure build where large segments share out their search
over a cluster of blocks: one segment and several beside small ones, as many as
leave two blocks or one to each, and more segments than multiprocessors.  The
tree is checked on the host (PT_VALIDATE_BVH, set by conftest), the image equals
the oracle's bit for bit, and a second build gives the same tree."""
import numpy as np
import pytest

import oracle
import pt_gb300 as P
from pt_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(tri_counts):
    rng = np.random.default_rng(len(tri_counts))
    meshes = []
    for k, t in enumerate(tri_counts):
        n = max(2, int(np.ceil(np.sqrt(t / 2))))
        p, nrm, uv, ix = scenes.displaced_grid(n, scenes.SceneRng(3 + k))
        M = np.eye(4)
        M[:3, :3] *= rng.uniform(0.2, 0.6)
        M[:3, 3] = rng.uniform(-2, 2, 3)
        meshes.append(((p, nrm, uv, ix[:t]), scenes.material_row(rng.uniform(0.2, 0.9, 3), 0.6), [M]))
    meshes.append((scenes.quad(2.0, 4.0, True), scenes.material_row((0, 0, 0), 1.0, 0.0, 8.0), [np.eye(4)]))
    cam = {"position": (0.0, -2.0, -6.0), "lookdir": (0.0, 2.0, 6.0), "fov_degrees": 55.0}
    return scenes.assemble_raw(meshes, (0.1, 0.15, 0.3)), cam


@pytest.mark.parametrize("tri_counts", [(4096,), (1500, 3, 700, 64, 65, 2048), (600,) * 20 + (40,) * 10, (530,) * 60, (520,) * 100,
                                        (513, 20) * 100],
                         ids=["one_of_4096", "some_beside_small", "20_large", "60_large", "100_large", "200_segments"])
def test_tree_is_valid_and_image_equals_oracle(tri_counts):
    raw, cam = _scene(tri_counts)
    hs = P.HostScene.from_raw(raw, cam)
    view = hs.pack()
    params = hs.render_params(40, 24, 1, 2)
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
