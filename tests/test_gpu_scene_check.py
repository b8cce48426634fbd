"""Positions and indices of an uploaded scene are checked on the device: the
first offender is named, in the order vertices, then meshes (a mesh's range
before its indices), and the context takes a good scene afterwards."""
import ctypes as C

import numpy as np
import pytest

import pt_gb300 as P
from pt_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


def _view():
    raw, cam = scenes.batch_scene(3, 700)
    hs = P.HostScene.from_raw(raw, cam)
    v = hs.pack()
    vert = np.ctypeslib.as_array(C.cast(v.vertices, C.POINTER(C.c_float)), shape=(v.vertex_count, 8))
    idx = np.ctypeslib.as_array(C.cast(v.indices, C.POINTER(C.c_uint32)), shape=(v.index_count,))
    ranges = np.ctypeslib.as_array(C.cast(v.meshes, C.POINTER(C.c_uint32)), shape=(v.mesh_count, 4))
    return hs, v, vert, idx, ranges


def _bad_vertices(vert, idx, ranges):
    vert[-1, 2] = np.nan
    vert[len(vert) // 2, 0] = -np.inf
    idx[0] = 1 << 30
    return f"vertex {len(vert) // 2} has a non-finite position"


def _last_vertex(vert, idx, ranges):
    vert[-1, 1] = np.inf
    return f"vertex {len(vert) - 1} has a non-finite position"


def _two_indices(vert, idx, ranges):
    m = len(ranges) - 1
    idx[ranges[m, 1] + 3 * ranges[m, 2] - 1] = ranges[m, 3]  # the last corner of the last mesh, one past its vertices
    idx[ranges[1, 1] + 1] = 0xFFFFFFFF
    return "mesh 1 has an index outside its vertices"


def _last_corner(vert, idx, ranges):
    m = len(ranges) - 1
    idx[ranges[m, 1] + 3 * ranges[m, 2] - 1] = ranges[m, 3]
    return f"mesh {m} has an index outside its vertices"


def _index_before_range(vert, idx, ranges):
    ranges[2, 2] = 0x10000000
    idx[ranges[1, 1]] = ranges[1, 3]
    return "mesh 1 has an index outside its vertices"


def _range(vert, idx, ranges):
    ranges[2, 2] = 0x10000000
    return "mesh 2 range outside the vertex/index arrays"


@pytest.mark.parametrize("spoil", [_bad_vertices, _last_vertex, _two_indices, _last_corner, _index_before_range, _range])
def test_first_offender_is_named(spoil):
    with P.Context(0) as ctx:
        hs, v, vert, idx, ranges = _view()
        want = spoil(vert, idx, ranges)
        with pytest.raises(P.PtError) as e:
            ctx.upload(v)
        assert e.value.status == abi.PT_ERR_INVALID and want in str(e.value), str(e.value)
        good, view, *_ = _view()
        ctx.upload(view)
        ctx.build_accel()
        assert ctx.render(good.render_params(16, 12, 1, 2)).error_word == 0
