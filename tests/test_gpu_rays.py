"""The ray entry (x2_trace_rays: closest hit and occlusion, each ray's two queries walked apart) and the BVH build's cuts of
the wide nodes, against every triangle tested in double precision: triangle counts about the sizes of a leaf and of a
wide node, ray counts about a warp's, and one beyond a lane for every query."""
import ctypes as C

import numpy as np
import pytest

from oracle_lib import x2

pytestmark = pytest.mark.gpu
# t: the watertight test's float error is a few ulps of the vertices' distances (under 4 here) times 1 / |det|'s spread; a
# ray that grazes its triangle at a cosine below 0.02 is left out.
RTOL, GRAZING = 1e-4, 0.02


def soup(ctx, count, seed):
    """`count` random triangles in one mesh under the box's light and camera."""
    s = x2.SyntheticScene(0)
    d = s.desc
    rng = np.random.default_rng(seed)
    centre = rng.uniform(-1, 1, (count, 1, 3))
    size = 0.4 if count <= 300 else 0.1
    v = (centre + rng.uniform(-size, size, (count, 3, 3))).astype(np.float32)
    vertices, triangles = np.ascontiguousarray(v.reshape(-1)), np.arange(3 * count, dtype=np.uint32)
    first, material = np.array([0, count], np.uint32), np.zeros(1, np.uint32)
    d.vertex_count, d.triangle_count, d.mesh_count = 3 * count, count, 1
    d.vertices, d.triangles = vertices.ctypes.data_as(C.POINTER(C.c_float)), triangles.ctypes.data_as(C.POINTER(C.c_uint32))
    d.mesh_first, d.mesh_material = first.ctypes.data_as(C.POINTER(C.c_uint32)), material.ctypes.data_as(C.POINTER(C.c_uint32))
    return x2.Scene(ctx, d, s.config), v.astype(np.float64)


def every_triangle(v, o, d, far):
    """The nearest hit's t in (0, far] of each ray (inf: none), its triangle, and the least margin of any triangle's edges."""
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    p = np.cross(d[:, None], e2[None])
    det = (p * e1[None]).sum(-1)
    q0 = o[:, None] - v[None, :, 0]
    u = (q0 * p).sum(-1) / det
    q = np.cross(q0, e1[None])
    w = (q * d[:, None]).sum(-1) / det
    t = (q * e2[None]).sum(-1) / det
    margin = np.minimum(np.minimum(u, w), 1 - u - w)
    cosine = np.abs(det) / np.linalg.norm(np.cross(e1, e2), axis=-1)[None]
    hit = np.where((margin >= 0) & (t > 0) & (t <= far[:, None]), t, np.inf)
    # Unclear to a float test: an edge passed closely, an end of the range met closely, a grazed triangle.
    near = (margin > -1e-3) & (t > -1e-3) & (t < far[:, None] + 1e-3)
    unclear = (near & ((margin < 1e-3) | (np.abs(t) < 1e-3) | (np.abs(t - far[:, None]) < 1e-3) | (cosine < GRAZING))).any(1)
    return hit.min(1), hit.argmin(1), unclear


@pytest.mark.parametrize("triangles,rays", [(1, 1), (2, 31), (3, 33), (4, 500), (5, 500), (8, 129), (9, 500), (24, 500), (25, 500), (300, 4097), (1500, 2001),
                                            (5, 90001), (1500, 90001), (29, 500), (30, 500)])  # 4 and 5 nodes: the two kernels
def test_rays_against_every_triangle(ctx, triangles, rays):
    scene, v = soup(ctx, triangles, 100 + triangles)
    rng = np.random.default_rng(triangles)
    o, target = rng.uniform(-2, 2, (rays, 3)), rng.uniform(-1, 1, (rays, 3))
    d = target - o
    length = np.linalg.norm(d, axis=1)
    q = np.zeros((rays, 8), np.float32)
    q[:, :3], q[:, 3:6] = o, d / length[:, None]
    q[:, 7] = np.where(rng.random(rays) < 0.5, length, 100.0)
    tri, t, occluded = scene.trace_rays(q)
    scene.free()
    assert np.array_equal(occluded == 1, tri != 0xffffffff)  # the same triangles on the same range
    some = np.arange(rays) if rays < 5000 else np.concatenate([np.arange(1000), np.arange(rays - 1000, rays)])
    q, tri, t = q[some], tri[some], t[some]
    want, which, unclear = every_triangle(v, q[:, :3].astype(np.float64), q[:, 3:6].astype(np.float64), q[:, 7].astype(np.float64))
    clear = ~unclear
    assert clear.mean() > 0.5 or rays == 1
    assert np.array_equal(tri[clear] != 0xffffffff, np.isfinite(want[clear]))
    hit = clear & np.isfinite(want)
    assert np.array_equal(tri[hit], which[hit])
    assert np.allclose(t[hit], want[hit], rtol=RTOL)
    assert (t[tri == 0xffffffff] == 0).all()
