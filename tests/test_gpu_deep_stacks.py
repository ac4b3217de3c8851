"""Traversal stacks on trees as deep as they get: a geometric series of triangles, whose
trees are chains.  Stack needs were counted on the CPU from the same trees."""
import numpy as np
import pytest

from vork_b200 import abi, scene as S

pytestmark = pytest.mark.gpu
RATIO, FIRST = 1.25, 1e-3


def _chain(renderer, count, first=FIRST, ratio=RATIO, **kw):
    # Triangle i: (x, 0, 0), (x, 0, x), (x, x, 0) at x = first * ratio^i, so the ray from the
    # origin along (1, a, a) crosses every triangle for a < 0.5 and every box for a < 1.
    x = (first * ratio ** np.arange(count)).astype(np.float32)
    z = np.zeros_like(x)
    pos = np.stack([np.stack([x, z, z], 1), np.stack([x, z, x], 1), np.stack([x, x, z], 1)], 1).reshape(-1, 3)
    nrm = np.tile(np.float32([-1, 0, 0]), (3 * count, 1))
    sc = S.spheres_scene(num_spheres=1, width=16, height=16)
    sc.meshes = [S.Mesh(pos, nrm, np.arange(3 * count, dtype=np.uint32).reshape(-1, 3))]
    sc.instance_rows = S.rows_from(1.0, (0.0, 0.0, 0.0)).reshape(1, 3, 4)
    sc.instance_mesh = sc.instance_material = np.zeros(1, np.uint32)
    for k, v in kw.items():
        setattr(sc, k, v)
    return renderer.install(sc)


def _ray(a):
    d = np.array([1.0, a, a]) / np.sqrt(1 + 2 * a * a)
    return np.concatenate([[0, 0, 0], d, [1e30]]).astype(np.float32)[None]


@pytest.mark.parametrize("count,need", [(100, 85), (141, 120), (144, 122), (150, 127)])
def test_8wide_stack_holds_128_entries(renderer, count, need):
    # `need` entries are on the stack when the first leaf, the nearest triangle, is reached.
    with _chain(renderer, count, blas_format=abi.BLAS_WIDE8) as s:
        t, ids, _ = s.trace(_ray(0.3))
        assert ids.tolist() == [[0, 0]]
        assert abs(t[0] / (FIRST * np.sqrt(1.18)) - 1) < 1e-5
        assert s.occluded(_ray(0.3)).all() and not s.occluded(_ray(0.6)).any()


# Chains of 400 triangles from 2e-23 (areas down to the smallest floats) to 1e9.
LONG = dict(count=400, first=1e9 * 1.2 ** -399, ratio=1.2, blas_builder=abi.BLAS_BUILD_PLOC)


@pytest.mark.parametrize("chain", [dict(count=n, blas_builder=abi.BLAS_BUILD_PLOC) for n in (100, 200, 220)] + [LONG])
def test_any_hit_rays_need_no_more_stack_than_sorted_children(renderer, chain):
    # A PLOC chain takes two triangles a level.  From the near end a ray that visits every
    # child far to near has at most three entries waiting; one that takes the chain ahead of
    # a nearer leaf has one more a level, and 64 (80 with the shared part) hold.
    with _chain(renderer, **chain) as s:
        assert s.occluded(_ray(0.3)).all() and not s.occluded(_ray(0.6)).any()


def test_an_occlusion_ray_that_runs_out_is_traced_again_in_order(renderer):
    # Along the ray: the long chain, whose triangles it misses; a wall; a triangle whose box
    # alone it meets.  Far to near it meets the wall before the chain, in slot order after it.
    with _chain(renderer, **LONG) as s:
        sc = s.scene
    tri = lambda *v: S.Mesh(np.float32(v), np.zeros((3, 3), np.float32), np.uint32([[0, 1, 2]]))
    sc.meshes = [sc.meshes[0], tri((3e9, -1e10, -1e10), (3e9, 4e10, -1e10), (3e9, -1e10, 4e10)), tri((5e9, 1e9, 1e9), (5e9, 4e9, 1e9), (5e9, 1e9, 4e9))]
    sc.instance_rows = np.stack([S.rows_from(1.0, (0.0, 0.0, 0.0))] * 3)
    sc.instance_mesh, sc.instance_material = np.uint32([0, 1, 2]), np.zeros(3, np.uint32)
    with renderer.install(sc) as s:
        assert s.occluded(np.repeat(_ray(0.6), 33, 0)).all()
        before_the_wall = _ray(0.6)
        before_the_wall[0, 6] = 3e9
        assert not s.occluded(before_the_wall).any()
