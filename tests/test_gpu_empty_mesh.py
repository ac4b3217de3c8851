"""Meshes without triangles (their vertices still have a box that rays enter), in device
buffers that another scene used before."""
import numpy as np
import pytest

from vork_b200 import Profile, abi, scene as S

pytestmark = pytest.mark.gpu
FORMATS = {"sah": dict(), "wide8": dict(blas_format=abi.BLAS_WIDE8), "lbvh": dict(blas_builder=abi.BLAS_BUILD_LBVH), "ploc": dict(blas_builder=abi.BLAS_BUILD_PLOC)}


def _scene(kind, where):
    sc = S.spheres_scene(num_spheres=12, seed=8, width=96, height=64, grid_cells=12)
    if where is not None:
        v = np.float32([[-9, -9, -9], [9, 9, 9], [-9, 9, 0]])
        empty = S.Mesh(v, np.zeros_like(v), np.zeros((0, 3), np.uint32))
        at = 0 if where == "first" else len(sc.meshes)
        sc.meshes = sc.meshes[:at] + [empty] + sc.meshes[at:]
        sc.instance_mesh = np.append(sc.instance_mesh + (sc.instance_mesh >= at), at).astype(np.uint32)
        sc.instance_material = np.append(sc.instance_material, 0).astype(np.uint32)
        sc.instance_rows = np.concatenate([sc.instance_rows, S.rows_from(1.0, (0.0, 1.0, 0.0))[None]])
    for k, v in FORMATS[kind].items():
        setattr(sc, k, v)
    return sc


@pytest.mark.parametrize("where", ["first", "last"])
@pytest.mark.parametrize("kind", list(FORMATS))
def test_an_empty_mesh_is_never_hit(renderer, kind, where):
    rng = np.random.default_rng(3)
    d = rng.normal(size=(5000, 3)); d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([rng.uniform(-12, 12, (5000, 3)), d, np.full((5000, 1), 1e30)], 1).astype(np.float32)
    with renderer.install(_scene(kind, None)) as s:
        want, image = s.trace(rays), s.render(Profile.reference_transport(4, 2)).image
        shade = s.occluded(rays)
    renderer.install(S.spheres_scene(num_spheres=14, seed=1, width=32, height=32, grid_cells=13)).close()
    with renderer.install(_scene(kind, where)) as s:
        got, res = s.trace(rays), s.render(Profile.reference_transport(4, 2))
        assert np.array_equal(s.occluded(rays), shade)
    assert (want[1][:, 0] != 0xFFFFFFFF).any()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert res.stats["traversal_overflows"] == 0 and np.array_equal(res.image, image)


def test_a_scene_of_an_empty_mesh_only(renderer):
    sc = _scene("sah", "first")
    sc.meshes, sc.instance_rows = sc.meshes[:1], sc.instance_rows[-1:]
    sc.instance_mesh = sc.instance_material = np.zeros(1, np.uint32)
    for kind in FORMATS:
        for k, v in {"blas_format": abi.BLAS_WIDE4, "blas_builder": abi.BLAS_BUILD_SAH, **FORMATS[kind]}.items():
            setattr(sc, k, v)
        with renderer.install(sc) as s:
            res = s.render(Profile.reference_transport(3, 2))
        assert res.stats["extension_rays"] == res.stats["paths"] and res.stats["traversal_overflows"] == 0
