"""Bounces whose rays all leave the scene, all hit it, or divide: the packed hit list of a
wave of any length (ends of a block, of a warp, one entry)."""
import numpy as np
import pytest

from vork_b200 import Profile, scene as S

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (31, 1), (33, 1), (511, 1), (512, 1), (513, 1), (1025, 3)]


def _plane(width, height, eye, target, radiance=(1.0, 0.75, 0.5), double_sided=False):
    m = S.material((1.0, 1.0, 1.0), 1.0, 0.0, double_sided)
    m.specular_weight = 0.0
    cam = S.look_at(eye, target, fov_y_degrees=20, width=width, height=height)
    return S.Scene([S.grid((1e5, 1e5), (2, 2))], S.rows_from(1.0, (0, 0, 0))[None], np.zeros(1, np.uint32), np.zeros(1, np.uint32), [m], [],
                   cam, S.environment(radiance))


@pytest.mark.parametrize("width,height", SIZES)
def test_all_rays_leave(renderer, width, height):
    with renderer.install(_plane(width, height, (0, 5, 0), (0, 9, 0.001))) as s:
        res = s.render(Profile.reference_transport(4, 3), ids=True)
    # Three equal samples summed and divided in fp32: at most three roundings.
    assert np.allclose(res.image[..., :3], [1.0, 0.75, 0.5], rtol=1e-6, atol=0)
    assert np.all(res.primary_ids == 0xFFFFFFFF)
    assert res.stats["extension_rays"] == res.stats["paths"] and res.stats["shadow_rays"] == 0


@pytest.mark.parametrize("width,height", SIZES)
def test_all_rays_hit_and_their_next_rays_leave(renderer, width, height):
    # A white Lambert plane under a constant environment returns it (1e-5, as the plane at
    # other sizes); every camera ray hits and every next ray leaves.
    with renderer.install(_plane(width, height, (0, 5, 0.001), (0, 0, 0))) as s:
        res = s.render(Profile.reference_transport(4, 3), ids=True)
    assert np.allclose(res.image[..., :3], [1.0, 0.75, 0.5], rtol=1e-5, atol=0)
    assert np.all(res.primary_ids[..., 0] == 0)
    assert res.stats["extension_rays"] == 2 * res.stats["paths"]


def test_one_image_of_both(renderer):
    # The horizon divides the image: every pixel above it is the environment's, and the
    # whole agrees with the same samples one per wave.
    sc = _plane(513, 65, (0, 5, 0), (0, 5, 10))
    with renderer.install(sc) as s:
        a = s.render(Profile.reference_transport(4, 4), ids=True)
        b = s.render(Profile.reference_transport(4, 4, wave_samples=1), ids=True)
    assert np.array_equal(a.image, b.image) and np.array_equal(a.primary_ids, b.primary_ids)
    hit = a.primary_ids[..., 0] == 0
    assert 0.3 < hit.mean() < 0.7
    assert np.allclose(a.image[:20, :, :3], [1.0, 0.75, 0.5], rtol=1e-6, atol=0)
