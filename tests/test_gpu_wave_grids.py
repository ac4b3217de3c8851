"""Waves whose kernels run on partial, exact and several blocks: every sample's bits are the
same however many path slots share its wave."""
import numpy as np
import pytest

from vork_b200 import Profile, abi, scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(1, 1), (127, 1), (128, 1), (129, 1), (512, 1), (171, 3), (641, 237)])
def test_image_does_not_depend_on_the_slots_of_a_wave(renderer, width, height):
    sc = S.spheres_scene(num_spheres=24, width=width, height=height)
    with renderer.install(sc) as s:
        whole = s.render(Profile.reference_transport(5, 3), ids=True)
        single = s.render(Profile.reference_transport(5, 3, wave_samples=1), ids=True)
        jobs, _ = renderer.render_batch([(s, Profile.reference_transport(5, 3)), (s, Profile.reference_transport(5, 3, wave_samples=1))])
    assert np.isfinite(whole.image).all() and whole.stats["traversal_overflows"] == 0
    assert whole.stats["paths"] == 3 * width * height
    for other in (single.image, *jobs):
        assert np.array_equal(whole.image, other)
    assert np.array_equal(whole.primary_ids, single.primary_ids)
    assert whole.stats["extension_rays"] == single.stats["extension_rays"]
    assert whole.stats["shadow_rays"] == single.stats["shadow_rays"]


def _lamps(w, h):
    return S.lamp_scene(w, h, seed=4), Profile.reference_transport(6, 2)


def _sky(w, h):
    sc = S.spheres_scene(num_spheres=12, width=w, height=h)
    sc.env_image = S.EnvironmentImage(S.sky_image(64, 32, seed=2))
    return sc, Profile.reference_transport(5, 2)


def _std(w, h):
    return S.spheres_scene(num_spheres=40, width=w, height=h), Profile(samples=2)


def _wide8(w, h):
    sc = S.spheres_scene(num_spheres=24, width=w, height=h)
    sc.blas_format = abi.BLAS_WIDE8
    return sc, Profile.reference_transport(5, 2)


def _empty(w, h):
    sc = S.spheres_scene(num_spheres=1, width=w, height=h)
    sc.environment = S.environment((0.5, 0.25, 0.125))
    sc.instance_rows, sc.instance_mesh, sc.instance_material = sc.instance_rows[:0], sc.instance_mesh[:0], sc.instance_material[:0]
    return sc, Profile.reference_transport(3, 2)


@pytest.mark.parametrize("make", [_lamps, _sky, _std, _wide8, _empty])
@pytest.mark.parametrize("width,height", [(3, 1), (97, 61), (200, 189), (211, 181), (331, 317)])
def test_paths_in_one_launch_equal_the_wavefront(renderer, make, width, height):
    # Small single renders run a wave's bounces (all of them, or the last ones) in one launch;
    # batches always run the wavefront's kernels.  The sizes lie on both sides of the lanes of
    # the one launch (148 SMs x 256) and where only its late bounces fit.
    sc, prof = make(width, height)
    with renderer.install(sc) as s:
        one = s.render(prof, ids=True)
        jobs, st = renderer.render_batch([(s, prof), (s, prof)])
    assert np.isfinite(one.image).all() and one.stats["traversal_overflows"] == 0
    for image in jobs:
        assert np.array_equal(one.image, image)
    assert 2 * one.stats["extension_rays"] == st["extension_rays"] and 2 * one.stats["shadow_rays"] == st["shadow_rays"]
    hit = one.primary_ids[..., 0] != 0xFFFFFFFF
    assert hit.any() == (len(sc.instance_rows) > 0) or width * height < 8
