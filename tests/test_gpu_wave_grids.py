"""Waves whose kernels run on partial, exact and several blocks: every sample's bits are the
same however many path slots share its wave."""
import numpy as np
import pytest

from vork_b200 import Profile, scene as S

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
