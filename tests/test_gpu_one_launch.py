"""Which bounces run in one launch, and that the wavefront's kernels (an instrumented render
runs nothing else) give the same image, rays and stopped samples."""
import numpy as np
import pytest

from vork_b200 import Profile, RadianceCache, abi, scene as S

pytestmark = pytest.mark.gpu


def _both(renderer, render, prof):
    one = render(prof)
    taken = renderer.lib.vkb_debug_path_bounces(renderer.h)
    front = render(Profile(**{**prof.__dict__, "flags": abi.PROFILE_COUNT_TRAVERSAL}))
    assert renderer.lib.vkb_debug_path_bounces(renderer.h) == 0 and front.stats["nodes_visited"] > 0
    for k in ("paths", "extension_rays", "shadow_rays", "samples_skipped", "traversal_overflows"):
        assert one.stats[k] == front.stats[k], k
    return one, front, taken


@pytest.mark.parametrize("width,height,bounces", [(1, 1, 0), (97, 61, 5), (256, 148, 5)])
def test_a_small_wave_runs_whole(renderer, width, height, bounces):
    # 256 x 148 paths are as many as the launch has lanes on 148 SMs.
    with renderer.install(S.spheres_scene(num_spheres=24, width=width, height=height)) as s:
        one, front, taken = _both(renderer, s.render, Profile.reference_transport(bounces, 1))
    assert taken == bounces + 1 and one.stats["trace_launches"] == 0 and front.stats["trace_launches"] == bounces + 1
    assert np.array_equal(one.image, front.image)


@pytest.mark.parametrize("make", [lambda: S.spheres_scene(num_spheres=24, width=331, height=317), lambda: S.lamp_scene(331, 317, seed=4)])
def test_late_bounces_of_a_larger_wave(renderer, make):
    with renderer.install(make()) as s:
        one, front, taken = _both(renderer, s.render, Profile.reference_transport(8, 1))
    assert 0 < taken < 9 and one.stats["trace_launches"] == 9
    assert np.array_equal(one.image, front.image)


@pytest.mark.parametrize("side", [128, 256])
def test_adaptive_waves(renderer, side):
    # 256 x 256 is more than the launch's lanes: only waves whose pixels have mostly stopped,
    # and late bounces, fit.
    prof = Profile(samples=32, adaptive=True, adaptive_threshold=0.05, adaptive_min_samples=16)
    with renderer.install(S.spheres_scene(num_spheres=64, width=side, height=side)) as s:
        one, front, taken = _both(renderer, s.render, prof)
    assert taken > 0 and 0 < one.stats["samples_skipped"] < 16 * side * side
    assert np.array_equal(one.image, front.image)


def test_cached_renders(renderer):
    prof = Profile.reference_transport(6, 2, wave_samples=1)
    sc = S.spheres_scene(num_spheres=24, width=160, height=120)
    with renderer.install(sc) as s, RadianceCache(s, seed=0) as cache:
        cache.train(prof)
        one, front, taken = _both(renderer, cache.render, prof)
        assert one.stats["cache_queries"] == front.stats["cache_queries"] > 0
    # Both waves' vertices up to the query (0, 1, 2).  The records reach the network in
    # another order; each one's answer is its own.
    assert taken == 6
    assert np.allclose(one.image, front.image, rtol=1e-5, atol=1e-7)
