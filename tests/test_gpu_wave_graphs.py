"""Waves replayed from captured graphs (a server on one stream): the images are those of
the requests rendered alone, whatever waves were captured before."""
import numpy as np
import pytest

from vork_b200 import Profile, abi, scene as S
from vork_b200.serving import Server

pytestmark = pytest.mark.gpu


def _serve(renderer, groups, spp=1):
    """Each group's sizes as requests of one wave, group after group on one server."""
    scenes = {}
    try:
        with Server(renderer, max_jobs=8, wave_capacity=20000, flags=abi.PROFILE_SERIAL_WAVES | abi.BATCH_FAIR) as srv:
            for group in groups:
                for w, h in group:
                    if (w, h) not in scenes:
                        scenes[w, h] = renderer.install(S.spheres_scene(num_spheres=6, seed=w, width=w, height=h, grid_cells=8))
                ids = [srv.submit(scenes[size], Profile.reference_transport(4, spp, seed=k)) for k, size in enumerate(group)]
                srv.run_until_idle()
                for k, (rid, size) in enumerate(zip(ids, group)):
                    alone = scenes[size].render(Profile.reference_transport(4, spp, seed=k)).image
                    assert np.array_equal(srv.images[rid], alone), (group, k)
    finally:
        for s in scenes.values():
            s.close()


def test_a_wave_is_not_replayed_from_a_graph_of_another_job_count(renderer):
    # 2 x 7500 paths, then 3 x 4484: trace grids of 938 and 841 blocks, equal shade grids.
    _serve(renderer, [[(75, 100)] * 2, [(59, 76)] * 3, [(75, 100)] * 2])


def test_waves_of_many_sizes_share_few_graphs(renderer):
    # More waves than are kept, their sizes on both sides of the grids' powers of two.
    rng = np.random.default_rng(5)
    sizes = [(int(w), int(h)) for w, h in zip(rng.integers(20, 60, 24), rng.integers(20, 90, 24))] + [(32, 32), (33, 31), (64, 64), (65, 63)]
    _serve(renderer, [[sizes[int(k)] for k in rng.integers(0, len(sizes), rng.integers(2, 9))] for _ in range(90)])
