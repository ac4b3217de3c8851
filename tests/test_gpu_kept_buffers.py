"""Device buffers kept between scenes and display calls of one context: what they hold never
shows, they are bounded, and threads do not share one."""
import threading

import numpy as np
import pytest

from vork_b200 import Profile, abi, scene as S
from vork_b200.display import display

pytestmark = pytest.mark.gpu
PROF = Profile.reference_transport(4, 2)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_scenes_in_reused_buffers_render_as_before(renderer):
    makes = [lambda: S.spheres_scene(num_spheres=30, width=65, height=43), lambda: S.lamp_scene(65, 43, seed=2),
             lambda: S.flock_scene(3000, width=65, height=43, terrain_cells=40)[0], lambda: S.spheres_scene(num_spheres=5, width=65, height=43, grid_cells=8)]
    builders = (abi.BLAS_BUILD_SAH, abi.BLAS_BUILD_LBVH, abi.BLAS_BUILD_PLOC)
    first = {}
    for turn in range(3):
        order = range(len(makes)) if turn != 1 else reversed(range(len(makes)))
        for k in order:
            for builder in builders:
                sc = makes[k]()
                sc.blas_builder = builder
                with renderer.install(sc) as s, s.fork() as f:
                    image = s.render(PROF).image
                    rows = sc.instance_rows.copy()
                    rows[0, :, 3] += 0.25
                    f.update_instances(rows)
                    moved = f.render(PROF).image
                want = first.setdefault((k, builder), (image, moved))
                assert np.array_equal(image, want[0]) and np.array_equal(moved, want[1])


def test_idle_buffers_are_bounded(renderer):
    img = np.random.default_rng(0).random((540, 960, 4), np.float32)
    for _ in range(3):
        display(renderer, img)
    before = _free()
    for _ in range(40):
        display(renderer, img)
    assert before - _free() < 32 << 20
    sc = S.flock_scene(400_000, width=16, height=16, terrain_cells=400)[0]
    for _ in range(2):
        with renderer.install(sc) as s:
            s.render(Profile.reference_transport(1, 1))
    assert before - _free() < (256 << 20) + (64 << 20)


def test_display_from_several_threads(renderer):
    rng = np.random.default_rng(1)
    jobs = [(rng.random((64 + 31 * k, 97, 4), np.float32), b) for k in range(6) for b in (8, 16, 32)]
    want = [display(renderer, img, bits=b) for img, b in jobs]
    bad = []

    def work(offset):
        for i in range(offset, len(jobs), 3):
            for _ in range(8):
                if not np.array_equal(display(renderer, jobs[i][0], bits=jobs[i][1]), want[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(o,)) for o in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
