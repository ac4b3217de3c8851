"""A server beside device buffers that its context keeps idle."""
import contextlib

import numpy as np
import pytest

from vork_b200 import Profile, Renderer, scene as S
from vork_b200.serving import Server

pytestmark = pytest.mark.gpu
MIB = 1 << 20


@contextlib.contextmanager
def _device_memory_left(most):
    """Another user of the device holds all of its memory but less than `most` bytes."""
    import torch
    blocks, step = [], None
    try:
        while (free := torch.cuda.mem_get_info()[0]) >= most:
            step = max(10 * MIB, min(step or free, free - most * 3 // 4))
            try:
                blocks.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                if step == 10 * MIB:
                    break
                step //= 2
        yield torch.cuda.mem_get_info()[0]
    finally:
        blocks.clear()
        torch.cuda.empty_cache()


def test_a_request_gets_the_memory_that_closed_scenes_left_idle():
    big = S.spheres_scene(num_spheres=6, width=1024, height=1024, grid_cells=8)   # 2 x 16 MiB of buffers
    small = S.spheres_scene(num_spheres=6, width=64, height=64, grid_cells=8)
    prof = Profile.reference_transport(3, 1)
    with Renderer(0) as r, r.install(big) as s, r.install(small) as t:
        want = s.render(prof).image
        with Server(r, max_jobs=2, wave_capacity=1024 * 1024) as srv:
            srv.submit(t, prof)
            srv.run_until_idle()   # the kernels are loaded
            r.install(S.flock_scene(300_000, width=16, height=16, terrain_cells=300)[0]).close()   # over 100 MiB idle
            with _device_memory_left(16 * MIB) as free:
                assert free < 16 * MIB
                rid = srv.submit(s, prof)
                srv.run_until_idle()
            assert np.array_equal(srv.images[rid], want)
