"""A server beside device buffers that its context keeps idle."""
import contextlib

import numpy as np
import pytest

from vork_b200 import Profile, Renderer, abi, scene as S
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


def test_kept_buffers_count_as_allocated_and_never_refuse_a_request():
    make = lambda n: S.spheres_scene(num_spheres=n, width=160, height=120, grid_cells=40)
    prof = Profile.reference_transport(3, 1)
    with Renderer(0) as r, r.install(make(50)) as s:
        asked = s.info()["scene_bytes"]
        want = s.render(prof).image
    with Renderer(0) as r:
        r.install(make(90)).close()
        with r.install(make(50)) as s:
            held = s.info()["scene_bytes"]
            assert asked < held <= asked + 40 * MIB
            cap = 160 * 120
            with Server(r, memory_budget_bytes=1 << 40, max_jobs=4, wave_capacity=cap) as srv:
                wave = srv.step()["used_bytes"]
            # Just the room that the scene asked for: one request at a time, each to its end.
            with Server(r, memory_budget_bytes=wave + asked + cap * 32, max_jobs=4, wave_capacity=cap) as srv:
                ids = [srv.submit(s, prof) for _ in range(3)]
                st = srv.step()
                assert st["running"] == 1 and st["queued"] == 2 and st["used_bytes"] == wave + held + cap * 32
                for _ in range(100):
                    st = srv.step()
                    if st["queued"] + st["running"] == 0:
                        break
                assert all(np.array_equal(srv.images[i], want) for i in ids)


def test_a_fork_that_runs_out_of_memory_leaves_its_base(renderer):
    # 2^26 emissive triangles: each fork needs a weight tree of 512 MiB of its own.
    sc = S.spheres_scene(num_spheres=1, width=48, height=32)
    sc.meshes = [S.grid((1.0, 1.0), (256, 128))]
    sc.instance_rows = np.stack([S.rows_from(1.0, (i % 32 - 16.0, 0.0, i // 32 - 16.0)) for i in range(1024)])
    sc.instance_mesh = sc.instance_material = np.zeros(1024, np.uint32)
    sc.materials = [S.emissive(luminance=2.0, double_sided=True)]
    sc.blas_builder = abi.BLAS_BUILD_LBVH
    prof = Profile.reference_transport(2, 2)
    with renderer.install(sc) as s:
        assert sc.num_triangles == 1 << 26
        want = s.render(prof).image
        s.fork().close()
        renderer.install(S.spheres_scene(num_spheres=2, width=16, height=16)).close()
        with _device_memory_left(256 * MIB):
            with pytest.raises(abi.VkbError) as e:
                s.fork()
            assert e.value.status == abi.VKB_OUT_OF_MEMORY
        assert want[..., :3].max() > 0 and np.array_equal(s.render(prof).image, want)
