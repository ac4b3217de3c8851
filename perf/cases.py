"""The work a program gives this backend, as cases that can be timed and compared.

Each case is one call path of a user's program through the package: a still, a frame of
an animated flock, a batch of previews, a cached frame, the first frame of a new scene,
the display transform of a finished image.  Scenes are the synthetic generators of
`vork_b200.scene`, seeded; one `Renderer` per process is kept, as a program keeps it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vork_b200 import Profile, RadianceCache, Renderer, abi
from vork_b200 import scene as S
from vork_b200.display import display

_renderer = None


def renderer() -> Renderer:
    global _renderer
    if _renderer is None:
        _renderer = Renderer(0)
    return _renderer


class State:
    """What the program keeps between calls; closes its scenes when it is dropped."""

    def __init__(self, case, **kw):
        self.case, self.frame, self.closers = case, 0, []
        self.__dict__.update(kw)

    def __del__(self):
        for obj in self.closers:
            obj.close()


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # The first look at a small scene while it is edited: one sample of a thumbnail.
        # All latency: a few short launches and the host around them.
        dict(name="thumbnail", kind="spheres", width=128, height=128, spp=1, depth=4, spheres=16, profile="reference"),
        # The small configuration of the bench: 64 spheres and a grid, 256x256, 16 spp.
        dict(name="small_still", kind="spheres", width=256, height=256, spp=16, depth=4, spheres=64, profile="reference"),
        # A still with vork's own std/path settings (12/4/4/12 bounces, clamped indirect,
        # light threshold) at an odd resolution.
        dict(name="std_still_odd", kind="spheres", width=641, height=359, spp=12, depth=12, spheres=208, profile="std"),
        # The large configuration of the bench: a frame of a million instanced birds over
        # two million triangles of terrain, its TLAS rebuilt from rows on the device, the
        # image left on the device.
        dict(name="flock_frame", kind="flock", width=1920, height=1080, spp=64, depth=8, birds=1_000_000, cells=1000, rows="device"),
        # One frame of an animated sequence as a server renders it: a frame slot forked
        # from the installed scene takes host rows, then a short render at 640x360.
        dict(name="sequence_frame", kind="flock", width=640, height=360, spp=8, depth=8, birds=50_000, cells=300, rows="host"),
        # Previews of many scenes rendered together in one shared wavefront.
        dict(name="preview_batch", kind="batch", jobs=24, max_side=512),
        # Emissive meshes: every light is a surface (mesh next-event estimation).
        dict(name="lamps_still", kind="lamps", width=480, height=360, spp=16, depth=6, lamps=3),
        # An image environment, with the denoiser's guide planes beside the image.
        dict(name="sky_guides", kind="sky", width=400, height=300, spp=16, depth=6, spheres=64),
        # A frame through the learned radiance cache: one online training round, then the
        # cached render.
        dict(name="cached_frame", kind="cached", width=960, height=540, spp=8, depth=8, birds=100_000, cells=300),
        # Adaptive sampling: one sample per wave, settled pixels stop.
        dict(name="adaptive_still", kind="adaptive", width=256, height=256, spp=64, spheres=64),
        # A scene that has to show at once: install with BLASes built on the GPU, a first
        # frame of a few samples, and the scene dropped again.
        dict(name="first_frame", kind="install", width=640, height=360, spp=4, depth=6, birds=20_000, cells=300, builder="lbvh"),
        # The finished image on its way to a file: the display transform of a 1080p frame.
        dict(name="display_1080p", kind="display", width=1920, height=1080, display="srgb", bits=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spheres", "spheres", "flock", "flock", "batch", "lamps", "sky", "cached", "adaptive", "install", "display"])
    w = _log_int(rng, 96, 960)
    h = max(64, int(w * rng.choice([0.5625, 0.75, 1.0])) + rng.choice([0, 0, 1, 3]))
    if kind == "spheres":
        return dict(kind=kind, width=w, height=h, spp=_log_int(rng, 1, 32), depth=rng.randint(2, 12), spheres=_log_int(rng, 4, 208),
                    profile=rng.choice(["reference", "std"]))
    if kind == "flock":
        return dict(kind=kind, width=w, height=h, spp=_log_int(rng, 1, 32), depth=rng.randint(4, 8), birds=_log_int(rng, 2000, 400_000),
                    cells=rng.choice([64, 300, 500]), rows=rng.choice(["device", "host"]))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(3, 32), max_side=rng.choice([256, 512, 700]))
    if kind == "lamps":
        return dict(kind=kind, width=w, height=h, spp=_log_int(rng, 1, 24), depth=rng.randint(2, 8), lamps=rng.randint(1, 8))
    if kind == "sky":
        return dict(kind=kind, width=w, height=h, spp=_log_int(rng, 1, 24), depth=rng.randint(2, 8), spheres=_log_int(rng, 4, 128))
    if kind == "cached":
        return dict(kind=kind, width=w, height=h, spp=_log_int(rng, 2, 16), depth=rng.randint(4, 8), birds=_log_int(rng, 5000, 200_000),
                    cells=rng.choice([64, 300]))
    if kind == "adaptive":
        side = _log_int(rng, 96, 400)
        return dict(kind=kind, width=side, height=side + rng.choice([0, 1, 5]), spp=_log_int(rng, 32, 128), spheres=_log_int(rng, 8, 128))
    if kind == "install":
        return dict(kind=kind, width=w, height=h, spp=_log_int(rng, 1, 8), depth=rng.randint(3, 8), birds=_log_int(rng, 1000, 100_000),
                    cells=rng.choice([64, 300]), builder=rng.choice(["lbvh", "ploc"]))
    return dict(kind="display", width=_log_int(rng, 128, 1920), height=_log_int(rng, 128, 1080),
                display=rng.choice(["srgb", "display_p3", "rec2100_pq", "rec2100_hlg"]), bits=rng.choice([8, 16, 32]))


# ----------------------------------------------------------------------------- running
def _flock_rows(flock, scene):
    flock.step()
    return np.ascontiguousarray(np.concatenate([flock.rows(), scene.instance_rows[-1:]], 0), np.float32).reshape(-1, 12)


def prepare(case, seed):
    kind, r = case["kind"], renderer()
    if kind == "display":
        rng = np.random.default_rng(seed)
        n = (case["height"], case["width"])
        img = np.ones((*n, 4), np.float32)
        img[..., :3] = np.exp(rng.standard_normal((*n, 3), np.float32) * 1.2 - 1.0)   # a mean image's radiances, a few highlights
        return State(case, image=img)
    if kind == "batch":
        st = State(case)
        items = []
        # The jobs' shapes come from the case, so their images keep their sizes; what they show from the seed.
        for j, (job, spp, depth) in enumerate(S.preview_jobs(case["jobs"], seed=case["jobs"], max_side=case["max_side"])):
            sc = S.spheres_scene(len(job.instance_rows) - 1, seed=(seed & 0xFFFF) * 64 + j, width=job.camera.width, height=job.camera.height,
                                 grid_cells=round(math.sqrt(job.meshes[1].num_triangles / 2)))
            inst = r.install(sc)
            st.closers.append(inst)
            items.append((inst, Profile.reference_transport(depth, spp, seed=seed & 0xFFFF)))
        st.items = items
        return st
    if kind == "lamps":
        sc = S.lamp_scene(case["width"], case["height"], seed=seed, lamps=case["lamps"])
        prof = Profile.reference_transport(case["depth"], case["spp"], seed=seed & 0xFFFF)
    elif kind in ("flock", "cached", "install"):
        sc, flock = S.flock_scene(case["birds"], seed=seed, width=case["width"], height=case["height"], terrain_cells=case["cells"])
        prof = Profile.reference_transport(case["depth"], case["spp"], seed=seed & 0xFFFF)
    else:
        sc = S.spheres_scene(case["spheres"], seed=seed, width=case["width"], height=case["height"])
        if kind == "adaptive":
            prof = Profile(samples=case["spp"], seed=seed & 0xFFFF, adaptive=True, adaptive_threshold=0.02)
        elif case.get("profile") == "std":
            prof = Profile(samples=case["spp"], seed=seed & 0xFFFF)
        else:
            prof = Profile.reference_transport(case["depth"], case["spp"], seed=seed & 0xFFFF)
    if kind == "sky":
        sc.env_image = S.EnvironmentImage(S.sky_image(seed=seed))
    if kind == "install":
        sc.blas_builder = abi.BLAS_BUILD_PLOC if case["builder"] == "ploc" else abi.BLAS_BUILD_LBVH
        return State(case, scene=sc, profile=prof)
    inst = r.install(sc)
    st = State(case, scene=inst, profile=prof)
    st.closers.append(inst)
    if kind == "flock":
        rows = [_flock_rows(flock, sc) for _ in range(2)]
        if case["rows"] == "device":
            st.rows = [torch.from_numpy(x).cuda() for x in rows]
            st.out = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        else:
            st.rows = rows
            st.scene = inst.fork()
            st.closers.insert(0, st.scene)
    if kind == "cached":
        st.cache = RadianceCache(inst, seed=seed & 0xFFFF)
        st.closers.insert(0, st.cache)
    return st


def run(st):
    kind = st.case["kind"]
    if kind == "display":
        return display(renderer(), st.image, st.case["display"], bits=st.case["bits"])
    if kind == "batch":
        return renderer().render_batch(st.items)[0]
    if kind == "install":
        with renderer().install(st.scene) as inst:
            return inst.render(st.profile).image
    if kind == "cached":
        loss = st.cache.train(st.profile)["loss"]
        return {"image": st.cache.render(st.profile).image, "loss": loss}
    if kind == "flock":
        rows = st.rows[st.frame & 1]
        st.frame += 1
        if st.case["rows"] == "device":
            st.scene.update_instances_device(rows.data_ptr(), rows.shape[0])
            st.scene.render(st.profile, device_ptr=st.out.data_ptr())
            return st.out
        st.scene.update_instances(rows)
        return st.scene.render(st.profile).image
    res = st.scene.render(st.profile, guides=kind == "sky")
    return [res.image, res.guide_albedo, res.guide_normal] if kind == "sky" else res.image


# ----------------------------------------------------------------------------- work
def work(case):
    """Bytes: the scene's rows, triangles and nodes once and the image once.  Flops: per
    path an average of 2.3 vertices, each an extension and a shadow ray through a 4-wide
    tree over the instances and the mesh (24 multiply-adds a node, 60 flops a triangle
    test) and about 600 flops of shading."""
    kind = case["kind"]
    if kind == "display":
        n = case["width"] * case["height"]
        return {"bytes": n * (16 + case["bits"] // 2), "flops": n * 60}
    if kind == "batch":
        pix = case["jobs"] * (case["max_side"] * 0.5) ** 2
        paths, inst, tris = pix * 18, 50, 9152
        scenes = case["jobs"]
    else:
        pix = case["width"] * case["height"]
        paths = pix * case["spp"]
        scenes = 1
        if kind in ("flock", "cached", "install"):
            inst, tris = case["birds"] + 1, 500 + 2 * case["cells"] ** 2
        elif kind == "lamps":
            inst, tris = 10 + case["lamps"], 1000
        else:
            inst, tris = case["spheres"] + 1, 9152
    nodes = math.ceil(math.log(max(inst, 2), 4)) + math.ceil(math.log(max(tris / 2, 2), 4))
    ray = nodes * 48 + 2 * 60 + 60
    planes = 3 if kind == "sky" else 1
    return {"bytes": scenes * (inst * (48 + 128) + tris * (96 + 128 / 3)) + pix * 16 * planes, "flops": paths * 2.3 * (2 * ray + 600)}


# ----------------------------------------------------------------------------- exact
def exact(case, seed):
    """The display transform in 64 bits, where it returns float codes; path-traced images
    have no closed value, and whole codes are compared as they are."""
    if case["kind"] != "display" or case["bits"] != 32:
        return None
    img = prepare(case, seed).image.astype(np.float64)
    c, a = img[..., :3], img[..., 3:]

    def srgb(x):
        return np.where(x > .0031308, 1.055 * np.maximum(x, 0.0) ** (1 / 2.4) - .055, 12.92 * x)

    def mix(rows):
        return np.stack([sum(k * c[..., i] for i, k in enumerate(row)) for row in rows], -1)

    if case["display"] == "srgb":
        v = srgb(c)
    elif case["display"] == "display_p3":
        v = srgb(mix([(.82246197, .17753803, 0), (.03319420, .96680580, 0), (.01708263, .07239744, .91051993)]))
    else:
        n = np.clip(mix([(.62740390, .32928304, .04331307), (.06909729, .91954040, .01136232), (.01639144, .08801331, .89559525)]) * 100.0, 0.0, 1000.0)
        if case["display"] == "rec2100_pq":
            l = (n / 10000.0) ** .1593017578125
            v = ((.8359375 + 18.8515625 * l) / (1 + 18.6875 * l)) ** 78.84375
        else:
            l = n / 1000.0
            y = np.maximum(l @ np.array([.2627, .6780, .0593]), 1e-4 / 3 ** 1.2)
            e = l * (y ** ((1 - 1.2) / 1.2))[..., None]
            v = np.where(e <= 1 / 12, np.sqrt(3 * np.maximum(e, 0)), .17883277 * np.log(np.maximum(12 * e - .28466892, 1e-6)) + .55991073)
    return np.concatenate([v, a], -1)
