"""The render work whose speed is tracked: a list of cases, each a call (or a
few) that a program built on this framework makes, with its inputs.

A case is a dict of plain values. ``prepare`` makes what the program holds
before the call (a loaded job, its scene generated from the seed), ``run``
makes the call through the public API and returns the images, ``work`` counts
what the call cannot do without, ``exact`` gives the closest-hit distances in
64 bits. Every scene comes from ``hastyrenderer_gb300.scenes`` with the sizes
of the benchmark workloads or generic ones.

Kinds:
  cornell, field, room, stress  render n passes of a job and read its images
  batch    several jobs of uneven size in one call
  photon   progressive photon-mapping iterations from the start
  load     a job file to its first image (parse, BVH build, upload, one pass)
  rays     closest hits of a list of rays
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from hastyrenderer_gb300 import scenes
from hastyrenderer_gb300.api import AOV_ALBEDO, AOV_COLOR, AOV_NORMAL, RenderJob, batch_render, load_jobs

RESOLUTIONS = [(128, 128), (256, 192), (512, 512), (1024, 768)]   # of the mixed-job workload


def listed():
    return [
        # an editor's preview: one pass of a small frame, shown after each pass
        {"name": "cornell_preview_128", "kind": "cornell", "width": 128, "height": 128, "spp": 1, "depth": 8,
         "mis": True, "aovs": False},
        # the small benchmark configuration: a closed room, all of its 64 passes
        {"name": "cornell_256", "kind": "cornell", "width": 256, "height": 256, "spp": 64, "depth": 8, "mis": True,
         "aovs": False},
        # a final frame of a closed room with deep paths, and the normal and
        # albedo images that a denoiser takes beside the colour
        {"name": "cornell_1024x768", "kind": "cornell", "width": 1024, "height": 768, "spp": 48, "depth": 16,
         "mis": True, "aovs": True},
        # an ordinary outdoor frame: 64 thousand triangles, sky light, thin lens
        {"name": "field_512", "kind": "field", "spheres": 50, "width": 512, "height": 512, "spp": 16, "depth": 10,
         "mis": True, "lens": True, "dispersion": False, "aovs": False},
        # the large benchmark configuration: 1.02 million triangles in full HD
        {"name": "field_1080p", "kind": "field", "spheres": 800, "width": 1920, "height": 1080, "spp": 16,
         "depth": 12, "mis": True, "lens": True, "dispersion": False, "aovs": False},
        # a ragged viewport refined by a few passes: pinhole camera, dispersive
        # glass, BSDF sampling only (the settings' use_mis off)
        {"name": "field_ragged", "kind": "field", "spheres": 200, "width": 333, "height": 257, "spp": 7, "depth": 9,
         "mis": False, "lens": False, "dispersion": True, "aovs": False},
        # an interior with albedo, roughness, metalness and normal maps, an
        # anisotropic panel and dispersive glass, with the denoiser's inputs
        {"name": "room_640x480", "kind": "room", "width": 640, "height": 480, "spp": 32, "depth": 8, "tex": 256,
         "mis": True, "aovs": True},
        # half glass, half glossy, sky and area lights together, depth 32: the
        # stress configuration at a fraction of its size
        {"name": "stress_960x540", "kind": "stress", "spheres": 400, "cuboids": 500, "tex": 512, "width": 960,
         "height": 540, "spp": 8, "depth": 32, "aovs": False},
        # a queue of jobs of uneven resolution, passes, depth and scene
        {"name": "batch_12_jobs", "kind": "batch", "jobs": 12, "mix": 3, "spp": 32},
        # caustics by the photon mapper: the first iterations of a frame
        {"name": "photon_room_640x480", "kind": "photon", "width": 640, "height": 480, "iterations": 4, "depth": 8,
         "tex": 256},
        # from a job file to the first images, as a viewer or a server starts
        {"name": "load_field", "kind": "load", "spheres": 200, "width": 640, "height": 480},
        # picking and visibility: closest hits of given rays, half from a
        # camera and half with scattered origins and directions
        {"name": "rays_1m", "kind": "rays", "spheres": 50, "rays": 1000000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _draw(rng)
        if work(c)["flops"] <= most:
            return c


def _draw(rng):
    kind = rng.choice(["cornell", "cornell", "field", "field", "room", "stress", "batch", "photon", "load", "rays"])
    w = _log(rng, 65, 1920)
    h = max(48, int(w * rng.uniform(0.5, 1.1)))
    frame = {"kind": kind, "width": w, "height": h, "spp": _log(rng, 1, 96)}
    aovs = rng.random() < 0.4
    if kind == "cornell":
        return dict(frame, depth=rng.randint(4, 16), mis=rng.random() < 0.8, aovs=aovs)
    if kind == "field":
        return dict(frame, spheres=_log(rng, 30, 800), depth=rng.randint(6, 16), mis=rng.random() < 0.8,
                    lens=rng.random() < 0.6, dispersion=rng.random() < 0.3, aovs=aovs)
    if kind == "room":
        return dict(frame, depth=rng.randint(4, 16), tex=_log(rng, 33, 700), mis=rng.random() < 0.8, aovs=aovs)
    if kind == "stress":
        return dict(frame, spheres=_log(rng, 40, 400), cuboids=_log(rng, 20, 500), tex=_log(rng, 65, 512),
                    depth=rng.randint(12, 32), aovs=aovs)
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 12), "mix": rng.randint(0, 1 << 20), "spp": _log(rng, 4, 32)}
    if kind == "photon":
        w = _log(rng, 97, 640)
        return {"kind": kind, "width": w, "height": max(64, int(w * rng.uniform(0.6, 1.0))),
                "iterations": rng.randint(1, 4), "depth": rng.randint(4, 12), "tex": _log(rng, 33, 512)}
    if kind == "load":
        return {"kind": kind, "spheres": _log(rng, 20, 400), "width": w // 4 + 16, "height": h // 4 + 16}
    return {"kind": kind, "spheres": _log(rng, 20, 200), "rays": _log(rng, 1000, 1500000)}


def _mix(case):
    """The jobs of a batch case: (kind, spheres, width, height, passes, depth)."""
    r = np.random.default_rng(case["mix"])
    jobs = []
    for _ in range(case["jobs"]):
        spheres = int(r.choice([0, 0, 50, 200]))
        w, h = RESOLUTIONS[int(r.integers(0, len(RESOLUTIONS)))]
        spp = max(1, int(round(case["spp"] * math.exp(r.uniform(-1.0, 1.0)))))
        jobs.append(("field" if spheres else "cornell", spheres, w, h, spp, int(r.integers(8, 17))))
    return jobs


# ----------------------------------------------------------------- inputs --
_sky = []


def _sky_path():
    """The sky picture of all field scenes (it has no seed), written once."""
    if not _sky:
        d = tempfile.TemporaryDirectory(prefix="perf_sky_")
        scenes.write_pfm(os.path.join(d.name, "sky.pfm"), scenes.sky_environment(2048, 1024))
        _sky.append(d)
    return os.path.join(_sky[0].name, "sky.pfm")


def _write(case, seed, folder):
    """The case's job file, its scene made from the seed."""
    kind = case["kind"]
    if kind == "cornell":
        return scenes.cornell_box(folder, seed=seed, width=case["width"], height=case["height"], spp=case["spp"],
                                  max_depth=case["depth"], use_mis=case["mis"])
    if kind in ("room", "photon"):
        return scenes.textured_room(folder, seed=seed, width=case["width"], height=case["height"], spp=64,
                                    max_depth=case["depth"], tex_size=case["tex"], use_mis=case.get("mis", True))
    if kind == "stress":
        return scenes.stress_scene(folder, seed=seed, n_spheres=case["spheres"], n_cuboids=case["cuboids"],
                                   tex_size=case["tex"], width=case["width"], height=case["height"],
                                   spp=case["spp"], max_depth=case["depth"], box=20.0)
    return scenes.sphere_field(folder, seed=seed, n_spheres=case["spheres"], width=case.get("width", 64),
                               height=case.get("height", 64), spp=case.get("spp", 16),
                               max_depth=case.get("depth", 12), aperture=0.15 if case.get("lens", True) else 0.0,
                               vary_glass_ior=case.get("dispersion", False), use_mis=case.get("mis", True),
                               sky_path=_sky_path())


def _rays(case, seed):
    """n x 6 rays through a sphere field (box 20): the first half from its
    camera, the rest from points in the box in uniform directions."""
    r = np.random.default_rng([seed, 77])
    n = case["rays"]
    k = n // 2
    target = np.stack([r.uniform(-10, 10, k), r.uniform(0, 20, k), r.uniform(-10, 10, k)], 1)
    eye = np.broadcast_to(np.array([0.0, 9.0, 27.0]), (k, 3))
    o = np.stack([r.uniform(-10, 10, n - k), r.uniform(0.5, 20, n - k), r.uniform(-10, 10, n - k)], 1)
    org = np.concatenate([eye, o])
    d = np.concatenate([target - eye, r.normal(size=(n - k, 3))])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([org, d], 1).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    folder = tempfile.TemporaryDirectory(prefix="perf_job_")
    if kind == "batch":
        paths, passes = [], []
        for k, (sub, spheres, w, h, spp, depth) in enumerate(_mix(case)):
            c = {"kind": sub, "spheres": spheres, "width": w, "height": h, "spp": spp, "depth": depth, "mis": True}
            paths.append(_write(c, 1000 * seed + k, os.path.join(folder.name, str(k))))
            passes.append(spp)
        return {"case": case, "jobs": load_jobs(paths), "passes": passes}
    path = _write(case, seed, folder.name)
    if kind == "load":
        return {"case": case, "path": path, "folder": folder}
    state = {"case": case, "job": RenderJob(path)}
    if kind == "rays":
        state["rays"] = _rays(case, seed)
    return state


# ------------------------------------------------------------------- run --
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        for j in state["jobs"]:
            j.reset()
        batch_render(state["jobs"], state["passes"])
        return [j.compute_estimate() for j in state["jobs"]]
    if kind == "load":
        with RenderJob(state["path"]) as job:
            job.render_passes(1)
            return [job.compute_estimate(a) for a in (AOV_COLOR, AOV_NORMAL, AOV_ALBEDO)]
    job = state["job"]
    if kind == "rays":
        return list(job.intersect(state["rays"]))
    if kind == "photon":
        job.pm_reset()
        job.pm_render(case["iterations"])
        return {"color": job.pm_read(), "radii": job.pm_radii()}
    job.reset()
    job.render_passes(case["spp"])
    if case["aovs"]:
        return [job.compute_estimate(a) for a in (AOV_COLOR, AOV_NORMAL, AOV_ALBEDO)]
    return job.compute_estimate()


# ------------------------------------------------------------------ work --
# Rays and shaded vertices of one camera sample, about as the scenes of each
# kind have them (the job statistics' counts; a closed room bounces longer
# than an open field); photon: of one pixel in one iteration, with its share
# of the photons.
_PER_SAMPLE = {"cornell": (7.0, 3.6), "room": (3.7, 1.6), "field": (2.5, 0.9), "load": (2.5, 0.9),
               "stress": (5.1, 3.6), "photon": (8.0, 3.5)}
_SKY_BYTES = 2048 * 1024 * 12
_SHADE_FLOPS = 400     # light sample, BSDF evaluation, pdf and sample of one vertex


def _triangles(case):
    kind = case["kind"]
    if kind == "cornell":
        return 36
    if kind in ("room", "photon"):
        return 330 + 80
    return 1280 * case["spheres"] + 12 * case.get("cuboids", 0) + 2


def _ray_flops(n_tris):
    """One descent of an 8-wide tree (48 plane tests, 2 flops each, a level)
    and two triangle tests: the least a closest-hit query computes."""
    return 96 * max(1, math.ceil(math.log(n_tris, 8))) + 2 * 45


def _scene_bytes(case):
    """Triangles (positions and shading indices), texels and sky, read once."""
    tex = case.get("tex", 0)
    sky = _SKY_BYTES if case["kind"] in ("field", "stress", "load") else 0
    return _triangles(case) * (36 + 48) + (32 * tex * tex if case["kind"] == "stress" else 8 * tex * tex) + sky


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for sub, spheres, w, h, spp, depth in _mix(case):
            parts.append(work({"kind": sub, "spheres": spheres, "width": w, "height": h, "spp": spp, "depth": depth,
                               "aovs": False}))
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    if kind == "rays":
        n = case["rays"]
        return {"bytes": n * (24 + 16) + _triangles(case) * 36, "flops": n * _ray_flops(_triangles(case))}
    npix = case["width"] * case["height"]
    samples = npix * {"photon": case.get("iterations"), "load": 1}.get(kind, case.get("spp"))
    rays, vertices = _PER_SAMPLE[kind]
    flops = samples * (rays * _ray_flops(_triangles(case)) + vertices * _SHADE_FLOPS)
    out = npix * 12 * (3 if case.get("aovs") or kind == "load" else 1) + (npix * 4 if kind == "photon" else 0)
    total = _scene_bytes(case) + out
    if kind == "load":      # the OBJ text (about 85 bytes a triangle) is read too
        total += 85 * _triangles(case)
    return {"bytes": total, "flops": flops}


# ----------------------------------------------------------------- exact --
def exact(case, seed):
    """Closest hits in 64 bits, by testing every triangle of each object whose
    bounding sphere a ray meets. The images are Monte Carlo estimates whose
    branches (which lobe, which light, absorbed or not) are decided on 32-bit
    numbers, so they have no 64-bit value to compare with: None."""
    if case["kind"] != "rays":
        return None
    with tempfile.TemporaryDirectory(prefix="perf_exact_") as folder:
        _write(case, seed, folder)
        verts, objects = [], []
        with open(os.path.join(folder, "scene.obj")) as f:
            for line in f:
                if line.startswith("v "):
                    verts.append(line.split()[1:4])
                elif line.startswith("o "):
                    objects.append([])
                elif line.startswith("f "):
                    objects[-1].append([int(p.split("/")[0]) - 1 for p in line.split()[1:4]])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.from_numpy(np.array(verts, dtype=np.float64).astype(np.float32).astype(np.float64)).to(dev)
    rays = torch.from_numpy(_rays(case, seed).astype(np.float64)).to(dev)
    o, d = rays[:, :3], rays[:, 3:]
    n = rays.shape[0]
    best = [torch.full((n,), math.inf, dtype=torch.float64, device=dev)] + [
        torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(2)]
    for faces in objects:
        tri = v[torch.tensor(faces, device=dev)]
        c = tri.reshape(-1, 3).mean(0)
        radius = (tri.reshape(-1, 3) - c).norm(dim=1).max() * 1.001
        near = (c - o) - d * (((c - o) * d).sum(1) / (d * d).sum(1))[:, None]
        for at in torch.nonzero(near.norm(dim=1) <= radius)[:, 0].split(max(1, (1 << 24) // len(faces))):
            _closest(o[at], d[at], tri, at, best)
    return [None] + [b.cpu().numpy() for b in best]


def _closest(o, d, tri, at, best):
    """Moeller-Trumbore of rays (o, d) and every triangle; ray at[i]'s closest
    hit is kept in best = (t, u, v), u and v the weights of vertices 2 and 3."""
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    p = torch.linalg.cross(d[:, None], e2[None])
    det = (p * e1).sum(-1)
    s = o[:, None] - tri[None, :, 0]
    u = (s * p).sum(-1) / det
    q = torch.linalg.cross(s, e1[None].expand_as(s))
    w = (d[:, None] * q).sum(-1) / det
    t = (e2 * q).sum(-1) / det
    ok = (det != 0) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-6)
    t = torch.where(ok, t, torch.full_like(t, math.inf))
    tm, k = t.min(1)
    rows = torch.arange(len(at), device=at.device)
    closer = tm < best[0][at]
    for b, val in zip(best, (tm, u[rows, k], w[rows, k])):
        b[at] = torch.where(closer, val, b[at])
