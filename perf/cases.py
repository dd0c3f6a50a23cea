"""The work a user of the engine has it do, as measured cases.

`listed()` names the cases, `draw()` gives more of the same ranges, `prepare()` builds what
a program holds before the call (resident scenes, films, guide images), `run()` is one pass
through the public entry points and `work()` what that pass cannot do without.  Every kind
of call is here once or twice: renders with the scene resident (the progressive viewer's and
the benchmark's call), renders through host buffers (`accumulate`, the reference's call),
batched stones, served requests, the Stokes film, metric sweeps and the display path.

A render adds onto its film, as a progressive render does, so a state can be run again.
One renderer serves the whole process and starts from the package's schedule table; a stone
the table does not hold is tuned while its state is prepared, as a program's first renders do.
"""
from __future__ import annotations

import ctypes as C
import math
import random
from pathlib import Path

import numpy as np
import torch

import gemray_studio_b200 as pkg
from gemray_studio_b200 import abi, denoise as D, metrics as M, scene as S, serve as V, workloads as W

TABLE = Path(pkg.__file__).resolve().parent / "tuning" / "b200_schedules.txt"
ENVS = {"uniform": abi.GR_ENV_UNIFORM, "studio": abi.GR_ENV_STUDIO, "latlong": abi.GR_ENV_LATLONG}
MAPS = {"latlong": (2048, 1024), "latlong_small": (1024, 512)}

_one: list = []


def _renderer():
    """The process's renderer, with the measured schedules of the known stones."""
    if not _one:
        r = pkg.GpuFrameRenderer()
        n = C.c_uint32()
        r.lib.gr_tuning_load(r.ctx, str(TABLE).encode(), C.byref(n))
        _one.append(r)
    return _one[0]


def _ok(r, status: int) -> None:
    if status != abi.GR_OK:
        raise RuntimeError((r.lib.gr_last_error_string() or b"").decode(errors="replace"))


# ---------------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------------
def _planes(stone: str, stone_seed: int) -> np.ndarray:
    if stone == "rb57":
        return S.round_brilliant_57()
    if stone == "srb":
        return S.standard_round_brilliant()
    if stone == "em49":
        return S.emerald_cut_49()
    return S.random_polyhedron(np.random.default_rng(stone_seed))


def _scene(case: dict, seed: int) -> S.Scene:
    """The case's stone (fixed) seen from a camera and in an environment made from the seed."""
    rng = np.random.default_rng(seed)
    planes = _planes(case["stone"], case.get("stone_seed", 0))
    ext, finishes = None, None
    if case["material"] == "dichroic emerald":
        mat, ext = W.birefringent_emerald_material()
    elif case["material"] == "crown glass":
        mat = W.material_tables()[0][1]
    else:
        mat = S.builtin_material(case["material"])
    if case.get("frosted"):  # a bruted girdle: the near-vertical planes
        finishes = (np.abs(planes[:, 1]) < 0.05).astype(np.uint32)
    if case.get("sigma_s"):
        mat.scattering_sigma_s, mat.scattering_g = float(case["sigma_s"]), 0.6
    env = case["env"]
    latlong = S.gaussian_blob_latlong(*MAPS[env], 12, seed=seed) if env in MAPS else None
    return S.Scene(width=case["width"], height=case["height"], planes=planes, material=mat,
                   cam=S.camera(float(rng.uniform(-math.pi, math.pi)), float(rng.uniform(0.2, 0.6)), 5.0, 18.0),
                   max_bounces=case["depth"], env_mode=ENVS[env.split("_")[0]], latlong=latlong, ext=ext,
                   finishes=finishes, light_yaw=float(rng.uniform(0.0, 1.5)), exposure=float(rng.uniform(0.8, 1.2)),
                   uniform_rgb=tuple(float(x) for x in rng.uniform(0.7, 1.0, 3)),
                   flags=abi.GR_FLAG_KAHAN_FILM if case.get("kahan") else 0)


class _Resident:
    """A scene kept on the device, released with the state that holds it."""

    def __init__(self, r, sc: S.Scene):
        self.r, self.width, self.height = r, sc.width, sc.height
        sid = C.c_uint64()
        _ok(r, r.lib.gr_scene_upload(r.ctx, C.byref(sc.c_scene()), C.byref(sid)))
        self.id = sid.value

    def __del__(self):
        self.r.lib.gr_synchronize(self.r.ctx)
        self.r.lib.gr_scene_release(self.r.ctx, self.id)


def _tuned(r, res: _Resident, spp: int, film: torch.Tensor) -> None:
    """Renders until the stone's schedule is chosen (at once for a known stone)."""
    c = [C.c_uint32() for _ in range(3)]
    for k in range(8):
        _ok(r, r.lib.gr_scene_schedule(r.ctx, res.id, *(C.byref(x) for x in c)))
        if c[0].value or res.width * res.height * spp < abi.GR_AUTO_STAGED_MIN_TUPLES:
            break
        _ok(r, r.lib.gr_render_resident(r.ctx, res.id, k * spp, spp, film.data_ptr(), None))
        _ok(r, r.lib.gr_synchronize(r.ctx))
    film.zero_()


def _offset(seed: int) -> int:
    """The first absolute sample of the pass: a progressive render is somewhere in its sequence."""
    return 16 * (seed % 61)


# ---------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # a thumbnail through host buffers, the smallest call: latency, copies and launches
        dict(name="thumbnail_24x16", kind="accumulate", stone="srb", material="Diamond", env="studio", width=24, height=16,
             spp=16, depth=12),
        # the CPU-runnable configuration through the reference's call, host buffers in and out
        dict(name="accumulate_256", kind="accumulate", stone="rb57", material="Diamond", env="uniform", width=256, height=256,
             spp=64, depth=32),
        # the headline frame, scene resident
        dict(name="brilliant_1080p", kind="resident", stone="rb57", material="Diamond", env="latlong", width=1920, height=1080,
             spp=256, depth=32),
        # the birefringent dichroic step cut, a tenth of its full sample count (one progressive pass)
        dict(name="emerald_1024", kind="resident", stone="em49", material="dichroic emerald", env="studio", width=1024,
             height=1024, spp=96, depth=64),
        # an odd-sized view of a tinted uniaxial stone with Kahan sums
        dict(name="tourmaline_317x211", kind="resident", stone="srb", material="Tourmaline", env="studio", width=317, height=211,
             spp=37, depth=24, kahan=True),
        # frosted girdle, volume scattering and a biaxial trichroic material together
        dict(name="frosted_tanzanite", kind="resident", stone="srb", material="Tanzanite", env="latlong_small", width=320,
             height=240, spp=48, depth=32, frosted=True, sigma_s=0.3),
        # many small random stones in one call, the catalogue's thumbnails
        dict(name="batch_64", kind="batch", stones=64, side_lo=16, side_hi=64, spp_lo=32, spp_hi=512, depth=32, stone_seed=0),
        # the Stokes film beside the XYZ film, host buffers
        dict(name="stokes_384x256", kind="stokes", stone="em49", material="dichroic emerald", env="studio", width=384,
             height=256, spp=64, depth=64),
        # the tilt sweep of brilliance, fire and scintillation
        dict(name="metrics_16", kind="metrics", stone="rb57", material="Diamond", poses=16),
        # a progressive viewer's display update: guide images, denoise and tone map, all on the device
        dict(name="display_1080p", kind="display", stone="rb57", material="Diamond", width=1920, height=1080, count=16,
             passes=5),
        # the filter alone on host images of an odd size
        dict(name="denoise_333x187", kind="denoise", stone="srb", width=333, height=187, count=9, passes=4),
        # a burst of requests to the serving loop, renders of several sizes and one metric sweep
        dict(name="serve_9", kind="serve", stones=8, side_lo=64, side_hi=256, spp_lo=16, spp_hi=96, depth=32, stone_seed=3),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["resident", "resident", "resident", "accumulate", "batch", "stokes", "metrics", "display", "denoise",
                       "serve"])
    stone = rng.choice(["rb57", "srb", "em49", "random", "random"])
    if kind in ("resident", "accumulate", "stokes"):
        c = dict(kind=kind, stone=stone, stone_seed=rng.randrange(1 << 16),
                 material=rng.choice(["Diamond", "Diamond", "Spinel", "Zircon", "Sapphire", "Quartz", "Tourmaline", "Topaz",
                                      "crown glass", "dichroic emerald"]),
                 env=rng.choice(["uniform", "studio", "latlong_small"]), width=_log_int(rng, 16, 1200),
                 height=_log_int(rng, 16, 900), spp=_log_int(rng, 4, 256), depth=rng.choice([8, 12, 24, 32, 64]),
                 kahan=rng.random() < 0.3)
        most = {"resident": 60_000_000, "accumulate": 20_000_000, "stokes": 8_000_000}[kind]
        c["spp"] = max(1, min(c["spp"], most // (c["width"] * c["height"])))
        if kind == "resident" and rng.random() < 0.2:
            c.update(frosted=True, sigma_s=round(rng.uniform(0.0, 0.5), 2))
        return c
    if kind in ("batch", "serve"):
        big = kind == "serve"
        return dict(kind=kind, stones=_log_int(rng, 2, 12 if big else 64), side_lo=16, side_hi=_log_int(rng, 24, 256 if big else 128),
                    spp_lo=16, spp_hi=_log_int(rng, 32, 128 if big else 256), depth=32, stone_seed=rng.randrange(1 << 16))
    if kind == "metrics":
        return dict(kind=kind, stone=stone, stone_seed=rng.randrange(1 << 16),
                    material=rng.choice(["Diamond", "Quartz", "Zircon", "Spinel"]), poses=_log_int(rng, 1, 64))
    if kind == "display":
        return dict(kind=kind, stone=stone, stone_seed=rng.randrange(1 << 16), material="Diamond", width=_log_int(rng, 160, 2048),
                    height=_log_int(rng, 120, 1200), count=_log_int(rng, 1, 256), passes=rng.choice([3, 4, 5, 5]))
    return dict(kind=kind, stone=stone, stone_seed=rng.randrange(1 << 16), width=_log_int(rng, 64, 700),
                height=_log_int(rng, 64, 500), count=_log_int(rng, 1, 128), passes=rng.choice([2, 4, 5]))


def _sizes(case: dict) -> list[tuple[int, int]]:
    """(side, spp) of each stone of a batched or served case."""
    rng = random.Random(case["stone_seed"])
    return [(_log_int(rng, case["side_lo"], case["side_hi"]), _log_int(rng, case["spp_lo"], case["spp_hi"]))
            for _ in range(case["stones"])]


def _stones(case: dict, seed: int) -> list[tuple[S.Scene, int]]:
    """Random stones, materials and cameras from the seed, one environment for all."""
    rng = np.random.default_rng(seed)
    mats = [m for _, m in W.material_tables()]
    env = S.gaussian_blob_latlong(512, 256, 12, seed=seed)
    out = []
    for i, (side, spp) in enumerate(_sizes(case)):
        planes = S.random_polyhedron(np.random.default_rng(case["stone_seed"] + i))
        cam = S.camera(float(rng.uniform(-math.pi, math.pi)), float(rng.uniform(0.15, 0.9)), 4.0, 30.0)
        out.append((S.Scene(width=side, height=side, planes=planes, material=mats[i % len(mats)], cam=cam,
                            max_bounces=case["depth"], env_mode=abi.GR_ENV_LATLONG, latlong=env,
                            flags=abi.GR_FLAG_KAHAN_FILM), spp))
    return out


def _tilts(n: int, seed: int) -> np.ndarray:
    """A tilt sweep in +-20 degrees around the viewing pitch, the light where the seed puts it."""
    rng = np.random.default_rng(seed)
    p = W.c2_tilt_poses(n)
    p[:, 0] = rng.uniform(0.0, 2.0 * math.pi)
    p[:, 2] = rng.uniform(0.5, 1.2)
    return p


def _noisy(guides: D.GuideBuffers, seed: int) -> np.ndarray:
    """A low-sample film over the guide images' facets: a level for each facet, and speckle."""
    rng = np.random.default_rng(seed)
    level = rng.uniform(0.02, 1.5, (600, 3))
    base = level[guides.facet_id.astype(np.int64) + 1]
    return (base * rng.gamma(2.0, 0.5, base.shape)).astype(np.float32)


# ---------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    r = _renderer()
    kind = case["kind"]
    st = dict(case=case, r=r, offset=_offset(seed))
    if kind in ("accumulate", "resident", "stokes"):
        sc = _scene(case, seed)
        n = sc.width * sc.height
        st.update(scene=sc)
        if kind == "resident":
            st.update(res=_Resident(r, sc), film=torch.zeros((n, 3), dtype=torch.float32, device="cuda"))
            torch.cuda.synchronize()
            _tuned(r, st["res"], case["spp"], st["film"])
        else:
            st.update(accum=np.zeros((n, 3), np.float32), stokes=np.zeros((n, 4), np.float32))
    elif kind == "batch":
        made = _stones(case, seed)
        res = [_Resident(r, sc) for sc, _ in made]
        films = [torch.zeros((sc.width * sc.height, 3), dtype=torch.float32, device="cuda") for sc, _ in made]
        items = (abi.gr_batch_item * len(made))()
        for i, (sc, spp) in enumerate(made):
            items[i].scene_id, items[i].film_device = res[i].id, films[i].data_ptr()
            items[i].sample_offset, items[i].spp = st["offset"], spp
        st.update(res=res, films=films, items=items)
    elif kind == "serve":
        made = _stones(case, seed)
        srv = V.RenderServer(r)
        st.update(srv=srv, scenes=[sc for sc, _ in made], spps=[spp for _, spp in made], poses=_tilts(64, seed),
                  ids=_Served(srv, [srv.upload(sc) for sc, _ in made]))
    elif kind == "metrics":
        st.update(planes=_planes(case["stone"], case.get("stone_seed", 0)), material=S.builtin_material(case["material"]),
                  poses=_tilts(case["poses"], seed))
    else:
        guide_case = dict(case, material="Diamond", env="uniform", depth=8)
        sc = _scene(guide_case, seed)
        guides = D.generate_guide_buffers(r, sc)
        film = _noisy(guides, seed)
        n = sc.width * sc.height
        st.update(scene=sc, params=D.AtrousParams(num_passes=case["passes"]))
        if kind == "display":
            dev = dict(dtype=torch.float32, device="cuda")
            st.update(film=torch.from_numpy(film * np.float32(case["count"])).cuda(), depth=torch.empty(n, **dev),
                      normal=torch.empty((n, 3), **dev), facet=torch.empty(n, dtype=torch.int32, device="cuda"),
                      rgba=torch.empty((n, 4), dtype=torch.uint8, device="cuda"))
        else:
            st.update(guides=guides, color=film)
    return st


class _Served:
    """The scenes of a served case, released with its state."""

    def __init__(self, srv, ids):
        self.srv, self.ids = srv, ids

    def __del__(self):
        for i in self.ids:
            self.srv.release_scene(i)


def run(st: dict):
    case, r = st["case"], st["r"]
    kind = case["kind"]
    if kind == "resident":
        _ok(r, r.lib.gr_render_resident(r.ctx, st["res"].id, st["offset"], case["spp"], st["film"].data_ptr(), None))
        return st["film"]
    if kind == "accumulate":
        r.accumulate(st["scene"], st["offset"], case["spp"], st["accum"])
        return st["accum"]
    if kind == "stokes":
        fp = C.POINTER(C.c_float)
        _ok(r, r.lib.gr_accumulate_stokes(r.ctx, C.byref(st["scene"].c_scene()), st["offset"], case["spp"],
                                          st["accum"].ctypes.data_as(fp), st["stokes"].ctypes.data_as(fp)))
        return {"xyz": st["accum"], "stokes": st["stokes"]}
    if kind == "batch":
        _ok(r, r.lib.gr_render_batch(r.ctx, st["items"], len(st["items"]), abi.GR_BATCH_GRAPH, None))
        return st["films"]
    if kind == "serve":
        srv = st["srv"]
        ids = [srv.submit_render(s, st["offset"], spp) for s, spp in zip(st["ids"].ids, st["spps"])]
        sweep = srv.submit_metrics(st["scenes"][0].planes, st["scenes"][0].material, st["poses"])
        films = []
        for q in ids:
            srv.wait(q)
            films.append(srv.film(q))
            srv.release(q)
        srv.wait(sweep)
        table = srv.metrics(sweep)
        srv.release(sweep)
        return {"films": films, "metrics": table}
    if kind == "metrics":
        return M.evaluate_poses(r, st["planes"], st["material"], st["poses"])
    sc = st["scene"]
    if kind == "display":
        _ok(r, r.lib.gr_guide_buffers_device(r.ctx, C.byref(sc.c_scene()), st["depth"].data_ptr(), st["normal"].data_ptr(),
                                             st["facet"].data_ptr(), None))
        p = st["params"].c()
        _ok(r, r.lib.gr_denoise_tonemap_device(r.ctx, st["film"].data_ptr(), case["count"], st["depth"].data_ptr(),
                                               st["normal"].data_ptr(), st["facet"].data_ptr(), sc.width, sc.height,
                                               C.byref(p), st["rgba"].data_ptr(), None))
        return {"rgba": st["rgba"], "depth": st["depth"], "normal": st["normal"], "facet": st["facet"]}
    return D.denoise(r, st["color"], st["guides"], sc.width, sc.height, case["count"], st["params"])


# ---------------------------------------------------------------------------------
# work / exact
# ---------------------------------------------------------------------------------
# Arithmetic of one path-sample (the engine's FLOP model over the event counts of the
# benchmark scenes, rounded): a clear isotropic stone, and one with absorption or
# birefringence; a miss costs the sampler, the camera ray and the film integral.
FLOPS_CLEAR, FLOPS_GENERAL = 6.9e3, 1.1e4


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("resident", "accumulate", "stokes"):
        n = case["width"] * case["height"]
        w, h = MAPS.get(case["env"], (0, 0))
        per = FLOPS_CLEAR if case["material"] in ("Diamond", "Spinel") and not case.get("frosted") else FLOPS_GENERAL
        return {"bytes": float(n * (24 + (32 if kind == "stokes" else 0)) + 12 * w * h), "flops": float(n) * case["spp"] * per}
    if kind in ("batch", "serve"):
        t = sum(s * s * p for s, p in _sizes(case))
        n = sum(s * s for s, _ in _sizes(case))
        return {"bytes": float(24 * n + 12 * 512 * 256), "flops": t * 9e3 + (64 * 1780 * 4000.0 if kind == "serve" else 0.0)}
    if kind == "metrics":
        return {"bytes": 4096.0 + 36.0 * case["poses"], "flops": case["poses"] * 1780 * 4000.0}
    n = case["width"] * case["height"]
    if kind == "display":  # guides out, film in, bytes out; a ray against ~70 planes, 25 taps a pass
        return {"bytes": float(n * (20 + 12 + 4)), "flops": float(n) * (70 * 12 + case["passes"] * 25 * 25)}
    return {"bytes": float(n * (12 + 12 + 20)), "flops": float(n) * case["passes"] * 25 * 25}


def exact(case: dict, seed: int):
    """The filtered image in 64 bits.  A render has no such value: its paths are decided by
    draws in 32 bits, and a 64-bit path leaves them at the first threshold; the metrics count
    rays that are decided likewise, and the display path's bytes and facets are whole."""
    if case["kind"] != "denoise":
        return None
    st = prepare(case, seed)
    w, h, p, g = case["width"], case["height"], st["params"], st["guides"]
    t = lambda a: torch.from_numpy(np.asarray(a)).to("cuda", torch.float64)  # noqa: E731
    color, depth = t(st["color"]).reshape(h, w, 3), t(g.depth).reshape(h, w)
    normal, facet = t(g.normal).reshape(h, w, 3), torch.from_numpy(g.facet_id).cuda().reshape(h, w)
    length = normal.norm(dim=2, keepdim=True)
    normal = torch.where(length <= 1e-8, torch.zeros_like(normal), normal / length.clamp_min(1e-30))
    flat = (normal == 0).all(dim=2)
    taper = 1.0 / math.sqrt(1.0 + case["count"] / max(p.taper_reference_spp, 1e-8))
    if taper < p.taper_identity_epsilon:
        return color.reshape(-1, 3).cpu().numpy()
    nisd, nits = -1.0 / max(p.sigma_depth, 1e-8), -1.0 / (2.0 * max((p.sigma_color * taper) ** 2, 1e-8))
    b3 = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    for k in range(p.num_passes):
        total, weight = torch.zeros_like(color), torch.zeros_like(depth)
        for ky in range(5):
            for kx in range(5):
                dy, dx = (ky - 2) << k, (kx - 2) << k
                y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
                if y0 >= y1 or x0 >= x1:
                    continue
                a, b = (slice(y0, y1), slice(x0, x1)), (slice(y0 + dy, y1 + dy), slice(x0 + dx, x1 + dx))
                cosine = (normal[a] * normal[b]).sum(dim=2).clamp(0.0, 1.0) ** p.normal_power
                wn = torch.where(flat[a] | flat[b], torch.ones_like(cosine), cosine)
                diff = color[a] - color[b]
                wt = b3[ky] * b3[kx] * wn * torch.exp((depth[a] - depth[b]).abs() * nisd + (diff * diff).sum(dim=2) * nits)
                wt = torch.where(facet[a] == facet[b], wt, torch.zeros_like(wt))
                total[a] += color[b] * wt[..., None]
                weight[a] += wt
        color = torch.where((weight > 1e-8)[..., None], total / weight.clamp_min(1e-30)[..., None], color)
    return color.reshape(-1, 3).cpu().numpy()
