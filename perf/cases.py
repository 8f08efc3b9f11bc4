"""Performance cases: the renders a user has this library do, through its public
entry points, from a viewer's preview frame to a 2^26-photon rainbow.

``listed()`` gives the named cases and ``draw(rng)`` further ones of the same
ranges.  ``prepare(case, seed)`` builds what a program holds before the call
(scene, film, tracer, batch or server), ``run(state)`` makes one pass and
returns its outputs, ``work(case)`` says what the pass cannot do without and
``exact(case, seed)`` computes the same images in 64 bits with torch alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import spectral_b200 as sb
from spectral_b200 import scenes, specs
from spectral_b200._lib import check, lib, sc_film_options, sc_trace_desc, sc_vol_weights
from spectral_b200.batch import Batch, job_from_spec, prism_jobs
from spectral_b200.serve import ORBIT_TARGET, Server

_CTX = []


def _ctx():
    """The program's one context."""
    if not _CTX:
        _CTX.append(sb.GpuContext(0))
    return _CTX[0]


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    prism = dict(scene="prism", sigma_s=0.05, sigma_t=0.05, g=0.0, max_dist=6.0, bounces=8, lo=380.0, hi=780.0)
    rainbow = dict(scene="rainbow", sigma_s=0.02, sigma_t=0.02, g=0.0, max_dist=8.0, bounces=6, lo=380.0, hi=780.0)
    dsotm = dict(scene="dsotm", sigma_s=0.5, sigma_t=0.06, g=0.5, max_dist=14.0, bounces=8, lo=380.0, hi=730.0)
    return [
        # one frame of the interactive viewer at its smallest: camera moved, film cleared, 2^16 photons, RGBA8 back
        dict(name="viewer_256", kind="viewer", w=256, h=256, photons=1 << 16, kradius=2.0, **dsotm),
        # the drop-in render of the reference's GPU path: one full dispatch into an XYZ film, exposed and read back
        dict(name="dsotm_800_4m", kind="object", w=800, h=800, bins=0, photons=4_000_000, estimator=0, exact=False,
             **dsotm),
        # the same with the haze samples in the reference's operation order, as a parity check renders it
        dict(name="haze_exact_400x300", kind="object", w=400, h=300, bins=0, photons=1 << 18, estimator=0, exact=True,
             **dsotm),
        # the single-prism benchmark scene: a 64-bin film on the device, traced and drained to XYZ
        dict(name="prism_640x360x64", kind="device", w=640, h=360, bins=64, photons=1 << 20, estimator=0, **prism),
        # ragged film, odd bin count, anisotropic haze, free-flight distances
        dict(name="freeflight_ragged", kind="device", w=1001, h=563, bins=31, photons=300_001, estimator=3,
             **dict(prism, g=0.3, sigma_s=0.4, sigma_t=0.5)),
        # the largest single launch: the rainbow benchmark scene, a 1.06 GB spectral film
        dict(name="rainbow_1080p_64m", kind="device", w=1920, h=1080, bins=64, photons=1 << 26, estimator=0,
             **rainbow),
        # the uneven batch of 256 scenes with the plan its autotuner keeps, images left on the device
        dict(name="batch_256", kind="batch", jobs=256, bins=32, tuned=True, photons_log2=22, side=1024),
        # a burst of render requests through the continuous-batching server
        dict(name="serve_burst", kind="serve", requests=40, photons_log2=20, side=1024),
        # the camera tracer's benchmark scene: prism on a diffuse floor, small emitter, black sky
        dict(name="tracer_720p_64spp", kind="tracer", scene="floor", w=1280, h=720, spp=64, background=0.0,
             illuminant=0),
        # an interactive preview of glass under a bright sky: few samples, odd size
        dict(name="tracer_sky_333x187", kind="tracer", scene="glass", w=333, h=187, spp=4, background=1.0,
             illuminant=1),
        # the photon-beam estimator on the DSOTM composition
        dict(name="beam_800", kind="device", w=800, h=800, bins=0, photons=1 << 18, estimator=2, **dsotm),
        # the prism-on-plane program from start to end: floor caustic, z-buffer, haze film behind it
        dict(name="prism_on_plane_800x600", kind="plane", w=800, h=600, texels=512, photons=1 << 18),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "device", "object", "viewer", "batch", "serve", "tracer", "tracer", "beam", "plane"])
    w = _log_int(rng, 64, 1600)
    h = max(33, int(w * rng.uniform(0.5, 1.0)))
    name = rng.choice(["prism", "dsotm", "rainbow"])
    haze = dict(scene=name, sigma_s=round(rng.uniform(0.01, 0.5), 4), sigma_t=round(rng.uniform(0.01, 0.5), 4),
                g=rng.choice([0.0, 0.3, 0.5, -0.2]), max_dist={"prism": 6.0, "dsotm": 14.0, "rainbow": 8.0}[name],
                bounces=rng.choice([4, 6, 8]), lo=380.0, hi=rng.choice([730.0, 780.0]))
    if kind == "device":
        return dict(kind=kind, w=w, h=h, bins=rng.choice([0, 1, 8, 16, 31, 32, 40, 64, 81]),
                    photons=_log_int(rng, 1 << 14, 1 << 24), estimator=rng.choice([0, 0, 0, 1, 3]), **haze)
    if kind == "object":
        return dict(kind=kind, w=w, h=h, bins=rng.choice([0, 0, 16, 33]), photons=_log_int(rng, 1 << 14, 1 << 22),
                    estimator=rng.choice([0, 0, 1, 3]), exact=rng.random() < 0.25, **haze)
    if kind == "viewer":
        w = _log_int(rng, 128, 1024)
        return dict(kind=kind, w=w, h=int(w * rng.uniform(0.5, 1.0)), photons=_log_int(rng, 1 << 14, 1 << 20),
                    kradius=float(rng.choice([1, 2, 3])), **haze)
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(4, 64), bins=rng.choice([16, 31, 32, 64]), tuned=rng.random() < 0.5,
                    photons_log2=rng.randint(18, 22), side=rng.choice([256, 500, 1024]))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(6, 40), photons_log2=rng.randint(17, 20),
                    side=rng.choice([256, 500, 1024]))
    if kind == "tracer":
        return dict(kind=kind, scene=rng.choice(["floor", "glass"]), w=w, h=h, spp=rng.choice([1, 3, 8, 16, 33]),
                    background=rng.choice([0.0, 0.2, 1.0]), illuminant=rng.randint(0, 1))
    if kind == "beam":
        return dict(kind="device", w=w, h=h, bins=rng.choice([0, 0, 16]), photons=_log_int(rng, 1 << 10, 1 << 16),
                    estimator=2, **haze)
    return dict(kind="plane", w=w, h=h, texels=_log_int(rng, 100, 1024), photons=_log_int(rng, 1 << 14, 1 << 20))


# ---------------------------------------------------------------------------
# scenes: plain numbers drawn from the seed
# ---------------------------------------------------------------------------
def _scene_spec(name, seed):
    g = specs.Pcg(7, seed)
    if name == "prism":
        return specs.prism_scene(60.0, 1.0, g.uniform(40.0, 50.0), 0.02, 1.0, specs.SF11)
    if name == "rainbow":
        return specs.rainbow_scene(g.uniform(2.1, 2.3))
    d = specs.dsotm_scene()
    o, t, up, vfov = d["camera"]
    d["camera"] = ((o[0] + g.uniform(-0.2, 0.2), o[1], o[2]), t, up, vfov)
    return d


def _photon_seed(seed):
    return (int(seed) * 2654435761 + 0xDED) & 0xFFFFFFFF


def _tracer_spec(case, seed):
    g = specs.Pcg(9, seed)
    if case["scene"] == "floor":
        return specs.tracer_scene()
    box = [((1, 0, 0), 1.5), ((-1, 0, 0), -3.0), ((0, 1, 0), -2.0), ((0, -1, 0), -2.0), ((0, 0, 1), 4.0),
           ((0, 0, -1), -6.0)]
    return dict(solids=[(box, ("glass", specs.BK7))],
                spheres=[((g.uniform(-0.2, 0.2), 0.0, -3.0), 1.0, ("glass", specs.SF11)),
                         ((1.8, 0.5, -4.0), 0.7, ("lambertian", 0.7))],
                camera=((0.0, 0.3, 0.5), (0.0, 0.0, -3.0), (0.0, 1.0, 0.0), 55.0), horizon=2.0, tracer=dict(max_depth=8))


def _vary(spec, index, seed):
    """The same film and photon budget with another prism, light and seed."""
    g = specs.Pcg(index, seed)
    return dict(spec, apex_deg=g.uniform(30.0, 75.0), incidence_deg=g.uniform(30.0, 60.0), seed=g.u32())


def _requests(case, seed):
    """Requests of the serving distribution: (job spec, frames, orbit step);
    every other session keeps its camera and accumulates a few frames."""
    stream = specs.poisson_request_specs(200.0, 2.0, photons=(2 ** 16, 2 ** case["photons_log2"]),
                                         side=(128, case["side"]))[:case["requests"]]
    out, sessions = [], 0
    for i, (_, spec, frames, orbit) in enumerate(stream):
        if frames > 1:
            sessions += 1
            if sessions % 2 == 0:
                frames, orbit = 4 + frames % 13, 0.0
        out.append((_vary(spec, i, seed), frames, orbit))
    return out


def _batch_specs(case, seed):
    jobs = specs.random_prism_jobs(case["jobs"], bins=case["bins"], photons=(2 ** 14, 2 ** case["photons_log2"]),
                                   side=(128, case["side"]))
    return [_vary(j, i, seed) for i, j in enumerate(jobs)]


def _look_at(camera, aspect):
    return sb.Camera.look_at(*camera, aspect)


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
class _DeviceFilm:
    """A film in torch tensors traced and drained through the device-pointer
    entry points, on torch's current stream."""

    def __init__(self, case, seed):
        d = _scene_spec(case["scene"], seed)
        w, h, bins = case["w"], case["h"], case["bins"]
        prims, n_prims, planes, n_planes, mats, n_mats = scenes.scene_from_spec(d).arrays()
        self.keep = [torch.frombuffer(bytearray(bytes(a)), dtype=torch.uint8).cuda() for a in (prims, planes, mats)]
        dp, dl, dm = (t.data_ptr() for t in self.keep)
        self.channels, self.scale = bins or 3, 40 if case["estimator"] == 2 else 32
        opts = sc_film_options(bins, case["lo"], case["hi"], case["bounces"], self.scale, case["estimator"], 0)
        self.desc = sc_trace_desc(dp, n_prims, dl, n_planes, dm, n_mats, _look_at(d["camera"], w / h).c,
                                  sb.Beam(*d["beam"]).c, sc_vol_weights(case["sigma_s"], case["sigma_t"], case["g"]),
                                  w, h, _photon_seed(seed), 1, case["max_dist"], opts, None)
        self.film = torch.zeros(lib.sc_film_bytes(w, h, self.channels) // 8, dtype=torch.int64, device="cuda")
        self.flags = torch.zeros(lib.sc_film_flag_bytes(w, h) // 4, dtype=torch.int32, device="cuda")
        self.xyz = torch.empty(3 * w * h, dtype=torch.float32, device="cuda")
        self.case = case


def _object_film(case, seed, zbuffer=None):
    d = _scene_spec(case["scene"], seed)
    scene, cam, beam = scenes.scene_from_spec(d), _look_at(d["camera"], case["w"] / case["h"]), sb.Beam(*d["beam"])
    return sb.GpuPhotonFilm(_ctx(), scene, cam, beam, case["w"], case["h"], case["photons"], _photon_seed(seed),
                            case["max_dist"], sb.VolWeights(case["sigma_s"], case["sigma_t"], case["g"]),
                            bins=case.get("bins", 0), lambda_min=case["lo"], lambda_max=case["hi"],
                            max_bounces=case["bounces"], estimator=case.get("estimator", 0),
                            haze_exact=case.get("exact", False)), cam


class _DeviceArray:
    """A float32 array in device memory of `owner`, which lives as long as it."""

    def __init__(self, owner, address, floats):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(floats,), typestr="<f4", data=(address, False), version=3)


def _device_images(batch):
    """The batch's XYZ images on the device, in job order, as one tensor (they
    lie one behind the other, which is checked here)."""
    at, floats, first = C.POINTER(C.c_float)(), 0, None
    for i, job in enumerate(batch.jobs):
        check(lib.sc_batch_device_xyz(batch.h, i, C.byref(at)))
        address = C.cast(at, C.c_void_p).value
        first = address if first is None else first
        if address != first + 4 * floats:
            raise RuntimeError("image %d is not behind image %d" % (i, i - 1))
        floats += 3 * job.width * job.height
    return torch.as_tensor(_DeviceArray(batch, first, floats), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case, seed=seed, photon_seed=_photon_seed(seed))
    if kind == "device":
        _ctx()
        state["film"] = _DeviceFilm(case, seed)
    elif kind in ("object", "viewer"):
        state["film"], state["cam"] = _object_film(case, seed)
    elif kind == "batch":
        tuning = dict(chunk_photons=8192, minb=4, per_photon=1, block=128) if case["tuned"] else {}
        state["batch"] = Batch(_ctx(), prism_jobs(_batch_specs(case, seed)), **tuning)
        state["images"] = _device_images(state["batch"])
    elif kind == "serve":
        state["server"] = Server(_ctx(), budget_bytes=8 << 30)
        state["requests"] = [(job_from_spec(s), frames, orbit) for s, frames, orbit in _requests(case, seed)]
    elif kind == "tracer":
        d = _tracer_spec(case, seed)
        scene = scenes.scene_from_spec(d)
        scene.background, scene.horizon = case["background"], d.get("horizon")
        state["tracer"] = sb.GpuTracer(_ctx(), scene, _look_at(d["camera"], case["w"] / case["h"]), case["w"], case["h"],
                                       case["illuminant"], state["photon_seed"], **d["tracer"])
    else:
        state["plane"] = scenes.prism_on_plane(case["w"], case["h"], case["texels"])
        _ctx()
    return state


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def _run_device(state):
    f = state["film"]
    c, stream = f.case, C.c_void_p(torch.cuda.current_stream().cuda_stream)
    film, flags, xyz = (C.c_void_p(t.data_ptr()) for t in (f.film, f.flags, f.xyz))
    check(lib.sc_trace_photons_device(_ctx().h, C.byref(f.desc), 0, c["photons"], film, flags, stream))
    check(lib.sc_sensor_reduce_device(_ctx().h, c["w"], c["h"], f.channels, c["lo"], c["hi"], f.scale, film, flags, xyz,
                                      1, stream))
    return f.xyz


def _run_object(state):
    film, c = state["film"], state["case"]
    film.clear_film()
    film.trace_and_resolve(c["photons"], state["photon_seed"])
    exposure = film.auto_expose_p997()
    return [film.accum(), exposure, film.to_rgb8(exposure)]


def _run_viewer(state):
    film, c = state["film"], state["case"]
    film.set_camera(state["cam"])
    film.clear_film()
    film.dispatch_photons(0, c["photons"], state["photon_seed"])
    return film.gather_rgba8(c["photons"], kradius=c["kradius"], exposure=20.0)


def _run_batch(state):
    state["batch"].run()
    return state["images"]


def _run_serve(state):
    server, got = state["server"], {}
    ids = [server.submit(job, frames, orbit) for job, frames, orbit in state["requests"]]
    while len(got) < len(ids):
        server.step()
        while (done := server.poll()) is not None:
            got[done[0]] = done[1]
    return [got[i] for i in ids]


def _run_tracer(state):
    t = state["tracer"]
    t.clear_accum()
    t.accumulate(state["case"]["spp"])
    return t.read_xyz()


def _run_plane(state):
    c, seed = state["case"], state["photon_seed"]
    scene, floor, beam, cam = state["plane"]
    caustic = sb.trace(_ctx(), scene, sb.Screen(floor.corner, floor.u, floor.v, floor.width, floor.height), beam,
                       c["photons"], seed)
    zbuf = sb.scene_zbuffer(_ctx(), scene, cam, c["w"], c["h"], floor)
    film = sb.GpuPhotonFilm(_ctx(), scene, cam, beam, c["w"], c["h"], c["photons"], seed, 22.0,
                            sb.VolWeights(0.5, 0.06, 0.5), zbuffer=zbuf)
    film.trace_and_resolve(c["photons"], seed)
    haze = film.accum()
    film.close()
    return [caustic.sum, zbuf, haze]


_RUN = dict(device=_run_device, object=_run_object, viewer=_run_viewer, batch=_run_batch, serve=_run_serve,
            tracer=_run_tracer, plane=_run_plane)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Path segments per photon of the scenes, and FP32 operations per emission,
# plane test, sphere test, haze sample, scatter, beam step with its footprint.
_SEGMENTS = dict(prism=3.2, dsotm=2.3, rainbow=2.6, plane=3.0)
_EMIT, _PLANE, _SPHERE, _SAMPLE, _SCATTER, _BEAM_STEP = 20, 14, 25, 60, 45, 300


def _photon_flops(name, photons, estimator=0):
    s = _SEGMENTS[name]
    hit = _SPHERE if name == "rainbow" else 5 * _PLANE
    haze = 350 * _BEAM_STEP if estimator == 2 else 4 * _SAMPLE
    return photons * (_EMIT + s * (hit + haze) + (s - 1.0) * _SCATTER)


def work(case):
    """Bytes: the images that go out.  Flops: the FP32 operations of the
    photons' or paths' arithmetic at the scenes' usual path lengths."""
    kind = case["kind"]
    if kind in ("device", "object", "viewer"):
        out = {"device": 12, "object": 15, "viewer": 4}[kind]
        return dict(bytes=out * case["w"] * case["h"],
                    flops=_photon_flops(case["scene"], case["photons"], case.get("estimator", 0)))
    if kind == "batch":
        jobs = _batch_specs(case, 1)
        return dict(bytes=sum(12 * j["width"] * j["height"] for j in jobs),
                    flops=sum(_photon_flops("prism", j["n_photons"]) for j in jobs))
    if kind == "serve":
        jobs = _requests(case, 1)
        return dict(bytes=sum(12 * j["width"] * j["height"] for j, _, _ in jobs),
                    flops=sum(_photon_flops("prism", j["n_photons"] * f) for j, f, _ in jobs))
    if kind == "tracer":
        paths = case["w"] * case["h"] * case["spp"]
        return dict(bytes=12 * case["w"] * case["h"], flops=paths * (60 + 2 * 6 * _PLANE + _SCATTER + 100))
    return dict(bytes=12 * case["texels"] ** 2 + 16 * case["w"] * case["h"],
                flops=2 * _photon_flops("plane", case["photons"]))


# ---------------------------------------------------------------------------
# exact: the same estimators in 64 bits, torch only
# ---------------------------------------------------------------------------
_M32 = 0xFFFFFFFF
_INF = float("inf")


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pcg(x):
    s = (x * 747796405 + 2891336453) & _M32
    w = (((s >> ((s >> 28) + 4)) ^ s) * 277803737) & _M32
    return (w >> 22) ^ w


def _f32(v):
    return float(np.float32(v))


def _vec(v):
    return torch.tensor([_f32(x) for x in v], dtype=torch.float64, device=_dev())


def _dot(a, b):
    return (a * b).sum(-1)


def _norm(v):
    return v / _dot(v, v).sqrt().unsqueeze(-1)


class _Rng:
    """One stream per row: state + 1 hashed per draw, 24 bits per number."""

    def __init__(self, key, seed):
        self.state = _pcg(key ^ _pcg(torch.tensor(seed, device=_dev())))

    def pick(self, keep):
        r = _Rng.__new__(_Rng)
        r.state = self.state[keep]
        return r

    def next(self, rows=None):
        if rows is None:
            self.state = (self.state + 1) & _M32
            return (_pcg(self.state) >> 8).double() / 16777216.0
        self.state = torch.where(rows, (self.state + 1) & _M32, self.state)
        return (_pcg(self.state) >> 8).double() / 16777216.0


def _glass_n(glass, nm):
    l2 = (nm / 1000.0) ** 2
    if glass == specs.WATER:
        return 1.3238 + 0.00314 / l2
    b, c = {specs.BK7: ((1.03961212, 0.231792344, 1.01046945), (0.00600069867, 0.0200179144, 103.560653)),
            specs.SF11: ((1.73759695, 0.313747346, 1.89878101), (0.013188707, 0.0623068142, 155.23629)),
            specs.FUSED_SILICA: ((0.6961663, 0.4079426, 0.8974794), (0.0684043 ** 2, 0.1162414 ** 2, 9.896161 ** 2))
            }[glass]
    return (1.0 + sum(bi * l2 / (l2 - ci) for bi, ci in zip(b, c))).sqrt()


def _tables():
    return torch.tensor(sb.sample_tables().reshape(5, 71), dtype=torch.float64, device=_dev())


def _lerp(table, nm):
    """Columns of `table` (k x 71) at the wavelengths nm: (..., k)."""
    f = ((nm - 380.0) / 5.0).clamp(0.0, 70.0)
    i = f.floor().clamp(max=69.0)
    a, b = table.T[i.long()], table.T[i.long() + 1]
    return a + (b - a) * (f - i).unsqueeze(-1)


class _Geometry:
    """Solids, then spheres, then an optional emitter sphere, in scene order."""

    def __init__(self, d):
        self.solids = [([(_vec(n), _f32(off)) for n, off in planes], m) for planes, m in d["solids"]]
        self.spheres = [(_vec(c), _f32(r), m) for c, r, m in d["spheres"]]
        self.mats = [m for _, m in self.solids] + [m for _, _, m in self.spheres]

    @staticmethod
    def sphere(c, r, o, d, far):
        oc = o - c
        a, hb = _dot(d, d), _dot(oc, d)
        disc = hb * hb - a * (_dot(oc, oc) - r * r)
        sq = disc.clamp(min=0.0).sqrt()
        near, back = (-hb - sq) / a, (-hb + sq) / a
        t = torch.where((near >= 1e-3) & (near <= far), near, back)
        return t, (disc >= 0) & (t >= 1e-3) & (t <= far)

    def hit(self, o, d):
        """(any, t, unit normal against the ray, front face, material row)."""
        n = o.shape[0]
        best = torch.full((n,), _INF, dtype=torch.float64, device=o.device)
        normal, mat = torch.zeros_like(o), torch.full((n,), -1, dtype=torch.int64, device=o.device)
        for k, (planes, _) in enumerate(self.solids):
            t_in, t_out = torch.full_like(best, -_INF), torch.full_like(best, _INF)
            n_in, n_out, out = torch.zeros_like(o), torch.zeros_like(o), torch.zeros_like(best, dtype=torch.bool)
            for pn, off in planes:
                den, dist = d @ pn, o @ pn + off
                flat = den.abs() < 1e-8
                out |= flat & (dist > 0)
                t = -dist / torch.where(flat, torch.ones_like(den), den)
                enter, leave = ~flat & (den < 0) & (t > t_in), ~flat & (den >= 0) & (t < t_out)
                t_in, t_out = torch.where(enter, t, t_in), torch.where(leave, t, t_out)
                n_in, n_out = torch.where(enter[:, None], pn, n_in), torch.where(leave[:, None], pn, n_out)
            first = t_in > 1e-3
            t = torch.where(first, t_in, t_out)
            ok = ~out & (t_in <= t_out) & (t > 1e-3) & (t <= best)
            best = torch.where(ok, t, best)
            normal = torch.where(ok[:, None], torch.where(first[:, None], n_in, n_out), normal)
            mat = torch.where(ok, torch.full_like(mat, k), mat)
        for k, (c, r, _) in enumerate(self.spheres):
            t, ok = self.sphere(c, r, o, d, best)
            best = torch.where(ok, t, best)
            at = o + d * torch.where(ok, t, torch.zeros_like(t))[:, None]
            normal = torch.where(ok[:, None], (at - c) / r, normal)
            mat = torch.where(ok, torch.full_like(mat, len(self.solids) + k), mat)
        front = _dot(normal, d) < 0
        return mat >= 0, best, torch.where(front[:, None], normal, -normal), front, mat

    def scatter(self, rng, lam, o, d, t, normal, front, mat):
        """(origin, direction, weight) after the hit; rows scattered by glass."""
        at = o + d * t[:, None]
        new, weight, glass = torch.zeros_like(d), torch.ones_like(t), torch.zeros_like(front)
        n_glass = torch.ones_like(t)
        for k, (kind, value) in enumerate(self.mats):
            rows = mat == k
            if kind == "glass":
                n_glass, glass = torch.where(rows, _glass_n(value, lam), n_glass), glass | rows
            else:
                weight = torch.where(rows, torch.full_like(weight, _f32(value)), weight)
        diffuse = ~glass
        u1 = rng.next()
        u2 = rng.next(diffuse)
        if diffuse.any():
            rr, phi = u1.sqrt(), 2.0 * math.pi * u2
            near_x = normal[:, 0].abs() > 0.9
            a = torch.where(near_x[:, None], _vec((0, 1, 0)), _vec((1, 0, 0)))
            tang = _norm(torch.linalg.cross(normal, a))
            local = (rr * phi.cos())[:, None] * tang + (rr * phi.sin())[:, None] * torch.linalg.cross(normal, tang)
            new = torch.where(diffuse[:, None], _norm(local + (1.0 - u1).clamp(min=0.0).sqrt()[:, None] * normal), new)
        if glass.any():
            cos_i = (-_dot(d, normal)).abs()
            one = torch.ones_like(n_glass)
            n1, n2 = torch.where(front, one, n_glass), torch.where(front, n_glass, one)
            eta = n1 / n2
            c = cos_i.clamp(0.0, 1.0)
            sin2 = eta * eta * (1.0 - c * c)
            cos_t = (1.0 - sin2).clamp(min=0.0).sqrt()
            rs, rp = (n1 * c - n2 * cos_t) / (n1 * c + n2 * cos_t), (n1 * cos_t - n2 * c) / (n1 * cos_t + n2 * c)
            mirror = (u1 < torch.where(sin2 >= 1.0, one, 0.5 * (rs * rs + rp * rp))) | (sin2 > 1.0)
            reflected = d - normal * (2.0 * _dot(d, normal))[:, None]
            refracted = _norm(d * eta[:, None] + normal * (eta * cos_i - cos_t)[:, None])
            new = torch.where(glass[:, None], torch.where(mirror[:, None], reflected, refracted), new)
        return at, new, weight, glass


class _View:
    def __init__(self, camera, w, h):
        origin, target, up, vfov = camera
        self.o = _vec(origin)
        half = 2.0 * math.tan(math.radians(_f32(vfov)) / 2.0)
        self.z = _norm(self.o - _vec(target))
        self.x = _norm(torch.linalg.cross(_vec(up), self.z))
        self.y = torch.linalg.cross(self.z, self.x)
        self.vw, self.vh, self.w, self.h = half * w / h, half, w, h

    def project(self, q):
        """(in frame, column, row from the top), both in pixels."""
        r = q - self.o
        c = r @ self.z
        front = c < -1e-6
        depth = torch.where(front, -c, torch.ones_like(c))
        s, t = 0.5 + (r @ self.x) / (depth * self.vw), 0.5 + (r @ self.y) / (depth * self.vh)
        return front & (s >= 0) & (s < 1) & (t >= 0) & (t < 1), s * self.w, (1.0 - t) * self.h

    def ray(self, s, t):
        d = self.x * ((s - 0.5) * self.vw)[:, None] + self.y * ((t - 0.5) * self.vh)[:, None] - self.z
        return _norm(d)


def _bin_weights(bins, lo, hi):
    nm = lo + (hi - lo) / bins * (torch.arange(bins, dtype=torch.float64, device=_dev())[:, None] +
                                  (torch.arange(16, dtype=torch.float64, device=_dev()) + 0.5) / 16.0)
    return _lerp(_tables()[:3], nm).mean(1)


def _colour(lam, bins, lo, hi, weights):
    if bins:
        return weights[((lam - lo) * (bins / (hi - lo))).long().clamp(0, bins - 1)]
    return _lerp(_tables()[:3], lam)


def _emit(d, first, count, seed, lo, hi):
    rng = _Rng(torch.arange(first, first + count, device=_dev()) & _M32, seed)
    corner, u, v, direction = (_vec(x) for x in d["beam"])
    o = corner + u * rng.next()[:, None] + v * rng.next()[:, None]
    lam = lo + (hi - lo) * rng.next()
    return rng, o, direction.expand(count, 3).clone(), lam


def _haze_sums(case, d, view, first, count, seed, zbuf=None):
    """Summed XYZ image (h*w, 3) of photons [first, first + count)."""
    w, h, est = case["w"], case["h"], case["estimator"]
    geo, img = _Geometry(d), torch.zeros(w * h, 3, dtype=torch.float64, device=_dev())
    ss, st, g = _f32(case["sigma_s"]), _f32(case["sigma_t"]), _f32(case["g"])
    lo, hi = _f32(case["lo"]), _f32(case["hi"])
    weights = _bin_weights(case["bins"], lo, hi) if case["bins"] else None
    step = 1 << 22
    for base in range(first, first + count, step):
        rng, o, ray, lam = _emit(d, base, min(step, first + count - base), seed, lo, hi)
        col, power = _colour(lam, case["bins"], lo, hi, weights), torch.ones_like(lam)
        for _ in range(case["bounces"]):
            hit, t, normal, front, mat = geo.hit(o, ray)
            seg = torch.where(hit, t, torch.full_like(t, _f32(case["max_dist"])))
            for _ in range(4):
                u = rng.next()
                span, dist = seg, u * seg
                if est == 3 and st > 0:
                    dist = -torch.log1p(u * torch.expm1(-st * seg)) / st
                    span = -torch.expm1(-st * seg) / (st * torch.exp(-st * dist))
                q = o + ray * dist[:, None]
                ok, x, y = view.project(q)
                pix = y.long().clamp(0, h - 1) * w + x.long().clamp(0, w - 1)
                if est == 1:
                    value = power * ss * seg / 4.0 / (4.0 * math.pi)
                else:
                    value, dd = _connect(view, q, ray, power, ss, st, g)
                    value = value * span / 4.0
                    if zbuf is not None:
                        ok = ok & (dd < zbuf[torch.where(ok, pix, torch.zeros_like(pix))])
                at = ok.nonzero()[:, 0]
                img.index_add_(0, pix[at], col[at] * value[at, None])
            keep = hit.nonzero()[:, 0]
            rng, lam, col, power = rng.pick(keep), lam[keep], col[keep], power[keep]
            o, ray, weight, _ = geo.scatter(rng, lam, o[keep], ray[keep], t[keep], normal[keep], front[keep], mat[keep])
            power = power * weight
            if not keep.numel():
                break
    return img


def _connect(view, q, ray, power, ss, st, g):
    """Weight of the camera connection at q before the path-length factor, and
    the distance to the camera."""
    to = view.o - q
    dd = _dot(to, to).sqrt().clamp(min=1e-3)
    den = (1.0 + g * g - 2.0 * g * _dot(ray, to) / dd).clamp(min=1e-6) ** 1.5
    return power * ss * (1.0 - g * g) / (4.0 * math.pi * den) * torch.exp(-st * dd) / (dd * dd), dd


def _beam_sums(case, d, view, seed):
    """The photon-beam estimator: each segment marched, a tent per step."""
    w, h = case["w"], case["h"]
    geo, img = _Geometry(d), torch.zeros(w * h, 3, dtype=torch.float64, device=_dev())
    ss, st, g = _f32(case["sigma_s"]), _f32(case["sigma_t"]), _f32(case["g"])
    lo, hi = _f32(case["lo"]), _f32(case["hi"])
    weights = _bin_weights(case["bins"], lo, hi) if case["bins"] else None
    step = 1 << 16
    for base in range(0, case["photons"], step):
        rng, o, ray, lam = _emit(d, base, min(step, case["photons"] - base), seed, lo, hi)
        col, power = _colour(lam, case["bins"], lo, hi, weights), torch.ones_like(lam)
        for _ in range(case["bounces"]):
            hit, t, normal, front, mat = geo.hit(o, ray)
            seg = torch.where(hit, t, torch.full_like(t, _f32(case["max_dist"])))
            ok0, x0, y0 = view.project(o)
            ok1, x1, y1 = view.project(o + ray * seg[:, None])
            on_film = torch.hypot(x1 - x0, y1 - y0) * 2.0
            m = torch.where(ok0 & ok1, on_film.ceil().clamp(0, 4096) + 1, (seg * 80.0).ceil().clamp(0, 4096))
            m = m.clamp(1, 4096).long()
            ends = m.cumsum(0)
            total, part = int(ends[-1]), 1 << 22
            for s0 in range(0, total, part):
                k = torch.arange(s0, min(s0 + part, total), device=_dev())
                row = torch.searchsorted(ends, k, right=True)
                ds = seg[row] / m[row]
                q = o[row] + ray[row] * ((k - ends[row] + m[row] + 0.5) * ds)[:, None]
                inside, px, py = view.project(q)
                at = inside.nonzero()[:, 0]
                _tents(img, view, q[at], ray[row[at]], power[row[at]], col[row[at]], ds[at], px[at], py[at], ss, st, g)
            keep = hit.nonzero()[:, 0]
            rng, lam, col, power = rng.pick(keep), lam[keep], col[keep], power[keep]
            o, ray, weight, _ = geo.scatter(rng, lam, o[keep], ray[keep], t[keep], normal[keep], front[keep], mat[keep])
            power = power * weight
            if not keep.numel():
                break
    return img


def _tents(img, view, q, ray, power, col, ds, px, py, ss, st, g):
    w, h = view.w, view.h
    value, dd = _connect(view, q, ray, power, ss, st, g)
    look = (view.o - q) / dd[:, None]
    perp = torch.linalg.cross(look, _vec((0, 1, 0)).expand_as(look))
    flat = _dot(perp, perp) < 1e-8
    perp = torch.where(flat[:, None], torch.linalg.cross(look, _vec((1, 0, 0)).expand_as(look)), perp)
    ok, ex, ey = view.project(q + _norm(perp) * _f32(0.03))
    r = torch.where(ok, torch.hypot(ex - px, ey - py).clamp(1.5, 24.0), torch.ones_like(px))
    cx, cy = px - 0.5, py - 0.5
    x0, y0 = (cx - r).floor().clamp(min=0.0), (cy - r).floor().clamp(min=0.0)
    x1, y1 = (cx + r).ceil().clamp(0, w - 1), (cy + r).ceil().clamp(0, h - 1)
    wide, high = int((x1 - x0).max()) + 1 if px.numel() else 0, int((y1 - y0).max()) + 1 if px.numel() else 0
    cells = [(i, j) for j in range(high) for i in range(wide)]

    def tent(i, j):
        x, y = x0 + i, y0 + j
        t = (1.0 - torch.hypot(x - cx, y - cy) / r).clamp(min=0.0)
        return x, y, torch.where((x <= x1) & (y <= y1), t, torch.zeros_like(t))
    total = torch.zeros_like(px)
    for i, j in cells:
        total = total + tent(i, j)[2]
    value = col * (value * ds)[:, None]
    share = torch.where(total > 0, 1.0 / total.clamp(min=1e-300), torch.zeros_like(total))
    for i, j in cells:
        x, y, t = tent(i, j)
        at = (t > 0).nonzero()[:, 0]
        img.index_add_(0, (y[at] * w + x[at]).long(), value[at] * (t[at] * share[at])[:, None])
    lost = (total <= 0).nonzero()[:, 0]
    img.index_add_(0, (cy[lost].round().clamp(0, h - 1) * w + cx[lost].round().clamp(0, w - 1)).long(), value[lost])


def _job_image(spec, first, count, camera=specs.PRISM_CAMERA):
    d = dict(solids=[(specs.prism_planes(spec["apex_deg"], 1.0, 1.0), ("glass", spec["glass"]))], spheres=[],
             beam=specs.prism_beam(spec["apex_deg"], 1.0, spec["incidence_deg"], 0.02))
    c = dict(w=spec["width"], h=spec["height"], bins=spec["bins"], estimator=0, sigma_s=spec["sigma_s"],
             sigma_t=spec["sigma_t"], g=spec["g"], lo=spec["lambda_min"], hi=spec["lambda_max"], max_dist=6.0, bounces=8)
    return _haze_sums(c, d, _View(camera, c["w"], c["h"]), first, count, spec["seed"]).reshape(-1)


def _orbit(frame, deg):
    (x, y, z), target, up, vfov = specs.PRISM_CAMERA
    a = math.radians(deg * frame)
    dx, dz = x - ORBIT_TARGET[0], z - ORBIT_TARGET[2]
    return ((ORBIT_TARGET[0] + dx * math.cos(a) + dz * math.sin(a), y,
             ORBIT_TARGET[2] - dx * math.sin(a) + dz * math.cos(a)), target, up, vfov)


def _request_image(spec, frames, orbit):
    n = spec["n_photons"]
    if orbit:
        return _job_image(spec, (frames - 1) * n, n, _orbit(frames - 1, orbit))
    return _job_image(spec, 0, frames * n) / frames


def _tracer_image(case, seed):
    d, w, h = _tracer_spec(case, seed), case["w"], case["h"]
    geo, view, table = _Geometry(d), _View(d["camera"], w, h), _tables()
    opt, n = d["tracer"], w * h
    emitter, rr = opt.get("emitter"), opt.get("rr_start", 0)
    horizon = d.get("horizon") or 0.0
    img = torch.zeros(n, 3, dtype=torch.float64, device=_dev())
    pixel = torch.arange(n, device=_dev())
    for sample in range(case["spp"]):
        rng = _Rng(_pcg(pixel ^ _pcg(torch.tensor(sample, device=_dev()))), _photon_seed(seed))
        s, t = ((pixel % w) + rng.next()) / w, 1.0 - ((pixel // w) + rng.next()) / h
        u = rng.next()
        ray, o, at = view.ray(s, t), view.o.expand(n, 3), pixel
        tp, four = torch.ones_like(u), torch.ones_like(u, dtype=torch.bool)
        for bounce in range(opt["max_depth"]):
            hit, dist, normal, front, mat = geo.hit(o, ray)
            light = torch.zeros_like(u)
            over = ~hit
            if emitter:
                _, lamp = geo.sphere(_vec(emitter[0]), _f32(emitter[1]), o, ray, dist)
                light, over = torch.where(lamp, torch.full_like(u, _f32(emitter[2])), light), over | lamp
                sky = ~hit & ~lamp
            else:
                sky = ~hit
            light = torch.where(sky, case["background"] + horizon * (ray[:, 1] > 0).double(), light)
            e = over.nonzero()[:, 0]
            for k in range(4):
                lam = 380.0 + (u[e] * 350.0 + k * 87.5) % 350.0
                share = torch.where(four[e], 0.25 * torch.ones_like(u[e]), float(k == 0) * torch.ones_like(u[e]))
                rad = tp[e] * light[e] * _lerp(table[3 + case["illuminant"]:4 + case["illuminant"]], lam)[:, 0]
                img.index_add_(0, at[e], _lerp(table[:3], lam) * (rad * share * 350.0)[:, None])
            keep = (~over).nonzero()[:, 0]
            if not keep.numel():
                break
            rng, u, at, tp, four = rng.pick(keep), u[keep], at[keep], tp[keep], four[keep]
            o, ray, weight, glass = geo.scatter(rng, 380.0 + (u * 350.0) % 350.0, o[keep], ray[keep], dist[keep],
                                                normal[keep], front[keep], mat[keep])
            tp, four = tp * weight, four & ~glass
            if rr and bounce + 1 >= rr:
                p = tp.clamp(max=_f32(0.95))
                alive = (rng.next() < p).nonzero()[:, 0]
                rng, u, at, four, o, ray = rng.pick(alive), u[alive], at[alive], four[alive], o[alive], ray[alive]
                tp = tp[alive] / p[alive]
    return (img / case["spp"]).reshape(-1)


def _rectangle(screen, o, d):
    """(hit parameter or inf, s, r) of the rays on a screen rectangle."""
    corner, u, v = _vec(screen.corner), _vec(screen.u), _vec(screen.v)
    n = _norm(torch.linalg.cross(u, v))
    den = d @ n
    flat = den.abs() < 1e-8
    t = ((corner - o) @ n) / torch.where(flat, torch.ones_like(den), den)
    rel = o + d * t[:, None] - corner
    s, r = (rel @ u) / _dot(u, u), (rel @ v) / _dot(v, v)
    ok = ~flat & (t > 1e-4) & (s >= 0) & (s < 1) & (r >= 0) & (r < 1)
    return torch.where(ok, t, torch.full_like(t, _INF)), s, r


def _caustic(floor, d, photons, seed):
    w, h = floor.width, floor.height
    geo, img = _Geometry(d), torch.zeros(w * h, 3, dtype=torch.float64, device=_dev())
    rng, o, ray, lam = _emit(d, 0, photons, seed, 380.0, 730.0)
    power = torch.ones_like(lam)
    for _ in range(8):
        hit, t, normal, front, mat = geo.hit(o, ray)
        ts, s, r = _rectangle(floor, o, ray)
        land = ts < t
        x, y = (s[land] * w - 0.5).clamp(0, w - 1), ((1.0 - r[land]) * h - 0.5).clamp(0, h - 1)
        x0, y0 = x.floor(), y.floor()
        value = _lerp(_tables()[:3], lam[land]) * power[land, None]
        for i, fx in ((0, 1.0 - (x - x0)), (1, x - x0)):
            for j, fy in ((0, 1.0 - (y - y0)), (1, y - y0)):
                cell = (y0 + j).clamp(max=h - 1) * w + (x0 + i).clamp(max=w - 1)
                img.index_add_(0, cell.long(), value * (fx * fy)[:, None])
        keep = (hit & ~land).nonzero()[:, 0]
        if not keep.numel():
            break
        rng, lam, power = rng.pick(keep), lam[keep], power[keep]
        o, ray, weight, _ = geo.scatter(rng, lam, o[keep], ray[keep], t[keep], normal[keep], front[keep], mat[keep])
        power = power * weight
    return img


def _plane_images(case, seed):
    _, floor, _, _ = scenes.prism_on_plane(case["w"], case["h"], case["texels"])
    d = dict(solids=[(scenes.wedge_planes(30.0, 1.0, 2.0), ("glass", specs.SF11))], spheres=[],
             beam=((-3.0, 0.55, -0.75), (0.0, 0.0, 1.5), (0.0, 0.12, 0.0), (1.0, 0.0, 0.0)))
    w, h = case["w"], case["h"]
    view = _View(((0.0, 4.5, 9.0), (4.0, -1.2, 0.0), (0.0, 1.0, 0.0), 50.0), w, h)
    pixel = torch.arange(w * h, device=_dev())
    ray = view.ray(((pixel % w) + 0.5) / w, 1.0 - ((pixel // w) + 0.5) / h)
    o = view.o.expand(w * h, 3)
    zbuf = torch.minimum(_Geometry(d).hit(o, ray)[1], _rectangle(floor, o, ray)[0])
    haze = dict(w=w, h=h, bins=0, estimator=0, sigma_s=0.5, sigma_t=0.06, g=0.5, lo=380.0, hi=730.0, max_dist=22.0,
                bounces=8)
    # pixels on the outline of the wedge or the floor hit one side or the other by rounding: no exact distance there
    return [_caustic(floor, d, case["photons"], _photon_seed(seed)), None,
            _haze_sums(haze, d, view, 0, case["photons"], _photon_seed(seed), zbuf).reshape(-1)]


def exact(case, seed):
    kind, ps = case["kind"], _photon_seed(seed)
    if kind == "viewer":
        return None  # bytes
    if kind in ("device", "object"):
        d = _scene_spec(case["scene"], seed)
        view = _View(d["camera"], case["w"], case["h"])
        if case["estimator"] == 2:
            return _beam_sums(case, d, view, ps).reshape(-1)
        img = _haze_sums(case, d, view, 0, case["photons"], ps).reshape(-1)
        return img if kind == "device" else [img, None, None]
    if kind == "batch":
        jobs = _batch_specs(case, seed)
        if sum(j["n_photons"] for j in jobs) > 1 << 26:
            return None  # over 20 seconds
        return torch.cat([_job_image(j, 0, j["n_photons"]) for j in jobs])
    if kind == "serve":
        return [_request_image(*r) for r in _requests(case, seed)]
    if kind == "tracer":
        return _tracer_image(case, seed)
    return _plane_images(case, seed)
