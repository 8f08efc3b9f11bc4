"""The grouped photon transport over the forms its launches take: photon counts
at the edges of a warp's chunk and of the rule that divides a launch, films with
and without the shared-memory cell cache, values too large for the cache, groups
of photons that end after very different numbers of bounces.

Films are sums of exact integers, so one launch and the same photons in many
small launches (32 photons a warp, no cache) must agree in every cell; paths
must equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle
import spectral_b200 as sb
from spectral_b200 import scenes, specs
from helpers import axis_box, device_desc, obeam, oscene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sb.GpuContext(0)
    yield c
    c.close()


def mixed_scene():
    """Spheres and solids of several glasses and a diffuse floor in a wide beam."""
    s = sb.Scene(background=0.0)
    s.add_sphere((0.0, 0.0, 0.0), 0.8, sb.Dielectric(sb.WATER))
    s.add_solid(specs.prism_planes(60.0, 1.0, 1.0), sb.Dielectric(sb.SF11))
    s.add_solid(axis_box((1.6, -0.5, -0.4), (2.2, 0.5, 0.4)), sb.Dielectric(sb.BK7))
    s.add_sphere((1.5, -0.5, 0.2), 0.5, sb.Lambertian(0.7))
    s.add_solid([((0.0, 1.0, 0.0), 1.2)], sb.Lambertian(0.6))
    beam = sb.Beam((-3.0, -0.7, -0.7), (0.0, 0.0, 1.4), (0.0, 1.4, 0.0), sb.f32_normalize((1.0, 0.02, 0.01)))
    return s, beam, ((0.5, 0.6, 6.0), (0.3, 0.0, 0.0), (0.0, 1.0, 0.0), 45.0)


def workload(name):
    if name == "mixed":
        return mixed_scene()
    d = {"prism": specs.prism_scene, "dsotm": specs.dsotm_scene, "rainbow": specs.rainbow_scene}[name]()
    return scenes.scene_from_spec(d), sb.Beam(*d["beam"]), d["camera"]


# 2^15: the cache's smallest launch; 151,552 photons: the most at 32 a warp on 148 SMs
@pytest.mark.parametrize("name,w,h,bins,n,kw", [
    ("prism", 160, 90, 0, (1 << 15) - 1, {}),
    ("prism", 160, 90, 0, 1 << 15, {}),
    ("prism", 161, 91, 0, 151_553, {}),
    ("prism", 161, 91, 8, 151_552, {}),
    ("prism", 160, 90, 9, 300_001, {}),
    ("dsotm", 333, 187, 0, 700_003, dict(g=0.5)),
    ("dsotm", 96, 64, 1, 400_000, dict(g=-0.3, estimator=1)),
    ("dsotm", 96, 64, 3, 200_000, dict(estimator=3, sigma_t=0.4)),
    ("rainbow", 320, 180, 0, 1_300_000, dict(max_bounces=20)),
    ("mixed", 200, 150, 0, 250_000, dict(max_bounces=64)),
    ("mixed", 64, 48, 2, 250_000, dict(z=5.9)),
    ("prism", 64, 36, 0, 100_000, dict(scale_log2=44))])  # deposits of 2^23 quanta and more pass the cache by
def test_one_launch_equals_many(ctx, name, w, h, bins, n, kw):
    kw = dict(kw)
    z = np.full(w * h, kw.pop("z"), np.float32) if "z" in kw else None
    wts = sb.VolWeights(0.3, kw.pop("sigma_t", 0.05), kw.pop("g", 0.0))
    scene, beam, cam = workload(name)
    cam = sb.Camera.look_at(*cam, w / h)
    f = sb.GpuPhotonFilm(ctx, scene, cam, beam, w, h, n, 5, 8.0, wts, zbuffer=z, bins=bins, **kw)
    f.trace_and_resolve(n, 5)
    whole = f.read_raw()
    f.clear_film()
    for a in range(0, n, 30_011):
        f.dispatch_photons(a, min(a + 30_011, n), 5)
    assert whole.sum() > 0 and np.array_equal(f.read_raw(), whole)
    f.close()


@pytest.mark.parametrize("bounces,n,part,bins", [
    (300, 96, 1, 4),           # photons set aside after more than 255 bounces
    (2000, 40_000, 4_000, 0)])  # more deposits of a CTA than the cell cache sums exactly
def test_long_paths(ctx, bounces, n, part, bins):
    """The device entry takes any bounce limit: photons totally reflected in a
    glass cube until it, beside others that miss the cube, so that lanes fall idle
    and photons of different bounces are set aside."""
    import ctypes as C

    import torch
    from spectral_b200 import _lib
    scene = sb.Scene(background=0.0)
    scene.add_solid(axis_box((-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)), sb.Dielectric(sb.SF11))
    beam = sb.Beam((0.2, 0.0, 0.0), (1.4, 0.0, 0.0), (0.0, 0.01, 0.0), sb.f32_normalize((1.0, 1.0, 1.0)))
    cam, keep, films = sb.Camera.look_at((0.0, 0.0, 8.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 40.0, 1.0), [], []
    desc = device_desc(sb, _lib, torch, scene, cam, beam, 16, 16, 3, bins, keep)
    desc.opts.max_bounces = bounces
    for step in (n, part):
        film = torch.zeros(_lib.lib.sc_film_bytes(16, 16, bins or 3) // 8, dtype=torch.int64, device="cuda")
        for a in range(0, n, step):
            _lib.check(_lib.lib.sc_trace_photons_device(ctx.h, C.byref(desc), a, min(step, n - a),
                                                        C.c_void_p(film.data_ptr()), None, None))
        torch.cuda.synchronize()
        films.append(film)
    assert films[0].sum().item() > 0 and torch.equal(films[0], films[1])


@pytest.mark.parametrize("bounces", [1, 2, 8, 20])
def test_paths_through_several_solids(ctx, bounces):
    """Bit-identical paths where rays start on, inside and outside spheres and
    solids, graze them and miss them."""
    scene = sb.Scene(background=0.0)
    scene.add_sphere((0.0, 0.0, 0.0), 0.8, sb.Dielectric(sb.WATER))
    scene.add_solid(specs.prism_planes(60.0, 1.0, 1.0), sb.Dielectric(sb.SF11))
    scene.add_solid(axis_box((0.9, -1.0, -1.0), (1.4, 1.0, 1.0)), sb.Dielectric(sb.BK7))
    scene.add_sphere((2.0, 0.1, 0.0), 0.37, sb.Dielectric(sb.FUSED_SILICA))
    _, beam, cam = mixed_scene()
    n = 3000
    f = sb.GpuPhotonFilm(ctx, scene, sb.Camera.look_at(*cam, 1.0), beam, 32, 32, n, 9, 9.0, max_bounces=bounces)
    num, lam, states = f.trace_debug(n, 9, n)
    p = oracle.vol_params(32, 32, 9, max_dist=9.0, max_bounces=bounces)
    osc, ob, longest = oscene(scene), obeam(beam), 0
    for i in range(n):
        k, wl, st, _ = oracle.simulate_photon(osc, ob, p, i)
        k = min(k, 9)
        longest = max(longest, k)
        assert num[i] == k and np.float32(lam[i]) == np.float32(wl)
        assert np.array_equal(states[i, :2 * k], st[:k].reshape(-1, 4)), i
    assert longest >= min(bounces, 5)
    f.close()


@pytest.mark.parametrize("n_jobs,photons,chunk", [
    (1, (1, 1), 0),               # one photon for all warps
    (1, (200_000, 200_000), 64),  # items at their smallest
    (3, (31, 70_001), 8192),      # shares far below the chunk
    (40, (2_000, 500_000), 512),  # shares above the chunk, then below it
    (2, (3_000_000, 3_000_000), 1 << 20)])
def test_uneven_items_cover_every_photon(ctx, n_jobs, photons, chunk):
    """Work items of any sizes trace each photon once: the batch's images equal
    the plain per-scene launches' (which have no items)."""
    from spectral_b200.batch import Batch, prism_jobs
    jobs = prism_jobs(specs.random_prism_jobs(n_jobs, 3, 8, photons=photons, side=(40, 90)))
    b = Batch(ctx, jobs, chunk_photons=chunk)
    b.run()
    b.synchronize()
    batched = b.read_all_xyz()
    b.run_plain()
    b.synchronize()
    assert np.array_equal(b.read_all_xyz(), batched)
    b.close()
