"""Calls at the edges of what the entry points accept: weights below zero, rays
without a direction, films so wide that 16-bit differences of their columns wrap,
films of more than 2^32 cells or of three bins, calls that take more memory than a
context keeps.

Films are sums of exact integers: every cell is compared."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
import spectral_b200 as sb
from spectral_b200 import _lib, scenes, specs
from spectral_b200.batch import Batch, prism_jobs
from helpers import axis_box, device_desc, obeam, oracle_job_xyz, oscene, rel_l1

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def _dsotm(ctx, n, w=64, h=48, weights=sb.VolWeights(), scene=None, **kw):
    d, beam, cam = sb.dsotm_scene(w / h)
    return sb.GpuPhotonFilm(ctx, scene or d, cam, beam, w, h, n, 3, 14.0, weights, **kw)


# 40,000 photons: films of up to 8 bins and XYZ films go through the cell cache
@pytest.mark.parametrize("bins", [0, 8, 16, 64])
@pytest.mark.parametrize("weights,kw", [
    ((-0.5, 0.06, 0.5), {}),
    ((-1e-9, 0.06, 0.0), {}),               # weights of a few quanta and of less than one
    ((0.5, 0.06, 1.2), {}),                 # 1 - g^2 < 0
    ((float("nan"), 0.06, 0.5), {}),
    ((-0.5, 0.3, 0.5), dict(estimator=3))])
def test_weights_below_zero_leave_a_film_black(ctx, bins, weights, kw):
    f = _dsotm(ctx, 40_000, weights=sb.VolWeights(*weights), bins=bins, **kw)
    f.trace_and_resolve(40_000, 3)
    assert not f.read_raw().any()
    f.close()


def test_a_batch_of_weights_below_zero_is_black(ctx):
    jobs = prism_jobs(specs.random_prism_jobs(2, 3, 16, photons=(20_000, 30_000), side=(40, 90)))
    jobs[0].weights.sigma_s = -0.5
    jobs[1].weights.g = 1.2
    b = Batch(ctx, jobs)
    b.run()
    b.synchronize()
    assert not b.read_all_xyz().any()
    b.close()


def test_weights_of_both_signs(ctx, monkeypatch):
    """A reflectance below zero turns a photon's weight at every diffuse hit: the
    samples below zero add nothing, whichever kernel deposits them."""
    scene = sb.Scene(background=0.0)
    scene.add_solid(axis_box((-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)), sb.Lambertian(-0.6))
    scene.add_solid([((-1.0, 0.0, 0.0), -3.5)], sb.Lambertian(0.9))
    raws = []
    for aggregate in ("0", "1"):
        monkeypatch.setenv("SPECTRAL_CUDA_AGGREGATE", aggregate)
        f = _dsotm(ctx, 50_000, scene=scene, bins=16)
        f.trace_and_resolve(50_000, 3)
        raws.append(f.read_raw())
        f.close()
    assert raws[0].sum() > 0 and np.array_equal(raws[0], raws[1])


@pytest.mark.parametrize("across", [True, False])
@pytest.mark.parametrize("bins", [0, 1])
def test_beam_film_whose_columns_differ_by_almost_2_to_16(ctx, across, bins):
    """Beams along a film of 65,535 columns (or rows).  Behind a thin slab every
    photon marches the frame from edge to edge: the last step of one lies on the
    last column, the first of the next on the first.  In the whole launch a warp has
    several photons, in the small ones a single photon."""
    side, thin, n, part = 65_535, 16, 60_000, 3_000
    w, h = (side, thin) if across else (thin, side)
    half, far = 700.0, 1000.0  # half the frame's long side, the camera's distance
    ds = 2.0 * half / 4090.0   # 4096 steps a segment: 4091 from edge to edge, 5 behind it
    vfov = 2.0 * np.degrees(np.arctan((half * thin / side if across else half) / far))
    cam = sb.Camera.look_at((0.0, 0.0, far), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), float(vfov), w / h)
    lo, hi = -half - 0.5 * ds - 0.05, -half - 0.495 * ds
    scene = sb.Scene(background=0.0)
    # they start within 0.1 units of the slab, 1 to 9 steps before it, and march
    # towards the last column, or the last row (downwards)
    if across:
        scene.add_solid([((1.0, 0.0, 0.0), -hi), ((-1.0, 0.0, 0.0), lo)], sb.Dielectric(sb.BK7))
        beam = sb.Beam((lo - 0.11, -0.02, 0.0), (0.1, 0.0, 0.0), (0.0, 0.04, 0.0), (1.0, 0.0, 0.0))
    else:
        scene.add_solid([((0.0, 1.0, 0.0), lo), ((0.0, -1.0, 0.0), -hi)], sb.Dielectric(sb.BK7))
        beam = sb.Beam((-0.02, 0.11 - lo, 0.0), (0.0, -0.1, 0.0), (0.04, 0.0, 0.0), (0.0, -1.0, 0.0))
    f = sb.GpuPhotonFilm(ctx, scene, cam, beam, w, h, n, 7, 4096.0 * ds * 0.99999, sb.VolWeights(0.5, 0.0, 0.0),
                         estimator=sb.BEAM, bins=bins, scale_log2=44)
    f.dispatch_photons(0, n, 7)
    whole = f.read_raw()
    f.clear_film()
    for a in range(0, n, part):
        f.dispatch_photons(a, a + part, 7)
    assert whole.sum() > 0 and np.array_equal(f.read_raw(), whole)
    f.close()


def test_cell_cache_of_a_film_of_more_than_2_to_32_cells(ctx):
    """A film one pixel high has eight times its pixels in padded cells: 83,886,080
    x 1 of 8 bins are 5 * 2^30 cells (43 GB).  A launch that is large enough for the
    cell cache gives the image of small launches that do without."""
    import torch
    w, n = 5 << 24, 60_000
    scene = sb.Scene(background=0.0)
    beam = sb.Beam((-3.0, -0.01, 0.0), (0.0, 0.02, 0.0), (0.0, 0.0, 0.02), (1.0, 0.0, 0.0))
    cam = sb.Camera.look_at((0.0, 0.0, 6.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 30.0, 1.0)
    keep, images = [], []
    desc = device_desc(sb, _lib, torch, scene, cam, beam, w, 1, 3, 8, keep, scale_log2=24)  # below 2^22 quanta
    film = torch.zeros(_lib.lib.sc_film_bytes(w, 1, 8) // 8, dtype=torch.int64, device="cuda")
    flags = torch.zeros(_lib.lib.sc_film_flag_bytes(w, 1) // 4, dtype=torch.int32, device="cuda")
    assert film.numel() > 1 << 32
    for step in (n, 20_000):  # the cache is taken from 2^15 photons on
        xyz = torch.empty(3 * w, dtype=torch.float32, device="cuda")
        for a in range(0, n, step):
            _lib.check(_lib.lib.sc_trace_photons_device(ctx.h, C.byref(desc), a, min(step, n - a),
                                                        C.c_void_p(film.data_ptr()), C.c_void_p(flags.data_ptr()),
                                                        None))
        _lib.check(_lib.lib.sc_sensor_reduce_device(ctx.h, w, 1, 8, 380.0, 730.0, 24, C.c_void_p(film.data_ptr()),
                                                    C.c_void_p(flags.data_ptr()), C.c_void_p(xyz.data_ptr()), 1,
                                                    None))
        torch.cuda.synchronize()
        images.append(xyz)
    same = torch.equal(images[0], images[1])
    beyond = images[1][3 << 26:].sum().item()  # cells from 2^32 on
    del film, images, xyz
    torch.cuda.empty_cache()
    assert same and beyond > 0


@pytest.mark.parametrize("direction", [(float("nan"), 0.0, 0.0), (0.0, 0.0, float("nan"))])
def test_rays_without_a_direction(ctx, direction):
    """A NaN direction passes every plane test of a solid by, whichever side of
    the planes the ray starts on: paths end where the CPU crate's do."""
    scene = sb.Scene(background=0.0)
    scene.add_solid(axis_box((-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)), sb.Dielectric(sb.SF11))
    beam = sb.Beam((-3.0, -0.5, -0.5), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0), direction)
    cam = sb.Camera.look_at((0.0, 0.0, 8.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 40.0, 1.0)
    f = sb.GpuPhotonFilm(ctx, scene, cam, beam, 32, 32, 64, 9, 9.0, max_bounces=5)
    num, _, _ = f.trace_debug(64, 9, 64)
    p = oracle.vol_params(32, 32, 9, max_dist=9.0, max_bounces=5)
    assert num.tolist() == [oracle.simulate_photon(oscene(scene), obeam(beam), p, i)[0] for i in range(64)]
    f.close()


def test_films_of_three_bins_are_spectral(ctx):
    """The images of a film of three bins (film object, allocation-free call, batch,
    plain launches) are its bins times the bin-averaged colour-matching functions."""
    import torch
    n, w, h = 20_000, 64, 48
    weights = oracle.bin_weights(3, 380.0, 730.0).astype(np.float64)
    f = _dsotm(ctx, n, w, h, bins=3)
    f.trace_and_resolve(n, 3)
    raw = f.read_raw().reshape(-1, 3).astype(np.float64)
    # three f64 products and sums, rounded to f32 once
    expect = (raw @ weights.T).reshape(-1) * 2.0 ** -32
    assert raw.sum() > 0 and np.abs(f.accum() - expect).max() <= 2.0 ** -23 * expect.max()
    scene, beam, cam = sb.dsotm_scene(w / h)
    keep = []
    desc = device_desc(sb, _lib, torch, scene, cam, beam, w, h, 3, 3, keep)
    xyz = torch.empty(3 * w * h, dtype=torch.float32, device="cuda")
    _lib.check(_lib.lib.sc_trace_xyz_noalloc(sb.sample_tables().ctypes.data_as(C.POINTER(C.c_float)), C.byref(desc),
                                             0, n, C.c_void_p(xyz.data_ptr()), None))
    torch.cuda.synchronize()
    assert np.array_equal(xyz.cpu().numpy(), f.accum())
    f.close()
    job = prism_jobs(specs.random_prism_jobs(1, 3, 3, photons=(20_000, 20_000), side=(40, 60)))
    j = job[0]
    b = Batch(ctx, job)
    images = []
    for run in (b.run, b.run_plain):
        run()
        b.synchronize()
        images.append(b.read_all_xyz())
    b.close()
    ref = oracle_job_xyz(j)
    assert ref.sum() > 0 and np.array_equal(images[0], images[1]) and rel_l1(images[0], ref) < 2e-3


def test_large_calls_give_their_memory_back(ctx):
    """A caustic and a z-buffer of more memory than a context keeps leave the
    device's free memory as it was."""
    import torch
    scene, beam, cam = sb.dsotm_scene(1.0)
    screen = sb.Screen((-4.0, -1.0, -4.0), (8.0, 0.0, 0.0), (0.0, 0.0, 8.0), 64, 64)
    sb.trace(ctx, scene, screen, beam, 1000, 3)  # kernels loaded
    sb.scene_zbuffer(ctx, scene, cam, 64, 64)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    large = sb.Screen((-4.0, -1.0, -4.0), (8.0, 0.0, 0.0), (0.0, 0.0, 8.0), 4096, 4096)  # 604 MB
    sb.trace(ctx, scene, large, beam, 1000, 3)
    sb.scene_zbuffer(ctx, scene, cam, 8192, 4096)  # 134 MB
    assert large.sum.sum() > 0
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20


@pytest.mark.parametrize("bins", [0, 16])
@pytest.mark.parametrize("g", [0.0, 0.4])
def test_free_flight_samples_with_and_without_a_z_buffer(ctx, bins, g):
    """A z-buffer that hides nothing has its samples worked out one by one: the
    same cells as the four of a segment together."""
    raws = []
    for z in (None, np.full(64 * 48, np.inf, np.float32)):
        f = _dsotm(ctx, 50_000, weights=sb.VolWeights(0.5, 0.3, g), bins=bins, estimator=3, zbuffer=z)
        f.trace_and_resolve(50_000, 3)
        raws.append(f.read_raw())
        f.close()
    assert raws[0].sum() > 0 and np.array_equal(raws[0], raws[1])


@pytest.mark.parametrize("bins", [0, 16])
@pytest.mark.parametrize("weights", [(-0.5, 0.06, 0.5), (0.5, 0.06, 1.2)])
def test_beam_weights_below_zero_leave_a_film_black(ctx, bins, weights):
    f = _dsotm(ctx, 500, weights=sb.VolWeights(*weights), bins=bins, estimator=sb.BEAM)
    f.trace_and_resolve(500, 3)
    assert not f.read_raw().any()
    f.close()


# samples a cell (32 x photons a warp / pixels under the beam) on both sides of the lines:
# empty scenes 0.4, single segments and launches below 2^16 photons 0.05, others 0.02
@pytest.mark.parametrize("name,w,h,n,kw", [
    ("prism", 96, 64, 40_000, {}), ("rainbow", 96, 64, 40_000, {}),
    ("rainbow", 200, 200, 65_535, {}), ("rainbow", 200, 200, 65_536, {}),
    ("rainbow", 128, 128, 65_535, dict(max_bounces=1)), ("rainbow", 256, 256, 65_536, dict(max_bounces=1))])
@pytest.mark.parametrize("empty", [False, True])
def test_cell_cache_on_both_sides_of_its_lines(ctx, name, w, h, n, kw, empty):
    d = {"prism": specs.prism_scene, "rainbow": specs.rainbow_scene}[name]()
    scene = sb.Scene(background=0.0) if empty else scenes.scene_from_spec(d)
    f = sb.GpuPhotonFilm(ctx, scene, sb.Camera.look_at(*d["camera"], w / h), sb.Beam(*d["beam"]), w, h, n, 5, 8.0,
                         sb.VolWeights(0.3, 0.05, 0.0), **kw)
    f.trace_and_resolve(n, 5)
    whole = f.read_raw()
    f.clear_film()
    for a in range(0, n, 30_011):  # too small for the cache
        f.dispatch_photons(a, min(a + 30_011, n), 5)
    assert whole.sum() > 0 and np.array_equal(f.read_raw(), whole)
    f.close()


def test_beam_film_whose_scene_grows():
    """A beam film created for a small scene takes the largest one afterwards.  In a
    process of its own: no other film has raised the kernel's shared memory there."""
    code = """
import spectral_b200 as sb
ctx = sb.GpuContext(0)
scene, beam, cam = sb.dsotm_scene(1.0)
f = sb.GpuPhotonFilm(ctx, scene, cam, beam, 320, 320, 200, 3, 14.0, sb.VolWeights(), estimator=sb.BEAM)
f.trace_and_resolve(200, 3)
one = f.read_raw()
box = [((1, 0, 0), -1e3), ((-1, 0, 0), -1e3), ((0, 1, 0), -1e3), ((0, -1, 0), -1e3)]
for i in range(50):  # far behind every photon and the camera
    scene.add_solid([((0, 0, 1), 1e3 + i), ((0, 0, -1), -1e3 - i - 0.5)] + box[:3], sb.Lambertian(0.5))
f.set_scene(scene, cam, beam)
f.clear_film()
f.trace_and_resolve(200, 3)
assert one.sum() > 0 and (f.read_raw() == one).all()
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
