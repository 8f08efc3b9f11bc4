"""Photon-beam films whose footprints take each splat path: boxes within 8x8 and
16x16 pixels (sliding windows), larger ones (on their own), boxes clipped by
every film edge, single-pixel films, deposits too large for the windows' 32-bit
sums, and photon counts from one to several per warp.

Bars: 1e-4 relative L1 against the oracle's f32 image, as for the other beam
films (per-deposit arithmetic within a few ulp, the oracle sums in f32); any
split of the photons into launches gives the same integers."""
import numpy as np
import pytest

import oracle
import spectral_b200 as sb
from spectral_b200 import scenes, specs
from helpers import obeam, ocam, oscene, rel_l1

pytestmark = pytest.mark.gpu


def workload(name, w, h):
    d = {"prism": specs.prism_scene, "dsotm": specs.dsotm_scene, "rainbow": specs.rainbow_scene}[name]()
    o, t, up, vfov = d["camera"]
    return scenes.scene_from_spec(d), sb.Beam(*d["beam"]), sb.Camera.look_at(o, t, up, vfov, w / h)


# projected beam radius in pixels: about 0.0033 h (dsotm), 0.0065 h (prism), 0.0035 h (rainbow), at least 1.5
@pytest.mark.parametrize("name,w,h,n,scale", [
    ("dsotm", 64, 48, 900, 40),      # 1.5 px: the smallest boxes
    ("dsotm", 9, 7, 400, 40),        # film smaller than a window
    ("dsotm", 1, 1, 60, 40),         # every box clipped to one pixel
    ("rainbow", 320, 240, 300, 40),  # photons that leave the frame on every side
    ("prism", 500, 460, 120, 40),    # 3 px: the 8x8 window nearly full
    ("prism", 701, 640, 60, 40),     # 4 px: both windows in use
    ("prism", 1201, 1200, 12, 40),   # 8 px: at the 16x16 window's edge
    ("prism", 1500, 1900, 6, 40),    # 12 px: boxes of their own
    ("dsotm", 100, 75, 200, 50),     # deposits of 2^23 quanta and more
    ("dsotm", 100, 75, 1, 40)])
def test_footprint_paths(name, w, h, n, scale):
    ctx = sb.GpuContext(0)
    scene, beam, cam = workload(name, w, h)
    f = sb.GpuPhotonFilm(ctx, scene, cam, beam, w, h, n, 11, 9.0, sb.VolWeights(), estimator=sb.BEAM, scale_log2=scale)
    f.trace_and_resolve(n, 11)
    whole = f.read_raw()
    p = oracle.vol_params(w, h, 11, 0.5, 0.06, 0.5, 9.0)
    ref = oracle.render_beam(oscene(scene), ocam(cam), obeam(beam), p, 0, n)
    assert ref.sum() > 0 and rel_l1(f.accum(), ref) < 1e-4
    f.clear_film()
    cuts = sorted({0, n // 3, n // 3 + n % 2, n})
    for a, b in zip(cuts, cuts[1:]):
        f.dispatch_photons(a, b, 11)
    assert np.array_equal(f.read_raw(), whole)
    f.close()
    ctx.close()


@pytest.mark.parametrize("bins,w,h", [(1, 64, 48), (31, 333, 187), (64, 900, 800)])
def test_spectral_windows_hold_one_bin(bins, w, h):
    """A spectral film's bins add up to the one-bin film of the same photons
    within the rounding of one quantum per deposit and bin."""
    ctx = sb.GpuContext(0)
    scene, beam, cam = workload("dsotm", w, h)
    n, films = 60, []
    for b in (1, bins):
        f = sb.GpuPhotonFilm(ctx, scene, cam, beam, w, h, n, 3, 9.0, sb.VolWeights(), estimator=sb.BEAM, bins=b)
        f.trace_and_resolve(n, 3)
        films.append(f.read_raw().sum(axis=2))
        f.close()
    assert films[0].sum() > 0 and np.array_equal(films[0], films[1])
    ctx.close()
