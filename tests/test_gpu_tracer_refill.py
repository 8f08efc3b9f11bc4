"""The camera tracer's warps at their edges: waves of fewer paths than a warp, one
pixel wide or high, claims that end inside a warp, with and without radiance under
the sky, at every number of compacted bounces: the CPU tracer's bits."""
import numpy as np
import pytest

import oracle
import spectral_b200 as sb
from helpers import axis_box, ocam, oscene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,wave_bounces", [(1, 1, 1, 0), (1, 7, 5, 1), (33, 1, 33, 2), (257, 3, 3, 8), (95, 67, 9, 1)])
@pytest.mark.parametrize("background", [0.0, 1.0])
def test_small_and_ragged_waves(w, h, spp, wave_bounces, background):
    s = sb.Scene(background=background, horizon=2.0)
    s.add_sphere((0, 0, -3), 1.0, sb.Dielectric(sb.SF11))
    s.add_solid(axis_box((-3, -2, -6), (-1.5, 2, -4)), sb.Dielectric(sb.BK7))
    cam = sb.Camera.look_at((0, 0.3, 0.5), (0, 0, -3), (0, 1, 0), 55.0, w / h)
    ctx = sb.GpuContext(0)
    t = sb.GpuTracer(ctx, s, cam, w, h, sb.D65, 0x51, max_depth=8, wave_bounces=wave_bounces)
    t.accumulate(spp)
    gpu = t.read_xyz()
    ref = oracle.tracer_accumulate(oscene(s), ocam(cam), w, h, sb.D65, 0x51, spp)
    assert np.array_equal(gpu, np.asarray(ref, np.float32).reshape(gpu.shape) / np.float32(spp))
    assert t.stats()[0] == w * h * spp
    t.close()
    ctx.close()
