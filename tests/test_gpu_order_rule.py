"""The wavelength-ordered dispatch on both sides of its rule, and forced on and off:
the same film bits."""
import numpy as np
import pytest

import spectral_b200 as sb
from spectral_b200 import scenes, specs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,w,h,bins,n", [
    ("rainbow", 1280, 720, 64, 900_000),   # film, beam and samples all beyond L2
    ("rainbow", 1280, 720, 64, 300_000),   # too few samples
    ("prism", 1024, 640, 64, 900_000)])    # a narrow beam
def test_order_keeps_the_film(monkeypatch, name, w, h, bins, n):
    d = {"prism": specs.prism_scene, "rainbow": specs.rainbow_scene}[name]()
    ctx, sums = sb.GpuContext(0), []
    for order in ("1", "0", "2"):
        monkeypatch.setenv("SPECTRAL_CUDA_ORDER", order)
        f = sb.GpuPhotonFilm(ctx, scenes.scene_from_spec(d), sb.Camera.look_at(*d["camera"], w / h),
                             sb.Beam(*d["beam"]), w, h, n, 5, 8.0, sb.VolWeights(0.1, 0.05, 0.0), bins=bins)
        f.trace_and_resolve(n, 5)
        sums.append(f.read_raw())
        f.close()
    assert sums[0].sum() > 0 and np.array_equal(sums[0], sums[1]) and np.array_equal(sums[0], sums[2])
    ctx.close()
