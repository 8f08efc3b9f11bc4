"""The 99.7th percentile exposure over images of one pixel to many CTAs, all black,
mostly black and all lit: the k-th smallest luminance, as a sort finds it."""
import numpy as np
import pytest

import spectral_b200 as sb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n,lit", [(1, 1, 0, False), (1, 1, 500, False), (3, 5, 300, True), (32, 32, 40_000, False),
                                       (333, 187, 200_000, False), (64, 48, 20_000, True), (800, 600, 100_000, True)])
def test_percentile_is_the_sorted_value(w, h, n, lit):
    ctx = sb.GpuContext(0)
    scene, beam, cam = sb.dsotm_scene(w / h)
    f = sb.GpuPhotonFilm(ctx, scene, cam, beam, w, h, max(n, 1), 3, 14.0, sb.VolWeights())
    if n:
        f.trace_and_resolve(n, 3)
    if lit:
        f.recompute_surface(cam)
    y = f.accum().reshape(-1, 3)[:, 1] + f.surface().reshape(-1, 3)[:, 1]
    y = np.sort(np.maximum(y, np.float32(0)))
    k = min(int(np.float32(w * h) * np.float32(0.997)), w * h - 1)
    assert f.auto_expose_p997() == np.float32(1) / max(y[k], np.float32(1e-9))
    assert f.auto_expose_p997() == np.float32(1) / max(y[k], np.float32(1e-9))  # the scratch is reusable
    f.close()
    ctx.close()
