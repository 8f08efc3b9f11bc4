"""The film's cell order as the raw read-back sees it: every pixel and channel of
ragged films of odd channel counts, against the same photons traced into an
XYZ film's image and the oracle's film."""
import numpy as np
import pytest

import oracle
import spectral_b200 as sb
from helpers import obeam, ocam, oscene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,bins", [(1, 1, 1), (8, 8, 2), (9, 7, 3), (17, 33, 5), (64, 40, 31), (23, 24, 256)])
def test_raw_cells_are_the_oracles(w, h, bins):
    ctx = sb.GpuContext(0)
    scene, beam, cam = sb.dsotm_scene(w / h)
    n, seed = 3000, 11
    f = sb.GpuPhotonFilm(ctx, scene, cam, beam, w, h, n, seed, 14.0, sb.VolWeights(), bins=bins, haze_exact=True)
    f.trace_and_resolve(n, seed)
    raw = f.read_raw().reshape(h, w, bins).astype(np.float64)
    p = oracle.vol_params(w, h, seed, 0.5, 0.06, 0.5, 14.0, bins=bins)
    _, _, fs = oracle.render_point(oscene(scene), ocam(cam), obeam(beam), p, 0, n, f32=False, xyz=False, spec=True)
    ref = fs.reshape(h, w, bins).astype(np.float64)
    assert ref.sum() > 0 and np.array_equal(raw > 0, ref > 0)
    # the haze arithmetic is the oracle's but for CUDA's expf and powf (2 and 4 ulp of 2^-24 each)
    assert np.abs(raw - ref).sum() <= 2e-6 * ref.sum() + raw[raw > 0].size
    f.close()
    ctx.close()
