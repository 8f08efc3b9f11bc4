"""Calls at the edges of what the entry points accept: weights below zero, rays
without a direction, films so wide that 16-bit differences of their columns wrap,
films of more than 2^32 cells, films of three bins, calls larger than the memory a
context keeps.

Films are sums of exact integers, so the comparisons are of every cell."""

import numpy as np
import pytest

import spectral_b200 as sb
from spectral_b200 import specs
from spectral_b200.batch import Batch, prism_jobs
from helpers import axis_box

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
