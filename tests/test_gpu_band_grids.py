"""The banded IC-GN loop on grids that it is launched for, against the CPU
oracle, bit for bit.

Few windows of affine and translation warps take a block each instead
(solver_partial.cu: at most six windows per SM with 16 lanes, five with 32),
and with 16 lanes a grid of up to 20 windows per SM (quadratic 16) has one
window to a warp.  The grids below lie above the first limit, and above or
below the second: two subsets to a warp, the lanes of the one that is done
first sampling the other's window, and a warp to a subset; with a launch over
the grid and with the persistent queue, which always pairs the subsets."""

from __future__ import annotations

import functools

import numpy as np
import pytest

from live_dic_gb300 import ICGNBatch, ICGNWGPU, synthetic
from oracle import oracle as oracle_c
from oracle import reference_prep as rp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SMALL, LARGE = (400, 330), (1000, 840)


@functools.cache
def _pair(size, kind):
    w, h = size
    ref, sp = synthetic.reference_image(w, h, seed=311, device="cpu")
    strong = synthetic.affine_field(0.6, 1e-2, -1.5e-2, 1.1, 1.2e-2, -8e-3)

    def bulge(X, Y):
        u, v = strong(X - w / 2, Y - h / 2)
        return u + 1e-4 * (X - w / 2) ** 2, v - 8e-5 * (Y - h / 2) ** 2

    field = {"affine": strong, "quadratic": bulge,
             "translation": synthetic.affine_field(1.37, 0.0, 0.0, -2.21, 0.0, 0.0)}[kind]
    return ref, synthetic.deformed_image(sp, field, noise_seed=312, device="cpu")


def _packed(result):
    return np.concatenate([result.parameters, result.status[..., None], result.iterations[..., None]], -1)


CASES = [("affine", 21, 5, 16, "gaussian", SMALL), ("affine", 31, 5, 16, "uniform", SMALL),
         ("affine", 41, 5, 16, "uniform", SMALL), ("affine", 31, 10, 16, "uniform", SMALL),
         ("affine", 61, 6, 16, "gaussian", SMALL), ("affine", 16, 16, 16, "uniform", LARGE),
         ("affine", 24, 24, 16, "gaussian", LARGE), ("affine", 31, 7, 32, "uniform", SMALL),
         ("affine", 41, 7, 32, "gaussian", SMALL), ("affine", 21, 21, 32, "uniform", LARGE),
         ("translation", 15, 5, 16, "uniform", SMALL), ("translation", 49, 5, 16, "gaussian", SMALL),
         ("translation", 27, 9, 16, "gaussian", SMALL), ("translation", 17, 17, 16, "uniform", LARGE),
         ("translation", 16, 6, 32, "uniform", SMALL), ("quadratic", 21, 6, 16, "uniform", SMALL),
         ("quadratic", 41, 6, 16, "gaussian", SMALL)]


@pytest.mark.parametrize("model,subset,stride,lanes,weighting,size", CASES)
def test_banded_grids_bit_exact(model, subset, stride, lanes, weighting, size):
    ref, tgt = _pair(size, model)
    w, h = size
    gw, gh = 1 + (w - subset) // stride, 1 + (h - subset) // stride
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if model != "quadratic":
        assert gw * gh > (6 if lanes == 16 else 5) * sms
    plane, inverse, metadata = rp.reference_arrays(ref, motion_model=model, subset_size=subset, subset_stride=stride,
                                                   spatial_weighting=weighting)
    n, width = (12, 16) if model == "quadratic" else (6, 8)
    rng = np.random.default_rng(subset)
    # seeds near and far from the field: unequal iteration counts within a warp, some windows pushed off the frame
    seeds = np.zeros((gh * gw, width), np.float32)
    seeds[:, 0], seeds[:, 3] = rng.normal(0.0, 1.5, (2, gh * gw))
    active = (rng.random((gh, gw)) < 0.9).astype(np.uint32)
    coef = oracle_c.prefilter(tgt, rp.runtime_fir_taps())
    kw = dict(subset_size=subset, subset_stride=stride, model=model, lanes=lanes, tolerance=1e-4)
    with ICGNWGPU(subset_size=subset, subset_stride=stride, motion_model=model, outlier_policy="disabled",
                  solver_workgroup_size=lanes, spatial_weighting=weighting) as engine:
        engine.set_reference_arrays(w, h, plane, metadata, inverse, tolerance=1e-4)
        weights = engine.export_weights() if weighting == "gaussian" else None
        fields, seeded = [], []
        for persistent in (False, True):
            engine.set_solver_variant(lanes, persistent)
            fields.append(_packed(engine.register(tgt)))
            seeded.append(engine._register_seeded_states(tgt, seeds.reshape(gh, gw, width), active))
    expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, weights=weights, **kw)
    for got in fields:
        np.testing.assert_array_equal(got, expected.reshape(gh, gw, -1)[..., :n + 2])
    expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, weights=weights, seed_state=seeds,
                              active=active.ravel(), **kw)
    for got in seeded:
        np.testing.assert_array_equal(got[..., :n + 2], expected.reshape(gh, gw, -1)[..., :n + 2])
    assert (fields[0][..., n] > 0.5).any()
    pairs = seeded[0][..., n + 1].reshape(-1)[:gh * gw // 2 * 2].reshape(-1, 2)
    assert (pairs[:, 0] != pairs[:, 1]).any()


@pytest.mark.parametrize("subset,stride,lanes,size", [(31, 6, 16, SMALL), (31, 10, 32, SMALL), (16, 16, 16, LARGE),
                                                      (21, 21, 32, LARGE)])
def test_planes_of_a_prepared_reference(subset, stride, lanes, size):
    """A reference prepared on the GPU gives the oracle's field on its exported
    arrays, also after another of the same size: the banded loop's f, gradients
    and pixel table, overlapping windows and tiled ones."""
    ref, tgt = _pair(size, "affine")
    with ICGNWGPU(subset_size=subset, subset_stride=stride, outlier_policy="disabled",
                  solver_workgroup_size=lanes) as engine:
        for image in (np.ascontiguousarray(ref[::-1]), ref):
            engine.set_reference(image)
        got = _packed(engine.register(tgt))
        plane, inverse, metadata = engine.export_reference()
    assert got[..., 0].size > 6 * torch.cuda.get_device_properties(0).multi_processor_count
    coef = oracle_c.prefilter(tgt, rp.runtime_fir_taps())
    expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, subset_size=subset, subset_stride=stride, lanes=lanes)
    np.testing.assert_array_equal(got, expected.reshape(got.shape))


def test_batch_branches_of_banded_jobs():
    """Branches whose jobs run the banded loop, paired subsets and single ones,
    against the launch over jobs of every kind."""
    jobs = [("affine", 31, 5, SMALL), ("translation", 21, 5, SMALL), ("quadratic", 21, 6, SMALL), ("affine", 16, 16, LARGE),
            ("affine", 31, 9, SMALL)]
    with ICGNBatch() as batch:
        targets = []
        for model, subset, stride, size in jobs:
            ref, tgt = _pair(size, model)
            batch.add(ref, motion_model=model, subset_size=subset, subset_stride=stride)
            targets.append(tgt)
        batch.set_variant(16, "single", 32)
        expected = [_packed(r) for r in batch.register(targets)]
        batch.set_variant(16, "single")
        for got, want in zip(batch.register(targets), expected, strict=True):
            np.testing.assert_array_equal(_packed(got), want)
