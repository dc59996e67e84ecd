"""The banded IC-GN loop (solver_band.cuh) against the CPU oracle, bit for bit.

Complete B-spline windows with 16 or 32 lanes are sampled by vertical runs
into shared memory and accumulated from there in the reference's order.  The
sizes below are where that can go wrong: runs of every length modulo the
ring's four rows, one to five bands (the last one overlapping the band above
it), windows narrower than the lanes, one more column than the lanes walk at
once, tiled grids (whose plane is centred per window), Gaussian weights, and
warps that leave the frame, cross tap rows and columns, bulge over the border
(quadratic) and stop after different iteration counts within a warp."""

from __future__ import annotations

import numpy as np
import pytest

from live_dic_gb300 import ICGNWGPU, synthetic
from oracle import oracle as oracle_c
from oracle import reference_prep as rp

pytestmark = pytest.mark.gpu

W, H = 203, 171


@pytest.fixture(scope="module")
def pairs():
    ref, sp = synthetic.reference_image(W, H, seed=301, device="cpu")
    strong = synthetic.affine_field(0.6, 2e-2, -3e-2, 1.1, 2.5e-2, -1.5e-2)

    def bulge(X, Y):
        u, v = strong(X - W / 2, Y - H / 2)
        return u + 3e-4 * (X - W / 2) ** 2, v - 2e-4 * (Y - H / 2) ** 2

    shift = synthetic.affine_field(1.37, 0.0, 0.0, -2.21, 0.0, 0.0)
    return ref, {name: synthetic.deformed_image(sp, field, noise_seed=302, device="cpu")
                 for name, field in (("affine", strong), ("quadratic", bulge), ("translation", shift))}


CASES = [("affine", 31, 8, 16, "uniform"), ("affine", 29, 14, 16, "uniform"), ("affine", 27, 9, 16, "gaussian"),
         ("affine", 21, 7, 16, "uniform"), ("affine", 41, 13, 16, "uniform"), ("affine", 16, 16, 16, "uniform"),
         ("affine", 61, 20, 16, "gaussian"), ("affine", 32, 11, 32, "uniform"), ("affine", 41, 41, 32, "gaussian"),
         ("affine", 25, 12, 32, "uniform"), ("quadratic", 41, 10, 16, "uniform"), ("quadratic", 13, 6, 16, "uniform"),
         ("quadratic", 33, 11, 16, "gaussian"), ("quadratic", 65, 21, 16, "uniform"),
         ("quadratic", 21, 21, 32, "uniform"), ("translation", 15, 5, 16, "uniform"),
         ("translation", 17, 17, 16, "gaussian"), ("translation", 49, 24, 16, "uniform"),
         ("translation", 16, 8, 32, "uniform"), ("translation", 81, 30, 32, "uniform")]


@pytest.mark.parametrize("model,size,stride,lanes,weighting", CASES)
def test_banded_loop_bit_exact(pairs, model, size, stride, lanes, weighting):
    ref, targets = pairs
    tgt = targets[model]
    plane, inverse, metadata = rp.reference_arrays(ref, motion_model=model, subset_size=size, subset_stride=stride,
                                                   spatial_weighting=weighting)
    gw, gh = 1 + (W - size) // stride, 1 + (H - size) // stride
    width = 16 if model == "quadratic" else 8
    n = 12 if model == "quadratic" else 6
    rng = np.random.default_rng(size)
    # seeds near and far from the field: unequal iteration counts, some windows pushed off the frame
    seeds = np.zeros((gh * gw, width), np.float32)
    seeds[:, 0], seeds[:, 3] = rng.normal(0.0, 1.5, (2, gh * gw))
    coef = oracle_c.prefilter(tgt, rp.runtime_fir_taps())
    kw = dict(subset_size=size, subset_stride=stride, model=model, lanes=lanes, tolerance=1e-4)
    with ICGNWGPU(subset_size=size, subset_stride=stride, motion_model=model, outlier_policy="disabled",
                  solver_workgroup_size=lanes, spatial_weighting=weighting) as engine:
        engine.set_reference_arrays(W, H, plane, metadata, inverse, tolerance=1e-4)
        weights = engine.export_weights() if weighting == "gaussian" else None
        result = engine.register(tgt)
        got = np.concatenate([result.parameters, result.status[..., None], result.iterations[..., None]], -1)
        seeded = engine._register_seeded_states(tgt, seeds.reshape(gh, gw, width), np.ones((gh, gw), np.uint32))
    expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, weights=weights, **kw)
    np.testing.assert_array_equal(got, expected.reshape(gh, gw, -1)[..., :n + 2])
    expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, weights=weights, seed_state=seeds,
                              active=np.ones(gh * gw, np.uint32), **kw)
    np.testing.assert_array_equal(seeded[..., :n + 2], expected.reshape(gh, gw, -1)[..., :n + 2])
    assert (got[..., n] > 0.5).any() and len(np.unique(got[..., n + 1])) > 1


@pytest.mark.parametrize("lanes", [16, 32])
def test_prepared_plane_copies(pairs, lanes):
    """A reference prepared on the GPU (overlapping and tiled windows) gives the oracle's field on its exported
    arrays, also after another reference of the same size replaced it."""
    ref, targets = pairs
    tgt = targets["affine"]
    coef = oracle_c.prefilter(tgt, rp.runtime_fir_taps())
    for size, stride in ((31, 10), (21, 21)):
        with ICGNWGPU(subset_size=size, subset_stride=stride, outlier_policy="disabled",
                      solver_workgroup_size=lanes) as engine:
            for image in (np.ascontiguousarray(ref[::-1]), ref):
                engine.set_reference(image)
            result = engine.register(tgt)
            plane, inverse, metadata = engine.export_reference()
        got = np.concatenate([result.parameters, result.status[..., None], result.iterations[..., None]], -1)
        expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, subset_size=size, subset_stride=stride,
                                  lanes=lanes)
        np.testing.assert_array_equal(got, expected.reshape(got.shape))


@pytest.mark.parametrize("size,stride", [(16, 16), (21, 10), (31, 8), (33, 11), (41, 13), (63, 20)])
def test_final_zncc_by_bands(size, stride):
    """The final ZNCC's band sampling against the oracle: a shift of about 2 px puts the first windows' corners
    within a sixteenth of a pixel of the bound, on either side of it."""
    ref, sp = synthetic.reference_image(W, H, seed=303, device="cpu")
    tgt = synthetic.deformed_image(sp, synthetic.affine_field(2.0, 4e-4, -3e-4, 2.0, 2e-4, 5e-4), noise_seed=304,
                                   device="cpu")
    with ICGNWGPU(subset_size=size, subset_stride=stride) as engine:
        engine.set_reference(ref)
        result = engine.register_seeded(tgt, np.tile(np.array([2, 0, 0, 2, 0, 0], np.float32),
                                                     (engine.grid_height, engine.grid_width, 1)),
                                        np.ones((engine.grid_height, engine.grid_width), bool), include_zncc=True)
        plane, _, _ = engine.export_reference()
    state = np.concatenate([result.parameters, result.status[..., None], result.iterations[..., None]], -1)
    coef = oracle_c.prefilter(tgt, rp.runtime_fir_taps())
    expected = oracle_c.final_zncc(tgt, coef, plane, state.reshape(-1, 8), subset_size=size, subset_stride=stride)
    expected[expected < -1.0] = np.nan
    np.testing.assert_array_equal(result.zncc.ravel(), expected)
    assert np.isfinite(expected).any()


@pytest.mark.parametrize("policy", ["replace", "flag"])
def test_quadratic_outliers_bit_exact(pairs, policy):
    """Planted outliers, rejected neighbours, infinities and NaNs in quadratic states."""
    ref, _ = pairs
    plane, inverse, metadata = rp.reference_arrays(ref, motion_model="quadratic", subset_size=21, subset_stride=10)
    gw, gh = 1 + (W - 21) // 10, 1 + (H - 21) // 10
    rng = np.random.default_rng(12)
    state = np.zeros((gh, gw, 16), np.float32)
    state[..., :12] = rng.normal(0, 1e-3, (gh, gw, 12))
    state[..., 0] += 0.3 + rng.normal(0, 0.05, (gh, gw))
    state[..., 3] += rng.normal(0, 0.05, (gh, gw))
    state[..., 12] = rng.choice(np.array([1.0] * 12 + [0.0, -1.0], np.float32), (gh, gw))
    state[..., 13] = 3.0
    state[rng.random((gh, gw)) < 0.1, 0] += 2.5
    state[2, 3, 0] = np.inf
    state[9, 11, 4] = np.nan
    state[12, 4, 3] = np.nan
    with ICGNWGPU(subset_size=21, subset_stride=10, motion_model="quadratic", outlier_policy=policy) as engine:
        engine.set_reference_arrays(W, H, plane, metadata, inverse)
        got = engine.apply_outlier_filter(state)
    expected = oracle_c.uod(state.reshape(-1, 16), metadata, grid=(gw, gh), subset_stride=10, model="quadratic",
                            policy=policy)
    np.testing.assert_array_equal(got.reshape(-1, 16), expected)
    assert (got[..., 12] == 2.0).sum() > 5


@pytest.mark.parametrize("scope", ["rejected", "all"])
@pytest.mark.parametrize("size", [3, 5])
@pytest.mark.parametrize("model", ["translation", "affine", "quadratic"])
def test_median_fields_in_registers_bit_exact(pairs, model, size, scope):
    """3x3 and 5x5 medians: rejected neighbours, grid edges, infinities, and NaNs
    (whose subsets take the general selection)."""
    ref, _ = pairs
    plane, inverse, metadata = rp.reference_arrays(ref, motion_model=model, subset_size=21, subset_stride=10)
    gw, gh = 1 + (W - 21) // 10, 1 + (H - 21) // 10
    rng = np.random.default_rng(size)
    stride, n = (16, 12) if model == "quadratic" else (8, 6)
    state = np.zeros((gh, gw, stride), np.float32)
    state[..., :n] = rng.normal(0, 1e-2, (gh, gw, n))
    if model == "translation":
        state[..., [1, 2, 4, 5]] = 0.0
    state[..., n] = rng.choice(np.array([1.0, 2.0, 1.0, 0.0, -1.0], np.float32), (gh, gw))
    state[2, 3, 0] = np.inf
    state[gh - 2, 4, 3] = -np.inf
    state[9, 11, 0] = np.nan
    with ICGNWGPU(subset_size=21, subset_stride=10, motion_model=model, outlier_policy="median",
                  median_filter_size=size, median_filter_scope=scope) as engine:
        engine.set_reference_arrays(W, H, plane, metadata, inverse)
        got = engine.apply_outlier_filter(state)
    expected = oracle_c.uod(state.reshape(-1, stride), metadata, grid=(gw, gh), subset_stride=10, model=model,
                            policy="median", median_size=size, scope_all=scope == "all")
    np.testing.assert_array_equal(got.reshape(-1, stride), expected)


@pytest.mark.parametrize("policy,size", [("replace", 3), ("flag", 3), ("median", 3), ("median", 5), ("median", 7),
                                         ("disabled", 3)])
@pytest.mark.parametrize("model", ["translation", "affine", "quadratic"])
def test_waiting_and_pipelined_calls_return_one_field(pairs, model, policy, size):
    """A waiting call's field is written to pinned memory by the outlier pass, a
    pipelined one's is copied: the same field, frame after frame."""
    ref, _ = pairs
    frames = [np.ascontiguousarray(np.roll(ref, k, 1)) for k in (1, 2, 0)]
    with ICGNWGPU(subset_size=21, subset_stride=10, motion_model=model, outlier_policy=policy,
                  median_filter_size=size) as engine:
        engine.set_reference(ref)
        waiting = [engine.register(f) for f in frames]
        for a, b in zip(waiting, engine.register_stream(frames), strict=True):
            np.testing.assert_array_equal(a.parameters, b.parameters)
            np.testing.assert_array_equal(a.status, b.status)
            np.testing.assert_array_equal(a.iterations, b.iterations)


@pytest.mark.parametrize("lanes", [16, 32])
@pytest.mark.parametrize("model,interp,weighting,subset,stride", [
    ("affine", "bspline", "uniform", 21, 11), ("affine", "bspline", "gaussian", 33, 33), ("affine", "cubic", "uniform", 15, 9),
    ("affine", "linear", "gaussian", 16, 13), ("translation", "bspline", "uniform", 41, 20),
    ("translation", "linear", "uniform", 12, 12)])
def test_few_windows_by_blocks_bit_exact(pairs, model, interp, weighting, subset, stride, lanes):
    """Launches of few windows, a block each: odd and even sides, more than one
    sampled chunk, tiled grids, windows that leave the frame, a masked reference."""
    ref, _ = pairs
    tgt = np.ascontiguousarray(np.roll(np.roll(ref, 2, 1), -1, 0))
    mask = None
    if weighting == "uniform":
        mask = np.ones(ref.shape, bool)
        mask[30:70, 40:110] = False
    with ICGNWGPU(subset_size=subset, subset_stride=stride, motion_model=model, interpolation=interp,
                  spatial_weighting=weighting, outlier_policy="disabled", solver_workgroup_size=lanes) as engine:
        engine.set_reference(ref, roi_mask=mask)
        result = engine.register(tgt)
        plane, inverse, metadata = engine.export_reference()
        coef = engine.export_coefficients() if interp == "bspline" else None
        weights = engine.export_weights() if weighting == "gaussian" else None
    assert result.status.size <= 912
    expected = oracle_c.solve(tgt, coef, plane, metadata, inverse, subset_size=subset, subset_stride=stride, model=model,
                              interpolation=interp, lanes=lanes, roi_enabled=mask is not None, weights=weights)
    got = np.concatenate([result.parameters, result.status[..., None], result.iterations[..., None]], -1)
    np.testing.assert_array_equal(got.reshape(-1, 8), expected.reshape(-1, 8))
