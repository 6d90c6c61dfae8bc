"""The fused training pass of the learned sensor's network at the edges of its tiles of 128
points and of its grid of one CTA per SM, against the NumPy oracle in 64 bits, and its
determinism.

Tolerance: a gradient entry sums, per point, products whose factors carry a few FP32
roundings of 112- and 64-term dot products (each below 112 * 6e-8 of its terms' magnitude
sum, under 1e-6 of the largest entry at these sizes), in partial sums of at most 5 * 64 points
per accumulator: 320 * 6e-8 = 2e-5 of the magnitude sum; 1e-4 of the tensor's largest entry,
as for the unfused pass."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures

import oracle_mlp as om

pytestmark = pytest.mark.gpu


def _solver():
    c = fixtures.case("jet96x64sc")
    s = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"],
                         axj.patches_from_records(c["records"], c["Nz"], c["Nr"]))
    s.set_state(c["pv"], c["target"])
    return s


def _model(seed):
    m = axj.mlp_init(seed)
    m["out_scale"] = np.array([2e-3, 5e-4], dtype=np.float32)
    return m


@pytest.mark.parametrize("B", [1, 2, 127, 128, 129, 148 * 128, 148 * 128 + 1, 5 * 148 * 128 - 77])
def test_gradients_at_tile_edges(B):
    dev = _solver()
    model = _model(31)
    dev.mlp_set(model)
    rng = np.random.default_rng(B)
    X = rng.standard_normal((B, 100)).astype(np.float32)
    T = rng.standard_normal((B, 2)).astype(np.float32)
    g, loss = dev.mlp_grad(X, T)
    lo, go = om.loss_and_grad(model, X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    for k in ("w1", "b1", "w2", "b2", "w3", "b3"):
        assert np.abs(g[k] - go[k]).max() <= 1e-4 * np.abs(go[k]).max(), k
    dev.close()


@pytest.mark.parametrize("B", [100, 129, 4096])
def test_sampled_steps_equal_given_batches_and_repeat(B):
    """Three training steps: each draws the batch that dataset_sample returns for it (the
    losses are those of the given batches on the same weights), and a repeated run gives the
    same bits."""
    dev = _solver()
    dev.dataset_reserve(2)
    for _ in range(2):
        dev.run(3)
        dev.dataset_add()
    runs = []
    for _ in range(2):
        dev.mlp_set(_model(9))
        loss = dev.mlp_train(steps=3, batch=B, seed=5, fit_normalization=1)
        runs.append((loss, dev.mlp_get()))
    assert np.array_equal(runs[0][0], runs[1][0])
    for k in runs[0][1]:
        assert np.array_equal(runs[0][1][k], runs[1][1][k]), k
    first = _model(9)
    for k in ("feat_mean", "feat_scale", "out_scale"):
        first[k] = runs[0][1][k]
    dev.mlp_set(first)
    X, T = dev.dataset_sample(B, 5, 0)
    lo, _ = om.loss_and_grad(first, X.astype(np.float64), T.astype(np.float64))
    assert abs(runs[0][0][0] - lo) <= 1e-5 * abs(lo)
    dev.close()
