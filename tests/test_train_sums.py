"""The parameter gradients of a batch of many tiles per CTA. Every point of the batch is the same, so
the gradient is that of one point, every term of a sum is of one sign, and the roundings of the
sums are biased: a sum of n terms one after the other can be off by n * 6e-8.

Tolerance: the longest chain is 8 tiles of 64 points, 4194304 / (128 * 148) = 222 tiles in
28 such groups, 37 partial rows and 8 threads' sums: 585 roundings, 3.5e-5; the biases and W3 sum 8 points
per tile and thread, 1776 + 16 of them: 1.1e-4; the point's own factors (dot products of up to 112
terms) add 7e-6. 5e-5 of the tensor's largest entry for W1 and W2, 1.2e-4 for the others."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures

import oracle_mlp as om


@pytest.mark.gpu
def test_large_batch():
    B = 1 << 22
    c = fixtures.case("jet96x64sc")
    dev = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"],
                           axj.patches_from_records(c["records"], c["Nz"], c["Nr"]))
    dev.set_state(c["pv"], c["target"])
    model = axj.mlp_init(31)
    dev.mlp_set(model)
    rng = np.random.default_rng(1)
    x, t = rng.standard_normal((1, 100)).astype(np.float32), rng.standard_normal((1, 2)).astype(np.float32)
    g, loss = dev.mlp_grad(np.repeat(x, B, 0), np.repeat(t, B, 0))
    lo, go = om.loss_and_grad(model, x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - lo) <= 1.2e-4 * lo
    for k, tol in (("w1", 5e-5), ("w2", 5e-5), ("w3", 1.2e-4), ("b1", 1.2e-4), ("b2", 1.2e-4), ("b3", 1.2e-4)):
        assert np.abs(g[k] - go[k]).max() <= tol * np.abs(go[k]).max(), k
    dev.close()
