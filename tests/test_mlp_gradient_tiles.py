"""The gradient kernel at the edges of its tiles: one sample, a tile of 64 and its neighbours,
two tiles per CTA, more tiles than the CTAs take in one round, against the FP64 oracle.

Tolerance: a weight's gradient is a sum over samples of products that pass through at most
three FP32 dot products of length 64 and the sum itself (64 terms, then tiles and CTAs), each
within a few hundred roundings of 6e-8: 5e-5 of the largest gradient covers it."""
import numpy as np
import pytest

from oracle import mlp as om


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 37889, 90001])
def test_gradient_tiles(pkg, n):
    rng = np.random.default_rng(n)
    p = (pkg.mlp_init(5).astype(np.float64) + rng.normal(0, 0.05, om.NPARAM)).astype(np.float32)
    x = rng.uniform(-1, 1, (n, om.NIN)).astype(np.float32)
    t = rng.normal(0, 1, (n, om.NOUT)).astype(np.float32)
    loss, grad = pkg.mlp_gradient(p, x, t)
    lref, gref = om.loss_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - lref) <= 5e-5 * abs(lref)
    for a, b in zip(om.unpack(grad), om.unpack(gref)):
        assert np.max(np.abs(a - b)) <= 5e-5 * np.max(np.abs(gref))
