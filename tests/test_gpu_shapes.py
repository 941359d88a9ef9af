"""Kernels at the sizes where their tiling can go wrong (edges of tiles,
remainders, the smallest and largest of a range), against the FP64 oracle.

Error bounds are derived per test from the longest chain of roundings of the
type, before any run."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# A sum of weighted terms (weights summing to one) is a chain of at most 128
# roundings per thread, then FP64; the weight itself holds at most 4 roundings.
# 256 eps of the terms' root-mean-square scale bounds both.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d", [(1, 1), (2, 3), (63, 4), (64, 5), (65, 16), (127, 17), (128, 8), (129, 24), (1000, 33),
                                 (4097, 64), (20011, 63), (30001, 2)])
def test_native_moments_shapes(issm, orc, cuda, dtype, n, d):
    rng = np.random.default_rng(1000 * d + n)
    X = (rng.normal(size=(n, d)) * (1.0 + rng.random(d)) + 3.0 * rng.normal(size=d)).astype(dtype)
    lw = (rng.normal(size=n) - 7.0).astype(dtype)
    if n > 2:
        lw[rng.integers(0, n, size=n // 8)] = -np.inf  # samples of zero weight
        lw[0] = -6.0
    tx, tl = torch.tensor(X, device=cuda), torch.tensor(lw, device=cuda)
    shift = rng.normal(size=d)
    mean, cov = issm.ops.weighted_moments(tx, tl, issm.ops.logweight_summary(tl), torch.tensor(shift, device=cuda))
    em, ec, _ = orc.weighted_moments(X.astype(np.float64).reshape(-1), d, lw.astype(np.float64))
    bound = 256 * float(np.finfo(dtype).eps)
    w = np.exp(lw.astype(np.float64) - lw.max())
    w /= w.sum()
    sd = np.sqrt(np.diag(ec).reshape(-1))
    spread = np.sqrt(w @ (X.astype(np.float64) - shift) ** 2) + np.abs(shift)
    assert np.all(np.abs(mean.cpu().numpy() - em) <= bound * spread)
    # the pass centres on the computed mean, rounded: its error enters squared
    scale = np.outer(sd, sd) + bound * np.outer(spread, spread) + np.finfo(np.float64).tiny
    assert np.all(np.abs(cov.cpu().numpy() - ec.reshape(d, d)) <= bound * scale)
    assert np.array_equal(cov.cpu().numpy(), cov.cpu().numpy().T)
