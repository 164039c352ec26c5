"""Plain FP32 Gram: work dealt to CTAs in runs that cut tiles at any 32-cell
group.  One, a few and many 128-gene tiles, cell counts from one group to
several per CTA, odd gene counts.

Tolerance: FP32 chains of 32 products and one rounding of each input give at
most 33 x 2^-24 = 2e-6 of the sum of absolute products per element (Higham,
Accuracy and Stability, 3.1); the norm bound below uses it for the whole matrix."""

import numpy as np
import pytest

from crest_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 2), (31, 130), (64, 129), (65, 300), (1000, 128), (3000, 777), (20_000, 257)])
def test_gram_fp32_over_runs(n, d):
    rng = np.random.default_rng(n + d)
    per = min(d, 40)
    idx = np.sort(rng.random((n, d)).argpartition(per - 1, axis=1)[:, :per], axis=1).astype(np.uint32)
    val = rng.integers(1, 9, idx.shape).astype(np.float32)
    indptr = np.arange(n + 1, dtype=np.int64) * per
    mean, std = rng.uniform(0.1, 1.0, d), rng.uniform(0.5, 2.0, d)
    gram, colsum = np.zeros((d, d)), np.zeros(d)
    args = (idx.ravel(), val.ravel(), np.arange(n, dtype=np.int64), np.arange(d, dtype=np.int32), 0.0, True, None, indptr, 0)
    _native.gram_accumulate(*args, np.arange(d, dtype=np.int32), gram, colsum, True, mean, std, 10.0, precision="fp32")
    S = np.zeros((n, d))
    z = (np.log1p(val.astype(np.float64)) - mean[idx]) / std[idx]
    S[np.arange(n)[:, None], idx] = np.clip(z, -10, 10) + np.clip(mean / std, -10, 10)[idx]
    ref, size = np.triu(S.T @ S), np.abs(S).T @ np.abs(S)
    shift = np.abs(mean / std)  # the products are formed of S - shift and corrected: their size bounds the error
    size = size + np.add.outer(shift, shift) * np.abs(S).sum(0) + n * np.outer(shift, shift)
    assert np.abs(np.triu(gram) - ref).max() <= 4e-6 * size.max()
    np.testing.assert_allclose(colsum, S.sum(0), rtol=1e-6, atol=1e-6 * n)


@pytest.mark.parametrize("n,d", [(64, 2000), (192, 1500), (193, 1500), (2176, 2000), (2177, 2000), (40, 2050)])
def test_gram_fp32_of_few_cells(n, d):
    """On both sides of the line between a CTA per tile and even runs (6 groups
    of 32 cells at 1,500 genes, 68 at 2,000, on 148 SMs), and more tiles than
    SMs."""
    test_gram_fp32_over_runs(n, d)
