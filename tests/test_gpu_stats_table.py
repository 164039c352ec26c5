"""gene_stats of a resident matrix from the per-cell table of small counts:
counts on both sides of the table's end (8, fewer for very many cells),
values that are no counts, dropped cells and genes, gene columns of one entry
up to several 2,048-entry segments.

Bar as for the other per-gene statistics: counts exact, f64 sums within
1e-12 relative of the oracle's (each term is the same f64 value; the order of
at most 3 x 10^4 additions of like-signed terms is not fixed)."""

import numpy as np
import pytest

import oracle
from crest_b200 import _lib, core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_genes,per_cell", [(1, 40, 12), (5000, 300, 150), (300_000, 50, 4)])
@pytest.mark.parametrize("target,log", [(1e4, True), (0.0, False)])
def test_gene_stats_around_the_table(n, n_genes, per_cell, target, log):
    rng = np.random.default_rng(n)
    weight = 1.0 / (1.0 + np.arange(n_genes)) if n > 1 else np.ones(n_genes)
    rank = rng.random((n, n_genes)) ** (1.0 / weight) if n < 10_000 else rng.random((n, n_genes))
    idx = np.sort(np.argpartition(-rank, per_cell - 1, axis=1)[:, :per_cell], axis=1).astype(np.uint32).ravel()
    indptr = np.arange(n + 1, dtype=np.int64) * per_cell
    val = rng.integers(1, 13, len(idx)).astype(np.float32)
    odd = rng.random(len(idx)) < 0.05
    val[odd] = rng.choice(np.array([0.0, 0.5, 2.5, 300.0, 70000.0], np.float32), odd.sum())
    cm = np.full(n, -1, np.int64)
    keep = rng.random(n) >= 0.1
    keep[0] = True
    cm[keep] = np.arange(keep.sum())
    gm = np.arange(n_genes, dtype=np.int32)
    gm[3::7] = -1
    gm[gm >= 0] = np.arange((gm >= 0).sum(), dtype=np.int32)
    nv = int(gm.max()) + 1
    m = core.DeviceMatrix(indptr, idx, val, n_genes)
    got, ref = np.zeros((nv, 5)), np.zeros((nv, 5))
    _lib.call("crest_matrix_gene_stats", m.handle, _lib.ptr(cm), _lib.ptr(gm), float(target), int(log), nv,
              _lib.ptr(got))
    m.close()
    oracle.gene_stats(idx, val, cm, gm, target, log, None, indptr, 0, ref)
    assert np.array_equal(got[:, 4], ref[:, 4])
    np.testing.assert_allclose(got[:, :4], ref[:, :4], rtol=1e-12, atol=1e-300)


def test_gene_stats_of_a_cell_without_a_factor():
    """An infinite total under an infinite target leaves a NaN factor: the
    cell's entries count and make their genes' sums NaN, for counts inside and
    outside the table alike."""
    indptr = np.array([0, 4, 6], np.int64)
    idx = np.array([0, 1, 2, 3, 1, 3], np.uint32)
    val = np.array([np.inf, 1.0, 20.0, 2.5, 3.0, 40.0], np.float32)
    cm, gm = np.arange(2, dtype=np.int64), np.arange(5, dtype=np.int32)
    m = core.DeviceMatrix(indptr, idx, val, 5)
    got, ref = np.zeros((5, 5)), np.zeros((5, 5))
    _lib.call("crest_matrix_gene_stats", m.handle, _lib.ptr(cm), _lib.ptr(gm), np.inf, 1, 5, _lib.ptr(got))
    m.close()
    oracle.gene_stats(idx, val, cm, gm, np.inf, True, None, indptr, 0, ref)
    assert np.array_equal(got[:, 4], ref[:, 4])
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))


@pytest.mark.parametrize("n", [524_288, 524_289, 2_100_000])
def test_gene_stats_of_very_many_cells(n):
    """A table of four counts up to 524,288 cells and none above; gene columns
    that end anywhere in a warp's step.  Up to 10^6 like-signed terms a gene: the
    oracle's sums in order are within 10^6 x 2^-53 = 1.1e-10 of the exact ones,
    the segments' far closer."""
    rng = np.random.default_rng(n)
    g0 = rng.integers(0, 5, n).astype(np.uint32)
    idx = np.stack([g0, g0 + 1 + rng.integers(0, 4, n).astype(np.uint32)], 1).ravel()
    val = rng.choice(np.array([1, 1, 1, 2, 3, 0.5], np.float32), 2 * n)
    indptr = np.arange(n + 1, dtype=np.int64) * 2
    cm = np.arange(n, dtype=np.int64)
    cm[::1000] = -1
    cm[cm >= 0] = np.arange((cm >= 0).sum())
    gm = np.arange(10, dtype=np.int32)
    m = core.DeviceMatrix(indptr, idx, val, 10)
    got, ref = np.zeros((10, 5)), np.zeros((10, 5))
    _lib.call("crest_matrix_gene_stats", m.handle, _lib.ptr(cm), _lib.ptr(gm), 1e4, 1, 10, _lib.ptr(got))
    m.close()
    oracle.gene_stats(idx, val, cm, gm, 1e4, True, None, indptr, 0, ref)
    assert np.array_equal(got[:, 4], ref[:, 4])
    np.testing.assert_allclose(got[:, :4], ref[:, :4], rtol=1.2e-10)
