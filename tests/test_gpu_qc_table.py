"""QC sums of a resident matrix at the edges of the one-table kernel
(k_sweep.cu: k_qc_table): the largest gene table and one gene more, more rows
per block than one table word can count, values on both sides of the 11-bit
split, duplicate entries (which the table must not see), and values that are
no small integers.

Bar: all results are integers (or f64 sums of integers below 2^53), so they
equal the oracle exactly; with other values the per-cell sums are in entry
order (equal) and the per-gene sums within 1e-13."""

import numpy as np
import pytest

import oracle
from crest_b200 import _lib, core

pytestmark = pytest.mark.gpu


def both(indptr, idx, val, n_genes, gm=None, cm=None):
    n = len(indptr) - 1
    cm = np.arange(n, dtype=np.int64) if cm is None else cm
    gm = np.arange(n_genes, dtype=np.int32) if gm is None else gm
    nr, nv = int(cm.max()) + 1, int(gm.max()) + 1
    flag = np.zeros(nv, np.bool_)
    flag[::7] = True

    def empty():
        return [np.zeros(nr), np.zeros(nr, np.uint32), np.zeros(nr), np.zeros(nv, np.uint32), np.zeros(nv)]

    m = core.DeviceMatrix(indptr, idx, val, n_genes, "device")
    got, ref = empty(), empty()
    _lib.call("crest_matrix_qc", m.handle, _lib.ptr(cm), _lib.ptr(gm), _lib.ptr(flag.view(np.uint8)), nr, nv,
              *[_lib.ptr(a) for a in got])
    m.close()
    oracle.qc(idx, val, cm, gm, 0.0, False, None, indptr, 0, flag, *ref)
    return got, ref


def rows(n, n_genes, per_row, seed):
    rng = np.random.default_rng(seed)
    nnz = rng.integers(0, per_row + 1, n)
    indptr = np.concatenate([[0], np.cumsum(nnz)]).astype(np.int64)
    idx = np.concatenate([np.sort(rng.choice(n_genes, k, replace=False)) for k in nnz] + [np.zeros(0)])
    return indptr, idx.astype(np.uint32), rng.integers(1, 9, len(idx)).astype(np.float32)


@pytest.mark.parametrize("n_genes", [1, 31, 33, 46_479, 46_480])
@pytest.mark.parametrize("n", [1, 149, 700])
def test_gene_counts(n_genes, n):
    indptr, idx, val = rows(n, n_genes, min(n_genes, 700), n_genes)
    idx[indptr[1:][np.diff(indptr) > 0] - 1] = n_genes - 1  # the last gene wherever a row ends
    for a, b in zip(*both(indptr, idx, val, n_genes)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("value", [2047.0, 2048.0, 4095.0, 16777215.0])
def test_rows_past_one_word(value):
    """One gene in every row of more rows than 148 blocks of 1023 hold, each
    with the value: the count and the sum of a word at their limits."""
    n = 148 * 1023 + 149
    idx = np.tile(np.array([3, 4], np.uint32), n)
    val = np.tile(np.array([value, 1.0], np.float32), n)
    for a, b in zip(*both(np.arange(0, 2 * n + 1, 2, dtype=np.int64), idx, val, 40)):
        assert np.array_equal(a, b)


def test_dense_row_and_values():
    """A row of every gene (the longest lane sums) beside rows of zeros, a
    negative zero and values around the split; dropped genes and cells."""
    n_genes = 46_000
    rng = np.random.default_rng(0)
    idx = np.concatenate([np.arange(n_genes), np.arange(0, 700, 7)]).astype(np.uint32)
    val = np.concatenate([np.full(n_genes, 2047.0), rng.choice([0.0, -0.0, 2047, 2048, 2049, 70000, 16777215], 100)])
    indptr = np.array([0, 0, n_genes, n_genes + 100], np.int64)
    gm = np.arange(n_genes, dtype=np.int32)
    gm[5::9] = -1
    gm[gm >= 0] = np.arange((gm >= 0).sum())
    for cm in (np.array([0, 1, 2], np.int64), np.array([0, -1, 1], np.int64), np.array([1, 0, 0], np.int64)):
        for a, b in zip(*both(indptr, idx, val.astype(np.float32), n_genes, gm, cm)):
            assert np.array_equal(a, b)


def test_duplicate_entries():
    """A gene stored 5000 times in one row would wrap a word's count."""
    idx = np.concatenate([np.full(5000, 2), [7, 9], [2, 2, 3]]).astype(np.uint32)
    indptr = np.array([0, 5002, 5005], np.int64)
    for a, b in zip(*both(indptr, idx, np.full(len(idx), 1500.0, np.float32), 12)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("odd", [0.5, 2047.75, -3.0, 3e7])
def test_other_values(odd):
    indptr, idx, val = rows(300, 900, 200, 5)
    val[len(val) // 2] = odd
    got, ref = both(indptr, idx, val, 900)
    for a, b in zip(got[:4], ref[:4]):
        assert np.array_equal(a, b)
    np.testing.assert_allclose(got[4], ref[4], rtol=1e-13)


@pytest.mark.parametrize("n", [60, 40_000])
@pytest.mark.parametrize("share,kernel", [(0.0, "qc_csr"), (0.01, "qc_csr"), (0.04, "qc_ranges_csr"), (1.0, "qc_ranges_csr")])
def test_large_values_take_the_ranges(n, share, kernel):
    """The table up to 2.8 % of values above 2047 at 1,000 genes, the gene ranges
    beyond (a sample of up to 65,536 values decides, so shares to either side)."""
    indptr, idx, val = rows(n, 1000, 200, 3)
    every = int(1 / share) if share else 0
    if every:
        val[::every] = 5000.0
    _lib.profile_enable(True)
    got, ref = both(indptr, idx, val, 1000)
    ran = _lib.profile_table()
    _lib.profile_enable(False)
    assert kernel in ran and {"qc_csr", "qc_ranges_csr"} & set(ran) == {kernel}
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
