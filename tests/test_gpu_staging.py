"""Large pageable arrays in and out through the staging buffers: results equal
to those of small pieces (which take the plain copies), for sizes around the
pieces and with two threads at once (one finds the buffers in use)."""

import mmap
import threading
import time

import numpy as np
import pytest

from crest_b200 import _lib, _native, core

pytestmark = pytest.mark.gpu

D = 600


def chunk(n, seed):
    rng = np.random.default_rng(seed)
    per = 300
    idx = np.sort(rng.random((n, D)).argpartition(per - 1, axis=1)[:, :per], axis=1).astype(np.uint32).ravel()
    val = rng.integers(1, 6, len(idx)).astype(np.float32)
    return idx, val, np.arange(n + 1, dtype=np.int64) * per


def sums(idx, val, indptr, n, cuts):
    """Per (group, gene) sums over the chunks between `cuts`, raw counts: exact in any order."""
    gm = np.arange(D, dtype=np.int32)
    cm = np.arange(n, dtype=np.int64)
    grp = (np.arange(n) % 700).astype(np.uint32)
    out = [np.zeros((700, D)) for _ in range(3)]
    for a, b in zip(cuts[:-1], cuts[1:]):
        lo, hi = int(indptr[a]), int(indptr[b])
        _native.group_gene_sums(idx[lo:hi], val[lo:hi], cm, gm, 0.0, False, None, np.ascontiguousarray(indptr[a:b + 1]),
                                a, grp, *out)
    return out


@pytest.mark.parametrize("n", [1747, 1748, 7000])  # 2,096,400 and 2,097,600 bytes an array; 8.4 MB
def test_staged_copies_equal_plain_ones(n):
    idx, val, indptr = chunk(n, n)
    whole = sums(idx, val, indptr, n, [0, n])
    parts = sums(idx, val, indptr, n, list(range(0, n, 500)) + [n])
    for a, b in zip(whole, parts):
        assert np.array_equal(a, b)
    assert whole[2].sum() == len(idx)


def test_two_threads_share_the_buffers():
    n = 20_000
    idx, val, indptr = chunk(n, 3)
    want = np.bincount(idx, val, D)
    flag = np.zeros(D, np.bool_)
    got, errors = {}, []

    def work(t):
        try:
            for _ in range(3):
                m = core.DeviceMatrix(indptr, idx, val, D)
                o = [np.zeros(n), np.zeros(n, np.uint32), np.zeros(n), np.zeros(D, np.uint32), np.zeros(D)]
                cm, gm = np.arange(n, dtype=np.int64), np.arange(D, dtype=np.int32)
                _lib.call("crest_matrix_qc", m.handle, _lib.ptr(cm), _lib.ptr(gm), _lib.ptr(flag), n, D,
                          *[_lib.ptr(a) for a in o])
                m.close()
                got.setdefault(t, []).append(o[4])
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    th = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors
    for rows in got.values():
        assert len(rows) == 3 and all(np.array_equal(r, want) for r in rows)


def test_a_matrix_after_another_does_not_pay_for_the_buffers():
    """Lives of a matrix with large arrays (8.4 MB each, through the buffers)
    and with small ones (1.9 MB, plain copies), the fastest of ten: the large
    one's extra 13 MB take 2 to 3 ms, taking and giving back the pinned buffers
    in every life took 12 to 16 ms more."""
    took = {}
    for n in (1600, 7000):
        idx, val, indptr = chunk(n, n)
        times = []
        for _ in range(10):
            t = time.perf_counter()
            core.DeviceMatrix(indptr, idx, val, D).close()
            times.append(time.perf_counter() - t)
        took[n] = min(times)
    assert took[7000] - took[1600] < 7e-3, took


@pytest.mark.parametrize("n", [4369, 4370])  # 5,242,800 and 5,244,000 bytes an array: around 5 MB
def test_copies_in_around_their_limit(n):
    idx, val, indptr = chunk(n, n)
    whole = sums(idx, val, indptr, n, [0, n])
    parts = sums(idx, val, indptr, n, list(range(0, n, 500)) + [n])
    for a, b in zip(whole, parts):
        assert np.array_equal(a, b)
    assert whole[2].sum() == len(idx)


@pytest.mark.parametrize("n", [262_143, 262_144, 1_572_863, 1_572_864])  # 8 bytes each: around 2 and 12 MB
@pytest.mark.parametrize("offset", [0, 8, 4088])
def test_copies_out_into_new_and_warm_arrays(n, offset):
    """Sums of every cell into pages that exist, that do not, and that are half
    there, at any place in a page; bytes around them stay."""
    indptr = np.arange(n + 1, dtype=np.int64)
    val = (np.arange(n) % 1000 + 1).astype(np.float32)
    m = core.DeviceMatrix(indptr, np.zeros(n, np.uint32), val, 1)
    cm, gm, flag = np.arange(n, dtype=np.int64), np.zeros(1, np.int32), np.ones(1, np.uint8)
    for touched in (0.0, 0.4, 1.0):
        mem = [mmap.mmap(-1, 8 * n + 8192) for _ in range(2)]
        for buf in mem:
            np.frombuffer(buf, np.uint8)[:int(touched * len(buf))] = 7
        whole = [np.frombuffer(buf, np.uint8) for buf in mem]
        total, flagged = (w[offset:offset + 8 * n].view(np.float64) for w in whole)
        ngenes, gn, gt = np.zeros(n, np.uint32), np.zeros(1, np.uint32), np.zeros(1)
        _lib.call("crest_matrix_qc", m.handle, _lib.ptr(cm), _lib.ptr(gm), _lib.ptr(flag), n, 1, _lib.ptr(total),
                  _lib.ptr(ngenes), _lib.ptr(flagged), _lib.ptr(gn), _lib.ptr(gt))
        assert np.array_equal(total, val) and np.array_equal(flagged, val)
        assert gn[0] == n and gt[0] == val.sum(dtype=np.float64)
        for w in whole:
            assert np.all(w[:offset] == (7 if touched else 0))
            assert np.all(w[offset + 8 * n:] == (7 if touched == 1.0 else 0))
    m.close()


@pytest.mark.parametrize("n", [4_194_303, 4_194_304, 4_456_449])  # 4 bytes each: around 16 MB, a ragged last piece
def test_copies_in_from_untouched_pages(n):
    """Values in pages that nothing has written (zeros), a third of them
    written, and all of them: the sums over every 300th gene of 64 cells."""
    cells = 64
    indptr = np.linspace(0, n, cells + 1).astype(np.int64)
    idx = np.concatenate([np.arange(k, dtype=np.uint32) for k in np.diff(indptr)])
    n_genes = int(idx.max()) + 1
    gm = np.full(n_genes, -1, np.int32)
    gm[::300] = np.arange(len(gm[::300]))
    nv = int(gm.max()) + 1
    cm, flag = np.arange(cells, dtype=np.int64), np.zeros(nv, np.uint8)
    for written in (0.0, 0.3, 1.0):
        val = np.frombuffer(mmap.mmap(-1, 4 * n), np.float32)
        val[:int(written * n)] = np.arange(int(written * n)) % 97 + 1
        m = core.DeviceMatrix(indptr, idx, val, n_genes)
        total, ngenes, flagged = np.zeros(cells), np.zeros(cells, np.uint32), np.zeros(cells)
        gn, gt = np.zeros(nv, np.uint32), np.zeros(nv)
        _lib.call("crest_matrix_qc", m.handle, _lib.ptr(cm), _lib.ptr(gm), _lib.ptr(flag), cells, nv, _lib.ptr(total),
                  _lib.ptr(ngenes), _lib.ptr(flagged), _lib.ptr(gn), _lib.ptr(gt))
        m.close()
        kept = np.where(gm[idx] >= 0, val, 0.0).astype(np.float64)
        assert np.array_equal(total, np.add.reduceat(kept, indptr[:-1]))
        assert np.array_equal(gt, np.bincount(gm[idx][gm[idx] >= 0], val[gm[idx] >= 0], minlength=nv))


@pytest.mark.parametrize("d", [886, 887, 1100])  # 6,279,968 and 6,294,152 bytes: around 6 MB
@pytest.mark.parametrize("fresh", [False, True])
def test_gram_in_and_out_around_its_limit(d, fresh):
    """A Gram of whole numbers added to what the caller holds, exactly: d genes
    of 40 cells in FP64."""
    rng = np.random.default_rng(d)
    dense = rng.integers(0, 4, (40, d)).astype(np.float32)
    rows, cols = np.nonzero(dense)
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=40))]).astype(np.int64)
    start = 0.0 if fresh else 5.0
    gram = np.zeros((d, d)) if fresh else np.full((d, d), start)
    colsum = np.full(d, 3.0)
    _native.gram_accumulate(cols.astype(np.uint32), dense[rows, cols], np.arange(40, dtype=np.int64),
                            np.arange(d, dtype=np.int32), 0.0, False, None, indptr, 0, np.arange(d, dtype=np.int32),
                            gram, colsum, False, None, None, 0.0)
    want = dense.astype(np.float64).T @ dense.astype(np.float64) + start
    iu = np.triu_indices(d)
    assert np.array_equal(gram[iu], want[iu])
    assert np.all(gram[np.tril_indices(d, -1)] == start)
    assert np.array_equal(colsum, dense.sum(0, dtype=np.float64) + 3.0)
