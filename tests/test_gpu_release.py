"""Freed matrices and plans give back all the device memory they held (the
library's own count, crest_memory_stats)."""

import threading

import numpy as np
import pandas as pd
import pytest

import crest_b200 as cb
from crest_b200 import _lib, core
from crest_b200.tl import PcaPlan

pytestmark = pytest.mark.gpu


def build(seed):
    rng = np.random.default_rng(seed)
    n, g, per = 4000, 900, 150
    idx = np.sort(rng.random((n, g)).argpartition(per - 1, axis=1)[:, :per], axis=1).astype(np.uint32).ravel()
    val = rng.integers(1, 9, len(idx)).astype(np.float32)
    return cb.BioFrame.from_csr(np.arange(n + 1, dtype=np.int64) * per, idx, val, g,
                                var=pd.DataFrame({"gene_name": [f"G{i}" for i in range(g)]}))


def one_life(seed, precision):
    bf = build(seed)
    cb.pp.calculate_qc_metrics(bf)
    cb.pp.normalize_total(bf, 1e4)
    cb.pp.log1p(bf)
    cb.pp.highly_variable_genes(bf, n_top_genes=300)
    cb.pp.scale(bf)
    cb.tl.pca(bf, n_comps=20, gram_precision=precision)
    cb.pp.group_gene_sums(bf, (np.arange(bf.n_obs) % 5).astype(np.uint32), 5)
    bf.store._dev.close()


@pytest.mark.parametrize("precision", ["bf16x3", "fp32", "fp64"])
def test_a_matrix_and_its_plans_leave_nothing(precision):
    one_life(0, precision)  # the solver's and the per-chunk workspaces stay
    before = _lib.memory_stats()[0]
    for seed in (1, 2):
        one_life(seed, precision)
    assert _lib.memory_stats()[0] == before


def test_unused_objects_leave_nothing():
    m = core.DeviceMatrix(np.array([0, 1]), np.array([0]), np.array([1.0]), 3)
    p = PcaPlan(50)
    m.close()
    p.close()
    before = _lib.memory_stats()[0]
    m = core.DeviceMatrix(np.array([0, 1]), np.array([0]), np.array([1.0]), 3)
    p = PcaPlan(50)
    m.close()
    p.close()
    assert _lib.memory_stats()[0] == before


def pass_over(m, n, g, d, precision, seed, keep=None):
    """One Gram pass and solve of d columns; the Gram and the leading variances."""
    rng = np.random.default_rng(seed)
    sub = np.full(g, -1, np.int32)
    sub[np.sort(rng.choice(g, d, replace=False))] = np.arange(d, dtype=np.int32)
    cm, gm = np.arange(n, dtype=np.int64), np.arange(g, dtype=np.int32)
    p = PcaPlan(d, precision)
    scale = _lib.Scale(0, None, None, 0.0)
    p.accumulate(m, cm, gm, 1e4, True, sub, g, scale)
    gram = np.triu(p.gram())
    p.solve(n, 5)
    v = p.results()[0]
    if keep is not None:
        keep.append(p)
    else:
        p.close()
    return gram, v


def matrix(n, g, per, seed):
    rng = np.random.default_rng(seed)
    idx = np.sort(rng.random((n, g)).argpartition(per - 1, axis=1)[:, :per], axis=1).astype(np.uint32).ravel()
    return core.DeviceMatrix(np.arange(n + 1, dtype=np.int64) * per, idx,
                             rng.integers(1, 9, len(idx)).astype(np.float32), g)


def test_matrices_share_one_tile():
    """Passes over several matrices that stay alive hold one Gram tile in all
    (d = 700 in FP64: 8,000 cells x 768 x 8 bytes = 49 MB), the widest so far;
    the last matrix gives it back."""
    n, g, per = 8000, 900, 40
    ms = [matrix(n, g, per, s) for s in range(3)]
    pass_over(ms[0], n, g, 300, "fp64", 0)
    held = [_lib.memory_stats()[0]]
    for m in ms:
        pass_over(m, n, g, 700, "fp64", 1)
        held.append(_lib.memory_stats()[0])
    tile = 8000 * 768 * 8
    assert held[1] - held[0] >= 8000 * (768 - 384) * 8
    assert held[2] - held[1] < tile / 2 and held[3] - held[2] < tile / 2  # their compact forms only
    for m in ms:
        m.close()
    assert _lib.memory_stats()[0] <= held[0] - 8000 * 384 * 8


def test_plans_of_other_shapes_in_turn():
    """Plans of different widths and precisions in turn over one matrix, alive
    together, each as over a matrix of its own."""
    n, g, per = 3001, 500, 60
    shapes = [(300, "fp64"), (70, "bf16x3"), (301, "fp32"), (400, "bf16x3"), (33, "fp64"), (300, "fp64")]
    alone = []
    for i, (d, precision) in enumerate(shapes):
        m = matrix(n, g, per, 4)
        alone.append(pass_over(m, n, g, d, precision, i))
        m.close()
    m, plans = matrix(n, g, per, 4), []
    for i, (d, precision) in enumerate(shapes):
        gram, v = pass_over(m, n, g, d, precision, i, plans)
        assert np.array_equal(gram, alone[i][0])
        assert np.array_equal(v, alone[i][1])
    for p in plans:
        p.close()
    m.close()


def test_passes_of_several_threads():
    """Passes over different matrices in several threads: the tile is lent to
    one of them at a time."""
    n, g, per, d = 20_000, 600, 50, 400
    ms = [matrix(n, g, per, s) for s in range(4)]
    alone = [pass_over(m, n, g, d, "bf16x3", 7) for m in ms]
    got = [[] for _ in ms]

    def work(i):
        for _ in range(6):
            got[i].append(pass_over(ms[i], n, g, d, "bf16x3", 7))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        assert len(got[i]) == 6
        for gram, v in got[i]:
            assert np.array_equal(gram, alone[i][0])
            np.testing.assert_allclose(v, alone[i][1], rtol=1e-12)
    for m in ms:
        m.close()
