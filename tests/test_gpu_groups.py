"""Per (group, gene) sums (src/kernels.rs:388-442) on the GPU against the
oracle, and rank_genes_groups (t-test) through crest_b200.tl against the
golden tables of the reference's own crest/tl.py.

Tolerances: the reference sums each (group, gene) in entry order, the GPU
with atomics in no fixed order: sums within 1e-12 relative, counts exact.
Differential-expression tables: the same genes in the same order per group,
scores / log fold changes within 1e-9 relative, p-values within 1e-6
relative (scipy's Student t in both the oracle and the product)."""

import os

import numpy as np
import pandas as pd
import pytest

import crest_b200 as cb
import oracle
from crest_b200 import _lib, _native, core

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def chunks(indptr, cuts):
    for a, b in zip(cuts[:-1], cuts[1:]):
        yield a, b, int(indptr[a]), int(indptr[b])


@pytest.mark.parametrize("clip", [False, True])
@pytest.mark.parametrize("coo", [False, True])
def test_group_gene_sums_match_oracle(small_counts, clip, coo):
    indptr, indices, data, n_genes = small_counts[:4]
    n = len(indptr) - 1
    rng = np.random.default_rng(21)
    keep_c = rng.random(n) >= 0.1
    cm = np.full(n, -1, np.int64)
    cm[keep_c] = np.arange(keep_c.sum())
    keep_g = rng.random(n_genes) >= 0.2
    gm = np.full(n_genes, -1, np.int32)
    gm[keep_g] = np.arange(keep_g.sum(), dtype=np.int32)
    nr, nv, G = int(keep_c.sum()), int(keep_g.sum()), 7
    grp = rng.integers(0, G, nr).astype(np.uint32)
    grp[rng.random(nr) < 0.1] = np.iinfo(np.uint32).max  # cells without a group
    cl = rng.uniform(0.5, 3.0, (G, nv)) if clip else None
    out = [[np.zeros((G, nv)) for _ in range(3)] for _ in range(2)]
    for a, b, lo, hi in chunks(indptr, [0, 701, n]):
        g, v = indices[lo:hi], data[lo:hi]
        if coo:
            cells = np.repeat(np.arange(a, b, dtype=np.uint32), np.diff(indptr[a:b + 1]))
            args = (g, v, cm, gm, 1e4, True, cells, None, 0)
        else:
            args = (g, v, cm, gm, 1e4, True, None, np.ascontiguousarray(indptr[a:b + 1]), a)
        _native.group_gene_sums(*args, grp, *out[0], cl)
        oracle.group_gene_sums(*args, grp, *out[1], cl)
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12, atol=1e-12)
    assert np.array_equal(out[0][2], out[1][2])
    tot = [np.zeros((G, nv)), np.zeros((G, nv))]
    p = np.ascontiguousarray(indptr)
    _native.group_gene_totals(indices, data, cm, gm, 0.0, False, None, p, 0, grp, tot[0])
    oracle.group_gene_totals(indices, data, cm, gm, 0.0, False, None, p, 0, grp, tot[1])
    assert np.array_equal(tot[0], tot[1])  # raw integer counts: exact sums


def test_group_gene_sums_rejects_bad_groups(small_counts):
    indptr, indices, data, n_genes = small_counts[:4]
    n = len(indptr) - 1
    cm = np.arange(n, dtype=np.int64)
    gm = np.arange(n_genes, dtype=np.int32)
    s = [np.zeros((3, n_genes)) for _ in range(3)]
    bad = np.full(n, 3, np.uint32)
    with pytest.raises(ValueError, match="group id out of range"):
        _native.group_gene_sums(indices, data, cm, gm, 0.0, False, None, indptr, 0, bad, *s)
    with pytest.raises(ValueError, match="group_of_row"):
        _native.group_gene_sums(indices, data, cm, gm, 0.0, False, None, indptr, 0, bad[:10], *s)


@pytest.mark.parametrize("name", ["small", "pbmc3k_like"])
@pytest.mark.parametrize("store", ["csr", "triplets"])
def test_rank_genes_groups_matches_reference_golden(name, store):
    import importlib.util
    spec = importlib.util.spec_from_file_location("make_golden", os.path.join(HERE, "golden", "make_golden.py"))
    mg = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mg)
    c = mg.CASES[name]
    indptr, indices, data, n_genes, names = mg.case_input(name)
    labels = mg.case_labels(name)
    g = dict(np.load(os.path.join(HERE, "golden", f"{name}.npz")))
    var = pd.DataFrame({"gene_name": names})
    if store == "csr":
        bf = cb.BioFrame.from_csr(indptr, indices, data, n_genes, var=var)
    else:
        cells = np.repeat(np.arange(len(indptr) - 1), np.diff(indptr)).astype(np.uint32)
        bf = cb.BioFrame.from_triplets(cells, indices, data, len(indptr) - 1, n_genes, var=var)
    bf = cb.pp.filter_cells(bf, min_genes=c["min_genes"])
    bf = cb.pp.filter_genes(bf, min_cells=c["min_cells"])
    cb.pp.normalize_total(bf, 1e4)
    cb.pp.log1p(bf)
    bf.obs["cluster"] = [f"c{x}" for x in labels[bf.obs["cell_id"].to_numpy()]]
    tab = cb.tl.rank_genes_groups(bf, "cluster", method="t-test", n_genes=mg.DE_TOP)
    assert np.array_equal(tab["group"].to_numpy().astype(str), g["de_group"])
    assert np.array_equal(tab["names"].to_numpy().astype(str), g["de_names"])
    np.testing.assert_allclose(tab["scores"].to_numpy(), g["de_scores"], rtol=1e-9)
    np.testing.assert_allclose(tab["logfoldchanges"].to_numpy(), g["de_logfoldchanges"], rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(tab["pvals"].to_numpy(), g["de_pvals"], rtol=1e-6, atol=1e-300)
    np.testing.assert_allclose(tab["pvals_adj"].to_numpy(), g["de_pvals_adj"], rtol=1e-6, atol=1e-300)
    assert "rank_genes_groups" in bf.uns


@pytest.mark.parametrize("name", ["small", "pbmc3k_like"])
@pytest.mark.parametrize("store", ["csr", "triplets"])
def test_seurat_v3_matches_reference_golden(name, store):
    """seurat_v3 HVG (two GPU passes of per (batch, gene) sums of the raw
    counts, the second clipped; loess trend and ranking on the host) against
    the reference's columns: the HVG set, ranks and batch counts identical,
    means / variances within 1e-12 relative, variances_norm within 1e-9."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("make_golden", os.path.join(HERE, "golden", "make_golden.py"))
    mg = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mg)
    c = mg.CASES[name]
    indptr, indices, data, n_genes, names = mg.case_input(name)
    labels = mg.case_labels(name)
    g = dict(np.load(os.path.join(HERE, "golden", f"{name}.npz")))
    var = pd.DataFrame({"gene_name": names})
    if store == "csr":
        bf = cb.BioFrame.from_csr(indptr, indices, data, n_genes, var=var)
    else:
        cells = np.repeat(np.arange(len(indptr) - 1), np.diff(indptr)).astype(np.uint32)
        bf = cb.BioFrame.from_triplets(cells, indices, data, len(indptr) - 1, n_genes, var=var)
    bf = cb.pp.filter_cells(bf, min_genes=c["min_genes"])
    bf = cb.pp.filter_genes(bf, min_cells=c["min_cells"])
    bf.obs["batch"] = [f"b{x % 3}" for x in labels[bf.obs["cell_id"].to_numpy()]]
    for tag, key in (("v3", None), ("v3b", "batch")):
        cb.pp.highly_variable_genes(bf, flavor="seurat_v3", n_top_genes=mg.V3_TOP, batch_key=key)
        assert np.array_equal(bf.var["highly_variable"].to_numpy(), g[f"{tag}_highly_variable"])
        assert np.array_equal(bf.var["highly_variable_nbatches"].to_numpy(), g[f"{tag}_highly_variable_nbatches"])
        assert np.array_equal(bf.var["highly_variable_rank"].to_numpy(), g[f"{tag}_highly_variable_rank"],
                              equal_nan=True)
        for col in ("means", "variances"):
            np.testing.assert_allclose(bf.var[col].to_numpy(), g[f"{tag}_{col}"], rtol=1e-12)
        np.testing.assert_allclose(bf.var["variances_norm"].to_numpy(), g[f"{tag}_variances_norm"], rtol=1e-9)


def resident(m, cm, gm, target, log, grp, G, nv, cl=None):
    out = [np.zeros((G, nv)) for _ in range(3)]
    _lib.call("crest_matrix_group_gene_sums", m.handle, _lib.ptr(cm), _lib.ptr(gm), float(target), int(log), _lib.ptr(grp),
              len(grp), G, nv, _lib.ptr(cl), *[_lib.ptr(a) for a in out])
    return out


@pytest.mark.parametrize("target,log", [(1e4, True), (0.0, True), (0.0, False)])
@pytest.mark.parametrize("clip", [False, True])
def test_resident_group_sums_around_the_lane_table(target, log, clip):
    """Counts on both sides of the 32 that a warp tabulates, zeros and
    fractions; a second gene map on the same matrix (other totals), then the
    first again."""
    rng = np.random.default_rng(31)
    n, ng, per, G = 700, 400, 90, 6
    idx = np.sort(rng.random((n, ng)).argpartition(per - 1, axis=1)[:, :per], axis=1).astype(np.uint32).ravel()
    indptr = np.arange(n + 1, dtype=np.int64) * per
    val = rng.choice(np.array([1, 2, 31, 32, 33, 0, 0.5, 31.5, 40000], np.float32), len(idx))
    cm = np.arange(n, dtype=np.int64)
    cm[::11] = -1
    cm[cm >= 0] = np.arange((cm >= 0).sum())
    nr = int(cm.max()) + 1
    grp = rng.integers(0, G, nr).astype(np.uint32)
    grp[::13] = np.iinfo(np.uint32).max
    maps = []
    for step in (5, 2):
        gm = np.arange(ng, dtype=np.int32)
        gm[::step] = -1
        gm[gm >= 0] = np.arange((gm >= 0).sum(), dtype=np.int32)
        maps.append(gm)
    m = core.DeviceMatrix(indptr, idx, val, ng)
    for gm in (maps[0], maps[1], maps[0]):
        nv = int(gm.max()) + 1
        cl = rng.uniform(0.5, 3.0, (G, nv)) if clip else None
        got = resident(m, cm, gm, target, log, grp, G, nv, cl)
        ref = [np.zeros((G, nv)) for _ in range(3)]
        oracle.group_gene_sums(idx, val, cm, gm, target, log, None, indptr, 0, grp, *ref, cl)
        np.testing.assert_allclose(got[0], ref[0], rtol=1e-12, atol=1e-12)
        np.testing.assert_allclose(got[1], ref[1], rtol=1e-12, atol=1e-12)
        assert np.array_equal(got[2], ref[2])
    m.close()


def test_resident_group_sums_of_very_many_genes():
    """More genes than a shared-memory bit set of them holds (1.86 million)."""
    ng, n = 1_900_000, 6
    idx = np.sort(np.random.default_rng(1).choice(ng, (n, 50), replace=False), axis=1).astype(np.uint32)
    idx[:, -1] = ng - 1
    indptr = np.arange(n + 1, dtype=np.int64) * 50
    val = np.tile(np.arange(1, 51, dtype=np.float32), n)
    cm, gm = np.arange(n, dtype=np.int64), np.arange(ng, dtype=np.int32)
    grp = (np.arange(n) % 2).astype(np.uint32)
    m = core.DeviceMatrix(indptr, idx.ravel(), val, ng)
    got = resident(m, cm, gm, 1e4, True, grp, 2, ng)
    m.close()
    ref = [np.zeros((2, ng)) for _ in range(3)]
    oracle.group_gene_sums(idx.ravel(), val, cm, gm, 1e4, True, None, indptr, 0, grp, *ref)
    np.testing.assert_allclose(got[0], ref[0], rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(got[1], ref[1], rtol=1e-12, atol=1e-12)
    assert np.array_equal(got[2], ref[2])


@pytest.mark.parametrize("groups", [3, 436, 437, 900])  # 600 genes: up to and from 2 MB an array, more than one huge page
@pytest.mark.parametrize("stats", [True, False])
def test_group_sums_are_arrays_of_their_own(small_counts, groups, stats):
    """Zero to begin with, writable, and none keeps another's memory alive."""
    indptr, indices, data, n_genes = small_counts[:4]
    bf = cb.BioFrame.from_csr(indptr, indices, data, n_genes, var=pd.DataFrame({"gene_name": small_counts[4]}))
    grp = (np.arange(bf.n_obs) % groups).astype(np.uint32)
    ref = [np.zeros((groups, n_genes)) for _ in range(3)]
    oracle.group_gene_sums(indices, data, np.arange(bf.n_obs, dtype=np.int64), np.arange(n_genes, dtype=np.int32), 0.0,
                           False, None, indptr, 0, grp, *ref)
    got = cb.pp.group_gene_sums(bf, grp, groups, stats=stats)
    got = got if stats else (got,)
    for a, r in zip(got, ref):
        assert a.flags.c_contiguous and a.flags.writeable and a.dtype == np.float64
        assert np.array_equal(a, r)  # raw integer counts: exact
        held = a
        while isinstance(held, np.ndarray) and held.base is not None:
            held = held.base
        size = held.nbytes if isinstance(held, np.ndarray) else len(held)
        assert size < a.nbytes + (1 << 21)
    for i, a in enumerate(got):
        assert not any(np.shares_memory(a, b) for b in got[i + 1:])


@pytest.mark.parametrize("groups,genes", [(1, 65_535), (3, 21_845), (4, 16_384), (2, 32_769), (1, 7)])
def test_group_counts_around_their_narrow_form(groups, genes):
    """Up to 65,535 pairs the counts are kept as wide as the sums, from 65,536
    on in 32 bits: the same whole numbers either way, added to what the caller
    holds, on a resident matrix and in chunks."""
    rng = np.random.default_rng(genes)
    n, per = 300, 7
    idx = np.sort(np.stack([rng.choice(genes, per, replace=False) for _ in range(n)]), axis=1).astype(np.uint32).ravel()
    indptr = np.arange(n + 1, dtype=np.int64) * per
    val = rng.integers(1, 40, len(idx)).astype(np.float32)
    cm, gm = np.arange(n, dtype=np.int64), np.arange(genes, dtype=np.int32)
    grp = rng.integers(0, groups, n).astype(np.uint32)
    ref = [np.full((groups, genes), 2.0) for _ in range(3)]
    oracle.group_gene_sums(idx, val, cm, gm, 1e4, True, None, indptr, 0, grp, *ref)
    m = core.DeviceMatrix(indptr, idx, val, genes)
    kept = [np.full((groups, genes), 2.0) for _ in range(3)]
    _lib.call("crest_matrix_group_gene_sums", m.handle, _lib.ptr(cm), _lib.ptr(gm), 1e4, 1, _lib.ptr(grp), n, groups,
              genes, None, *[_lib.ptr(a) for a in kept])
    m.close()
    chunk = [np.full((groups, genes), 2.0) for _ in range(3)]
    _native.group_gene_sums(idx, val, cm, gm, 1e4, True, None, indptr, 0, grp, *chunk)
    totals = np.full((groups, genes), 2.0)
    _native.group_gene_totals(idx, val, cm, gm, 1e4, True, None, indptr, 0, grp, totals)
    for got in (kept, chunk):
        np.testing.assert_allclose(got[0], ref[0], rtol=1e-12)
        np.testing.assert_allclose(got[1], ref[1], rtol=1e-12)
        assert np.array_equal(got[2], ref[2])
    np.testing.assert_allclose(totals, ref[0], rtol=1e-12)
