"""Differentiable normalise -> log1p -> scale -> project map (K7).

The CUDA forward and backward (crest_fused_forward / crest_fused_backward
behind crest_b200.autograd) are checked against an FP64 PyTorch reference of
the same map and its autograd gradient (tests/fused_case.py); that reference
gradient is itself checked against central finite differences in
tests/test_fused_reference.py.
Tolerances: scores 1e-5 and gradients 1e-4, relative in the 2-norm (the
CUDA path keeps y and log1p(y) in f32, as the reference's transform does).
"""

import numpy as np
import pytest
import torch

from crest_b200 import _lib
from crest_b200.autograd import fused_scale_project
from fused_case import loss_of, make_case, ref_run, rel

pytestmark = pytest.mark.gpu


def gpu_run(c):
    dev = torch.device("cuda")
    values = torch.tensor(c["values"], device=dev, requires_grad=True)
    sf = torch.tensor(c["sf"], device=dev, requires_grad=True)
    W = torch.tensor(c["W"], device=dev, requires_grad=True)
    scores = fused_scale_project(values, sf, W, torch.tensor(c["indptr"], device=dev),
                                 torch.tensor(c["indices"], device=dev), torch.tensor(c["mean"], device=dev),
                                 torch.tensor(c["std"], device=dev), c["max_value"])
    loss_of(scores.double(), torch.tensor(c["wts"], device=dev)).backward()
    return (scores.detach().cpu().double(), values.grad.cpu().double(), sf.grad.cpu().double(),
            W.grad.cpu().double())


@pytest.mark.parametrize("k,max_value", [(24, 10.0), (50, 10.0), (100, 10.0), (24, 0.75), (50, 0.0)])
def test_forward_and_gradients_match_fp64_reference(k, max_value):
    c = make_case(k=k, max_value=max_value)
    s_gpu, gx, gsf, gW = gpu_run(c)
    s_ref, rx, rsf, rW = ref_run(c)
    assert rel(s_gpu, s_ref) <= 1e-5
    assert rel(gx, rx) <= 1e-4
    assert rel(gsf, rsf) <= 1e-4
    assert rel(gW, rW) <= 1e-4


def test_differentiation_workload_shape():
    """The differentiation workload at its own shape: 50,000 cells x 2,000 HVG
    genes (~200 stored entries per cell), k = 50, scale max 10; the FP64
    reference runs with float64 PyTorch ops on the GPU."""
    c = make_case(n=50_000, d=2_000, k=50, max_value=10.0, seed=4, nnz_per_cell=200.0, clusters=20,
                  dispersion=0.2)
    s_gpu, gx, gsf, gW = gpu_run(c)
    s_ref, rx, rsf, rW = ref_run(c, device="cuda")
    assert rel(s_gpu, s_ref) <= 1e-5
    assert rel(gx, rx) <= 1e-4
    assert rel(gsf, rsf) <= 1e-4
    assert rel(gW, rW) <= 1e-4


def test_out_of_range_gene_id_is_rejected():
    c = make_case(n=50, d=40, k=8)
    c["indices"][3] = c["d"] + 5
    dev = torch.device("cuda")
    with pytest.raises(ValueError, match=r"gene ids in \[0, d\)"):
        fused_scale_project(torch.tensor(c["values"], device=dev), torch.tensor(c["sf"], device=dev),
                            torch.tensor(c["W"], device=dev), torch.tensor(c["indptr"], device=dev),
                            torch.tensor(c["indices"], device=dev), torch.tensor(c["mean"], device=dev),
                            torch.tensor(c["std"], device=dev), 10.0)
    assert _lib.EINVAL == -22


def test_wide_gene_set_counts_entries_with_global_atomics():
    """d above the shared-memory histogram of the backward (12,288 genes): the
    per-gene entry counts come from global atomics; the same gradients."""
    c = make_case(n=2000, d=13_000, k=24, max_value=10.0, seed=7, nnz_per_cell=300.0)
    s_gpu, gx, gsf, gW = gpu_run(c)
    s_ref, rx, rsf, rW = ref_run(c)
    assert rel(s_gpu, s_ref) <= 1e-5
    assert rel(gx, rx) <= 1e-4
    assert rel(gsf, rsf) <= 1e-4
    assert rel(gW, rW) <= 1e-4


@pytest.mark.parametrize("k", [1, 7, 31, 32, 33, 63, 64, 65, 127, 128])
def test_row_widths_and_segment_chunks(k):
    """Rows padded to 32, 64 and 128 columns with every remainder, genes with
    none, a few and several chunks of entries in the W gradient, cells with
    none to several 32-entry segments; the tolerances of this file."""
    c = make_case(n=1501, d=45, k=min(k, 45), max_value=10.0, seed=11 + k, nnz_per_cell=30.0)
    rng = np.random.default_rng(k)
    c["W"] = (rng.standard_normal((c["d"], k)) / np.sqrt(c["d"])).astype(np.float32)
    c["wts"] = rng.standard_normal((c["n"], k))
    c["k"] = k
    s_gpu, gx, gsf, gW = gpu_run(c)
    s_ref, rx, rsf, rW = ref_run(c)
    assert rel(s_gpu, s_ref) <= 1e-5
    assert rel(gx, rx) <= 1e-4
    assert rel(gsf, rsf) <= 1e-4
    assert rel(gW, rW) <= 1e-4


@pytest.mark.parametrize("n,d,k,per", [(1, 30, 50, 20.0), (300, 600, 50, 330.0), (592, 90, 20, 40.0), (593, 90, 100, 40.0)])
def test_few_cells_spread_over_blocks(n, d, k, per):
    """A block per cell (up to four blocks on each of 148 SMs), its eight warps
    taking none to two 32-entry segments each; the tolerances of this file."""
    c = make_case(n=max(n, 2), d=d, k=min(k, d), max_value=10.0, seed=n, nnz_per_cell=per)
    if n == 1:
        for key in ("sf", "wts"):
            c[key] = c[key][:1]
        c["indptr"] = c["indptr"][:2]
        for key in ("indices", "values"):
            c[key] = c[key][:c["indptr"][1]]
        c["n"] = 1
    s_gpu, gx, gsf, gW = gpu_run(c)
    s_ref, rx, rsf, rW = ref_run(c)
    assert rel(s_gpu, s_ref) <= 1e-5
    assert rel(gx, rx) <= 1e-4
    assert rel(gsf, rsf) <= 1e-4
    assert rel(gW, rW) <= 1e-4


@pytest.mark.parametrize("k", [1, 50, 128])
@pytest.mark.parametrize("n", [40, 5000])
def test_no_genes(n, k):
    """d = 0 through the C interface: entries are rejected (no gene id is in
    range) without a row of W being read - the padded copy has a zero row 0 for
    them - and an empty matrix has zero scores and gradients."""
    dev = torch.device("cuda")
    per = 37
    f32 = dict(dtype=torch.float32, device=dev)
    W, mean = torch.full((4,), float("nan"), **f32), torch.zeros(1, dtype=torch.float64, device=dev)
    sf, G = torch.ones(n, **f32), torch.ones((n, k), **f32)
    indices, values = torch.zeros(n * per, dtype=torch.int32, device=dev), torch.ones(n * per, **f32)
    for entries in (per, 0):
        indptr = torch.arange(n + 1, device=dev) * entries
        scores, gx, gsf = (torch.full(s, 7.0, **f32) for s in ((n, k), (n * per,), (n,)))
        a = (indptr.data_ptr(), indices.data_ptr(), values.data_ptr(), n, 0, sf.data_ptr(), W.data_ptr(), k,
             mean.data_ptr(), mean.data_ptr(), 10.0)
        out = (G.data_ptr(), gx.data_ptr(), gsf.data_ptr(), W.data_ptr())
        torch.cuda.synchronize()
        if entries:
            with pytest.raises(ValueError, match=r"gene ids in \[0, d\)"):
                _lib.call("crest_fused_forward", *a, scores.data_ptr())
            with pytest.raises(ValueError, match=r"gene ids in \[0, d\)"):
                _lib.call("crest_fused_backward", *a, *out)
        else:
            _lib.call("crest_fused_forward", *a, scores.data_ptr())
            _lib.call("crest_fused_backward", *a, *out)
        assert torch.all(scores == 0) and torch.all(gsf == 0)
        assert torch.all(gx[:n * entries] == 0)
        assert torch.all(torch.isnan(W))  # an output of no rows, and an input of none


@pytest.mark.parametrize("n,per", [(593, 330.0), (9472, 330.0), (9473, 330.0), (700, 110.0), (600, 140.0)])
def test_spread_of_the_backward_over_blocks(n, per):
    """The backward takes a block per cell up to 9,472 cells (148 SMs) that
    average 128 entries: both sides of either line; the tolerances of this file."""
    c = make_case(n=n, d=600, k=20, max_value=10.0, seed=n, nnz_per_cell=per)
    s_gpu, gx, gsf, gW = gpu_run(c)
    s_ref, rx, rsf, rW = ref_run(c)
    assert rel(s_gpu, s_ref) <= 1e-5
    assert rel(gx, rx) <= 1e-4
    assert rel(gsf, rsf) <= 1e-4
    assert rel(gW, rW) <= 1e-4


@pytest.mark.parametrize("n,k", [(3, 1), (700, 50)])
def test_rejected_call_leaves_no_trace(n, k):
    """The flag of an out-of-range gene id is the next call's again: rejected,
    accepted with the right scores, rejected, forward and backward."""
    rng = np.random.default_rng(n)
    dev, d, per = torch.device("cuda"), 30, 40
    indptr = torch.arange(n + 1, device=dev) * per
    good = torch.from_numpy(rng.integers(0, d, n * per).astype(np.int32)).to(dev)
    bad = good.clone()
    bad[-1] = d
    v = torch.ones(n * per, device=dev, requires_grad=True)
    sf = torch.full((n,), 2.0, device=dev, requires_grad=True)
    W = torch.ones((d, k), device=dev, requires_grad=True)
    mean, std = torch.zeros(d, dtype=torch.float64, device=dev), torch.ones(d, dtype=torch.float64, device=dev)
    want = per * np.log1p(0.5)
    for _ in range(2):
        with pytest.raises(Exception, match="gene ids"):
            fused_scale_project(v, sf, W, indptr, bad, mean, std, 10.0)
        s = fused_scale_project(v, sf, W, indptr, good, mean, std, 10.0)
        assert torch.allclose(s, torch.full_like(s, want), rtol=1e-6)
        g = torch.autograd.grad(s.sum(), (v, sf, W))
        assert torch.allclose(g[0], torch.full_like(g[0], k / 3.0), rtol=1e-6)
