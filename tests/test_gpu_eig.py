"""The block eigensolver behind ``pca_from_gram`` against LAPACK (FP64) at the
sizes where its kernels change shape: block widths of one and several 16-wide
steps, above the one-CTA Cholesky (64), odd and even matrix sizes, one more
than the whole-matrix Jacobi limit, locked columns leaving odd blocks.

Tolerances: the solver stops at residuals of 1e-11 of the largest eigenvalue.
An eigenvalue is then within 1e-11 of it (Bauer-Fike; 1e-10 with the rounding
of the products), the loadings are orthonormal to 1e-12, and the sine of the
angle between the leading subspaces is at most residual / gap (Davis-Kahan);
the test's gaps are at least 1e-3, so 1e-7 with the square root of k terms."""

import numpy as np
import pytest

from crest_b200 import _lib, _native

pytestmark = pytest.mark.gpu


def spectrum_case(d, k, seed):
    """Gram of a covariance with well separated leading values over a dense bulk."""
    rng = np.random.default_rng(seed)
    lam = np.concatenate([1.5 + 0.05 * np.arange(k, 0, -1) + np.r_[20.0, np.zeros(k - 1)],
                          np.sort(rng.uniform(0.2, 1.0, d - k))[::-1]])
    Q = np.linalg.qr(rng.standard_normal((d, d)))[0]
    C = (Q * lam) @ Q.T
    return 0.5 * (C + C.T), lam, Q


@pytest.mark.parametrize("d,k", [(161, 1), (162, 2), (200, 7), (333, 18), (256, 34), (777, 50), (500, 51), (640, 60),
                                 (2001, 50)])
def test_block_eigensolver_matches_lapack(d, k):
    C, lam, Q = spectrum_case(d, k, d + k)
    n = 5000
    vals, vecs, total = _native.pca_from_gram(np.triu(C * (n - 1)), np.zeros(d), n, k)
    ref = np.linalg.eigvalsh(C)[::-1][:k]
    assert np.abs(vals - ref).max() <= 1e-10 * ref[0]
    assert abs(total - np.trace(C)) <= 1e-12 * np.trace(C)
    assert np.abs(vecs.T @ vecs - np.eye(k)).max() <= 1e-12
    assert np.linalg.norm(vecs - Q[:, :k] @ (Q[:, :k].T @ vecs), 2) <= 1e-7
    big = np.abs(vecs).argmax(0)
    assert np.all(vecs[big, np.arange(k)] > 0)


@pytest.mark.parametrize("d,run", [(2639, "eig_lanczos"), (2764, "eig_lanczos"), (2765, "eig_lanczos_steps")])
def test_spectrum_bounds_at_the_shared_memory_limit(d, run):
    """The one-launch Lanczos run holds its rows and one vector in shared memory
    up to 2,764 rows (148 SMs); one more takes a launch per step."""
    k = 10
    C, lam, Q = spectrum_case(d, k, d)
    n = 5000
    _lib.profile_enable(True)
    vals, vecs, _ = _native.pca_from_gram(np.triu(C * (n - 1)), np.zeros(d), n, k)
    ran = _lib.profile_table()
    _lib.profile_enable(False)
    assert run in ran and {"eig_lanczos", "eig_lanczos_steps"} & set(ran) == {run}
    assert np.abs(vals - lam[:k]).max() <= 1e-10 * lam[0]
    assert np.linalg.norm(vecs - Q[:, :k] @ (Q[:, :k].T @ vecs), 2) <= 1e-7


@pytest.mark.parametrize("d,k", [(2, 2), (37, 37), (160, 160), (160, 50)])
def test_nan_covariance_ranks_stay_a_permutation(d, k):
    """With a NaN off the diagonal no rotation is taken (its threshold is NaN),
    so the values are the diagonal: descending, ties by index, NaN last (and
    reported as 0 like a negative one), each with its own unit vector.  The
    ranks index the vectors, so they have to be a permutation."""
    rng = np.random.default_rng(d)
    diag = rng.integers(1, 1 + d // 3 + 1, d).astype(np.float64)
    if d > 2:
        diag[[3, d // 2, d - 2]] = np.nan
    G = np.diag(diag)
    G[0, 1] = np.nan
    vals, vecs, _ = _native.pca_from_gram(G, np.zeros(d), 2, k)
    order = sorted(range(d), key=lambda i: (np.isnan(diag[i]), -diag[i] if diag[i] == diag[i] else 0.0, i))[:k]
    assert np.array_equal(vals, np.nan_to_num(diag[order], nan=0.0))
    assert np.array_equal(vecs, np.eye(d)[:, order])
