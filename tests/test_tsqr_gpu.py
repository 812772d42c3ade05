"""GPU tests of the TSQR panel (csrc/tsqr_fp64.cu) at its edges.

Block 1 of bcgsi2 is the explicit TSQR of the first s columns alone, so a QR of 2s
columns gives the panel's Q and R. Checked against the contract of a Householder QR:
Q orthonormal to a few units of roundoff whatever the panel's condition, every column
reproduced to a few units of roundoff of its own norm, R upper triangular with a
non-negative diagonal. Widths at and around the column groups and the kernels'
widths, row counts at the tile edges (256 rows), columns whose squares overflow or
underflow, zero and dependent columns.
"""
import numpy as np
import pytest

from bcgs_gb300 import orth

pytestmark = pytest.mark.gpu
U = np.finfo(np.float64).eps / 2


def _panel(P):
    m, s = P.shape
    other = np.random.default_rng(5).standard_normal((m, s))
    Q, R, rc, st = orth.qr("bcgsi2", np.hstack([P, other]), s)
    assert rc == 0 and st["cuda_error"] == 0
    return Q[:, :s], R[:s, :s]


def _check(P):
    Q, R = _panel(P)
    s = P.shape[1]
    # Householder QR over at most 48 levels of 256-row tiles: errors of order s u per
    # level, few levels here.
    tol = 40 * (s + 10) * U
    assert np.linalg.norm(Q.T @ Q - np.eye(s)) <= tol
    assert np.all(np.tril(R, -1) == 0) and np.all(np.diag(R) >= 0)
    scale = np.max(np.abs(P), axis=0)
    scale[scale == 0] = 1.0
    D = P / scale - Q @ (R / scale)
    assert np.max(np.linalg.norm(D, axis=0) / np.sqrt(P.shape[0])) <= tol


@pytest.mark.parametrize("s", [1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 20, 31, 32, 33, 47, 63, 64])
@pytest.mark.parametrize("m", [255, 256, 257, 4100])
def test_tsqr_widths_and_tiles(lib, m, s):
    rng = np.random.default_rng(1000 * s + m)
    _check(rng.standard_normal((m, s)) * np.logspace(0, -12, s))


@pytest.mark.parametrize("s", [4, 10, 16, 40])
def test_tsqr_out_of_range_columns(lib, s):
    rng = np.random.default_rng(s)
    P = rng.standard_normal((3000, s))
    P *= np.ldexp(1.0, np.array([[-600, 0, 600, 300][j % 4] for j in range(s)]))
    _check(P)


@pytest.mark.parametrize("s", [4, 10, 16, 40])
def test_tsqr_rank_deficient(lib, s):
    rng = np.random.default_rng(s)
    P = rng.standard_normal((1500, s))
    P[:, 1] = 0.0
    P[:, 3] = P[:, 0]
    P[600:, 2] = 0.0
    _check(P)


@pytest.mark.parametrize("s", [8, 9, 11, 12, 14, 16, 17, 20, 33, 64])
@pytest.mark.parametrize("kappa", [1e2, 1e4, 3e4, 1e5, 1e8, 1e13])
def test_tsqr_conditions(lib, s, kappa):
    """Panels of 8 columns and more (in bcgsi2) take Cholesky QR where no column is too close to
    those before it and the tree otherwise; the contract is the same on both sides."""
    rng = np.random.default_rng(s)
    V, _ = np.linalg.qr(rng.standard_normal((3000, s)))
    W, _ = np.linalg.qr(rng.standard_normal((s, s)))
    _check((V * np.logspace(0, -np.log10(kappa), s)) @ W)


@pytest.mark.parametrize("s", [15, 21, 24, 25, 28, 29, 32])
@pytest.mark.parametrize("m", [2999, 40001])
def test_tsqr_checked_gram_widths(lib, m, s):
    """Widths at the edges of the narrow Gram kernel's forms, with fewer row groups than CTAs and with
    several to each."""
    rng = np.random.default_rng(m + s)
    _check(rng.standard_normal((m, s)) * np.logspace(0, -3, s))
