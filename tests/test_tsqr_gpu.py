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


def _unit_upper(s, kind, a):
    """Triangular factors whose diagonal says little about their condition: Kahan's
    (unit columns, diagonal a^j) and I - a triu(ones, 1) (unit diagonal, inverse of
    norm about (1 + a)^(s - 2))."""
    if kind == "kahan":
        T = np.eye(s) - np.sqrt(1.0 - a * a) * np.triu(np.ones((s, s)), 1)
        return T * (a ** np.arange(s))[:, None]
    return np.eye(s) - a * np.triu(np.ones((s, s)), 1)


@pytest.mark.parametrize("kind,a", [("kahan", 0.9), ("kahan", 0.8), ("kahan", 0.7), ("kahan", 0.5), ("triu", 0.25),
                                    ("triu", 0.5), ("triu", 1.0), ("triu", 2.0)])
@pytest.mark.parametrize("s", [8, 12, 16, 20, 24, 32, 40, 48, 64])
def test_tsqr_conditions_pivots_do_not_show(lib, s, kind, a):
    """Panels whose Cholesky pivots stay large next to their diagonal while the condition grows
    exponentially with the width: from harmless (8 columns) to numerically singular
    (64), so both sides of the check that admits Cholesky QR are covered."""
    for seed in range(3):
        V, _ = np.linalg.qr(np.random.default_rng(100 * s + seed).standard_normal((4000, s)))
        _check(V @ _unit_upper(s, kind, a))


@pytest.mark.parametrize("s", [20, 32, 64])
@pytest.mark.parametrize("variant", ["bcgsi2P1s", "bcgsi2P2s"])
def test_first_block_pivots_do_not_show(lib, variant, s):
    """Block 1 is orthogonalized once in every variant."""
    rng = np.random.default_rng(s)
    V, _ = np.linalg.qr(rng.standard_normal((4000, s)))
    X = np.hstack([V @ _unit_upper(s, "triu", 1.0), rng.standard_normal((4000, s))])
    Q, R, rc, st = orth.qr(variant, X, s)
    assert rc == 0 and st["cuda_error"] == 0
    Q1 = Q[:, :s]
    assert np.linalg.norm(Q1.T @ Q1 - np.eye(s)) <= 40 * (s + 10) * U
