"""GPU tests of the FP64 Gram's tiles and the FP64 update's forms at their edges.

The Gram picks its tile (16, 32 or 64 columns of A by 1 to 8 columns of B per thread)
and its chunks by na, nb and m, and leaves out tiles below the diagonal of X^T X where
only the upper part is used; the update has code per width and splits K over four warps
by a rule on m and K. Every entry must be the product whatever was picked.
"""
import numpy as np
import pytest

from bcgs_gb300 import inputs, orth
from helpers import qr_tolerance, sign_normalize

pytestmark = pytest.mark.gpu
U = np.finfo(np.float64).eps / 2


@pytest.mark.parametrize("na,b0,nb", [(1, 0, 1), (4, 0, 4), (16, 0, 16), (17, 12, 5), (33, 23, 10), (64, 44, 20),
                                      (65, 60, 3), (100, 68, 32), (129, 95, 34), (200, 136, 64), (128, 0, 128)])
@pytest.mark.parametrize("m", [1, 15, 16, 63, 65, 1000, 70001])
def test_gram_tiles(lib, m, na, b0, nb):
    torch = pytest.importorskip("torch")
    n, ld = max(na, b0 + nb), m + 3
    g = torch.Generator(device="cuda")
    g.manual_seed(m + na)
    X = torch.randn((n, ld), generator=g, device="cuda", dtype=torch.float64)
    C = torch.full((nb, na + 1), 7.0, device="cuda", dtype=torch.float64)
    assert orth.gram_dev(m, na, b0, nb, X.data_ptr(), ld, C.data_ptr(), na + 1, orth.FP64) == 0
    torch.cuda.synchronize()
    A, B = X[:na, :m], X[b0:b0 + nb, :m]
    # An FMA chain of m terms: at most (m + 2) u times the sum of the magnitudes.
    err = (C[:, :na] - B @ A.T).abs()
    assert bool((err <= 2 * (m + 2) * U * (B.abs() @ A.abs().T)).all())
    assert bool((C[:, na] == 7.0).all())


@pytest.mark.parametrize("s,n", [(1, 40), (3, 100), (6, 80), (10, 101), (11, 143), (13, 90), (15, 150), (16, 150),
                                 (18, 108), (27, 110), (31, 95), (36, 150), (50, 190)])
@pytest.mark.parametrize("variant", ["bcgsi2P1s", "bcgsi2"])
@pytest.mark.parametrize("m", [2000, 2049])
def test_update_widths_and_splits(lib, variant, s, n, m):
    """K runs through both sides of the split rule; both m leave a partial last tile."""
    X = inputs.graded_host(m, n, 1e3, seed=s * 1000 + n)
    Q, R, rc, st = orth.qr(variant, X, s)
    assert rc == 0 and st["breakdown_step"] == 0
    Q, R = sign_normalize(Q, np.triu(R))
    Qo, Ro = sign_normalize(*np.linalg.qr(X))
    tol = qr_tolerance(1e3)
    assert np.max(np.abs(Q - Qo)) <= tol
    assert np.max(np.abs(R - Ro)) <= tol * np.max(np.abs(Ro))


@pytest.mark.parametrize("m", [599999, 600001])
def test_update_split_rule_edge(lib, m):
    torch = pytest.importorskip("torch")
    n, s = 60, 10
    X0 = inputs.graded_device(m, n, 1e3, seed=m)
    X, R = X0.clone(), torch.zeros((n, n), device="cuda", dtype=torch.float64)
    rc, st = orth.run_dev("bcgspipi2", m, n, s, X.data_ptr(), m, R.data_ptr(), n, orth.FP64)
    assert rc == 0 and st["breakdown_step"] == 0
    E = X @ X.T - torch.eye(n, device="cuda", dtype=torch.float64)
    assert float(E.norm()) <= 1e-13
    assert float((X0 - torch.triu(R.T).T @ X).norm() / X0.norm()) <= 1e-14


def test_gram_more_tiles_than_a_grid_dimension(lib):
    """C of 8208 x 8208 has over 65535 tiles."""
    torch = pytest.importorskip("torch")
    m, n = 24, 8208
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    X = torch.randn((n, m), generator=g, device="cuda", dtype=torch.float64)
    C = torch.full((n, n), 7.0, device="cuda", dtype=torch.float64)
    assert orth.gram_dev(m, n, 0, n, X.data_ptr(), m, C.data_ptr(), n, orth.FP64) == 0
    torch.cuda.synchronize()
    C -= X @ X.T
    assert bool((C.abs() <= 2 * (m + 2) * U * (X.abs() @ X.abs().T)).all())
