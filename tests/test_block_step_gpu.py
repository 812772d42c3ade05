"""GPU tests of the small work of a block step (csrc/small_fp64.cu) at its edges.

One launch per block step factors the joint matrix of the current and the next
block, by one CTA where the products are few and by a cluster of eight otherwise,
with or without the carried identity, and over the first block's pivots only in the
variants whose first pass is unscaled. Checked through whole QRs, against the
restated reference algorithm: block widths at and around the kernel's groups of 8
and 32 columns, ragged last blocks of one and s - 1 columns, and inputs scaled so far
that every pivot leaves the range of the elimination (the dot-product path).
"""
import numpy as np
import pytest

import bcgs_port as port
from bcgs_gb300 import inputs, orth
from helpers import qr_tolerance, sign_normalize

pytestmark = pytest.mark.gpu

KAPPA = 1e3


def _run(torch, variant, X, s, prec):
    m, n = X.shape
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    dR = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    rc, st = orth.run_dev(variant, m, n, s, dX.data_ptr(), m, dR.data_ptr(), n, prec,
                          torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and st["breakdown_step"] == 0 and st["timeout"] == 0, (rc, st)
    return dX.cpu().numpy().T, np.triu(dR.cpu().numpy().T)


@pytest.mark.parametrize("prec", [orth.FP64, orth.SPLIT_BF16])
@pytest.mark.parametrize("variant", ["bcgsi2P1s", "bcgsi21s", "bcgspipi2", "bcgsi2P2s"])
@pytest.mark.parametrize("s,n", [(1, 5), (4, 35), (7, 50), (16, 33), (17, 67), (33, 100), (64, 193), (64, 255)])
def test_block_step_edges(lib, variant, s, n, prec):
    torch = pytest.importorskip("torch")
    X = inputs.graded_host(1500, n, KAPPA, seed=100 * s + n)
    Q, R = sign_normalize(*_run(torch, variant, X, s, prec))
    Qo, Ro = sign_normalize(*np.linalg.qr(X))
    tol = qr_tolerance(KAPPA)
    assert np.max(np.abs(Q - Qo)) <= tol
    assert np.max(np.abs(R - Ro)) <= tol * np.max(np.abs(Ro))
    # 21s loses orthogonality with the block's condition number; the others do not.
    if variant != "bcgsi21s":
        assert port.loo_2(Q) <= 10 * max(port.loo_2(Qo), 1e-15)


@pytest.mark.parametrize("variant", ["bcgsi2P1s", "bcgsi21s", "bcgspipi2"])
@pytest.mark.parametrize("s,n", [(5, 27), (16, 80), (40, 120)])
@pytest.mark.parametrize("scale", [2.0 ** -480, 2.0 ** 480])
def test_block_step_pivots_out_of_range(lib, variant, s, n, scale):
    """A power-of-two scaling changes no rounding of the FP64 form, so Q must agree
    with the unscaled run's to the parity tolerance and R by the scale."""
    torch = pytest.importorskip("torch")
    X = inputs.graded_host(1500, n, KAPPA, seed=7 * s + n)
    Q1, R1 = _run(torch, variant, X, s, orth.FP64)
    Q2, R2 = _run(torch, variant, X * scale, s, orth.FP64)
    tol = qr_tolerance(KAPPA)
    assert np.max(np.abs(Q1 - Q2)) <= tol
    assert np.max(np.abs(R1 - R2 / scale)) <= tol * np.max(np.abs(R1))


@pytest.mark.parametrize("m,n,s", [(300, 64, 8), (4000, 128, 16), (1000, 48, 1), (3000, 96, 32)])
@pytest.mark.parametrize("variant", ["bcgsi2P1s", "bcgspipi2"])
@pytest.mark.parametrize("precision", ["fp64", "split7"])
@pytest.mark.parametrize("kappa", [1e10, 1e12])
def test_after_a_breakdown(lib, variant, precision, m, n, s, kappa):
    """Beyond the Pythagorean Cholesky's range the status reports the breakdown, and Q stays
    finite with columns of ordinary size: the pivots of columns that are noise are noise,
    but not exact zeros, which would end in NaN. The second pass of each block (or the
    lagged one) brings its columns back to norm 1 up to sqrt(s) where its Cholesky, too,
    breaks down part way."""
    prec = orth.FP64 if precision == "fp64" else orth.SPLIT_BF16
    assert orth.set_host_precision(prec) == 0
    norms = []
    try:
        for seed in range(9):
            X = inputs.graded_host(m, n, kappa, seed=seed)
            Q, R, rc, st = orth.qr(variant, X, s)
            assert rc == 0 and st["cuda_error"] == 0
            assert s == 1 or st["breakdown_step"] > 0
            assert np.isfinite(Q).all() and np.isfinite(np.triu(R)).all()
            norms.append(np.max(np.abs(np.linalg.norm(Q, axis=0) - 1.0)))
    finally:
        orth.set_host_precision(orth.FP64)
    assert np.median(norms) <= np.sqrt(s)
