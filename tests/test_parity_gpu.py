"""GPU parity tests: the CUDA path through the C ABI against the oracle.

Every test calls liborth_gb300.so through ctypes (the orth.h entry points or the
device-pointer entry point). The oracle is the reference's own output (golden
fixtures made by oracle/_ref) and the numpy restatement (oracle/bcgs_port.py).
Tolerances: Q and R/||R|| entries within 200*u*cond(X) + 1e-13 after sign
normalization; LOO and relative residual within 10x of the reference's (with an
n*u floor), the parity rule.
"""
import numpy as np
import pytest

import bcgs_port as port
from bcgs_gb300 import inputs, orth
from helpers import U, VARIANTS, load_golden, metric_ok, qr_tolerance, sign_normalize

pytestmark = pytest.mark.gpu
GOLD = load_golden()


def _compare(X, Q, R, Qref, Rref, cond):
    Qs, Rs = sign_normalize(Q, R)
    Qr, Rr = sign_normalize(Qref, Rref)
    tol = qr_tolerance(cond)
    assert np.max(np.abs(Rs - Rr)) <= tol * np.max(np.abs(Rr))
    assert np.max(np.abs(Qs - Qr)) <= tol


@pytest.mark.parametrize("precision", ["fp64", "split7"])
@pytest.mark.parametrize("case", sorted(GOLD))
@pytest.mark.parametrize("variant", VARIANTS)
def test_golden(lib, case, variant, precision):
    """The reference's own outputs (tests/golden/bcgs_golden.npz) through the orth.h
    host entry points, in FP64 and in the 56-bit split form."""
    g = GOLD[case]
    X, n, s = g["X"], g["n"], g["s"]
    gv = g[variant]
    assert orth.set_host_precision(orth.FP64 if precision == "fp64" else orth.SPLIT_BF16) == 0
    try:
        Q, R, rc, st = orth.qr(variant, X, s)
    finally:
        orth.set_host_precision(orth.FP64)
    assert rc == 0 and st["cuda_error"] == 0
    if gv["info"] != 0:
        if case == "edge_n2s_plus4" and variant == "bcgsi2P1s":
            # The reference reads its first-step X_3^T X_3 buffer with the wrong
            # leading dimension when 2s < n < 3s (SRC/orth.c:129-131 vs :160-163),
            # which breaks its Cholesky. This library forms the intended Omega:
            # no breakdown, and a Q at least as orthogonal as the reference's.
            assert st["breakdown_step"] == 0
            assert port.loo_fro(Q) <= gv["metrics"][0]
            assert port.rel_residual(X, Q, R) <= 10 * max(gv["metrics"][2], n * U)
        else:
            # Both break down. Near breakdown the first failing step depends on
            # rounding (the Gram sums are ordered differently from OpenBLAS), so
            # ours may fail one step earlier or later than the reference.
            assert st["breakdown_step"] > 0
            assert abs(st["breakdown_step"] - gv["info"]) <= 1
        return
    assert st["breakdown_step"] == 0
    Rg = gv["R"]
    d = np.sign(np.diag(Rg)).copy()
    d[d == 0] = 1
    tol = qr_tolerance(g["cond"])
    Qs, Rs = sign_normalize(Q, R)
    assert np.max(np.abs(Rs - Rg * d[:, None])) <= tol * np.max(np.abs(Rg))
    assert np.max(np.abs(Qs[:: g["qstride"], :] - gv["Qrows"] * d)) <= tol
    loo_f, _, res = gv["metrics"]
    assert metric_ok(port.loo_fro(Q), loo_f, n * U)
    assert metric_ok(port.rel_residual(X, Q, R), res, n * U)


@pytest.mark.parametrize("precision", ["fp64", "split7"])
@pytest.mark.parametrize("variant", ["bcgsi2", "bcgsi2P2s"])
def test_golden_monomial_median(lib, variant, precision):
    """The golden monomial case over 31 roundings of its input.

    Its blocks are exactly dependent in FP64 (condition 3e29), so the panels that bcgsi2 and
    bcgsi2P2s hand to the TSQR are rounding noise and the LOO is a draw, in the reference
    too: with every entry of X moved by at most one unit in the last place, 8 % (bcgsi2) and
    12 % (bcgsi2P2s) of 128 FP64 draws are over test_golden's limit, 12 to 27 % when every
    panel went through the tree. test_golden sees one draw, which one order of the TSQR's
    sums passes and another does not; the median over many says whether the kernels got
    worse. The residual is no draw.
    """
    g = GOLD["monomial_s8"]
    X, n, s = g["X"], g["n"], g["s"]
    loo_f, _, res = g[variant]["metrics"]
    rng = np.random.default_rng(11)
    assert orth.set_host_precision(orth.FP64 if precision == "fp64" else orth.SPLIT_BF16) == 0
    loos = []
    try:
        for k in range(31):
            Xk = X if k == 0 else np.asfortranarray(X + rng.integers(-1, 2, X.shape) * np.spacing(X))
            Q, R, rc, st = orth.qr(variant, Xk, s)
            assert rc == 0 and st["cuda_error"] == 0
            assert metric_ok(port.rel_residual(Xk, Q, R), res, n * U)
            loos.append(np.inf if st["breakdown_step"] else port.loo_fro(Q))
    finally:
        orth.set_host_precision(orth.FP64)
    assert metric_ok(float(np.median(loos)), loo_f, n * U)


@pytest.mark.parametrize("shape", [(3000, 50, 7), (2048, 10, 1), (4096, 128, 32), (6000, 128, 64),
                                   (1000, 37, 16), (777, 24, 12)])
@pytest.mark.parametrize("variant", VARIANTS)
def test_random_shapes_vs_oracle(lib, shape, variant):
    m, n, s = shape
    X = inputs.graded_host(m, n, 1e4, seed=m + n + s)
    Q, R, rc, st = orth.qr(variant, X, s)
    assert rc == 0 and st["breakdown_step"] == 0
    Qp, Rp, info = port.run_variant(variant, X, n, s)
    if variant == "bcgsi2P1s" and 2 * s < n < 3 * s:
        # The reference's leading-dimension quirk (SRC/orth.c:129-131 vs
        # :160-163), reproduced by the oracle, perturbs its first loop step;
        # this library forms the intended Omega. Compare accuracy only.
        assert port.loo_fro(Q) <= max(port.loo_fro(Qp), n * U)
        assert metric_ok(port.rel_residual(X, Q, R), port.rel_residual(X, Qp, Rp), n * U)
        return
    assert info == 0
    _compare(X, Q, R, Qp, Rp, 1e4)
    assert metric_ok(port.loo_fro(Q), port.loo_fro(Qp), n * U)
    assert metric_ok(port.rel_residual(X, Q, R), port.rel_residual(X, Qp, Rp), n * U)


@pytest.mark.parametrize("variant", VARIANTS)
def test_bit_exact_run_to_run(lib, variant):
    X = inputs.graded_host(20000, 96, 1e6, seed=42)
    Q1, R1, rc1, _ = orth.qr(variant, X, 16)
    Q2, R2, rc2, _ = orth.qr(variant, X, 16)
    assert rc1 == rc2 == 0
    assert np.array_equal(Q1, Q2) and np.array_equal(R1, R2)


def test_leading_dimension_and_untouched_lower_blocks(lib):
    m, n, s, ldx = 1500, 40, 8, 1600
    X = inputs.graded_host(m, n, 1e3, seed=9)
    Xb = np.full((ldx, n), 7.0, order="F")
    Xb[:m, :] = X
    R = np.full((n, n), -3.0, order="F")
    rc = orth.call("bcgsi2P1s", m, n, s, Xb, ldx, R, n)
    assert rc == 0
    assert np.all(Xb[m:, :] == 7.0)                 # rows past m untouched
    for j in range(n):                              # lower block triangle untouched
        b = j // s
        assert np.all(R[(b + 1) * s:, j] == -3.0)
    Qp, Rp, _ = port.run_variant("bcgsi2P1s", X, n, s)
    Rm = R.copy()
    for j in range(n):
        Rm[(j // s + 1) * s:, j] = 0.0
    _compare(X, Xb[:m, :], Rm, Qp, Rp, 1e3)


def test_device_entry_point_matches_host(lib):
    torch = pytest.importorskip("torch")
    m, n, s = 50000, 64, 16
    X = inputs.graded_host(m, n, 1e5, seed=3)
    Qh, Rh, rc, _ = orth.qr("bcgsi2P1s", X, s)
    assert rc == 0
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()      # (n, m) row-major == X col-major
    dR = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rc, st = orth.run_dev("bcgsi2P1s", m, n, s, dX.data_ptr(), m, dR.data_ptr(), n,
                          orth.FP64, stream)
    assert rc == 0 and st["breakdown_step"] == 0
    Qd = dX.cpu().numpy().T
    Rd = dR.cpu().numpy().T
    assert np.array_equal(Qd, Qh)
    assert np.array_equal(np.triu(Rd), np.triu(Rh))


@pytest.mark.parametrize("variant,precision", [("bcgsi2P1s", "fp64"), ("bcgsi2", "fp64"),
                                               ("bcgsi2P1s", "split"), ("bcgsi21s", "split")])
def test_device_leading_dimension(lib, variant, precision):
    """Device buffers with ldX > m (the reference's ldXsub >= msub): the same bits
    as with tight storage, and the padding rows keep their sentinel."""
    torch = pytest.importorskip("torch")
    m, n, s, pad = 30000, 64, 16, 37
    X = inputs.graded_host(m, n, 1e5, seed=21)
    prec = orth.FP64 if precision == "fp64" else orth.SPLIT_BF16
    st = torch.cuda.current_stream().cuda_stream
    tight = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    wide = torch.full((n, m + pad), 7.0, dtype=torch.float64, device="cuda")
    wide[:, :m] = tight
    outs = []
    for buf, ld in ((tight, m), (wide, m + pad)):
        R = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        rc, status = orth.run_dev(variant, m, n, s, buf.data_ptr(), ld, R.data_ptr(), n, prec, st)
        assert rc == 0 and status["breakdown_step"] == 0 and status["timeout"] == 0, (rc, status)
        outs.append(R.cpu().numpy())
    assert torch.equal(wide[:, :m], tight)
    assert bool((wide[:, m:] == 7.0).all())
    assert np.array_equal(np.triu(outs[0].T), np.triu(outs[1].T))


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_host_path_timeline(lib, precision):
    """orth.h host-buffer runs overlap the copies with the QR and record a timeline:
    X is resident before the kernels finish, Q is back after them, and the call's
    wall time covers all three. The result equals the device entry point's."""
    torch = pytest.importorskip("torch")
    m, n, s = 300000, 128, 16
    X = inputs.graded_host(m, n, 1e4, seed=11)
    prec = orth.FP64 if precision == "fp64" else orth.SPLIT_BF16
    assert orth.set_host_precision(prec) == 0
    try:
        Qh, Rh, rc, st = orth.qr("bcgsi2P1s", X, s)
    finally:
        orth.set_host_precision(orth.FP64)
    assert rc == 0 and st["breakdown_step"] == 0
    t = orth.last_host_timing()
    assert 0.0 < t["x_resident_ms"] <= t["compute_done_ms"] + 1e-3, t
    assert t["compute_done_ms"] <= t["q_back_ms"] + 1e-3, t
    assert t["q_back_ms"] <= t["wall_ms"] + 1.0, t
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    dR = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    rc, _ = orth.run_dev("bcgsi2P1s", m, n, s, dX.data_ptr(), m, dR.data_ptr(), n, prec,
                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert np.array_equal(dX.cpu().numpy().T, Qh)
    assert np.array_equal(np.triu(dR.cpu().numpy().T), np.triu(Rh))


def test_large_properties_fp64(lib):
    """Size-independent properties at m = 2^20: orthogonality and residual."""
    torch = pytest.importorskip("torch")
    m, n, s = 1 << 20, 256, 16
    Xt = inputs.graded_device(m, n, 1e6, seed=5)          # (n, m) == X column-major
    X0 = Xt.clone()
    for variant in VARIANTS:
        Xt.copy_(X0)
        R = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        rc, st = orth.run_dev(variant, m, n, s, Xt.data_ptr(), m, R.data_ptr(), n, orth.FP64,
                              torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and st["breakdown_step"] == 0, (variant, st)
        Q = Xt.t()
        Rm = R.t()
        G = (Q.t() @ Q - torch.eye(n, dtype=torch.float64, device="cuda")).cpu().numpy()
        loo = float(np.max(np.abs(np.linalg.eigvalsh(0.5 * (G + G.T)))))
        E = X0.t() - Q @ Rm
        res = float(((E * E).sum() / (X0 * X0).sum()).sqrt().item())
        assert loo < 1e-12, (variant, loo)
        assert res < 1e-14, (variant, res)


@pytest.mark.parametrize("precision", ["fp64", "split7"])
@pytest.mark.parametrize("variant", VARIANTS)
def test_measured_sync_count(lib, variant, precision):
    """The number of device-wide reductions a run launches (counted where the
    reduction kernel is launched) equals the variant's structure: p + 1 for the
    one-sync variants (one per block step after the first step's two), 2p for
    bcgspipi2 and bcgsi2. Reference: the MPI_Allreduce calls at SRC/orth.c:113,132,
    187/196 (P1s); :277,286,332/341 (21s); :423,437 (PIPI); :514,526 (BCGS2);
    :607,619,663/672 (P2s)."""
    torch = pytest.importorskip("torch")
    m, n, s = 20000, 96, 16
    X = inputs.graded_host(m, n, 1e4, seed=8)
    prec = orth.FP64 if precision == "fp64" else orth.SPLIT_BF16
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    dR = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    rc, st = orth.run_dev(variant, m, n, s, dX.data_ptr(), m, dR.data_ptr(), n, prec,
                          torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and st["breakdown_step"] == 0
    p = (n - s) // s
    expected = {"bcgsi2P1s": p + 1, "bcgsi21s": p + 1, "bcgsi2P2s": p + 1,
                "bcgspipi2": 2 * p, "bcgsi2": 2 * p}[variant]
    assert orth.sync_count(variant, n, s) == expected
    assert orth.last_reduction_count() == expected


@pytest.mark.parametrize("variant", ["bcgsi2P1s", "bcgsi21s", "bcgsi2"])
@pytest.mark.parametrize("r_on_device", [True, False])
def test_orth_h_with_device_pointers(lib, variant, r_on_device):
    """The orth.h entry points given device buffers (detected with
    cudaPointerGetAttributes): the QR runs in place on them, bit-identical to
    the host-buffer call; R gets exactly the reference's part (the rest keeps
    its sentinel), in device or host memory."""
    torch = pytest.importorskip("torch")
    m, n, s, ldx = 30000, 64, 16, 30011
    X = inputs.graded_host(m, n, 1e5, seed=13)
    Qh, Rh, rc, _ = orth.qr(variant, X, s)
    assert rc == 0
    dX = torch.full((n, ldx), 7.0, dtype=torch.float64, device="cuda")
    dX[:, :m] = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    if r_on_device:
        Rbuf = torch.full((n, n), -3.0, dtype=torch.float64, device="cuda")
        r_ptr = Rbuf.data_ptr()
    else:
        Rnp = np.full((n, n), -3.0, order="F")
        r_ptr = Rnp.ctypes.data
    torch.cuda.synchronize()
    rc = orth.call_ptr(variant, m, n, s, dX.data_ptr(), ldx, r_ptr, n)
    assert rc == 0
    Q = dX[:, :m].cpu().numpy().T
    R = Rbuf.cpu().numpy().T if r_on_device else Rnp
    assert np.array_equal(Q, Qh)
    assert bool((dX[:, m:] == 7.0).all())
    for j in range(n):
        b = j // s
        rows = min((b + 1) * s, n) if not (variant == "bcgsi21s" and b >= 1) else j + 1
        assert np.array_equal(R[:rows, j], Rh[:rows, j]), j
        assert np.all(R[(b + 1) * s:, j] == -3.0), j
