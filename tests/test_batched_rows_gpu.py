"""GPU tests of the batched FP64 plan's choice of Gram chunk rows (csrc/batched.cu).

One value for the whole plan, from the shapes of every block step: a power of two from
256 to 32768. With the same chunk rows the single-matrix driver gives the same bits,
whichever value is chosen: small chunks where the late steps have few matrices, large
ones where every step fills the GPU, chunks longer than a matrix, one matrix alone.
"""
import numpy as np
import pytest

from bcgs_gb300 import orth

pytestmark = pytest.mark.gpu

BATCHES = {
    "one": [(5000, 64, 8)],
    "late steps of one matrix": [(12000, 256, 16)] + [(2000, 32, 16)] * 9 + [(2100, 8, 4)] * 5,
    "even": [(3001, 40, 8)] * 40,
    "many": [(4000, 96, 16)] * 300,
}


@pytest.mark.parametrize("name", list(BATCHES))
def test_rows_and_bits(lib, name):
    torch = pytest.importorskip("torch")
    shapes = BATCHES[name]
    rng = np.random.default_rng(len(shapes))
    mats = [rng.standard_normal((n, m)) for m, n, _ in shapes]
    dX = [torch.from_numpy(x).cuda() for x in mats]
    dR = [torch.zeros((n, n), dtype=torch.float64, device="cuda") for _, n, _ in shapes]
    st = torch.cuda.current_stream().cuda_stream
    plan = orth.Batch([m for m, _, _ in shapes], [n for _, n, _ in shapes], [s for _, _, s in shapes],
                      [x.data_ptr() for x in dX], [r.data_ptr() for r in dR], stream=st)
    assert plan.rc == 0 and plan.run(st) == 0
    torch.cuda.synchronize()
    rows = {v[1] for v in plan.info()["tuned"].values()}
    assert len(rows) == 1
    rows = rows.pop()
    assert 256 <= rows <= 32768 and rows & (rows - 1) == 0
    plan.close()
    for b in sorted({0, len(shapes) // 2, len(shapes) - 1}):
        m, n, s = shapes[b]
        Q = torch.from_numpy(mats[b]).cuda()
        R = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        orth.set_gram_chunk_rows(rows)
        try:
            rc, _ = orth.run_dev("bcgsi2P1s", m, n, s, Q.data_ptr(), m, R.data_ptr(), n, orth.FP64, st)
        finally:
            orth.set_gram_chunk_rows(0)
        assert rc == 0
        assert torch.equal(Q, dX[b]) and torch.equal(R, dR[b])


def test_report_and_tune_flag(lib):
    """The report has no panel width (it differs from Gram to Gram), and the flag changes nothing."""
    torch = pytest.importorskip("torch")
    shapes = BATCHES["late steps of one matrix"]
    X = [torch.zeros((n, m), dtype=torch.float64, device="cuda") for m, n, _ in shapes]
    R = [torch.zeros((n, n), dtype=torch.float64, device="cuda") for _, n, _ in shapes]
    infos = []
    for tune in (False, True):
        plan = orth.Batch([m for m, _, _ in shapes], [n for _, n, _ in shapes], [s for _, _, s in shapes],
                          [x.data_ptr() for x in X], [r.data_ptr() for r in R], tune=tune,
                          stream=torch.cuda.current_stream().cuda_stream)
        assert plan.rc == 0
        infos.append(plan.info())
        plan.close()
    assert infos[0] == infos[1]
    assert all(v[0] == 0 for v in infos[0]["tuned"].values())
