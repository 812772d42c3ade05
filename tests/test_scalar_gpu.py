"""GPU test of the reciprocal and square root that the block step and the TSQR compute
with fewer dependent instructions than a division and sqrt (csrc/common.cuh), against
CUDA's own over the exponents that their callers admit (2^-930 .. 2^930).

Both end in one fused operation on a correction of relative size 2^-19 or less, known to
far more than the bits that count, so they are within about 0.6 units in the last place
of the exact value, and CUDA's are correctly rounded: the two are equal or neighbours.
"""
import numpy as np
import pytest

from bcgs_gb300 import orth

pytestmark = pytest.mark.gpu


def _values():
    rng = np.random.default_rng(7)
    n = 1 << 21
    some = np.ldexp(1.0 + rng.random(n), rng.integers(-930, 930, n).astype(np.int32))
    edge = []
    for e in range(-929, 930):
        p = np.ldexp(1.0, e)
        edge += [p, np.nextafter(p, 0.0), np.nextafter(p, np.inf), 1.5 * p]
    near = 1.0 + np.arange(-2048, 2049) * np.finfo(np.float64).eps
    # Mantissas around the steps of any table of up to 2^12 entries.
    steps = 1.0 + np.arange(1, 4096) / 4096.0
    return np.concatenate([some, edge, near, steps, np.nextafter(steps, 0.0), np.nextafter(steps, 2.0),
                           [np.ldexp(1.0, -930), np.ldexp(1.0, 930)]])


def test_reciprocal_and_root_against_cuda(lib):
    torch = pytest.importorskip("torch")
    x = torch.from_numpy(_values()).cuda()
    r, u = torch.zeros_like(x), torch.zeros_like(x)
    assert orth.scalar_probe(x.numel(), x.data_ptr(), r.data_ptr(), u.data_ptr(),
                             torch.cuda.current_stream().cuda_stream) == 0
    for mine, cuda in ((r, 1.0 / x), (u, torch.sqrt(x))):
        ulps = (mine.view(torch.int64) - cuda.view(torch.int64)).abs()
        assert int(ulps.max()) <= 1


def test_scalar_probe_rejects_null(lib):
    assert orth.scalar_probe(4, 0, 0, 0) == 2
