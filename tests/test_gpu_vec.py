"""The vector kernels at odd lengths and off 16-byte boundaries: elementwise
results bit for bit, sums independent of the alignment and within rounding of
numpy's."""
import numpy as np
import pytest

from tflows_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 2047, 2048, 2049, 300001, 1300001])
def test_vec_kernels(gpu_ctx, n):
    import torch
    rng = np.random.default_rng(n)
    a, b, y = (rng.uniform(0.5, 2.0, n) * rng.choice([-1, 1], n) for _ in range(3))
    sums = []
    for off in (0, 1):   # doubles past a 16-byte boundary
        def up(v):
            t = torch.zeros(n + 4, dtype=torch.float64, device="cuda")
            t[off:off + n] = torch.from_numpy(v)
            return t
        da, db, dy, dz = up(a), up(b), up(y), up(np.zeros(n))
        out = torch.zeros(8, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        p = [t.data_ptr() + 8 * off for t in (da, db, dy, dz)]
        o = out.data_ptr()
        native.vec_axpby(gpu_ctx, n, 0.3, p[0], -1.7, p[2])
        native.vec_dot(gpu_ctx, n, p[0], p[1], o)
        native.vec_dot(gpu_ctx, n, p[0], None, o + 8)
        native.vec_nrms_sum(gpu_ctx, n, p[0], p[1], o + 16)
        native.vec_jacobi(gpu_ctx, n, p[0], p[1], p[3], o + 24)
        native.vec_minmax(gpu_ctx, n, p[0], o + 32)
        gpu_ctx.sync()
        cut = slice(off, off + n)
        assert np.array_equal(dy[cut].cpu().numpy(), 0.3 * a + -1.7 * y)
        assert np.array_equal(dz[cut].cpu().numpy(), a * b)
        assert not dy[off + n:].any() and not dz[off + n:].any()
        sums.append(out.cpu().numpy())
    assert np.array_equal(sums[0], sums[1])
    want = [a @ b, a.sum(), np.sum((a * a) / (b * b)), (a * b) @ a, a.min(), a.max()]
    mass = [np.abs(a * b).sum(), np.abs(a).sum(), want[2], np.abs(a * b * a).sum(), 0, 0]
    # each sum is within (log2 of its length + a few) roundings of its terms' mass
    for got, w, m in zip(sums[0], want, mass):
        assert abs(got - w) <= 40 * 2.3e-16 * m
