"""The FP64 residual where sigma x / dt and b nearly cancel, on cubic and other cells.

In a uniform conductor a constant potential has no differences: a row's residual is (b - m x) / d with
m = sigma (1 / dt).  With sigma a power of two m is exact.  On cubic cells the row forms b - m x in one
fused operation, and the quotient's operands carry the roundings of that difference and of d's five sums
and products: 16 ulp of r bound them (at most 8 halves of an ulp, and those of the reference's own d).
A time term that was rounded once more, by scaling it to the unit of the links, would be off by an ulp
of m x, which is up to 1e9 times r d here.  Other cells form m x first: half an ulp of m x / d more.
"""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MU0 = 1.25663706e-6


@pytest.mark.parametrize("h", [(1e-3, 1e-3, 1e-3), (0.7e-3, 0.7e-3, 0.7e-3), (1e-3, 1.1e-3, 0.9e-3)])
@pytest.mark.parametrize("dt", [1e-5, 3.7e-6])
def test_a_residual_that_cancels_keeps_its_digits(h, dt):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300 import _lib
    xs, ys, zs = 37, 12, 21
    sigma, c = 2.0 ** 25, 3.1e-4
    m = sigma * (1.0 / dt)
    rng = np.random.default_rng(2)
    values = m * c * (1.0 + rng.uniform(-1, 1, 40) * 10.0 ** rng.uniform(-9, -3, 40))
    d = sum(Fraction(2) / Fraction(MU0) / (Fraction(q) * Fraction(q)) for q in h) + Fraction(m)
    exact = np.array([float((Fraction(v) - Fraction(m) * Fraction(c)) / d) for v in values])
    nx, ny, nz = xs + 1, ys + 1, zs + 1
    n = [xs * ny * nz, nx * ys * nz, nx * ny * zs, nx * ny * nz]
    x = np.full(sum(n), c)
    x[sum(n[:3]):] = 0.0
    pick = rng.integers(0, values.size, sum(n[:3]))
    b = np.concatenate([values[pick], np.zeros(n[3])])
    L = _lib.load()
    slots = torch.ones(xs * ys * zs, dtype=torch.uint8, device="cuda")
    rows = np.array([[1.0, 1.0, 1.0, sigma, sigma, sigma]])
    t_x, t_b = torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda()
    t_r, t_s = torch.empty_like(t_x), torch.empty(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert L.qms_residual_noalloc(xs, ys, zs, *h, dt, 1, _lib.dvec([0.0, 0.0, 0.0]), slots.data_ptr(), rows.ctypes.data,
                                  1, t_x.data_ptr(), t_b.data_ptr(), t_r.data_ptr(), t_s.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream) == 0
    r, at = t_r.cpu().numpy(), 0
    for shape, size in zip([(nz, ny, xs), (nz, ys, nx), (zs, ny, nx)], n):
        inner = (slice(3, -3),) * 3                     # rows whose links and sigma are the conductor's
        got = r[at:at + size].reshape(shape)[inner]
        ref = exact[pick[at:at + size]].reshape(shape)[inner]
        eps = np.finfo(float).eps
        bound = 16 * eps * np.abs(ref) + (0.0 if h[0] == h[1] else 0.5 * eps * m * c / float(d))
        assert (np.abs(got - ref) <= bound).all(), float((np.abs(got - ref) / bound).max())
        at += size
