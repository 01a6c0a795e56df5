"""The operator rows on cubic cells, whose links leave out 1/h^2, against the oracle's CSR.

Cubic cells take the unit-scaled rows in the FP64 residual (qms_residual_noalloc, qms_residual_norm)
and in the inner operator; others the general ones.  For every set of velocity components that has an
instantiation of its own, and for the general form, the residual of random states must agree with
D^-1 (b - M x) from the oracle's CSR row by row: a row sums at most 37 products of magnitude
|m_ij x_j| / d_i, each with a handful of roundings, so 64 ulp of that sum bounds the difference.
"""
import ctypes

import numpy as np
import pytest

import qms_oracle as o

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("h", [(1e-3, 1e-3, 1e-3), (1e-3, 1.1e-3, 0.9e-3)])
@pytest.mark.parametrize("v,transient", [((0, 0, 0), False), ((0, 0, 0), True), ((-7, 0, 0), True), ((0, 3, 0), True),
                                         ((0, 0, 5), True), ((2, -3, 1), True), ((2, -3, 1), False)])
def test_residual_rows_match_the_csr(h, v, transient):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300 import _lib
    xs, ys, zs, dt = 35, 10, 19, 1e-5
    rng = np.random.default_rng(3)
    geom = rng.integers(0, 3, size=(xs, ys, zs)).astype(np.float64)
    table = np.array([[1, 1, 2, 3, 3.5e7, 1e7, 5e6], [2, 50, 40, 60, 2e6, 3e6, 4e6]], np.float64)
    c = o.materials(xs, ys, zs, geom.flatten(order="F"), table)
    n = int(o.sizes(xs, ys, zs)[0])
    x, b0 = rng.standard_normal(n) * 1e-4, rng.standard_normal(n)
    ia, ja, a, _ = o.assemble(xs, ys, zs, *h, c, transient, dt, np.array(v, float), np.zeros(3), np.zeros(9), x)
    M = o.to_scipy(ia, ja, a, n)
    d = np.abs(M.diagonal())
    b = b0 * d * 1e-4
    ref = (b - M @ x) / d
    size = (abs(M) @ np.abs(x) + np.abs(b)) / d
    L = _lib.load()
    fn = L.qms_residual_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int] * 3 + [ctypes.c_double] * 4 + [ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                                                                 ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int] + [ctypes.c_void_p] * 5
    slots = torch.from_numpy(geom.flatten(order="F").astype(np.uint8)).cuda()
    rows = np.ascontiguousarray(table[:, 1:7])
    t_x, t_b = torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda()
    t_r, t_s = torch.empty_like(t_x), torch.empty(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = fn(xs, ys, zs, *h, dt, int(transient), _lib.dvec(v), slots.data_ptr(), rows.ctypes.data, 2, t_x.data_ptr(),
            t_b.data_ptr(), t_r.data_ptr(), t_s.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    err = np.abs(t_r.cpu().numpy() - ref)
    assert (err <= 64 * np.finfo(float).eps * size).all(), float((err / size).max())
