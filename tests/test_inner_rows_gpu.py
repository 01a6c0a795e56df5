"""The inner operator's rows, row by row, against the oracle's CSR.

Every instantiation that a solve launches: D^-1 M x (each velocity axis, the general form and none), the
coupling of the potential rows to A, and the A rows without motion; on cubic cells, whose links leave
out 1/h^2, and on others; FP32 and FP64 vectors; sizes at and beyond a tile's edges.  A row sums at
most 37 products of magnitude |m_ij x_j| / d_i; in the vectors' precision a coefficient carries a handful
of roundings, its products two, their sum half an ulp per term and the quotient two: 64 ulp of
sum |m_ij x_j| / d_i bound the difference.  Vectors are zero on the Dirichlet rows, as a solve's are.
(The conductor regions of a random geometry have no part in it.)
"""
import numpy as np
import pytest

import qms_oracle as o

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SCALED, COUPLE, A_ROWS = 0, 1, 2


def _interior(size):
    xs, ys, zs = size
    nx, ny, nz = xs + 1, ys + 1, zs + 1
    out = []
    for q, shape in enumerate([(nz, ny, xs), (nz, ys, nx), (zs, ny, nx), (nz, ny, nx)]):
        f = np.zeros(shape, bool)
        box = [slice(2, nz - 2), slice(2, ny - 2), slice(2, nx - 2)]
        if q < 3:
            box[2 - q] = slice(1, (xs, ys, zs)[q] - 1)
        f[tuple(box)] = True
        out.append(f.ravel())
    return np.concatenate(out)


@pytest.mark.parametrize("size,h", [((35, 10, 19), (1e-3, 1e-3, 1e-3)), ((35, 10, 19), (1e-3, 1.1e-3, 0.9e-3)),
                                    ((33, 17, 9), (0.25e-3, 0.25e-3, 0.25e-3)), ((66, 24, 12), (1e-3, 1e-3, 1e-3))])
@pytest.mark.parametrize("v,transient", [((0, 0, 0), False), ((0, 0, 0), True), ((-7, 0, 0), True), ((0, 3, 0), True),
                                         ((0, 0, 5), True), ((2, -3, 1), True), ((2, -3, 1), False)])
def test_inner_rows_match_the_csr(size, h, v, transient):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300 import _lib
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = size
    dt = 1e-5
    rng = np.random.default_rng(3)
    geom = rng.integers(0, 3, size=size).astype(np.float64).flatten(order="F")
    table = np.array([[1, 1, 2, 3, 3.5e7, 1e7, 5e6], [2, 50, 40, 60, 2e6, 3e6, 4e6]], np.float64)
    c = o.materials(xs, ys, zs, geom, table)
    n, inner = int(o.sizes(xs, ys, zs)[0]), _interior(size)
    oV = o.block_offsets(xs, ys, zs)[3]
    x, w = (np.where(inner, rng.standard_normal(n) * s, 0.0) for s in (1e-4, 1e-3))
    is_v = np.arange(n) >= oV
    ia, ja, a, _ = o.assemble(xs, ys, zs, *h, c, transient, dt, np.array(v, float), np.zeros(3), np.zeros(9), x)
    M = o.to_scipy(ia, ja, a, n)
    d, M_abs = np.abs(M.diagonal()), abs(M)
    t_x, t_w = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    t_y = torch.empty_like(t_x)
    torch.cuda.synchronize()
    for precision, eps in (("mixed", np.finfo(np.float32).eps), ("fp64", np.finfo(np.float64).eps)):
        with QMSSolver(default_desc(xs, ys, zs, *h, dt, precision=precision, mg_region_cut=-1.0)) as s:
            s.set_geometry_f64(geom, table)
            for rows in (SCALED, COUPLE) + (() if any(v) else (A_ROWS,)):
                xi = x if rows == SCALED else np.where(is_v, 0.0, x)
                ref, bound = M @ xi, M_abs @ np.abs(xi)
                if rows == A_ROWS:
                    ref, bound = np.where(is_v, 0.0, ref), np.where(is_v, 0.0, bound)
                else:
                    ref, bound = ref / d, bound / d
                if rows == COUPLE:
                    ref, bound = np.where(is_v & inner, w - ref, 0.0), np.where(is_v, np.abs(w) + bound, 0.0)
                rc = s.L.qms_apply_inner(s.h, rows, int(transient), _lib.dvec(v), t_x.data_ptr(), t_w.data_ptr(),
                                         t_y.data_ptr())
                assert rc == 0
                err = np.abs(t_y.cpu().numpy() - ref)
                assert (err <= 64 * eps * bound).all(), (precision, rows, float((err - 64 * eps * bound).max()))
            assert s.L.qms_apply_inner(s.h, 3, 1, _lib.dvec(v), t_x.data_ptr(), t_w.data_ptr(), t_y.data_ptr()) == -1
