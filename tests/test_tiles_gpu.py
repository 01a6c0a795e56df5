"""The tiles of the stencil kernels at the edges of their range.

The kernels over the inner solver's vectors cover the nodes 1..xs-1, 1..ys-1, 1..zs-1 (rows beyond
are Dirichlet rows) in tiles of 32 x 8 columns that march over 16, 8, 4 or 2 planes, by the number
of tiles.  At sizes one below, at and one above a tile's edge, and at each march length, a steady
state and two steps must meet the tolerance in the exact FP64 residual over ALL rows
(qms_residual_norm, which runs the reference-layout operator) and keep the Dirichlet rows at their
values.  The bound is 1.5 tol: the solver stops at tol by its own residual, whose double-float
rounding stays below tol / 10 (test_chained_residual_does_not_drift).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size,precision", [
    ((32, 8, 9), "mixed"), ((33, 9, 8), "mixed"), ((34, 10, 18), "mixed"), ((65, 17, 35), "fp64"),
    ((33, 25, 12), "fp64"), ((97, 66, 41), "mixed"), ((129, 89, 97), "mixed"), ((225, 161, 161), "mixed")])
def test_every_row_of_a_step_is_solved(size, precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = size
    geom = np.zeros(size)
    geom[2:xs - 2, 2:ys - 2, 3:zs - 3] = 1               # conductor up to the Dirichlet shell
    geom[xs // 2, 3:ys - 3, 3:zs - 3] = 2
    table = np.array([[1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7], [2, 50, 50, 50, 2e6, 2e6, 2e6]], np.float64)
    B, G = np.array([1e-3, -2e-3, 5e-3]), np.array([-0.05, 0, 0, 0, -0.05, 0, 0, 0, 0.1])
    nx, ny, nz = xs + 1, ys + 1, zs + 1
    fixed = []
    for q, shape in enumerate([(nz, ny, xs), (nz, ys, nx), (zs, ny, nx), (nz, ny, nx)]):
        f = np.ones(shape, bool)
        box = [slice(2, nz - 2), slice(2, ny - 2), slice(2, nx - 2)]
        if q < 3:
            box[2 - q] = slice(1, (xs, ys, zs)[q] - 1)
        f[tuple(box)] = False
        fixed.append(f.ravel())
    fixed = np.concatenate(fixed)
    with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1.1e-3, 0.9e-3, 1e-5, precision=precision)) as s:
        s.set_geometry_f64(geom.flatten(order="F"), table)
        st = s.steady([0.0, 0.0, 0.0], B, G)
        assert st["status"] == 0
        for v, scale in (([-4.0, 0.0, 0.0], 1.0), ([-4.0, 0.0, 0.0], 0.9)):
            st = s.step(v, scale * B, scale * G)
            assert st["status"] == 0 and st["r"] <= s.desc.tol
            assert s.residual_norm(True, v) <= 1.5 * s.desc.tol
            assert np.array_equal(s.get_state()[fixed], s.get_rhs()[fixed])
