"""Sweep counts whose weights differ: one (omega), several (Chebyshev), more than the coarse table holds.

With each count the one-launch sub-cycle and the launches of its own per level are the same cycle but
for rounding, so FGMRES and conjugate-gradient counts may differ by the granularity of the looks at the
estimate, two steps per cycle, and the fields by the solver's own tolerance (1e-8, as for every comparison
of two solves); so may the fields of different counts.  Conjugate gradients need the cycle symmetric.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("sweeps", [1, 2, 5, 8, 9])
def test_sweep_counts_agree(sweeps, precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = size = (45, 38, 41)
    geom = np.zeros(size)
    geom[5:xs - 6, 4:ys - 5, 6:zs - 4] = 1
    geom[xs // 2:xs - 4, 3:ys // 2, 4:zs // 2] = 2
    table = np.array([[1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7], [2, 60, 60, 60, 3e6, 3e6, 3e6]], np.float64)
    B, G = np.array([1e-3, 2e-3, -4e-3]), np.zeros(9)
    out = []
    for n, points in ((3, 0), (sweeps, -1), (sweeps, 0)):
        with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1e-3, 1e-3, 1e-5, precision=precision, mg_sweeps=n,
                                    mg_tail_points=points)) as s:
            s.set_geometry_f64(geom.flatten(order="F"), table)
            st = [s.steady([0.0, 0.0, 0.0], B, G), s.step([3.0, 0.0, -2.0], B, G)]
            assert all(q["status"] == 0 and q["r"] <= s.desc.tol for q in st), st
            out.append((st, np.stack(s.fields())))
    for a, b in zip(out[1][0], out[2][0]):
        assert abs(a["inner"] - b["inner"]) <= 2 * max(a["outer"], b["outer"]), (a, b)
    ref = out[0][1]
    for st, H in out[1:]:
        assert np.linalg.norm(H - ref) <= 1e-8 * np.linalg.norm(ref)
