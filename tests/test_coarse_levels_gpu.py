"""The coarse sub-cycle in one launch against the same cycle level by level.

mg_tail_points says which levels the one-launch sub-cycle takes: -1 leaves it the coarsest level alone
(every other level by launches of its own), 0 gives it all that fit, a number in between splits the
levels elsewhere.  The cycle is the same but for rounding (1e-6 of a preconditioner whose cycles reduce
by 1e-3), so the FGMRES and conjugate-gradient counts may differ by the granularity of the looks at
the estimate, two steps per cycle, and the fields by the solver's own tolerance (1e-8, as for every
comparison of two solves here).  Sizes: one level above the coarsest, odd plane counts, fewer planes
than CTAs, long and flat grids, levels at and around the one-CTA bound (8^3 .. 11^3 points).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size,precision", [((9, 8, 9), "mixed"), ((21, 19, 17), "mixed"), ((23, 20, 90), "mixed"),
                                           ((100, 40, 7), "mixed"), ((66, 66, 66), "mixed"), ((40, 35, 30), "fp64")])
def test_one_launch_and_level_by_level_cycles_agree(size, precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = size
    geom = np.zeros(size)
    geom[3:xs - 3, 3:ys - 3, 2:zs - 2] = 1
    geom[xs // 2:xs - 2, 2:ys // 2, 2:zs // 2 + 1] = 2
    table = np.array([[1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7], [2, 60, 60, 60, 3e6, 3e6, 3e6]], np.float64)
    B, G = np.array([1e-3, 2e-3, -4e-3]), np.zeros(9)
    out = {}
    for points in (-1, 0, 700):
        with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1e-3, 1e-3, 1e-5, precision=precision,
                                    mg_tail_points=points)) as s:
            s.set_geometry_f64(geom.flatten(order="F"), table)
            st = [s.steady([0.0, 0.0, 0.0], B, G), s.step([3.0, 0.0, -2.0], B, G), s.step([3.0, 0.0, -2.0], B, G)]
            assert all(q["status"] == 0 and q["r"] <= s.desc.tol for q in st), st
            out[points] = st, np.stack(s.fields())
    for points in (0, 700):
        for a, b in zip(out[points][0], out[-1][0]):
            assert abs(a["inner"] - b["inner"]) <= 2 * max(a["outer"], b["outer"]), (points, a, b)
        H, ref = out[points][1], out[-1][1]
        assert np.linalg.norm(H - ref) <= 1e-8 * np.linalg.norm(ref), points
