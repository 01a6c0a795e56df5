"""FGMRES cycles that end by their residual estimate, replayed from graphs or launched directly.

A velocity that repeats replays the cycle's steps from graphs, a new one launches them directly and
drops the graphs of the one before; bases of odd and of the largest length end a cycle in the middle
of a graph's steps.  Whatever the route, every step meets the tolerance in the exact FP64 residual
(1.5 tol: the double-float residual's rounding stays below tol / 10), also after a state that was
set from outside.  The solver's tolerance is relative to the larger of |x| before and after the solve
(a frame that stops loses its potential, and |x| shrinks), qms_residual_norm's to |x| after it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision,m,krylov_graphs", [("mixed", 32, 1), ("mixed", 5, 1), ("mixed", 64, 1),
                                                       ("mixed", 32, 0), ("fp64", 7, 1)])
def test_steps_meet_the_tolerance_on_every_route(precision, m, krylov_graphs):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = 22, 17, 19
    geom = np.zeros((xs, ys, zs))
    geom[5:16, 5:12, 6:12] = 1
    geom[9:12, 4:9, 8:14] = 2
    table = np.array([[1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7], [2, 80, 80, 80, 4e6, 4e6, 4e6]], np.float64)
    B, G = np.array([2e-3, -1e-3, 5e-3]), np.zeros(9)
    moves = [[-5.0, 0, 0], [-5.0, 0, 0], [-5.0, 0, 0], [0, 3.0, 1.0], [0, 3.0, 1.0], [-5.0, 0, 0], [0, 0, 0], [0, 0, 0]]
    with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1e-3, 1e-3, 1e-5, precision=precision, gmres_m=m,
                                use_graphs=krylov_graphs)) as s:
        s.set_geometry_f64(geom.flatten(order="F"), table)
        s.steady([0.0, 0.0, 0.0], B, G)
        start = s.get_state()
        for again in range(2):
            s.set_state(start)
            for n, v in enumerate(moves):
                before = np.linalg.norm(s.get_state())
                st = s.step(v, (1.0 - 0.05 * n) * B, G)
                after = np.linalg.norm(s.get_state())
                assert st["status"] == 0 and st["r"] <= s.desc.tol, (again, n, st)
                assert s.residual_norm(True, v) * after <= 1.5 * s.desc.tol * max(before, after), (again, n)
