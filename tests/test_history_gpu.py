"""A run from a state that was set does not depend on what the handle solved before.

The counts and rates that a solve leaves for the next one belong to the run: the same set_state and
steps give the same bits whether they are a handle's first calls or follow runs of other motions,
other fields and magnetostatic solves.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size,precision,steps", [((10, 9, 8), "mixed", 12), ((33, 40, 21), "mixed", 9),
                                                  ((33, 40, 21), "fp64", 4), ((80, 75, 90), "mixed", 7)])
def test_a_run_from_a_set_state_is_the_same_after_any_other(size, precision, steps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = size
    geom = np.zeros(size)
    geom[3:xs - 3, 3:ys - 3, 3:zs - 3] = 1
    geom[3:xs // 2, 3:ys // 2, 3:zs // 2] = 2
    table = np.array([[1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7], [2, 20, 20, 20, 5e6, 5e6, 5e6]], np.float64)
    B, G = np.array([1e-3, -1e-3, 3e-3]), np.array([-0.05, 0, 0, 0, -0.05, 0, 0, 0, 0.1])
    with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1e-3, 1e-3, 1e-5, precision=precision)) as s:
        s.set_geometry_f64(geom.flatten(order="F"), table)
        s.steady([0.0, 0.0, 0.0], B, G)
        start = s.get_state()

        def run():
            s.set_state(start)
            counts = []
            for _ in range(steps):
                st = s.step([4.0, 0.0, 0.0], B, G)
                counts.append((st["outer"], st["inner"]))
            return counts, s.get_state()

        first = run()
        for between in ((), ([0.0, 9.0, 0.0], 0.3), ([0.0, 0.0, 0.0], -1.0)):
            if between:
                s.set_state(start)               # (a magnetostatic solve takes a state without potential)
                s.steady([0.0, 0.0, 0.0], between[1] * B, G)
                for n in range(3):
                    s.step(between[0], between[1] * (1.0 + 0.3 * n) * B, G)
            again = run()
            assert again[0] == first[0], between
            assert np.array_equal(again[1], first[1]), between
