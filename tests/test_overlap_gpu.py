"""Kernels that start before the one before them has ended (qms_pdl.cuh) keep the stream's order.

A kernel that read what its predecessor had not written yet would read differently from run to run:
the whole solve is a fixed sequence of fixed-order sums, so two handles that go through the same calls
(a first run, and repeated ones that replay its graphs) must be equal bit for bit after each.  (A
handle's later runs may differ from its first in rounding: their cycles are sized with its rate.)  Sizes: single-CTA launches, one
wave, and launches above the line where the overlap ends beside ones below it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size,precision,steps", [((10, 9, 8), "mixed", 12), ((33, 40, 21), "mixed", 8),
                                                  ((33, 40, 21), "fp64", 4), ((150, 130, 140), "mixed", 6)])
def test_repeated_runs_are_equal_bit_for_bit(size, precision, steps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = size
    geom = np.zeros(size)
    geom[3:xs - 3, 3:ys - 3, 3:zs - 3] = 1
    geom[3:xs // 2, 3:ys // 2, 3:zs // 2] = 2
    table = np.array([[1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7], [2, 20, 20, 20, 5e6, 5e6, 5e6]], np.float64)
    B, G = np.array([1e-3, -1e-3, 3e-3]), np.array([-0.05, 0, 0, 0, -0.05, 0, 0, 0, 0.1])
    runs = []
    for _ in range(2):
        with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1e-3, 1e-3, 1e-5, precision=precision)) as s:
            s.set_geometry_f64(geom.flatten(order="F"), table)
            s.steady([0.0, 0.0, 0.0], B, G)
            start = s.get_state()
            for _ in range(3):
                s.set_state(start)
                for _ in range(steps):
                    s.step([4.0, 0.0, 0.0], B, G)
                runs.append(s.get_state())
    for q in range(3):
        assert np.array_equal(runs[q], runs[q + 3]), q
