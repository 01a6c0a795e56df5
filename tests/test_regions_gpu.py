"""The conductor-region coarse space of the potential block with many bodies and bodies of many rows.

Its sums run over chunks of at most 1024 rows of one body.  A grid with one body of several chunks,
one just above a chunk, small ones and touching bodies of other conductivities (the modes the space is
for) must converge as with FP64 inner vectors: every step meets the tolerance in the exact FP64
residual (1.5 tol, the double-float residual's rounding below tol / 10), and repeated runs are equal
bit for bit (the sums' order is fixed).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("bodies,precision", [(1, "mixed"), (40, "mixed"), (40, "fp64")])
def test_steps_with_bodies_of_every_chunk_count(bodies, precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    xs, ys, zs = 40, 36, 34
    geom = np.zeros((xs, ys, zs))
    geom[4:26, 4:20, 4:16] = 1                       # 4224 cells: several chunks
    if bodies > 1:
        geom[4:14, 4:14, 16:27] = 2                  # touches body 1: about one chunk
        for q in range(3, bodies + 1):               # small bodies, some touching their neighbours
            i, j, k = 27 + 3 * (q % 4), 4 + 3 * (q // 4 % 9), 4 + 5 * (q % 5)
            geom[i:i + 3, j:j + 3, k:k + 3] = q
    rng = np.random.default_rng(5)
    table = np.array([[q, m, m, m, c, c, c] for q, m, c in
                      zip(range(1, bodies + 1), 10 ** rng.uniform(0, 2, bodies), 10 ** rng.uniform(5, 7.7, bodies))])
    B, G = np.array([2e-3, 1e-3, 4e-3]), np.zeros(9)
    states = []
    for _ in range(2):
        with QMSSolver(default_desc(xs, ys, zs, 1e-3, 1e-3, 1e-3, 2e-5, precision=precision)) as s:
            s.set_geometry_f64(geom.flatten(order="F"), table)
            s.steady([0.0, 0.0, 0.0], B, G)
            for scale in (0.8, 0.5):
                before = np.linalg.norm(s.get_state())
                st = s.step([0.0, 0.0, 0.0], scale * B, G)
                x = s.get_state()
                assert st["status"] == 0 and st["r"] <= s.desc.tol, st
                bound = 1.5 * s.desc.tol * max(before, np.linalg.norm(x))
                assert s.residual_norm(True, [0.0, 0.0, 0.0]) * np.linalg.norm(x) <= bound
            states.append(x)
    assert np.array_equal(states[0], states[1])
