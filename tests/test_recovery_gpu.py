"""Solves that turn non-finite: how they are reported, and that nothing of them stays behind.

A material whose coefficients overflow FP32 makes the inner operator infinite while the FP64 residual
stays finite: the solve enters its inner iteration and turns non-finite there.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZE = XS, YS, ZS = 33, 17, 12
SOUND = [1, 1, 1, 1, 3.5e7, 3.5e7, 3.5e7]
OVERFLOWS = [[1, 1e-33, 1e-33, 1e-33, 3.5e7, 3.5e7, 3.5e7], [1, 1e-40, 1e-40, 1e-40, 3.5e7, 3.5e7, 3.5e7],
             [1, 1, 1, 1, 1e36, 1e36, 1e36], [1, 1, 1, 1, 1e45, 1e45, 1e45]]
B, G, V = np.array([1e-3, -2e-3, 5e-3]), np.zeros(9), [-4.0, 0.0, 0.0]


def _geometry():
    geom = np.zeros(SIZE)
    geom[8:24, 5:12, 4:8] = 1
    return geom.flatten(order="F")


def _solver(**kw):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from alpineqms_gb300.solver import QMSSolver, default_desc
    return QMSSolver(default_desc(XS, YS, ZS, 1e-3, 1e-3, 1e-3, 1e-5, **kw))


def _non_finite_step(s, state, row):
    """A step from `state` with the material `row` ends as one that is not finite."""
    from alpineqms_gb300 import _lib
    s.set_geometry_f64(_geometry(), np.array([row], np.float64))
    s.set_state(state)
    with pytest.raises(_lib.QMSError):
        s.step(V, 0.9 * B, G)
    st = s.stats()
    assert st["status"] & _lib.QMS_STATUS_NAN and st["inner"] > 0, st


def _steady_state(s):
    s.set_geometry_f64(_geometry(), np.array([SOUND], np.float64))
    s.steady([0.0, 0.0, 0.0], B, G)
    return s.get_state()


@pytest.mark.parametrize("row", OVERFLOWS)
def test_a_state_that_is_not_finite_is_reported_as_such(row):
    with _solver() as s:
        _non_finite_step(s, _steady_state(s), row)


@pytest.mark.parametrize("row", OVERFLOWS[1:3])
@pytest.mark.parametrize("krylov,graphs", [(0, 1), (0, 0), (1, 1)])
def test_a_handle_solves_again_after_a_non_finite_solve(krylov, graphs, row):
    """XS - 1 = 32 and YS - 1 = 16 leave Dirichlet rows beyond the last tile, which only sums over whole
    vectors write.  The run after the non-finite solve is bit for bit that of a handle without one."""
    def run(s, state):
        s.set_geometry_f64(_geometry(), np.array([SOUND], np.float64))
        s.set_state(state)
        for scale in (0.9, 0.8, 0.8, 0.8, 0.8):
            st = s.step(V, scale * B, G)
            assert st["status"] == 0 and st["r"] <= s.desc.tol, st
        return s.get_state()

    with _solver(krylov=krylov, use_graphs=graphs) as s:
        state = _steady_state(s)
        ref = run(s, state)
    with _solver(krylov=krylov, use_graphs=graphs) as s:
        _non_finite_step(s, state, row)
        assert np.array_equal(run(s, state), ref)
