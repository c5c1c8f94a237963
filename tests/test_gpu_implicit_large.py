"""The implicit solver on a mesh with more groups of 32 elements than its sums have blocks: every block
adds several groups.  The solution of one implicit Euler step is put into the explicit solver's operator,
which shares no code with the implicit one: x - tau cDot(x) has to give the state before the step.  With
a constant velocity both problems' quadrature is exact.

Bar: the solver's residual tolerance of 1e-12, times the 1e2 by which the difference of two Euler states
loses digits at this step size.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dim', [139, 150])       # 1208 and 1407 groups; 1216 blocks
@pytest.mark.parametrize('p', [0, 1, 2])
def test_implicit_euler_step_solves_the_explicit_operator(lib, p, dim):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    from festung_gb300.testcases import jitter_coords, square_coords
    coordV, V0T, _, h = square_coords(1.0 / dim)
    coordV = jitter_coords(coordV, h, 0.1, 3)
    K, N = len(V0T), (p + 1) * (p + 2) // 2
    c = np.asfortranarray(np.random.default_rng(2).standard_normal((K, N)) * 2.0 ** -np.arange(N))
    g = L.grid_build(coordV, V0T)
    vn = np.asfortranarray(np.repeat((g['nuE0T'] @ [0.6, 0.8])[:, :, None], p + 1, axis=2))
    u1, u2 = np.zeros((K, N), order='F'), np.zeros((K, N), order='F')
    u1[:, 0], u2[:, 0] = 0.6 / np.sqrt(2), 0.8 / np.sqrt(2)
    tau = 1.0 / dim
    impl = DeviceSolver(coordV, V0T, p, 1, precision='fp64', flags=L.FLAG_IMPLICIT)
    expl = DeviceSolver(coordV, V0T, p, 1, precision='fp64', isSlopeLim=False)
    try:
        for s in (impl, expl):
            s.set_velocity(u1, u2, vn)
        impl.set_state(c)
        it, res = impl.step_implicit(1, 0, tau, 1, tol=1e-12)
        x = impl.get_state()
        assert res <= 1e-12 and it > 0
        expl.set_state(x)
        expl.step(1, 0, tau)
        back = 2.0 * x - expl.get_state()
        assert np.linalg.norm(back - c) <= 1e-10 * np.linalg.norm(c)
    finally:
        impl.close()
        expl.close()
