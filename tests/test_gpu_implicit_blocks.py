"""The implicit solver on meshes with diagonal blocks that are singular up to rounding: elements whose
edges carry no flow while their inside does.  The mean then stands in no equation of its block (a row of
rounding), and elimination leaves a pivot of that size; the systems stay solvable, as the right-hand
sides have no mean there.

Bar: the solver's own tolerance on the relative residual of the whole operator.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision,tol', [('fp64', 1e-10), ('fp32', 1e-4)])
@pytest.mark.parametrize('p', [1, 2, 3])
def test_blocks_singular_up_to_rounding(lib, p, precision, tol):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    from festung_gb300.testcases import jitter_coords, square_coords
    coordV, V0T, dim, h = square_coords(1.0 / 7)
    cell = np.floor(coordV[V0T].mean(axis=1) * dim).astype(int) % 3
    coordV = jitter_coords(coordV, h, 0.1, 3)
    K, N = len(V0T), (p + 1) * (p + 2) // 2
    r = np.random.default_rng(4)
    closed = np.all(cell == 1, axis=1)          # both triangles of squares apart: every other element keeps an outflow
    g = L.grid_build(coordV, V0T)
    edges = np.unique(g['E0T'][closed])
    vn = np.where(np.isin(g['E0T'], edges), 0.0, g['nuE0T'].sum(axis=2) / np.sqrt(2))
    u1, u2 = (np.asfortranarray(a) for a in r.standard_normal((2, K, N)) * 2.0 ** -np.arange(N))
    u1[~closed], u2[~closed] = 0.0, 0.0
    u1[~closed, 0] = u2[~closed, 0] = 0.5
    rhs = r.standard_normal((K, N))
    rhs[closed, 0] = 0.0
    s = DeviceSolver(coordV, V0T, p, 1, precision=precision, flags=L.FLAG_IMPLICIT)
    try:
        s.set_velocity(u1, u2, np.asfortranarray(np.repeat(vn[:, :, None], p + 1, axis=2)))
        s.set_source_terms([0], [np.asfortranarray(rhs)])
        s.set_state(np.zeros((K, N), order='F'))
        it, res = s.solve_stationary(tol=tol, restart=200)
        assert res <= tol and it > 0
        assert np.all(np.isfinite(s.get_state()))
    finally:
        s.close()
