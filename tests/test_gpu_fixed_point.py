"""The FP64 kernels' fixed-point sums (festung_gb300/csrc/dgadv_fixed.cuh) against plain FP64 arithmetic,
at the edges of their range: meshes around one block of 128 elements, every degree, states
scaled to the ends of the exponents the sums take and beyond them (those elements run in
FP64), exact zeros beside them, infinities and NaN.

Bars.  A fixed-point sum of n terms is off by about n 2^-57 of its scale, an FP64 chain by n 2^-53;
n <= 10 per row and at most 12 edge points, and neighbouring terms cancel to a few per cent of
their scale at these mesh widths: 100 * 22 * 2^-53 = 2.4e-13 between the two, 1e-12 is the
suite's FP64 bar.  Scaling a state by a power of two scales every FP64 operation exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def mesh(dim, jitter=0.2, seed=3):
    from festung_gb300.testcases import jitter_coords, square_coords
    coordV, V0T, _, h = square_coords(1.0 / dim)
    return jitter_coords(coordV, h, jitter, seed), V0T


def solver(dim, p, lim=False, elem=1, **kw):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    coordV, V0T = mesh(dim)
    s = DeviceSolver(coordV, V0T, p, min(p + 1, 3), precision='fp64', isSlopeLim=lim, **kw)
    s.set_option(L.OPT_ELEMENT_OPERATOR, elem)
    s.set_velocity_function((L.VEL_TRANSIENT, []))
    return s


def state(K, N, seed, zeros=False):
    c = np.random.default_rng(seed).standard_normal((K, N)) * 2.0 ** -np.arange(N)
    if zeros:
        c[K // 3:2 * K // 3] = 0.0
    return np.asfortranarray(c)


def step(s, c, tau):
    s.set_state(c)
    s.step(2, 0, tau)
    return s.get_state()


@pytest.mark.parametrize('dim', [1, 8, 9])        # 2, 128 and 162 elements
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_operator_matches_quadrature_form(lib, p, dim):
    c = state(2 * dim * dim, (p + 1) * (p + 2) // 2, p + dim, zeros=dim > 1)
    a, b = solver(dim, p), solver(dim, p, elem=0)
    try:
        assert rel(step(a, c, 1e-3), step(b, c, 1e-3)) <= TOL
    finally:
        a.close()
        b.close()


# the exponent range is 2^-400 .. 2^400: inside, at both ends, and past them (FP64)
@pytest.mark.parametrize('e', [-480, -401, -399, 300, 398, 402, 480])
@pytest.mark.parametrize('p', [1, 2, 3])
def test_operator_over_the_exponent_range(lib, p, e):
    c = state(2 * 81, (p + 1) * (p + 2) // 2, 5, zeros=True)
    s = solver(9, p)
    try:
        r = step(s, c, 1e-3)
        assert rel(np.ldexp(step(s, np.ldexp(c, e), 1e-3), -e), r) <= TOL
    finally:
        s.close()


def test_operator_with_sources_and_mixed_scales(lib):
    """Sources with the element operator on, and blocks of elements 600 binary orders apart."""
    K, N = 2 * 81, 6
    c = state(K, N, 7)
    c[:K // 2] = np.ldexp(c[:K // 2], -600)
    r = [state(K, N, 8), state(K, N, 9)]
    a, b = solver(9, 2), solver(9, 2, elem=0)
    try:
        for s in (a, b):
            s.set_source_terms([0, 1], r)
        assert rel(step(a, c, 1e-3), step(b, c, 1e-3)) <= TOL
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize('lim', [False, True])
def test_non_finite_state_is_reported(lib, bad, lim):
    from festung_gb300 import _lib as L
    s = solver(9, 2, lim)
    try:
        c = state(2 * 81, 6, 1)
        c[40, 0] = bad
        s.set_state(c)
        s.step(1, 0, 1e-3)
        with pytest.raises(L.DgadvError):
            s.sync()
    finally:
        s.close()


# one solution-limiter pass against the entry point that limits in plain FP64, means from 2^-40
# (every value below the limiter's tolerance) to 2^420 (past the range: FP64 there too)
@pytest.mark.parametrize('e', [-40, -8, 0, 16, 390, 420])
@pytest.mark.parametrize('p', [1, 2, 3])
def test_linear_limiter_matches_fp64_pass(lib, p, e):
    from test_zz_no_alloc import _case, _no_alloc, _with_handle
    cs = _case(1.0 / 9, p, seed=11 + p, jitter=0.2, with_data=True)
    cs['c'] = np.asfortranarray(np.ldexp(cs['c'], e))
    cs['data'] = np.asfortranarray(np.ldexp(cs['data'], e))
    assert rel(_with_handle(cs), _no_alloc(cs)) <= TOL


# ... and each element on its own, down to states of 2^-720: none loses its mean or what is left of its slopes
@pytest.mark.parametrize('e', [-399, -401, -410, -450, -470, -690, -720])
@pytest.mark.parametrize('p', [1, 2, 3])
def test_linear_limiter_of_small_states_element_by_element(lib, p, e):
    from test_zz_no_alloc import _case, _no_alloc, _with_handle
    cs = _case(1.0 / 9, p, seed=11 + p, jitter=0.2, with_data=True)
    cs['c'] = np.asfortranarray(np.ldexp(cs['c'], e))
    cs['data'] = np.asfortranarray(np.ldexp(cs['data'], e))
    a, b = (np.ldexp(x, -e) for x in (_with_handle(cs), _no_alloc(cs)))
    assert np.all(np.linalg.norm(a - b, axis=1) <= TOL * np.linalg.norm(b, axis=1))


# the range of the matrices, 2^-200 .. 2^400: a velocity scaled by a power of two and the step by its inverse
@pytest.mark.parametrize('e', [-230, -201, -180, 380, 420])
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_operator_over_the_velocity_range(lib, p, e):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    coordV, V0T = mesh(9)
    K, N = len(V0T), (p + 1) * (p + 2) // 2
    vn = np.repeat(L.grid_build(coordV, V0T)['nuE0T'].sum(axis=2)[:, :, None], p + 1, axis=2)
    c, out = state(K, N, 6), []
    for sc in (0, e):
        s = DeviceSolver(coordV, V0T, p, min(p + 1, 3), precision='fp64', isSlopeLim=False)
        try:
            u = np.zeros((K, N), order='F')
            u[:, 0] = 2.0 ** sc / np.sqrt(2)
            s.set_velocity(u, u, np.asfortranarray(np.ldexp(vn, sc)))
            out.append(step(s, c, 1e-3 * 2.0 ** -sc))
        finally:
            s.close()
    assert rel(out[1], out[0]) <= TOL


# The time-derivative limiter's sums in fixed point against its FP64 form (the correction rebuilt from the
# mesh, whose tables differ by rounding; a derivative of order 3 carries 1e-11 of the mean from them)
@pytest.mark.parametrize('e', [-720, -460, -40, 0, 390, 420])
@pytest.mark.parametrize('p', [2, 3])
def test_derivative_limiter_matches_fp64_form(lib, p, e):
    from festung_gb300 import _lib as L
    out = []
    for fly in (0, 1):
        s = solver(9, p, lim=True)
        try:
            s.set_option(L.OPT_TAYLOR_MASS, fly)
            c = state(2 * 81, (p + 1) * (p + 2) // 2, 5)
            c[:, 0] += 3.0
            out.append(step(s, np.ldexp(c, e), 1e-3))
        finally:
            s.close()
    a, b = (np.ldexp(x, -e) for x in out)
    assert np.all(np.linalg.norm(a - b, axis=1) <= 1e-10 * np.linalg.norm(b, axis=1))


# Blocks with more vertices than threads: elements in random order (NO_REORDER keeps it), so 128 of
# them touch up to 384 vertices.  Minima and maxima do not depend on the order, and an
# element's arithmetic does not either: bitwise equal to the library's own order.
@pytest.mark.parametrize('precision,p,lim', [('fp32', 1, 'linear'), ('fp32', 3, 'hierarch_vert'),
                                             ('fp32', 2, 'strict'), ('fp64', 2, 'linear'),
                                             ('fp64', 3, 'hierarch_vert'), ('df32', 2, 'linear')])
def test_block_vertex_tables(lib, precision, p, lim):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    coordV, V0T = mesh(20)
    V0T = np.random.default_rng(2).permutation(V0T)
    out = []
    for flags in (0, L.FLAG_NO_REORDER):
        s = DeviceSolver(coordV, V0T, p, min(p + 1, 3), precision=precision, isSlopeLim=True, typeSlopeLim=lim,
                         flags=flags)
        try:
            s.set_velocity_function((L.VEL_ROTATION, []))
            s.project_state((L.FN_GAUSS_SLOT, []), 0.0, 2 * p + 1)
            s.limit_state(0.0)
            s.step(4, 0, 1e-3)
            out.append(s.get_state())
        finally:
            s.close()
    assert np.array_equal(out[0], out[1])


# Lists between the two: the caller's rows (NO_REORDER), three vertex lines of 65 per 128 elements.  The
# Taylor limiters then read every element's own keys, the library's own order has tables.
@pytest.mark.parametrize('precision,p,lim', [('fp32', 2, 'hierarch_vert'), ('fp32', 3, 'strict'), ('df32', 2, 'strict'),
                                             ('df32', 3, 'hierarch_vert'), ('fp64', 2, 'hierarch_vert'),
                                             ('fp64', 3, 'strict')])
def test_block_vertex_tables_in_row_order(lib, precision, p, lim):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    coordV, V0T = mesh(64)
    out = []
    for flags in (0, L.FLAG_NO_REORDER):
        s = DeviceSolver(coordV, V0T, p, min(p + 1, 3), precision=precision, isSlopeLim=True, typeSlopeLim=lim,
                         flags=flags)
        try:
            s.set_velocity_function((L.VEL_ROTATION, []))
            s.project_state((L.FN_GAUSS_SLOT, []), 0.0, 2 * p + 1)
            s.limit_state(0.0)
            s.step(3, 0, 1e-4)
            out.append(s.get_state())
        finally:
            s.close()
    assert np.array_equal(out[0], out[1])


# Species share their launches; each must come out as if it ran alone, also on a handle whose
# buffers an earlier, larger set of species left behind.
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
def test_transported_species_do_not_mix(lib, precision):
    from festung_gb300 import transport_gpu as GT

    def run(sets):
        pd = GT.Struct(hmax=1.0 / 9, p=1, numSpecies=max(map(len, sets)), numSteps=6, tEnd=6 * 4e-3, precision=precision)
        GT.configureProblem(pd)
        GT.preprocessProblem(pd)
        K = pd.K
        h = np.zeros((K, 3), order='F')
        h[:, 0] = 0.1 / np.sqrt(2)
        got = []
        for members in sets:
            cH = np.zeros((K, 3, len(members)), order='F')
            for i, m in enumerate(members):
                cH[:, 0, i] = (np.random.default_rng(m).random(K) > 0.7) * (m + 1.0)
            pd.solver.transport_init(h, cH, 1e-6, True)
            pd.solver.transport_step(pd.numSteps, 0, pd.tau)
            got.append([pd.solver.transport_get(i) for i in range(len(members))])
        pd.solver.close()
        return got
    together, fewer = run([[0, 1, 2, 3, 4], [3, 1]])
    for m in range(5):
        alone = run([[m]])[0][0]
        for a, b in zip(together[m], alone):
            assert np.array_equal(a, b)
    for i, m in enumerate([3, 1]):
        for a, b in zip(fewer[i], together[m]):
            assert np.array_equal(a, b)


# The implicit solver's Arnoldi step takes the local part of A P^-1 for the identity, except where a
# diagonal block has no inverse: an element without any velocity, in the stationary problem.
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_implicit_with_singular_blocks(lib, p):
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    coordV, V0T = mesh(5, jitter=0.1)
    K, N = len(V0T), (p + 1) * (p + 2) // 2
    s = DeviceSolver(coordV, V0T, p, 1, precision='fp64', flags=L.FLAG_IMPLICIT)
    try:
        still = np.arange(K) < 6
        u1, u2 = np.zeros((K, N), order='F'), np.zeros((K, N), order='F')
        u1[~still, 0] = u2[~still, 0] = 1.0 / np.sqrt(2)
        g = L.grid_build(coordV, V0T)
        vn = np.repeat((g['nuE0T'].sum(axis=2) * ~still[:, None])[:, :, None], p + 1, axis=2)
        s.set_velocity(u1, u2, np.asfortranarray(vn))
        rhs = state(K, N, 4) * ~still[:, None]
        s.set_source_terms([0], [np.asfortranarray(rhs)])
        s.set_state(np.zeros((K, N), order='F'))
        it, res = s.solve_stationary(tol=1e-10, restart=200)
        assert res <= 1e-10 and it > 0          # the residual of the whole operator
        x = s.get_state()
        assert np.all(x[still] == 0.0) and np.linalg.norm(x[~still]) > 0
    finally:
        s.close()
