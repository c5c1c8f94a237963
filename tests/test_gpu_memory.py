"""Device memory that runs out: what the kernels can do without is left out, what they need fails the
call, and a later call, with room again, starts over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def hold_all_but(torch, leave):
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device='cuda')


def release(torch, held):
    del held[:]
    torch.cuda.empty_cache()


def test_fixed_point_digits_do_without_room(lib):
    """131072 triangles, p = 2, linear limiter: 50 MB of digits of the element operator that do not fit, nor
    then the 25 MB of the source terms' second form."""
    torch = pytest.importorskip('torch')
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    from festung_gb300.testcases import square_coords
    coordV, V0T = square_coords(1.0 / 256)[:2]
    K, N = len(V0T), 6
    c = np.asfortranarray(np.random.default_rng(1).standard_normal((K, N)) * 2.0 ** -np.arange(N))
    rhs = np.asfortranarray(np.random.default_rng(2).standard_normal((K, N)) * 1e-3)

    def run():
        s = DeviceSolver(coordV, V0T, 2, 3, precision='fp64', isSlopeLim=True)
        try:
            s.set_velocity_function((L.VEL_TRANSIENT, []))
            s.set_state(c)
            s.step(3, 0, 1e-5)
            a = s.get_state()
            s.set_source_terms([0], [rhs])
            s.set_state(c)
            s.step(3, 0, 1e-5)
            return a, s.get_state(), torch.cuda.mem_get_info()[0]
        finally:
            s.close()
    run()                                         # modules loaded
    free = torch.cuda.mem_get_info()[0]
    a, b, left = run()
    held = [hold_all_but(torch, free - left - 60 * 2 ** 20)]
    try:
        x, y, _ = run()
    finally:
        release(torch, held)
    for p, q in ((x, a), (y, b)):
        assert np.linalg.norm(p - q) <= TOL * np.linalg.norm(q)


def test_a_failed_allocation_stays_with_its_call(lib):
    """The error of one handle's call does not surface in the next handle's."""
    torch = pytest.importorskip('torch')
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    from festung_gb300.testcases import square_coords
    coordV, V0T = square_coords(1.0 / 512)[:2]
    held = [hold_all_but(torch, 48 * 2 ** 20)]
    try:
        with pytest.raises(L.DgadvError):
            DeviceSolver(coordV, V0T, 3, 3, precision='fp64', isSlopeLim=True)
    finally:
        release(torch, held)
    s = DeviceSolver(*square_coords(1.0 / 8)[:2], 1, 2, precision='fp64', isSlopeLim=False)
    try:
        s.set_velocity_function((L.VEL_ROTATION, []))
    finally:
        s.close()


def test_implicit_step_after_memory_ran_out(lib):
    torch = pytest.importorskip('torch')
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    from festung_gb300.testcases import square_coords
    coordV, V0T = square_coords(1.0 / 64)[:2]
    K, N = len(V0T), 6
    c = np.asfortranarray(np.random.default_rng(1).standard_normal((K, N)) * 2.0 ** -np.arange(N))
    out = []
    for squeeze in (False, True):
        s = DeviceSolver(coordV, V0T, 2, 1, precision='fp64', flags=L.FLAG_IMPLICIT)
        try:
            s.set_velocity_function((L.VEL_ROTATION, []))
            s.set_state(c)
            s.sync()
            if squeeze:                           # 256 vectors take 100 MB
                held = [hold_all_but(torch, 32 * 2 ** 20)]
                try:
                    with pytest.raises(L.DgadvError):
                        s.step_implicit(1, 0, 0.02, 1, restart=256)
                finally:
                    release(torch, held)
            s.step_implicit(1, 0, 0.02, 1, restart=256)
            out.append(s.get_state())
        finally:
            s.close()
    assert np.array_equal(out[0], out[1])


def test_transport_after_memory_ran_out(lib):
    torch = pytest.importorskip('torch')
    from festung_gb300 import _lib as L
    from festung_gb300 import transport_gpu as GT
    out = []
    for squeeze in (False, True):
        pd = GT.Struct(hmax=1.0 / 256, p=1, numSpecies=4, numSteps=4, tEnd=4e-4, precision='fp64')
        GT.configureProblem(pd)
        GT.preprocessProblem(pd)
        h = np.zeros((pd.K, 3), order='F')
        h[:, 0] = 0.1 / np.sqrt(2)
        cH = np.zeros((pd.K, 3, 4), order='F')
        cH[:, 0, :] = np.random.default_rng(3).random((pd.K, 4)) > 0.7
        try:
            if squeeze:                           # c h, concentrations and work of four species take 50 MB
                held = [hold_all_but(torch, 24 * 2 ** 20)]
                try:
                    with pytest.raises(L.DgadvError):
                        pd.solver.transport_init(h, cH, 1e-6, True)
                    with pytest.raises(L.DgadvError):
                        pd.solver.transport_step(1, 0, 1e-4)
                finally:
                    release(torch, held)
            pd.solver.transport_init(h, cH, 1e-6, True)
            pd.solver.transport_step(4, 0, 1e-4)
            out.append([pd.solver.transport_get(i) for i in range(4)])
        finally:
            pd.solver.close()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
