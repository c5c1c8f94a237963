"""Linked groups with vertex tables of different length, stepped from threads of their own: their launches
share kernels, and neither may set the other's limits."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def group(dim, seed, shuffle):
    """A p = 1 and a p = 2 handle, linked; with `shuffle` the elements keep a random order, so that
    a block of 128 touches up to 384 vertices instead of about 90."""
    from festung_gb300 import _lib as L
    from festung_gb300.solver import DeviceSolver
    from festung_gb300.testcases import jitter_coords, square_coords
    coordV, V0T, _, h = square_coords(1.0 / dim)
    coordV = jitter_coords(coordV, h, 0.1, seed)
    if shuffle:
        V0T = np.random.default_rng(seed).permutation(V0T)
    out = []
    for p in (1, 2):
        s = DeviceSolver(coordV, V0T, p, p + 1, precision='fp32', isSlopeLim=True,
                         flags=L.FLAG_NO_GRAPH | (L.FLAG_NO_REORDER if shuffle else 0))
        s.set_velocity_function((L.VEL_ROTATION, []))
        s.project_state((L.FN_GAUSS_SLOT, []), 0.0, 2 * p + 1)
        s.limit_state(0.0)
        out.append(s)
    out[0].link(out[1])
    return out


def run(groups, nSteps):
    from festung_gb300 import _lib as L
    failed = []

    def work(g):
        try:
            for n in range(nSteps // 50):
                g[0].step(50, 50 * n, 1e-4)
            g[0].sync()
        except L.DgadvError as e:
            failed.append(str(e))
    threads = [threading.Thread(target=work, args=(g,)) for g in groups]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    return [[s.get_state() for s in g] for g in groups]


def test_groups_of_different_tables_step_side_by_side(lib):
    what = [(16, 1, True), (16, 2, False), (16, 3, True), (16, 4, False)]
    both = []
    for together in (False, True):
        groups = [group(*w) for w in what]
        try:
            both.append(run(groups, 1000) if together else [run([g], 1000)[0] for g in groups])
        finally:
            for g in groups:
                for s in g:
                    s.close()
    for a, b in zip(*both):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
