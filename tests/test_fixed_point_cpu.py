"""The FP64 kernels' fixed-point sums (festung_gb300/csrc/dgadv_fixed.cuh) against FP64 multiply-add chains,
both against long double sums of the same terms, element by element and coefficient by coefficient.
The header runs on the host (fixed_point_host.cpp).

Bars.  Fixed point takes the place of FP64 sums, so its error has to be no larger: the root mean square
over a mesh of an element's error, relative to the element's result, at most that of the chain.  Every
coefficient on its own: at most 64 units of 2^-53 of the sum of its terms' magnitudes (the chain's bound
is one unit per term, 22 to 48), or, where that sum is far below the scales of its factors (a table entry
that happens to vanish at the one inflow point), half a unit of the element's largest such sum: the
scheme's bound for 12 terms is 31 2^-60 of the scales, a quarter of a unit.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from festung_gb300 import build as BLD
from festung_gb300.testcases import jitter_coords, slotted_cylinder, square_coords
from oracle import assembly as OA
from oracle import basis as OB
from oracle import grid as OG

EPS = 2.0 ** -53
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope='module')
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp('fx') / 'fixed_point_host.so')
    cuda = os.path.join(BLD._cuda_home(), 'include')
    subprocess.run(['g++', '-O2', '-std=c++17', '-shared', '-fPIC', '-ffp-contract=off', '-w', '-I', BLD.CSRC, '-I', cuda,
                    os.path.join(HERE, 'fixed_point_host.cpp'), os.path.join(BLD.CSRC, 'dgadv_host.cpp'), '-o', out],
                   check=True)
    return C.CDLL(out)


def mesh(dim, jitter=0.2):
    coordV, V0T, _, h = square_coords(1.0 / dim)
    return jitter_coords(coordV, h, jitter, 3), V0T


def state(m, p, data, seed=1):
    """Random coefficients, or the projection of a function."""
    coordV, V0T = m
    N = (p + 1) * (p + 2) // 2
    if data == 'random':
        return np.random.default_rng(seed).standard_normal((len(V0T), N))
    f = {'waves': lambda x, y: np.sin(7 * x) * np.cos(5 * y), 'offset': lambda x, y: 2 + np.sin(7 * x) * np.cos(5 * y),
         'hump': lambda x, y: np.exp(-((x - 0.3) ** 2 + (y - 0.5) ** 2) / 0.01),
         'slot': lambda x, y: slotted_cylinder(x, y) + np.exp(-60 * (x + y))}[data]
    g = OG.generateGridData(coordV, V0T)
    b = OB.computeBasesOnQuad(N)
    return OA.projectFuncCont2DataDisc(g, f, max(2 * p, 1), np.eye(N), b)


class Result:
    def __init__(self, K, N):
        self.value, self.fixed, self.fp64, self.size = (np.zeros((K, N)) for _ in range(4))
        self.taken = np.zeros(K, dtype=np.int32)

    def args(self):
        return [a.ctypes.data_as(C.c_void_p) for a in (self.value, self.fixed, self.fp64, self.size, self.taken)]

    def relative(self, err):
        """Every element's error relative to its result."""
        n = np.linalg.norm(self.value, axis=1)
        return np.linalg.norm(err, axis=1)[n > 0] / n[n > 0]


def call(fn, m, p, how, c, vscale=None):
    coordV, V0T = m
    xy = np.asfortranarray(coordV, dtype=np.float64).ravel(order='F')
    tri = np.asfortranarray(V0T, dtype=np.int32).ravel(order='F')
    c = np.ascontiguousarray(c, dtype=np.float64)
    r = Result(*c.shape)
    ptr = [a if a is None else a.ctypes.data_as(C.c_void_p) for a in (vscale, c)]
    mid = [ptr[1]] if fn.__name__ == 'fixed_point_limiter' else ptr
    assert fn(p, len(coordV), xy.ctypes.data_as(C.c_void_p), len(V0T), tri.ctypes.data_as(C.c_void_p), how, *mid,
              *r.args()) == 0
    return r


def rms(x):
    return float(np.sqrt(np.mean(x ** 2)))


def close(r, units=64):
    assert np.all(r.fixed <= EPS * (units * r.size + 0.5 * r.size.max(axis=1, keepdims=True)))


def no_less_accurate(r):
    assert rms(r.relative(r.fixed)) <= rms(r.relative(r.fp64))
    close(r)


@pytest.mark.parametrize('data', ['random', 'waves', 'offset', 'hump', 'slot'])
@pytest.mark.parametrize('velocity', [0, 1])
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_operator_is_no_less_accurate_than_fp64(host, p, velocity, data):
    m = mesh(24)
    r = call(host.fixed_point_operator, m, p, velocity, state(m, p, data))
    assert np.mean(r.taken) > 0.9
    no_less_accurate(r)
    if p:                                       # the mean's row on its own
        assert rms(r.fixed[:, 0] / (r.size[:, 0] + 1e-300)) <= rms(r.fp64[:, 0] / (r.size[:, 0] + 1e-300))


# Elements, neighbours and edge velocities of very different size side by side: each element's result
# keeps the accuracy of its own terms.
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_operator_with_scales_far_apart(host, p):
    m = mesh(16)
    K = len(m[1])
    r = np.random.default_rng(5)
    c = np.ldexp(state(m, p, 'random'), r.choice([0, -20, -40, -90], size=(K, 1)))
    v = np.ldexp(1.0, r.choice([0, -15, -50], size=3 * K)).astype(np.float64)
    q = call(host.fixed_point_operator, m, p, 1, c, v)
    assert np.all(q.taken)
    no_less_accurate(q)


# The mean far below or above the other coefficients.
@pytest.mark.parametrize('e', [-60, -30, 30, 60])
@pytest.mark.parametrize('p', [1, 2, 3])
def test_operator_with_a_mean_of_another_size(host, p, e):
    m = mesh(16)
    c = state(m, p, 'random')
    c[:, 0] = np.ldexp(c[:, 0], e)
    q = call(host.fixed_point_operator, m, p, 1, c)
    assert np.all(q.taken)
    no_less_accurate(q)


# Both sides of the exponent ranges: vectors 2^-700 .. 2^400, matrices 2^-200 .. 2^400; beyond them, and for
# an infinity or a NaN, the element is handed back.
@pytest.mark.parametrize('e,taken', [(-760, False), (-690, True), (380, True), (420, False)])
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_operator_at_the_ends_of_the_state_range(host, p, e, taken):
    m = mesh(4)
    c = np.sign(state(m, p, 'random'))
    q = call(host.fixed_point_operator, m, p, 1, np.ldexp(c, e))
    ref = call(host.fixed_point_operator, m, p, 1, c)
    assert np.all(q.taken == taken)
    if taken:                                   # powers of two scale every sum exactly
        assert np.array_equal(np.ldexp(q.value, -e), ref.value)


@pytest.mark.parametrize('e,taken', [(-230, False), (-180, True), (380, True), (420, False)])
@pytest.mark.parametrize('p', [0, 1, 2, 3])
def test_operator_at_the_ends_of_the_velocity_range(host, p, e, taken):
    m = mesh(4)
    c = state(m, p, 'random')
    v = np.full(3 * len(m[1]), 2.0 ** e)
    q = call(host.fixed_point_operator, m, p, 1, c, v)
    if p == 0:                                  # no volume term: the matrix scales with the edges
        assert np.all(q.taken == taken)
    elif not taken:
        assert not np.any(q.taken)
    no_less_accurate(q)


@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan, 5e-324])
@pytest.mark.parametrize('p', [1, 2, 3])
def test_operator_hands_back_what_it_cannot_hold(host, p, bad):
    m = mesh(4)
    for j in range((p + 1) * (p + 2) // 2):
        c = np.zeros((len(m[1]), (p + 1) * (p + 2) // 2))
        c[7, j] = bad
        q = call(host.fixed_point_operator, m, p, 1, c)
        assert not q.taken[7]
        assert q.taken[0] and np.all(q.value[0] == 0.0)


@pytest.mark.parametrize('data', ['random', 'waves', 'offset', 'hump', 'slot'])
@pytest.mark.parametrize('solution', [0, 1])
@pytest.mark.parametrize('p', [2, 3])
def test_limiter_is_no_less_accurate_than_fp64(host, p, solution, data):
    m = mesh(24)
    r = call(host.fixed_point_limiter, m, p, solution, state(m, p, data))
    assert np.mean(r.taken) > 0.9
    assert rms(r.relative(r.fixed)) <= rms(r.relative(r.fp64))


# States of any size, down to where an element is handed back, keep their means and slopes: a mean is a sum
# of N terms, a limited slope takes a factor with three roundings.
@pytest.mark.parametrize('e', [-40, -100, -399, -401, -410, -440, -450, -456, -470, -690, -720])
@pytest.mark.parametrize('solution', [0, 1])
@pytest.mark.parametrize('p', [2, 3])
def test_limiter_of_small_states(host, p, solution, e):
    m = mesh(8)
    c = np.ldexp(state(m, p, 'random') + 3.0 * (np.arange((p + 1) * (p + 2) // 2) == 0), e)
    r = call(host.fixed_point_limiter, m, p, solution, c)
    assert np.all(r.taken) or e < -690 or solution   # (a tiny slope times a tiny factor is handed back too)
    close(r, 16)


# Sums over a warp's lanes: shares alike, of one sign, decades apart, one far above the rest.
@pytest.mark.parametrize('data', ['normal', 'squares', 'decades', 'one'])
def test_lane_sums_are_no_less_accurate_than_fp64(host, data):
    r = np.random.default_rng(1)
    x = {'normal': r.standard_normal, 'squares': lambda s: r.standard_normal(s) ** 2,
         'decades': lambda s: np.exp(10 * r.standard_normal(s)),
         'one': lambda s: r.random(s) * np.where(np.arange(32) == 0, 1.0, 1e-6)}[data]((20000, 32))
    out = np.zeros(len(x))
    host.fixed_point_lane_sums(len(x), np.ascontiguousarray(x).ctypes.data_as(C.c_void_p),
                               out.ctypes.data_as(C.c_void_p))
    tree, exact = x, x.astype(np.longdouble).sum(axis=1)
    while tree.shape[1] > 1:
        tree = tree[:, :tree.shape[1] // 2] + tree[:, tree.shape[1] // 2:]
    size = np.abs(x).sum(axis=1)
    assert rms((out - exact) / size) <= rms((tree[:, 0] - exact) / size)
