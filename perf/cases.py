"""The work this library does for its users, as cases to be timed.

Every case goes through the package's public entry points: the ``DeviceSolver`` calls, the step
functions of the ``advection_gpu``, ``advection_implicit_gpu`` and ``transport_gpu`` problems,
``Ensemble`` and ``adjoint.misfit_gradient``.  One pass hands over the initial coefficients, runs
some time steps and reads the result back, as a program does between two outputs.

``exact`` is a restatement of the same discrete problems in plain torch, FP64: the DG operator of
degree p on triangles with upwind fluxes, SSP-RK / DIRK steps, the vertex-based Taylor limiters,
the masked transport of several species, and gradients by automatic differentiation.
"""
import math

import numpy as np
import torch

from festung_gb300 import _lib as L
from festung_gb300 import adjoint as ADJ
from festung_gb300 import advection_gpu as G
from festung_gb300 import advection_implicit_gpu as GI
from festung_gb300 import ensemble as ENS
from festung_gb300 import transport_gpu as GT
from festung_gb300.solver import DeviceSolver

ENSEMBLE_TAU = 2e-4
FLOAT_BYTES = {'fp64': 8, 'df32': 8, 'fp32': 4}


# ---------------------------------------------------------------------------------------------
# The cases
def listed():
    return [
        # The reference's own loop, main('advection', ...): one call per time step, on the small
        # mesh of its plain configuration (2048 triangles, p = 1, SSP-RK2, limiter on).
        dict(name='loop_2k_p1_fp64', kind='loop', dim=32, p=1, steps=50),
        # Production size in the reference's precision: 131072 triangles, p = 2, SSP-RK3, linear
        # limiter, rotating hump and slotted cylinder.
        dict(name='solve_131k_p2_fp64', kind='solve', dim=256, jitter=0.0, p=2, limiter='linear',
             precision='fp64', velocity='rotation', steps=50),
        # The same in single precision, where the mesh lives in the L2 cache.
        dict(name='solve_131k_p2_fp32', kind='solve', dim=256, jitter=0.0, p=2, limiter='linear',
             precision='fp32', velocity='rotation', steps=60),
        # Double-float on an odd, jittered mesh (34322 triangles, not a multiple of a block).
        dict(name='solve_34k_p2_df32', kind='solve', dim=131, jitter=0.1, p=2, limiter='linear',
             precision='df32', velocity='stream', steps=50),
        # A mesh whose data come from HBM: 2,097,152 triangles, p = 2, single precision.
        dict(name='solve_2M_p2_fp32', kind='solve', dim=1024, jitter=0.0, p=2, limiter='linear',
             precision='fp32', velocity='rotation', steps=20),
        # The large jittered mesh with p = 3 and the hierarchical limiter, a quarter of its size.
        dict(name='solve_524k_p3_hier_fp32', kind='solve', dim=512, jitter=0.1, p=3,
             limiter='hierarch_vert', precision='fp32', velocity='rotation', steps=8),
        # A convergence study's run: analytical solution with source and boundary data that change
        # in time, odd mesh (6498 triangles), error against the exact solution at the end.
        dict(name='transient_6k_p2_fp64', kind='transient', dim=57, p=2, steps=30),
        # An ensemble of uneven instances (2048 to 32768 triangles, p = 1 and 2) in FP32.
        dict(name='ensemble_24_fp32', kind='ensemble', count=24, steps=60),
        # Gradients of a misfit with respect to initial data and velocity: few snapshots in FP64,
        # every stage stored in FP32.
        dict(name='grad_32k_p2_fp64', kind='grad', dim=128, p=2, precision='fp64', steps=60, snapshots=10),
        dict(name='grad_32k_p2_fp32', kind='grad', dim=128, p=2, precision='fp32', steps=100, snapshots=0),
        # Implicit steps of the reference's default size: 8192 triangles, p = 2, DIRK3.
        dict(name='implicit_8k_p2_fp64', kind='implicit', dim=64, p=2, ordRK=3, precision='fp64', steps=4),
        # Masked transport of four species, the reference's default size (8192 triangles, p = 1).
        dict(name='transport_8k_p1_4sp_fp64', kind='transport', dim=64, p=1, species=4,
             precision='fp64', steps=40),
    ]


def draw(rng):
    kind = rng.choice(['loop', 'solve', 'solve', 'solve', 'solve', 'transient', 'ensemble', 'grad',
                       'implicit', 'transport'])

    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    if kind == 'loop':
        return dict(kind=kind, dim=log_int(10, 128), p=rng.choice([1, 2]), steps=rng.randint(10, 60))
    if kind == 'solve':
        p = rng.choice([0, 1, 1, 2, 2, 2, 3])
        precision = rng.choice(['fp64', 'fp32', 'fp32', 'df32'])
        # without a limiter, or the one the degree and the precision are run with
        limiter = 'none' if p == 0 else rng.choice(['none', 'linear', 'linear'])
        if p >= 2 and precision == 'fp32' and rng.random() < 0.3:
            limiter = 'hierarch_vert'
        dim = log_int(24, 400 if precision == 'fp32' else 200)
        return dict(kind=kind, dim=dim, jitter=rng.choice([0.0, 0.1, 0.2]), p=p, limiter=limiter,
                    precision=precision, velocity=rng.choice(['rotation', 'stream']),
                    steps=rng.randint(4, 10) if limiter == 'hierarch_vert' else rng.randint(5, 40))
    if kind == 'transient':
        return dict(kind=kind, dim=log_int(12, 100), p=rng.choice([1, 2]), steps=rng.randint(5, 30))
    if kind == 'ensemble':
        return dict(kind=kind, count=rng.randint(4, 24), steps=rng.randint(10, 60))
    if kind == 'grad':
        return dict(kind=kind, dim=log_int(16, 128), p=rng.choice([1, 2]), precision=rng.choice(['fp64', 'fp32']),
                    steps=rng.randint(10, 60), snapshots=rng.choice([0, 5, 10]))
    if kind == 'implicit':
        return dict(kind=kind, dim=log_int(12, 90), p=rng.choice([1, 2]), ordRK=rng.choice([1, 2, 3, 4]),
                    precision='fp64', steps=rng.randint(1, 4))
    return dict(kind=kind, dim=log_int(12, 90), p=rng.choice([1, 2]), species=rng.randint(1, 5),
                precision='fp64', steps=rng.randint(5, 40))


# ---------------------------------------------------------------------------------------------
# Inputs: meshes, velocities and initial data, from the case and the seed
def square_mesh(dim, jitter=0.0, seed=0):
    """The unit square in 2 dim^2 triangles (the reference's domainSquare), interior vertices moved
    by up to jitter / dim."""
    n = dim + 1
    v = np.arange(n) * (1.0 / dim)
    v[-1] = 1.0
    xy = np.stack([np.repeat(v, n), np.tile(v, n)], axis=1)
    if jitter > 0:
        d = np.random.default_rng(seed).uniform(-1.0, 1.0, size=xy.shape) * (jitter * (1.0 / dim))
        inner = (xy[:, 0] > 0) & (xy[:, 0] < 1) & (xy[:, 1] > 0) & (xy[:, 1] < 1)
        xy[inner] += d[inner]
    r = (np.arange(dim)[:, None] * n + np.arange(dim)[None, :]).ravel()
    tri = np.concatenate([np.stack([r, r + n, r + 1], 1), np.stack([r + n, r + n + 1, r + 1], 1)])
    return xy, tri.astype(np.int64)


def humps(seed, amplitude=1.0):
    """A Gaussian hump and a slotted cylinder at seeded places, turned about the centre."""
    r = np.random.default_rng([int(seed), 71])
    ang, width = r.uniform(0, 2 * math.pi), r.uniform(0.06, 0.12)
    co, si = math.cos(ang), math.sin(ang)

    def c0(x, y):
        a, b = co * (x - 0.5) + si * (y - 0.5) + 0.5, -si * (x - 0.5) + co * (y - 0.5) + 0.5
        hump = (-((a - 0.25) ** 2 + (b - 0.5) ** 2) / width ** 2)
        exp = torch.exp if isinstance(x, torch.Tensor) else np.exp
        slot = ((a - 0.5) ** 2 + (b - 0.75) ** 2 <= 0.0225) & ((abs(a - 0.5) >= 0.025) | (b >= 0.85))
        return amplitude * (exp(hump) + slot * 1.0)
    return c0


def smooth(seed):
    """Two Gaussian humps at seeded places."""
    r = np.random.default_rng([int(seed), 72])
    q = r.uniform(0.3, 0.7, size=4)

    def c0(x, y):
        exp = torch.exp if isinstance(x, torch.Tensor) else np.exp
        return (exp(-((x - q[0]) ** 2 + (y - q[1]) ** 2) / 0.01)
                + 0.5 * exp(-((x - q[2]) ** 2 + (y - q[3]) ** 2) / 0.02))
    return c0


def stream_modes(seed):
    """A streamfunction of eight seeded modes: (k, l, amplitude)."""
    r = np.random.default_rng([int(seed), 73])
    return r.integers(1, 4, size=8), r.integers(1, 4, size=8), r.normal(0.0, 0.1, size=8)


def stream_velocity(k, l, a):
    def u1(x, y):
        lib = torch if isinstance(x, torch.Tensor) else np
        return sum(am * lm * math.pi * lib.sin(km * math.pi * x) * lib.cos(lm * math.pi * y)
                   for km, lm, am in zip(map(float, k), map(float, l), map(float, a)))

    def u2(x, y):
        lib = torch if isinstance(x, torch.Tensor) else np
        return -sum(am * km * math.pi * lib.cos(km * math.pi * x) * lib.sin(lm * math.pi * y)
                    for km, lm, am in zip(map(float, k), map(float, l), map(float, a)))
    return u1, u2


def rotation():
    return (lambda x, y: 0.5 - y), (lambda x, y: x - 0.5)


def instance(seed):
    """What one seeded instance of the 'ensemble' test case draws: mesh level, degree,
    streamfunction, mesh seed."""
    r = np.random.default_rng(seed)
    d = dict(seed=seed, level=int(r.choice([5, 6, 7])), p=int(r.choice([1, 2])))
    d['k'], d['l'], d['a'] = r.integers(1, 4, size=8), r.integers(1, 4, size=8), r.normal(0.0, 0.1, size=8)
    r.uniform(0.2, 0.8, size=2), r.uniform(0.05, 0.15)
    d['mesh'] = int(r.integers(0, 2 ** 31 - 1))
    return d


MIX = [(5, 1), (6, 2), (7, 1), (5, 2), (6, 1), (7, 2)]   # (level, degree) of an ensemble's instances


def instances(count, seed):
    """`count` instances of the mix, the first ones that a count-up from the seed meets."""
    out, s = [], 100000 * (int(seed) % 20000) + 1
    for i in range(count):
        while True:
            d = instance(s)
            s += 1
            if (d['level'], d['p']) == MIX[i % len(MIX)]:
                out.append(d)
                break
    return out


def pinned(a):
    """A K x N array in column-major order, in pinned host memory."""
    t = torch.from_numpy(np.ascontiguousarray(a.T))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy().T


def host_projection(xy, tri, p, f):
    """L2 projection of f on every triangle (volume rule of order 2p), K x N."""
    q1, q2, w = rule2(max(2 * p, 1))
    x = [xy[tri[:, n]] for n in range(3)]
    px = x[0][:, None, 0] + (x[1] - x[0])[:, None, 0] * q1 + (x[2] - x[0])[:, None, 0] * q2
    py = x[0][:, None, 1] + (x[1] - x[0])[:, None, 1] * q1 + (x[2] - x[0])[:, None, 1] * q2
    return f(px, py) @ (w[:, None] * basis(p, q1, q2)[0])


def species_fields(case, seed):
    """Initial c h of every species: discs around seeded centres, scaled by the species index."""
    r = np.random.default_rng([int(seed), 74])
    at = r.uniform(0.25, 0.75, size=(case['species'], 3, 2))

    def field(s):
        def f(x, y):
            on = sum((((x - cx) ** 2 + (y - cy) ** 2) <= 0.0225 / math.sqrt(2)) * 1.0 for cx, cy in at[s])
            return (s + 1) * 0.1 * on
        return f
    return [field(s) for s in range(case['species'])]


def transient_data():
    """The reference's analytical case: velocity, solution, and sources as (g(t), f(x, y))."""
    def lib(x):
        return torch if isinstance(x, torch.Tensor) else np
    u1 = lambda x, y: lib(x).exp(0.5 * (x + y))   # noqa: E731
    u2 = lambda x, y: lib(x).exp(0.5 * (x - y))   # noqa: E731
    cc = lambda x, y: lib(x).cos(7 * x) * lib(x).cos(7 * y)   # noqa: E731
    adv = lambda x, y: (-7 * u1(x, y) * lib(x).sin(7 * x) * lib(x).cos(7 * y)   # noqa: E731
                        - 7 * u2(x, y) * lib(x).cos(7 * x) * lib(x).sin(7 * y)
                        + 0.5 * (u1(x, y) - u2(x, y)) * cc(x, y))
    decay = lambda x, y: -1 + 0.5 * (u1(x, y) - u2(x, y))   # noqa: E731
    return u1, u2, cc, adv, decay


def ord_rk(p):
    return min(p + 1, 3)


def tau_of(case):
    """The benchmark's step size on its meshes, scaled with the mesh width."""
    return 0.0256 / case['dim'] if case['kind'] != 'transport' else 2 * math.pi / 3142 * 64 / max(case['dim'], 64)


# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case['kind']
    if kind == 'loop':
        pd = G.Struct(testcase='gauss_slot', hmax=1.0 / case['dim'], p=case['p'], isSlopeLim=True,
                      numSteps=case['steps'], tEnd=case['steps'] * tau_of(case))
        G.configureProblem(pd)
        G.preprocessProblem(pd)
        xy, tri = square_mesh(case['dim'])
        return dict(kind=kind, pd=pd, c0=pinned(host_projection(xy, tri, case['p'], humps(seed))))
    if kind == 'solve':
        xy, tri = square_mesh(case['dim'], case['jitter'], 5)
        p = case['p']
        s = DeviceSolver(xy, tri, p, ord_rk(p), precision=case['precision'], isSlopeLim=case['limiter'] != 'none',
                         typeSlopeLim=case['limiter'] if case['limiter'] != 'none' else 'linear')
        if case['velocity'] == 'rotation':
            s.set_velocity_function((L.VEL_ROTATION, []))
        else:
            s.set_velocity_function((L.VEL_STREAM, np.concatenate(stream_modes(seed)).astype(np.float64)))
        c0 = pinned(host_projection(xy, tri, p, humps(seed)))
        return dict(kind=kind, solver=s, c0=c0, out=pinned(np.zeros_like(c0)), steps=case['steps'],
                    tau=tau_of(case), limit=case['limiter'] != 'none', single=case['precision'] == 'fp32')
    if kind == 'transient':
        pd = G.Struct(testcase='transient', hmax=1.0 / case['dim'], p=case['p'], isSlopeLim=True,
                      numSteps=case['steps'], tEnd=case['steps'] * tau_of(case))
        G.configureProblem(pd)
        G.preprocessProblem(pd)
        xy, tri = square_mesh(case['dim'])
        c0, extra = transient_data()[2], smooth(seed)
        return dict(kind=kind, pd=pd, c0=pinned(host_projection(
            xy, tri, case['p'], lambda x, y: c0(x, y) + 1.0 + extra(x, y))))
    if kind == 'ensemble':
        insts = instances(case['count'], seed)
        e = ENS.Ensemble([d['seed'] for d in insts], precision='fp32', tau=ENSEMBLE_TAU)
        c0 = {}
        for p, members in e.groups.items():
            c0[p] = pinned(np.concatenate([host_projection(*square_mesh(2 ** insts[i]['level'], 0.2, insts[i]['mesh']),
                                                           p, smooth(insts[i]['seed'])) for i in members]))
        return dict(kind=kind, ensemble=e, c0=c0, steps=case['steps'])
    if kind == 'grad':
        r = np.random.default_rng([int(seed), 75])
        pd = ADJ.setup(hmax=1.0 / case['dim'], p=case['p'], precision=case['precision'], numSteps=case['steps'],
                       tEnd=case['steps'] * tau_of(case))
        xy, tri = square_mesh(case['dim'])
        return dict(kind=kind, pd=pd, theta=r.normal(0.0, 0.04, size=16), snapshots=case['snapshots'],
                    c0=pinned(host_projection(xy, tri, case['p'], smooth(seed))),
                    target=pinned(host_projection(xy, tri, case['p'], smooth(seed + 1))),
                    single=case['precision'] == 'fp32')
    if kind == 'implicit':
        pd = GI.Struct(testcase='solid_body', hmax=1.0 / case['dim'], p=case['p'], ordRK=case['ordRK'],
                       precision=case['precision'], numSteps=320, tEnd=320 * implicit_tau(case))
        GI.configureProblem(pd)
        GI.preprocessProblem(pd)
        xy, tri = square_mesh(case['dim'])
        return dict(kind=kind, pd=pd, steps=case['steps'], c0=pinned(host_projection(xy, tri, case['p'], humps(seed))))
    pd = GT.Struct(hmax=1.0 / case['dim'], p=case['p'], numSpecies=case['species'], precision=case['precision'],
                   numSteps=case['steps'], tEnd=case['steps'] * tau_of(case))
    GT.configureProblem(pd)
    GT.preprocessProblem(pd)
    xy, tri = square_mesh(case['dim'])
    depth = host_projection(xy, tri, case['p'], lambda x, y: 0.1 + 0.0 * x)
    cH = np.stack([host_projection(xy, tri, case['p'], f) for f in species_fields(case, seed)], axis=2)
    return dict(kind='transport', pd=pd, depth=np.asfortranarray(depth), cH=np.asfortranarray(cH))


def implicit_tau(case):
    return 2 * math.pi / 320 * 64 / case['dim']


def run(state):
    kind = state['kind']
    if kind == 'loop':
        pd = state['pd']
        pd.solver.set_state(state['c0'])
        pd.solver.limit_state(0.0)
        pd.isFinished, n = False, 0
        while not pd.isFinished:
            n += 1
            for f in G.STEP:
                pd = f(pd, n)
        return G.cDisc(pd)
    if kind == 'solve':
        s = state['solver']
        s.set_state(state['c0'])
        if state['limit']:
            s.limit_state(0.0)
        s.step(state['steps'], 0, state['tau'])
        s.get_state(state['out'])
        return single_of(state['out']) if state['single'] else state['out']
    if kind == 'transient':
        pd = state['pd']
        pd.solver.set_state(state['c0'])
        pd.solver.limit_state(0.0)
        pd.solver.step(pd.numSteps, 0, pd.tau)
        pd._stale = True
        G.postprocessProblem(pd)
        return [pd.cDisc, pd.error]
    if kind == 'ensemble':
        e = state['ensemble']
        for p, s in e.solvers.items():
            s.set_state(state['c0'][p])
            s.limit_state(0.0)
        e.step(state['steps'])
        return [c.astype(np.float32) for c in e.states()]
    if kind == 'grad':
        J, g0, gth = ADJ.misfit_gradient(state['pd'], state['c0'], state['theta'], state['target'],
                                         state['snapshots'])
        if state['single']:
            return [np.float32(J), single_of(g0), gth.astype(np.float32)]
        return [J, g0, gth]
    if kind == 'implicit':
        pd = state['pd']
        pd.iterations = 0
        pd.solver.set_state(state['c0'])
        for n in range(1, state['steps'] + 1):
            GI.solveStep(pd, n)
        return pd.solver.get_state()
    pd = state['pd']
    pd.solver.transport_init(state['depth'], state['cH'], pd.maskTol, pd.isMask)
    pd.solver.transport_step(pd.numSteps, 0, pd.tau)
    GT.postprocessProblem(pd)
    return [list(pd.cDisc), list(pd.concDisc), list(pd.mask)]


def single_of(a):
    """The values of an FP32 handle's state, which the call gives in FP64, in single precision."""
    return torch.from_numpy(a.T).float().T


# ---------------------------------------------------------------------------------------------
def work(case):
    """Bytes: per stage the coefficients read and written (also the step's start, where a
    Runge-Kutta stage needs it), the velocity at the volume and edge points and the neighbour map,
    each once; with a limiter the vertex values; per pass the coefficients in and out in FP64.
    Flops: the point values, the volume and edge sums and the limiter's reconstruction, a
    multiply-add as two."""
    def stage(p, w, lim):
        n, q, r = (p + 1) * (p + 2) // 2, (1, 3, 6, 12)[p], p + 1
        by = w * (3 * n + 2 * q + 3 * r) + 16 + (2 * w if lim else 0)
        fl = 2 * (3 * q * n + 3 * r * 2 * n + 2 * n) + (2 * 6 * n if lim else 0)
        return by, fl, n
    kind = case['kind']
    if kind == 'ensemble':
        by = fl = 0.0
        for i in range(case['count']):
            level, p = MIX[i % len(MIX)]
            b, f, n = stage(p, 4, True)
            k = 2 * 4 ** level
            by += k * (case['steps'] * (p + 1) * b + 16 * n)
            fl += k * case['steps'] * (p + 1) * f
        return dict(bytes=by, flops=fl)
    k, p = 2 * case['dim'] ** 2, case['p']
    w = FLOAT_BYTES[case.get('precision', 'fp64')]
    lim = kind in ('loop', 'transient', 'transport') or case.get('limiter', 'none') != 'none'
    b, f, n = stage(p, w, lim)
    if kind == 'grad':      # the recorded run, and the reverse stages with the velocity's sensitivities
        st = case['steps'] * ord_rk(p)
        return dict(bytes=k * (st * 3.0 * b + 5 * 8 * n), flops=k * st * 3.5 * f)
    if kind == 'implicit':  # about a dozen operator and preconditioner products a stage
        st = case['steps'] * (case['ordRK'] + (case['ordRK'] == 4))
        return dict(bytes=k * (st * 12.0 * (b + w * (n * n + 4 * n)) + 16 * n), flops=k * st * 12.0 * (f + 2 * n * n))
    m = case.get('species', 1)
    st = case['steps'] * ord_rk(p)
    return dict(bytes=float(k * m * (st * b + (32 if m > 1 else 16) * n)), flops=float(k * m * st * f))


# ---------------------------------------------------------------------------------------------
# The same problems in plain torch, FP64
def rule2(order):
    """Rules on the reference triangle: points and weights (sum 1/2) of Gauss, Strang and Fix,
    Dunavant, exact for polynomials of the given degree."""
    if order <= 1:
        return np.array([1 / 3]), np.array([1 / 3]), np.array([0.5])
    if order == 2:
        return np.array([1 / 6, 2 / 3, 1 / 6]), np.array([1 / 6, 1 / 6, 2 / 3]), np.full(3, 1 / 6)
    if order == 3:
        s3, s6 = math.sqrt(3), math.sqrt(6)
        a, b = np.array([(3 + s3) / 6, (3 - s3) / 6]), np.array([(6 + s6) / 10, (6 - s6) / 10])
        w = np.array([1 / 8 + s6 / 72, 1 / 8 - s6 / 72])
        return (np.array([a[0] * b[0], a[1] * b[0], a[0] * b[1], a[1] * b[1]]),
                np.array([a[1] * b[0], a[0] * b[0], a[1] * b[1], a[0] * b[1]]), np.repeat(w, 2))

    def orbit3(a, w):
        return [(a, a, w), (1 - 2 * a, a, w), (a, 1 - 2 * a, w)]
    if order == 4:
        pts = orbit3(0.445948490915965, 0.111690794839005) + orbit3(0.091576213509771, 0.054975871827661)
    elif order == 5:
        s = math.sqrt(15)
        pts = [(1 / 3, 1 / 3, 9 / 80)] + orbit3((6 - s) / 21, (155 - s) / 2400) + orbit3((6 + s) / 21, (155 + s) / 2400)
    elif order == 6:
        pts = orbit3(0.063089014491502, 0.025422453185103) + orbit3(0.249286745170910, 0.058393137863189)
        a, b, c, w = 0.310352451033785, 0.053145049844816, 0.636502499121399, 0.041425537809187
        pts += [(x, y, w) for x, y in ((a, b), (b, a), (a, c), (c, a), (b, c), (c, b))]
    else:
        raise ValueError('no rule of order %d here' % order)
    return tuple(np.array(c) for c in zip(*pts))


def basis(p, x, y):
    """The orthonormal modal basis on the reference triangle and its two derivatives: values
    (points x N) each."""
    x, y = np.asarray(x, dtype=np.float64), np.asarray(y, dtype=np.float64)
    one, nul = np.ones_like(x), np.zeros_like(x)
    f = [(math.sqrt(2) * one, nul, nul)]
    if p >= 1:
        f += [(2 - 6 * x, -6 * one, nul)]
        s = 2 * math.sqrt(3)
        f += [(s * (1 - x - 2 * y), -s * one, -2 * s * one)]
    if p >= 2:
        s = math.sqrt(6)
        f += [(s * (10 * x * x - 8 * x + 1), s * (20 * x - 8), nul)]
        s = math.sqrt(3)
        f += [(s * (5 * x * x - 4 * x - 15 * y * y + 12 * y - 1), s * (10 * x - 4), s * (12 - 30 * y))]
        s = 3 * math.sqrt(5)
        f += [(s * (3 * x * x + 8 * x * y - 4 * x + 3 * y * y - 4 * y + 1), s * (6 * x + 8 * y - 4), s * (8 * x + 6 * y - 4))]
    if p >= 3:
        s = 2 * math.sqrt(2)
        f += [(s * (35 * x ** 3 - 45 * x * x + 15 * x - 1), s * (105 * x * x - 90 * x + 15), nul)]
        s = 2 * math.sqrt(6)
        f += [(s * (21 * x ** 3 - 33 * x * x + 13 * x - 1 + (42 * x * x - 24 * x + 2) * y),
               s * (63 * x * x - 66 * x + 13 + (84 * x - 24) * y), s * (42 * x * x - 24 * x + 2))]
        s = 2 * math.sqrt(10)
        f += [(s * (7 * x ** 3 - 15 * x * x + 9 * x - 1 + (42 * x * x - 48 * x + 6) * y + (42 * x - 6) * y * y),
               s * (21 * x * x - 30 * x + 9 + (84 * x - 48) * y + 42 * y * y),
               s * (42 * x * x - 48 * x + 6 + 2 * (42 * x - 6) * y))]
        s = 2 * math.sqrt(14)
        f += [(s * (x ** 3 - 3 * x * x + 3 * x - 1 + (12 * x * x - 24 * x + 12) * y + (30 * x - 30) * y * y + 20 * y ** 3),
               s * (3 * x * x - 6 * x + 3 + (24 * x - 24) * y + 30 * y * y),
               s * (12 * x * x - 24 * x + 12 + 2 * (30 * x - 30) * y + 60 * y * y))]
    return tuple(np.stack([g[m] for g in f], axis=-1) for m in range(3))


def edge_point(n, s):
    """Point s in [0, 1] of reference edge n (opposite to vertex n, counter-clockwise)."""
    return ((1 - s, s), (0 * s, 1 - s), (s, 0 * s))[n]


class Scheme:
    """The semi-discrete problem on one mesh: dc/dt = rhs(c), and its limiters."""

    def __init__(self, xy, tri, p, order=None):
        dev = 'cuda' if torch.cuda.is_available() else 'cpu'
        self.t = lambda a: torch.as_tensor(np.asarray(a), device=dev)
        t = self.t
        self.p, self.N, self.K = p, (p + 1) * (p + 2) // 2, len(tri)
        self.order = max(2 * p, 1) if order is None else order
        self.nv = len(xy)
        self.tri = t(tri)
        X = t(xy)[self.tri]                                   # K x 3 x 2
        self.X = X
        self.B = torch.stack([X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]], dim=2)   # B[k, m, n]
        self.det = self.B[:, 0, 0] * self.B[:, 1, 1] - self.B[:, 0, 1] * self.B[:, 1, 0]
        q1, q2, w = rule2(self.order)
        self.q, self.w = (q1, q2), t(w)
        self.phi, self.d1, self.d2 = (t(a) for a in basis(p, q1, q2))
        s, ws = np.polynomial.legendre.leggauss(p + 1)
        self.s, self.ws = (s + 1) / 2, t(ws / 2)
        self.edge = t(np.stack([basis(p, *edge_point(n, self.s))[0] for n in range(3)]))       # 3 x R x N
        self.back = t(np.stack([basis(p, *edge_point(n, 1 - self.s))[0] for n in range(3)]))   # the neighbour's side
        a, b = X[:, [1, 2, 0]], X[:, [2, 0, 1]]
        self.areanu = torch.stack([b[..., 1] - a[..., 1], a[..., 0] - b[..., 0]], dim=2)       # |E| nu, K x 3 x 2
        # neighbours: the two sides of an edge, found by its sorted vertex pair
        e = np.sort(np.stack([tri[:, [1, 2]], tri[:, [2, 0]], tri[:, [0, 1]]], axis=1), axis=2).reshape(-1, 2)
        key = e[:, 0].astype(np.int64) * self.nv + e[:, 1]
        o = np.argsort(key, kind='stable')
        same = key[o][1:] == key[o][:-1]
        other = np.full(len(key), -1, dtype=np.int64)
        i, j = o[:-1][same], o[1:][same]
        other[i], other[j] = j, i
        other = other.reshape(-1, 3)
        self.bdr = t(other < 0)
        self.nb, self.ne = t(np.where(other < 0, 0, other // 3)), t(np.where(other < 0, 0, other % 3))
        vd = np.zeros(self.nv, dtype=bool)
        vd[np.concatenate([tri[:, [1, 2]][other[:, 0] < 0].ravel(), tri[:, [2, 0]][other[:, 1] < 0].ravel(),
                           tri[:, [0, 1]][other[:, 2] < 0].ravel()])] = True
        self.vdir = t(vd)[self.tri]
        self.F1 = self.F2 = self.vn = None
        self.active = None

    def points(self, q1, q2):
        q1, q2 = self.t(np.asarray(q1)), self.t(np.asarray(q2))
        return [self.X[:, 0, m, None] + self.B[:, m, 0, None] * q1 + self.B[:, m, 1, None] * q2 for m in range(2)]

    def project(self, f, order=None):
        q1, q2, w = rule2(self.order if order is None else order)
        v = f(*self.points(q1, q2))
        return v @ (self.t(w)[:, None] * self.t(basis(self.p, q1, q2)[0]))

    def factors(self, u1, u2):
        """The volume and edge factors of a velocity: its projection at the volume points, its
        normal component at the edge points."""
        a, b = self.project(u1) @ self.phi.T, self.project(u2) @ self.phi.T
        B, d = self.B, self.det[:, None]
        f1 = self.w * (B[:, 1, 1, None] * a - B[:, 0, 1, None] * b) / d
        f2 = self.w * (B[:, 0, 0, None] * b - B[:, 1, 0, None] * a) / d
        vn = []
        for n in range(3):
            x, y = self.points(*edge_point(n, self.s))
            vn.append(self.ws * (self.areanu[:, n, 0, None] * u1(x, y) + self.areanu[:, n, 1, None] * u2(x, y)) / d)
        return f1, f2, torch.stack(vn, dim=1)

    def set_velocity(self, u1, u2):
        self.F1, self.F2, self.vn = self.factors(u1, u2)

    def rhs(self, c):
        cq = c @ self.phi.T
        out = (self.F1 * cq) @ self.d1 + (self.F2 * cq) @ self.d2
        for n in range(3):
            own = c @ self.edge[n].T
            cn = c[self.nb[:, n]]
            far = torch.einsum('krj,kj->kr', self.back[self.ne[:, n]], cn)
            v = self.vn[:, n]
            inner = ~self.bdr[:, n, None]
            outer = torch.ones_like(inner)
            if self.active is not None:      # an active element sees active neighbours only
                act = inner & self.active[self.nb[:, n], None]
                inner, outer = act, act | self.bdr[:, n, None]
            zero = torch.zeros((), dtype=c.dtype, device=c.device)
            trace = torch.where((v > 0) & outer, own, torch.where((v < 0) & inner, far, zero))
            out = out - (v * trace) @ self.edge[n]
        return out

    def inflow(self, f):
        """Boundary term of the data f on the inflow edges."""
        out = 0.0
        for n in range(3):
            v = torch.where((self.vn[:, n] < 0) & self.bdr[:, n, None], self.vn[:, n], torch.zeros_like(self.vn[:, n]))
            out = out + (v * f(*self.points(*edge_point(n, self.s)))) @ self.edge[n]
        return out

    # ---- limiters -----------------------------------------------------------------------------
    def taylor(self):
        """Taylor basis of every element at the volume points and the vertices, the map from Taylor
        to modal coefficients and its inverse, and the Taylor mass correction."""
        dx = 2 / torch.sqrt(self.det)
        q1, q2, _ = rule2(max(2 * self.p, 1))
        bary = self.X.mean(dim=1)
        P = [z - bary[:, m, None] for m, z in enumerate(self.points(q1, q2))]
        V = [self.X[:, :, m] - bary[:, m, None] for m in range(2)]
        w = self.t(rule2(max(2 * self.p, 1))[2])
        phi = self.t(basis(self.p, q1, q2)[0])

        def functions(z):
            f = [torch.ones_like(z[0]), z[0] * dx[:, None], z[1] * dx[:, None]]
            for d in range(2, self.p + 1):
                for j in range(d + 1):
                    c = 1 / (math.factorial(d - j) * math.factorial(j))
                    mean = 2 * ((P[0] ** (d - j) * P[1] ** j) @ w)
                    f.append(c * (z[0] ** (d - j) * z[1] ** j - mean[:, None]) * dx[:, None] ** d)
            return torch.stack(f, dim=2)
        at = functions(P)
        self.tv = functions(V)
        self.t2c = torch.einsum('q,qi,kqj->kij', w, phi, at)
        self.c2t = torch.linalg.inv(self.t2c)
        m = torch.einsum('q,kqi,kqj->kij', w, at, at)
        self.mcorr = m / torch.diagonal(m, dim1=1, dim2=2)[:, :, None]

    def extremes(self, v):
        lo = torch.full((self.nv,), math.inf, dtype=v.dtype, device=v.device)
        at, val = self.tri.reshape(-1), v[:, None].expand(-1, 3).reshape(-1)
        return (lo.scatter_reduce(0, at, val, 'amin')[self.tri], (-lo).scatter_reduce(0, at, val, 'amax')[self.tri])

    def factor(self, mean, at, data):
        lo, hi = self.extremes(mean)
        if data is not None:
            lo, hi = torch.where(self.vdir, torch.fmin(lo, data), lo), torch.where(self.vdir, torch.fmax(hi, data), hi)
        dv, lo, hi = at - mean[:, None], lo - mean[:, None], hi - mean[:, None]
        one = torch.ones_like(dv)
        a = torch.where(dv < lo + 1e-8, (lo / (dv - 1e-8)).clamp(0, 1), one)
        a = torch.where(dv > hi - 1e-8, (hi / (dv + 1e-8)).clamp(0, 1), a)
        return a.amin(dim=1)

    def limit_taylor(self, c, kind, data):
        if kind == 'linear':
            a = self.factor(c[:, 0], torch.einsum('knj,kj->kn', self.tv[:, :, :3], c[:, :3]), data)[:, None]
            return torch.cat([c[:, :1], a * c[:, 1:3], (a == 1) * c[:, 3:]], dim=1)
        out, alpha = c.clone(), torch.zeros_like(c[:, 0])
        for o in range(self.p, 0, -1):
            a = torch.ones_like(alpha)
            for j in range(o):
                i0, i1 = o * (o - 1) // 2 + j, o * (o + 1) // 2 + j
                at = torch.einsum('knj,kj->kn', self.tv[:, :, :3], c[:, [i0, i1, i1 + 1]])
                a = torch.minimum(a, self.factor(c[:, i0], at, at if o > 1 else data))
            alpha = torch.maximum(alpha, a)
            out[:, o * (o + 1) // 2:(o + 1) * (o + 2) // 2] *= alpha[:, None]
        return out

    def limit(self, c, kind, data):
        u = torch.einsum('kij,kj->ki', self.c2t, c)
        return torch.einsum('kij,kj->ki', self.t2c, self.limit_taylor(u, kind, data))

    def limit_dot(self, c, kind):
        u = torch.einsum('kij,kj->ki', self.c2t, c)
        l = self.limit_taylor(u, kind, None)
        return torch.einsum('kij,kj->ki', self.t2c, l + torch.einsum('kij,kj->ki', self.mcorr, u - l))

    def zero_data(self):
        return torch.zeros((self.K, 3), dtype=torch.float64, device=self.X.device)

    def solve(self, c, tau, steps, kind, sources=None, data=None):
        """SSP-RK steps of the degree's order from t = 0 (kind: limiter or 'none')."""
        om = ((0.0,), (0.0, 0.5), (0.0, 0.75, 1 / 3))[ord_rk(self.p) - 1]
        at = ((0.0,), (0.0, 1.0), (0.0, 1.0, 0.5))[ord_rk(self.p) - 1]
        data = data or (lambda t: self.zero_data())
        if kind != 'none':
            self.taylor()
            c = self.limit(c, kind, data(0.0))
        for n in range(steps):
            c0, t0 = c, n * tau
            for s in range(len(om)):
                d = self.rhs(c)
                if sources is not None:
                    d = d + sources(t0 + at[s] * tau)
                if kind != 'none' and self.p > 1:
                    d = self.limit_dot(d, kind)
                c = om[s] * c0 + (1 - om[s]) * (c + tau * d)
                if kind != 'none':
                    c = self.limit(c, kind, data(t0 + (at[s + 1] if s + 1 < len(om) else 1.0) * tau))
        return c


def gmres(op, b, x, tol=1e-14, m=80):
    """(op) x = b, restarted GMRES."""
    nb = b.norm()
    for _ in range(20):
        r = b - op(x)
        beta = r.norm()
        if beta <= tol * nb:
            break
        V, H = [r / beta], torch.zeros((m + 1, m), dtype=b.dtype)
        for j in range(m):
            w = op(V[j])
            for _ in range(2):
                h = torch.stack([(v * w).sum() for v in V])
                H[:j + 1, j] += h.cpu()
                w = w - sum(hi * v for hi, v in zip(h, V))
            H[j + 1, j] = w.norm().cpu()
            V.append(w / w.norm())
            rhs = torch.zeros(j + 2, dtype=b.dtype)
            rhs[0] = beta.cpu()
            y = torch.linalg.lstsq(H[:j + 2, :j + 1], rhs[:, None]).solution[:, 0]
            if (H[:j + 2, :j + 1] @ y - rhs).norm() <= 0.3 * tol * nb.cpu():
                break
        x = x + sum(float(yi) * v for yi, v in zip(y, V))
    return x


def dirk(order):
    if order == 1:
        return [[1.0]]
    if order == 2:
        g = 1 - math.sqrt(0.5)
        return [[g], [1 - g, g]]
    if order == 3:
        g = 0.435866521508459
        b1, b2 = -0.25 * (6 * g * g - 16 * g + 1), 0.25 * (6 * g * g - 20 * g + 5)
        return [[g], [0.5 * (1 - g), g], [b1, b2, g]]
    return [[1 / 4], [1 / 2, 1 / 4], [17 / 50, -1 / 25, 1 / 4], [371 / 1360, -137 / 2720, 15 / 544, 1 / 4],
            [25 / 24, -49 / 48, 125 / 16, -85 / 12, 1 / 4]]


def exact(case, seed):
    kind = case['kind']
    if kind == 'ensemble':
        out = []
        for d in instances(case['count'], seed):
            mesh = square_mesh(2 ** d['level'], 0.2, d['mesh'])
            s = Scheme(*mesh, d['p'])
            s.set_velocity(*stream_velocity(d['k'], d['l'], d['a']))
            c = s.t(host_projection(*mesh, d['p'], smooth(d['seed'])))
            out.append(s.solve(c, ENSEMBLE_TAU, case['steps'], 'linear'))
        return out
    p, tau = case['p'], tau_of(case)
    mesh = square_mesh(case['dim'], case.get('jitter', 0.0), 5)
    start = lambda s, f: s.t(host_projection(*mesh, p, f))   # noqa: E731
    if kind in ('loop', 'solve'):
        s = Scheme(*mesh, p)
        s.set_velocity(*(stream_velocity(*stream_modes(seed)) if case.get('velocity') == 'stream' else rotation()))
        return s.solve(start(s, humps(seed)), tau, case['steps'], case.get('limiter', 'linear'))
    if kind == 'transient':
        s = Scheme(*mesh, p)
        u1, u2, cc, adv, decay = transient_data()
        s.set_velocity(u1, u2)
        extra = smooth(seed)
        one = lambda x, y: torch.ones_like(x)   # noqa: E731
        a, b = s.project(adv) - s.inflow(cc), s.project(decay) - s.inflow(one)
        at = cc(s.X[:, :, 0], s.X[:, :, 1])
        c = s.solve(start(s, lambda x, y: cc(x, y) + 1.0 + extra(x, y)), tau, case['steps'], 'linear',
                    sources=lambda t: a + math.exp(-t) * b, data=lambda t: at + math.exp(-t))
        q1, q2, w = rule2(2 * p + 1)
        d = c @ s.t(basis(p, q1, q2)[0]).T - cc(*s.points(q1, q2)) - math.exp(-case['steps'] * tau)
        return [c, float(torch.sqrt(((d * d) @ s.t(w) * s.det).sum()))]
    if kind == 'grad':
        s = Scheme(*mesh, p)
        r = np.random.default_rng([int(seed), 75])
        theta = s.t(r.normal(0.0, 0.04, size=16)).requires_grad_()
        f = [s.factors(*stream_velocity([k], [l], [1.0])) for k in (1, 2, 3, 4) for l in (1, 2, 3, 4)]
        s.F1, s.F2, s.vn = (torch.tensordot(theta, torch.stack([m[i] for m in f]), 1) for i in range(3))
        c0 = start(s, smooth(seed)).requires_grad_()
        J = 0.5 * ((s.solve(c0, tau, case['steps'], 'none') - start(s, smooth(seed + 1))) ** 2).sum()
        g0, gth = torch.autograd.grad(J, (c0, theta))
        return [float(J), g0, gth]
    if kind == 'implicit':
        s = Scheme(*mesh, p, order=2 * p + 1)
        s.set_velocity(*rotation())
        c, tau = start(s, humps(seed)), implicit_tau(case)
        for _ in range(case['steps']):
            k, x = [], c
            for row in dirk(case['ordRK']):
                b = c + sum(tau * a * d for a, d in zip(row, k))
                x = gmres(lambda z: z - tau * row[-1] * s.rhs(z), b, x)
                k.append(s.rhs(x))
            c = x
        return c
    s = Scheme(*mesh, p)
    s.set_velocity(lambda x, y: 0.1 * (0.5 - y), lambda x, y: 0.1 * (x - 0.5))
    s.taylor()
    om = ((0.0,), (0.0, 0.5), (0.0, 0.75, 1 / 3))[ord_rk(p) - 1]

    def spread(c):
        lo, hi = s.extremes(math.sqrt(2) * c[:, 0])
        z = torch.zeros_like(lo)
        lo, hi = torch.where(s.vdir, torch.minimum(lo, z), lo), torch.where(s.vdir, torch.maximum(hi, z), hi)
        return (hi - lo).amax(dim=1) >= 1e-6
    outH, outC = [], []
    for f in species_fields(case, seed):
        raw = start(s, f) / 0.1
        mask, c = spread(raw), s.limit(raw, 'linear', s.zero_data())
        for _ in range(case['steps']):
            c0 = c
            for i, w in enumerate(om):
                s.active = mask
                raw = w * c0 + (1 - w) * (c + tau / 0.1 * (mask[:, None] * s.rhs(c)))
                c = s.limit(raw, 'linear', s.zero_data())
            mask = spread(raw)
        s.active = None
        outH.append(c * 0.1)
        outC.append(c)
    return [outH, outC, None]
