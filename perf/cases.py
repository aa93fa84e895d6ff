"""What a user of this package has it do, as timed cases through its public entry points.

Kinds of case:
  step     KDK steps of one simulation from a state in hand (Solver.nbody), with
           or without a monitor that takes P(k) of every force's delta_k
  ics      whitenoise -> linear field -> 2LPT state (Solver.whitenoise / linear / lpt)
  power    P(k) of a density mesh (power)
  catalog  a particle catalogue on a mesh: paint, r2c, c2r, readout (ParticleMesh)
  grad     loss and gradient of the differentiable forward model (ForwardModel)
  serve    a batch of whole simulations (ServingEngine)
Inputs come from seeded torch generators and cuFFT alone, so every build of the
package sees the same bits; exact() restates each kind in float64 torch.
"""
import gc
import importlib
import math

import numpy
import torch

import fastpm_gb300 as G

OM0, H, OB0, NS, SIGMA8, TCMB = 0.3089, 0.6774, 0.0486, 0.9667, 0.8159, 2.7255
MESHES = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 1024)
DEV = 'cuda'


def listed():
    return [
        # the smallest simulation of the tests: all launches and host time
        dict(name='step-16x2-cic', kind='step', nc=16, B=2, box=32.0, window='cic', shift=0.0, a0=0.1, a1=0.2, steps=3,
             monitor=False, explicit=0),
        # a laptop-scale run, the 64^3 / 128^3 configuration, mid-way through
        dict(name='step-64x2-cic', kind='step', nc=64, B=2, box=256.0, window='cic', shift=0.0, a0=0.4, a1=0.6, steps=2,
             monitor=False, explicit=0),
        # a mesh whose size is no power of two, late and clustered
        dict(name='step-192x2-tsc', kind='step', nc=192, B=2, box=384.0, window='tsc', shift=0.5, a0=0.8, a1=0.9, steps=2,
             monitor=False, explicit=0),
        # the 256^3 / 512^3 CIC configuration at late times
        dict(name='step-256x2-cic', kind='step', nc=256, B=2, box=512.0, window='cic', shift=0.0, a0=0.7, a1=0.85, steps=2,
             monitor=False, explicit=0),
        # the production configuration: 512^3 particles, 1024^3 TSC mesh
        dict(name='step-512x2-tsc', kind='step', nc=512, B=2, box=1024.0, window='tsc', shift=0.0, a0=0.5, a1=0.6, steps=2,
             monitor=False, explicit=0),
        # a run that watches its P(k), as a user's script does at every force
        dict(name='watch-128x2-tsc', kind='step', nc=128, B=2, box=512.0, window='tsc', shift=0.5, a0=0.5, a1=0.7, steps=2,
             monitor=True, explicit=0),
        # initial conditions of a mid-sized run
        dict(name='ics-256', kind='ics', nc=256, B=2, box=512.0, a0=0.05, order=2, unitary=False),
        # the power spectrum of a finished run's density
        dict(name='power-512', kind='power', n=512, box=1024.0),
        # a halo / galaxy catalogue: a few million points on a mid-sized mesh
        dict(name='catalog-3M-256-tsc', kind='catalog', np=3000001, n=256, box=1000.0, window='tsc', clustered=True),
        # a small catalogue on a small mesh
        dict(name='catalog-20k-48-cic', kind='catalog', np=20011, n=48, box=200.0, window='cic', clustered=False),
        # one evaluation of loss and gradient, as a sampler over initial conditions does
        dict(name='grad-64x2', kind='grad', nc=64, B=2, box=256.0, window='cic', a0=0.1, a1=1.0, steps=3, ck=2),
        # a service run: eight requests of one shape class
        dict(name='serve-128x2', kind='serve', nc=128, B=2, window='cic', requests=8, steps=4, a0=0.1, a1=0.6),
    ]


def _log_pick(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(('step', 'ics', 'power', 'catalog', 'grad', 'serve'), (10, 2, 2, 4, 1, 1))[0]
    window = rng.choice(('cic', 'tsc'))
    if kind == 'step':
        B = rng.choice((1, 2, 2, 2, 3, 4))
        nc = rng.choice([m for m in MESHES if m <= 512 and m * B in MESHES and (m, B) != (512, 2)])
        a0 = round(rng.uniform(0.05, 0.9), 3)
        # an explicit particle load (a glass, a selection) of any number of particles
        explicit = _log_pick(rng, 1000, 4000000) if nc <= 128 and rng.random() < 0.3 else 0
        return dict(kind='step', nc=nc, B=B, box=round(nc * rng.uniform(1.0, 4.0), 2), window=window,
                    shift=rng.choice((0.0, 0.5)), a0=a0, a1=round(a0 + rng.uniform(0.02, 0.1), 3),
                    steps=rng.choice((1, 2)), monitor=rng.random() < 0.25 and nc * B <= 512, explicit=explicit)
    if kind == 'ics':
        nc = rng.choice([m for m in MESHES if 32 <= m <= 512])
        return dict(kind='ics', nc=nc, B=1, box=round(nc * rng.uniform(1.0, 4.0), 2), a0=round(rng.uniform(0.02, 0.1), 3),
                    order=rng.choice((1, 2, 2)), unitary=rng.random() < 0.3)
    if kind == 'power':
        n = rng.choice([m for m in MESHES if m >= 32])
        return dict(kind='power', n=n, box=round(n * rng.uniform(1.0, 4.0), 2))
    if kind == 'catalog':
        return dict(kind='catalog', np=_log_pick(rng, 1000, 20000000), n=rng.choice([m for m in MESHES if m <= 512]),
                    box=round(rng.uniform(100.0, 2000.0), 1), window=window, clustered=rng.random() < 0.5)
    if kind == 'grad':
        nc = rng.choice((24, 32, 48, 64, 96, 128))
        return dict(kind='grad', nc=nc, B=rng.choice((1, 2)), box=round(nc * rng.uniform(2.0, 4.0), 2), window=window,
                    a0=0.1, a1=round(rng.uniform(0.4, 1.0), 2), steps=rng.choice((2, 3)), ck=rng.choice((1, 2, 4)))
    return dict(kind='serve', nc=rng.choice((64, 96, 128, 192)), B=rng.choice((1, 2)), window='cic',
                requests=rng.randint(2, 8), steps=rng.randint(2, 5), a0=0.1, a1=0.6)


# ---------------------------------------------------------------------------
# linear power: the Eisenstein & Hu (1998, ApJ 496, 605) no-wiggle fit, sigma8-normalised
# ---------------------------------------------------------------------------
def _transfer(k, Om0):
    wm, wb, fb, th = Om0 * H * H, OB0 * H * H, OB0 / Om0, TCMB / 2.7
    s = 44.5 * math.log(9.83 / wm) / math.sqrt(1 + 10 * wb ** 0.75)
    al = 1 - 0.328 * math.log(431 * wm) * fb + 0.38 * math.log(22.3 * wm) * fb ** 2
    q = k * th ** 2 / (Om0 * H * (al + (1 - al) / (1 + (0.43 * k * H * s) ** 4)))
    L0 = numpy.log(2 * math.e + 1.8 * q)
    return L0 / (L0 + (14.2 + 731 / (1 + 62.5 * q)) * q * q)


def _linear_power(Om0=OM0, sigma8=SIGMA8):
    """P(k) in (Mpc/h)^3 at redshift 0, a callable of k in h/Mpc."""
    lnk = numpy.linspace(math.log(1e-5), math.log(1e3), 20001)
    k = numpy.exp(lnk)
    x = 8 * k
    w = 3 * (numpy.sin(x) - x * numpy.cos(x)) / x ** 3
    amp = sigma8 ** 2 / numpy.trapezoid(k ** 3 * k ** NS * _transfer(k, Om0) ** 2 / (2 * math.pi ** 2) * w ** 2, lnk)

    def P(kk):
        kk = numpy.asarray(kk, dtype='f8')
        with numpy.errstate(divide='ignore', invalid='ignore'):
            p = amp * kk ** NS * _transfer(kk, Om0) ** 2
        return numpy.where(kk > 0, p, 0.0)
    return P


def _shell_table(n, box, P):
    k = numpy.sqrt(numpy.arange(3 * (n // 2) ** 2 + 1, dtype='f8')) * (2 * math.pi / box)
    return P(k) ** 0.5 / box ** 1.5


# ---------------------------------------------------------------------------
# inputs (float32, seeded; gathers and cuFFT only, so they repeat bit for bit)
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _freq(n, dtype):
    f = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=dtype)
    return f.view(n, 1, 1), f.view(1, n, 1), torch.arange(n // 2 + 1, device=DEV, dtype=dtype).view(1, 1, -1)


def _delta_k(n, box, g):
    """A Gaussian field of the linear power at redshift 0 (torch's rfftn, unnormalised)."""
    d = torch.fft.rfftn(torch.randn(n, n, n, generator=g, device=DEV))
    ix, iy, iz = _freq(n, torch.float32)
    t = torch.from_numpy((_shell_table(n, box, _linear_power()) * n ** 1.5).astype('f4')).to(DEV)
    for i in range(n):
        d[i] *= t[(ix[i] ** 2 + iy[0] ** 2 + iz[0] ** 2).long()]
    return d


def _psi(n, box, g):
    """The Zel'dovich displacement per unit growth on the nodes of an n^3 mesh, [n^3, 3]."""
    d = _delta_k(n, box, g)
    f = _freq(n, torch.float32)
    kk = f[0] ** 2 + f[1] ** 2 + f[2] ** 2
    kk[0, 0, 0] = 1.0
    d /= kk * (2 * math.pi / box)
    del kk
    out = torch.empty(n ** 3, 3, device=DEV)
    for ax in range(3):
        odd = torch.where(f[ax].abs() == n // 2, torch.zeros_like(f[ax]), f[ax])
        out[:, ax] = torch.fft.irfftn(1j * odd * d, s=(n, n, n)).reshape(-1)
    return out


def _interp(mesh, n, x):
    """Trilinear interpolation of [n^3, 3] at positions in cells."""
    i0 = torch.floor(x)
    f = x - i0
    i0 = i0.long() % n
    i1 = (i0 + 1) % n
    out = torch.zeros_like(x)
    for a in range(2):
        ia, wa = ((i1, f) if a else (i0, 1 - f))
        for b in range(2):
            ib, wb = ((i1, f) if b else (i0, 1 - f))
            for c in range(2):
                ic, wc = ((i1, f) if c else (i0, 1 - f))
                out += (wa[:, 0] * wb[:, 1] * wc[:, 2])[:, None] * mesh[(ia[:, 0] * n + ib[:, 1]) * n + ic[:, 2]]
    return out


def _evolved(nc, box, q, a, seed):
    """Displacement S, momentum P and force F of particles at q (a function of the
    chunk, in lattice cells) that moved in the frozen linear potential from
    a = 0.05 to a: sheets and clumps grow as they do in a run (Brainerd, Scherrer
    & Villumsen 1993).  In units of the growth factor ~ a (Einstein-de Sitter)
    du/dlna = 3/2 (psi(x) - u), dx/da = u."""
    psi = _psi(nc, box, _gen(seed))
    h = box / nc
    np_ = q(None)
    S, P, F = (torch.empty(np_, 3, device=DEV) for _ in range(3))
    lna = numpy.linspace(math.log(0.05), math.log(a), 5)
    E = math.sqrt(OM0 / a ** 3 + 1 - OM0)
    f1 = (OM0 / a ** 3 / E ** 2) ** 0.55
    for at in range(0, np_, 1 << 22):
        sl = slice(at, min(at + (1 << 22), np_))
        q0 = q(sl)
        u = _interp(psi, nc, q0)
        s = u * math.exp(lna[0])
        for l0, l1 in zip(lna[:-1], lna[1:]):
            g = _interp(psi, nc, q0 + s / h)
            w = 1 - math.exp(-1.5 * (l1 - l0))
            u = u + w * (g - u)
            s = s + u * (math.exp(l1) - math.exp(l0))
        S[sl] = s
        P[sl] = u * (a ** 3 * E * f1)
        F[sl] = _interp(psi, nc, q0 + s / h) * (1.5 * OM0 * a)
    return S, P, F


def _lattice_of(nc, shift):
    def q(sl):
        if sl is None:
            return nc ** 3
        p = torch.arange(sl.start, sl.stop, device=DEV)
        return torch.stack([p // (nc * nc), (p // nc) % nc, p % nc], dim=1).float() + shift
    return q


def _explicit_of(np_, nc, seed):
    x = torch.rand(np_, 3, generator=_gen(seed + 77), device=DEV) * nc

    def q(sl):
        return np_ if sl is None else x[sl]
    return q, x


def _stages(c):
    return [float(x) for x in numpy.linspace(c['a0'], c['a1'], c['steps'] + 1)]


def _catalog(c, seed):
    """float32 positions: uniform, or three quarters of them in clumps."""
    g = _gen(seed)
    pos = torch.rand(c['np'], 3, generator=g, device=DEV) * c['box']
    if c['clustered']:
        m = c['np'] * 3 // 4
        k = max(1, m // 200)
        centres = torch.rand(k, 3, generator=g, device=DEV) * c['box']
        who = torch.randint(k, (m,), generator=g, device=DEV)
        r = torch.randn(m, 3, generator=g, device=DEV) * (0.003 * c['box'])
        pos[:m] = torch.remainder(centres[who] + r, c['box'])
        pos = pos[torch.randperm(c['np'], generator=g, device=DEV)]
    return pos.contiguous()


def _density(c, seed):
    """1 + delta of a lognormal field of the linear power."""
    d = torch.fft.irfftn(_delta_k(c['n'], c['box'], _gen(seed)), s=(c['n'],) * 3)
    d = torch.exp(d.clamp_(-6.0, 6.0))
    return d / d.mean(dtype=torch.float64).float()


def _requests(c, seed):
    serving = importlib.import_module('fastpm_gb300.serving')
    rng = numpy.random.RandomState(seed % (1 << 31))
    return [serving.Request(i, nc=c['nc'], B=c['B'], Om0=float(rng.uniform(0.25, 0.35)), sigma8=float(rng.uniform(0.7, 0.9)),
                            nsteps=c['steps'], a0=c['a0'], a1=c['a1'], seed=int(rng.randint(1 << 30)), resampler=c['window'])
            for i in range(c['requests'])]


# the meshes, solvers and engines of the case in hand: a program makes them once
# and has many inputs go through them
_plan = {}


def _planned(c, make):
    key = repr(sorted((k, v) for k, v in c.items() if k != 'name'))
    if key not in _plan:
        _plan.clear()
        gc.collect()
        _plan[key] = make()
    return _plan[key]


def prepare(case, seed):
    c = dict(case)
    if c['kind'] == 'step':
        def make():
            pm = G.ParticleMesh(BoxSize=c['box'], Nmesh=[c['nc']] * 3, resampler=c['window'])
            return G.Solver(pm, G.Cosmology(Om0=OM0), B=c['B']), \
                None if c['explicit'] else pm.generate_uniform_particle_grid(shift=c['shift'])
        solver, Q = _planned(c, make)
        q = _lattice_of(c['nc'], c['shift'])
        if c['explicit']:
            q, x = _explicit_of(c['explicit'], c['nc'], seed)
            Q = x.double() * (c['box'] / c['nc'])
        S, P, F = _evolved(c['nc'], c['box'], q, c['a0'], seed)
        state = G.StateVector(solver, Q)
        state.S, state.P, state.F = S, P, F
        state.a = dict(S=c['a0'], P=c['a0'], F=c['a0'])
        return dict(c=c, solver=solver, state=state, stages=_stages(c))
    if c['kind'] == 'ics':
        def make():
            pm = G.ParticleMesh(BoxSize=c['box'], Nmesh=[c['nc']] * 3)
            return G.Solver(pm, G.Cosmology(Om0=OM0), B=c['B']), pm.generate_uniform_particle_grid(shift=0.0), _linear_power()
        return dict(c=c, plan=_planned(c, make), seed=int(seed))
    if c['kind'] == 'power':
        pm = _planned(c, lambda: G.ParticleMesh(BoxSize=c['box'], Nmesh=[c['n']] * 3))
        return dict(c=c, field=G.RealField(pm, _density(c, seed)))
    if c['kind'] == 'catalog':
        pm = _planned(c, lambda: G.ParticleMesh(BoxSize=c['box'], Nmesh=[c['n']] * 3, resampler=c['window']))
        return dict(c=c, pm=pm, pos=_catalog(c, seed))
    if c['kind'] == 'grad':
        adjoint = importlib.import_module('fastpm_gb300.adjoint')

        def make():
            n = c['nc'] * c['B']
            target = torch.exp(0.3 * torch.randn(n, n, n, generator=_gen(5), device=DEV))
            return adjoint.ForwardModel(c['nc'], c['B'], c['box'], _stages(c), target=target, checkpoint_every=c['ck'],
                                        resampler=c['window'])
        model = _planned(c, make)
        return dict(c=c, model=model, wn=model.pm.generate_whitenoise(int(seed)))
    serving = importlib.import_module('fastpm_gb300.serving')
    # the variant is fixed: what a tuner picks may differ from run to run
    engine = _planned(c, lambda: serving.ServingEngine([_requests(c, 0)[0].key], max_slots=c['requests'], use_graphs=True,
                                                       keep_state=True, tune=False, hbm_budget=60e9))
    return dict(c=c, engine=engine, seed=int(seed))


def run(state):
    c = state['c']
    if c['kind'] == 'step':
        seen = []

        def monitor(action, ai, ac, af, st, event):
            if action == 'F':
                seen.append(_spectrum(G.power(event['delta_k'], average=False)))
        st = state['state'].copy()   # the state in hand stays what it was
        state['solver'].nbody(st, G.leapfrog_with_lpt(state['stages']), monitor=monitor if c['monitor'] else None)
        return dict(S=st.S, P=st.P, F=st.F, RHO=st.RHO, seen=seen)
    if c['kind'] == 'ics':
        solver, Q, P = state['plan']
        wn = solver.whitenoise(state['seed'], unitary=c['unitary'])
        dlin = solver.linear(wn, P)
        st = solver.lpt(dlin, Q, c['a0'], order=c['order'])
        return dict(wn=wn.value, dlin=dlin.value, S=st.S, P=st.P, F=st.F)
    if c['kind'] == 'power':
        return _spectrum(G.power(state['field'], average=False))
    if c['kind'] == 'catalog':
        rho = state['pm'].paint(state['pos'])
        dk = rho.r2c()
        back = dk.c2r()
        return dict(rho=rho.value, dk=dk.value, back=back.value, at=back.readout(state['pos']))
    if c['kind'] == 'grad':
        loss = state['model'].forward(state['wn'], OM0)
        g, dom = state['model'].backward()
        return dict(loss=loss, g=g.value, dom=dom)
    reqs = state['engine'].run(_requests(c, state['seed']), realtime=False)
    reqs = sorted(reqs, key=lambda r: r.rid)
    return dict(k=[r.k.astype('f4') for r in reqs], pk=[r.pk.astype('f4') for r in reqs], S=[r.X for r in reqs])


def _spectrum(kpn):
    """k, P N and N; the spectrum of a float32 field is kept as float32."""
    k, p, N = kpn
    return dict(k=k.astype('f4'), p=p.astype('f4'), N=N.astype('i8'))


def work(case):
    c = case
    fft = lambda n: 2.5 * n ** 3 * math.log2(float(n) ** 3)   # noqa: E731
    if c['kind'] == 'step':
        n, np_ = c['nc'] * c['B'], c['explicit'] or c['nc'] ** 3
        # per step: S, P, F and the 16-bit compensation terms of S, P read and
        # written, RHO written; density and potential meshes written and read
        return dict(bytes=c['steps'] * (100.0 * np_ + 16.0 * n ** 3), flops=c['steps'] * (2 * fft(n) + 400.0 * np_))
    if c['kind'] == 'ics':
        n = c['nc']
        return dict(bytes=(8.0 + 36.0) * n ** 3, flops=(3 if c['order'] == 1 else 13) * fft(n))
    if c['kind'] == 'power':
        return dict(bytes=4.0 * c['n'] ** 3, flops=fft(c['n']))
    if c['kind'] == 'catalog':
        return dict(bytes=16.0 * c['np'] + 12.0 * c['n'] ** 3, flops=2 * fft(c['n']) + 300.0 * c['np'])
    if c['kind'] == 'grad':
        n, nc = c['nc'] * c['B'], c['nc']
        forces = c['steps'] + 1
        return dict(bytes=16.0 * nc ** 3 + forces * (2 * 100.0 * nc ** 3 + 80.0 * n ** 3),
                    flops=forces * 14 * fft(n) + 40 * fft(nc))
    n, nc = c['nc'] * c['B'], c['nc']
    one = 44.0 * nc ** 3 + (c['steps'] + 1) * (100.0 * nc ** 3 + 16.0 * n ** 3)
    return dict(bytes=c['requests'] * one, flops=c['requests'] * (13 * fft(nc) + (2 * c['steps'] + 3) * fft(n)))


# ---------------------------------------------------------------------------
# float64 restatement
# ---------------------------------------------------------------------------
class _Growth(object):
    """D1, D2 and their ln a derivatives in flat LambdaCDM, normalised at a = 1:
    Runge-Kutta in ln a from the matter-dominated solution at a = 1e-7."""

    def __init__(self, Om0, N=6000):
        self.Om0 = Om0
        lna = numpy.linspace(math.log(1e-7), 0.0, N + 1)
        y = numpy.empty((N + 1, 4))
        a0 = 1e-7
        y[0] = [a0, a0, -3. / 7 * a0 ** 2, -6. / 7 * a0 ** 2]
        h = lna[1] - lna[0]
        for i in range(N):
            k1 = self.rhs(y[i], lna[i])
            k2 = self.rhs(y[i] + h / 2 * k1, lna[i] + h / 2)
            k3 = self.rhs(y[i] + h / 2 * k2, lna[i] + h / 2)
            k4 = self.rhs(y[i] + h * k3, lna[i] + h)
            y[i + 1] = y[i] + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        self.lna, self.y, self.h = lna, y, h

    def E(self, a):
        return math.sqrt(self.Om0 / a ** 3 + 1 - self.Om0)

    def dE(self, a):   # dE / dlna
        return -1.5 * self.Om0 / a ** 3 / self.E(a)

    def rhs(self, y, lna):
        a = math.exp(lna)
        hf = -2 - self.dE(a) / self.E(a)
        om = self.Om0 / a ** 3 / self.E(a) ** 2
        return numpy.array([y[1], hf * y[1] + 1.5 * om * y[0], y[3], hf * y[3] + 1.5 * om * (y[2] - y[0] ** 2)])

    def at(self, a):
        """(D1, D1', D1'', D2, D2', D2'') at a."""
        l = math.log(a)
        i = min(int((l - self.lna[0]) / self.h), len(self.lna) - 2)
        y, x, d = self.y[i], self.lna[i], l - self.lna[i]
        k1 = self.rhs(y, x)
        k2 = self.rhs(y + d / 2 * k1, x + d / 2)
        k3 = self.rhs(y + d / 2 * k2, x + d / 2)
        k4 = self.rhs(y + d * k3, x + d)
        y = y + d / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        r = self.rhs(y, l)
        n1, n2 = self.y[-1][0], self.y[-1][2]
        return y[0] / n1, y[1] / n1, r[1] / n1, y[2] / n2, y[3] / n2, r[3] / n2

    def Gf(self, a):
        return self.at(a)[1] * a ** 2 * self.E(a)

    def gf(self, a, second=False):
        D, d1, d2 = self.at(a)[3:] if second else self.at(a)[:3]
        return (d2 * a ** 2 * self.E(a) + d1 * (a ** 2 * self.dE(a) + 2 * a ** 2 * self.E(a))) / a

    def kick(self, ai, ac, af):
        return (self.Gf(af) - self.Gf(ai)) / (ac ** 2 * self.E(ac) * self.gf(ac))

    def drift(self, ai, ac, af):
        return (self.at(af)[0] - self.at(ai)[0]) / (ac ** 3 * self.E(ac) * self.at(ac)[1] / ac)

    def lpt(self, a):
        D1, d1, _, D2, d2, _ = self.at(a)
        return (D1, D2, a ** 2 * self.E(a) * d1, a ** 2 * self.E(a) * d2,
                a ** 2 * self.E(a) * self.gf(a), a ** 2 * self.E(a) * self.gf(a, second=True))


def _window64(x, window):
    """First-cell offsets and weights (differentiable in x) along one axis, x in cells."""
    if window == 'cic':
        i0 = torch.floor(x.detach())
        f = x - i0
        return i0.long(), (0, 1), (1 - f, f)
    i0 = torch.floor(x.detach() + 0.5)
    d = x - i0
    return i0.long(), (-1, 0, 1), (0.5 * (0.5 - d) ** 2, 0.75 - d ** 2, 0.5 * (0.5 + d) ** 2)


def _cells64(x, n, window):
    """(flat cell, weight) over the window's cells; x [m, 3] float64 in cells."""
    ax = [_window64(x[:, d], window) for d in range(3)]
    for oa, wa in zip(ax[0][1], ax[0][2]):
        ia = torch.remainder(ax[0][0] + oa, n) * n
        for ob, wb in zip(ax[1][1], ax[1][2]):
            iab, wab = (ia + torch.remainder(ax[1][0] + ob, n)) * n, wa * wb
            for oc, wc in zip(ax[2][1], ax[2][2]):
                yield iab + torch.remainder(ax[2][0] + oc, n), wab * wc


CHUNK = 1 << 23


def _paint64(pos, n, window):
    out = torch.zeros(n ** 3, dtype=torch.float64, device=DEV)
    for sl, np_ in _chunks(pos):
        for idx, w in _cells64(pos(sl), n, window):
            out = out.index_add(0, idx, w) if w.requires_grad else out.index_add_(0, idx, w)
    return out.view(n, n, n)


def _read64(meshes, pos, n, window):
    outs = []
    for sl, np_ in _chunks(pos):
        acc = [0.0] * len(meshes)
        for idx, w in _cells64(pos(sl), n, window):
            acc = [a + w * m.reshape(-1)[idx] for a, m in zip(acc, meshes)]
        outs.append(torch.stack(acc, dim=1))
    return torch.cat(outs)


def _chunks(pos):
    np_ = pos(None)
    for at in range(0, np_, CHUNK):
        yield slice(at, min(at + CHUNK, np_)), np_


def _r2c64(x):
    return torch.fft.rfftn(x) / float(x.numel())


def _c2r64(k, n):
    return torch.fft.irfftn(k, s=(n, n, n)) * float(n) ** 3


def _pot64(dk, n, box):
    """dk / k^2, 0 at k = 0."""
    f = _freq(n, torch.float64)
    out = torch.empty_like(dk) if not dk.requires_grad else None
    if out is None:
        kk = (f[0] ** 2 + f[1] ** 2 + f[2] ** 2) * (2 * math.pi / box) ** 2
        kk[0, 0, 0] = math.inf
        return dk / kk
    for i in range(n):
        kk = (f[0][i] ** 2 + f[1][0] ** 2 + f[2][0] ** 2) * (2 * math.pi / box) ** 2
        if i == 0:
            kk[0, 0] = math.inf
        out[i] = dk[i] / kk
    return out


def _grad64(d, n, box):
    """i (8 sin w - sin 2w) / (6 h) along axis d."""
    w = _freq(n, torch.float64)[d] * (2 * math.pi / n)
    return 1j * ((8 * torch.sin(w) - torch.sin(2 * w)) * (n / (6.0 * box)))


def _force64(rho, nbar, factor, pos, n, box, window, want_rho=True):
    """F [np, 3], RHO [np] (or None), delta_k of the painted density."""
    dk = _r2c64(rho / nbar)
    pot = _pot64(dk, n, box)
    F = []
    for d in range(3):   # one force mesh at a time
        mesh = _c2r64(pot * _grad64(d, n, box), n)
        F.append(_read64([mesh], pos, n, window)[:, 0] * factor)
        del mesh
    RHO = _read64([rho / nbar], pos, n, window)[:, 0] if want_rho else None
    return torch.stack(F, dim=1), RHO, dk


def _spectrum64(dk, n, box):
    """k, P N, N of utils.power's integer shells (floor |n|), normalised by |dk(0)|^2."""
    nb = n // 2
    sums = torch.zeros(3, nb, dtype=torch.float64, device=DEV)
    f = _freq(n, torch.float64)
    w1 = torch.full((n, n // 2 + 1), 2.0, dtype=torch.float64, device=DEV)
    w1[:, 0] = w1[:, n // 2] = 1.0
    for i in range(n):
        q = f[0][i] ** 2 + f[1][0] ** 2 + f[2][0] ** 2
        r = torch.sqrt(q)
        s = torch.floor(r).long()
        ok = s < nb
        for j, v in enumerate((r * (2 * math.pi / box), dk[i].abs() ** 2, torch.ones_like(r))):
            sums[j].index_add_(0, s[ok], (v * w1)[ok])
    z = float(dk[0, 0, 0].abs())
    k, p, N = sums.cpu().numpy()
    return dict(k=k / N, p=p / (z * z) * box ** 3, N=None)


def _steps64(S, P, F, q, c, gr, Om0, n, box, window, acts, spectra):
    """Run K / D / F actions on float64 arrays; q(slice): positions in lattice cells of the base mesh."""
    np_ = q(None)
    nbar = np_ / float(n) ** 3
    B, RHO, seen = c['B'], None, []

    def pos(sl):
        return np_ if sl is None else q(sl).double() * B + S[sl] * (n / box)
    for t, ai, ac, af in acts:
        if t == 'K':
            P += gr.kick(ai, ac, af) * F
        elif t == 'D':
            S += gr.drift(ai, ac, af) * P
        else:
            F, RHO, dk = _force64(_paint64(pos, n, window), nbar, 1.5 * Om0, pos, n, box, window)
            if spectra:
                seen.append(_spectrum64(dk, n, box))
            del dk
    return S, P, F, RHO, seen


def _u32mul(a, b):
    """High and low words of the product of 32-bit words held in int64."""
    lo = a * (b & 0xFFFF)
    mid = a * (b >> 16) + (lo >> 16)
    return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)


def _uniforms(lin, seed):
    """Two uniforms per counter: Philox4x32-10 (Salmon et al. 2011), key = seed."""
    c = [lin & 0xFFFFFFFF, lin >> 32, torch.zeros_like(lin), torch.zeros_like(lin)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for r in range(10):
        h0, l0 = _u32mul(c[0], 0xD2511F53)
        h1, l1 = _u32mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = lambda a, b: ((a >> 5).double() * 67108864.0 + (b >> 6).double() + 0.5) * 2.0 ** -53   # noqa: E731
    return u(c[0], c[1]), u(c[2], c[3])


def _whitenoise64(n, seed, unitary):
    """Unit-variance Hermitian modes, Box-Muller on the mode's own counter; the
    l = 0 and l = n/2 planes take the smaller of a pair's counters."""
    nz = n // 2 + 1
    out = torch.empty(n, n, nz, dtype=torch.complex128, device=DEV)
    l = torch.arange(nz, device=DEV).view(1, nz)
    j = torch.arange(n, device=DEV).view(n, 1)
    for i in range(n):
        me, mirror = i * n + j, ((n - i) % n) * n + (n - j) % n
        plane = (l == 0) | (l == n // 2)
        low = plane & (mirror < me)
        u1, u2 = _uniforms(torch.where(low, mirror, me) * nz + l, seed)
        amp = torch.ones_like(u1) if unitary else torch.sqrt(-torch.log(u1))
        re, im = amp * torch.cos(2 * math.pi * u2), amp * torch.sin(2 * math.pi * u2)
        own = plane & (mirror == me)
        real = torch.where(re >= 0, 1.0, -1.0).double() if unitary else re * math.sqrt(2.0)
        out[i] = torch.complex(torch.where(own, real, re), torch.where(own, 0.0, torch.where(low, -im, im)))
    out[0, 0, 0] = 0
    return out


def _linear64(wn, table, n):
    f = _freq(n, torch.float64)
    out = torch.empty_like(wn)
    for i in range(n):
        out[i] = wn[i] * table[(f[0][i] ** 2 + f[1][0] ** 2 + f[2][0] ** 2).long()]
    return out


def _lpt64(dlin, n, box, q, order=2):
    """First- and second-order displacement fields read out (CIC) at the lattice."""
    def psi(dk):
        pot = _pot64(dk, n, box)
        return torch.cat([_read64([_c2r64(pot * _grad64(d, n, box), n)], q, n, 'cic') for d in range(3)], dim=1)
    if order == 1:
        return psi(dlin), None
    pot = _pot64(dlin, n, box)
    g = [_grad64(d, n, box) for d in range(3)]
    ii = [_c2r64(pot * g[d] * g[d], n) for d in range(3)]
    src = ii[0] * (ii[1] + ii[2]) + ii[1] * ii[2]
    del ii
    for a, b in ((0, 1), (1, 2), (2, 0)):
        src = src - _c2r64(pot * g[a] * g[b], n) ** 2
    return psi(dlin), psi(_r2c64(src * (3.0 / 7)))


def _leapfrog(st, first):
    acts = [('F', st[0], st[0], st[0])] if first else []
    for a0, a1 in zip(st[:-1], st[1:]):
        ah = (a0 * a1) ** 0.5
        acts += [('K', a0, a0, ah), ('D', a0, ah, a1), ('F', a0, a1, a1), ('K', ah, a1, a1)]
    return acts


def _positions64(q):
    return lambda sl: q(None) if sl is None else q(sl).double()


def exact(case, seed):
    c = dict(case)
    if c['kind'] == 'grad':
        return _grad_exact(c, seed)
    with torch.no_grad():
        if c['kind'] == 'step':
            n = c['nc'] * c['B']
            q = _explicit_of(c['explicit'], c['nc'], seed)[0] if c['explicit'] else _lattice_of(c['nc'], c['shift'])
            S, P, F = (x.double() for x in _evolved(c['nc'], c['box'], q, c['a0'], seed))
            S, P, F, RHO, seen = _steps64(S, P, F, q, c, _Growth(OM0), OM0, n, c['box'], c['window'],
                                          _leapfrog(_stages(c), False), c['monitor'])
            return dict(S=S, P=P, F=F, RHO=RHO, seen=seen)
        if c['kind'] == 'ics':
            n, box = c['nc'], c['box']
            wn = _whitenoise64(n, int(seed), c['unitary'])
            dlin = _linear64(wn, torch.from_numpy(_shell_table(n, box, _linear_power())).to(DEV), n)
            x1, x2 = _lpt64(dlin, n, box, _positions64(_lattice_of(n, 0.0)), c['order'])
            D1, D2, A1, A2, g1, g2 = _Growth(OM0).lpt(c['a0'])
            out = [D1 * x1, A1 * x1, g1 * x1]
            if x2 is not None:
                out = [out[0] + D2 * x2, out[1] + A2 * x2, out[2] + g2 * x2]
            return dict(wn=wn, dlin=dlin, S=out[0], P=out[1], F=out[2])
        if c['kind'] == 'power':
            return _spectrum64(_r2c64(_density(c, seed).double()), c['n'], c['box'])
        if c['kind'] == 'catalog':
            x = _catalog(c, seed)
            pos = lambda sl: x.shape[0] if sl is None else x[sl].double() * (c['n'] / c['box'])   # noqa: E731
            rho = _paint64(pos, c['n'], c['window'])
            return dict(rho=rho, dk=_r2c64(rho), back=rho, at=_read64([rho], pos, c['n'], c['window'])[:, 0])
        ks, pks, Ss = [], [], []
        n, nc, box = c['nc'] * c['B'], c['nc'], 4.0 * c['nc']
        q = _lattice_of(nc, 0.0)
        st = [float(x) for x in numpy.linspace(c['a0'], c['a1'], c['steps'] + 1)]
        for r in _requests(c, seed):
            gr = _Growth(r.Om0)
            table = torch.from_numpy(_shell_table(nc, box, _linear_power(r.Om0, r.sigma8))).to(DEV)
            x1, x2 = _lpt64(_linear64(_whitenoise64(nc, r.seed, False), table, nc), nc, box, _positions64(q))
            D1, D2, A1, A2 = gr.lpt(c['a0'])[:4]
            S, P, _, _, _ = _steps64(D1 * x1 + D2 * x2, A1 * x1 + A2 * x2, torch.zeros_like(x1), q, c, gr, r.Om0, n, box,
                                     c['window'], _leapfrog(st, True), False)
            rho = _paint64(lambda sl: nc ** 3 if sl is None else q(sl).double() * c['B'] + S[sl] * (n / box), n, c['window'])
            sp = _spectrum64(_r2c64(rho), n, box)
            N = _spectrum_counts(n)
            ks.append(sp['k'])
            pks.append(sp['p'] / N)
            Ss.append(S)
        return dict(k=ks, pk=pks, S=Ss)


def _spectrum_counts(n):
    f = _freq(n, torch.float64)
    w = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device=DEV)
    w[0] = w[n // 2] = 1.0
    s = torch.floor(torch.sqrt(f[0] ** 2 + f[1] ** 2 + f[2] ** 2)).long().reshape(-1)
    ok = s < n // 2
    return torch.bincount(s[ok], weights=w.repeat(n * n)[ok], minlength=n // 2).cpu().numpy()


def _grad_exact(c, seed):
    """The forward model in float64 and its gradient by torch's reverse mode."""
    nc, B, box = c['nc'], c['B'], c['box']
    n = nc * B
    if n > 128:
        return None
    q = _lattice_of(nc, 0.0)
    q64 = q(slice(0, nc ** 3)).double()
    st, nbar = _stages(c), nc ** 3 / float(n) ** 3
    acts = _leapfrog(st, True)
    target = torch.exp(0.3 * torch.randn(n, n, n, generator=_gen(5), device=DEV)).double()

    def scalars(Om0):
        gr = _Growth(Om0)
        f = [gr.kick(*a[1:]) if a[0] == 'K' else gr.drift(*a[1:]) if a[0] == 'D' else 1.5 * Om0 for a in acts]
        return numpy.array(f + list(gr.lpt(st[0])[:4]))
    table = lambda Om0: _shell_table(nc, box, _linear_power(Om0))   # noqa: E731
    wn = _whitenoise64(nc, int(seed), False).to(torch.complex64).to(torch.complex128).requires_grad_(True)
    sc = torch.from_numpy(scalars(OM0)).requires_grad_(True)
    T = torch.from_numpy(table(OM0)).to(DEV).requires_grad_(True)
    fr = _freq(nc, torch.float64)
    shell = (fr[0] ** 2 + fr[1] ** 2 + fr[2] ** 2).long()
    m = len(acts)
    x1, x2 = _lpt64(wn * T[shell], nc, box, _positions64(q))
    S, P = sc[m].to(DEV) * x1 + sc[m + 1].to(DEV) * x2, sc[m + 2].to(DEV) * x1 + sc[m + 3].to(DEV) * x2
    F = None
    for i, (t, _, _, _) in enumerate(acts):
        if t == 'K':
            P = P + sc[i].to(DEV) * F
        elif t == 'D':
            S = S + sc[i].to(DEV) * P
        else:
            pos = lambda sl, S=S: nc ** 3 if sl is None else (q64 * B + S * (n / box))[sl]   # noqa: E731
            F = _force64(_paint64(pos, n, c['window']), nbar, sc[i].to(DEV), pos, n, box, c['window'], want_rho=False)[0]
    rho = _paint64(lambda sl: nc ** 3 if sl is None else (q64 * B + S * (n / box))[sl], n, 'cic') / nbar
    loss = ((rho - target) ** 2).sum()
    gw, gs, gT = torch.autograd.grad(loss, (wn, sc, T))
    w = torch.full((nc, nc, nc // 2 + 1), 2.0, dtype=torch.float64, device=DEV)
    w[:, :, 0] = w[:, :, nc // 2] = 1.0
    # torch's gradient treats the modes of the l = 0 and l = n/2 planes as free
    # and counts every stored mode once; the Hermitian half-space gradient g has
    # dL = sum w Re(conj(g) dmode)
    h = 1e-5
    dom = float((gs * torch.from_numpy((scalars(OM0 + h) - scalars(OM0 - h)) / (2 * h))).sum())
    dom += float((gT * torch.from_numpy((table(OM0 + h) - table(OM0 - h)) / (2 * h)).to(DEV)).sum())
    return dict(loss=float(loss.detach()), g=gw / w, dom=dom)
