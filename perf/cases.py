"""Measured cases: the calls a DGFS program makes, through the public entry
points of ``frfs_b200``, over the sizes it makes them at.

Kinds
  point    Q(f) at one solution point (``sm.fs``), the call frfs's own
           collision loop makes
  collide  Q(f) at every point of a bank (``DGFSSystem.collide``)
  stage    face values, wall sums and the fused Runge-Kutta residual
           (``DGFSSystem.updatebc`` + ``rk_stage``)
  step     one SSP-RK2 step with its two collision sweeps (the stepper)
  mixture  the four Q_pq of a binary VSS mixture on a bank (``fs_all``)
  sur      the surrogate-assisted collision sweep (``VHSSurrogate.collide``)
  train    forward and backward pass of the surrogate's network

``listed()`` holds the configurations of ``frfs_b200.workloads`` and of the
test suite; ``draw()`` spreads the same kinds over element counts (blocks of
32 with ragged tails), velocity grids, orders and precisions.  ``exact()``
evaluates the same formulas in 64 bits with torch and numpy alone.
"""

import glob
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(ROOT, 'dgfs-be-solver_b200')
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

_F64 = torch.float64


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: frfs's per-point collision of the 0D relaxation
        dict(name='relax-point-f64', kind='point', prec=64, mesh='strip',
             nx=1, ny=1, order=1, Nv=16, Nrho=8, M=6, project=0),
        # the headline sweep: Couette slab, 576 points, conservation on
        dict(name='couette-collide-f32', kind='collide', prec=32,
             mesh='strip', nx=64, ny=1, order=2, Nv=24, Nrho=12, M=16,
             project=1),
        # the same sweep in the FP64 parity mode
        dict(name='couette-collide-f64', kind='collide', prec=64,
             mesh='strip', nx=64, ny=1, order=2, Nv=24, Nrho=12, M=16,
             project=0),
        # the largest velocity grid: channel on 24x12 quads, 2,592 points
        dict(name='channel-collide-f32', kind='collide', prec=32, mesh='box',
             nx=24, ny=12, order=2, Nv=32, Nrho=16, M=24, project=1),
        # a coarse velocity grid on a ragged bank (37 elements: one full and
        # one 5-element block), p = 3
        dict(name='ragged-collide-f32', kind='collide', prec=32,
             mesh='strip', nx=37, ny=1, order=3, Nv=16, Nrho=8, M=6,
             project=0),
        # the transport half of a Couette stage: 64 elements, two blocks
        dict(name='couette-stage-f32', kind='stage', prec=32, mesh='strip',
             nx=64, ny=1, order=2, Nv=24, Nrho=12, M=16, project=0),
        # transport on the cylinder's O-grid at p = 3: 640 elements, 1.3 GB
        # per register
        dict(name='cylinder-stage-f32', kind='stage', prec=32, mesh='ogrid',
             nx=40, ny=16, order=3, Nv=32, Nrho=16, M=24, project=0),
        # transport in FP64 on a ragged channel mesh (91 elements)
        dict(name='channel-stage-f64', kind='stage', prec=64, mesh='box',
             nx=13, ny=7, order=2, Nv=24, Nrho=12, M=16, project=0),
        # a whole time step of the Couette run, stages replayed as graphs
        dict(name='couette-step-f32', kind='step', prec=32, mesh='strip',
             nx=64, ny=1, order=2, Nv=24, Nrho=12, M=16, project=1),
        # argon-krypton mixture: all four ordered pairs on 144 points
        dict(name='mixture-collide-f32', kind='mixture', prec=32, nupts=9,
             nx=16, Nv=24, Nrho=12, M=32),
        # the surrogate-assisted sweep on Couette-like near-equilibrium states
        dict(name='couette-surrogate-f32', kind='sur', prec=32, mesh='strip',
             nx=64, ny=1, order=2, Nv=24, Nrho=12, M=16, project=1),
        # one training batch of the surrogate's network, both directions
        dict(name='surrogate-train', kind='train', prec=32, batch=1024),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# velocity grids of the configurations: (Nv, Nrho, M)
_GRIDS = {16: (8, 6), 24: (12, 16), 32: (16, 24)}


def draw(rng):
    top = max(_cost(c) for c in listed())
    most = max(work(c)['bytes'] for c in listed())
    while True:
        kind = rng.choice(['point', 'collide', 'collide', 'collide', 'stage',
                           'stage', 'stage', 'step', 'mixture', 'sur',
                           'train'])
        c = dict(kind=kind, prec=32)
        if kind == 'train':
            c['batch'] = 8*_logint(rng, 16, 512)
            return c
        if kind == 'mixture':
            c['Nv'] = rng.choice([16, 24])
            c.update(nupts=rng.choice([4, 9]), nx=_logint(rng, 1, 48),
                     Nrho=c['Nv']//2, M=rng.choice([12, 32]))
        else:
            if kind in ('point', 'collide', 'stage'):
                c['prec'] = rng.choice([32, 32, 64])
            Nv = {'point': [16, 24, 32], 'collide': [16, 24, 24, 32],
                  'stage': [16, 24, 32], 'step': [16, 24], 'sur': [24]}
            c['Nv'] = rng.choice(Nv[kind])
            c['Nrho'], c['M'] = _GRIDS[c['Nv']]
            c['order'] = rng.choice([1, 2, 3] if kind == 'stage' else [1, 2])
            c['mesh'] = rng.choice(['strip', 'box', 'ogrid']) \
                if kind == 'stage' else rng.choice(['strip', 'box'])
            if kind == 'sur':
                c['mesh'] = 'strip'
            if c['mesh'] == 'ogrid' and c['Nv'] == 16:
                c['mesh'] = 'box'      # too coarse for the Mach-2 inflow
            if c['mesh'] == 'strip':
                c['nx'], c['ny'] = _logint(rng, 8 if kind == 'sur' else 1,
                                           256 if kind == 'stage' else 96), 1
                if kind == 'point':
                    c['nx'] = 1
            elif c['mesh'] == 'box':
                c['nx'], c['ny'] = _logint(rng, 3, 40), _logint(rng, 2, 24)
            else:
                c['nx'], c['ny'] = _logint(rng, 8, 48), _logint(rng, 2, 20)
            c['project'] = rng.choice([0, 1]) if c['prec'] == 32 else 0
        if _cost(c) <= top and work(c)['bytes'] <= most:
            return c


def _cost(c):
    """Rough time of a pass in ms, to keep drawn cases within the listed."""
    if c['kind'] == 'train':
        return 0.2
    w = work(c)
    rate = 8e12 if c['prec'] == 64 else 2e13
    return max(w['flops']/rate, w['bytes']/2e12)*1e3


def _npts(c):
    if c['kind'] == 'mixture':
        return c['nupts']*c['nx']
    return (c['order'] + 1)**2*c['nx']*c['ny']


def work(case):
    """Bytes: every input read once and every output written once.  FLOPs:
    a real-input Q(f) needs one complex transform per radial node and
    direction, one real transform of f, per radial node and for gain and
    loss, the phase products and the squares; a mixture pair two real
    inverse and one real forward transform per node and direction."""
    k = case['kind']
    if k == 'train':
        b, nin, wd, nout = case['batch'], 256, 512, 256
        fwd = 2*(nin*wd + 2*wd*wd + wd*nout + nin*nout)
        npar = fwd//2 + 3*wd + nout
        return {'bytes': float(b*4*(nin + 2*nout) + npar*(2 + 4)),
                'flops': float(b*(2*fwd + 2*(wd*nout + 2*wd*wd)))}
    N, P, M, es = case['Nv'], case['Nrho'], case['M'], case['prec']//8
    V, n = N**3, _npts(case)
    fft = 5.0*V*math.log2(V)
    if k == 'mixture':
        return {'bytes': float(n*V*es*4),
                'flops': n*4*((1.5*P*M + 2)*fft + 8.0*P*M*V)}
    q = (P*M + 0.5*(P + 3))*fft + 6.0*P*M*V
    if k == 'point':
        return {'bytes': 2.0*V*es, 'flops': q}
    if k in ('collide', 'sur'):
        return {'bytes': 2.0*n*V*es, 'flops': n*q if k == 'collide' else
                n*(2*0.5*fft + 2.0*220*V)}
    p1 = case['order'] + 1
    # u, two Runge-Kutta terms and Q in, one bank out; face values are an
    # intermediate.  Per element and velocity: normal interface fluxes,
    # the flux divergence and the lift
    U, F = p1*p1, 4*p1
    ne = case['nx']*case['ny']
    st = {'bytes': 5.0*n*V*es,
          'flops': float(ne*V*2*(F*p1 + 2*U*p1 + F*p1 + 6*U))}
    if k == 'stage':
        return st
    return {'bytes': 2*(2.0*n*V*es) + 2*st['bytes'],
            'flops': 2*(n*q + st['flops'])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _config(case):
    from frfs_b200 import workloads
    from frfs_b200.inifile import Inifile
    prec = 'double' if case['prec'] == 64 else 'single'
    N, order = case['Nv'], case['order']
    if case['mesh'] == 'strip':
        ini = workloads.couette_n24(prec, M=case['M'], nele=case['nx'])
    elif case['mesh'] == 'box':
        ini = workloads.channel_n32(prec, nx=case['nx'], ny=case['ny'],
                                    Nv=N, Nrho=case['Nrho'], M=case['M'])
    else:
        ini = workloads.cylinder_n32(prec, ntheta=case['nx'], nr=case['ny'],
                                     order=order, Nv=N, Nrho=case['Nrho'],
                                     M=case['M'])
    cfg = Inifile(ini)
    cfg.set('constants', 'Nv', N)
    cfg.set('constants', 'NvBatchSize', N**3)
    cfg.set('constants', 'Nrho', case['Nrho'])
    cfg.set('solver', 'order', order)
    cfg.set('backend-b200', 'vhs-project', case['project'])
    cfg.set('backend-b200', 'cuda-graphs', 1 if case['kind'] == 'step' else 0)
    # spatially uniform initial condition: the banks are filled below
    cfg.set('soln-ics', 'noise', 0.0)
    if N < 24:
        # a coarse grid resolves the walls' Maxwellians in a narrower box
        cfg.set('velocity-mesh', 'dev', 4.8)
    return cfg


def _halfwidth(case):
    if case['kind'] == 'mixture':
        return 5.0
    if case['mesh'] == 'ogrid':
        return 6.0
    dev = 4.8 if case['Nv'] < 24 else 5.0
    return dev + (0.5 if case['mesh'] == 'strip' else 0.0)


def _states(case, seed, nupts, neles, mass=1.0):
    """Per-point parameters of a two-Maxwellian mixture: moments that vary
    smoothly along the mesh and by a little from point to point, and a
    distance from equilibrium between 0.3 % and order one per element."""
    r = np.random.default_rng(seed)
    x = np.arange(neles)/max(neles, 1)
    wave = lambda lo, hi: (0.5*(lo + hi) + 0.5*(hi - lo)*np.sin(
        2*np.pi*(r.integers(1, 4)*x + r.uniform()))[None, :] *
        r.uniform(0.5, 1.0) + 0.01*r.uniform(-1, 1, (nupts, neles)))
    rho, T = wave(0.7, 1.5), wave(0.8, 1.15)
    u = [wave(-0.4, 0.4) for _ in range(3)]
    lo, hi = (3e-3, 0.3) if case['kind'] == 'sur' else (1e-2, 1.0)
    d = np.exp(r.uniform(np.log(lo), np.log(hi), neles))[None, :]
    if case['kind'] == 'sur':
        # most of the slab is close to equilibrium, the wall layers are not
        d = np.where(r.uniform(size=neles) < 0.85, np.minimum(d, 2e-2), d)
    w = r.uniform(0.3, 0.7, (nupts, neles))
    du = [0.7*d*r.uniform(-1, 1, (nupts, neles)) for _ in range(3)]
    dT = 0.3*d*r.uniform(-1, 1, (nupts, neles))
    out = dict(rho=rho, w=w, T1=T*(1 + dT), T2=T*(1 - dT), mass=mass)
    for i in range(3):
        out[f'u1{i}'] = u[i] + (1 - w)*du[i]
        out[f'u2{i}'] = u[i] - w*du[i]
    return out


def _distribution(st, upt, L, N, dev, noise, seed):
    """f[V, neles] of one solution point index, 64 bits."""
    t = lambda k: torch.as_tensor(st[k][upt], dtype=_F64, device=dev)
    c = torch.linspace(-L + L/N, L - L/N, N, dtype=_F64, device=dev)[:, None]
    m = st['mass']
    f = 0
    for s, w in (('1', t('w')), ('2', 1 - t('w'))):
        T = t('T' + s)/m
        a, b, g = (torch.exp(-(c - t(f'u{s}{i}'))**2/T) for i in range(3))
        a = a*(w*t('rho')/(math.pi*T)**1.5)
        f = f + a[:, None, None]*b[None, :, None]*g[None, None]
    f = f.reshape(N**3, -1)
    if noise:
        gen = torch.Generator(device=dev).manual_seed(1000*seed + upt)
        f = f*(1 + noise*torch.randn(f.shape, generator=gen, device=dev,
                                     dtype=_F64))
    return f


def _fill(view, case, seed, L, mass=1.0):
    """A bank's (nupts, leaddim) storage: frfs's AoSoA(32) order, padding
    lanes of the last element block zero."""
    N = case['Nv']
    if case['kind'] == 'mixture':
        nupts, neles = case['nupts'], case['nx']
    else:
        nupts, neles = (case['order'] + 1)**2, case['nx']*case['ny']
    st = _states(case, seed, nupts, neles, mass)
    nblk = -(-neles//32)
    noise = 0.01 if case.get('mesh') == 'box' else 0.0
    for i in range(nupts):
        f = _distribution(st, i, L, N, view.device, noise, seed)
        f = torch.nn.functional.pad(f, (0, nblk*32 - neles))
        view[i, :nblk*32*N**3] = f.view(N**3, nblk, 32).transpose(
            0, 1).reshape(-1).to(view.dtype)


def _network_inputs(batch, seed, dev):
    """Standardised features and an output gradient of the loss's size."""
    g = torch.Generator(device=dev).manual_seed(seed)
    X = torch.randn(batch, 256, generator=g, device=dev)
    dY = torch.randn(batch, 256, generator=g, device=dev)/batch
    return X, dY


def prepare(case, seed):
    dev = torch.device('cuda', torch.cuda.current_device())
    kind = case['kind']
    if kind == 'train':
        from frfs_b200.surrogate import MLP
        mlp = MLP(dev, seed=seed)
        X, dY = _network_inputs(case['batch'], seed, dev)
        # a training loop replays the captured step
        mlp.forward(X, keep=True)
        mlp.backward(dY)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            Y = mlp.forward(X, keep=True)
            mlp.backward(dY)
        return dict(case=case, mlp=mlp, X=X, dY=dY, Y=Y, graph=graph)
    from frfs_b200.backend import B200Backend
    if kind == 'mixture':
        from frfs_b200 import workloads
        from frfs_b200.inifile import Inifile
        from frfs_b200.mixture import (DGFSBiVelocityMesh,
                                       DGFSBiVSSGLLScatteringModel)
        cfg = Inifile(workloads.mixture_n24(
            'single', Nv=case['Nv'], Nrho=case['Nrho'], M=case['M'], Mpre=32))
        be = B200Backend(cfg)
        vm = DGFSBiVelocityMesh(be, cfg)
        sm = DGFSBiVSSGLLScatteringModel(be, cfg, vm)
        shape = (case['nupts'], vm.vsize(), case['nx'])
        f = [be.matrix(shape) for _ in range(2)]
        Q = [be.matrix(shape) for _ in range(2)]
        for s in range(2):
            _fill(f[s].view2d(), case, 2*seed + s, vm.L(), vm.masses()[s])
        return dict(case=case, sm=sm, f=f, Q=Q)
    from frfs_b200.system import DGFSSystem
    cfg = _config(case)
    system = DGFSSystem(B200Backend(cfg), cfg,
                        nreg=4 if kind == 'stage' else 3)
    bank = system.bank
    for r in range(3 if kind == 'stage' else 1):
        _fill(bank[r].view2d(), case, seed + 7919*r, system.vm.L())
    st = dict(case=case, system=system, dt=cfg.getfloat(
        'solver-time-integrator', 'dt'))
    if kind == 'step':
        from frfs_b200.steppers import get_stepper
        st['stepper'] = get_stepper(system, cfg)
        st['f0'] = bank[0].data.clone()
    if kind == 'sur':
        from frfs_b200.surrogate import VHSSurrogate
        system.surrogate = VHSSurrogate(system.sm, seed=seed)
    return st


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'train':
        state['graph'].replay()
        return {'Y': state['Y'], 'grad': state['mlp'].flat_g}
    if kind == 'mixture':
        f, Q = state['f'], state['Q']
        state['sm'].fs_all(*f, *Q)
        return {'Q0': Q[0].data, 'Q1': Q[1].data}
    s = state['system']
    if kind == 'point':
        s.sm.fs(s.bank[0], s.bank[1], 0, 0)
        return s.bank[1].data
    if kind in ('collide', 'sur'):
        s.collide(0.0, 0, 1)
        return s.bank[1].data
    if kind == 'stage':
        # the second stage of SSP-RK2 into a register of its own
        s.updatebc(0.0, 0, 3, 0, 0)
        s.rk_stage(0, 3, 0.5, 1, 0.5, 0, 0.5*state['dt'], 2, interp=False)
        return s.bank[3].data
    # the step updates register 0 in place: the state to advance arrives there
    s.bank[0].data.copy_(state['f0'])
    i = state['stepper'].step(0.0, state['dt'])
    return s.bank[i].data


# ---------------------------------------------------------------------------
# the same results in 64 bits, torch and numpy alone
# ---------------------------------------------------------------------------
_GAS = dict(R0=8.3144598, NA=6.0221409e+23, m=39.96e-3, H0=1e-3, rho0=1.5e-3,
            dRef=4.17e-10, omega=0.81)


def _design(npts):
    f = glob.glob(os.path.join(_PKG, 'frfs_b200', 'data', 'sphericaldesign',
                               f'womersley-*-m{npts:05d}.txt'))
    return np.loadtxt(f[0])


def _freq(N):
    return np.concatenate((np.arange(N//2), np.arange(-N//2, 0))).astype(float)


def _sinc(x):
    return np.sin(x + 1e-15)/(x + 1e-15)


def _lnorm(N):
    l = _freq(N)
    return np.sqrt(l[:, None, None]**2 + l[None, :, None]**2 + l**2)


def _phases(N, fac, sz, sign, dev):
    """e^{sign i fac s.l} on the grid."""
    l = torch.as_tensor(_freq(N), device=dev)
    e = [torch.exp(1j*sign*fac*float(sz[a])*l) for a in range(3)]
    return e[0][:, None, None]*e[1][None, :, None]*e[2][None, None, :]


def _vhs_exact(f, case, L):
    """Q(f) of the rows f (n, V): 64-bit FFTs of the fast spectral VHS
    operator, with the optional projection onto zero collision moments."""
    N, P, M, dev = case['Nv'], case['Nrho'], case['M'], f.device
    V, g = N**3, _GAS
    n0 = g['rho0']/g['m']*g['NA']
    invKn = g['H0']*math.sqrt(2.0)*math.pi*n0*g['dRef']**2
    pre = invKn/(2.0**(3 - g['omega'])*math.gamma(2.5 - g['omega'])*math.pi)
    gam = 2.0*(1 - g['omega'])
    R = 4.0*L/(3.0 + math.sqrt(2.0))
    z, w = np.polynomial.legendre.leggauss(P)
    qz, qw = 0.5*R*(1 + z), 0.5*R*w
    sz, sw = _design(2*M)[:M], 2*math.pi/M
    ln = _lnorm(N)
    b1 = [torch.as_tensor(2*qw[p]*sw/V*qz[p]**(gam + 2)*4*math.pi *
                          _sinc(math.pi/L*qz[p]/2*ln), device=dev)
          for p in range(P)]
    b2 = torch.as_tensor(sum(qw[p]*qz[p]**(gam + 2)*16*math.pi**2 *
                             _sinc(math.pi/L*qz[p]*ln) for p in range(P)),
                         device=dev)
    ax = (1, 2, 3)
    fwd = lambda a: torch.fft.fftn(a, dim=ax)
    inv = lambda a: torch.fft.ifftn(a, dim=ax, norm='forward')
    out = torch.empty_like(f)
    step = max(1, (1 << 23)//V)
    for i in range(0, f.shape[0], step):
        x = f[i:i + step].view(-1, N, N, N)
        F = fwd(x.to(torch.complex128))/V
        G = torch.zeros_like(F)
        for p in range(P):
            S = torch.zeros_like(x)
            for q in range(M):
                e = _phases(N, math.pi/L*qz[p]/2, sz[q], 1, dev)
                S += (inv(e*F)*inv(e.conj()*F)).real
            G += b1[p]*fwd(S.to(torch.complex128))
        Q = pre*(inv(G).real - x*inv(b2*F).real)
        out[i:i + step] = Q.reshape(-1, V)
    if case['project']:
        c = np.linspace(-L + L/N, L - L/N, N)
        X = np.meshgrid(c, c, c, indexing='ij')
        phi = np.stack([np.ones(V)] + [a.ravel() for a in X] +
                       [sum(a*a for a in X).ravel()])
        phi = torch.as_tensor(phi, device=dev)
        out -= torch.linalg.solve(phi @ phi.T, phi @ out.T).T @ phi
    return out


def _legendre(n, x):
    """Orthonormal Legendre polynomials 0..n and derivatives at x."""
    x = np.asarray(x, float)
    p, d = [], []
    for k in range(n + 1):
        c = np.zeros(k + 1)
        c[k] = math.sqrt(k + 0.5)
        p.append(np.polynomial.legendre.legval(x, c))
        d.append(np.polynomial.legendre.legval(
            x, np.polynomial.legendre.legder(c)) if k else 0*x)
    return np.array(p), np.array(d)


def _lobatto(n):
    """n-point Gauss-Lobatto rule."""
    c = np.zeros(n)
    c[-1] = 1
    x = np.r_[-1.0, np.sort(np.polynomial.legendre.legroots(
        np.polynomial.legendre.legder(c))) if n > 2 else [], 1.0]
    return x, 2.0/(n*(n - 1)*np.polynomial.legendre.legval(x, c)**2)


def _stage_exact(u, case, L, A, a, B, b, C, g):
    """a A + b B + g (-div F(u) + C) on a box of nx x ny rectangles, u
    (U, V, E): nodal flux reconstruction on Gauss-Legendre points, upwind
    faces, diffuse walls; lifts integrated with the (p+1)-point Lobatto
    rule."""
    nx, ny, p1, N, dev = case['nx'], case['ny'], case['order'] + 1, \
        case['Nv'], u.device
    strip = case['mesh'] == 'strip'
    hx, hy = 1.0/nx, (1.0/nx if strip else 0.5/ny)
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=_F64,
                                  device=dev)
    z, _ = np.polynomial.legendre.leggauss(p1)
    pz, dz = _legendre(p1 - 1, z)
    nod = lambda x: np.linalg.solve(pz, _legendre(p1 - 1, x)[0])  # (node, x)
    D = np.linalg.solve(pz, dz).T                 # d/dxi at node i of node j
    E = nod([-1.0, 1.0])                          # node values at the ends
    zq, wq = _lobatto(p1)
    # lift of a face function: along the face, and across it from each end
    K = lambda x: pz.T @ _legendre(p1 - 1, x)[0]  # reproducing kernel (node, x)
    along = (K(zq)*wq) @ nod(zq).T                # (node, face node)
    cross = K([-1.0, 1.0])                        # (node, end)
    c1 = np.linspace(-L + L/N, L - L/N, N)
    cx, cy, cz = (a_.ravel() for a_ in np.meshgrid(c1, c1, c1, indexing='ij'))
    V = N**3
    U = u.view(p1, p1, V, ny, nx)                 # (eta, xi, v, j, i)
    D, E, along, cross = t(D), t(E), t(along), t(cross)
    out = torch.zeros_like(U)

    def axis(Ua, c, h, periodic, wall):
        """-d/dx along the second index and last element index of Ua
        (s, n, V, q, m): s runs along the face, q over the other element
        direction."""
        ctv = t(c)
        end = torch.einsum('sjvqm,jf->fsvqm', Ua, E)
        lo, hi = end[0], end[1]                   # own traces at -1, +1
        left, right = hi.roll(1, -1), lo.roll(-1, -1)
        if not periodic:
            for side, own, nb, n in ((0, lo, left, -1.0), (-1, hi, right,
                                                           1.0)):
                fw = t(wall[side])
                out_ = ctv*n >= 0
                ul = own[..., side]               # (s, V, q)
                num = torch.einsum('svq,v->sq', ul, torch.where(
                    out_, ctv*n, 0*ctv))
                den = torch.sum(torch.where(out_, 0*ctv, ctv*n)*fw)
                gh = fw[None, :, None]*(-num/den)[:, None, :]
                nb[..., side] = torch.where(out_[None, :, None], ul, gh)
        cc = ctv[None, :, None, None]
        flo = torch.where(cc >= 0, left, lo)*cc   # upwind flux at the ends
        fhi = torch.where(cc >= 0, hi, right)*cc
        div = torch.einsum('ij,sjvqm->sivqm', D, Ua)*ctv[None, None, :, None,
                                                         None]
        for k, jump in ((0, -(flo - lo*cc)), (1, fhi - hi*cc)):
            div += torch.einsum('st,i,tvqm->sivqm', along, cross[:, k], jump)
        return -div*(2.0/h)

    maxw = lambda uy: np.exp(-cx**2 - (cy - uy)**2 - cz**2)/math.pi**1.5
    wx = {0: maxw(-0.5), -1: maxw(0.5)}
    wy = {0: maxw(0.0), -1: maxw(0.0)}
    out += axis(U, cx, hx, not strip, wx)
    Ut = U.permute(1, 0, 2, 4, 3)
    out += axis(Ut, cy, hy, strip, wy).permute(1, 0, 2, 4, 3)
    return a*A + b*B + g*(out.reshape(u.shape) + C)


def _rows(view, case, nupts, neles):
    """(nupts, V, neles) of AoSoA storage, 64 bits."""
    V, nblk = case['Nv']**3, -(-neles//32)
    x = view[:, :nblk*32*V].view(nupts, nblk, V, 32).transpose(1, 2)
    return x.reshape(nupts, V, nblk*32)[:, :, :neles].to(_F64)


def _store(x, like):
    """x (nupts, V, neles) in the AoSoA storage shape ``like``, flat."""
    nupts, V, neles = x.shape
    nblk = -(-neles//32)
    x = torch.nn.functional.pad(x, (0, nblk*32 - neles))
    buf = torch.zeros(like, dtype=_F64, device=x.device)
    buf[:, :nblk*32*V] = x.view(nupts, V, nblk, 32).transpose(1, 2).reshape(
        nupts, -1)
    return buf.view(-1)


def _mixture_exact(f, case, L):
    """Q_p = sum_q Q(f_p, f_q), f two (n, V) arrays."""
    N, P, M, dev, g = case['Nv'], case['Nrho'], case['M'], f[0].device, _GAS
    V = N**3
    ms = [1.0, 83.8e-3/g['m']]
    mr = max(ms)
    S = min(2*L/(max(4*mr/(1 + mr), 2) + math.sqrt(1 + mr) + 1),
            2*L/(max(4/(1 + mr), 2) + math.sqrt(1 + 1/mr) + 1))
    z, w = np.polynomial.legendre.leggauss(P)
    qz, qw = S*(1 + z), S*w
    sz, sp = _design(M), _design(32)
    sw, swp = 4*math.pi/M, 4*math.pi/32
    n0 = g['rho0']/g['m']*g['NA']
    gas = {0: (1.40, 0.81, 4.11e-10), 1: (1.32, 0.80, 4.76e-10)}
    dot = 1 + sz @ sp.T
    dot = np.where(np.abs(dot) < 1e-12, 0, np.maximum(dot, 0))
    ax = (1, 2, 3)
    fwd = lambda a: torch.fft.fftn(a, dim=ax)
    inv = lambda a: torch.fft.ifftn(a, dim=ax, norm='forward')
    spec = [fwd(x.view(-1, N, N, N).to(torch.complex128))/V for x in f]
    out = [torch.zeros_like(x) for x in f]
    for p in range(2):
        for q in range(2):
            al, om, d = (0.5*(gas[p][i] + gas[q][i]) for i in range(3))
            mu = ms[p]*ms[q]/(ms[p] + ms[q])
            rt = math.sqrt(1 + ms[p]/ms[q])
            pre = (rt*math.pi*n0*d*d*g['H0'])*al/(
                rt*mu**(om - 0.5)*2.0**(1 + al)*math.gamma(2.5 - om)*math.pi)
            gam, eta = 2*(1 - om), al - 1
            kq, kp = ms[q]/(ms[p] + ms[q]), ms[p]/(ms[p] + ms[q])
            Bm = torch.as_tensor(dot**eta, device=dev).to(torch.complex128)
            c = torch.zeros((N, N, N), dtype=torch.complex128, device=dev)
            G = torch.zeros_like(spec[p])
            for x in range(P):
                fac = math.pi/L*qz[x]
                fb = swp*qz[x]**(gam + 2)
                eb = torch.stack([_phases(N, kq*fac, s, -1, dev) for s in sp])
                b = fb*(Bm @ eb.view(32, V)).view(M, N, N, N)
                ec = torch.stack([_phases(N, fac, s, -1, dev) for s in sp])
                c += qw[x]*sw*fb*(Bm.sum(0) @ ec.view(32, V)).view(N, N, N)
                for y in range(M):
                    h = inv(_phases(N, fac*kq, sz[y], 1, dev)*spec[p]) * \
                        inv(_phases(N, fac*kp, sz[y], -1, dev)*spec[q])
                    G += (qw[x]*sw/V)*b[y]*fwd(h)
            out[p] += pre*(inv(G).real.reshape(-1, V) -
                           f[p]*inv(c*spec[q]).real.reshape(-1, V))
    return out


def _train_exact(case, seed, dev):
    """Forward pass and gradients of the 256-512-512-512-256 tanh network
    with a linear skip; the products read the weights in their 16-bit
    storage, everything else in 64 bits."""
    r = np.random.default_rng(seed)
    nin, wd, nout = 256, 512, 256
    W1, W2, W3, W4 = (r.standard_normal(s)/np.sqrt(s[0]) for s in
                      ((nin, wd), (wd, wd), (wd, wd), (wd, nout)))
    W4 = 0.1*W4
    W = [torch.as_tensor(w, device=dev).float().bfloat16().to(_F64)
         for w in (W1, W2, W3, W4)]
    X, dY = (a.to(_F64) for a in _network_inputs(case['batch'], seed, dev))
    H = [X]
    for w in W[:3]:
        H.append(torch.tanh(H[-1] @ w))
    Y = H[3] @ W[3]
    gW, gb, dZ = [], [], dY
    for i in (3, 2, 1, 0):
        gW.append(H[i].T @ dZ)
        gb.append(dZ.sum(0))
        if i:
            dZ = (dZ @ W[i].T)*(1 - H[i]**2)
    gW, gb = gW[::-1] + [X.T @ dY], gb[::-1]
    return {'Y': Y, 'grad': torch.cat([a.reshape(-1) for a in gW + gb])}


def exact(case, seed):
    dev = torch.device('cuda', torch.cuda.current_device())
    kind = case['kind']
    if kind == 'sur' or case.get('mesh') == 'ogrid':
        return None
    if kind == 'train':
        return _train_exact(case, seed, dev)
    V, L = case['Nv']**3, _halfwidth(case)
    if kind == 'mixture':
        nupts, neles = case['nupts'], case['nx']
    else:
        nupts, neles = (case['order'] + 1)**2, case['nx']*case['ny']
    dt = torch.float64 if case['prec'] == 64 else torch.float32
    like = (nupts, -(-neles//32)*32*V)

    def bank(sd, mass=1.0):
        v = torch.zeros(like, dtype=dt, device=dev)
        _fill(v, case, sd, L, mass)
        return _rows(v, case, nupts, neles)

    points = lambda x: x.transpose(1, 2).reshape(-1, V).contiguous()
    back = lambda r: r.view(nupts, neles, V).transpose(1, 2)
    if kind == 'mixture':
        Q = _mixture_exact([points(bank(2*seed + s, m)) for s, m in
                            enumerate((1.0, 83.8/39.96))], case, L)
        return {'Q0': _store(back(Q[0]), like), 'Q1': _store(back(Q[1]),
                                                             like)}
    u = bank(seed)
    if kind in ('point', 'collide'):
        q = torch.zeros(nupts*neles, V, dtype=_F64, device=dev)
        n = 1 if kind == 'point' else nupts*neles
        q[:n] = _vhs_exact(points(u)[:n].contiguous(), case, L)
        return _store(back(q), like)
    if kind == 'stage':
        A, C = bank(seed + 7919), bank(seed + 2*7919)
        return _store(_stage_exact(u, case, L, A, 0.5, u, 0.5, C, 0.5*1e-4),
                      like)
    Qf = lambda x: back(_vhs_exact(points(x), case, L))
    u1 = _stage_exact(u, case, L, u, 1.0, u, 0.0, Qf(u), 1e-4)
    u2 = _stage_exact(u1, case, L, u, 0.5, u1, 0.5, Qf(u1), 0.5e-4)
    return _store(u2, like)
