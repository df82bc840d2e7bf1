"""What is timed when this library's speed is judged: a list of propagations (and the other work its
users have it do) over the sizes and options in use, each through the public entry points.

    listed()           the cases, smallest calls to largest
    draw(rng)          one more case of the same ranges
    prepare(case, s)   inputs of seed s on the GPU (or on the host, for the host entry point) and what a
                       program keeps between calls: the plan, the multi-electron object, the network
    run(state)         one pass; returns everything it computes
    work(case)         the bytes and operations a pass cannot do without
    exact(case, s)     what run returns for the same inputs, in 64 bits with plain torch

A propagation is a chain of optical elements; four chains are used, those of the library's tests and
benchmark: "drifts" (drift, rectangular aperture, lens, drift: angular-representation drifts, two 2D
transforms each way), "waist" (circular aperture, resize, lens, drift to the waist: one 2D transform
on the resized grid), "quad" (drift, lens, drift with the quadratic phase treated analytically).
"""
import math
from array import array

import numpy as np
import torch

from srw_b200 import learned, srwlib, srwlpy
from srw_b200.multie import MultiE
from srw_b200.plan import Plan

DEV = 'cuda' if torch.cuda.is_available() else 'cpu'

# source phase space of the multi-electron runs: x [m], x' [rad], y [m], y' [rad], relative energy
SIGMA = (30e-6, 5e-6, 5e-6, 2e-6, 1e-3)
STEPS = 1000
LAYERS = (learned.N_IN, 256, 256, 256, learned.N_OUT)


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def listed():
    plan = dict(kind='plan', pxm=1., pxd=1., pzm=1., pzd=1.)
    return [
        # the smallest call of an alignment or optimisation loop: launches and latency
        dict(plan, name='drifts 64', chain='drifts', nx=64, ny=64),
        # the everyday coherent propagation, a power of two
        dict(plan, name='drifts 512', chain='drifts', nx=512, ny=512),
        # a ragged small mesh: lengths without a kernel of their own
        dict(plan, name='drifts 216x200', chain='drifts', nx=216, ny=200),
        # a ragged large mesh: general lengths
        dict(plan, name='drifts 2240x1536', chain='drifts', nx=2240, ny=1536),
        # the benchmark's beamline with its configured factors: 1024^2 resized to 4096^2
        dict(plan, name='waist 1024 to 4096', chain='waist', nx=1024, ny=1024, pxm=2., pxd=2., pzm=2., pzd=2.),
        # the largest coherent propagation: analytic quadratic-phase drifts at 4096^2
        dict(plan, name='quad 4096', chain='quad', nx=4096, ny=4096),
        # a stack of small wavefronts with one mesh (coherent modes, scans): one launch per pass
        dict(kind='batch', name='drifts 8 of 256', chain='drifts', nx=256, ny=256, batch=8, pxm=1., pxd=1., pzm=1., pzd=1.),
        # partially coherent runs (macro-electrons), small grid with its factors
        dict(kind='electrons', name='electrons 256', chain='waist', nx=256, ny=256, batch=64, acc=512,
             pxm=1., pxd=1.5, pzm=1., pzd=2.),
        # the benchmark's headline: 1024^2 with the learned factors, launches of 64 electrons
        dict(kind='electrons', name='electrons 1024', chain='waist', nx=1024, ny=1024, batch=64, acc=512,
             pxm=1., pxd=1.5, pzm=1.25, pzd=1.25),
        # the same run with the configured factors (what it falls back to): 4096^2 per electron
        dict(kind='electrons', name='electrons 1024 configured', chain='waist', nx=1024, ny=1024, batch=16, acc=512,
             pxm=2., pxd=2., pzm=2., pzd=2.),
        # the drop-in call on host arrays, the wavefront carrying its source's moments (the aperture
        # then recomputes them from the field)
        dict(kind='host', name='host 512 to 2048', chain='waist', nx=512, ny=512, pxm=2., pxd=2., pzm=2., pzd=2.),
        # a training step of the resize-factor network: forward, loss, backward, Adam
        dict(kind='train', name='train 128', batch=128),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """The next even number >= n with no prime factor above 7 (what a transform of the input mesh takes)."""
    n += n & 1
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 2


def draw(rng):
    kind = rng.choice(['drifts', 'drifts', 'quad', 'waist', 'waist', 'batch', 'electrons', 'electrons', 'electrons', 'host',
                       'train'])
    one = dict(pxm=1., pxd=1., pzm=1., pzd=1.)
    # factors as the users set them and as the network chooses them
    fac = dict(pxm=rng.choice([0.75, 1., 1.25, 1.5, 2.]), pxd=rng.choice([1.25, 1.5, 1.75, 2.]),
               pzm=rng.choice([0.75, 1., 1.25, 1.5, 2.]), pzd=rng.choice([1.25, 1.5, 1.75, 2.]))
    if kind in ('drifts', 'quad'):
        return dict(kind='plan', chain=kind, nx=_smooth(_spread(rng, 64, 3000)), ny=_smooth(_spread(rng, 64, 3000)), **one)
    if kind == 'waist':
        return dict(kind='plan', chain='waist', nx=_spread(rng, 96, 1024), ny=_spread(rng, 96, 1024), **fac)
    if kind == 'batch':
        return dict(kind='batch', chain='drifts', nx=_smooth(_spread(rng, 64, 512)), ny=_smooth(_spread(rng, 64, 512)),
                    batch=rng.randint(2, 16), **one)
    if kind == 'electrons':
        n = _spread(rng, 200, 1024)
        most = 16 if fac['pxm'] * fac['pxd'] * fac['pzm'] * fac['pzd'] > 8. else 32
        return dict(kind='electrons', chain='waist', nx=n, ny=n + rng.randint(-9, 0), batch=_spread(rng, 8, most),
                    acc=_spread(rng, 200, 700), **fac)
    if kind == 'host':
        return dict(kind='host', chain='waist', nx=_spread(rng, 96, 512), ny=_spread(rng, 96, 512), **fac)
    return dict(kind='train', batch=_spread(rng, 1, 512))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _mesh(case):
    """(photon energy [eV], half range [m], radius of curvature [m]) of the chain's input wavefront."""
    return {'drifts': (1000., 1e-3, 0.), 'waist': (2012., 1.5e-3, 20.), 'quad': (10000., 1e-3, 30.)}[case['chain']]


def _fields(case, seed, count=1):
    """Two lists of complex64 fields [ny, nx] on the device: beams whose size, centre, phase and weak
    vertical component follow from the seed.  "waist": the ring structure of an undulator harmonic."""
    rng = np.random.default_rng([seed, 71])
    E, r, R = _mesh(case)
    lam = 1.239842e-06 / E
    x = torch.linspace(-r, r, case['nx'], dtype=torch.float64, device=DEV)[None, :]
    y = torch.linspace(-r, r, case['ny'], dtype=torch.float64, device=DEV)[:, None]
    ex, ey = [], []
    for _ in range(count):
        s, cx, cy, ph, v = rng.uniform(0.85, 1.2), rng.normal() * 0.01 * r, rng.normal() * 0.01 * r, rng.uniform(0, 6.28), \
            rng.uniform(0.01, 0.03)
        rr = (x - cx) ** 2 + (y - cy) ** 2
        if case['chain'] == 'waist':
            q = 100. * (5870.85 / 20.) ** 2 * rr / 2.125 * s
            a = torch.polar(3.0e7 * torch.sinc(q), ph - math.pi * q)
        else:
            sig = (80e-6 if case['chain'] == 'drifts' else 60e-6) * s
            a = torch.polar(1e6 * torch.exp(-rr / (4. * sig * sig)), ph + 0. * rr)
        if R:
            p = math.pi / (lam * R) * (x * x + y * y)
            a = a * torch.polar(torch.ones_like(p), p)
        ex.append(a.to(torch.complex64))
        ey.append((a * (v * torch.polar(torch.tensor(1., dtype=torch.float64), torch.tensor(2. * ph, dtype=torch.float64)).to(DEV)
                        * (1. + 0.3 * x * y / (r * r)))).to(torch.complex64))
    return ex, ey


def _wfr(case):
    """The wavefront's description (no field arrays)."""
    E, r, R = _mesh(case)
    w = srwlib.SRWLWfr()
    m = w.mesh
    m.ne, m.nx, m.ny = 1, case['nx'], case['ny']
    m.eStart = m.eFin = E
    m.xStart, m.xFin, m.yStart, m.yFin = -r, r, -r, r
    m.zStart = R
    w.Rx = w.Ry = R
    w.dRx = w.dRy = 0.01 * R
    return w


def _host_wfr(case, ex, ey):
    w = _wfr(case)
    w.arEx, w.arEy = ex, ey
    return w


def _chain(case):
    def pp(mode=0, f=(1., 1., 1., 1.)):
        return [0, 0, 1., mode, 0, f[0], f[1], f[2], f[3], 0, 0, 0]
    L = srwlib
    if case['chain'] == 'drifts':
        return L.SRWLOptC([L.SRWLOptD(10.), L.SRWLOptA('r', 'a', 1e-3, 1e-3), L.SRWLOptL(5., 5.), L.SRWLOptD(5.)],
                          [pp(), pp(), pp(), pp()])
    if case['chain'] == 'quad':
        return L.SRWLOptC([L.SRWLOptD(30.), L.SRWLOptL(15., 15.), L.SRWLOptD(30.)], [pp(2), pp(), pp(2)])
    return L.SRWLOptC([L.SRWLOptA('c', 'a', 0.8e-3, 0.8e-3), L.SRWLOptL(10., 10.), L.SRWLOptD(10.)],
                      [pp(), pp(0, (case['pxm'], case['pxd'], case['pzm'], case['pzd'])), pp(4)])


def _offsets(case, seed):
    return np.random.default_rng([seed, 72]).normal(size=(case['batch'], 5)) * np.array(SIGMA)


def _acc_mesh(case):
    """The detector: the output range of the configured factors (2, 2) on acc x acc points."""
    E, r, _ = _mesh(case)
    d = {}
    for a, n in (('x', case['nx']), ('y', case['ny'])):
        half = 1.239842e-06 / E * 10. / (2. * 2. * r / (2. * n - 1.))
        d[a + 'Start'], d[a + 'Fin'] = -half, half
    return dict(d, nx=case['acc'], ny=case['acc'], eStart=E)


def _train_data(case, seed):
    """Normalised features, targets (log2 of factors), He-initialised weights, and Adam's two moments of
    weights and biases as they stand in the middle of a training run (after STEPS steps)."""
    rng = np.random.default_rng([seed, 73])
    X = rng.standard_normal((case['batch'], LAYERS[0])).astype(np.float32)
    T = rng.uniform(-1., 1., (case['batch'], LAYERS[-1])).astype(np.float32)
    W = [(rng.standard_normal((a, b)) * math.sqrt(2. / a)).astype(np.float32) for a, b in zip(LAYERS[:-1], LAYERS[1:])]
    b = [(0.1 * rng.standard_normal(n)).astype(np.float32) for n in LAYERS[1:]]
    to = lambda v: torch.from_numpy(v).to(DEV)  # noqa: E731
    m = [(1e-3 * rng.standard_normal(p.shape)).astype(np.float32) for p in W + b]
    v = [(1e-6 * rng.uniform(0.5, 2., p.shape)).astype(np.float32) for p in W + b]
    return to(X), to(T), [to(w) for w in W], [to(a) for a in b], [to(a) for a in m], [to(a) for a in v]


def _interleaved(a):
    return torch.view_as_real(a).reshape(-1).cpu().numpy()


def prepare(case, seed):
    if case['kind'] == 'train':
        X, T, W, b, m, v = _train_data(case, seed)
        net = learned.ResizeMLP(device=0)
        for p, a in zip(net.W + net.b + net.mW + net.mb + net.vW + net.vb, W + b + m + v):
            p.copy_(a)
        net.t = STEPS
        return dict(case=case, net=net, X=X, T=T)
    ex, ey = _fields(case, seed, case['batch'] if case['kind'] == 'batch' else 1)
    if case['kind'] == 'plan':
        plan = Plan(_wfr(case), _chain(case))
        ox, oy = plan.new_output()
        return dict(case=case, plan=plan, ins=(ex[0], ey[0]), outs=(ox, oy))
    if case['kind'] == 'batch':
        plan = Plan(_wfr(case), _chain(case))
        ox, oy = plan.new_output(case['batch'])
        return dict(case=case, plan=plan, ins=(torch.stack(ex), torch.stack(ey)), outs=(ox, oy))
    hx, hy = _interleaved(ex[0]), _interleaved(ey[0])
    if case['kind'] == 'electrons':
        me = MultiE(_host_wfr(case, hx, hy), _chain(case), _acc_mesh(case), max_batch=case['batch'], graph=True)
        acc = torch.zeros((case['acc'], case['acc']), dtype=torch.float64, device=DEV)
        me.use_accumulator(acc.data_ptr())
        st = torch.cuda.Stream()
        return dict(case=case, me=me, acc=acc, stream=st, offsets=_offsets(case, seed))
    # host arrays; the moments of the intensity as a source calculation leaves them
    I = (ex[0].abs().double() ** 2 + ey[0].abs().double() ** 2).cpu().numpy()
    r = _mesh(case)[1]
    x, y = np.linspace(-r, r, case['nx'])[None, :], np.linspace(-r, r, case['ny'])[:, None]
    n = I.sum()
    mom = [n, (I * x).sum() / n, 0., (I * y).sum() / n, 0., (I * x * x).sum() / n, 0., 0., (I * y * y).sum() / n, 0., 0.]
    return dict(case=case, chain=_chain(case), hx=hx, hy=hy, mom=[float(v) for v in mom])


def run(state):
    kind = state['case']['kind']
    if kind == 'plan':
        state['plan'].execute(*state['ins'], *state['outs'])
        return dict(ex=state['outs'][0], ey=state['outs'][1])
    if kind == 'batch':
        state['plan'].execute_batch(*state['ins'], *state['outs'])
        return dict(ex=state['outs'][0], ey=state['outs'][1])
    if kind == 'electrons':
        # a run's mean intensity, kept in the single precision of the reference's Stokes arrays
        st = state['stream']
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            state['acc'].zero_()
            state['me'].add(state['offsets'], st.cuda_stream)
            mean = (state['acc'] / state['case']['batch']).float()
        torch.cuda.current_stream().wait_stream(st)
        mean.record_stream(torch.cuda.current_stream())
        return mean
    if kind == 'host':
        w = _host_wfr(state['case'], state['hx'], state['hy'])
        w.arMomX, w.arMomY = array('d', state['mom']), array('d', state['mom'])
        srwlpy.PropagElecField(w, state['chain'])
        return dict(ex=w.arEx, ey=w.arEy, momx=np.frombuffer(w.arMomX), momy=np.frombuffer(w.arMomY))
    net = state['net']
    out = net.forward(state['X'])
    loss, dout = net.loss_grad(out, state['T'])
    dW, db = net.backward(dout)
    net.adam(dW, db)
    return dict(out=out, loss=loss.float(), dW=dW, db=db, W=net.W, b=net.b)


# ------------------------------------------------------------------------------------------------
# the bytes and operations a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _grid(case):
    """The grid the transforms run on: the input's, or the resized one."""
    g = []
    for n, m, d in ((case['nx'], case['pxm'], case['pxd']), (case['ny'], case['pzm'], case['pzd'])):
        g.append(n if m * d == 1. else _good(int(m * d * n + 0.5)))
    return g


def work(case):
    """Each input read once, each output written once; the operations of the 2D transforms
    (5 N log2 N per complex transform of N points), or of the network's multiplications."""
    if case['kind'] == 'train':
        n = sum(a * b for a, b in zip(LAYERS[:-1], LAYERS[1:]))
        first = LAYERS[0] * LAYERS[1]
        B = case['batch']
        # weights and both Adam moments read and written; no gradient with respect to the features
        return dict(bytes=4. * (6 * n + B * (LAYERS[0] + 2 * LAYERS[-1])), flops=2. * B * (3 * n - first))
    gx, gz = _grid(case)
    n_in, n_out = case['nx'] * case['ny'], gx * gz
    fft = {'drifts': 4, 'quad': 4, 'waist': 1}[case['chain']] * 2 * 5. * n_out * math.log2(n_out)
    B = case.get('batch', 1)
    if case['kind'] == 'electrons':
        return dict(bytes=16. * n_in + 8. * case['acc'] ** 2, flops=B * fft)
    return dict(bytes=16. * B * (n_in + n_out), flops=B * fft)


# ------------------------------------------------------------------------------------------------
# the same in 64 bits (the reference's definitions and physical constants, plain torch)
# ------------------------------------------------------------------------------------------------
def _good(n):
    """Transform lengths of a resized mesh: even, 2^a 3^b 5^c 7^d times at most one 11 and one 13."""
    n += n & 1
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m in (1, 11, 13, 143):
            return n
        n += 2


class _Wave(object):
    """Two complex128 components on a mesh, with the wavefront's radii and centre."""

    def __init__(self, ex, ey, E, xs, xf, zs, zf, R):
        self.f = [ex.to(torch.complex128), ey.to(torch.complex128)]
        self.nz, self.nx = ex.shape
        self.E, self.lam = E, 1.239842e-06 / E
        self.x0, self.dx = xs, (xf - xs) / (self.nx - 1)
        self.z0, self.dz = zs, (zf - zs) / (self.nz - 1)
        self.Rx = self.Rz = R
        self.eRx = self.eRz = 0.01 * R
        self.xc = self.zc = 0.

    def axes(self):
        x = self.x0 + torch.arange(self.nx, dtype=torch.float64, device=DEV) * self.dx
        z = self.z0 + torch.arange(self.nz, dtype=torch.float64, device=DEV) * self.dz
        return x[None, :], z[:, None]

    def mult(self, fx, fz=None):
        self.f = [a * fx if fz is None else a * fx * fz for a in self.f]

    def phase(self, px, pz):
        """exp(i (px(x) + pz(z)))"""
        self.mult(torch.polar(torch.ones_like(px), px), torch.polar(torch.ones_like(pz), pz))


def _transform(w, sign):
    """Centred 2D transform with the mesh's origin; w's mesh becomes the conjugate one."""
    n = (w.nx, w.nz)
    step = (w.dx, w.dz)
    off = [s + 0.5 * m * d for s, m, d in zip((w.x0, w.z0), n, step)]
    off = [o if abs(o) > 1e-6 * m * d else 0. for o, m, d in zip(off, n, step)]
    out = []
    for a in w.f:
        a = torch.fft.ifftshift(a)
        a = torch.fft.fft2(a) if sign < 0 else torch.fft.ifft2(a, norm='forward')
        out.append(torch.fft.fftshift(a) * (w.dx * w.dz))
    w.f = out
    w.x0, w.z0 = -0.5 / w.dx, -0.5 / w.dz
    w.dx, w.dz = -w.x0 / (w.nx >> 1), -w.z0 / (w.nz >> 1)
    qx = (torch.arange(w.nx, dtype=torch.float64, device=DEV)[None, :] - (w.nx >> 1)) * w.dx
    qz = (torch.arange(w.nz, dtype=torch.float64, device=DEV)[:, None] - (w.nz >> 1)) * w.dz
    w.phase(sign * 2. * math.pi * off[0] * qx, sign * 2. * math.pi * off[1] * qz)


def _after_drift(w, L):
    w.Rx += L
    w.Rz += L


def _drift(w, L):
    x0, z0 = w.x0, w.z0
    w.x0, w.z0 = -(w.nx >> 1) * w.dx, -(w.nz >> 1) * w.dz
    _transform(w, -1)
    qx, qz = w.axes()
    q2 = qx * qx + qz * qz
    c = 0.25 * w.lam * w.lam * q2
    p = -3.1415926536 * L * w.lam * q2 * (1. + c + 2. * c * c)
    w.mult(torch.polar(torch.ones_like(p), p))
    _transform(w, 1)
    w.x0, w.z0 = x0, z0
    _after_drift(w, L)


def _aperture(w, shape, D):
    x, z = w.axes()
    if shape == 'r':
        h = 0.5 * D + 1e-10
        inside = (x >= -h) & (x <= h) & (z >= -h) & (z <= h)
    else:
        inside = x * x + z * z <= (0.5 * D) * (0.5 * D)
    w.f = [torch.where(inside, a, torch.zeros((), dtype=a.dtype, device=DEV)) for a in w.f]
    for e, R in (('eRx', 'Rx'), ('eRz', 'Rz')):
        if getattr(w, R) != 0. and getattr(w, e) == 0.:
            setattr(w, e, abs(0.1 * getattr(w, R)))


def _lens(w, F):
    x, z = w.axes()
    k = w.E * 2.533865612e+06
    w.phase(-k * (x * x / F), -k * (z * z / F))
    for R, e, c in (('Rx', 'eRx', 'xc'), ('Rz', 'eRz', 'zc')):
        r = getattr(w, R)
        m = F / (F - r if F != r else 1e-23)
        setattr(w, R, r * m)
        setattr(w, e, getattr(w, e) * m * m)
        setattr(w, c, getattr(w, c) * m)
        if r * m != 0. and getattr(w, e) == 0.:
            setattr(w, e, abs(0.1 * r * m))


def _quad_drift(w, L):
    """The quadratic phase of radius R (kept three error bars away from 0 and -L) taken out analytically."""
    def radius(R, err):
        m = 3. * err
        if abs(R) < m:
            return m if R >= 0. else -m
        if abs(R + L) < m:
            return (m if R + L >= 0. else -m) - L
        return R
    Rx, Rz = radius(w.Rx, w.eRx), radius(w.Rz, w.eRz)
    big = 1e23
    inv = [1. / R if R else 0. for R in (Rx, Rz)]
    k = [(R + L) / R if R else big for R in (Rx, Rz)]
    kc = [L / R if R else big for R in (Rx, Rz)]
    le = [(L / (1. + L / R) if R != -L else big) if R else 0. for R in (Rx, Rz)]
    invL = [(1. / (L + R) if R != -L else big) if R else 1. / L for R in (Rx, Rz)]
    pl = 3.1415926536 / w.lam
    x, z = w.axes()
    w.phase(-pl * inv[0] * (x - w.xc) ** 2, -pl * inv[1] * (z - w.zc) ** 2)
    x0, z0 = w.x0, w.z0
    w.x0, w.z0 = -(w.nx >> 1) * w.dx, -(w.nz >> 1) * w.dz
    _transform(w, -1)
    qx, qz = w.axes()
    sg = [(v > 0) - (v < 0) for v in le]
    c = 0.25 * math.pi * (2. - sg[0] - sg[1])
    w.phase(-3.1415926536 * w.lam * le[0] * qx * qx + c, -3.1415926536 * w.lam * le[1] * qz * qz)
    w.mult(math.sqrt(abs(le[0] * le[1])) / L)
    _transform(w, 1)
    w.x0, w.z0 = k[0] * x0 - kc[0] * w.xc, k[1] * z0 - kc[1] * w.zc
    w.dx, w.dz = w.dx * k[0], w.dz * k[1]
    x, z = w.axes()
    w.phase(pl * invL[0] * (x - w.xc) ** 2, pl * invL[1] * (z - w.zc) ** 2)
    flip = [d for d, v in ((1, k[0]), (0, k[1])) if v < 0.]
    if flip:
        w.f = [torch.flip(a, flip) for a in w.f]
    if k[0] < 0.:
        w.x0, w.dx = w.x0 + (w.nx - 1) * w.dx, -w.dx
    if k[1] < 0.:
        w.z0, w.dz = w.z0 + (w.nz - 1) * w.dz, -w.dz
    _after_drift(w, L)


def _waist_drift(w, L):
    pl = w.E * 2.53384080189e+06
    il = w.E * 806546.577258
    x, z = w.axes()
    w.phase(pl / L * x * x + 2. * pl * w.xc / w.Rx * x, pl / L * z * z + 2. * pl * w.zc / w.Rz * z)
    _transform(w, -1)
    s = L / il
    w.x0, w.dx = (w.x0 - w.xc * il / w.Rx) * s, w.dx * s
    w.z0, w.dz = (w.z0 - w.zc * il / w.Rz) * s, w.dz * s
    x, z = w.axes()
    w.phase(pl / L * x * x, pl / L * z * z)
    w.mult(-1j * il / L)
    _after_drift(w, L)


def _axis(n, start, step, n_new, start_new, step_new, first, last):
    """Per new node of [first, last]: start of its 4-node stencil on the old axis, sub-cell for the
    two-node fallback, and its coordinate relative to the stencil's second node."""
    i = torch.arange(first, last + 1, device=DEV)
    a = start_new + i.double() * step_new
    ic = ((a - start) * (1. / step) + 1e-6).long()
    rel = a - (start + ic.double() * step)
    st = ic - 1
    for at, move in ((n - 1, 2), (n - 2, 1), (0, -1)):
        st = torch.where(ic == at, ic - 1 - move, st)
        rel = torch.where(ic == at, rel + move * step, rel)
    t = rel / step
    wt = torch.stack([-t * (t - 1.) * (t - 2.) / 6., (t + 1.) * (t - 1.) * (t - 2.) / 2., -(t + 1.) * t * (t - 2.) / 2.,
                      (t + 1.) * t * (t - 1.) / 6.])
    return st, (ic - st).clamp(0, 2), t, wt


def _resize(w, pxm, pxd, pzm, pzd):
    """Range and resolution factors per axis: the mesh about the same centre, then interpolation of
    the field with its quadratic phase removed (cubic; linear where a stencil holds an exact zero),
    its modulus corrected by the interpolated intensity; zero outside the old range."""
    new = []
    for n, start, step, m, d in ((w.nx, w.x0, w.dx, pxm, pxd), (w.nz, w.z0, w.dz, pzm, pzd)):
        nn = _good(int(m * d * n) + (m * d * n - int(m * d * n) >= 0.5)) if m * d != 1. else n
        mag = (n - 1) * step
        if m > 1.:
            inner = int(nn / m) if d != 1. else n
            left = (nn - inner + 1) >> 1
            st = mag / (inner - 1)
            new.append([nn, start - left * st, st, left, left + inner - 1])
        else:
            st = step if d == 1. else mag * m / (nn - 1)
            new.append([nn, 0.5 * (start + (start + mag)) - 0.5 * (nn - 1) * st, st, 0, nn - 1])
    k = 3.14159265358979e+06 / 1.23984186 * w.E
    cx = k / w.Rx if abs(w.eRx) < 0.4 * abs(w.Rx) else 0.
    cz = k / w.Rz if abs(w.eRz) < 0.4 * abs(w.Rz) else 0.
    x, z = w.axes()
    w.phase(-cx * (x - w.xc) ** 2, -cz * (z - w.zc) ** 2)
    (nx, x0, dx, xa, xb), (nz, z0, dz, za, zb) = new
    stx, irx, tx, wx = _axis(w.nx, w.x0, w.dx, nx, x0, dx, xa, xb)
    stz, irz, tz, wz = _axis(w.nz, w.z0, w.dz, nz, z0, dz, za, zb)
    out = []
    for a in w.f:
        g = torch.zeros((nz, nx), dtype=torch.complex128, device=DEV)
        rows = max(1, (1 << 21) // max(1, stx.numel()))
        for r in range(0, stz.numel(), rows):
            sz = stz[r:r + rows]
            F = I = low = 0.
            for j in range(4):
                for i in range(4):
                    v = a[(sz + j)[:, None], (stx + i)[None, :]]
                    wgt = wz[j, r:r + rows][:, None] * wx[i][None, :]
                    F = F + wgt * v
                    I = I + wgt * (v.real ** 2 + v.imag ** 2)
                    z0v = (v.real == 0.) | (v.imag == 0.)
                    low = z0v if i + j == 0 else (low | z0v)
            q = [a[(sz + irz[r:r + rows] + j)[:, None], (stx + irx + i)[None, :]] for j in (0, 1) for i in (0, 1)]
            X, Z = tx[None, :], tz[r:r + rows][:, None]
            bil = lambda c: c[0] + (c[1] - c[0]) * X + (c[2] - c[0]) * Z + (c[0] - c[2] - c[1] + c[3]) * X * Z  # noqa: E731
            F = torch.where(low, bil(q), F)
            I = torch.where(low, bil([c.real ** 2 + c.imag ** 2 for c in q]), I).clamp(min=0.)
            A = F.real ** 2 + F.imag ** 2
            g[za + r:za + r + sz.numel(), xa:xb + 1] = F * torch.where(A != 0., torch.sqrt(I / torch.where(A != 0., A, 1.)), 1.)
        out.append(g)
    w.f = out
    # the mesh as the wavefront's description holds it: first and last point
    w.nx, w.nz = nx, nz
    w.x0, w.dx = x0, ((x0 + dx * (nx - 1)) - x0) / (nx - 1)
    w.z0, w.dz = z0, ((z0 + dz * (nz - 1)) - z0) / (nz - 1)
    x, z = w.axes()
    w.phase(cx * (x - w.xc) ** 2, cz * (z - w.zc) ** 2)


def _propagate(case, w):
    if case['chain'] == 'drifts':
        _drift(w, 10.)
        _aperture(w, 'r', 1e-3)
        _lens(w, 5.)
        _drift(w, 5.)
    elif case['chain'] == 'quad':
        _quad_drift(w, 30.)
        _lens(w, 15.)
        _quad_drift(w, 30.)
    else:
        _aperture(w, 'c', 0.8e-3)
        _resize(w, case['pxm'], case['pxd'], case['pzm'], case['pzd'])
        _lens(w, 10.)
        _waist_drift(w, 10.)
    return w


def _electron(case, ex, ey, off):
    """The field of one macro-electron: kicked on the base mesh, the mesh moved, the energy shifted."""
    E, r, R = _mesh(case)
    x, xp, y, yp, de = off
    w = _Wave(ex, ey, E * (1. + 2. * de), -r, r, -r, r, R)
    ax, az = w.axes()
    w.phase(5.06773065e+06 * w.E * xp * ax, 5.06773065e+06 * w.E * yp * az)
    w.x0, w.z0, w.xc, w.zc = w.x0 + x + xp * R, w.z0 + y + yp * R, x, y
    return w


def _sample(w, m):
    """|Ex|^2 + |Ey|^2 interpolated linearly on the detector's mesh; nothing outside w's."""
    I = sum(a.real ** 2 + a.imag ** 2 for a in w.f)
    at = []
    for s, f, n, s0, d, k in ((m['xStart'], m['xFin'], m['nx'], w.x0, w.dx, w.nx), (m['yStart'], m['yFin'], m['ny'], w.z0, w.dz, w.nz)):
        p = (s + torch.arange(n, dtype=torch.float64, device=DEV) * ((f - s) / (n - 1)) - s0) / d
        i = torch.trunc(p + 1e-9).long()
        ok = (i >= 0) & (i < k - 1)
        i = i.clamp(0, k - 2)
        at.append((i, p - i.double(), ok))
    (ix, tx, okx), (iz, tz, okz) = at
    g = lambda j, i: I[(iz + j)[:, None], (ix + i)[None, :]]  # noqa: E731
    X, Z = tx[None, :], tz[:, None]
    v = g(0, 0) * (1. - X) * (1. - Z) + g(0, 1) * X * (1. - Z) + g(1, 0) * (1. - X) * Z + g(1, 1) * X * Z
    return torch.where(okz[:, None] & okx[None, :], v, torch.zeros_like(v))


def _train_exact(case, seed):
    X, T, W, b, m, v = _train_data(case, seed)
    X, T = X.double(), T.double()
    W, b = [w.double().requires_grad_() for w in W], [v.double().requires_grad_() for v in b]
    a = X
    for k, (w, c) in enumerate(zip(W, b)):
        a = a @ w + c
        if k + 1 < len(W):
            a = torch.nn.functional.gelu(a, approximate='tanh')
    loss = ((a - T) ** 2).mean()
    g = torch.autograd.grad(loss, W + b)
    n, t = len(W), STEPS + 1
    new = []
    for p, d, mp, vp in zip(W + b, g, m, v):                # Adam
        mp, vp = 0.9 * mp.double() + 0.1 * d, 0.999 * vp.double() + 0.001 * d * d
        new.append((p - 1e-3 * (mp / (1. - 0.9 ** t)) / (torch.sqrt(vp / (1. - 0.999 ** t)) + 1e-8)).detach())
    return dict(out=a.detach(), loss=loss.detach().reshape(1), dW=list(g[:n]), db=list(g[n:]), W=new[:n], b=new[n:])


def exact(case, seed):
    if DEV == 'cpu' and case['kind'] != 'train' and case['nx'] * case['ny'] * case['pxm'] * case['pxd'] * case['pzm'] * \
            case['pzd'] * case.get('batch', 1) > 5e7:
        return None
    if case['kind'] == 'train':
        return _train_exact(case, seed)
    E, r, R = _mesh(case)
    ex, ey = _fields(case, seed, case['batch'] if case['kind'] == 'batch' else 1)
    if case['kind'] == 'electrons':
        mean = 0.
        for off in _offsets(case, seed):
            mean = mean + _sample(_propagate(case, _electron(case, ex[0], ey[0], off)), _acc_mesh(case))
        return mean / case['batch']
    ws = [_propagate(case, _Wave(a, c, E, -r, r, -r, r, R)).f for a, c in zip(ex, ey)]
    if case['kind'] == 'batch':
        return dict(ex=torch.stack([f[0] for f in ws]), ey=torch.stack([f[1] for f in ws]))
    ex, ey = ws[0]
    if case['kind'] == 'host':
        # the moments are rounded to single precision by definition: no 64-bit value
        return dict(ex=torch.view_as_real(ex).reshape(-1), ey=torch.view_as_real(ey).reshape(-1), momx=None, momy=None)
    return dict(ex=ex, ey=ey)
