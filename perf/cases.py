"""Workloads of the library as a user's program runs them, with their inputs, their compulsory work and their values in 64 bits.

Every case is a dict of plain values with a "kind":

  step       one integrator step of a resident state and the density on the grid (the loop body of pendulum.m / pendulum_reduced.m)
  sequence   device arrays in the MATLAB layout through forward transform, Euler step and backward transform (the MEX calls)
  gyro       one Euler step of the gyro-bias model on a device array (gyro_bias.m)
  hybrid     one hybrid step with the collision operator, and the density after it (pendulum_reduced_hybrid.m)
  adjoint    gradients of a terminal loss through Euler steps
  round      density -> coefficients -> density, the precision stress of the transforms
  batch      uneven densities advanced together, and their densities
  product    the Clebsch-Gordan product of batched coefficients (fftSO3_prod.m)
  real       real-harmonic transforms there and back of batched functions (fftSO3.m / ifftSO3.m)

B is the bandlimit (2B points per Euler angle), N the points per omega axis.
"""
import importlib
import math

import numpy as np
import torch

hp = importlib.import_module('hybridpendulum-up_b200')

DT = 1e-3
DT_EULER = 1e-4                          # a resident state takes thousands of passes: forward Euler grows on the imaginary axis
L3, L2 = 8.0, 3.4                        # omega periods of the 3-D and the reduced pendulum
J, B3, G3 = (0.02, 0.02, 0.01), 0.05, 0.02     # inertia, damping, noise H H^T / 2 with H = 0.2 I
GYRO = ((J[1] - J[2]) / J[0], (J[2] - J[0]) / J[1], (J[0] - J[1]) / J[2])
MGR = 1.0 * 9.8 * 0.1                    # m g rho, rho along the third body axis
GRAV3 = np.array([[0, MGR / J[0], 0], [-MGR / J[1], 0, 0], [0, 0, 0]])      # J^-1 (-m g rho x R^T e3)
B2, G2 = 0.2, 0.5                        # reduced pendulum: damping, noise
GRAV2 = np.array([[0, 1.0, 0], [-1.0, 0, 0]])                               # [R32; -R31]
GB_G1, GB_G2 = 0.01 * np.eye(3) + 0.002, 0.005 * np.eye(3) + 0.001          # gyro-bias random walks
LAMBDA_MAX, RESTITUTION, TAPS = 100.0, 0.8, 10                              # collision operator


def listed():
    return [
        # the headline: Euler step and density of the 3-D pendulum in mixed precision, B = 15 on 32^3
        dict(name='step_mixed_B15_w32', kind='step', B=15, N=32, ndim=3, mixed=True, method='euler'),
        # the same loop in FP64, where a study asks for it, on the grid of the differentiation workload
        dict(name='step_fp64_B12_w24', kind='step', B=12, N=24, ndim=3, mixed=False, method='euler'),
        # sizes whose FFT lengths have a large prime factor, with the stable integrator
        dict(name='rk4_mixed_B11_w22', kind='step', B=11, N=22, ndim=3, mixed=True, method='rk4'),
        # the reduced pendulum, small: a few short launches per step, latency counts
        dict(name='rk4_mixed_2d_B8_w16', kind='step', B=8, N=16, ndim=2, mixed=True, method='rk4'),
        # plain FP64 single step through the MEX-shaped calls, B = 10 on 16^3
        dict(name='sequence_fp64_B10_w16', kind='sequence', B=10, N=16, ndim=3),
        # gyro_bias.m at its driver's sizes (BR = 10, Bx = 15)
        dict(name='gyro_fp64_B10_w30', kind='gyro', B=10, N=30),
        # the hybrid pendulum with density gravity and wall collisions, omega grid above 32 points
        dict(name='hybrid_mixed_B16_w40', kind='hybrid', B=16, N=40, mixed=True),
        # gradients of a terminal loss (the 50-step workload, cut to four steps with two checkpoints)
        dict(name='adjoint_fp64_B12_w24', kind='adjoint', B=12, N=24, steps=4, every=2),
        # transform round trip at the largest bandlimit, complex coefficients
        dict(name='round_mixed_B32_w24', kind='round', B=32, N=24, ndim=2, mixed=True),
        # an estimator bank: densities of uneven bandlimit and omega grid in one batch
        dict(name='batch_mixed_6', kind='batch', members='8x16,12x16,16x16,8x24,12x24,8x32', method='rk2'),
        # measurement updates multiply coefficient arrays: batched products
        dict(name='product_B12_16', kind='product', B=12, batch=16),
        # SO(3)-only models work in real harmonics on batches of functions
        dict(name='real_B16_64', kind='real', B=16, batch=64),
    ]


def _coefficients(B, real=True):
    """Stored coefficients of one omega point: (l, m, n) with m >= 0 for real densities."""
    return B * (B + 1) * (4 * B - 1) // 6 if real else B * (2 * B - 1) * (2 * B + 1) // 3


def _cost(case):
    """A rough size, to keep drawn cases within the largest listed one."""
    k = case['kind']
    if k == 'product':
        return case['batch'] * case['B'] ** 7 * 2.0
    if k == 'real':
        return case['batch'] * (2 * case['B']) ** 4 * 4.0
    if k == 'batch':
        return sum(2 * (2 * B) ** 3 * N ** 3 for B, N in _members(case))
    points = case['N'] ** case.get('ndim', 2 if k == 'hybrid' else 3)
    per = (2 * case['B']) ** 3
    if k == 'step':
        stages = {'euler': 1, 'midpoint': 2, 'rk2': 2, 'rk4': 4}[case['method']]
        return points * per * (1 if case['mixed'] else 3) * (0.5 + 0.5 * stages)
    factor = {'sequence': 8, 'gyro': 4, 'hybrid': 16 if case.get('mixed') else 40, 'adjoint': 20 * case.get('steps', 1),
              'round': 6 if case.get('mixed') else 20}[k]
    return points * per * factor


def draw(rng):
    def even(lo, hi):                    # even sizes, spread over their logarithm
        return 2 * int(round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2)))))

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    cap = _cost(listed()[0])
    while True:
        kind = rng.choice(['step', 'step', 'step', 'sequence', 'gyro', 'hybrid', 'adjoint', 'round', 'batch', 'product', 'real'])
        if kind == 'step':
            ndim = rng.choice([2, 3])
            case = dict(kind=kind, B=size(4, 24), N=even(8, 32 if ndim == 3 else 64), ndim=ndim, mixed=rng.random() < 0.6,
                        method=rng.choice(['euler', 'midpoint', 'rk2', 'rk4']))
        elif kind == 'sequence':
            case = dict(kind=kind, B=size(4, 16), N=even(8, 24), ndim=3)
        elif kind == 'gyro':
            case = dict(kind=kind, B=size(4, 12), N=even(8, 32))
        elif kind == 'hybrid':
            case = dict(kind=kind, B=size(6, 20), N=even(16, 48), mixed=rng.random() < 0.6)
        elif kind == 'adjoint':
            case = dict(kind=kind, B=size(4, 12), N=even(8, 24), steps=rng.randint(1, 4), every=rng.randint(1, 3))
        elif kind == 'round':
            case = dict(kind=kind, B=size(8, 32), N=even(8, 32), ndim=2, mixed=rng.random() < 0.6)
        elif kind == 'batch':
            members = ['%dx%d' % (size(6, 16), even(8, 24)) for _ in range(rng.randint(2, 8))]
            case = dict(kind=kind, members=','.join(members), method=rng.choice(['rk2', 'rk4']))
        elif kind == 'product':
            case = dict(kind=kind, B=size(4, 14), batch=size(1, 64))
        else:
            case = dict(kind=kind, B=size(4, 20), batch=size(1, 128))
        if _cost(case) <= cap:
            return case


def _dt(method):
    return DT_EULER if method == 'euler' else DT


def _members(case):
    return [tuple(int(v) for v in m.split('x')) for m in case['members'].split(',')]


def work(case):
    """Compulsory bytes and operations of one pass: inputs read once (of a full coefficient array the entries that carry
    information), outputs written once; the operations of the beta contractions, FFTs and pointwise products that the path is made of."""
    k = case['kind']
    if k == 'batch':
        parts = [work(dict(kind='step', B=B, N=N, ndim=3, mixed=True, method=case['method'])) for B, N in _members(case)]
        return {key: float(sum(p[key] for p in parts)) for key in ('bytes', 'flops')}
    B = case['B']
    if k == 'product':
        n = (2 * B - 1) ** 2 * B * case['batch']
        grid = (3 * B) ** 3                # the product of the two functions on a grid that resolves it
        return {'bytes': 48.0 * n, 'flops': 3.0 * case['batch'] * grid * (4 * B + 30 * math.log2(3 * B))}
    if k == 'real':
        n = (2 * B) ** 3 * case['batch']
        c = (2 * B - 1) ** 2 * B * case['batch']
        return {'bytes': 16.0 * (n + c), 'flops': 2.0 * n * (2 * B + 10 * math.log2(2 * B))}
    N, ndim = case['N'], case.get('ndim', 2 if k == 'hybrid' else 3)
    real = k != 'round'
    mixed = case.get('mixed', False)
    points, coeffs, grid = N ** ndim, _coefficients(B, real), (2 * B) ** 3 * (1 if real else 2)
    state, full = 16.0 * coeffs * points, 16.0 * (2 * B - 1) ** 2 * B * points
    density = (4.0 if mixed else 8.0) * grid * points
    transform = points * (4.0 * coeffs * 2 * B + 5 * grid * math.log2(2 * B) + 5 * coeffs * ndim * math.log2(N))
    deriv = coeffs * points * (10.0 * (2 * ndim + 1) * math.log2(N) + 120)
    stages = {'euler': 1, 'midpoint': 2, 'rk2': 2, 'rk4': 4}.get(case.get('method', 'euler'))
    if k == 'step':
        return {'bytes': 2 * state + density, 'flops': stages * deriv + transform}
    if k == 'sequence':
        return {'bytes': 2 * density + 2 * full + 2 * state, 'flops': deriv + 2 * transform}
    if k == 'gyro':
        return {'bytes': state + full, 'flops': deriv}
    if k == 'hybrid':
        tables = (4.0 if mixed else 8.0) * (TAPS + 1) + 2 * TAPS
        return {'bytes': 2 * state + 2 * density + tables * _colliding(B) * points, 'flops': deriv + 4 * transform}
    if k == 'adjoint':
        return {'bytes': state + 16.0 * _coefficients(B, False) * points + full, 'flops': case['steps'] * 4.0 * deriv}
    return {'bytes': 2 * density, 'flops': 2 * transform}


# ------------------------------------------------------------------------------------------------- inputs ----
def _rng(seed):
    return np.random.default_rng(seed)


def _device():
    return torch.device('cuda' if torch.cuda.is_available() else 'cpu')


def _third_row(B, dev):
    """R^T e3 on the Euler grid, broadcastable over [c, b, a]."""
    k = torch.arange(2 * B, dtype=torch.float64, device=dev)
    beta, gamma = (math.pi / (4 * B) * (2 * k + 1))[None, :, None], (math.pi / B * k)[:, None, None]
    return torch.stack([(-torch.sin(beta) * torch.cos(gamma)).expand(2 * B, 2 * B, 1),
                        (torch.sin(beta) * torch.sin(gamma)).expand(2 * B, 2 * B, 1),
                        torch.cos(beta).expand(2 * B, 2 * B, 1)])


def _rotations(B, dev):
    """R = Rz(alpha) Ry(beta) Rz(gamma) as [c, b, a, 3, 3]."""
    k = torch.arange(2 * B, dtype=torch.float64, device=dev)
    a, b, c = math.pi / B * k, math.pi / (4 * B) * (2 * k + 1), math.pi / B * k
    z, o = torch.zeros_like(k), torch.ones_like(k)

    def rz(t):
        return torch.stack([torch.cos(t), -torch.sin(t), z, torch.sin(t), torch.cos(t), z, z, z, o], -1).view(-1, 3, 3)
    ry = torch.stack([torch.cos(b), z, torch.sin(b), z, o, z, -torch.sin(b), z, torch.cos(b)], -1).view(-1, 3, 3)
    return torch.einsum('aij,bjk,ckl->cbail', rz(a), ry, rz(c))


def _omega(N, L, dev):
    return -L / 2 + L / N * torch.arange(N, dtype=torch.float64, device=dev)


def _density(B, N, ndim, L, seed, dtype, dev, sigma=0.5):
    """A matrix Fisher distribution times a Gaussian, of unit peak mass scale: [omega..., c, b, a]."""
    r = _rng(seed)

    def haar():
        q, t = np.linalg.qr(r.standard_normal((3, 3)))
        q = q * np.sign(np.diag(t))
        q[:, 0] *= np.linalg.det(q)
        return q
    F = haar() @ np.diag(np.sort(r.uniform(5, 20, 3))[::-1]) @ haar().T
    mu = r.uniform(-0.125 * L, 0.125 * L, ndim)
    e = torch.einsum('ij,cbaij->cba', torch.as_tensor(F, device=dev), _rotations(B, dev))
    fR = torch.exp(e - e.max())
    fR = fR / fR.mean()
    x, fx = _omega(N, L, dev), None
    for i in reversed(range(ndim)):      # the last omega axis is the slowest in memory
        g = torch.exp(-0.5 * ((x - mu[i]) / sigma) ** 2) / math.sqrt(2 * math.pi) / sigma
        fx = g if fx is None else fx[..., None] * g
    out = torch.empty((N,) * ndim + (2 * B,) * 3, dtype=dtype, device=dev)
    for w in range(N):
        out[w] = fx[w][(...,) + (None,) * 3] * fR
    return out


def _gravity_MR(B, A, ndim):
    """fftSO3R of mR_i = sum_j A_ij (R^T e3)_j in the MATLAB layout: degree 1, m = 0 only."""
    t = _Transform(B, torch.device('cpu'))
    MR = np.zeros((2 * B - 1, 2 * B - 1, B, ndim), np.complex128)
    rows = _third_row(B, torch.device('cpu')).expand(3, 2 * B, 2 * B, 2 * B)
    c = t.forward(torch.einsum('ij,jcba->icba', torch.as_tensor(A), rows))          # [i, l, n, m]
    lo = B - 2
    MR[B - 1, lo:lo + 3, 1, :] = c[:, 1, lo:lo + 3, B - 1].numpy().T
    return MR


def _plan(B, N, ndim, mixed, symmetry=None):
    return hp.Plan(B, N // 2, ndim, hp.HP_MIXED if mixed else hp.HP_FP64, hp.HP_REAL if symmetry is None else symmetry)


def _set_pendulum(plan):
    if plan.ndim == 3:
        plan.set_model(L3, [B3] * 3, G3 * np.eye(3), _gravity_MR(plan.B, GRAV3, 3), GYRO)
    else:
        plan.set_model(L2, [B2] * 2, G2 * np.eye(2), _gravity_MR(plan.B, GRAV2, 2))


def _dtype(mixed):
    return torch.float32 if mixed else torch.float64


def _period(ndim):
    return L3 if ndim == 3 else L2


def _colliding(B):
    """Attitudes at which the tip touches the wall: about a fifth of the grid."""
    return int((_tilt(B, torch.device('cpu')) > 0.6).sum())


def _tilt(B, dev):
    """First component of R e3 on [c, b, a]: how far the pendulum leans toward the wall."""
    k = torch.arange(2 * B, dtype=torch.float64, device=dev)
    return (torch.cos(math.pi / B * k)[None, None, :] * torch.sin(math.pi / (4 * B) * (2 * k + 1))[None, :, None]).expand((2 * B,) * 3)


def _collision_tables(B, N, dev):
    """A wall: the switching rate ramps with the lean where the tip moves toward the wall, the landing velocity is the
    mirrored one with restitution, its Gaussian kernel is kept at the nearest grid points."""
    tilt = _tilt(B, dev).reshape(-1)
    ind = torch.nonzero(tilt > 0.6).reshape(-1)
    gamma = (math.pi / B * torch.arange(2 * B, dtype=torch.float64, device=dev))[:, None, None].expand((2 * B,) * 3).reshape(-1)[ind]
    n = torch.stack([torch.sin(gamma), torch.cos(gamma)], -1)               # wall normal seen from the body
    x = _omega(N, L2, dev)
    om = torch.stack([x.repeat(N), x.repeat_interleave(N)], -1)             # [ix, 2], first component fastest
    s = om @ n.T                                                           # [ix, k]
    lam = LAMBDA_MAX * ((tilt[ind] - 0.6) / 0.1).clamp(0, 1) * (s > 0)
    land = om[:, None] - (1 + RESTITUTION) * s.clamp(min=0)[..., None] * n
    first = ((land + L2 / 2) * N / L2).round().long() - 2                   # 4 x 4 window around the landing point
    first = first.clamp(0, N - 4)
    q = torch.arange(4, device=dev)
    cell = torch.stack([q.repeat(4), q.repeat_interleave(4)], -1)
    p = first[:, :, None] + cell                                           # [ix, k, 16, 2]
    d2 = ((x[p] - land[:, :, None]) ** 2).sum(-1)
    d2, at = d2.topk(TAPS, dim=-1, largest=False)
    w = torch.exp(-(d2 - d2[..., :1]) / (2 * 0.05 ** 2))
    w = lam[..., None] * w / w.sum(-1, keepdim=True)
    p = (p[..., 0] + N * p[..., 1]).gather(-1, at)
    return lam, ind.to(torch.int32), w, p.to(torch.int16)


def _random_full(shape, seed, dev):
    g = torch.Generator(device=dev).manual_seed(int(seed))
    return torch.randn(shape, dtype=torch.complex128, device=dev, generator=g)


def _lmn(B, dev):
    l = torch.arange(B, device=dev).view(-1, 1, 1)
    k = torch.arange(2 * B - 1, device=dev) - (B - 1)
    return l, k.view(1, 1, -1), k.view(1, -1, 1)


def _mask(B, dev):
    l, m, n = _lmn(B, dev)
    return ((m.abs() <= l) & (n.abs() <= l)).to(torch.float64)


def _spectrum(B, batch, seed, dev):
    """Random band-limited coefficients, N(0, 1) / (2l + 1): [batch, l, n, m]."""
    l, _, _ = _lmn(B, dev)
    return _random_full((batch, B, 2 * B - 1, 2 * B - 1), seed, dev) * (_mask(B, dev) / (2 * l + 1))


def _round_density(case, seed, dev):
    B, N = case['B'], case['N']
    t = _Transform(B, dev)
    f = t.backward(_spectrum(B, N ** case['ndim'], seed, dev))
    return f.to(torch.complex64 if case['mixed'] else torch.complex128)


def _real_functions(case, seed, dev):
    g = torch.Generator(device=dev).manual_seed(int(seed))
    F = torch.randn((case['batch'], case['B'], 2 * case['B'] - 1, 2 * case['B'] - 1), dtype=torch.float64, device=dev, generator=g)
    l, _, _ = _lmn(case['B'], dev)
    return _Real(case['B'], dev).backward(F * _mask(case['B'], dev) / (2 * l + 1)) + 0.01 * torch.randn(
        (case['batch'],) + (2 * case['B'],) * 3, dtype=torch.float64, device=dev, generator=g)


def _adjoint_inputs(case, seed, dev):
    B, N = case['B'], case['N']
    f0 = _density(B, N, 3, L3, seed, torch.float64, dev)
    lam = _random_full((N, N, N, B, 2 * B - 1, 2 * B - 1), seed + 1, dev) * _mask(B, dev)
    return f0, lam


def prepare(case, seed):
    k, dev = case['kind'], _device()
    s = {'kind': k}
    if k in ('step', 'hybrid'):
        ndim = case.get('ndim', 2)
        plan = _plan(case['B'], case['N'], ndim, case['mixed'])
        if k == 'step':
            _set_pendulum(plan)
            s['method'] = case['method']
        else:
            rows = _third_row(case['B'], torch.device('cpu')).expand((3,) + (2 * case['B'],) * 3)
            mR = torch.einsum('ij,jcba->iabc', torch.as_tensor(GRAV2), rows).contiguous().numpy()
            plan.set_den_model(L2, [B2] * 2, G2 * np.eye(2), mR)
            lam, ind, w, at = (t.cpu().numpy() for t in _collision_tables(case['B'], case['N'], dev))
            s['coll'] = hp.Collision.from_tables(plan, lam, ind, w, at)
        s['f'] = _density(case['B'], case['N'], ndim, _period(ndim), seed, _dtype(case['mixed']), dev)
        s['state'] = hp.State(plan)
        s['state'].load_density(s['f'].data_ptr())
    elif k == 'sequence':
        plan = s['plan'] = _plan(case['B'], case['N'], 3, False)
        _set_pendulum(plan)
        s['f'] = _density(case['B'], case['N'], 3, L3, seed, torch.float64, dev).reshape(-1)
        n = int(np.prod(plan.F_shape))
        s['F'], s['Fnew'] = (torch.empty(n, dtype=torch.complex128, device=dev) for _ in range(2))
        s['fnew'] = torch.empty_like(s['f'])
    elif k in ('gyro', 'adjoint'):
        plan = s['plan'] = _plan(case['B'], case['N'], 3, False)
        if k == 'gyro':
            plan.set_gyro_bias_model(2.0, GB_G1, GB_G2)
            f0 = _density(case['B'], case['N'], 3, 2.0, seed, torch.float64, dev, sigma=0.15)
        else:
            _set_pendulum(plan)
            f0, lam = _adjoint_inputs(case, seed, dev)
            s.update(lam=lam.reshape(-1), steps=case['steps'], every=case['every'])
        s['F'] = plan.forward(f0.reshape(-1))
        s['Fnew'] = torch.empty_like(s['F'])
    elif k == 'round':
        plan = _plan(case['B'], case['N'], case['ndim'], case['mixed'], hp.HP_COMPLEX)
        s['f'] = _round_density(case, seed, dev)
        s['out'] = torch.empty_like(s['f'])
        s['state'] = hp.State(plan)
    elif k == 'batch':
        s['states'], s['f'] = [], []
        for i, (B, N) in enumerate(_members(case)):
            plan = _plan(B, N, 3, True)
            _set_pendulum(plan)
            f = _density(B, N, 3, L3, seed + 1000 * i, torch.float32, dev)
            st = hp.State(plan)
            st.load_density(f.data_ptr())
            s['states'].append(st)
            s['f'].append(f)
        s.update(batch=hp.Batch(s['states']), method=case['method'])
    elif k == 'product':
        B, D = case['B'], 2 * case['B'] - 1
        s['plan'] = _plan(B, 4, 2, False)
        s['F'], s['G'] = (_spectrum(B, case['batch'], seed + i, dev).view(D, D, B, case['batch']) for i in range(2))
        s['out'] = torch.empty_like(s['F'])
    else:
        s['plan'] = _plan(case['B'], 4, 2, False)
        s['f'] = _real_functions(case, seed, dev).reshape(-1)
        s['F'] = torch.empty(case['batch'] * (2 * case['B'] - 1) ** 2 * case['B'], dtype=torch.float64, device=dev)
        s['out'] = torch.empty_like(s['f'])
    if dev.type == 'cuda':
        torch.cuda.empty_cache()
    return s


def run(s):
    k = s['kind']
    if k == 'step':
        s['state'].step(_dt(s['method']), s['method'], 1)
        s['state'].density_into(s['f'].data_ptr())
        return s['f']
    if k == 'sequence':
        s['plan'].forward(s['f'], out=s['F'])
        s['plan'].propagate(s['F'], DT, 'euler', out=s['Fnew'])
        s['plan'].backward(s['Fnew'], out=s['fnew'])
        return s['F'], s['Fnew'], s['fnew']
    if k == 'gyro':
        return s['plan'].gyrobias_propagate(s['F'], DT, out=s['Fnew'])
    if k == 'hybrid':
        s['state'].hybrid_step(s['coll'], DT, 'euler', 1)
        s['state'].density_into(s['f'].data_ptr())
        return s['f']
    if k == 'adjoint':
        return s['plan'].adjoint(s['F'], s['lam'], s['steps'], DT, s['every'])
    if k == 'round':
        s['state'].load_density(s['f'].data_ptr())
        s['state'].density_into(s['out'].data_ptr())
        return s['out']
    if k == 'batch':
        s['batch'].step(DT, s['method'], 2)
        for st, f in zip(s['states'], s['f']):
            st.density_into(f.data_ptr())
        return s['f']
    if k == 'product':
        return s['plan'].prod(s['F'], s['G'], out=s['out'])
    s['plan'].real_forward(s['f'], out=s['F'])
    s['plan'].real_backward(s['F'], out=s['out'])
    return s['F'], s['out']


# --------------------------------------------------------------------------------------- values in 64 bits ----
class _Transform:
    """SO(3) transforms of [..., c, b, a] samples and [..., l, n, m] coefficients, plain and in FP64."""

    def __init__(self, B, dev):
        self.B, self.dev = B, dev
        k = torch.arange(2 * B, dtype=torch.float64)
        beta = math.pi / (4 * B) * (2 * k + 1)
        q = 2 * torch.arange(B, dtype=torch.float64) + 1
        self.w = (torch.sin(beta) / (4 * B ** 3) * (torch.sin(beta[:, None] * q) / q).sum(1)).to(dev)
        d = torch.zeros((2 * B, B, 2 * B - 1, 2 * B - 1), dtype=torch.float64)       # [b, l, n, m]
        for l in range(B):
            # d^l(beta) = exp(-i beta J_y), J_y from its ladder
            m = torch.arange(-l, l, dtype=torch.float64)
            up = torch.sqrt(l * (l + 1) - m * (m + 1)) / 2
            Jy = torch.diag(-1j * up, -1) + torch.diag(1j * up, 1)
            e, U = torch.linalg.eigh(Jy)
            rot = torch.einsum('mk,bk,nk->bnm', U, torch.exp(-1j * beta[:, None] * e.round()), U.conj()).real
            d[:, l, B - 1 - l:B + l, B - 1 - l:B + l] = rot
        self.d = d.to(dev)
        self.bins = ((torch.arange(2 * B - 1) - (B - 1)) % (2 * B)).to(dev)

    def _chunks(self, n, per):
        step = max(1, int(2e9 / (per * 16)))
        return [(i, min(n, i + step)) for i in range(0, n, step)]

    def forward(self, f, mult=None):
        """[..., c, b, a] -> [..., l, n, m]."""
        B, lead = self.B, f.shape[:-3]
        f = f.reshape((-1,) + f.shape[-3:])
        D = 2 * B - 1
        out = torch.empty((f.shape[0], B, D, D), dtype=torch.complex128, device=f.device)
        dw = self.d * self.w[:, None, None, None]
        for i, j in self._chunks(f.shape[0], (2 * B) ** 3):
            g = f[i:j].to(torch.complex128 if f.is_complex() else torch.float64)
            g = (g if mult is None else g * mult).to(torch.complex128)
            y = torch.fft.ifft(torch.fft.ifft(g, dim=-1, norm='forward')[..., self.bins], dim=1, norm='forward')[:, self.bins]
            out[i:j] = torch.einsum('blnm,wnbm->wlnm', dw.to(torch.complex128), y)
        return out.reshape(lead + out.shape[1:])

    def backward(self, F):
        """[..., l, n, m] -> complex [..., c, b, a]."""
        B, lead = self.B, F.shape[:-3]
        F = F.reshape((-1,) + F.shape[-3:])
        out = torch.empty((F.shape[0],) + (2 * B,) * 3, dtype=torch.complex128, device=F.device)
        dl = (self.d * (2 * torch.arange(B, device=self.dev) + 1).view(1, -1, 1, 1)).to(torch.complex128)
        for i, j in self._chunks(F.shape[0], (2 * B) ** 3):
            y = torch.zeros((j - i,) + (2 * B,) * 3, dtype=torch.complex128, device=F.device)
            g = torch.einsum('blnm,wlnm->wnbm', dl, F[i:j])
            z = torch.zeros(g.shape[:-1] + (2 * B,), dtype=g.dtype, device=g.device)
            z[..., self.bins] = g
            y[:, self.bins] = torch.fft.fft(z, dim=-1)
            out[i:j] = torch.fft.fft(y, dim=1)
        return out.reshape(lead + out.shape[1:])


class _Real(_Transform):
    """Transforms in the real harmonics of fftSO3.m, by their cosine and sine sums."""

    def __init__(self, B, dev):
        super().__init__(B, dev)
        D, lm = 2 * B - 1, B - 1
        k = torch.arange(D, device=dev) - lm
        am, m = k.abs(), k
        sign = 1 - 2 * ((m[None, :] - m[:, None]).abs() % 2).to(torch.float64)               # (-1)^(m-n), [n, m]
        d1 = self.d[:, :, lm + am][..., lm + am]                                             # d_{|m| |n|}
        d2 = self.d[:, :, lm - am][..., lm + am]                                             # d_{|m|, -|n|}
        both = sign * d1 + (1 - 2 * (am % 2)).to(torch.float64) * torch.sign(m).to(torch.float64) * d2
        zero_m, zero_n = (m == 0)[None, :].expand(D, D), (m == 0)[:, None].expand(D, D)
        psi = torch.where(zero_m | zero_n, math.sqrt(2) * sign * d1, both)
        self.psi = torch.where(zero_m & zero_n, d1, psi)
        self.same = (m >= 0)[None, :] == (m >= 0)[:, None]
        t = math.pi / B * torch.arange(2 * B, dtype=torch.float64, device=dev)[:, None] * k
        self.cos, self.sin = torch.cos(t), torch.sin(t)                                      # [point, order]

    def forward(self, f):
        out = []
        for g in f.split(8):
            S = torch.einsum('wcba,am,cn->wbnm', g.to(torch.complex128), torch.complex(self.cos, -self.sin), torch.complex(self.cos, -self.sin))
            x = torch.where(self.same, S.real, -S.imag)
            y = torch.where(self.same, S.real.flip(2), -S.imag.flip(2))
            p = torch.where(self.same, 0.5 * (y + x), 0.5 * (x - y))
            q = torch.where(self.same, 0.5 * (x - y), -0.5 * (x + y))
            out.append(torch.einsum('b,wbnm,blnm->wlnm', self.w, p, self.psi) + torch.einsum('b,wbnm,blnm->wlnm', self.w, q, self.psi.flip(3)))
        return torch.cat(out)

    def backward(self, F):
        out, l1 = [], (2 * torch.arange(self.B, device=self.dev) + 1).view(-1, 1, 1)
        for g in F.split(8):
            S = torch.einsum('wlnm,blnm->wbnm', l1 * g, self.psi)
            T = torch.einsum('wlnm,blnm->wbnm', l1 * g, self.psi.flip(3))
            s, o = self.same.to(torch.float64), (~self.same).to(torch.float64)
            f = torch.einsum('wbnm,cn,am->wcba', S * s, self.cos, self.cos) + torch.einsum('wbnm,cn,am->wcba', S * o, self.sin, self.cos)
            f -= torch.einsum('wbnm,cn,am->wcba', T * s, self.sin, self.sin) + torch.einsum('wbnm,cn,am->wcba', T * o, self.cos, self.sin)
            out.append(f)
        return torch.cat(out)


class _Model:
    """The Fokker-Planck derivative on [k_nd, ..., k_1, l, n, m] coefficients."""

    def __init__(self, B, N, ndim, L, dev, b, G, gyro=(0.0, 0.0, 0.0), A=None, G1=None, density_gravity=False):
        self.t = _Transform(B, dev)
        self.B, self.N, self.ndim, self.dev = B, N, ndim, dev
        self.x = _omega(N, L, dev)
        k = torch.arange(N, device=dev)
        kd = torch.where(k < N // 2, k, k - N).to(torch.float64) * (2 * math.pi / L)
        k1 = torch.where(k == N // 2, torch.zeros_like(kd), kd)
        self.kd, self.k1 = kd, k1
        self.b, self.G, self.gyro = b, G, gyro
        self.scale = torch.ones(3, dtype=torch.float64, device=dev)                 # factors of the gravity components
        self.A, self.G1, self.density_gravity = A, G1, density_gravity
        # u^l_i: F^l[E_i f] = F^l[f] (u^l_i)^T, as [l, row, column]
        D, lm = 2 * B - 1, B - 1
        u = torch.zeros((3, B, D, D), dtype=torch.complex128)
        for l in range(B):
            for n in range(-l, l + 1):
                if n > -l:
                    v = math.sqrt((l + n) * (l - n + 1))
                    u[0, l, n + lm - 1, n + lm], u[1, l, n + lm - 1, n + lm] = -0.5j * v, 0.5 * v
                if n < l:
                    v = math.sqrt((l - n) * (l + n + 1))
                    u[0, l, n + lm + 1, n + lm], u[1, l, n + lm + 1, n + lm] = -0.5j * v, -0.5 * v
                u[2, l, n + lm, n + lm] = -1j * n
        self.u = u.to(dev)
        if A is not None and not density_gravity:
            rows = _third_row(B, dev).expand((3,) + (2 * B,) * 3)
            mr = self.t.forward(torch.einsum('ij,jcba->icba', torch.as_tensor(A, device=dev), rows))
            self.mr = mr[:, 1, lm - 1:lm + 2, lm]                                    # [i, n2 + 1]
            self.taps = self._taps()

    def _taps(self):
        """Degree-1 product weights (2 l1 + 1) 3 / (2l + 1) <l1 m; 1 0|l m> <l1 n-n2; 1 n2|l n>, as {(l1 - l, n2): [l, n, m]}."""
        l, m, n = (v.to(torch.float64) for v in _lmn(self.B, self.dev))
        taps = {}
        for dl in (-1, 0, 1):
            l1 = l + dl

            def cg(mu, m2):
                r = lambda p: torch.sqrt(p.clamp(min=0))                            # noqa: E731
                j = l1.clamp(min=0)
                if dl == -1:                                                         # l = l1 + 1
                    return {1: r((j + mu) * (j + mu + 1) / ((2 * j + 1) * (2 * j + 2))),
                            0: r((j - mu + 1) * (j + mu + 1) / ((2 * j + 1) * (j + 1))),
                            -1: r((j - mu) * (j - mu + 1) / ((2 * j + 1) * (2 * j + 2)))}[m2]
                p = (2 * j * (j + 1)).clamp(min=1)
                if dl == 0:
                    return {1: -r((j + mu) * (j - mu + 1) / p), 0: mu / torch.sqrt(p / 2), -1: r((j - mu) * (j + mu + 1) / p)}[m2]
                p = (2 * j * (2 * j + 1)).clamp(min=1)                               # l = l1 - 1
                return {1: r((j - mu) * (j - mu + 1) / p), 0: -r((j - mu) * (j + mu) * 2 / p), -1: r((j + mu + 1) * (j + mu) / p)}[m2]
            for n2 in (-1, 0, 1):
                ok = (l1 >= 0) & (l1 < self.B) & (m.abs() <= l1) & ((n - n2).abs() <= l1) & (m.abs() <= l) & (n.abs() <= l)
                taps[dl, n2] = torch.where(ok, (2 * l1 + 1) * 3 / (2 * l + 1) * cg(m, 0) * cg(n, n2), torch.zeros_like(l))
        return taps

    def _along(self, v, i):
        """v over omega axis i (0-based), broadcast against coefficients."""
        shape = [1] * (self.ndim + 3)
        shape[self.ndim - 1 - i] = self.N
        return v.view(shape)

    def times_x(self, F, i):
        dim = self.ndim - 1 - i
        return torch.fft.fft(self._along(self.x, i) * torch.fft.ifft(F, dim=dim), dim=dim)

    def D(self, F, i):
        return 1j * self._along(self.k1, i) * F

    def right(self, F, i):
        return torch.matmul(self.u[i], F)

    def __call__(self, F, f=None):
        nd = self.ndim
        M = [self.times_x(F, i) for i in range(nd)]
        out = 0
        for i in range(nd):
            out = out - self.right(M[i], i)
            if self.b is not None:
                out = out + self.b[i] * self.D(M[i], i)
        if nd == 3 and self.gyro is not None:
            for i, j, k in ((0, 1, 2), (1, 0, 2), (2, 0, 1)):
                out = out - self.gyro[i] * self.D(self.times_x(M[k], j), i)
        if self.density_gravity:
            rows = _third_row(self.B, self.dev)
            mr = torch.einsum('ij,jcba->icba', torch.as_tensor(self.A, device=self.dev), rows)
            for i in range(nd):
                g = torch.fft.fftn(self.t.forward(f, mr[i]), dim=tuple(range(nd)))
                out = out - self.D(g, i)
        elif self.A is not None:
            for q, n2 in enumerate((-1, 0, 1)):
                s = 0
                for dl in (-1, 0, 1):
                    g = torch.roll(F, (-dl, n2), dims=(nd, nd + 1))                  # F^{l + dl}_{m, n - n2}
                    s = s + self.taps[dl, n2] * g
                for i in range(nd):
                    out = out - self.scale[i] * self.mr[i, q] * self.D(s, i)
        if self.G1 is not None:
            for i in range(3):
                g = self.right(F, i)
                for j in range(3):
                    out = out + float(self.G1[i, j]) * self.right(g, j)
        c = 0
        for i in range(nd):
            for j in range(nd):
                c = c - self.G[i, j] * (self._along(self.kd, i) ** 2 if i == j else self._along(self.k1, i) * self._along(self.k1, j))
        return out + c * F

    def step(self, F, dt, method, f=None):
        k1 = self(F, f)
        if method == 'euler':
            return F + dt * k1
        if method == 'rk2':
            return F + dt / 2 * (k1 + self(F + dt * k1))
        k2 = self(F + dt / 2 * k1)
        if method == 'midpoint':
            return F + dt * k2
        k3 = self(F + dt / 2 * k2)
        return F + dt / 6 * (k1 + 2 * k2 + 2 * k3 + self(F + dt * k3))

    def forward(self, f):
        return torch.fft.fftn(self.t.forward(f), dim=tuple(range(self.ndim)))

    def backward(self, F):
        """The real density, a slice of the slowest omega axis at a time."""
        Fx = torch.fft.ifftn(F, dim=tuple(range(self.ndim)))
        return torch.stack([self.t.backward(Fx[w]).real for w in range(self.N)])


def _pendulum(B, N, ndim, dev, density_gravity=False):
    def v(a):
        return torch.as_tensor(a, dtype=torch.float64, device=dev)
    if ndim == 3:
        return _Model(B, N, 3, L3, dev, v([B3] * 3), v(G3 * np.eye(3)), v(GYRO), A=GRAV3)
    return _Model(B, N, 2, L2, dev, v([B2] * 2), v(G2 * np.eye(2)), None, A=GRAV2, density_gravity=density_gravity)


def exact(case, seed):
    k, dev = case['kind'], _device()
    if k == 'step':
        f = _density(case['B'], case['N'], case['ndim'], _period(case['ndim']), seed, _dtype(case['mixed']), dev)
        p = _pendulum(case['B'], case['N'], case['ndim'], dev)
        return p.backward(p.step(p.forward(f), _dt(case['method']), case['method']))
    if k == 'sequence':
        f = _density(case['B'], case['N'], 3, L3, seed, torch.float64, dev)
        p = _pendulum(case['B'], case['N'], 3, dev)
        F = p.forward(f)
        Fnew = p.step(F, DT, 'euler')
        return F, Fnew, p.backward(Fnew)
    if k == 'gyro':
        f = _density(case['B'], case['N'], 3, 2.0, seed, torch.float64, dev, sigma=0.15)
        p = _Model(case['B'], case['N'], 3, 2.0, dev, None, torch.as_tensor(GB_G2, device=dev), None, G1=GB_G1)
        return p.step(p.forward(f), DT, 'euler')
    if k == 'hybrid':
        B, N = case['B'], case['N']
        f = _density(B, N, 2, L2, seed, _dtype(case['mixed']), dev)
        p = _pendulum(B, N, 2, dev, density_gravity=True)
        F = p.forward(f)
        f = p.backward(p.step(F, DT, 'euler', p.backward(F))).reshape(N * N, -1)
        lam, ind, w, at = _collision_tables(B, N, dev)
        g = f[:, ind.long()]
        df = -lam * g
        for d in range(TAPS):
            df += w[..., d] * g.gather(0, at[..., d].long())
        f[:, ind.long()] += DT * df
        return f.reshape((N, N) + (2 * B,) * 3)
    if k == 'adjoint':
        return _exact_adjoint(case, seed, dev)
    if k == 'round':
        t = _Transform(case['B'], dev)
        return t.backward(t.forward(_round_density(case, seed, dev)))
    if k == 'batch':
        out = []
        for i, (B, N) in enumerate(_members(case)):
            f = _density(B, N, 3, L3, seed + 1000 * i, torch.float32, dev)
            p = _pendulum(B, N, 3, dev)
            F = p.forward(f)
            for _ in range(2):
                F = p.step(F, DT, case['method'])
            out.append(p.backward(F))
        return out
    if k == 'product':
        # the product of two functions of bandlimit B, resolved on the grid of twice the bandlimit
        B, D = case['B'], 2 * case['B'] - 1
        t, z = _Transform(2 * B, dev), []
        for i in range(2):
            F = torch.zeros((case['batch'], 2 * B, 4 * B - 1, 4 * B - 1), dtype=torch.complex128, device=dev)
            F[:, :B, B:B + D, B:B + D] = _spectrum(B, case['batch'], seed + i, dev)
            z.append(t.backward(F))
        return (t.forward(z[0] * z[1])[:, :B, B:B + D, B:B + D] * _mask(B, dev)).reshape(D, D, B, case['batch'])
    t = _Real(case['B'], dev)
    F = t.forward(_real_functions(case, seed, dev)) * _mask(case['B'], dev)
    return F.reshape(-1), t.backward(F).reshape(-1)


def _exact_adjoint(case, seed, dev):
    """Reverse mode through the plain steps, one step's graph at a time."""
    f, lam = _adjoint_inputs(case, seed, dev)
    p = _pendulum(case['B'], case['N'], 3, dev)
    states = [p.forward(f)]
    for _ in range(case['steps'] - 1):
        states.append(p.step(states[-1], DT, 'euler'))
    # the loss gradient on the subspace of real densities: F^l_mn[k] -> (-1)^(m-n) conj F^l_{-m,-n}[-k]
    _, m, n = _lmn(case['B'], dev)
    flip = torch.roll(lam.flip(0, 1, 2), (1, 1, 1), dims=(0, 1, 2)).flip(4, 5).conj()
    lam = 0.5 * (lam + (1 - 2 * ((m - n).abs() % 2)).to(torch.float64) * flip)
    params = [p.b, p.G, p.gyro, p.scale]
    total = [torch.zeros_like(v) for v in params]
    for F in reversed(states):
        F = F.detach().requires_grad_(True)
        p.b, p.G, p.gyro, p.scale = leaves = [v.detach().clone().requires_grad_(True) for v in params]
        grads = torch.autograd.grad(p.step(F, DT, 'euler'), [F] + leaves, lam)
        lam = grads[0]
        total = [a + g for a, g in zip(total, grads[1:])]
    grads = dict(zip(('b', 'G', 'gyro', 'gscale'), (v.cpu().numpy() for v in total)))
    return lam.reshape(-1), grads
