"""The work that programs have this library do, as cases that can be timed and checked.

Each case is one pass through the library's public calls on the inputs, workspaces and plans
that a program holds: 1D and 3D sweeps of the Daubechies-16 operators (MagicFilter, kinetic,
wavelet analysis and synthesis), the local Hamiltonian, batches of uneven grids, the Poisson
finite differences, one layer of the preconditioner network, and a call on host arrays; in the
compute modes that the library offers.  `exact` gives the same results in plain torch FP64.
"""
import ctypes
import math
import os
import sys
from fractions import Fraction

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PERIODIC, GROW, SHRINK, FREE = 0, 1, -1, 2
MODES = {'fp64': 0, 'exact': 1, 'bf16x3': 2, 'tf32x3': 3}
H = 0.45                                  # grid spacing of the kinetic operator (bohr)
A_KIN = -0.5 / H ** 2


def _pkg():
    """The package, imported by the repository's own entry module."""
    if os.getcwd() not in sys.path:
        sys.path.insert(0, os.getcwd())
    import __graft_entry__
    return __graft_entry__.package()


# ---- the cases --------------------------------------------------------------------------------
def listed():
    return [
        # one 1D sweep over a 32^3 grid, in the library's default mode: the unit call of the
        # generated procedures' own tests, where launch and call overhead count
        {'name': 'sweep_32_default', 'op': 'sweep', 'filter': 'md', 'axis': 0, 'bc': PERIODIC,
         'mode': 'fp64', 'n0': 32, 'n1': 32, 'n2': 32, 'narr': 1},
        # MagicFilter of a single small orbital grid, called once per orbital
        {'name': 'mf_32', 'op': 'mf', 'bc': PERIODIC, 'mode': 'exact',
         'n0': 32, 'n1': 32, 'n2': 32, 'narr': 1},
        # the benchmark's step: MagicFilter and kinetic operator over 32 orbitals of 128^3
        {'name': 'mfkin_128x32', 'op': 'mfkin', 'bc': PERIODIC, 'mode': 'exact',
         'n0': 128, 'n1': 128, 'n2': 128, 'narr': 32},
        # kinetic operator with its energies on one isolated system's grid of odd extents
        {'name': 'kin_energy_odd', 'op': 'kin_ekin', 'bc': FREE, 'mode': 'exact',
         'n0': 61, 'n1': 83, 'n2': 97, 'narr': 1},
        # wavelet synthesis of 48^3 coefficients to 96^3 and analysis back, 16 orbitals
        {'name': 'wavelet_96x16', 'op': 'wavelet', 'bc': PERIODIC, 'mode': 'exact',
         'n0': 48, 'n1': 48, 'n2': 48, 'narr': 16},
        # local Hamiltonian of an isolated system's 8 orbitals, density accumulated
        {'name': 'hamiltonian_48x8', 'op': 'hamiltonian', 'bc': FREE, 'mode': 'exact',
         'n0': 48, 'n1': 48, 'n2': 48, 'narr': 8},
        # MagicFilter and kinetic operator over orbitals with localisation regions of their own
        {'name': 'uneven_128', 'op': 'batch', 'mode': 'exact', 'ngrids': 128, 'lo': 24, 'hi': 72},
        # divergence and correction term of the generalised Poisson solver
        {'name': 'poisson_256', 'op': 'poisson', 'mode': 'exact', 'geocode': 3, 'nord': 16,
         'n0': 256, 'n1': 256, 'n2': 256},
        # kinetic operator in the default mode
        {'name': 'kin_64x8_default', 'op': 'kin', 'bc': PERIODIC, 'mode': 'fp64',
         'n0': 64, 'n1': 64, 'n2': 64, 'narr': 8},
        # MagicFilter with growth of 64^3 orbitals to 79^3 at split precision
        {'name': 'mf_grow_64x16_split', 'op': 'mf', 'bc': GROW, 'mode': 'bf16x3',
         'n0': 64, 'n1': 64, 'n2': 64, 'narr': 16},
        # the generated procedures' own form of call: arrays in host memory
        {'name': 'host_mf_96x16', 'op': 'host_mf', 'bc': PERIODIC, 'mode': 'exact',
         'n0': 96, 'n1': 96, 'n2': 96, 'narr': 16},
        # a hidden layer of the kinetic solves' preconditioner network
        {'name': 'network_layer_48x64', 'op': 'layer', 'mode': 'exact', 'n0': 48, 'narr': 64},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi, most, even=False):
        """Extents (a third of them powers or multiples of 16) and a number of arrays whose
        points together stay under `most`."""
        n = [log(lo, hi) for _ in range(3)]
        if rng.random() < 0.33:
            n = [max(16, 16 * round(v / 16)) for v in n]
        if rng.random() < 0.4:
            n = [n[0]] * 3
        top = max(1, min(64, int(most // (n[0] * n[1] * n[2]))))
        return {'n0': n[0], 'n1': n[1], 'n2': n[2], 'narr': log(1, top) if top > 1 else 1}

    op = rng.choice(['sweep', 'mf', 'mf', 'kin', 'mfkin', 'kin_ekin', 'wavelet', 'wavelet',
                     'hamiltonian', 'batch', 'poisson', 'host_mf', 'layer'])
    mode = rng.choice(['exact', 'exact', 'exact', 'fp64', 'bf16x3', 'tf32x3'])
    most = 8e6 if mode == 'fp64' else 4e7
    c = {'op': op, 'mode': mode}
    if op == 'sweep':
        c.update(grid(17, 160, most), filter=rng.choice(['md', 'imd', 'd1', 'd2']),
                 axis=rng.choice([0, 1, 2]), bc=rng.choice([PERIODIC, FREE, GROW]))
    elif op in ('mf', 'host_mf'):
        c.update(grid(17, 160, most / 2), bc=rng.choice([PERIODIC, GROW]))
    elif op in ('kin', 'kin_ekin'):
        c.update(grid(17, 160, most / 2), bc=rng.choice([PERIODIC, FREE]))
        if op == 'kin_ekin':
            c['narr'] = 1
    elif op == 'mfkin':
        c.update(grid(17, 160, most / 2), bc=PERIODIC)
    elif op == 'wavelet':
        c.update(grid(9, 72, most / 16), bc=rng.choice([PERIODIC, GROW]))
    elif op == 'hamiltonian':
        c.update(grid(9, 56, most / 64), bc=rng.choice([PERIODIC, FREE]))
    elif op == 'batch':
        lo = log(17, 40)
        c.update(ngrids=log(2, 128), lo=lo, hi=lo + log(4, 40))
        c['mode'] = 'exact'
    elif op == 'poisson':
        c.update(grid(24, 256, 1.7e7), geocode=rng.choice([1, 2, 3]), nord=rng.choice([4, 6, 16]))
        del c['narr']
    else:
        n = 8 * rng.choice([2, 3, 4, 5, 6, 8])
        c.update(n0=n, narr=log(1, min(128, max(2, int(1.4e7 / n ** 3)))), mode='exact')
    return c


# ---- inputs -----------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed) + 1)


def _smooth(seed, narr, n):
    """Unit-RMS Gaussian-filtered noise on periodic grids [narr, n2, n1, n0]."""
    x = torch.randn(narr, *n[::-1], dtype=torch.float64, device='cuda', generator=_gen(seed))
    w = torch.exp(-0.5 * (torch.arange(-4, 5, dtype=torch.float64) / 1.5) ** 2)
    w = (w / w.sum()).tolist()
    for d in (1, 2, 3):
        if x.shape[d] > 1:
            x = sum(v * torch.roll(x, i - 4, d) for i, v in enumerate(w))
    return (x / x.square().mean().sqrt()).contiguous()


def _orbital(seed, narr, n):
    """Centred Gaussian envelopes times noise: a localised orbital on its own box."""
    x = torch.randn(narr, *n[::-1], dtype=torch.float64, device='cuda', generator=_gen(seed))
    for d, m in ((3, n[0]), (2, n[1]), (1, n[2])):
        r = (torch.arange(m, dtype=torch.float64, device='cuda') - (m - 1) / 2) * H
        e = torch.exp(-r * r / 32.0)
        x *= e.view([m if k == d else 1 for k in range(4)])
    return x


def _coefficients(seed, narr, n):
    """Wavelet coefficients: smooth scaling subband, details 1e-3 of it."""
    x = _smooth(seed, narr, [2 * v for v in n])
    x[:, n[2]:] *= 1e-3
    x[:, :, n[1]:] *= 1e-3
    x[:, :, :, n[0]:] *= 1e-3
    return x


def _n(c):
    return [c['n0'], c['n1'], c['n2']]


def _dims(c):
    r = np.random.default_rng(c['ngrids'] * 1000 + c['lo'])
    return r.integers(c['lo'], c['hi'] + 1, (c['ngrids'], 3)).tolist()


def _inputs(c, seed):
    op = c['op']
    if op == 'batch':
        return [_orbital(seed * 1000 + g, 1, d) for g, d in enumerate(_dims(c))]
    if op == 'poisson':
        return _smooth(seed, 3, _n(c))
    if op in ('wavelet', 'hamiltonian'):
        return _coefficients(seed, c['narr'], _n(c))
    if op == 'layer':
        m = c['n0']
        g = _gen(seed)
        x = torch.randn(c['narr'], m, m, m, 16, device='cuda', generator=g).clamp_(min=0)
        w = torch.randn(27, 16, 16, device='cuda', generator=g) * (2.0 / 432) ** 0.5
        b = torch.randn(16, device='cuda', generator=g) * 0.05
        return x.to(torch.bfloat16), w.to(torch.bfloat16), b
    if c.get('bc') in (FREE, GROW):
        return _orbital(seed, c['narr'], _n(c))
    return _smooth(seed, c['narr'], _n(c))


def _potential(seed, nreal):
    return -1.0 + 0.1 * torch.randn(nreal, dtype=torch.float64, device='cuda', generator=_gen(seed + 77))


# ---- one pass ---------------------------------------------------------------------------------
def prepare(case, seed):
    P = _pkg()
    c, op = case, case['op']
    P.set_mode(MODES[c['mode']])
    s = {'pkg': P, 'mode': MODES[c['mode']], 'op': op, 'case': c}
    x = _inputs(c, seed)
    new = lambda k: torch.empty(int(k), dtype=torch.float64, device='cuda')  # noqa: E731
    if op in ('sweep', 'mf', 'kin', 'mfkin', 'kin_ekin', 'wavelet', 'host_mf'):
        n, narr, bc = _n(c), c['narr'], c['bc']
        grown = [v + 15 if bc == GROW else v for v in n]
        s.update(n=n, narr=narr, bc=[bc] * 3, x=x.reshape(-1))
        size = narr * math.prod(n)
    if op == 'sweep':
        up = 7 if c['filter'] in ('md', 'imd') else 14
        ny = [v + (2 * up + (up == 7) if bc == GROW and i == c['axis'] else 0) for i, v in enumerate(n)]
        s.update(k=P.Kernel({'md': 'd_s0s0_1d_sym8_md', 'imd': 'd_s0s0_1d_sym8_imd', 'd1': 'd_s0s0_1d_sym8_d1',
                             'd2': 'd_s0s0_1d_sym8_d2_dotin'}[c['filter']]), ny=ny, y=new(narr * math.prod(ny)))
        if c['filter'] == 'd2':
            s['dot'] = new(1)
    elif op == 'mf':
        m = narr * math.prod(grown)
        s.update(k=P.Kernel('d_sfrf_ld_narr'), ny=grown, y=new(m), w1=new(m), w2=new(m))
    elif op in ('kin', 'kin_ekin'):
        s.update(k=P.Kernel('d_kin_narr' if op == 'kin' else 'd_kin_ekin'), y=new(size), w1=new(size), w2=new(size))
        if op == 'kin_ekin':
            s['ekin'] = new(3)
    elif op == 'mfkin':
        s.update(k=P.Kernel('d_sfrf_ld_narr'), k2=P.Kernel('d_kin_narr'), y=new(size), y2=new(size),
                 w1=new(size), w2=new(size))
    elif op == 'wavelet':
        m = narr * math.prod(2 * (v + 7) if bc == GROW else 2 * v for v in n)
        s.update(k=P.Kernel('d_idwt_sym8_narr'), k2=P.Kernel('d_dwt_sym8_narr'), y=new(m), y2=new(8 * size),
                 w1=new(m), w2=new(m), back=[SHRINK if bc == GROW else bc] * 3)
    elif op == 'host_mf':
        m = narr * math.prod(grown)
        s.update(k=P.Kernel('d_sfrf_ld_narr'), ny=grown, x=x.reshape(-1).cpu().pin_memory().numpy(),
                 y=torch.empty(m, dtype=torch.float64).pin_memory().numpy(), w=np.zeros(1))
    elif op == 'hamiltonian':
        ham = P.Hamiltonian(_n(c), [c['bc']] * 3, [A_KIN] * 3, c['narr'])
        s.update(ham=ham, x=x.reshape(-1), pot=_potential(seed, ham.nreal), y=new(c['narr'] * ham.nsig),
                 rho=torch.zeros(ham.nreal, dtype=torch.float64, device='cuda'))
    elif op == 'batch':
        b = P.Batch(_dims(c), mf_bc=[GROW] * 3, kin_bc=[FREE] * 3, kin_a=[A_KIN] * 3)
        _, n_mf, n_kin = b.sizes()
        s.update(batch=b, x=torch.cat([v.reshape(-1) for v in x]), y=new(n_mf), y2=new(n_kin),
                 stream=torch.cuda.Stream())
    elif op == 'poisson':
        f = P.lib().div_u_i_dev
        dp = ctypes.POINTER(ctypes.c_double)
        f.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p] * 2 + [ctypes.c_int, dp] + [ctypes.c_void_p] * 3
        f.restype = ctypes.c_int
        N = math.prod(_n(c))
        s.update(f=f, n=_n(c), h=(ctypes.c_double * 3)(0.1, 0.1, 0.1), x=x.reshape(-1), y=new(N), cc=new(N),
                 work=new(5 * N))
    else:
        f = P.lib().libconv_cnn_conv
        v = ctypes.c_void_p
        f.argtypes = [ctypes.c_int] * 4 + [v] * 8 + [ctypes.c_int, v, v]
        f.restype = ctypes.c_int
        s.update(f=f, x=x[0], w=x[1], b=x[2], y=torch.empty_like(x[0]))
    torch.cuda.synchronize()
    return s


def run(s):
    P, op, c = s['pkg'], s['op'], s['case']
    P.set_mode(s['mode'])
    if op == 'sweep':
        if c['filter'] == 'd2':
            s['k'].run_dev(3, c['axis'], s['n'], c['bc'], s['n'], s['ny'], s['narr'], s['x'], s['y'],
                           A_KIN, 0.0, 0.0, s['dot'])
            return s['y'], s['dot']
        s['k'].run_dev(3, c['axis'], s['n'], c['bc'], s['n'], s['ny'], s['narr'], s['x'], s['y'], 1.0, 0.0, 0.0)
        return s['y'],
    if op == 'mf':
        s['k'].run_dev(3, s['n'], s['bc'], s['n'], s['ny'], s['narr'], s['x'], s['y'], s['w1'], s['w2'])
        return s['y'],
    if op == 'kin':
        s['k'].run_dev(3, s['n'], s['bc'], s['narr'], s['x'], s['y'], s['w1'], s['w2'], [A_KIN] * 3, 0.0, 0.0)
        return s['y'],
    if op == 'kin_ekin':
        s['k'].run_dev(3, s['n'], s['bc'], s['x'], s['y'], s['w1'], s['w2'], [A_KIN] * 3, 0.5, 0.0, s['ekin'])
        return s['y'], s['ekin']
    if op == 'mfkin':
        s['k'].run_dev(3, s['n'], s['bc'], s['n'], s['n'], s['narr'], s['x'], s['y'], s['w1'], s['w2'])
        s['k2'].run_dev(3, s['n'], s['bc'], s['narr'], s['x'], s['y2'], s['w1'], s['w2'], [A_KIN] * 3, 0.0, 0.0)
        return s['y'], s['y2']
    if op == 'wavelet':
        s['k'].run_dev(3, s['n'], s['bc'], s['narr'], s['x'], s['y'], s['w1'], s['w2'])
        s['k2'].run_dev(3, s['n'], s['back'], s['narr'], s['y'], s['y2'], s['w1'], s['w2'])
        return s['y'], s['y2']
    if op == 'host_mf':
        s['k'].run(3, s['n'], s['bc'], s['n'], s['ny'], s['narr'], s['x'], s['y'], s['w'], s['w'])
        return s['y'],
    if op == 'hamiltonian':
        s['rho'].zero_()
        e = s['ham'](s['x'], s['pot'], s['y'], rho=s['rho'])
        return s['y'], s['rho'], e
    if op == 'batch':
        s['batch'].run(s['x'], s['y'], s['y2'], stream=s['stream'])
        return s['y'], s['y2']
    if op == 'poisson':
        st = s['f'](c['geocode'], *s['n'], s['x'].data_ptr(), s['y'].data_ptr(), c['nord'], s['h'],
                    s['cc'].data_ptr(), s['work'].data_ptr(), None)
        if st:
            raise RuntimeError(P.last_error())
        return s['y'], s['cc']
    st = s['f'](c['n0'], c['narr'], 0, 0, s['x'].data_ptr(), None, None, s['w'].data_ptr(), s['b'].data_ptr(),
                s['y'].data_ptr(), None, None, 16, None, None)
    if st:
        raise RuntimeError(P.last_error())
    return s['y'],


def work(case):
    c, op = case, case['op']
    if op == 'batch':
        pts = [math.prod(d) for d in _dims(c)]
        out = [math.prod(v + 15 for v in d) for d in _dims(c)]
        return {'bytes': 8.0 * (2 * sum(pts) + sum(out)), 'flops': 96.0 * sum(out) + 174.0 * sum(pts)}
    if op == 'layer':
        pts = c['narr'] * c['n0'] ** 3
        return {'bytes': 64.0 * pts + 27 * 512, 'flops': 2.0 * 27 * 256 * pts}
    n = _n(c)
    N = math.prod(n)
    if op == 'poisson':
        return {'bytes': 8.0 * 5 * N, 'flops': 6 * 2.0 * (c['nord'] + 1) * N}
    N *= c['narr']
    bc = c['bc']
    if op == 'sweep':
        taps = 16 if c['filter'] in ('md', 'imd') else 29
        out = N // n[c['axis']] * (n[c['axis']] + taps - 1 if bc == GROW else n[c['axis']])
        return {'bytes': 8.0 * (N + out), 'flops': 2.0 * taps * out}
    if op in ('mf', 'host_mf'):
        out = c['narr'] * math.prod(v + 15 if bc == GROW else v for v in n)
        return {'bytes': 8.0 * (N + out), 'flops': 96.0 * out}
    if op in ('kin', 'kin_ekin'):
        return {'bytes': 16.0 * N, 'flops': 174.0 * N}
    if op == 'mfkin':
        return {'bytes': 24.0 * N, 'flops': 270.0 * N}
    if op == 'wavelet':
        out = c['narr'] * math.prod(2 * (v + 7) if bc == GROW else 2 * v for v in n)
        return {'bytes': 8.0 * (8 * N + 8 * N + 2 * out), 'flops': 2 * 96.0 * out}
    free = bc == FREE
    fscf = c['narr'] * math.prod(2 * v + (14 if free else 0) for v in n)
    real = math.prod(2 * v + (29 if free else 0) for v in n)
    return {'bytes': 8.0 * (16 * N + 3 * real), 'flops': 2 * 96.0 * fscf + 174.0 * fscf + 2 * 96.0 * real * c['narr']}


# ---- the same results in plain FP64 -------------------------------------------------------------
# SYM8 family: scaling filter, MagicFilter, first and second derivative (positive half: k = 0..14)
LP = [float(v) for v in """
-0.003382415951005002595457699235919135128 -0.000542132331800010689347836944017347858
0.03169508781152599143142570752391597485 0.00760748732497660819192100801219238392
-0.1432942383512726628440955443992739699 -0.0612733590678110778430467690736584126
0.481359651259053391589568580264984525 0.777185751699628028624333566639210809
0.3644418948361789367595594323842960136 -0.0519458381078818007357107290625634285
-0.02721902991710348632196412421624687935 0.0491371796737302867869109881551654429
0.003808752013894489463071922223049694342 -0.01495225833706219911849029822472598879
-0.0003029205147241330812639124399571849886 0.001889950332767689184274432603245581173
""".split()]
MF = [float(v) for v in """
2.727344929119796596577153130172279928e-6 -0.00005185986881173432922848639136911486
0.0004944322768868991919228225947675097 -0.003441281444934938572808815096868218611
0.013372634148547947527334234670132209 -0.02103025160930381434955489412839065067
-0.06048952891969835160028346363993374 0.99404156978340039931786167125707312696
0.06126258958312079821953805969111734845 0.02373821463724942397566389712597274534
-0.00942047030201080385922711540948195 0.001747237136729939034494478127498529416
-0.000301580381326904631671637038261698 0.000087629844762105595646891618941163970
-0.00001290557201342060969516786758559028 8.4334247333529341094733325815816e-7
""".split()]
D2_HALF = [float(v) for v in """
-3.553692289913190194129680937424076424953 2.219146593891116389879454640457705235616
-0.6156141465570069496314853948700762181 0.2371780582153805636239247475762231531
-0.0822663999742123340987663520631668159 0.02207029188482255523789911295638968408
-0.004097656893426338238993270511883154847 0.000451679202875022353494800376397584960
-0.00002398228524507599670405555359023134 2.09042349529203659579228894473609842e-6
-3.723076304736927584879149697304408803e-7 -1.058570554967414703734941322870242653e-8
-5.813879830282540547959250667464887365e-11 2.708004936263194382698566890376475760e-13
-6.924474940639200152025730585882115968e-18
""".split()]
D1_HALF = [float(v) for v in """
0 0.8834460460908270942785855643941098713157598590915 -0.3032593514765938346887962440931660566677778365
0.1063640682894442760934532284702982844094052663346 -0.03129014783948023634381563995259325360348542944
0.006958379116450707495020407536758241511060163284 -0.001031530213375445369097964780217146384828800932
0.00007667706908380351933901775234801819926013328 2.451992111053665419191564123434446284949933594e-7
3.993810456408053712133667496514167576517175934e-8 -7.207948238588481597101904067961163265788433149e-8
-9.697184925637300947553068758362746388131353737e-10 -7.252206916665149851135591529994603533072998149e-13
1.240078536096648534547438612731567439237828505e-14 -1.585464751677102510097179308121926878193105545e-19
""".split()]
D2 = D2_HALF[:0:-1] + D2_HALF
D1 = [-v for v in D1_HALF[:0:-1]] + D1_HALF
HP = [v if i % 2 == 0 else -v for i, v in enumerate(LP)][::-1]
FILTERS = {'md': (MF[::-1], -8), 'imd': (MF, -7), 'd1': (D1, -14), 'd2': (D2, -14)}


def _taps(x, axis, taps, low, bc):
    """sum_k taps[k] x[q + low + k] along grid axis `axis` (the tensor's last dimension is axis 0)."""
    d, n, t = x.dim() - 1 - axis, x.shape[x.dim() - 1 - axis], len(taps)
    if bc == PERIODIC:
        return sum(v * torch.roll(x, -(low + k), d) for k, v in enumerate(taps))
    if bc == SHRINK:
        return sum(v * x.narrow(d, k, n - t + 1) for k, v in enumerate(taps))
    pad = list(x.shape)
    pad[d] = n + 2 * (t - 1)
    p = torch.zeros(pad, dtype=x.dtype, device=x.device)
    p.narrow(d, t - 1, n).copy_(x)
    first, count = (0, n + t - 1) if bc == GROW else (t - 1 + low, n)
    return sum(v * p.narrow(d, first + k, count) for k, v in enumerate(taps))


def _three(x, f, bc):
    for a in range(3):
        x = _taps(x, a, *FILTERS[f], bc)
    return x


def _kinetic(x, bc):
    parts = [A_KIN * _taps(x, a, *FILTERS['d2'], bc) for a in range(3)]
    return parts[0] + parts[1] + parts[2], [(x * p).flatten(1).sum(1) for p in parts]


def _synthesis(x, bc):
    le, lo, he, ho = LP[::-1][0::2], LP[::-1][1::2], HP[::-1][0::2], HP[::-1][1::2]
    for a in range(3):
        d = x.dim() - 1 - a
        n = x.shape[d] // 2
        s, w = x.narrow(d, 0, n), x.narrow(d, n, n)
        e0 = _taps(s, a, lo, -3, bc) + _taps(w, a, ho, -3, bc)
        e1 = _taps(s, a, le, -3, bc) + _taps(w, a, he, -3, bc)
        x = torch.stack([e0, e1], d + 1).flatten(d, d + 1)
    return x


def _analysis(x, bc):
    le, lo, he, ho = LP[0::2], LP[1::2], HP[0::2], HP[1::2]
    for a in range(3):
        d = x.dim() - 1 - a
        p = x.unflatten(d, (-1, 2))
        x0, x1 = p.select(d + 1, 0), p.select(d + 1, 1)
        x = torch.cat([_taps(x0, a, le, -4, bc) + _taps(x1, a, lo, -4, bc),
                       _taps(x0, a, he, -4, bc) + _taps(x1, a, ho, -4, bc)], d)
    return x


def _weights(at, nodes):
    """First-derivative weights at node `at` on nodes 0..nodes-1 (derivatives of the Lagrange basis)."""
    out = []
    for j in range(nodes):
        den = Fraction(1)
        for i in range(nodes):
            if i != j:
                den *= j - i
        num = Fraction(0)
        for m in range(nodes):
            if m != j:
                p = Fraction(1)
                for i in range(nodes):
                    if i not in (j, m):
                        p *= at - i
                num += p
        out.append(float(num / den))
    return out


def _derivative(u, axis, nord, periodic, inv_h):
    d, n, m = u.dim() - 1 - axis, u.shape[u.dim() - 1 - axis], nord // 2
    out = torch.empty_like(u)
    mid = _weights(m, nord + 1)
    if periodic:
        return inv_h * sum(v * torch.roll(u, m - k, d) for k, v in enumerate(mid))
    out.narrow(d, m, n - 2 * m).copy_(sum(v * u.narrow(d, k, n - 2 * m) for k, v in enumerate(mid)))
    for e in range(m):
        for at, base, to in ((e, 0, e), (m + 1 + e, n - 1 - nord, n - m + e)):
            w = _weights(at, nord + 1)
            out.select(d, to).copy_(sum(v * u.select(d, base + k) for k, v in enumerate(w)))
    return inv_h * out


def exact(case, seed):
    c, op = case, case['op']
    x = _inputs(c, seed)
    flat = lambda t: t.reshape(-1)  # noqa: E731
    if op == 'sweep':
        y = _taps(x, c['axis'], *FILTERS[c['filter']], c['bc'])
        if c['filter'] == 'd2':
            y = A_KIN * y
            at = y.narrow(3 - c['axis'], 14, _n(c)[c['axis']]) if c['bc'] == GROW else y
            return flat(y), (x * at).sum().reshape(1)
        return flat(y),
    if op in ('mf', 'host_mf'):
        y = flat(_three(x, 'md', c['bc']))
        return (y.cpu().numpy() if op == 'host_mf' else y),
    if op == 'kin':
        return flat(_kinetic(x, c['bc'])[0]),
    if op == 'kin_ekin':
        y, e = _kinetic(x, c['bc'])
        return flat(y + 0.5 * x), torch.cat(e)
    if op == 'mfkin':
        return flat(_three(x, 'md', c['bc'])), flat(_kinetic(x, c['bc'])[0])
    if op == 'wavelet':
        y = _synthesis(x, c['bc'])
        return flat(y), flat(_analysis(y, SHRINK if c['bc'] == GROW else c['bc']))
    if op == 'hamiltonian':
        free = c['bc'] == FREE
        out, back = (GROW, SHRINK) if free else (PERIODIC, PERIODIC)
        fscf = _synthesis(x, out)
        psir = _three(fscf, 'md', out)
        pot = _potential(seed, psir[0].numel()).view(psir.shape[1:])
        hpsi = _three(pot * psir, 'imd', back)
        t, e = _kinetic(fscf, c['bc'])
        en = torch.stack(e + [(pot * psir * psir).flatten(1).sum(1)], 1)
        return flat(_analysis(hpsi + t, back)), flat(psir.square().sum(0)), en
    if op == 'batch':
        return (torch.cat([flat(_three(v, 'md', GROW)) for v in x]),
                torch.cat([flat(_kinetic(v, FREE)[0]) for v in x]))
    if op == 'poisson':
        per = [c['geocode'] != 1, c['geocode'] == 2, c['geocode'] != 1]
        d = lambda k, a: _derivative(x[k], a, c['nord'], per[a], 10.0)  # noqa: E731
        d0, d1, d2 = d(0, 0), d(1, 1), d(2, 2)
        cc = x[0] ** 2 * d0 + x[1] ** 2 * d1 + x[2] ** 2 * d2 + 2 * (
            x[0] * x[1] * d(1, 0) + x[0] * x[2] * d(2, 0) + x[1] * x[2] * d(2, 1))
        return flat(d0 + d1 + d2), flat(cc)
    a, w, b = x[0].double(), x[1].double(), x[2].double()
    y = b.expand(*a.shape[:4], 16).clone()
    for t in range(27):
        shift = (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3)
        y += torch.roll(a, shift, (1, 2, 3)) @ w[t].T
    return y.clamp(min=0),
