"""The work a user of this package has it do, as cases that a timing harness can run: image formation by factorized
backprojection (ImageFormer) in both precisions, exact backprojection on a grid and at points, and the pair products
of formed images. Sizes are those of the package's own workloads (fastsar_b200/sim.py) and of its tests, and generic
ones between them.

    listed()             the cases; draw(rng): one more of the same ranges
    prepare(case, seed)  the inputs and the plan a program keeps; run(state): one pass through the public call
    work, tolerance, exact: the least bytes and operations of a pass, how far two correct results may differ, and the
    result in 64 bits

Histories are seeded: log-normal point targets of random phase on the grid and a -40 dB noise floor, the CPHD phase
convention exp(-j 4 pi f dR / c). They are synthesized here with torch (float64 phases)."""
import math

import numpy as np
import torch

C = 299792458.0
FC = 9.6e9                      # every collection is X band, as the package's workloads are
E1, E2 = (0.0, 1.0, 0.0), (1.0, 0.0, 0.0)


def listed():
    return [
        # the smallest call: a 128-pixel chip from 256 pulses, where launches and latency count
        _form('form_f32_chip_128', 256, 256, 300e6, 600e3, 45.0, 1.5, 128, 128, 0.25),
        # the package's small spotlight (spotlight_512), default options
        _form('form_f32_spotlight_512', 512, 1024, 300e6, 600e3, 45.0, 1.5, 512, 512, 0.25),
        # the ordinary call: 4,096 pulses x 4,096 samples to 2,048 x 2,048 (spotlight_4k), default options
        _form('form_f32_spotlight_2k', 4096, 4096, 300e6, 600e3, 45.0, 1.5, 2048, 2048, 0.25),
        # an odd-sized patch of a short-range collection, which needs 16-pixel final tiles
        _form('form_f32_near_odd', 2777, 2301, 900e6, 20e3, 40.0, 2.0, 1499, 701, 0.45, T=16),
        # the largest: the full spotlight_12k image in the plain float32 form
        _form('form_f32_spotlight_12k', 16384, 8192, 1.2e9, 500e3, 55.0, 3.0, 12288, 8832, 0.2),
        # the mixed-precision form with learned decimation taps at the same sizes
        _form('form_f16_spotlight_512', 512, 1024, 300e6, 600e3, 45.0, 1.5, 512, 512, 0.25, precision='float16',
              taps='learned', pmax=0.5),
        _form('form_f16_spotlight_2k', 4096, 4096, 300e6, 600e3, 45.0, 1.5, 2048, 2048, 0.25, precision='float16',
              taps='learned', pmax=0.5),
        _form('form_f16_near_odd', 2777, 2301, 900e6, 20e3, 40.0, 2.0, 1499, 701, 0.45, T=16, precision='float16',
              taps='learned', pmax=0.5),
        # the package's headline: the chosen form of spotlight_12k
        _form('form_f16_spotlight_12k', 16384, 8192, 1.2e9, 500e3, 55.0, 3.0, 12288, 8832, 0.2, precision='float16',
              taps='learned', pmax=0.52),
        # the exact former (cubic reads of 8x oversampled profiles) on a 1,024-pixel grid
        dict(name='exact_grid_1k', kind='exact', P=2048, K=2048, bw=300e6, r0=600e3, graze=45.0, ap=1.5, nx=1024,
             ny=1024, sp=0.25, interp='cubic'),
        # float64 backprojection at scattered points: how an image is checked
        dict(name='points_20k', kind='points', P=2048, K=2048, bw=300e6, r0=600e3, graze=45.0, ap=1.5, N=20000, nx=512,
             ny=512, sp=0.25, upsample=8),
        # the pair products of two formed images on a ragged grid: coherence map and multilooked interferogram
        dict(name='pair_4k', kind='pair', n1=4097, n2=3911, w1=7, w2=7, la=4, lr=4),
    ]


def _form(name, P, K, bw, r0, graze, ap, nx, ny, sp, precision='float32', taps='kaiser', pmax=0.4, T=0, window=True):
    """A formation case. T 0: the former chooses the final tile."""
    return dict(name=name, kind='form', P=P, K=K, bw=bw, r0=r0, graze=graze, ap=ap, nx=nx, ny=ny, sp=sp,
                precision=precision, taps=taps, pmax=pmax, T=T, window=window)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _geometry(rng, lo, hi):
    """A collection and a grid it leaves unambiguous: sides log-uniform in lo .. hi, as many pulses and samples as
    the grid's extent needs with a margin, or up to twice as many."""
    graze = rng.uniform(35.0, 55.0)
    ap = rng.uniform(1.3, 4.0)
    r0 = rng.choice([20e3, 100e3, 500e3, 600e3])
    res_a = C / FC / (2.0 * math.radians(ap))
    res_r = res_a * rng.uniform(0.8, 1.0)       # a bandwidth that matches the aperture: nearly square resolution
    bw = C / (2.0 * res_r * math.cos(math.radians(graze)))
    sp = math.ceil(res_a / 0.05) * 0.05
    nx = _log_int(rng, lo, hi)
    ny = _log_int(rng, max(lo, nx / 2), min(hi, nx * 2))
    if r0 < 50e3:                               # a short range holds no image of more than a few hundred metres
        nx, ny = min(nx, int(900.0 / sp)), min(ny, int(900.0 / sp))
    K = max(192, int(rng.uniform(1.3, 2.5) * ny * sp / res_r))
    P = max(192, int(rng.uniform(1.3, 2.5) * nx * sp / res_a))
    return dict(P=min(P, 12000), K=min(K, 12000), bw=bw, r0=r0, graze=graze, ap=ap, nx=nx, ny=ny, sp=sp)


def draw(rng):
    u = rng.random()
    if u < 0.75:
        g = _geometry(rng, 100, 3000)
        f16 = rng.random() < 0.5
        T = 16 if g['r0'] < 50e3 or rng.random() < 0.2 else 0
        form = dict(precision='float16', taps=rng.choice(['learned', 'kaiser']),
                    pmax=rng.choice([0.4, 0.5])) if f16 else dict(precision='float32', taps='kaiser', pmax=0.4)
        return dict(kind='form', T=T, window=rng.random() < 0.8, **form, **g)
    if u < 0.85:
        return dict(kind='exact', interp=rng.choice(['cubic', 'linear']), **_geometry(rng, 200, 1100))
    if u < 0.92:
        return dict(kind='points', N=_log_int(rng, 300, 60000), upsample=rng.choice([4, 8]), **_geometry(rng, 200, 800))
    return dict(kind='pair', n1=_log_int(rng, 300, 8000), n2=_log_int(rng, 300, 8000), w1=rng.randint(3, 11),
                w2=rng.randint(3, 11), la=rng.randint(1, 6), lr=rng.randint(1, 6))


# ------------------------------------------------------------------------------------------------ inputs
def _track(case):
    """(antenna positions [P, 3], fmin, df): a straight broadside track, as fastsar_b200.sim.spotlight lays it."""
    g = math.radians(case['graze'])
    ground = case['r0'] * math.cos(g)
    half = ground * math.tan(0.5 * math.radians(case['ap']))
    P, K = case['P'], case['K']
    ant = np.empty((P, 3))
    ant[:, 0], ant[:, 1], ant[:, 2] = -ground, np.linspace(-half, half, P), case['r0'] * math.sin(g)
    df = case['bw'] / K
    return ant, FC - (K // 2) * df, df


def _scene(case, seed):
    """64 point targets on the middle 80 % of the grid, powers log-normal (6 dB), random phases."""
    rng = np.random.default_rng(seed)
    n = 64
    a = rng.uniform(-0.4, 0.4, (n, 2)) * (case['nx'] * case['sp'], case['ny'] * case['sp'])
    pos = a[:, :1] * np.array(E1) + a[:, 1:] * np.array(E2)
    amp = 10.0 ** (6.0 * rng.standard_normal(n) / 20.0) * np.exp(2j * np.pi * rng.uniform(0.0, 1.0, n))
    return pos, amp


def _history(case, seed):
    """The phase history [P, K] complex64 on the GPU: per pulse the targets' phases at every 64th sample times their
    phases at the 64 samples between (float64 phases, complex64 products), plus the noise."""
    dev = 'cuda'
    ant, fmin, df = _track(case)
    pos, amp = _scene(case, seed)
    P, K = case['P'], case['K']
    A = torch.from_numpy(ant).to(dev)
    X = torch.from_numpy(pos).to(dev)
    a = torch.from_numpy(amp).to(dev)
    dR = (X[None] - A[:, None]).norm(dim=2) - A.norm(dim=1)[:, None]                      # [P, N]

    def cis(cycles):
        return torch.polar(torch.ones_like(cycles), -2.0 * math.pi * (cycles - cycles.round())).to(torch.complex64)
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    S = torch.view_as_complex(torch.randn((P, K, 2), device=dev, generator=g) * (0.01 / math.sqrt(2.0)))
    nb = -(-K // 64)
    hi = torch.arange(nb, device=dev, dtype=torch.float64) * 64.0
    lo = torch.arange(64, device=dev, dtype=torch.float64)
    for p0 in range(0, P, 1024):
        d = dR[p0:p0 + 1024] * (2.0 / C)
        U = cis(d[:, None, :] * (fmin + df * hi)[None, :, None]) * a.to(torch.complex64)     # [p, nb, N]
        V = cis(d[:, :, None] * (df * lo)[None, None, :])                                   # [p, N, 64]
        S[p0:p0 + 1024] += torch.bmm(U, V).reshape(len(d), nb * 64)[:, :K]
    return S


def _points(case, seed):
    """Points scattered uniformly over the grid's extent."""
    rng = np.random.default_rng(seed + 1)
    a = rng.uniform(-0.5, 0.5, (case['N'], 2)) * (case['nx'] * case['sp'], case['ny'] * case['sp'])
    return a[:, :1] * np.array(E1) + a[:, 1:] * np.array(E2)


def _pair(case, seed):
    """Two complex speckle images of one scene: a common part, a little noise of each, and a smooth phase between."""
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed))
    n1, n2 = case['n1'], case['n2']
    z = torch.view_as_complex(torch.randn((3, n1, n2, 2), device='cuda', generator=g))
    t = torch.arange(n2, device='cuda', dtype=torch.float32) * (12.0 / n2)
    return z[0] + 0.3 * z[1], (z[0] + 0.3 * z[2]) * torch.polar(torch.ones_like(t), t)


# ------------------------------------------------------------------------------------------------ the passes
def prepare(case, seed):
    kind = case['kind']
    if kind == 'pair':
        a, b = _pair(case, seed)
        return dict(case=case, a=a, b=b)
    ant, fmin, df = _track(case)
    st = dict(case=case, S=_history(case, seed), ant=ant, fmin=fmin, df=df)
    if kind == 'points':
        return dict(st, points=_points(case, seed))
    grid = (case['nx'], case['ny'], case['sp'], case['sp'], E1, E2)
    if kind == 'exact':
        from fastsar_b200 import ExactFormer
        return dict(st, former=ExactFormer(ant, fmin, df, case['K'], *grid, interp=case['interp']))
    from fastsar_b200 import ImageFormer
    return dict(st, former=ImageFormer(ant, fmin, df, case['K'], *grid, precision=case['precision'], taps=case['taps'],
                                       pmax=case['pmax'], T=case['T'] or 'auto', window=case['window']))


def run(state):
    case = state['case']
    if case['kind'] == 'pair':
        from fastsar_b200 import products
        return dict(coherence=products.coherence(state['a'], state['b'], case['w1'], case['w2']),
                    interferogram=products.interferogram(state['a'], state['b'], case['la'], case['lr']))
    if case['kind'] == 'points':
        from fastsar_b200.exact import backproject_device
        return backproject_device(state['S'], state['ant'], state['fmin'], state['df'], state['points'],
                                  upsample=case['upsample'])
    return state['former'].form_device(state['S'])


def work(case):
    """Histories (or images) read once and results written once. Operations: formation, the final sums alone (each
    T x T tile over the T x T samples its band and aperture need, as one complex product of 8 operations); exact
    backprojection, per pixel and pulse the range (10), the read of the profile (cubic 16, linear 8) and the
    rotation and sum (10); the pair products, per pixel the three products and their running sums."""
    if case['kind'] == 'pair':
        n = case['n1'] * case['n2']
        return dict(bytes=n * 20 + (n // (case['la'] * case['lr'])) * 8 + n * 16, flops=n * 40)
    hist = case['P'] * case['K'] * 8
    if case['kind'] == 'points':
        return dict(bytes=hist + case['N'] * 40, flops=case['N'] * case['P'] * 28)
    px = case['nx'] * case['ny']
    if case['kind'] == 'exact':
        return dict(bytes=hist + px * 8, flops=px * case['P'] * (36 if case['interp'] == 'cubic' else 28))
    T = case['T'] or 32
    return dict(bytes=hist + px * 8, flops=8 * px * T * T)


def tolerance(case):
    """Two correct results of one plan differ by the arithmetic alone."""
    if case['kind'] == 'points':
        return dict(rel=5e-8)                # float64 sums of a history windowed in float32 (1.2e-8 from 64 bits)
    if case['kind'] == 'pair':
        return dict(rel=2e-6)                # float64 window sums, float32 results
    if case['kind'] == 'exact':
        return dict(rel=3e-4)                # float32 ranges about the tile centres (7e-5 from 64 bits)
    if case['precision'] == 'float16':
        return dict(rel=2e-3, max=0.2)       # 4.5e-4 from the same plan's float32 kernels, at a faint pixel 0.05
    return dict(rel=2e-5, max=2e-3)          # 3e-6 from the same plan in 64 bits or in split-bfloat16 final sums


# ------------------------------------------------------------------------------------------------ 64 bits
def _taylor(n, nbar=4, sll=35.0):
    """The Taylor window (scipy's convention, not normalised), float64."""
    B = 10.0 ** (sll / 20.0)
    A = math.acosh(B) / math.pi
    s2 = nbar ** 2 / (A ** 2 + (nbar - 0.5) ** 2)
    ma = np.arange(1, nbar)
    F = np.empty(nbar - 1)
    signs = np.ones(nbar - 1)
    signs[1::2] = -1
    for i, m in enumerate(ma):
        num = signs[i] * np.prod(1.0 - m * m / s2 / (A ** 2 + (ma - 0.5) ** 2))
        F[i] = num / (2.0 * np.prod(1.0 - m * m / ma[:i] ** 2) * np.prod(1.0 - m * m / ma[i + 1:] ** 2))
    x = (np.arange(n) - n / 2.0 + 0.5) / n
    return 1.0 + 2.0 * (F[:, None] * np.cos(2.0 * math.pi * ma[:, None] * x[None, :])).sum(0)


def _backproject(case, seed, up, interp, pts):
    """Sum over pulses of the range profile at each point (the zero-padded inverse transform at `up` times the
    samples, read linearly or by cubic Lagrange) turned by the carrier's phase, all in float64."""
    ant, fmin, df = _track(case)
    S = _history(case, seed).to(torch.complex128)
    P, K = S.shape
    if case.get('window', True):
        S *= torch.from_numpy(_taylor(P)).cuda()[:, None] * torch.from_numpy(_taylor(K)).cuda()[None, :]
    h = K // 2
    nfft = 1 << int(math.ceil(math.log2(up * K)))
    inv_dr, kcyc = 2.0 * df * nfft / C, 2.0 * (fmin + h * df) / C
    out = torch.zeros(len(pts[0]), dtype=torch.complex128, device='cuda')
    r0 = np.linalg.norm(ant, axis=1)
    nb = max(1, (1 << 25) // nfft)
    for p0 in range(0, P, nb):
        n = min(nb, P - p0)
        z = torch.zeros((n, nfft), dtype=torch.complex128, device='cuda')
        z[:, :K - h], z[:, nfft - h:] = S[p0:p0 + n, h:], S[p0:p0 + n, :h]
        z = torch.fft.ifft(z, dim=1) * nfft
        for q in range(n):
            a = ant[p0 + q]
            dR = torch.sqrt((pts[0] - a[0]) ** 2 + (pts[1] - a[1]) ** 2 + (pts[2] - a[2]) ** 2) - r0[p0 + q]
            t = dR * inv_dr
            i = torch.floor(t)
            w = t - i
            i = i.to(torch.int64)
            if interp == 'linear':
                wts = ((0, 1.0 - w), (1, w))
            else:
                wts = ((-1, -w * (w - 1) * (w - 2) / 6), (0, (w + 1) * (w - 1) * (w - 2) / 2),
                       (1, -(w + 1) * w * (w - 2) / 2), (2, (w + 1) * w * (w - 1) / 6))
            v = sum(z[q][torch.remainder(i + o, nfft)] * c for o, c in wts)
            ph = kcyc * dR
            out += v * torch.polar(torch.ones_like(ph), (2.0 * math.pi) * (ph - ph.round()))
    return out


def _grid_points(case):
    x = (torch.arange(case['nx'], device='cuda', dtype=torch.float64) - case['nx'] / 2.0) * case['sp']
    y = (torch.arange(case['ny'], device='cuda', dtype=torch.float64) - case['ny'] / 2.0) * case['sp']
    X, Y = torch.meshgrid(x, y, indexing='ij')
    X, Y = X.reshape(-1), Y.reshape(-1)
    return tuple(X * E1[k] + Y * E2[k] for k in range(3))


def exact(case, seed):
    """The pixels in 64 bits: for the formers the exact backprojection of the history (the factorized former's own
    approximation is then part of its distance from it), for the point and grid backprojections the same profiles and
    reads in float64."""
    if case['kind'] == 'pair':
        return _exact_pair(case, seed)
    if case['kind'] == 'points':
        p = torch.from_numpy(_points(case, seed)).cuda()
        return _backproject(case, seed, case['upsample'], 'linear', (p[:, 0], p[:, 1], p[:, 2]))
    if case['nx'] * case['ny'] * case['P'] > 3e10:
        return None                                                 # minutes
    up, interp = (8, case['interp']) if case['kind'] == 'exact' else (32, 'cubic')
    return _backproject(case, seed, up, interp, _grid_points(case)).reshape(case['nx'], case['ny'])


def _exact_pair(case, seed):
    a, b = (x.to(torch.complex128) for x in _pair(case, seed))
    n1, n2, la, lr = case['n1'], case['n2'], case['la'], case['lr']
    ab = a * b.conj()

    def box(x, n, w, dim):
        # moving mean of w along dim, the window from -(w // 2), the edge pixels repeated
        i = torch.arange(-(w // 2), n + w - 1 - w // 2, device='cuda').clamp(0, n - 1)
        c = torch.cumsum(x.index_select(dim, i), dim)
        c = torch.cat([torch.zeros_like(c.narrow(dim, 0, 1)), c], dim)
        return (c.narrow(dim, w, n) - c.narrow(dim, 0, n)) / w

    def mean(x):
        return box(box(x, n1, case['w1'], 0), n2, case['w2'], 1)
    coh = mean(ab).abs() / torch.sqrt(mean(a.abs() ** 2) * mean(b.abs() ** 2))
    m1, m2 = n1 // la, n2 // lr
    ifg = ab[:m1 * la, :m2 * lr].reshape(m1, la, m2, lr).mean((1, 3))
    return dict(coherence=coh, interferogram=ifg)
