"""The tensor-core kernels of the float32 and mixed-precision forms at the sizes where their layouts change: the level's
product (residues per row, several pulses per unit, partial units and tiles, children in groups, planes of 8 samples,
short tiles), the float32 form's images against the float64 oracle of the same plan, and the point backprojection's lanes
per point and the coherence's window forms against plain NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')
if not torch.cuda.is_available():
    pytest.skip('no CUDA device', allow_module_level=True)

from test_gpu_parity import (_level_case, _oracle_level_full, _rel, _run_level_gpu, _run_level_tc,  # noqa: E402,F401
                             lib)


# Np, P, K, C, Dk, Dp, frequency pass fraction
LAYOUTS = [
    (5, 37, 60, 4, 2, 2, 0.6),        # a row needs half of the accumulator's rows: two pulses a unit, the last alone
    (3, 43, 30, 9, 1, 3, 0.6),        # Dk = 1 and 30 columns: four pulses a unit, two groups of 8 child columns
    (2, 21, 44, 8, 3, 2, 0.6),        # 23 columns, 25 taps
    (1, 65, 1100, 17, 2, 3, 0.6),     # two residues a row, the last tile's columns odd
    (1, 33, 515, 3, 1, 1, 0.6),       # no filter on either axis, four columns a row
    (1, 24, 700, 64, 8, 2, 0.45),     # 8 samples a row, 64 children
    (1, 40, 500, 64, 11, 3, 0.3),     # two planes of 8 samples
    (1, 30, 900, 40, 9, 3, 0.45),     # a plane of 8 samples and a gathered one, two steps of it (9 taps a phase)
    (2, 26, 640, 12, 10, 4, 0.3),     # two gathered planes
    (1, 20, 1500, 5, 17, 2, 0.2),     # two planes of 8 samples and a gathered one
]


def _layout_id(c):
    return 'Np%d-P%d-K%d-C%d-Dk%d-Dp%d' % c[:6]


@pytest.mark.parametrize('case', LAYOUTS, ids=_layout_id)
def test_level_layouts_match_oracle(lib, oracle_lib, case):  # noqa: F811
    """The mixed-precision level against the float64 oracle: split float16 products (2^-22) and a float16 intermediate
    (2^-12 rms a sample, averaged by the pulse filter): below 5e-4."""
    Np, P, K, C, Dk, Dp, pk = case
    rng = np.random.default_rng(sum(case[:6]))
    x, c0, sl, fk, fp, Ko, Po = _level_case(rng, Np, P, K, C, Dk, Dp, pk=pk)
    got, st = _run_level_tc(lib, x, c0, sl, fk, fp, Ko, Po, Dk, Dp)
    e = _rel(got, _oracle_level_full(oracle_lib, x, c0, sl, fk, fp, Ko, Po, Dk, Dp))
    print(f'level {case} Ko {Ko}: rel {e:.2e}')
    assert st[0] == 0 and e < 5e-4


def _level_float64(x, c0, sl, fk, fp, Ko, Po, Dk, Dp):
    """The level in float64: each child's rotated rows, the frequency FIR, the pulse FIR."""
    def fir(v, f, D, n):                               # along the last axis; zeros outside
        if f is None:
            return v
        h, L, pl = np.asarray(f['kern'], np.float32).astype(float), f['L'], f['pl']
        v = np.pad(v, [(0, 0)] * (v.ndim - 1) + [(pl, D * n + L)])
        return np.lib.stride_tricks.sliding_window_view(v, L, -1)[..., :D * n:D, :] @ h[:L]
    Np, P, K = x.shape
    C = c0.shape[1]
    k = np.arange(K) - (K - 1) / 2.0
    out = np.empty((Np, C, Po, Ko), complex)
    for n in range(Np):
        for c in range(C):
            z = x[n] * np.exp(2j * np.pi * (c0[n, c].astype(float)[:, None] + sl[n, c].astype(float)[:, None] * k))
            out[n, c] = fir(fir(z, fk, Dk, Ko).T, fp, Dp, Po).T
    return out.reshape(Np * C, Po, Ko)


@pytest.mark.parametrize('case', LAYOUTS + [
    (1, 21, 2600, 5, 40, 2, 0.4),     # long filters: a tile of 64 columns or fewer
    (4, 19, 1100, 12, 2, 3, 0.6),     # several parents, columns and children at a time (below)
], ids=_layout_id)
def test_float32_level_layouts(lib, case):  # noqa: F811
    """The float32 form's level through the same layouts, whole and in the pieces that less scratch leaves (parents; columns
    of one, the last ones odd; 8 of its children and 128 columns), against float64: split float16 products (2^-22), the
    hardware sine and cosine (4e-7) and float32 sums, 5e-6 (a missing low part of either operand is 1e-4)."""
    Np, P, K, C, Dk, Dp, pk = case
    rng = np.random.default_rng(sum(case[:6]))
    x, c0, sl, fk, fp, Ko, Po = _level_case(rng, Np, P, K, C, Dk, Dp, pk=pk)
    want = _level_float64(x, c0, sl, fk, fp, Ko, Po, Dk, Dp)
    L = lib.load()
    dx, dph = torch.from_numpy(x).cuda(), torch.from_numpy(np.stack([c0, sl], -1).astype(np.float32)).cuda()
    tk, tp = (torch.from_numpy(np.asarray(f['kern'], np.float32)).cuda() if f else None for f in (fk, fp))
    parent, column = C * P * (-(-Ko // 4) * 4) * 8, P * 8
    least = min(parent, 8 * column * (128 if Ko > 128 else -(-Ko // 4) * 4))
    args = (dx.data_ptr(), Np, P, K, dph.data_ptr(), C, lib.tptr(tk), fk['L'] if fk else 1, fk['pl'] if fk else 0, Dk, Ko,
            (K - 1) / 2.0, lib.tptr(tp), fp['L'] if fp else 1, fp['pl'] if fp else 0, Dp, Po, None, None)
    stream = torch.cuda.current_stream().cuda_stream
    for size in sorted({Np * parent, min(2, Np) * parent, parent, min(parent, C * column * 128), least}, reverse=True):
        scratch = torch.empty(size // 4 + 4, dtype=torch.int32, device='cuda')
        out = torch.full((Np * C, Po, Ko), float('nan'), dtype=torch.complex64, device='cuda')
        status = torch.zeros(3, dtype=torch.int32, device='cuda')
        lib.check(L.ffbp_level_tc32(*args, out.data_ptr(), None, scratch.data_ptr(), size, status.data_ptr(), stream), 'level')
        got, st = out.cpu().numpy(), status.cpu().numpy()
        e = _rel(got, want)
        print(f'level {case} Ko {Ko}, scratch {size} of {Np * parent}: rel {e:.2e}')
        assert st[0] == 0 and e < 5e-6
        assert st[2:].view(np.float32)[0] == max(abs(got.real).max(), abs(got.imag).max())
    with pytest.raises(ValueError, match='too small'):
        lib.check(L.ffbp_level_tc32(*args, out.data_ptr(), None, scratch.data_ptr(), column, status.data_ptr(), stream), 'level')


@pytest.mark.parametrize('Dp,pp,form', [
    (700, 0.4, 'both'),               # pulse taps of 44 KB: the most in the memory a launch has without asking
    (1351, 0.4, 'both'),              # 84 KB
    (3300, 0.4, 'both'),              # 206 KB: too much beside the CUDA-core level's rows, whose taps stay in global memory
    (4000, 0.4, 'cores'),             # 250 KB: the CUDA-core level alone
    (2400, 0.75, 'cores'),            # 14 taps a phase, 300 KB
])
def test_levels_of_long_pulse_filters(lib, Dp, pp, form):  # noqa: F811
    """Levels that decimate thousands of pulses to one (chips of collections of 10^5 pulses) on both kernels, against
    float64: as above 5e-6 (sums of some 10^4 products add float32 roundings of about 1e-7 each, averaged)."""
    rng = np.random.default_rng(Dp)
    x, c0, sl, fk, fp, Ko, Po = _level_case(rng, 1, 14 * Dp, 21, 3, 1, Dp, pp=pp)
    want = _level_float64(x, c0, sl, fk, fp, Ko, Po, 1, Dp)
    e = _rel(_run_level_gpu(lib, x, c0, sl, fk, fp, Ko, Po, 1, Dp), want)
    print(f'Dp {Dp}, {fp["L"]} taps: CUDA cores {e:.2e}')
    assert e < 5e-6
    L = lib.load()
    P, K, C = x.shape[1], x.shape[2], 3
    dx, dph = torch.from_numpy(x).cuda(), torch.from_numpy(np.stack([c0, sl], -1).astype(np.float32)).cuda()
    tp = torch.from_numpy(np.asarray(fp['kern'], np.float32)).cuda()
    size = C * P * (-(-Ko // 4) * 4) * 8
    scratch = torch.empty(size // 4, dtype=torch.int32, device='cuda')
    out = torch.empty((C, Po, Ko), dtype=torch.complex64, device='cuda')
    status = torch.zeros(3, dtype=torch.int32, device='cuda')

    def run():
        lib.check(L.ffbp_level_tc32(dx.data_ptr(), 1, P, K, dph.data_ptr(), C, None, 1, 0, 1, Ko, (K - 1) / 2.0, tp.data_ptr(),
                                    fp['L'], fp['pl'], Dp, Po, None, None, out.data_ptr(), None, scratch.data_ptr(), size,
                                    status.data_ptr(), torch.cuda.current_stream().cuda_stream), 'ffbp_level_tc32')
    if form == 'cores':
        with pytest.raises(ValueError, match='pulse taps'):
            run()
        return
    run()
    e = _rel(out.cpu().numpy(), want)
    print(f'Dp {Dp}, {fp["L"]} taps: tensor cores {e:.2e}')
    assert e < 5e-6 and int(status[0].item()) == 0


def test_chip_of_many_pulses(oracle_lib):
    """A 64-pixel chip of 65,536 pulses, whose first level takes 1,351 pulses to one: the float32 image against the oracle's
    (1e-5, as the other float32 images)."""
    from fastsar_b200 import ImageFormer, sim
    P, K, n = 65536, 96, 64
    col = sim.spotlight(P, K, 9.6e9, 300e6, 600e3, 45.0, 1.5)
    f = ImageFormer(col.ant, col.fmin, col.df, K, n, n, 0.25, 0.25, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0), T=16)
    assert max(l['Dp'] for l in f._plan['levels']) > 1000
    rng = np.random.default_rng(6)
    S = (rng.standard_normal((P, K)) + 1j * rng.standard_normal((P, K))).astype(np.complex64)
    form, _ = oracle_lib.image_former(col.ant, col.fmin, col.df, K, n, n, 0.25, 0.25, e1=(0.0, 1.0, 0.0),
                                      e2=(1.0, 0.0, 0.0), T=16, kind='port')
    e = _rel(f(S), form(S))
    print(f'{P} pulses: rel {e:.2e}')
    assert e < 1e-5


@pytest.mark.parametrize('P,K,nx,ny,T,window', [
    (97, 83, 33, 65, 16, True),       # odd sizes, T = 16: the last unit of two tiles half empty
    (128, 96, 64, 64, 32, True),
    (256, 700, 100, 130, 32, False),  # a first level with long filters
    (300, 260, 150, 120, 16, True),
])
def test_float32_form_matches_float64_oracle(oracle_lib, P, K, nx, ny, T, window):
    """The float32 former's image against the float64 oracle of the same plan. Per factor float32 rounding, the split
    float16 products (2^-22) and the hardware sine and cosine (5e-7) leave 1e-6 to 3e-6; the phases here are tens of
    cycles (float32: 2e-6 rad). Below 1e-5, with the tensor cores in the levels and the final stage."""
    from fastsar_b200 import ImageFormer, sim
    col = sim.spotlight(P, K, 9.6e9, 300e6, 600e3, 45.0, 1.5)
    rng = np.random.default_rng(P + K)
    pos, amp = sim.scene(rng, nx, ny, 0.25, 0.25, n_points=12)
    S = sim.add_noise(sim.simulate_brute(col, pos, amp), 0.01, rng).astype(np.complex64)
    f = ImageFormer(col.ant, col.fmin, col.df, K, nx, ny, 0.25, 0.25, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0), T=T, window=window)
    img = f(S)
    form, _ = oracle_lib.image_former(col.ant, col.fmin, col.df, K, nx, ny, 0.25, 0.25, e1=(0.0, 1.0, 0.0),
                                      e2=(1.0, 0.0, 0.0), T=T, window_on=window, kind='port')
    e = _rel(img, form(S))
    out = torch.empty((nx, ny), dtype=torch.complex64, device='cuda')
    kinds = [k for k, _, _ in f._dev.form_profile(torch.from_numpy(S).cuda(), out)]
    print(f'{P} x {K} -> {nx} x {ny}, T {T}: rel {e:.2e}, {kinds}')
    assert e < 1e-5
    assert 'level_tc_gemm' in kinds and kinds[-1] == 'final_tc'


@pytest.mark.parametrize('P,K,bw,ap,sp,T,items,odd', [
    (200, 16, 20e6, 1.5, 0.25, 32, 2, True),       # final subapertures of 2, 4 and 6 items for the twelve warps that
    (201, 16, 20e6, 1.5, 0.25, 32, 2, False),      # build operands, odd and even counts of them: a row's samples up to
    (300, 260, 300e6, 1.5, 0.1, 32, 4, True),      # 16, 32 and 48
    (301, 260, 300e6, 1.2, 0.1, 32, 4, False),
    (420, 400, 300e6, 1.5, 0.25, 32, 6, True),
    (400, 400, 300e6, 1.5, 0.25, 32, 6, False),
    (300, 260, 300e6, 1.5, 0.15, 16, 4, True),
    (300, 260, 300e6, 1.5, 0.1, 16, 4, False),
])
def test_final_stage_with_fewer_items_than_warps(oracle_lib, P, K, bw, ap, sp, T, items, odd):
    """625 tiles of 32 x 32 pixels or 2,500 of 16 x 16, several units for every block, whose producer warps have items in
    some subapertures only: against the float64 oracle (as above: below 1e-5), and the same bits twenty times."""
    from fastsar_b200 import ImageFormer, sim
    n = 800
    col = sim.spotlight(P, K, 9.6e9, bw, 600e3, 45.0, ap)
    rng = np.random.default_rng(P + K)
    pos, amp = sim.scene(rng, n, n, sp, sp, n_points=12)
    S = sim.add_noise(sim.simulate_brute(col, pos, amp), 0.01, rng).astype(np.complex64)
    f = ImageFormer(col.ant, col.fmin, col.df, K, n, n, sp, sp, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0), T=T)
    last = f._plan['levels'][-1]
    groups = -(-last['Ko'] // 8)                   # of 8 samples: 64 / T to an item, A and B, 32 / T tiles to a unit
    assert (32 // T) * 2 * -(-groups // (64 // T)) == items and last['Po'] % 2 == odd
    form, _ = oracle_lib.image_former(col.ant, col.fmin, col.df, K, n, n, sp, sp, e1=(0.0, 1.0, 0.0),
                                      e2=(1.0, 0.0, 0.0), T=T, kind='port')
    dS = torch.from_numpy(S).cuda()
    img = f.form_device(dS).clone()
    e = _rel(img.cpu().numpy(), form(S))
    print(f'{P} x {K} at T {T}: {items} items, rel {e:.2e}')
    assert e < 1e-5
    for _ in range(19):
        assert torch.equal(torch.view_as_real(f.form_device(dS)), torch.view_as_real(img))


@pytest.mark.parametrize('precision', ['float32', 'float16'])
def test_history_between_16_byte_boundaries(precision):
    """The second history of a stack of odd-sized ones starts 8 bytes past a 16-byte boundary: the bits of its copy's
    image, also with the largest sample at the ends, which the scan reads apart (a scan that misses it scales by 256 too
    much and reports the sample as non-finite)."""
    from fastsar_b200 import ImageFormer, sim
    P, K, n = 97, 83, 65
    col = sim.spotlight(P, K, 9.6e9, 300e6, 600e3, 45.0, 1.5)
    f = ImageFormer(col.ant, col.fmin, col.df, K, n, n, 0.25, 0.25, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0), T=16,
                    precision=precision)
    gen = torch.Generator(device='cuda').manual_seed(1)
    stack = torch.randn((2, P, K), dtype=torch.complex64, device='cuda', generator=gen)
    assert stack[1].data_ptr() % 16 == 8
    for at in (None, (0, 0), (0, 1), (P - 1, K - 1), (P - 1, K - 2)):
        if at is not None:
            stack[1][at] = 1e6
        a = f.form_device(stack[1]).clone()
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(f.form_device(stack[1].clone())))
        if at is not None:
            stack[1][at] = 0.0


@pytest.mark.parametrize('precision', ['float32', 'float16'])
@pytest.mark.parametrize('pulses,samples,amplitude', [
    (1 / 4096.0, 1 / 2048.0, 1.0),    # a window normalised to a sum of one: products of 2^-23
    (2.0 ** 12, 1.0, 1.0),            # products past float16's range
    (1.0, 1.0, 2.0 ** 108),           # histories near either end of float32's range
    # (at the lower end t = 2^-126 / 2^-112 of a sample, a level's output a tenth of it: flushed values below 10 t, of
    # which there are 0.8 10 t, cost sqrt(0.27 (10 t)^3) = 8e-6 a level in any float32 kernel; at 2^-104 2e-9)
    (1.0, 1.0, 2.0 ** -104),
])
def test_scales_of_window_and_history(precision, pulses, samples, amplitude):
    """The image of a scaled window or history is the scaled image: powers of two, so that nothing but the split products'
    place in float16's range can differ (2^-22 to 2^-24 a factor: below 2e-6, in the float16 form a rounding of the
    intermediate here and there, 2^-12 each: below 5e-4), and nothing is taken for non-finite."""
    from fastsar_b200 import ImageFormer, sim
    from fastsar_b200.api import DevicePlan, _final_mode
    P, K, n = 128, 96, 64
    col = sim.spotlight(P, K, 9.6e9, 300e6, 600e3, 45.0, 1.5)
    f = ImageFormer(col.ant, col.fmin, col.df, K, n, n, 0.25, 0.25, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0), precision=precision)
    S = torch.randn((P, K), dtype=torch.complex64, device='cuda', generator=torch.Generator(device='cuda').manual_seed(3))
    out = torch.empty((n, n), dtype=torch.complex64, device='cuda')
    want = f.form_device(S).cpu().numpy().astype(complex)
    dev = DevicePlan(f._plan, (f.wp * np.float32(pulses)), (f.wk * np.float32(samples)), None, None, _final_mode(precision))
    dev.form(S * amplitude, out)
    got = out.cpu().numpy().astype(complex) / (pulses * samples * amplitude)
    e = _rel(got, want)
    print(f'{precision}: window {pulses * samples:.1e}, history {amplitude:.1e}: rel {e:.1e}')
    assert e < (2e-6 if precision == 'float32' else 5e-4)


def test_pulse_of_a_non_finite_sample_among_large_ones():
    """An infinite or undefined sample names its pulse and no other, whatever the finite samples near it."""
    from fastsar_b200 import ImageFormer, sim
    P, K, n = 128, 96, 64
    col = sim.spotlight(P, K, 9.6e9, 300e6, 600e3, 45.0, 1.5)
    f = ImageFormer(col.ant, col.fmin, col.df, K, n, n, 0.25, 0.25, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0))
    for bad in (float('inf'), float('nan')):
        S = torch.ones((P, K), dtype=torch.complex64, device='cuda')
        S[40, 50] = 1e9                                       # read by the same thread as the next sample
        S[70, 51] = bad
        S[40, 51] = bad
        with pytest.raises(ValueError, match='pulse 40'):
            f.form_device(S)
        S[40, 51] = 0.0
        with pytest.raises(ValueError, match='pulse 70'):
            f.form_device(S)


@pytest.mark.parametrize('name,value,precision,kinds,bound', [
    ('FASTSAR_FINAL', 'fp32', 'float32', {'final_fp32'}, 1e-5),
    ('FASTSAR_FINAL', 'tc3', 'float32', {'final_tc'}, 1e-4),          # split bfloat16: 16 bits
    ('FASTSAR_LEVELS', 'fp32', 'float16', {'level_fp32', 'final_tc'}, 2e-3),    # a float16 final stage: 2^-11
])
def test_switches_choose_their_kernels(monkeypatch, name, value, precision, kinds, bound):
    """FASTSAR_FINAL=fp32 keeps the float32 form's final stage on the CUDA cores and FASTSAR_LEVELS=fp32 all of the float16
    form's levels, also where the tensor cores cover the shape: the kernels by name, and the default form's image."""
    from fastsar_b200 import ImageFormer, sim
    P, K, n = 128, 96, 64
    col = sim.spotlight(P, K, 9.6e9, 300e6, 600e3, 45.0, 1.5)
    args = (col.ant, col.fmin, col.df, K, n, n, 0.25, 0.25, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0))
    S = torch.randn((P, K), dtype=torch.complex64, device='cuda', generator=torch.Generator(device='cuda').manual_seed(2))
    out = torch.empty((n, n), dtype=torch.complex64, device='cuda')
    monkeypatch.delenv('FASTSAR_FINAL', raising=False)
    monkeypatch.delenv('FASTSAR_LEVELS', raising=False)
    want = ImageFormer(*args, precision=precision).form_device(S).cpu().numpy()
    monkeypatch.setenv(name, value)
    f = ImageFormer(*args, precision=precision)
    run = [k for k, _, _ in f._dev.form_profile(S, out)]
    assert {k for k in run if k.startswith(name[8:13].lower())} | {run[-1]} == kinds, run
    assert _rel(f.form_device(S).cpu().numpy(), want) < bound


def test_float32_form_with_large_phases_keeps_its_kernel(oracle_lib):
    """A level whose rotation phases pass the bound runs on the CUDA cores (its image is what it was), the later ones on
    the tensor cores; a non-finite sample is named by either."""
    from fastsar_b200 import ImageFormer, sim
    col = sim.spotlight(200, 1500, 9.6e9, 900e6, 20e3, 40.0, 2.0)
    f = ImageFormer(col.ant, col.fmin, col.df, 1500, 96, 700, 0.3, 0.3, (0.0, 1.0, 0.0), (1.0, 0.0, 0.0), T=16)
    S = torch.randn((200, 1500), dtype=torch.complex64, device='cuda')
    out = torch.empty((96, 700), dtype=torch.complex64, device='cuda')
    kinds = [k for k, _, _ in f._dev.form_profile(S, out)]
    assert kinds[0] == 'level_fp32' and 'level_tc_gemm' in kinds, kinds
    S[123, 45] = float('nan')
    with pytest.raises(ValueError, match='pulse 123'):
        f.form_device(S)


@pytest.mark.parametrize('N,P', [(1, 5), (700, 40), (9000, 33), (400000, 3)])
def test_points_lanes_match_numpy(N, P):
    """backproject_device at point counts that take 32, some and one lane per point (and fewer pulses than lanes),
    float64 throughout. The two sides round ranges of 1e4 m (1.8e-12 m) in different orders, 64 cycles a metre: 7e-10
    rad; below 2e-9."""
    from fastsar_b200.exact import C, backproject_device
    rng = np.random.default_rng(N)
    K, fmin, df = 48, 9.6e9, 2e6
    ant = np.stack([np.full(P, -7e3), np.linspace(-60, 60, P), np.full(P, 7e3)], 1)
    S = rng.standard_normal((P, K)) + 1j * rng.standard_normal((P, K))
    pts = rng.uniform(-20, 20, (N, 3))
    got = backproject_device(S, ant, fmin, df, pts, window=False, upsample=4).cpu().numpy()
    nfft, h = 256, K // 2
    pad = np.zeros((P, nfft), complex)
    pad[:, :K - h], pad[:, nfft - h:] = S[:, h:], S[:, :h]
    prof = np.fft.ifft(pad, axis=1) * nfft
    want = np.zeros(N, complex)
    for p in range(P):
        dR = np.linalg.norm(pts - ant[p], axis=1) - np.linalg.norm(ant[p])
        t = dR * (2 * df * nfft / C)
        i = np.floor(t).astype(int)
        w = t - i
        want += ((1 - w) * prof[p, i % nfft] + w * prof[p, (i + 1) % nfft]) * np.exp(2j * np.pi * (2 * (fmin + h * df) / C) * dR)
    assert _rel(got, want) < 2e-9


@pytest.mark.parametrize('window', [True, False])
@pytest.mark.parametrize('make', [
    lambda S: S.conj(),                                    # conjugated when read
    lambda S: S.T.contiguous().T,                          # pulses the fast axis
    lambda S: S.to(torch.complex64).conj()[:, ::2],
    lambda S: S.real,                                      # a real view of complex storage
    lambda S: torch._neg_view(S.conj()),                   # negated and conjugated when read
    lambda S: S[:1].expand(9, -1),
], ids=['conj', 'transposed', 'strided', 'real', 'neg', 'expanded'])
def test_points_take_any_view_of_a_history(make, window):
    """backproject_device on views whose buffer is not the history as it reads: the bits of the materialised copy's."""
    from fastsar_b200.exact import backproject_device
    gen = torch.Generator(device='cuda').manual_seed(4)
    S = torch.randn((9, 48), dtype=torch.complex128, device='cuda', generator=gen)
    v = make(S)
    ant = np.stack([np.full(9, -7e3), np.linspace(-60, 60, 9), np.full(9, 7e3)], 1)
    pts = np.random.default_rng(1).uniform(-20, 20, (50, 3))
    got = backproject_device(v, ant, 9.6e9, 2e6, pts, window=window)
    want = backproject_device(torch.from_numpy(v.cpu().resolve_conj().resolve_neg().numpy().copy()), ant, 9.6e9, 2e6, pts, window=window)
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))


@pytest.mark.parametrize('w1,w2', [(1, 3), (2, 2), (5, 7), (8, 3), (11, 10), (12, 5)])
@pytest.mark.parametrize('n1,n2', [(7, 5), (67, 250)])
def test_coherence_windows(n1, n2, w1, w2):
    """The coherence at window and run edges, images smaller than a window among them, against float64 window sums: up to 10
    column sums, each rounded to float32 and added in float32, and the result's rounding, 2e-6; and exactly 0 inside a strip
    where one image is zero."""
    from scipy.ndimage import uniform_filter
    from fastsar_b200 import products
    rng = np.random.default_rng(n1 + w1)
    a = (rng.standard_normal((n1, n2)) + 1j * rng.standard_normal((n1, n2))).astype(np.complex64)
    b = (a + rng.standard_normal((n1, n2))).astype(np.complex64)
    a[:, n2 // 2:n2 // 2 + w2 + 3] = 0
    A, B = a.astype(complex), b.astype(complex)

    def mean(v):
        return uniform_filter(v, (w1, w2), mode='nearest')
    ab = A * B.conj()
    den = mean(np.abs(A) ** 2) * mean(np.abs(B) ** 2)
    want = np.sqrt(np.where(den > 1e-20, (mean(ab.real) ** 2 + mean(ab.imag) ** 2) / np.maximum(den, 1e-20), 0.0))
    got = products.coherence(a, b, w1, w2)
    zero = mean(np.abs(A) ** 2) < 1e-12
    np.testing.assert_allclose(got[~zero], want[~zero], rtol=0, atol=2e-6)
    np.testing.assert_array_equal(got[zero], 0.0)
    assert n2 < 50 or zero.any()


def test_coherence_of_the_longest_images():
    """More rows than 65,535 runs of 48 hold: the middle and the last rows against float64 window sums, as above."""
    from fastsar_b200 import products
    n1, n2 = 48 * 65535 + 1000, 2
    gen = torch.Generator(device='cuda').manual_seed(7)
    a = torch.randn((n1, n2), dtype=torch.complex64, device='cuda', generator=gen)
    b = a + torch.randn((n1, n2), dtype=torch.complex64, device='cuda', generator=gen)
    got = products.coherence(a, b, 3, 2)
    for r in (n1 // 2, n1 - 500):
        A, B = (v[r - 1:r + 500].to(torch.complex128) for v in (a, b))

        def window(v):                                        # rows i - 1 .. i + 1, columns j - 1 .. j, the edges repeated
            v = v[:-2] + v[1:-1] + v[2:]
            return torch.stack([2 * v[:, 0], v[:, 0] + v[:, 1]], 1)
        want = window(A * B.conj()).abs() / (window(A.abs() ** 2) * window(B.abs() ** 2)).sqrt()
        assert float((got[r:r + len(want)] - want).abs().max()) < 2e-6
