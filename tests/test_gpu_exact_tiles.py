"""The exact former's tile kernel (ffbp_exact_backproject) and the pair coherence at the sizes where their indexing can
go wrong, against float64 numpy evaluations of the same sums."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')
if not torch.cuda.is_available():
    pytest.skip('no CUDA device', allow_module_level=True)

from fastsar_b200 import _lib, products  # noqa: E402


def _tiles_float64(prof, ant, ref, cen, nty, tx, ty, nx, ny, sp, inv_dr, kcyc, cubic):
    """The tile sum in float64: the third-order range about the tile's centre, Lagrange or linear reads."""
    nfft = prof.shape[1]
    out = np.zeros((nx, ny), complex)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing='ij')
    c = cen[(i // tx) * nty + j // ty]
    dx, dy = ((i % tx) - 0.5 * (tx - 1)) * sp, ((j % ty) - 0.5 * (ty - 1)) * sp
    most = 0.0
    for p in range(len(prof)):
        w = c - ant[p]
        r = np.sqrt((w ** 2).sum(-1))
        du = (dx * w[..., 0] + dy * w[..., 1]) / r
        de = du + (dx ** 2 + dy ** 2 - du ** 2) * (0.5 / r - du * 0.5 / r ** 2)
        x = (r - ref[p]) * inv_dr + de * inv_dr
        b = np.floor(x).astype(int)
        f = x - b
        if cubic:
            lag = [-f * (f - 1) * (f - 2) / 6, (f * f - 1) * (f - 2) / 2, -f * (f + 1) * (f - 2) / 2, f * (f * f - 1) / 6]
            v = sum(l * prof[p][(b - 1 + k) % nfft] for k, l in enumerate(lag))
        else:
            v = (1 - f) * prof[p][b % nfft] + f * prof[p][(b + 1) % nfft]
        out += v * np.exp(2j * np.pi * kcyc * (r - ref[p] + de))
        most = max(most, abs(kcyc * de).max())
    return out * nfft, most


@pytest.mark.parametrize('cubic', [1, 0])
@pytest.mark.parametrize('tx,ty', [(32, 32), (16, 16), (8, 16), (8, 8)])
def test_tile_sums_match_float64(tx, ty, cubic):
    rng = np.random.default_rng(tx * 100 + ty + cubic)
    n, nfft, nx, ny, sp = 37, 1024, 2 * tx + 5, ty + 3, 0.3          # partial tiles, a last group of pulses not full
    inv_dr, kcyc = 3.0, 60.0
    ntx, nty = -(-nx // tx), -(-ny // ty)
    ant = np.stack([rng.uniform(-50, 50, n), np.full(n, -3000.0), np.full(n, 2000.0)], 1)
    ref = np.sqrt((ant ** 2).sum(1)) + rng.uniform(-150, 150, n)     # bands that wrap past a profile's end too
    bx, by = np.meshgrid(np.arange(ntx), np.arange(nty), indexing='ij')
    cen = np.stack([(bx - 0.5) * tx * sp, (by - 0.5) * ty * sp, 0.0 * bx], -1).reshape(-1, 3)
    prof = (rng.normal(size=(n, nfft)) + 1j * rng.normal(size=(n, nfft))).astype(np.complex64)
    want, most = _tiles_float64(prof, ant, ref, cen, nty, tx, ty, nx, ny, sp, inv_dr, kcyc, cubic)
    L = _lib.load()
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (prof, ant, ref, cen)]
    got = {}
    for along1 in (0, 1):
        out = torch.zeros((nx, ny), dtype=torch.complex64, device='cuda')
        err = torch.zeros(1, dtype=torch.int32, device='cuda')
        _lib.check(L.ffbp_exact_backproject(d[0].data_ptr(), n, nfft, d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), ntx,
                                            nty, tx, ty, nx, ny, sp, sp, (ctypes.c_double * 3)(1, 0, 0),
                                            (ctypes.c_double * 3)(0, 1, 0), inv_dr, kcyc, cubic, along1, err.data_ptr(),
                                            out.data_ptr(), torch.cuda.current_stream().cuda_stream), 'exact')
        assert int(err.item()) == 0
        got[along1] = out.cpu().numpy()
    assert np.array_equal(got[0], got[1])
    # float32: the bin's place is a sum below 256 of three rounded terms (3 2^-17 bins, white samples changing by up to
    # 3 a bin), the phase one of `most` cycles at most rounded three times, the sine and cosine 4e-7, the sums 37 2^-24
    bound = 9 * 2.0 ** -17 + 2 * np.pi * 3 * (most + 1) * 2.0 ** -24 + 1e-6 + n * 2.0 ** -24
    e = np.linalg.norm(got[0] - want) / np.linalg.norm(want)
    assert e < bound, (e, bound)


@pytest.mark.parametrize('n1,n2,w1,w2', [(1, 1, 1, 1), (49, 131, 1, 2), (50, 127, 8, 1), (97, 260, 9, 64), (65, 123, 7, 7),
                                         (130, 300, 5, 6), (3, 200, 64, 63)])
def test_coherence_windows_match_float64(n1, n2, w1, w2):
    rng = np.random.default_rng(n1 + n2 + w1 + w2)
    a = (rng.normal(size=(n1, n2)) + 1j * rng.normal(size=(n1, n2))).astype(np.complex64)
    b = (0.6 * a + rng.normal(size=(n1, n2)) + 1j * rng.normal(size=(n1, n2))).astype(np.complex64)

    def windows(x):
        x = np.pad(x, ((w1 // 2, w1 - 1 - w1 // 2), (w2 // 2, w2 - 1 - w2 // 2)), mode='edge')
        return np.lib.stride_tricks.sliding_window_view(x, (w1, w2)).sum((-1, -2))

    A, B = a.astype(complex), b.astype(complex)
    want = abs(windows(A * B.conj())) / np.sqrt(windows(abs(A) ** 2) * windows(abs(B) ** 2))
    got = products.coherence(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), w1, w2)
    got = got.cpu().numpy() if hasattr(got, 'cpu') else np.asarray(got)
    # w2 column sums, each rounded to float32 and added in float32: (w2 + 1) 2^-24 of sum |a||b|, of each intensity sum
    # and (half twice) of the root of their product; the coherence's own rounding
    assert abs(got - want).max() < (2 * (w2 + 1) + 2) * 2.0 ** -24 * 1.5
