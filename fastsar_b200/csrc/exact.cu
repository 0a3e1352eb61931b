// Exact backprojection and phase-history synthesis on the device: the oracle family of the former.
//
// bp_points_f64  exact backprojection at arbitrary points in float64 throughout (fastsar/bp.py:99-137's bp_points,
//                with float64 profiles as well): for every point and pulse the range offset
//                dR = |x - tx_p| (+ |x - rcv_p|, halved, bistatic) - ref_p, the range profile read at bin
//                dR inv_dr + nfft/2 by linear interpolation (circularly), turned by exp(2 pi i kcyc dR) and summed.
//                The profiles are the caller's (a zero-padded inverse FFT per pulse: cuFFT through torch).
// simulate       the phase history of point scatterers, S[p, k] += sum_n a_n exp(-2 pi i (2 f_k / c) dR_pn),
//                dR_pn = |x_n - ant_p| - |ant_p| (the CPHD convention, fastsar/sim.py:1-8): ranges and phases in
//                float64 per thread's run of 8 samples, a float32 complex recurrence along the run, the sum over
//                each chunk of 256 scatterers in float32 and over the chunks in float64.
#include "common.cuh"

namespace ffbp {

namespace {

// LPP lanes share a point, each taking every LPP-th pulse, and add their sums by shuffles: with a thread per point a few
// thousand points leave most of the device idle behind one thread's chain of dependent reads (20,000 points: 157 blocks). The launch takes the fewest lanes that fill the device.
template <int LPP>
__global__ void __launch_bounds__(128) bp_points_f64_kernel(const double2 *__restrict__ prof, int P, int nfft,
                                                            const double *__restrict__ tx, const double *__restrict__ rcv,
                                                            const double *__restrict__ ref, const double *__restrict__ pts,
                                                            long N, double inv_dr, double kcyc, double2 *__restrict__ out)
{
    const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x, n = gid / LPP;
    const int l = (int)(gid % LPP);
    const bool in = n < N;
    const double x = in ? pts[3 * n] : 0.0, y = in ? pts[3 * n + 1] : 0.0, z = in ? pts[3 * n + 2] : 0.0;
    double ar = 0.0, ai = 0.0;
    for (int p = l; in && p < P; p += LPP) {
        const double ax = x - tx[3 * p], ay = y - tx[3 * p + 1], az = z - tx[3 * p + 2];
        double dR = sqrt(ax * ax + ay * ay + az * az);
        if (rcv) {
            const double bx = x - rcv[3 * p], by = y - rcv[3 * p + 1], bz = z - rcv[3 * p + 2];
            dR = 0.5 * (dR + sqrt(bx * bx + by * by + bz * bz));
        }
        dR -= ref[p];
        const double t = dR * inv_dr + (double)(nfft / 2);
        const double fl = floor(t);
        long i = (long)fl % nfft;
        if (i < 0) i += nfft;
        const long i1 = (i + 1 == nfft) ? 0 : i + 1;
        const double w = t - fl;
        const double2 v0 = prof[(size_t)p * nfft + i], v1 = prof[(size_t)p * nfft + i1];
        const double vr = v0.x + w * (v1.x - v0.x), vi = v0.y + w * (v1.y - v0.y);
        double ph = kcyc * dR;
        ph -= rint(ph);
        double s, c;
        sincospi(2.0 * ph, &s, &c);
        ar += vr * c - vi * s;
        ai += vr * s + vi * c;
    }
#pragma unroll
    for (int o = LPP / 2; o > 0; o >>= 1) {
        ar += __shfl_xor_sync(0xffffffffu, ar, o);
        ai += __shfl_xor_sync(0xffffffffu, ai, o);
    }
    if (in && l == 0) out[n] = make_double2(out[n].x + ar, out[n].y + ai);
}

// The rows of S (complex64, or complex128) windowed (the float32 product wp[p] wk[k], then the sample times it in
// float32), times (-1)^i at place i of the zero-padded row, sample K / 2 at place 0: the unscaled inverse transform of
// the row is then the profile with zero delay at nfft / 2 (nfft even: the sign is the half-length shift, exactly).
template <class T>
__global__ void bp_pad_kernel(const T *__restrict__ S, long n, int K, const float *__restrict__ wp,
                              const float *__restrict__ wk, int nfft, double2 *__restrict__ pad)
{
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n * K; q += (long)gridDim.x * blockDim.x) {
        const long p = q / K;
        const int k = (int)(q - p * K), h = K / 2, i = k >= h ? k - h : nfft - h + k;
        const T v = S[q];
        double2 o = make_double2(v.x, v.y);
        if (wp) {
            const float w = __fmul_rn(wp[p], wk[k]);
            o = make_double2(__fmul_rn((float)v.x, w), __fmul_rn((float)v.y, w));
        }
        const double g = (i & 1) ? -1.0 : 1.0;
        pad[p * nfft + i] = make_double2(o.x * g, o.y * g);
    }
}

constexpr int SIM_NT = 256;
constexpr int SIM_RUN = 8;                               // consecutive samples per thread

// One block: pulse p, SIM_NT * SIM_RUN consecutive samples. Per scatterer the block stages in shared memory the
// phase at its first sample (float64, reduced) and the per-sample step (float64 phase, its phasor in float32); each
// thread seeds its run's phasor from the float64 phase of its first sample and advances it by the step's phasor
// across its SIM_RUN samples (a complex recurrence of SIM_RUN - 1 steps: about 1e-6 relative).
__global__ void __launch_bounds__(SIM_NT) simulate_kernel(const double *__restrict__ ant, int P, int K, double fmin,
                                                          double df, const double *__restrict__ pos,
                                                          const double2 *__restrict__ amp, int N,
                                                          float2 *__restrict__ S)
{
    __shared__ double s_ph[SIM_NT], s_st[SIM_NT];
    __shared__ float2 s_w[SIM_NT];
    __shared__ double2 s_a[SIM_NT];
    const int span = SIM_NT * SIM_RUN;
    const int nkb = (K + span - 1) / span;
    const int p = blockIdx.x / nkb;
    const int k0 = (blockIdx.x % nkb) * span;
    const int t = threadIdx.x;
    const double ax = ant[3 * p], ay = ant[3 * p + 1], az = ant[3 * p + 2];
    const double r0 = sqrt(ax * ax + ay * ay + az * az);
    const double two_c = 2.0 / C_LIGHT;
    double sr[SIM_RUN], si[SIM_RUN];
#pragma unroll
    for (int j = 0; j < SIM_RUN; ++j) sr[j] = si[j] = 0.0;
    for (int n0 = 0; n0 < N; n0 += SIM_NT) {
        const int n = n0 + t;
        if (n < N) {
            const double dx = pos[3 * n] - ax, dy = pos[3 * n + 1] - ay, dz = pos[3 * n + 2] - az;
            const double dR = sqrt(dx * dx + dy * dy + dz * dz) - r0;
            const double ph = -two_c * (fmin + k0 * df) * dR;     // cycles at this block's first sample
            double st = -two_c * df * dR;                         // cycles per sample
            st -= rint(st);
            s_ph[t] = ph - rint(ph);
            s_st[t] = st;
            float sn, cs;
            sincospif(2.f * (float)st, &sn, &cs);
            s_w[t] = make_float2(cs, sn);
            s_a[t] = amp[n];
        } else {
            s_ph[t] = 0.0; s_st[t] = 0.0; s_w[t] = make_float2(1.f, 0.f); s_a[t] = make_double2(0.0, 0.0);
        }
        __syncthreads();
        const int nn = min(SIM_NT, N - n0);
        float cr[SIM_RUN], ci[SIM_RUN];
#pragma unroll
        for (int j = 0; j < SIM_RUN; ++j) cr[j] = ci[j] = 0.f;
        for (int m = 0; m < nn; ++m) {
            const double ph = fma((double)(SIM_RUN * t), s_st[m], s_ph[m]);
            float sn, cs;
            sincospif(2.f * (float)(ph - rint(ph)), &sn, &cs);
            const float2 st = s_w[m];
            const double2 a = s_a[m];
            float wr = (float)a.x * cs - (float)a.y * sn, wi = (float)a.x * sn + (float)a.y * cs;
#pragma unroll
            for (int j = 0; j < SIM_RUN; ++j) {
                cr[j] += wr;
                ci[j] += wi;
                const float nr = wr * st.x - wi * st.y;
                wi = wr * st.y + wi * st.x;
                wr = nr;
            }
        }
#pragma unroll
        for (int j = 0; j < SIM_RUN; ++j) { sr[j] += cr[j]; si[j] += ci[j]; }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < SIM_RUN; ++j) {
        const int k = k0 + SIM_RUN * t + j;
        if (k < K) {
            const float2 o = S[(size_t)p * K + k];
            S[(size_t)p * K + k] = make_float2(o.x + (float)sr[j], o.y + (float)si[j]);
        }
    }
}

}  // namespace

cudaError_t launch_bp_points_f64(const double2 *prof, int P, int nfft, const double *tx, const double *rcv,
                                 const double *ref, const double *pts, long N, double inv_dr, double kcyc, double2 *out,
                                 cudaStream_t s)
{
    if (N <= 0 || P <= 0) return cudaSuccess;
    const int nt = 128;
    int lpp = 1;
    while (lpp < 32 && N * lpp < 148L * 2048 && P >= 16 * lpp) lpp *= 2;
    const unsigned nb = (unsigned)((N * lpp + nt - 1) / nt);
    auto run = [&](auto kern) { kern<<<nb, nt, 0, s>>>(prof, P, nfft, tx, rcv, ref, pts, N, inv_dr, kcyc, out); };
    switch (lpp) {
        case 1: run(bp_points_f64_kernel<1>); break;
        case 2: run(bp_points_f64_kernel<2>); break;
        case 4: run(bp_points_f64_kernel<4>); break;
        case 8: run(bp_points_f64_kernel<8>); break;
        case 16: run(bp_points_f64_kernel<16>); break;
        default: run(bp_points_f64_kernel<32>); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_bp_pad(const void *S, int c128, long n, int K, const float *wp, const float *wk, int nfft,
                          double2 *pad, cudaStream_t s)
{
    if (n <= 0 || K <= 0) return cudaSuccess;
    const long nb = (n * K + 255) / 256;
    const unsigned g = (unsigned)(nb < 148 * 16 ? nb : 148 * 16);
    if (c128) bp_pad_kernel<<<g, 256, 0, s>>>(static_cast<const double2 *>(S), n, K, wp, wk, nfft, pad);
    else bp_pad_kernel<<<g, 256, 0, s>>>(static_cast<const float2 *>(S), n, K, wp, wk, nfft, pad);
    return cudaGetLastError();
}

cudaError_t launch_simulate(const double *ant, int P, int K, double fmin, double df, const double *pos,
                            const double2 *amp, int N, float2 *S, cudaStream_t s)
{
    if (P <= 0 || K <= 0 || N <= 0) return cudaSuccess;
    const long nb = (long)((K + SIM_NT * SIM_RUN - 1) / (SIM_NT * SIM_RUN)) * P;
    if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
    simulate_kernel<<<(unsigned)nb, SIM_NT, 0, s>>>(ant, P, K, fmin, df, pos, amp, N, S);
    return cudaGetLastError();
}

}  // namespace ffbp
