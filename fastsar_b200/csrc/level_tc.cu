// A level on the tcgen05 tensor cores (sm_100a): one merge stage of the FFBP (the reference's rot_fir_k + fir_p:
// fastsar/ffbp_cpu.cpp:146-293, fastsar/ffbp_cuda.py:48-256), in two passes.
//
// Pass 1 (level_mma.cu): per parent and pulse the rotation and the frequency FIR of every child as one product on the
// tensor cores, written at the input pulse rate as the intermediate y [Np, C, P, Kop]: float16 in the mixed-precision
// form, float32 in the float32 form, times a power of two (2^level_exponent).
//
// Pass 2: the pulse FIR of the intermediate, written as complex64 with the largest component recorded: on the CUDA
// cores in float32 (level_fir here: a thread per two columns with the ceil(Lp / Dp) outputs it feeds in registers), or
// for a float16 intermediate on the tensor cores as a banded product per row (level_fir_tc.cu); a launch option, by
// default the tensor cores for output pulse axes of 512 or more.
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace ffbp {

namespace {

// --------------------------------------------------------------------------------------------------- pass 2
struct FirArgs {
    const void *__restrict__ y;       // [rows, P, Kop] float16 or float32 complex, times 2^level_exponent
    const float *__restrict__ tp;     // [Lp]
    float2 *__restrict__ out;         // [rows, Po, Ko], columns nj of it from this pointer on
    int *amax;
    const int *amax_in;
    int rows, P, Kop, nj, Ko, Po, Dp, Lp, plp, SEG, nseg;
    int wexp;                         // (last: the loads of the others pair up; ahead of them 104 registers, 96 here)
};

// Two complex samples of the intermediate: 8 bytes of float16 or 16 of float32.
template <bool F32> struct Pair { using T = uint2; };
template <> struct Pair<true> { using T = float4; };

__device__ __forceinline__ void unpack(const uint2 &v, float2 &a, float2 &b)
{
    a = __half22float2(*reinterpret_cast<const __half2 *>(&v.x));
    b = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
}

__device__ __forceinline__ void unpack(const float4 &v, float2 &a, float2 &b)
{
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
}

template <int AP, bool F32>
__global__ void __launch_bounds__(128) level_fir(const FirArgs a)
{
    constexpr int APP = (AP + 3) & ~3;
    // [Dp][APP] pairs: s_tp[b APP + s] = (tp[Dp s + b], tp[Dp s + b]), a tap twice for the packed multiply-adds
    extern __shared__ __align__(16) float2 s_tp[];
    // thread -> (row, pair of columns j, j + 1), consecutive threads along a row's pairs and on into the next row;
    // blockIdx.y: the segment of output pulses
    const int t = threadIdx.x;
    for (int r = t; r < a.Dp * APP; r += 128) {
        const int b = r / APP, s = r - b * APP;
        const int tap = a.Dp * s + b;
        const float v = (s < AP && tap < a.Lp) ? (a.tp ? a.tp[tap] : 1.f) : 0.f;   // Dp = 1: one tap 1
        s_tp[r] = make_float2(v, v);
    }
    __syncthreads();
    using PT = typename Pair<F32>::T;
    const int npair = (a.nj + 1) / 2;
    const long gid = (long)blockIdx.x * 128 + t;
    if (gid >= (long)a.rows * npair) return;
    const int row = (int)(gid / npair), j = 2 * (int)(gid - (long)row * npair);
    const int seg = blockIdx.y;
    const float inv = pow2(-level_exponent(a.amax_in, a.wexp));
    const int i_s = seg * a.SEG, i_e = min(a.Po, i_s + a.SEG);
    const int g_end = i_e + AP - 1;
    const PT *__restrict__ yr = static_cast<const PT *>(a.y) + ((size_t)row * a.P * a.Kop + j) / 2;   // Kop, j even
    const size_t ypitch = a.Kop / 2;
    float2 acc[2][AP];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int s = 0; s < AP; ++s) acc[h][s] = make_float2(0.f, 0.f);
    float vmax = 0.f;
    // input pulses p_start .. p_stop - 1 in chunks of U, the next chunk's loads in flight while one is filtered
    constexpr int U = F32 ? 4 : 8;                        // float32: fewer registers, more warps (605 -> 533 us at 30 children
                                                          // x 448 parents of the 12,288 x 8,832 spotlight's third level)
    const int p_start = a.Dp * i_s - a.plp, p_stop = a.Dp * g_end - a.plp;
    auto ld = [&](int pp) -> PT { return (pp >= 0 && pp < a.P) ? __ldg(yr + (size_t)pp * ypitch) : PT{}; };
    PT cur[U], nxt[U];
#pragma unroll
    for (int u = 0; u < U; ++u) cur[u] = ld(p_start + u);
    int b = 0, gi = i_s;
    for (int pc = p_start; pc < p_stop; pc += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) nxt[u] = ld(pc + U + u);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (pc + u >= p_stop) break;
            float2 v0, v1;
            unpack(cur[u], v0, v1);
            float2 tb[APP];
#pragma unroll
            for (int s2 = 0; s2 < APP; s2 += 2) {
                const float4 q4 = *reinterpret_cast<const float4 *>(&s_tp[b * APP + s2]);
                tb[s2] = make_float2(q4.x, q4.y);
                tb[s2 + 1] = make_float2(q4.z, q4.w);
            }
#pragma unroll
            for (int s = 0; s < AP; ++s) {
                acc[0][s] = ffma2(tb[s], v0, acc[0][s]);
                acc[1][s] = ffma2(tb[s], v1, acc[1][s]);
            }
            if (++b == a.Dp) {                                // group gi complete: output gi - (AP - 1) finished
                b = 0;
                const int i = gi - (AP - 1);
                if (i >= i_s) {
                    float2 *o = a.out + ((size_t)row * a.Po + i) * a.Ko + j;
                    const float2 o0 = make_float2(acc[0][AP - 1].x * inv, acc[0][AP - 1].y * inv);
                    const float2 o1 = make_float2(acc[1][AP - 1].x * inv, acc[1][AP - 1].y * inv);
                    o[0] = o0;
                    vmax = fmaxf(vmax, fmaxf(fabsf(o0.x), fabsf(o0.y)));
                    if (j + 1 < a.nj) {
                        o[1] = o1;
                        vmax = fmaxf(vmax, fmaxf(fabsf(o1.x), fabsf(o1.y)));
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int s = AP - 1; s > 0; --s) acc[h][s] = acc[h][s - 1];
                    acc[h][0] = make_float2(0.f, 0.f);
                }
                ++gi;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) cur[u] = nxt[u];
    }
    if (a.amax) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        if ((t & 31) == 0 && vmax > 0.f) atomicMax(a.amax, __float_as_int(vmax));
    }
}

template <int AP, bool F32>
cudaError_t launch_fir(FirArgs f, cudaStream_t s)
{
    constexpr int APP = (AP + 3) & ~3;
    const long nb = ((long)f.rows * ((f.nj + 1) / 2) + 127) / 128;
    // segments of output pulses: the count whose waves of blocks (about 8 a multiprocessor) times the pulses a thread
    // sweeps (its outputs' and the AP - 1 of its halo) are fewest (the 512-pixel spotlight's first level: 1 segment 60
    // us, 7 segments 16)
    int nseg = 1;
    double best = 1e30;
    for (int k = 1; k <= 64 && k <= f.Po; ++k) {
        const double w = (double)nb * k / (148.0 * 8), cost = (w < 8 ? std::ceil(w) : w) * ((f.Po + k - 1) / k + AP - 1);
        if (cost < best) { best = cost; nseg = k; }
    }
    f.SEG = (f.Po + nseg - 1) / nseg;
    f.nseg = (f.Po + f.SEG - 1) / f.SEG;
    if (nb > 0x7fffffffL || f.nseg > 65535) return cudaErrorInvalidValue;
    const size_t smem = (size_t)f.Dp * APP * sizeof(float2);
    if (smem > 48 * 1024) {                               // 768 pulses to an output and more, of 8 taps each
        cudaError_t e = cudaFuncSetAttribute(level_fir<AP, F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    level_fir<AP, F32><<<dim3((unsigned)nb, (unsigned)f.nseg), 128, smem, s>>>(f);
    return cudaGetLastError();
}

// The largest |component| of n floats of complex samples, the non-finite ones left out (the level's kernel reports them).
// 16-byte reads from the first 16-byte boundary on: a history is aligned to its samples' 8 bytes (one of a stack of
// odd-sized histories lies between two boundaries).
__global__ void amax_kernel(const float *__restrict__ v, size_t n, int *amax)
{
    float m = 0.f;
    auto take = [&](float a) {
        a = fabsf(a);
        if (a <= FLT_MAX) m = fmaxf(m, a);
    };
    const size_t gid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    const size_t head = ((uintptr_t)v & 15) && n >= 2 ? 2 : 0, n4 = (n - head) / 4;
    const float4 *v4 = reinterpret_cast<const float4 *>(v + head);
    for (size_t i = gid; i < n4; i += step) {
        const float4 q = __ldg(v4 + i);
        const float most = fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w)));   // fmaxf passes NaNs over
        if (most <= FLT_MAX) {
            m = fmaxf(m, most);
        } else {
            take(q.x);
            take(q.y);
            take(q.z);
            take(q.w);
        }
    }
    for (size_t i = head + n4 * 4 + gid; i < n; i += step) take(v[i]);
    if (gid < head) take(v[gid]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(amax, __float_as_int(m));
}

}  // namespace

size_t level_tc_scratch_bytes(int Np, int C, int P, int Ko)
{
    const int Kop = (Ko + 3) & ~3;
    return (size_t)Np * C * P * Kop * sizeof(__half2);
}

// The shapes of the mixed-precision form and its launch options' limits: what a tile of nt columns with sb operand
// stages and pc plane copies took of shared memory in the kernel the options were made for. Which levels run in float16,
// and which option sets are refused, is part of the interface.
static size_t option_smem(int Lkp, int Dk, int nt, int sb, int pc)
{
    const int W = Dk * (nt - 1) + Lkp, Wp = pc == 4 ? (W + 11) & ~3 : (W + 9) & ~1;
    return (size_t)4 * 256 * Lkp + (size_t)sb * 8 * nt * Lkp + (size_t)16 * pc * Wp + (size_t)Lkp * 4 + (size_t)32 * Wp +
           (size_t)(13 + 2 * sb) * 8;
}

constexpr size_t OPTION_SMEM_MAX = 225 * 1024;

bool level_tc_supported(int C, int Lk, int Dk)
{
    const int Lkp = ((Lk + 15) / 16) * 16;
    return C >= 1 && C <= 64 && Lkp <= 96 && Dk >= 1 && option_smem(Lkp, Dk, 32, 2, 2) <= OPTION_SMEM_MAX;
}

// Whether the launch options of a level's first pass (ffbp_tc_opts) are ones it takes; they no longer change its
// schedule.
static bool options_ok(const LevelLaunch &L, int Lkp, const char **why)
{
    const int pc = L.tc_pc == 4 ? 4 : 2, cw = L.tc_cw ? L.tc_cw : 8;
    if (L.tc_pc != 0 && L.tc_pc != 2 && L.tc_pc != 4) { *why = "plane copies: 2 or 4"; return false; }
    if (cw != 4 && cw != 8 && cw != 12) { *why = "consumer warps: 4, 8 or 12"; return false; }
    const int rp = (Lkp > 32 && L.C <= 32 && L.tc_rp != 1) ? 2 : 1, unit = std::max(16, 8 * (cw / 4) * rp);
    auto fits = [&](int nt, int sb) { return option_smem(Lkp, L.Dk, nt, sb, pc) <= OPTION_SMEM_MAX; };
    int nt = L.tc_nt;
    if (nt) {
        if (nt % unit || nt > 128 || !fits(nt, 2)) {
            *why = "columns per tile: a multiple of 16 and of 8 x consumer warps / 4 (x 2 with repeated rows), up to 128, whose operands fit shared memory";
            return false;
        }
    } else {
        const int step = 32 % unit == 0 ? 32 : unit;
        int bestw = 1 << 30;
        for (int n = (128 / step) * step; n >= step; n -= step) {
            if (!fits(n, 2)) continue;
            const int nti = (L.Ko + n - 1) / n, waste = nti * n - L.Ko + nti * 32;
            if (waste < bestw) { bestw = waste; nt = n; }
        }
    }
    if (!nt || nt % unit != 0 || (nt / (cw / 4) / rp) % 8 != 0) {
        *why = "columns per tile do not split into the consumer warps' 8-column chunks";
        return false;
    }
    if (L.tc_sb && (L.tc_sb < 2 || L.tc_sb > 4 || !fits(nt, L.tc_sb))) { *why = "B stages: 2 to 4 that fit shared memory"; return false; }
    return true;
}

cudaError_t launch_amax(const float2 *x, size_t n, int *amax, cudaStream_t s)
{
    amax_kernel<<<148 * 4, 256, 0, s>>>(reinterpret_cast<const float *>(x), 2 * n, amax);
    return cudaGetLastError();
}

cudaError_t launch_level_tc_gemm(const LevelLaunch &L, const int *amax_in, void *scratch, int *err, cudaStream_t s,
                                 const char **why)
{
    *why = nullptr;
    const int Lk = L.Dk > 1 ? L.Lk : 1;
    if (!level_tc_supported(L.C, Lk, L.Dk)) { *why = "the tensor-core level takes C <= 64 children and Lk <= 96 taps"; return cudaErrorNotSupported; }
    if (!options_ok(L, ((Lk + 15) / 16) * 16, why)) return cudaErrorNotSupported;
    return launch_level_mma(L, amax_in, scratch, true, 0, L.Np, 0, L.Ko, err, s, why);
}

template <bool F32>
static cudaError_t run_fir(const FirArgs &f, cudaStream_t s, const char **why)
{
    const int AP = (f.Lp + f.Dp - 1) / f.Dp;
    switch (AP) {
        case 1: return launch_fir<1, F32>(f, s);
        case 2: return launch_fir<2, F32>(f, s);
        case 3: return launch_fir<3, F32>(f, s);
        case 4: return launch_fir<4, F32>(f, s);
        case 5: return launch_fir<5, F32>(f, s);
        case 6: return launch_fir<6, F32>(f, s);
        case 7: return launch_fir<7, F32>(f, s);
        case 8: return launch_fir<8, F32>(f, s);
        case 9: return launch_fir<9, F32>(f, s);
        case 10: return launch_fir<10, F32>(f, s);
        case 11: return launch_fir<11, F32>(f, s);
        case 12: return launch_fir<12, F32>(f, s);
        default: break;
    }
    if (F32 && AP <= 16) return AP <= 14 ? launch_fir<14, true>(f, s) : launch_fir<16, true>(f, s);
    *why = "pulse FIR spans more than 12 output pulses (16 in float32)";
    return cudaErrorNotSupported;
}

static FirArgs fir_args(const LevelLaunch &L, const int *amax_in, const void *scratch)
{
    FirArgs f;
    f.y = scratch; f.tp = L.Dp > 1 ? L.tp : nullptr; f.out = L.out; f.amax = L.amax; f.amax_in = amax_in; f.wexp = L.wexp;
    f.rows = L.Np * L.C; f.P = L.P; f.Kop = (L.Ko + 3) & ~3; f.nj = f.Ko = L.Ko; f.Po = L.Po; f.Dp = L.Dp;
    f.Lp = L.Dp > 1 ? L.Lp : 1; f.plp = L.Dp > 1 ? L.plp : 0;
    return f;
}

cudaError_t launch_level_fir_cc(const LevelLaunch &L, const int *amax_in, const void *scratch, cudaStream_t s,
                                const char **why)
{
    *why = nullptr;
    return run_fir<false>(fir_args(L, amax_in, scratch), s, why);
}

bool level_fir32_supported(int Lp, int Dp)
{
    const int AP = (Lp + Dp - 1) / Dp;
    return AP <= 16 && (size_t)Dp * ((AP + 3) & ~3) * sizeof(float2) <= 227 * 1024;
}

cudaError_t launch_level_fir32(const LevelLaunch &L, const int *amax_in, const void *y, int n0, int nn, int j0, int nj,
                               cudaStream_t s, const char **why)
{
    *why = nullptr;
    FirArgs f = fir_args(L, amax_in, y);
    f.out += (size_t)n0 * L.C * L.Po * L.Ko + j0;
    f.rows = nn * L.C;
    f.nj = nj;
    f.Kop = (nj + 3) & ~3;
    return run_fir<true>(f, s, why);
}

}  // namespace ffbp

namespace ffbp {

cudaError_t launch_level_tc(const LevelLaunch &L, const int *amax_in, void *scratch, int *err, cudaStream_t s,
                            const char **why)
{
    cudaError_t e = launch_level_tc_gemm(L, amax_in, scratch, err, s, why);
    if (e != cudaSuccess || *why) return e;
    return launch_level_tc_fir(L, amax_in, scratch, err, s, why);
}

cudaError_t launch_level_tc_fir(const LevelLaunch &L, const int *amax_in, const void *scratch, int *err,
                                cudaStream_t s, const char **why)
{
    // the pulse FIR on the tensor cores (a banded product per row, level_fir_tc.cu) or on the CUDA cores (level_fir);
    // by default the tensor cores where the output pulse axis fills several 128-row tiles (short axes leave most
    // of a tile's rows and the chunks' pulses empty, where the CUDA-core kernel is faster)
    const int Lp = L.Dp > 1 ? L.Lp : 1;
    const int AP = (Lp + L.Dp - 1) / L.Dp;
    const bool tc = L.tc_fir == 2 || (L.tc_fir == 0 && (L.Po >= 512 || AP > 12));
    if (L.tc_fir != 0 && L.tc_fir != 1 && L.tc_fir != 2) { *why = "pulse FIR kernel: 1 (CUDA cores) or 2 (tensor cores)"; return cudaErrorNotSupported; }
    return tc ? launch_level_fir_tc(L, amax_in, scratch, err, s, why) : launch_level_fir_cc(L, amax_in, scratch, s, why);
}

}  // namespace ffbp
