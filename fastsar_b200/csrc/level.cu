// The fused level kernel: for every parent, each child's phase re-centring (rotation), the pulse-axis decimation
// FIR and the frequency-axis decimation FIR in one pass over the parent's samples.
//
// The reference (fastsar/ffbp_cuda.py:48-256, fastsar/ffbp_cpu.cpp:146-293) rotates and filters along frequency
// first, writes the [children, P, Ko] intermediate, and filters along pulses in a second kernel; at the 16,384-pulse
// x 8,192-sample spotlight that intermediate is 23 GB of the first level alone. The two FIRs act on different axes
// and commute, so this kernel takes the other order: rotation, then the pulse FIR, then the frequency FIR, with the
// pulse FIR held in registers and the frequency FIR applied from shared memory to each finished output row. Nothing
// at the input pulse rate reaches global memory; the output is written once.
//
// Work decomposition. A thread block owns one parent n, G consecutive children, a block of JB output columns
// (whose NK = Dk (JB - 1) + Lk input columns fit the block's NT threads, one column per thread) and a segment of
// output pulses. It sweeps the input pulses of its segment in order. Input pulse p = Dp g + b - plp (group g, phase
// b) feeds outputs i = g - s with tap r = Dp s + b for s < AP = ceil(Lp / Dp): each thread keeps those AP
// accumulators per child in registers, and after each group the oldest is finished, handed to shared memory, and
// the registers shift by one. Consecutive blocks are the child groups of one column block and segment, so the
// parent's rows they all read are served from L2.
//
// Per input sample and child the inner loop is one fused multiply-add for the phase, the hardware sine and cosine,
// a complex multiply and AP complex-by-real multiply-adds. Each thread's column of the input arrives RX rows ahead
// by asynchronous copies into a shared-memory ring that only that thread reads (so no barrier orders them).
//
// Bound: float32 issue. The pulse FIR's multiply-adds are packed (a tap on a sample's two components in one
// instruction), its taps and the frequency taps lie twice in shared memory for that, the children's phases come in
// batches of PHB pulses through shared memory. 12,288 x 8,832 spotlight, first and second level: 24.8 -> 19.0 and
// 47.7 -> 37.5 ms, the same bits.
//
// Arithmetic: float32, the reference's. The rotation phase c0 + sl (k - kc) cycles is evaluated per sample in float32 and
// turned by the hardware sine and cosine, which are accurate to 2^-20.5 absolute over +-100 pi radians. c0 is wrapped to
// +-0.5; the slope term is the child's range offset across half the band, hundreds of cycles at the first level of a wide
// grid, and its rounding (about 1e-7 per cycle) is the error of this kernel there.
#include <cmath>
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"

namespace ffbp {

namespace {

constexpr int RX = 8;         // input rows in flight per thread (its own column, copied asynchronously)

struct LevelArgs {
    const float2 *__restrict__ x;
    const float2 *__restrict__ ph;
    const float *__restrict__ tk;
    const float *__restrict__ tp;
    const float *__restrict__ wp;
    const float *__restrict__ wk;
    float2 *__restrict__ out;
    int *bad;
    int *amax;
    int Np, C, P, K, Ko, Po, Dk, Lk, plk, Dp, Lp, plp;
    int JB, NK, ncb, ngrp, nseg, SEG;
    float kc;
};

constexpr int PHB = 16;       // input pulses per batch of child phases (and pulse weights)

// Dynamic shared memory: the pulse taps by phase b, [Dp][APE] pairs (t, t) with t = tp[Dp s + b] (zero past Lp), and the
// frequency taps as pairs (for the packed multiply-adds); the next RX input rows, one column a thread; two finished
// rows ahead of the frequency FIR; two batches of the children's phases and the pulse weights. Where the pulse taps do not
// fit (more than about 3,000 pulses to an output of 8 taps each: chips of collections of 10^5 pulses) they stay in global
// memory (FAR: the block's threads read the same few each pulse).
template <int AP, int G, int NT, bool FAR>
__host__ __device__ constexpr size_t level_smem(int Dp, int Lk)
{
    return (FAR ? 0 : (size_t)Dp * ((AP + 1) & ~1) * 8) + (size_t)((Lk + 1) & ~1) * 8 + (size_t)RX * NT * 8 + (size_t)2 * G * NT * 8 +
           (size_t)2 * PHB * G * 8 + (size_t)2 * PHB * 4;
}

template <int AP, int G, int NT, bool FAR>
__global__ void __launch_bounds__(NT, AP <= 10 ? 512 / NT : 1) level_kernel(const LevelArgs a)
{
    constexpr int APE = (AP + 1) & ~1;
    extern __shared__ __align__(16) float2 smem[];
    float2 *s_tp = smem;
    float2 *s_tk = s_tp + (FAR ? 0 : a.Dp * APE);
    float2 *s_x = s_tk + ((a.Lk + 1) & ~1);
    float2 *s_z = s_x + RX * NT;
    float2 *s_ph = s_z + 2 * G * NT;                      // [2][PHB][G]
    float *s_wp = reinterpret_cast<float *>(s_ph + 2 * PHB * G);   // [2][PHB]

    int bid = blockIdx.x;
    const int grp = bid % a.ngrp;
    bid /= a.ngrp;
    const int cb = bid % a.ncb;
    bid /= a.ncb;
    const int seg = bid % a.nseg;
    const int n = bid / a.nseg;

    const int t = threadIdx.x;
    const int j0 = cb * a.JB;
    const int k = a.Dk * j0 - a.plk + t;
    const bool colok = (t < a.NK) && (k >= 0) && (k < a.K);
    const float kf = (float)k - a.kc;                     // exact: |k| < 2^24 and kc is a multiple of 1/2

    for (int r = t; !FAR && r < a.Dp * APE; r += NT) {
        const int b = r / APE, s = r - b * APE;
        const int tap = a.Dp * s + b;
        const float v = (s < AP && tap < a.Lp) ? (a.tp ? a.tp[tap] : 1.f) : 0.f;
        s_tp[r] = make_float2(v, v);
    }
    for (int r = t; r < ((a.Lk + 1) & ~1); r += NT) {
        const float v = r < a.Lk ? (a.tk ? a.tk[r] : 1.f) : 0.f;
        s_tk[r] = make_float2(v, v);
    }

    const float wkk = (a.wk && colok) ? a.wk[k] : 1.f;
    const int i_s = seg * a.SEG;
    const int i_e = min(a.Po, i_s + a.SEG);
    const int c0 = grp * G;
    const int nc = min(G, a.C - c0);
    const float2 *__restrict__ phb = a.ph + ((size_t)n * a.C + c0) * a.P;
    const int jbc = min(a.JB, a.Ko - j0);

    float2 acc[G][AP];
#pragma unroll
    for (int c = 0; c < G; ++c)
#pragma unroll
        for (int s = 0; s < AP; ++s) acc[c][s] = make_float2(0.f, 0.f);

    float vmax = 0.f;                                     // the largest |component| this thread writes
    const int g_end = i_e + AP - 1;
    const int p_start = a.Dp * i_s - a.plp;
    const int p_stop = a.Dp * g_end - a.plp;              // rows p_start .. p_stop - 1 are swept
    const int p_last = min(a.P, p_stop);
    // the input ring: row p sits in slot (p - p_start) % RX of this thread's column, copied RX rows ahead
    const float2 *src = a.x + ((ptrdiff_t)n * a.P + p_start) * a.K + k;      // row pr's sample of this column
    int pr = p_start;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(s_x + t);
    auto issue = [&](int slot) {
        const bool ok = pr >= 0 && pr < p_last && colok;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n"
                     :: "r"(ring + (uint32_t)(slot * NT * 8)), "l"(ok ? src : a.x), "r"(ok ? 8 : 0) : "memory");
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        src += a.K;
        ++pr;
    };
#pragma unroll
    for (int r = 0; r < RX; ++r) issue(r);
    // the children's phases in batches of PHB pulses, the next batch's in registers
    float2 qn = make_float2(0.f, 0.f);
    float wn = 1.f;
    int pb = p_start;                                     // the batch in registers
    auto fetch = [&]() {
        if (t < G * PHB) {
            const int pp = pb + t % PHB, c = t / PHB;
            const bool ok = pp >= 0 && pp < a.P;
            qn = (ok && c < nc) ? __ldg(&phb[(size_t)c * a.P + pp]) : make_float2(0.f, 0.f);
            if (a.wp && t < PHB) wn = ok ? __ldg(&a.wp[pp]) : 0.f;
        }
        pb += PHB;
    };
    auto put = [&](int buf) {
        if (t < G * PHB) s_ph[(buf * PHB + t % PHB) * G + t / PHB] = qn;
        if (t < PHB) s_wp[buf * PHB + t] = wn;
    };
    fetch();
    put(0);
    fetch();
    int b = 0, slot = 0, buf = 0, qi = 0;
    __syncthreads();                                      // the taps, the first batch
    int p = p_start;
    for (int g = i_s; g < g_end;) {
        asm volatile("cp.async.wait_group %0;\n" :: "n"(RX - 1) : "memory");
        if (p >= 0 && p < a.P) {                          // the same for every thread of the block
            float2 v = s_x[slot * NT + t];
            if (a.wp) {
                const float w = s_wp[buf * PHB + qi] * wkk;   // the reference's float32 window product
                v.x *= w;
                v.y *= w;
                if (a.bad && colok && !(isfinite(v.x) && isfinite(v.y))) atomicMin(a.bad, p);
            }
            float2 tb[APE];
#pragma unroll
            for (int s2 = 0; s2 < APE; s2 += 2) {
                if (FAR) {
#pragma unroll
                    for (int s = s2; s < s2 + 2; ++s) {
                        const int tap = a.Dp * s + b;
                        const float f = (s < AP && tap < a.Lp) ? (a.tp ? __ldg(a.tp + tap) : 1.f) : 0.f;
                        tb[s] = make_float2(f, f);
                    }
                    continue;
                }
                const float4 q4 = *reinterpret_cast<const float4 *>(&s_tp[b * APE + s2]);
                tb[s2] = make_float2(q4.x, q4.y);
                tb[s2 + 1] = make_float2(q4.z, q4.w);
            }
            const float2 *q = s_ph + (buf * PHB + qi) * G;
#pragma unroll
            for (int c = 0; c < G; ++c) {
                float sn, cs;
                __sincosf(TWO_PI_F * fmaf(q[c].y, kf, q[c].x), &sn, &cs);
                const float2 r = make_float2(fmaf(v.x, cs, -v.y * sn), fmaf(v.x, sn, v.y * cs));
#pragma unroll
                for (int s = 0; s < AP; ++s) acc[c][s] = ffma2(tb[s], r, acc[c][s]);
            }
        }
        issue(slot);                                      // refill the slot just consumed
        slot = (slot + 1 == RX) ? 0 : slot + 1;
        ++p;
        if (++qi == PHB) {                                // the next batch (its buffer's readers are a barrier behind)
            qi = 0;
            buf ^= 1;
            put(buf);
            fetch();
            __syncthreads();
        }
        if (++b == a.Dp) {                                // group g is complete: output g - (AP - 1) is finished
            b = 0;
            const int i = g - (AP - 1);
            if (i >= i_s) {
                float2 *zb = s_z + (i & 1) * (G * NT);
#pragma unroll
                for (int c = 0; c < G; ++c) zb[c * NT + t] = acc[c][AP - 1];
                __syncthreads();
                // the frequency FIR of the finished row: outputs (c, j0 + jj), jj < jbc; even and odd taps apart
                int c = t / jbc, jj = t - c * jbc;
                while (c < nc) {
                    const float2 *zr = zb + c * NT + a.Dk * jj;
                    float2 s0 = make_float2(0.f, 0.f), s1 = s0;
                    int r = 0;
                    for (; r + 1 < a.Lk; r += 2) {
                        const float4 t4 = *reinterpret_cast<const float4 *>(&s_tk[r]);
                        s0 = ffma2(make_float2(t4.x, t4.y), zr[r], s0);
                        s1 = ffma2(make_float2(t4.z, t4.w), zr[r + 1], s1);
                    }
                    if (r < a.Lk) s0 = ffma2(s_tk[r], zr[r], s0);
                    const float2 o = make_float2(s0.x + s1.x, s0.y + s1.y);
                    vmax = fmaxf(vmax, fmaxf(fabsf(o.x), fabsf(o.y)));
                    a.out[(((size_t)n * a.C + c0 + c) * a.Po + i) * a.Ko + j0 + jj] = o;
                    jj += NT;
                    while (jj >= jbc) { jj -= jbc; ++c; }
                }
            }
#pragma unroll
            for (int c = 0; c < G; ++c) {
#pragma unroll
                for (int s = AP - 1; s > 0; --s) acc[c][s] = acc[c][s - 1];
                acc[c][0] = make_float2(0.f, 0.f);
            }
            ++g;
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (a.amax) {                                         // non-negative floats order as their bits
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        if ((t & 31) == 0 && vmax > 0.f) atomicMax(a.amax, __float_as_int(vmax));
    }
}

constexpr size_t LEVEL_SMEM_MAX = 227 * 1024;

template <int AP, int G, int NT, bool FAR = false>
cudaError_t launch_t(LevelArgs a, cudaStream_t s)
{
    a.JB = (a.Dk > 1) ? (NT - a.Lk) / a.Dk + 1 : NT;
    a.NK = a.Dk * (a.JB - 1) + a.Lk;
    a.ncb = (a.Ko + a.JB - 1) / a.JB;
    a.ngrp = (a.C + G - 1) / G;
    // output segments: the count whose waves of blocks times the rows a block sweeps (its outputs and the AP - 1 of its
    // halo) are fewest
    const long base = (long)a.Np * a.ngrp * a.ncb, slots = 148L * (512 / NT);
    int nseg = 1;
    double best = 1e30;
    for (int s2 = 1; s2 <= 64 && s2 <= a.Po; ++s2) {
        const double w = (double)base * s2 / slots, cost = (w < 8 ? ceil(w) : w) * ((a.Po + s2 - 1) / s2 + AP - 1);
        if (cost < best) { best = cost; nseg = s2; }
    }
    a.SEG = (a.Po + nseg - 1) / nseg;
    a.nseg = (a.Po + a.SEG - 1) / a.SEG;
    const long nblocks = base * a.nseg;
    if (nblocks > 0x7fffffffL) return cudaErrorInvalidValue;
    const size_t smem = level_smem<AP, G, NT, FAR>(a.Dp, a.Lk);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(level_kernel<AP, G, NT, FAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    level_kernel<AP, G, NT, FAR><<<(unsigned)nblocks, NT, smem, s>>>(a);
    return cudaGetLastError();
}

template <int G, int NT>
cudaError_t launch_g(const LevelArgs &a, int ap, cudaStream_t s)
{
    const size_t taps = (size_t)a.Dp * ((ap + 1) & ~1) * 8;       // the rest of the shared memory: level_smem
    if (taps + level_smem<1, G, NT, true>(0, a.Lk) > LEVEL_SMEM_MAX)
        return ap <= 8 ? launch_t<8, G, NT, true>(a, s) : launch_t<16, G, NT, true>(a, s);
    switch (ap) {
        case 1: return launch_t<1, G, NT>(a, s);
        case 2: return launch_t<2, G, NT>(a, s);
        case 3: return launch_t<3, G, NT>(a, s);
        case 4: return launch_t<4, G, NT>(a, s);
        case 5: return launch_t<5, G, NT>(a, s);
        case 6: return launch_t<6, G, NT>(a, s);
        case 7: return launch_t<7, G, NT>(a, s);
        case 8: return launch_t<8, G, NT>(a, s);
        case 9: return launch_t<9, G, NT>(a, s);
        case 10: return launch_t<10, G, NT>(a, s);
        case 11: return launch_t<11, G, NT>(a, s);
        case 12: return launch_t<12, G, NT>(a, s);
        case 14: return launch_t<14, G, NT>(a, s);
        default: return launch_t<16, G, NT>(a, s);
    }
}

cudaError_t launch_g8(const LevelArgs &a, int ap, cudaStream_t s)
{
    switch (ap) {
        case 1: return launch_t<1, 8, 256>(a, s);
        case 2: return launch_t<2, 8, 256>(a, s);
        case 3: return launch_t<3, 8, 256>(a, s);
        case 4: return launch_t<4, 8, 256>(a, s);
        case 5: return launch_t<5, 8, 256>(a, s);
        case 6: return launch_t<6, 8, 256>(a, s);
        case 7: return launch_t<7, 8, 256>(a, s);
        case 8: return launch_t<8, 8, 256>(a, s);
        default: return launch_t<9, 8, 256>(a, s);
    }
}

// Whether 512 threads (input columns) per block waste clearly fewer columns on the frequency FIR's halo than 256.
bool wide_blocks(int Dk, int Lk, int Ko)
{
    auto useful = [&](int nt) {
        const int jb = (nt - Lk) / Dk + 1;
        if (jb < 1) return 0.0;
        const int nblk = (Ko + jb - 1) / jb;
        return (double)Ko * Dk / ((double)nblk * nt);
    };
    return useful(512) > 1.08 * useful(256);
}

}  // namespace

cudaError_t launch_level(const LevelLaunch &L, cudaStream_t s, const char **why)
{
    *why = nullptr;
    LevelArgs a;
    a.x = L.x; a.ph = L.phase; a.tk = L.tk; a.tp = L.tp; a.wp = L.wp; a.wk = L.wk; a.out = L.out; a.bad = L.bad;
    a.amax = L.amax;
    a.Np = L.Np; a.C = L.C; a.P = L.P; a.K = L.K; a.Ko = L.Ko; a.Po = L.Po;
    a.Dk = L.Dk; a.Lk = L.Dk > 1 ? L.Lk : 1; a.plk = L.Dk > 1 ? L.plk : 0;
    a.Dp = L.Dp; a.Lp = L.Dp > 1 ? L.Lp : 1; a.plp = L.Dp > 1 ? L.plp : 0;
    a.kc = (float)L.kc;
    const int AP = (a.Lp + a.Dp - 1) / a.Dp;
    int apt = 0;
    const int choices[] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 14, 16};
    for (int c : choices) if (c >= AP) { apt = c; break; }
    if (!apt) { *why = "pulse FIR spans more than 16 output pulses (Lp / Dp > 16)"; return cudaErrorInvalidValue; }
    if (a.Lk > 512) { *why = "frequency FIR longer than a block's columns (Lk > 512)"; return cudaErrorInvalidValue; }
    // 512 threads where a long frequency FIR would leave a 256-thread block little useful width. Blocks of 4
    // children by default; FFBP_LEVEL_G=8 selects 8 (one block per multiprocessor at 230 registers: measured 35%
    // slower on the 16,384-pulse spotlight, kept for other shapes)
    const bool wide = a.Lk > 256 || (a.Dk > 1 && wide_blocks(a.Dk, a.Lk, a.Ko));
    const char *gsel = getenv("FFBP_LEVEL_G");
    const int G = gsel ? atoi(gsel) : 4;
    cudaError_t e;
    if (wide) e = launch_g<4, 512>(a, apt, s);
    else if (G == 8 && (size_t)a.Dp * apt * 8 < 96 * 1024) e = launch_g8(a, apt, s);
    else e = launch_g<4, 256>(a, apt, s);
    if (e == cudaErrorInvalidValue) *why = "too many level blocks";
    return e;
}

}  // namespace ffbp
