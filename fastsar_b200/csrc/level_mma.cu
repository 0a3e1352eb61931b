// The first pass of a tensor-core level (sm_100a): the rotation and the frequency FIR of every child as one product per
// pulse (the reference's rot_fir_k, fastsar/ffbp_cpu.cpp:146-255, fastsar/ffbp_cuda.py:48-193), written at the input
// pulse rate as the intermediate y that the pulse FIR (level_fir, level_fir_tc, level_fir32) reads.
//
// With m_c,p[r] = hk[r] exp(2 pi i sl r) and R_c,p[j] = exp(2 pi i (c0 + sl (Dk j - plk - kc))),
//     y_c[p, j] = R_c,p[j] sum_r m_c,p[r] x[p, Dk j + r - plk],
// a complex product of output columns x taps by taps x children, followed by a ramp. As one real product per pulse and
// tile of columns the accumulator's rows are 128 output columns and its columns the children's real and imaginary parts:
//     D[j, c] = Re, D[j, Ch + c] = Im,   A[j, :] = (re x | im x) of column j's window,
//     B[c, :] = (Re m | -Im m),  B[Ch + c, :] = (Im m | Re m).
//
// The window operand without its Hankel copies. A K-major operand without swizzle is made of 16-byte rows of 8 values,
// rows 16 bytes apart, and a descriptor may start at any row. Samples are laid out as rows Z[m] = x[Dk m .. Dk m + 7]
// (a row per output column step, Dk > 8: G such planes 8 samples apart), each sample stored once: the taps r = Dk a +
// 8 g + e of column j are then Z_g[j + a][e], that is, step a of the product is the same plane one row on. The taps are
// laid out to match, 8 per (a, g) with zeros past Dk. For Dk <= 4, S columns share a row of S Dk <= 8 samples: S planes
// (one per residue of j modulo S) and S accumulators, a third to a half of the steps.
//
// Arithmetic: every operand is split into float16 hi + lo (22 bits) after scaling by powers of two (the samples to
// below 2^8 from the input's largest component, the taps by 2^3), and hi hi + hi lo + lo hi are accumulated in float32:
// the products' error is 2^-22, below that of the float32 sums; with a full row of 8 taps a step is 16 long (8 real, 8
// imaginary parts).
//
// The first level's window lies in shared memory (K floats) where it fits: read through L1, which the operands leave
// little of, its latency bound the sample warps (2,048 x 2,048 float32: 886 -> 524 us).
//
// Measured (B200, first passes of the levels in us, against the kernel that copied the windows into Hankel rows): the
// 12,288 x 8,832 spotlight's mixed form 4,610 / 4,830 / 6,200 (7,570 / 7,210 / 12,890), the 1,499 x 701 patch at T = 16
// 265 / 348 / 439 (840 / 850 / 895), the 512-pixel spotlight 25 / 23 / 38 (221 / 88 / 96). The sine, cosine and stores of
// the read-out and, with few children, the latency of a pulse's chain of roles bound it; the MMAs take a quarter to a half.
//
// Warps: 0..7 read the accumulators (a thread an output column, 8 children at a time), apply the ramp and store; 8..11
// build a pulse's taps; 12..14 stage the tile's samples by cp.async and write the planes; 15 issues the MMAs. Blocks are
// persistent over a contiguous run of (parent, child group, column group, pulse) units; every wait is bounded.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace ffbp {

namespace {

using namespace tc;

constexpr int M_NCW = 8;                     // consumer warps 0..7
constexpr int M_TW0 = 8, M_NTW = 4;          // tap warps
constexpr int M_XW0 = 12, M_NXW = 3;         // sample warps
constexpr int M_MW = 15;                     // MMA issuer
constexpr int M_NTHR = 512;
constexpr int M_PB = 8;                      // pulses per batch of child phases
constexpr int M_PHB = 3;                     // ring of phase batches
constexpr int M_ND = 4;                      // most accumulator buffers
constexpr int M_NBAR = 2 * 4 + 2 * 4 + 2 * M_ND + 2 * M_PHB + 2;   // barriers
constexpr uint64_t M_WAIT_NS = 2000000000ull;
constexpr float M_TAP_SCALE = 8.f;           // the taps' power of two; the samples' is y_scale / M_TAP_SCALE

struct MmaArgs {
    const float2 *__restrict__ x;     // [Np, P, K]
    const float2 *__restrict__ ph;    // [Np, C, P] (c0, sl)
    const float *__restrict__ tk;     // [Lk] or null (Dk == 1)
    const float *__restrict__ wp;     // [P] or null
    const float *__restrict__ wk;     // [K] or null
    int *bad;                         // first non-finite pulse or null
    const int *amax_in;
    void *y;                          // [nn, C, P, Kop] from parent n0, column j0: half2 or float2, times y_scale
    int *err;
    int n0, C, P, K, Dk, Lk, plk;
    int j0, nj, Kop;                  // the first column, the columns and their pitch in y
    int G, A, ks;                     // planes per row of samples, steps a, G A
    int Ch, ncg;                      // children per group (a multiple of 8) and groups
    int TM, ntile, TG, ntg;           // column steps per tile, tiles of TM S columns, tiles per unit, units per row
    int ROWS, W;                      // rows of a plane, staged samples of a tile
    int NT, ZS, XR, nd;               // buffers: taps, planes, staged samples, accumulators
    int wtab;                         // the window's samples in shared memory (K floats)
    int TW;                           // tap warps that build a unit's taps together (4, or 1 a unit each with NT = 4)
    long nunits;
    float kc;
    unsigned test_wait_ns;
};

struct Unit {                         // a unit (parent from n0, child group, column group, pulse) and its successor
    int n, cg, tg, p;
    __device__ __forceinline__ void set(const MmaArgs &a, long u)
    {
        p = (int)(u % a.P);
        u /= a.P;
        tg = (int)(u % a.ntg);
        u /= a.ntg;
        cg = (int)(u % a.ncg);
        n = (int)(u / a.ncg);
    }
    __device__ __forceinline__ void next(const MmaArgs &a)
    {
        if (++p < a.P) return;
        p = 0;
        if (++tg < a.ntg) return;
        tg = 0;
        if (++cg < a.ncg) return;
        cg = 0;
        ++n;
    }
};

// 8 values -> 16 bytes of float16 hi and of float16 lo
__device__ __forceinline__ void split8(const float *v, uint4 &hi, uint4 &lo)
{
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const __half2 x = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
        const float2 f = __half22float2(x);
        const __half2 y = __floats2half2_rn(v[2 * e] - f.x, v[2 * e + 1] - f.y);
        h[e] = *reinterpret_cast<const uint32_t *>(&x);
        l[e] = *reinterpret_cast<const uint32_t *>(&y);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ uint4 negate(uint4 v)
{
    const uint32_t sg = 0x80008000u;
    return make_uint4(v.x ^ sg, v.y ^ sg, v.z ^ sg, v.w ^ sg);
}

// exp(2 pi i u r) to float32's rounding: the step of a recurrence, whose error every following value adds.
__device__ __forceinline__ float2 cis_accurate(float u, float r)
{
    const float m = u * r;
    float s, c;
    sincospif(2.f * ((m - rintf(m)) + fmaf(u, r, -m)), &s, &c);
    return make_float2(c, s);
}

__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}

// GC consecutive columns of this thread's lane (not waited for)
template <int GC>
__device__ __forceinline__ void tmem_ldc(uint32_t addr, float *v)
{
    if constexpr (GC == 8) {
        tmem_ld8(addr, v);
    } else {
        uint32_t r[4];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
    }
}

// Dynamic shared memory: taps [NT][hi, lo][ks][2][N][16 B], planes [ZS][S][G][re hi, im hi, re lo, im lo][ROWS][16 B],
// staged samples [XR][W], the phase batches [PHB][PB][Ch] (float4: c0, sl, the phasor of Dk samples; float2: of one),
// the taps' values [ks][8], the barriers.
__host__ __device__ constexpr size_t mma_tap_bytes(int Ch, int ks) { return (size_t)2 * ks * 2 * (2 * Ch) * 16; }
__host__ __device__ constexpr size_t mma_plane_bytes(int S, int G, int rows) { return (size_t)S * G * 4 * rows * 16; }
// (16 bytes on: the pulse's window weight)
__host__ __device__ constexpr size_t mma_raw_bytes(int W) { return (((size_t)W * 8 + 15) & ~(size_t)15) + 16; }
__host__ __device__ constexpr size_t mma_smem(int S, int G, int rows, int W, int Ch, int ks, int NT, int ZS, int XR,
                                              size_t wtab)
{
    // a product always reads 128 rows from its first: with shorter planes the last one's overrun (at most 96 rows, whose
    // accumulator rows nobody reads) ends inside what follows the planes
    const size_t after = XR * mma_raw_bytes(W) + (size_t)M_PHB * M_PB * Ch * 24 + (size_t)ks * 32 +
                         (size_t)M_NBAR * 8 + wtab;
    return NT * mma_tap_bytes(Ch, ks) + ZS * mma_plane_bytes(S, G, rows) + (after > 96 * 16 ? after : 96 * 16);
}

template <int S, bool HALF, bool WIN, int GC>
__global__ void __launch_bounds__(M_NTHR, 1) level_mma_kernel(const MmaArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int N = 2 * a.Ch, Dks = S * a.Dk;                    // accumulator columns, samples per row
    const uint32_t hipart = (uint32_t)a.ks * 2u * N * 16u, tapbytes = 2u * hipart;
    const uint32_t plane = (uint32_t)a.ROWS * 16u, gbytes = 4u * plane, zbytes = (uint32_t)S * a.G * gbytes;
    unsigned char *sT = smem;
    unsigned char *sZ = sT + (size_t)a.NT * tapbytes;
    unsigned char *sR = sZ + (size_t)a.ZS * zbytes;
    const uint32_t rawbytes = (uint32_t)mma_raw_bytes(a.W);
    float4 *sP = reinterpret_cast<float4 *>(sR + (size_t)a.XR * rawbytes);     // [PHB][PB][Ch]: c0, sl, step
    float2 *sS = reinterpret_cast<float2 *>(sP + (size_t)M_PHB * M_PB * a.Ch); // [PHB][PB][Ch]: a sample's phasor
    float *sH = reinterpret_cast<float *>(sS + (size_t)M_PHB * M_PB * a.Ch);   // [ks][8]
    uint64_t *bars = reinterpret_cast<uint64_t *>(sH + (size_t)a.ks * 8);
    float *sW = reinterpret_cast<float *>(bars + M_NBAR);                       // [K] the window's samples (wtab)
    uint64_t *tfull = bars, *tempty = tfull + 4, *zfull = tempty + 4, *zempty = zfull + 4, *dfull = zempty + 4,
             *dempty = dfull + M_ND, *pfull = dempty + M_ND, *pempty = pfull + M_PHB, *drain = pempty + M_PHB,
             *never = drain + 1;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;

    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const long u0 = a.nunits * (long)blockIdx.x / gridDim.x, u1 = a.nunits * ((long)blockIdx.x + 1) / gridDim.x;
    const int nu = (int)(u1 - u0);

    if (t == 0) {
        s_abort = 0;
        for (int i = 0; i < 4; ++i) { mbar_init(&tfull[i], a.TW); mbar_init(&tempty[i], 1); }
        for (int i = 0; i < 4; ++i) { mbar_init(&zfull[i], M_NXW); mbar_init(&zempty[i], 1); }
        for (int i = 0; i < M_ND; ++i) { mbar_init(&dfull[i], 1); mbar_init(&dempty[i], M_NCW); }
        for (int i = 0; i < M_PHB; ++i) { mbar_init(&pfull[i], M_NTW); mbar_init(&pempty[i], M_NTW + M_NCW); }
        mbar_init(drain, 1);
        mbar_init(never, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the taps' values in the product's order: step (g, a), 8 each, zero past Dks or Lk
    for (int i = t; i < a.ks * 8; i += M_NTHR) {
        const int st = i >> 3, e = i & 7, g = st / a.A, ia = st - g * a.A;
        const int r = Dks * ia + 8 * g + e;
        sH[i] = (8 * g + e < Dks && r < a.Lk) ? (a.tk ? a.tk[r] : 1.f) * M_TAP_SCALE : 0.f;
    }
    if (WIN && a.wtab)
        for (int i = t; i < a.K; i += M_NTHR) sW[i] = a.wk ? a.wk[i] : 1.f;
    if (warp == M_MW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_u32(&s_tmem)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    const bool leader = warp == M_MW && elect_one();           // the one thread that issues (and drains) the MMAs
    if (warp == M_MW) {
        // ------------------------------------------------------------------ MMA issue
        if (leader) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t sT0 = smem_u32(sT), sZ0 = smem_u32(sZ);
            // tests of the failure report: a wait that runs out before any MMA, as a stuck pipeline's would
            const bool stuck = a.test_wait_ns && !mbar_wait(never, 0, 2000, &s_abort, a.err, a.test_wait_ns);
            Unit un;
            un.set(a, u0);
            int ts = 0, zs = 0, d = 0;
            uint32_t tpar = 0, zpar = 0, dpar = 1;
            bool ok = !stuck;
            for (int i = 0; ok && i < nu; ++i, un.next(a)) {
                if (!mbar_wait(&tfull[ts], tpar, 500, &s_abort, a.err, M_WAIT_NS)) break;
                const uint64_t dt = smem_desc(sT0 + (uint32_t)ts * tapbytes, (uint32_t)N * 16u, 128u);
                const int t1 = min(a.ntile, (un.tg + 1) * a.TG);
                for (int tl = un.tg * a.TG; tl < t1; ++tl) {
                    if (!mbar_wait(&zfull[zs], zpar, 500, &s_abort, a.err, M_WAIT_NS) ||
                        !mbar_wait(&dempty[d], dpar, 500, &s_abort, a.err, M_WAIT_NS)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t dz = smem_desc(sZ0 + (uint32_t)zs * zbytes, plane, 128u);
#pragma unroll
                    for (int rho = 0; rho < S; ++rho) {
                        const uint32_t acc = tmem + (uint32_t)(d * S + rho) * N;
                        // the small products first: the accumulator's truncation then weighs on the short chain of hi hi
                        uint32_t on = 0;
#pragma unroll 1
                        for (int part = 0; part < 3; ++part) {       // lo hi, hi lo, hi hi (samples, taps)
                            const uint64_t zo = dz + (uint64_t)(((uint32_t)(rho * a.G) * gbytes + (part == 0 ? 2u * plane : 0u)) >> 4);
                            const uint64_t to = dt + (uint64_t)((part == 1 ? hipart : 0u) >> 4);
                            for (int g = 0; g < a.G; ++g) {
                                const uint64_t zg = zo + (uint64_t)(((uint32_t)g * gbytes) >> 4);
                                const uint64_t tg = to + (uint64_t)(((uint32_t)(g * a.A) * 2u * N * 16u) >> 4);
                                for (int ia = 0; ia < a.A; ++ia) {
                                    mma_bf16(acc, zg + (uint64_t)ia, tg + (uint64_t)((uint32_t)ia * 2u * N), idesc, on);   // kind::f16
                                    on = 1u;
                                }
                            }
                        }
                    }
                    mma_commit(&zempty[zs]);
                    mma_commit(&dfull[d]);
                    if (++zs == a.ZS) { zs = 0; zpar ^= 1u; }
                    if (++d == a.nd) { d = 0; dpar ^= 1u; }
                }
                if (!ok) break;
                mma_commit(&tempty[ts]);
                if (++ts == a.NT) { ts = 0; tpar ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp >= M_XW0) {
        // ------------------------------------------------------------------ samples
        // The three warps step through the tiles together (a named barrier each), also after a failed wait.
        const int xt = t - M_XW0 * 32;
        constexpr int NX = M_NXW * 32;
        const float xs = ([&]() {
            const float m = a.amax_in ? __int_as_float(*a.amax_in) : 0.f;
            if (!(m > 0.f) || !isfinite(m)) return 1.f;
            int ex;
            frexpf(4.f * m, &ex);
            ex = ex < -100 ? -100 : (ex > 100 ? 100 : ex);
            return ldexpf(1.f, 13 - ex);
        })() * (1.f / M_TAP_SCALE);
        Unit un, ld;                                            // the tile converted and the tile staged ahead
        un.set(a, u0);
        ld = un;
        int ui = 0, li = 0, tl = un.tg * a.TG, ltl = tl, lslot = 0, slot = 0, zs = 0;
        uint32_t zpar = 1;
        auto rows_of = [&](int tile) {
            const int c = min(a.TM * S, a.nj - tile * a.TM * S);
            return (c + S - 1) / S + a.A - 1;
        };
        auto stage = [&]() {                                    // the next tile's samples into the ring
            if (li < nu) {
                const int kb = a.Dk * (a.j0 + ltl * a.TM * S) - a.plk, n = Dks * rows_of(ltl) + a.Dk * (S - 1);
                const float2 *row = a.x + ((size_t)(a.n0 + ld.n) * a.P + ld.p) * a.K;
                const uint32_t dst = smem_u32(sR) + (uint32_t)lslot * rawbytes;
                for (int i = xt; i < n; i += NX) {
                    const int k = kb + i;
                    const bool v = k >= 0 && k < a.K;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
                                 :: "r"(dst + 8u * i), "l"(v ? row + k : a.x), "r"(v ? 8 : 0) : "memory");
                }
                if (WIN && xt == 0)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
                                 :: "r"(dst + rawbytes - 16u), "l"(a.wp + ld.p) : "memory");
                if (++lslot == a.XR) lslot = 0;
                if (++ltl == min(a.ntile, (ld.tg + 1) * a.TG)) {
                    ld.next(a);
                    ltl = ld.tg * a.TG;
                    ++li;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int k = 0; k < a.XR - 1; ++k) stage();
        bool live = true;
        while (ui < nu) {
            if (a.XR == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("bar.sync 2, %0;" :: "n"(NX) : "memory");  // this tile staged, the previous one's slot free
            stage();
            if (live) live = mbar_wait(&zempty[zs], zpar, 500, &s_abort, a.err, M_WAIT_NS);
            if (live) {
                const float2 *raw = reinterpret_cast<const float2 *>(sR + (size_t)slot * rawbytes);
                unsigned char *zb = sZ + (size_t)zs * zbytes;
                const int rows = rows_of(tl), items = rows * a.G * S;
                const int kb = a.Dk * (a.j0 + tl * a.TM * S) - a.plk;
                const float wpp = WIN ? *reinterpret_cast<const float *>(sR + (size_t)slot * rawbytes + rawbytes - 16) : 1.f;
                uint32_t worst = 0;
                int m = xt, gr = 0;
                while (m >= rows) { m -= rows; ++gr; }
                for (int it = xt; it < items; it += NX) {
                    const int rho = gr / a.G, g = gr - rho * a.G, ev = min(8, Dks - 8 * g);
                    const int o = Dks * m + a.Dk * rho + 8 * g;
                    float re[8], im[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        float2 v = make_float2(0.f, 0.f);
                        if (e < ev) {
                            v = raw[o + e];
                            if (WIN) {
                                const int k = min(max(kb + o + e, 0), a.K - 1);
                                const float w = wpp * (a.wtab ? sW[k] : a.wk ? __ldg(&a.wk[k]) : 1.f);   // the reference's float32 window product
                                v.x *= w;
                                v.y *= w;
                            }
                            if (a.bad) worst = max(worst, max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu));
                        }
                        re[e] = v.x * xs;
                        im[e] = v.y * xs;
                    }
                    unsigned char *z = zb + (size_t)gr * gbytes + (size_t)m * 16;
                    uint4 h, l;
                    split8(re, h, l);
                    *reinterpret_cast<uint4 *>(z) = h;
                    *reinterpret_cast<uint4 *>(z + 2 * plane) = l;
                    split8(im, h, l);
                    *reinterpret_cast<uint4 *>(z + plane) = h;
                    *reinterpret_cast<uint4 *>(z + 3 * plane) = l;
                    m += NX;
                    while (m >= rows) { m -= rows; ++gr; }
                }
                if (a.bad && worst >= 0x7f800000u) atomicMin(a.bad, un.p);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&zfull[zs]);
            }
            if (++zs == a.ZS) { zs = 0; zpar ^= 1u; }
            if (++slot == a.XR) slot = 0;
            if (++tl == min(a.ntile, (un.tg + 1) * a.TG)) {
                un.next(a);
                tl = un.tg * a.TG;
                ++ui;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp >= M_TW0) {
        // ------------------------------------------------------------------ taps
        const int tt = t - M_TW0 * 32;
        constexpr int NTT = M_NTW * 32;
        const int nph = a.Ch * M_PB;                            // at most 4 per thread (Ch <= 64)
        // a batch is a run of up to PB units of one (parent, child group, column group) within an aligned group of PB
        // pulses; the next batch's phases are in registers while one is used
        Unit un, nb;
        un.set(a, u0);
        nb = un;
        int nbi = 0;                                            // the unit the batch in registers starts at
        float2 reg[4];
        auto fetch = [&]() {
            if (nbi >= nu) return;
            const int pb = nb.p & ~(M_PB - 1), c0 = nb.cg * a.Ch;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = tt + q * NTT, pp = pb + (e & (M_PB - 1)), c = e / M_PB;
                reg[q] = make_float2(0.f, 0.f);
                if (e < nph && pp < a.P && c0 + c < a.C)
                    reg[q] = __ldg(&a.ph[((size_t)(a.n0 + nb.n) * a.C + c0 + c) * a.P + pp]);
            }
        };
        auto skip = [&]() {                                     // to the batch after the one in registers
            const int len = min(min(M_PB - (nb.p & (M_PB - 1)), a.P - nb.p), nu - nbi);
            nbi += len;
            nb.p += len - 1;
            nb.next(a);
        };
        auto put = [&](int slot) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = tt + q * NTT;
                if (e < nph) {
                    const size_t at = ((size_t)slot * M_PB + (e & (M_PB - 1))) * a.Ch + e / M_PB;
                    const float2 st = cis_accurate(reg[q].y, (float)a.Dk);
                    sP[at] = make_float4(reg[q].x, reg[q].y, st.x, st.y);
                    sS[at] = cis_accurate(reg[q].y, 1.f);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&pfull[slot]);
        };
        // the first batch
        fetch();
        put(0);
        skip();
        fetch();
        int b = -1, bslot = 0;
        uint32_t bpar = 0;
        int pslot = 1;                                          // the ring slot of the batch in registers
        uint32_t ppar = 1;
        // a unit's taps by the four warps together, or (few of them) by one warp, the warps taking the units in turn
        int ts = 0;
        uint32_t tpar = 1;
        const int nth = a.TW * 32, th = a.TW == 1 ? lane : tt, dc = nth % a.Ch, dk = nth / a.Ch;
        bool ok = true;
        for (int i = 0; ok && i < nu; ++i, un.next(a)) {
            if (i == 0 || (un.p & (M_PB - 1)) == 0) {           // a new batch
                if (++b > 0) {
                    if (lane == 0) mbar_arrive(&pempty[bslot]);
                    if (++bslot == M_PHB) { bslot = 0; bpar ^= 1u; }
                }
                if (nbi < nu) {                                 // the next batch into its slot, the one after it fetched
                    if (!mbar_wait(&pempty[pslot], ppar, 500, &s_abort, a.err, M_WAIT_NS)) break;
                    put(pslot);
                    if (++pslot == M_PHB) { pslot = 0; ppar ^= 1u; }
                    skip();
                    fetch();
                }
                if (!mbar_wait(&pfull[bslot], bpar, 200, &s_abort, a.err, M_WAIT_NS)) break;
            }
            if (a.TW == 1 && ts != warp - M_TW0) {              // another warp's unit (NT = 4: ts is its warp)
                if (++ts == a.NT) { ts = 0; tpar ^= 1u; }
                continue;
            }
            if (!mbar_wait(&tempty[ts], tpar, 500, &s_abort, a.err, M_WAIT_NS)) break;
            const float4 *pr = sP + ((size_t)bslot * M_PB + (un.p & (M_PB - 1))) * a.Ch;
            const float2 *ps = sS + ((size_t)bslot * M_PB + (un.p & (M_PB - 1))) * a.Ch;
            unsigned char *tb = sT + (size_t)ts * tapbytes;
            int c = th % a.Ch, st = th / a.Ch;
            while (st < a.ks) {
                const int g = st / a.A, ia = st - g * a.A, ev = min(8, Dks - 8 * g);
                const float sl = pr[c].y;
                const float4 h0 = *reinterpret_cast<const float4 *>(sH + 8 * st), h1 = *reinterpret_cast<const float4 *>(sH + 8 * st + 4);
                const float hv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                const float r0 = (float)(Dks * ia + 8 * g), m = sl * r0;
                float2 w = cis_cycles((m - rintf(m)) + fmaf(sl, r0, -m));
                const float2 step = ps[c];
                float mr[8], mi[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (e < ev) {
                        mr[e] = hv[e] * w.x;
                        mi[e] = hv[e] * w.y;
                        w = cmul(w, step);
                    } else {
                        mr[e] = mi[e] = 0.f;
                    }
                }
                uint4 rh, rl, ih, il;
                split8(mr, rh, rl);
                split8(mi, ih, il);
                // chunk 0 (real samples) and chunk 1 (imaginary) of rows c (the child's real part) and Ch + c
                unsigned char *o = tb + ((size_t)st * 2 * N + c) * 16;
                *reinterpret_cast<uint4 *>(o) = rh;
                *reinterpret_cast<uint4 *>(o + (size_t)a.Ch * 16) = ih;
                *reinterpret_cast<uint4 *>(o + (size_t)N * 16) = negate(ih);
                *reinterpret_cast<uint4 *>(o + (size_t)(N + a.Ch) * 16) = rh;
                o += hipart;
                *reinterpret_cast<uint4 *>(o) = rl;
                *reinterpret_cast<uint4 *>(o + (size_t)a.Ch * 16) = il;
                *reinterpret_cast<uint4 *>(o + (size_t)N * 16) = negate(il);
                *reinterpret_cast<uint4 *>(o + (size_t)(N + a.Ch) * 16) = rl;
                c += dc;
                st += dk;
                if (c >= a.Ch) { c -= a.Ch; ++st; }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tfull[ts]);
            if (++ts == a.NT) { ts = 0; tpar ^= 1u; }
        }
    } else {
        // ------------------------------------------------------------------ consumers
        // Warp w: accumulator lanes 32 (w % 4) .. + 31 (an output column step each), the groups of GC children of
        // parity w / 4 (4 where there are few). A thread's S columns S j' .. S j' + S - 1 are adjacent.
        constexpr int SP = S < 2 ? 1 : 2;                       // columns read together
        const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
        Unit un;
        un.set(a, u0);
        int b = -1, bslot = 0, d = 0;
        uint32_t bpar = 0, dpar = 0;
        const size_t cstride = (size_t)a.P * a.Kop;
        bool ok = true;
        for (int i = 0; ok && i < nu; ++i, un.next(a)) {
            if (i == 0 || (un.p & (M_PB - 1)) == 0) {
                if (++b > 0) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&pempty[bslot]);
                    if (++bslot == M_PHB) { bslot = 0; bpar ^= 1u; }
                }
                ok = mbar_wait(&pfull[bslot], bpar, 500, &s_abort, a.err, M_WAIT_NS);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            const float4 *pr = sP + ((size_t)bslot * M_PB + (un.p & (M_PB - 1))) * a.Ch;
            const int nc = min(a.Ch, a.C - un.cg * a.Ch);
            const int t1 = min(a.ntile, (un.tg + 1) * a.TG);
            for (int tl = un.tg * a.TG; tl < t1; ++tl) {
                ok = mbar_wait(&dfull[d], dpar, 500, &s_abort, a.err, M_WAIT_NS);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int jp = 32 * (warp & 3) + lane, j = S * (a.TM * tl + jp);
                const bool in = jp < a.TM && j < a.nj, any = __any_sync(0xffffffffu, in);
                const float uf = (float)(a.Dk * (a.j0 + j) - a.plk) - a.kc;
                const uint32_t base = tmem + lanes + (uint32_t)(d * S) * N;
                const size_t yo = (((size_t)un.n * a.C + un.cg * a.Ch) * a.P + un.p) * a.Kop + j;
                if (any) {
                    for (int cb = GC * (warp >> 2); cb < nc; cb += 2 * GC) {
#pragma unroll
                        for (int r0 = 0; r0 < S; r0 += SP) {
                            float re[SP][GC], im[SP][GC];
#pragma unroll
                            for (int r = 0; r < SP; ++r) {
                                tmem_ldc<GC>(base + (uint32_t)((r0 + r) * N + cb), re[r]);
                                tmem_ldc<GC>(base + (uint32_t)((r0 + r) * N + a.Ch + cb), im[r]);
                            }
                            tmem_wait_ld();
                            // the ramps of the children side by side (no branch between them: the chain phase ->
                            // sine and cosine -> product is long), children past nc computed and not stored
                            const float u = uf + (float)(r0 * a.Dk);
                            float2 e[GC];
#pragma unroll
                            for (int c = 0; c < GC; ++c) {
                                const float2 q = *reinterpret_cast<const float2 *>(&pr[cb + c]);
                                // in float32 with the product's rounding error carried along (hundreds of cycles leave
                                // few bits for the fraction), which float16 does not need
                                float f = fmaf(q.y, u, q.x);
                                if (!HALF) {
                                    const float m = q.y * u;
                                    f = (m - rintf(m)) + (fmaf(q.y, u, -m) + q.x);
                                }
                                e[c] = cis_cycles(f);
                            }
#pragma unroll
                            for (int r = 0; r < SP; ++r)
#pragma unroll
                                for (int c = 0; c < GC; ++c) {
                                    const float2 o = cmul(make_float2(re[r][c], im[r][c]), e[c]);
                                    re[r][c] = o.x;
                                    im[r][c] = o.y;
                                    if (r + 1 < SP) e[c] = cmul(e[c], *reinterpret_cast<const float2 *>(&pr[cb + c].z));
                                }
                            if (in) {
                                const size_t at = yo + (size_t)cb * cstride + r0;
                                if (HALF) {
                                    __half2 *yp = static_cast<__half2 *>(a.y) + at;
#pragma unroll
                                    for (int c = 0; c < GC; ++c) {
                                        const __half2 v0 = __floats2half2_rn(re[0][c], im[0][c]), v1 = __floats2half2_rn(re[SP - 1][c], im[SP - 1][c]);
                                        if (cb + c < nc) {
                                            if (SP == 1) *yp = v0;
                                            else *reinterpret_cast<uint2 *>(yp) = make_uint2(*reinterpret_cast<const uint32_t *>(&v0),
                                                                                            *reinterpret_cast<const uint32_t *>(&v1));
                                        }
                                        yp += cstride;
                                    }
                                } else {
                                    float2 *yp = static_cast<float2 *>(a.y) + at;
#pragma unroll
                                    for (int c = 0; c < GC; ++c) {
                                        if (cb + c < nc) {
                                            if (SP == 1) *yp = make_float2(re[0][c], im[0][c]);
                                            else *reinterpret_cast<float4 *>(yp) = make_float4(re[0][c], im[0][c], re[SP - 1][c], im[SP - 1][c]);
                                        }
                                        yp += cstride;
                                    }
                                }
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&dempty[d]);
                if (++d == a.nd) { d = 0; dpar ^= 1u; }
            }
        }
    }

    __syncthreads();
    if (warp == M_MW) {
        if (leader) {
            // drain: completes once every earlier MMA of the issuer has
            mma_commit(drain);
            const uint64_t t0 = global_ns();
            bool drained = false;
            while (!(drained = mbar_test(drain, 0, 0)) && global_ns() - t0 < M_WAIT_NS) {
            }
            if (!drained && a.err) atomicAdd(a.err, 1);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem));
    }
}

constexpr size_t MMA_SMEM_MAX = 226 * 1024;                  // the opt-in limit less the static shared memory

constexpr int TW1_ITEMS = 128;                               // most taps (8 each) of a unit built by one warp

struct MmaShape { int S, TM, G, A, ks, Ch, ROWS, W, NT, ZS, XR; size_t smem; };

// The shape of a level's product: the residues S and the column steps per tile TM (fewer than 128 only where long
// filters at large decimations leave no room) that need the fewest MMA cycles for the row's tiles, and the most children
// per group whose operands fit with two tap buffers (one where that doubles the group).
bool mma_shape(int C, int Lk, int Dk, int nj, size_t wtab, MmaShape *out)
{
    long best = 0;
    for (int TM = 128; TM >= 32 && !best; TM /= 2)
        for (int S = 1; S <= 4; S *= 2) {
            if (S > 1 && S * Dk > 8) break;
            MmaShape s;
            s.S = S;
            s.TM = TM;
            const int Dks = S * Dk;
            s.G = (Dks + 7) / 8;
            s.A = (Lk + Dks - 1) / Dks;
            s.ks = s.G * s.A;
            s.ROWS = TM + s.A - 1;
            s.W = Dks * s.ROWS + Dk * (S - 1);
            const int cmax = std::min((C + 7) & ~7, S == 4 ? 32 : 64);
            // buffers (taps, planes, staged samples): four tap buffers where one warp builds a unit's taps
            const int opt[5][3] = {{4, 3, 3}, {2, 2, 3}, {2, 2, 2}, {1, 2, 2}, {1, 1, 2}};
            s.Ch = 0;
            int groups = 1 << 30;
            for (const auto &o : opt) {
                int ch = cmax;
                if (o[0] == 4 && s.ks * std::min(cmax, (C + 7) & ~7) > TW1_ITEMS) continue;
                while (ch >= 8 && mma_smem(S, s.G, s.ROWS, s.W, ch, s.ks, o[0], o[1], o[2], wtab) > MMA_SMEM_MAX) ch -= 8;
                if (ch < 8) continue;
                const int g = (C + ch - 1) / ch;
                if (g * 2 > groups) continue;                // fewer buffers only for half the groups
                groups = g;
                s.NT = o[0]; s.ZS = o[1]; s.XR = o[2];
                s.Ch = (((C + g - 1) / g) + 7) & ~7;
                s.smem = mma_smem(S, s.G, s.ROWS, s.W, s.Ch, s.ks, s.NT, s.ZS, s.XR, wtab);
            }
            if (!s.Ch) continue;
            const int ntile = (nj + TM * S - 1) / (TM * S);
            const int cyc = std::max(32 + s.Ch / 2, s.Ch);   // measured cycles of an MMA of N = 2 Ch
            const long cost = (long)groups * ntile * S * s.ks * 3 * cyc;
            if (!best || cost < best) {
                best = cost;
                *out = s;
            }
        }
    return best != 0;
}

}  // namespace

bool level_mma_supported(int C, int Lk, int Dk, int Ko)
{
    MmaShape s;
    return C >= 1 && Dk >= 1 && Lk >= 1 && Lk <= 512 && mma_shape(C, Lk, Dk, Ko, 0, &s);
}

cudaError_t launch_level_mma(const LevelLaunch &L, const int *amax_in, void *y, bool half, int n0, int nn, int j0,
                             int nj, int *err, cudaStream_t s, const char **why)
{
    *why = nullptr;
    const int Lk = L.Dk > 1 ? L.Lk : 1, plk = L.Dk > 1 ? L.plk : 0;
    MmaShape m;
    // the first level's window over the samples in shared memory, where that costs no children per group
    const size_t wtab = L.wp ? ((size_t)L.K * 4 + 15) & ~(size_t)15 : 0;
    MmaShape m0;
    const bool tab = wtab && mma_shape(L.C, Lk, L.Dk, nj, wtab, &m) && mma_shape(L.C, Lk, L.Dk, nj, 0, &m0) && m.Ch == m0.Ch;
    if (!tab && !mma_shape(L.C, Lk, L.Dk, nj, 0, &m)) { *why = "the level's operands do not fit shared memory"; return cudaErrorNotSupported; }
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    MmaArgs a;
    a.x = L.x; a.ph = L.phase; a.tk = L.Dk > 1 ? L.tk : nullptr; a.wp = L.wp; a.wk = L.wk; a.bad = L.bad;
    a.amax_in = amax_in; a.y = y; a.err = err; a.wtab = tab; a.n0 = n0; a.C = L.C; a.P = L.P; a.K = L.K; a.Dk = L.Dk; a.Lk = Lk;
    a.plk = plk; a.j0 = j0; a.nj = nj; a.Kop = (nj + 3) & ~3; a.G = m.G; a.A = m.A; a.ks = m.ks; a.Ch = m.Ch;
    a.ncg = (L.C + m.Ch - 1) / m.Ch; a.TM = m.TM; a.ntile = (nj + m.TM * m.S - 1) / (m.TM * m.S);
    a.ROWS = m.ROWS; a.W = m.W; a.NT = m.NT; a.ZS = m.ZS; a.XR = m.XR; a.TW = m.NT == 4 ? 1 : M_NTW;
    a.nd = std::min(M_ND, 512 / (m.S * 2 * m.Ch));
    a.kc = (float)L.kc; a.test_wait_ns = L.test_wait_ns;
    // tiles per unit: all of the row's share a pulse's taps, unless that leaves too few units for the device
    a.TG = a.ntile;
    while (a.TG > 1 && (long)nn * a.ncg * ((a.ntile + a.TG - 1) / a.TG) * L.P < 8L * nsm) a.TG = (a.TG + 1) / 2;
    a.ntg = (a.ntile + a.TG - 1) / a.TG;
    a.nunits = (long)nn * a.ncg * a.ntg * L.P;
    if (a.nunits <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)std::min<long>(a.nunits, nsm);
    if (a.nunits / grid >= (1L << 30)) { *why = "too many pulses for one launch"; return cudaErrorNotSupported; }
    auto run = [&](auto kern) -> cudaError_t {
        cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m.smem);
        if (r != cudaSuccess) return r;
        kern<<<grid, M_NTHR, m.smem, s>>>(a);
        return cudaGetLastError();
    };
    const bool win = L.wp != nullptr;
#define FFBP_MMA_RUN2(SV, GV)                                                                               \
    (half ? (win ? run(level_mma_kernel<SV, true, true, GV>) : run(level_mma_kernel<SV, true, false, GV>))   \
          : (win ? run(level_mma_kernel<SV, false, true, GV>) : run(level_mma_kernel<SV, false, false, GV>)))
#define FFBP_MMA_RUN(SV) (m.Ch <= 16 ? FFBP_MMA_RUN2(SV, 4) : FFBP_MMA_RUN2(SV, 8))
    return m.S == 4 ? FFBP_MMA_RUN(4) : m.S == 2 ? FFBP_MMA_RUN(2) : FFBP_MMA_RUN(1);
#undef FFBP_MMA_RUN2
#undef FFBP_MMA_RUN
}

}  // namespace ffbp
