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
// Where a row has one or two samples past a multiple of 8 (Dk = 9, 10, 17, ...), a plane of their own would be mostly
// zeros: such a sample's plane gathers it from 8 rows instead (one step for 8 values of a).
//
// Arithmetic: every operand is split into float16 hi + lo (22 bits) after scaling by powers of two (the samples to
// below 2^8 from the input's largest component, the taps by 2^3), and hi hi + hi lo + lo hi are accumulated in float32:
// the products' error is 2^-22, below that of the float32 sums; with a full row of 8 taps a step is 16 long (8 real, 8
// imaginary parts).
//
// Measured (B200, first passes of the levels in us, against the kernel that copied the windows into Hankel rows): the
// 12,288 x 8,832 spotlight's mixed form 3,760 / 3,690 / 6,400 (7,570 / 7,210 / 12,890), the 1,499 x 701 patch at T = 16
// 219 / 371 / 401 (840 / 850 / 895), the 512-pixel spotlight 25 / 24 / 28 (221 / 88 / 96). The sine, cosine and stores of
// the read-out and, with few children, the latency of a pulse's chain of roles bound it; the MMAs take a quarter to a half.
//
// Warps: 0..7 read the accumulators (a thread an output column, 8 children at a time), apply the ramp and store; 8..14
// build a pulse's taps (3 or 4 of them, as the work divides: mma_shape) and stage the tile's samples by cp.async and write
// the planes; 15 issues the MMAs. Blocks are
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
constexpr int M_TW0 = 8, M_NAUX = 7;         // 3 or 4 tap warps, the others of these for the samples (MmaArgs::ntw)
constexpr int M_MW = 15;                     // MMA issuer
constexpr int M_NTHR = 512;
constexpr int M_PB = 8;                      // pulses per batch of child phases
constexpr int M_PHB = 3;                     // ring of phase batches
constexpr int M_ND = 4;                      // most accumulator buffers
constexpr int M_NBAR = 2 * 4 + 2 * 4 + 2 * M_ND + 2 * M_PHB + 2;   // barriers
constexpr uint64_t M_WAIT_NS = 2000000000ull;
constexpr float M_TAP_SCALE = 8.f;           // the taps' power of two; the samples' is 2^level_exponent / M_TAP_SCALE

struct MmaArgs {
    const float2 *__restrict__ x;     // [Np, P, K]
    const float2 *__restrict__ ph;    // [Np, C, P] (c0, sl)
    const float *__restrict__ tk;     // [Lk] or null (Dk == 1)
    const float *__restrict__ wp;     // [P] or null
    const float *__restrict__ wk;     // [K] or null
    int *bad;                         // first non-finite pulse or null
    const int *amax_in;
    void *y;                          // [nn, C, P, Kop] from parent n0, column j0: half2 or float2, times 2^level_exponent
    int *err;
    int n0, C, P, K, Dk, Lk, plk;
    int j0, nj, Kop;                  // the first column, the columns and their pitch in y
    int G, A, ks;                     // planes per row of samples, steps a, steps in all
    int Gf, A8;                       // planes of 8 neighbouring samples (the others gather 8 rows' samples), ceil(A / 8)
    int Ch, ncg;                      // children per group (a multiple of 8) and groups
    int PP, RP, PG, Chv;              // pulses per unit, each on RP of a plane's rows; units along the pulses; PP Ch
    int TM, ntile, TG, ntg;           // column steps per tile, tiles of TM S columns, tiles per unit, units per row
    int ROWS, W;                      // rows of a plane, staged samples of a tile
    int NT, ZS, XR, nd;               // buffers: taps, planes, staged samples, accumulators
    int wtab;                         // the window's samples in shared memory (K floats)
    int ntw, TW;                      // tap warps; those that build a unit's taps together (all, or 1 a unit each, NT = ntw)
    long nunits;
    float kc;
    unsigned test_wait_ns;
    int wexp;                         // the window's power of two (LevelLaunch::wexp)
};

struct Unit {                         // a unit (parent from n0, child group, column group, PP pulses) and its successor
    int n, cg, tg, p;                 // p: the unit along the pulses, pulses PP p .. PP p + PP - 1
    __device__ __forceinline__ void set(const MmaArgs &a, long u)
    {
        p = (int)(u % a.PG);
        u /= a.PG;
        tg = (int)(u % a.ntg);
        u /= a.ntg;
        cg = (int)(u % a.ncg);
        n = (int)(u / a.ncg);
    }
    __device__ __forceinline__ void next(const MmaArgs &a)
    {
        if (++p < a.PG) return;
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

// Bits 15 and 31 set where one of 8 float16 values is not finite (its exponent all ones carries into the sign's place): a
// finite sample is scaled below 2^8, its product with the window below 2^10 (LevelLaunch::wexp), finite in float16.
__device__ __forceinline__ uint32_t non_finite(uint4 v)
{
    auto c = [](uint32_t x) { return (x & 0x7c007c00u) + 0x04000400u; };
    return c(v.x) | c(v.y) | c(v.z) | c(v.w);
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
__host__ __device__ constexpr size_t mma_smem(int S, int G, int rows, int W, int Ch, int PP, int ks, int NT, int ZS, int XR,
                                              size_t wtab)
{
    // a product always reads 128 rows from its first: with shorter planes the last one's overrun (at most 96 rows, whose
    // accumulator rows nobody reads) ends inside what follows the planes
    const size_t after = XR * mma_raw_bytes(W) + (size_t)M_PHB * M_PB * Ch * 24 + (size_t)ks * 32 +
                         (size_t)M_NBAR * 8 + wtab;
    return NT * mma_tap_bytes(PP * Ch, ks) + ZS * mma_plane_bytes(S, G, rows) + (after > 96 * 16 ? after : 96 * 16);
}

template <int S, bool HALF, bool WIN, int GC, bool GA>
__global__ void __launch_bounds__(M_NTHR, 1) level_mma_kernel(const MmaArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int N = 2 * a.Chv, Dks = S * a.Dk;                   // accumulator columns, samples per row
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
    const int PBG = M_PB / a.PP;                               // units per batch of child phases

    if (t == 0) {
        s_abort = 0;
        for (int i = 0; i < 4; ++i) { mbar_init(&tfull[i], a.TW); mbar_init(&tempty[i], 1); }
        for (int i = 0; i < 4; ++i) { mbar_init(&zfull[i], M_NAUX - a.ntw); mbar_init(&zempty[i], 1); }
        for (int i = 0; i < M_ND; ++i) { mbar_init(&dfull[i], 1); mbar_init(&dempty[i], M_NCW); }
        for (int i = 0; i < M_PHB; ++i) { mbar_init(&pfull[i], a.ntw); mbar_init(&pempty[i], a.ntw + M_NCW); }
        mbar_init(drain, 1);
        mbar_init(never, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the taps' values in the product's order: step (g, a), 8 each, zero past Dks or Lk
    for (int i = t; i < a.ks * 8; i += M_NTHR) {
        const int st = i >> 3, e = i & 7, gs = st - a.Gf * a.A;
        const int g = GA && gs >= 0 ? a.Gf : st / a.A, ia = st - g * a.A;
        const int r = GA && gs >= 0 ? Dks * (8 * (gs % a.A8) + e) + 8 * a.Gf + gs / a.A8 : Dks * ia + 8 * g + e;
        const bool in = (GA || 8 * g + e < Dks) && r < a.Lk;
        sH[i] = in ? (a.tk ? a.tk[r] : 1.f) * M_TAP_SCALE : 0.f;
    }
    // the samples' power of two, which the window's table carries too (exact)
    const float xs = ldexpf(1.f / M_TAP_SCALE, level_exponent(a.amax_in, WIN ? a.wexp : 0));
    if (WIN && a.wtab)
        for (int i = t; i < a.K; i += M_NTHR) sW[i] = (a.wk ? a.wk[i] : 1.f) * xs;
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
                            for (int g = 0; g < a.Gf; ++g) {
                                const uint64_t zg = zo + (uint64_t)(((uint32_t)g * gbytes) >> 4);
                                const uint64_t tg = to + (uint64_t)(((uint32_t)(g * a.A) * 2u * N * 16u) >> 4);
                                for (int ia = 0; ia < a.A; ++ia) {
                                    mma_bf16(acc, zg + (uint64_t)ia, tg + (uint64_t)((uint32_t)ia * 2u * N), idesc, on);   // kind::f16
                                    on = 1u;
                                }
                            }
                            if (GA) {                                // the gathered planes: a step covers 8 rows
                                uint64_t tg = to + (uint64_t)((uint32_t)(a.Gf * a.A) * 2u * N);
                                for (int g = a.Gf; g < a.G; ++g)
                                    for (int u = 0; u < a.A8; ++u) {
                                        mma_bf16(acc, zo + (uint64_t)(((uint32_t)g * gbytes) >> 4) + (uint64_t)(8 * u), tg, idesc, on);
                                        tg += (uint64_t)(2u * N);
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
    } else if (warp >= M_TW0 + a.ntw) {
        // ------------------------------------------------------------------ samples
        // The warps step through the tiles together (a named barrier each), also after a failed wait.
        const int xt = t - (M_TW0 + a.ntw) * 32, NX = (M_NAUX - a.ntw) * 32;
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
                const uint32_t dst = smem_u32(sR) + (uint32_t)lslot * rawbytes;
                for (int q = 0; q < a.PP; ++q) {
                    const int p = ld.p * a.PP + q;
                    const float2 *row = a.x + ((size_t)(a.n0 + ld.n) * a.P + p) * a.K;
                    for (int i = xt; i < n; i += NX) {
                        const int k = kb + i;
                        const bool v = k >= 0 && k < a.K && p < a.P;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
                                     :: "r"(dst + 8u * (q * n + i)), "l"(v ? row + k : a.x), "r"(v ? 8 : 0) : "memory");
                    }
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
            asm volatile("bar.sync 2, %0;" :: "r"(NX) : "memory");  // this tile staged, the previous one's slot free
            stage();
            if (live) live = mbar_wait(&zempty[zs], zpar, 500, &s_abort, a.err, M_WAIT_NS);
            if (live) {
                const float2 *raw = reinterpret_cast<const float2 *>(sR + (size_t)slot * rawbytes);
                unsigned char *zb = sZ + (size_t)zs * zbytes;
                const int rows = rows_of(tl), items = rows * a.G * S * a.PP, nq = Dks * rows + a.Dk * (S - 1);
                const int kb = a.Dk * (a.j0 + tl * a.TM * S) - a.plk;
                const float wpp = WIN ? *reinterpret_cast<const float *>(sR + (size_t)slot * rawbytes + rawbytes - 16) : 1.f;
                uint32_t worst = 0;
                int m = xt, gr = 0;
                while (m >= rows) { m -= rows; ++gr; }
                for (int it = xt; it < items; it += NX) {
                    // S residues of one pulse, or (S = 1) PP pulses
                    const int hi = gr / a.G, g = gr - hi * a.G, rho = S > 1 ? hi : 0, q = S > 1 ? 0 : hi;
                    // a gathered plane's row: one sample of each of 8 rows of the tile
                    const bool ga = GA && g >= a.Gf;
                    const int sd = ga ? Dks : 1, ev = ga ? rows - m : min(8, Dks - 8 * g);
                    const int o = Dks * m + a.Dk * rho + (ga ? 8 * a.Gf + g - a.Gf : 8 * g);
                    const float2 *rp = raw + q * nq + o;
                    float re[8], im[8];
                    if (WIN) {
                        const int k0 = kb + o;
                        if (a.wtab && k0 >= 0 && k0 + 7 * (GA ? sd : 1) < a.K) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const float2 v = e < ev ? rp[GA ? e * sd : e] : make_float2(0.f, 0.f);
                                const float w = wpp * sW[k0 + (GA ? e * sd : e)];   // the reference's float32 window product
                                re[e] = v.x * w;
                                im[e] = v.y * w;
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const float2 v = e < ev ? rp[GA ? e * sd : e] : make_float2(0.f, 0.f);
                                const int k = min(max(k0 + (GA ? e * sd : e), 0), a.K - 1);
                                const float w = wpp * (a.wtab ? sW[k] : (a.wk ? __ldg(&a.wk[k]) : 1.f) * xs);
                                re[e] = v.x * w;
                                im[e] = v.y * w;
                            }
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float2 v = e < ev ? rp[GA ? e * sd : e] : make_float2(0.f, 0.f);
                            re[e] = v.x * xs;
                            im[e] = v.y * xs;
                        }
                    }
                    unsigned char *z = zb + (size_t)(rho * a.G + g) * gbytes + (size_t)(q * a.RP + m) * 16;
                    uint4 h, l;
                    split8(re, h, l);
                    worst |= non_finite(h);
                    *reinterpret_cast<uint4 *>(z) = h;
                    *reinterpret_cast<uint4 *>(z + 2 * plane) = l;
                    split8(im, h, l);
                    worst |= non_finite(h);
                    *reinterpret_cast<uint4 *>(z + plane) = h;
                    *reinterpret_cast<uint4 *>(z + 3 * plane) = l;
                    m += NX;
                    while (m >= rows) { m -= rows; ++gr; }
                }
                if (WIN || a.bad) {
                    if (a.bad && (worst & 0x80008000u)) atomicMin(a.bad, un.p);
                }
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
        const int NTT = a.ntw * 32;
        const int nph = a.Ch * M_PB;
        // a batch is a run of up to PB units of one (parent, child group, column group) within an aligned group of PB
        // pulses; the next batch's phases are in registers while one is used
        Unit un, nb;
        un.set(a, u0);
        nb = un;
        int nbi = 0;                                            // the unit the batch in registers starts at
        constexpr int NR = (64 * M_PB + 95) / 96;               // phases per thread (Ch <= 64)
        float2 reg[NR];
        auto fetch = [&]() {
            if (nbi >= nu) return;
            const int pb = nb.p * a.PP & ~(M_PB - 1), c0 = nb.cg * a.Ch;
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                const int e = tt + q * NTT, pp = pb + (e & (M_PB - 1)), c = e / M_PB;
                reg[q] = make_float2(0.f, 0.f);
                if (e < nph && pp < a.P && c0 + c < a.C)
                    reg[q] = __ldg(&a.ph[((size_t)(a.n0 + nb.n) * a.C + c0 + c) * a.P + pp]);
            }
        };
        auto skip = [&]() {                                     // to the batch after the one in registers
            const int len = min(min(PBG - (nb.p & (PBG - 1)), a.PG - nb.p), nu - nbi);
            nbi += len;
            nb.p += len - 1;
            nb.next(a);
        };
        auto put = [&](int slot) {
#pragma unroll
            for (int q = 0; q < NR; ++q) {
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
        const int nth = a.TW * 32, th = a.TW == 1 ? lane : tt, dc = nth % a.Chv, dk = nth / a.Chv;
        bool ok = true;
        for (int i = 0; ok && i < nu; ++i, un.next(a)) {
            if (i == 0 || (un.p & (PBG - 1)) == 0) {           // a new batch
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
            if (a.TW == 1 && ts != warp - M_TW0) {              // another warp's unit (NT = ntw: ts is its warp)
                if (++ts == a.NT) { ts = 0; tpar ^= 1u; }
                continue;
            }
            if (!mbar_wait(&tempty[ts], tpar, 500, &s_abort, a.err, M_WAIT_NS)) break;
            const float4 *pr = sP + ((size_t)bslot * M_PB + (un.p * a.PP & (M_PB - 1))) * a.Ch;
            const float2 *ps = sS + ((size_t)bslot * M_PB + (un.p * a.PP & (M_PB - 1))) * a.Ch;
            unsigned char *tb = sT + (size_t)ts * tapbytes;
            int c = th % a.Chv, st = th / a.Chv;
            while (st < a.ks) {
                const int gs = st - a.Gf * a.A;
                const bool ga = GA && gs >= 0;
                const int g = ga ? a.Gf : st / a.A, ia = st - g * a.A, ev = ga ? 8 : min(8, Dks - 8 * g);
                const float sl = pr[c].y;
                const float4 h0 = *reinterpret_cast<const float4 *>(sH + 8 * st), h1 = *reinterpret_cast<const float4 *>(sH + 8 * st + 4);
                const float hv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                const float r0 = (float)(ga ? Dks * 8 * (gs % a.A8) + 8 * a.Gf + gs / a.A8 : Dks * ia + 8 * g), m = sl * r0;
                float2 w = cis_cycles((m - rintf(m)) + fmaf(sl, r0, -m));
                const float2 step = ga ? make_float2(pr[c].z, pr[c].w) : ps[c];   // a row's phasor, or a sample's
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
                // chunk 0 (real samples) and chunk 1 (imaginary) of rows c (the child's real part) and Chv + c (the phases
                // of a unit's pulses follow one another, so do their children here)
                unsigned char *o = tb + ((size_t)st * 2 * N + c) * 16;
                *reinterpret_cast<uint4 *>(o) = rh;
                *reinterpret_cast<uint4 *>(o + (size_t)a.Chv * 16) = ih;
                *reinterpret_cast<uint4 *>(o + (size_t)N * 16) = negate(ih);
                *reinterpret_cast<uint4 *>(o + (size_t)(N + a.Chv) * 16) = rh;
                o += hipart;
                *reinterpret_cast<uint4 *>(o) = rl;
                *reinterpret_cast<uint4 *>(o + (size_t)a.Chv * 16) = il;
                *reinterpret_cast<uint4 *>(o + (size_t)N * 16) = negate(il);
                *reinterpret_cast<uint4 *>(o + (size_t)(N + a.Chv) * 16) = rl;
                c += dc;
                st += dk;
                if (c >= a.Chv) { c -= a.Chv; ++st; }
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
        const int qw = 32 * (warp & 3) / a.RP;                 // this warp's pulse of a unit
        Unit un;
        un.set(a, u0);
        int b = -1, bslot = 0, d = 0;
        uint32_t bpar = 0, dpar = 0;
        const size_t cstride = (size_t)a.P * a.Kop;
        bool ok = true;
        for (int i = 0; ok && i < nu; ++i, un.next(a)) {
            if (i == 0 || (un.p & (PBG - 1)) == 0) {
                if (++b > 0) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&pempty[bslot]);
                    if (++bslot == M_PHB) { bslot = 0; bpar ^= 1u; }
                }
                ok = mbar_wait(&pfull[bslot], bpar, 500, &s_abort, a.err, M_WAIT_NS);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            const float4 *pr = sP + ((size_t)bslot * M_PB + (un.p * a.PP & (M_PB - 1)) + qw) * a.Ch;
            const int p = un.p * a.PP + qw;
            const int nc = min(a.Ch, a.C - un.cg * a.Ch);
            const int t1 = min(a.ntile, (un.tg + 1) * a.TG);
            for (int tl = un.tg * a.TG; tl < t1; ++tl) {
                ok = mbar_wait(&dfull[d], dpar, 500, &s_abort, a.err, M_WAIT_NS);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int jp = 32 * (warp & 3) + lane - qw * a.RP, j = S * (a.TM * tl + jp);
                const bool in = jp < a.TM && j < a.nj && p < a.P, any = __any_sync(0xffffffffu, in);
                const float uf = (float)(a.Dk * (a.j0 + j) - a.plk) - a.kc;
                const uint32_t base = tmem + lanes + (uint32_t)(d * S) * N + (uint32_t)(qw * a.Ch);
                const size_t yo = (((size_t)un.n * a.C + un.cg * a.Ch) * a.P + p) * a.Kop + j;
                if (any) {
                    for (int cb = GC * (warp >> 2); cb < nc; cb += 2 * GC) {
#pragma unroll
                        for (int r0 = 0; r0 < S; r0 += SP) {
                            float re[SP][GC], im[SP][GC];
#pragma unroll
                            for (int r = 0; r < SP; ++r) {
                                tmem_ldc<GC>(base + (uint32_t)((r0 + r) * N + cb), re[r]);
                                tmem_ldc<GC>(base + (uint32_t)((r0 + r) * N + a.Chv + cb), im[r]);
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

struct MmaShape { int ntw, S, PP, TM, G, Gf, A, ks, Ch, ROWS, W, NT, ZS, XR; size_t smem; };

// The shape of a level's product: the residues S, or the pulses PP that share a unit where a row needs at most half or a
// quarter of the accumulator's 128 rows (a product of N = 2 Ch <= 32 columns takes as long as one of 64), and the column
// steps per tile TM (fewer than 128 only where long filters at large decimations leave no room), by the MMA cycles and a
// unit's fixed cost for a row's tiles; and the most children per group whose operands fit with two tap buffers (one where
// that doubles the group).
bool mma_shape(int C, int Lk, int Dk, int nj, size_t wtab, bool stack, MmaShape *out)
{
    double best = 0.0;
    for (int TM = 128; TM >= 32 && best == 0.0; TM /= 2)
        for (int v = 0; v < 6; ++v) {
            const int S = v == 1 ? 2 : v == 2 ? 4 : 1, PP = v == 3 ? 2 : v == 4 ? 4 : 1;
            MmaShape s;
            s.S = S;
            s.PP = PP;
            s.TM = TM;
            const int Dks = S * Dk;
            s.A = (Lk + Dks - 1) / Dks;
            // v = 5: one or two samples past a multiple of 8 as planes that gather 8 rows' samples, ceil(A / 8) steps each
            // instead of A
            if (v == 5 && (Dks < 8 || Dks % 8 < 1 || Dks % 8 > 2)) continue;
            s.Gf = v == 5 ? Dks / 8 : (Dks + 7) / 8;
            s.G = v == 5 ? s.Gf + Dks % 8 : s.Gf;
            s.ks = s.Gf * s.A + (s.G - s.Gf) * ((s.A + 7) / 8);
            s.ROWS = TM + s.A - 1;
            if ((S > 1 && Dks > 8) || (PP > 1 && (!stack || TM != 128 || nj + s.A - 1 > 128 / PP))) continue;
            s.W = PP > 1 ? PP * Dks * (nj + s.A - 1) : Dks * s.ROWS + Dk * (S - 1);
            const int cmax = std::min((C + 7) & ~7, (S == 4 ? 32 : 64) / PP);
            // buffers (taps, planes, staged samples): a tap buffer per warp where one builds a unit's taps
            const int opt[6][3] = {{4, 3, 3}, {3, 3, 3}, {2, 2, 3}, {2, 2, 2}, {1, 2, 2}, {1, 1, 2}};
            // 3 or 4 warps for the taps, the other 4 or 3 for the samples: a row's taps are built once, its samples for
            // every tile; the split with the shorter longest role, at a tie with the shorter sum (3 for the 4,096-pulse
            // spotlight's third level: 291 against 360 us with 4; 4 for the 12,288 x 8,832 one's second and third: 4.8
            // and 6.4 ms against 5.2 and 7.2 with 3)
            auto turns = [&](int n, int ch, int nt) {
                const int ti = s.ks * PP * ch, xi = std::min(s.ROWS, (nj + S - 1) / S + s.A - 1) * s.G * S * PP;
                const int tap = nt > 2 ? (ti + 31) / 32 * 4 / n : (ti + 32 * n - 1) / (32 * n) * 4;
                const int smp = (nj + TM * S - 1) / (TM * S) * ((xi + 32 * (M_NAUX - n) - 1) / (32 * (M_NAUX - n))) * 3;
                return 8 * std::max(tap, smp) + tap + smp;
            };
            s.Ch = 0;
            int groups = 1 << 30;
            for (const auto &o : opt) {
                int ch = cmax;
                if (o[0] > 2 && (s.ks * PP * ch > TW1_ITEMS || o[0] != (turns(3, ch, 3) < turns(4, ch, 4) ? 3 : 4))) continue;
                while (ch >= 8 && mma_smem(S, s.G, s.ROWS, s.W, ch, PP, s.ks, o[0], o[1], o[2], wtab) > MMA_SMEM_MAX) ch -= 8;
                if (ch < 8) continue;
                const int g = (C + ch - 1) / ch;
                if (g * 2 > groups) continue;                // fewer buffers only for half the groups
                groups = g;
                s.NT = o[0]; s.ZS = o[1]; s.XR = o[2];
                s.Ch = (((C + g - 1) / g) + 7) & ~7;
                s.smem = mma_smem(S, s.G, s.ROWS, s.W, s.Ch, PP, s.ks, s.NT, s.ZS, s.XR, wtab);
            }
            if (!s.Ch) continue;
            const int ntile = (nj + TM * S - 1) / (TM * S), N = 2 * PP * s.Ch;
            s.ntw = s.NT > 2 ? s.NT : turns(3, s.Ch, s.NT) < turns(4, s.Ch, s.NT) ? 3 : 4;
            const int cyc = std::max(32 + N / 4, N / 2);     // measured cycles of an MMA of N columns
            const double cost = (double)groups * ntile * (S * s.ks * 3 * cyc + 400) / PP;
            if (best == 0.0 || cost < best) {
                best = cost;
                *out = s;
            }
        }
    return best != 0.0;
}

}  // namespace

bool level_mma_supported(int C, int Lk, int Dk, int Ko)
{
    MmaShape s;
    return C >= 1 && Dk >= 1 && Lk >= 1 && Lk <= 512 && mma_shape(C, Lk, Dk, Ko, 0, false, &s);
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
    const bool tab = wtab && mma_shape(L.C, Lk, L.Dk, nj, wtab, false, &m) &&
                     mma_shape(L.C, Lk, L.Dk, nj, 0, false, &m0) && m.Ch == m0.Ch;
    // the first level keeps a pulse per unit (its scan names the pulse of a non-finite sample)
    if (!tab && !mma_shape(L.C, Lk, L.Dk, nj, 0, !L.bad && !L.wp, &m)) { *why = "the level's operands do not fit shared memory"; return cudaErrorNotSupported; }
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    MmaArgs a;
    a.x = L.x; a.ph = L.phase; a.tk = L.Dk > 1 ? L.tk : nullptr; a.wp = L.wp; a.wk = L.wk; a.bad = L.bad;
    a.amax_in = amax_in; a.wexp = L.wexp; a.y = y; a.err = err; a.wtab = tab; a.n0 = n0; a.C = L.C; a.P = L.P; a.K = L.K; a.Dk = L.Dk; a.Lk = Lk;
    a.plk = plk; a.j0 = j0; a.nj = nj; a.Kop = (nj + 3) & ~3; a.G = m.G; a.Gf = m.Gf; a.A = m.A; a.A8 = (m.A + 7) / 8; a.ks = m.ks; a.Ch = m.Ch;
    a.ncg = (L.C + m.Ch - 1) / m.Ch; a.TM = m.TM; a.ntile = (nj + m.TM * m.S - 1) / (m.TM * m.S);
    a.ROWS = m.ROWS; a.W = m.W; a.NT = m.NT; a.ZS = m.ZS; a.XR = m.XR; a.ntw = m.ntw; a.TW = m.NT > 2 ? 1 : m.ntw;
    a.PP = m.PP; a.RP = 128 / m.PP; a.PG = (L.P + m.PP - 1) / m.PP; a.Chv = m.PP * m.Ch;
    a.nd = std::min(M_ND, 512 / (m.S * 2 * a.Chv));
    a.kc = (float)L.kc; a.test_wait_ns = L.test_wait_ns;
    // tiles per unit: all of the row's share a pulse's taps, unless that leaves too few units for the device
    a.TG = a.ntile;
    while (a.TG > 1 && (long)nn * a.ncg * ((a.ntile + a.TG - 1) / a.TG) * a.PG < 8L * nsm) a.TG = (a.TG + 1) / 2;
    a.ntg = (a.ntile + a.TG - 1) / a.TG;
    a.nunits = (long)nn * a.ncg * a.ntg * a.PG;
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
#define FFBP_MMA_RUN3(SV, GV, GA)                                                                           \
    (half ? (win ? run(level_mma_kernel<SV, true, true, GV, GA>) : run(level_mma_kernel<SV, true, false, GV, GA>)) \
          : (win ? run(level_mma_kernel<SV, false, true, GV, GA>) : run(level_mma_kernel<SV, false, false, GV, GA>)))
#define FFBP_MMA_RUN2(SV, GA) (m.Ch <= 16 ? FFBP_MMA_RUN3(SV, 4, GA) : FFBP_MMA_RUN3(SV, 8, GA))
    if (m.S == 4) return FFBP_MMA_RUN2(4, false);
    if (m.S == 2) return FFBP_MMA_RUN2(2, false);
    return m.G > m.Gf ? FFBP_MMA_RUN2(1, true) : FFBP_MMA_RUN2(1, false);
#undef FFBP_MMA_RUN3
#undef FFBP_MMA_RUN2
}

}  // namespace ffbp
