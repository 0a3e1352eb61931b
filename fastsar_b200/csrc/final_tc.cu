// The final stage on the tcgen05 tensor cores (sm_100a): the chosen form of fastsar/ffbp_cpu.cpp:302-469's
// final_tiles (the reference's CUDA counterpart is the wmma kernel final_tile_tc2, fastsar/ffbp_cuda.py:1371-1524).
//
// Each T = 32 tile is the complex sum out[i, j] = sum_n A[i, n] B[j, n] over n = (p, q) (final subaperture p,
// frequency sample q) with A = d wx exp(-2 pi i ux dlx (a0 + a1 q)) and B = wy exp(-2 pi i uy dly (a0 + a1 q)).
// As one real product, D = [Ar; Ai] [Br; Bi]^T (64 x 64, K = Pf Qfp with Qf padded to a multiple of 16 by zeros):
// re = D[i][j] - D[i+32][j+32], im = D[i][j+32] + D[i+32][j] (the weighted and the bfloat16 forms).
//
// The folded product (float16 and split float16 without aperture weights): rows r and T - 1 - r lie at offsets dl and
// -dl and columns likewise, so their ramps are conjugates, cos +- i sin. The operands hold the cosine and sine of one
// row of a pair: A' = [dr cos; di cos; dr sin; di sin] (2 T rows), B' = [cos; sin] (T rows), D = A' B'^T (2 T x T), and the
// epilogue forms a pair of pairs' four pixels from sums and differences of 8 of its values (tile_fold). Against the full
// product that is half of B' and of the accumulator, an addition less per value of A', N = 64 instead of 128, and the
// same roundings per pixel: 107,520 tiles of 36 x 71 in float16 12.46 -> 10.76 ms, 44 x 88 in split float16 27.6 -> 24.8 ms,
// 4,096 of 40 x 46 696 -> 637 us, 4,320 of 48 x 97 at T = 16 890 -> 837 us.
//
// One MMA is M = 128, N = 128 (folded 64), K = 16, and a "unit" is what one accumulator holds:
//   FFBP_FINAL_TC_BF16X3  one tile, operands split x = hi + lo in bfloat16: A' = [A_hi; A_lo], B' = [B_hi; B_lo], so
//                         one product gives hi hi, hi lo, lo hi and lo lo of the tile, summed in the epilogue;
//   the float32 form      one T = 32 or two T = 16 tiles, operands split x = hi + lo in float16 (22 bits; the samples
//                         scaled by a power of two) the same way. Its error against float64 is that of the CUDA-core
//                         kernel it replaces (images 1.4e-6 to 2.1e-6 against 1.5e-6 to 8.8e-6): the ramps' seeds
//                         come from the plan as hi + lo, their steps are computed to float32's rounding by the loader
//                         warp, and the accumulations are cut into short segments (the tensor core's sums truncate).
//                         4,096 tiles of 40 x 46: 533 us (CUDA cores 1,714); 107,520 of 44 x 88: 23.8 ms (83.9);
//                         4,320 of 48 x 97 at T = 16: 714 us (2,057). The producers' conversions bound it.
//   FFBP_FINAL_TC_F16     two T = 32 tiles in float16, A' = [A_1; A_2], B' = [B_1; B_2]: the two diagonal blocks of the
//                         product are the tiles; or four T = 16 tiles, the four diagonal blocks, each epilogue warp
//                         reading one of them from its own lane quarter. The samples are
//                         scaled by a power of two (from the largest sample component, which the last level kernel
//                         records) into float16's range, and the pixels by its inverse.
// M = 128 takes max(32 + N / 4, N / 2) cycles per K step, so the larger shape does two or four times the work per
// instruction; two issuing warps overlap one's waits on its stage with the other's products.
//
// Block roles (persistent over units; one block per SM):
//   warp 6, 7    loaders, one or two that alternate (loaders): stage each final subaperture's samples and geometry by cp.async into a ring of LS
//                slots, LS - 1 subapertures ahead (its copies' completion arrives on the slot's barrier);
//   12 warps after them  producers: per final subaperture they build A' and B' (128 and 128 or 64 rows x Qfp) in shared memory from
//                the staged slot, a row's ramp by a complex recurrence along q seeded in float64, converted to the
//                operand type, into a ring of S stages (K-major, no swizzle: core matrices of 8 rows x 16 bytes);
//   warps 4, 5   one thread each issues tcgen05.mma: warp 4 + k takes the final subapertures p = k mod 2 of every
//                unit into its own accumulator (two 128-column accumulators per issuer, 512 TMEM columns), from its
//                own stages k, k + 2, ... of the ring (a stage with one consumer, so that no parity wait can run two
//                phases ahead of its barrier), commits each stage to the stage's "empty" barrier and the unit to the
//                accumulator's "full" barrier;
//   warps 0..3   epilogue: sum the issuers' accumulators (and, for bfloat16, the four split products), combine
//                re/im through shared memory, apply the quadratic phase and write the tile into the image (cropped).
//
// Every wait on a barrier is bounded: a wait that runs out sets *err (when given) and the block winds down without
// touching the barrier again; each issuing thread drains its MMAs (bounded) before the accumulator columns are freed.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace ffbp {

namespace {

constexpr int NEPI = 4;                    // epilogue warps 0..3 (TMEM lane quarters 0..3)
constexpr int NISS = 2;                    // MMA issuing warps 4, 5
constexpr int NPW = 12;                    // producer warps, after the loaders
constexpr int FS = 6;                      // most stages of folded operands (of the full ones 4): 512-pixel spotlight 36.8
                                           // against 38.9 us with 4, the larger cases the same
constexpr int LS = 8;                      // the loader's ring of staged final subapertures
constexpr int TMEM_COLS = 512;             // NISS issuers x 2 accumulators x 128 columns
constexpr uint64_t WAIT_NS = 2000000000ull;   // a barrier that has not completed after 2 s counts as stuck
constexpr uint32_t PRODUCER_HINT_NS = 1000;   // suspend-time hints of the waits: producers on a free stage or
                                              // a staged subaperture, the loader on a free ring slot,
constexpr uint32_t ISSUER_HINT_NS = 2000;     // the issuers on a filled stage,
constexpr uint32_t EPILOGUE_HINT_NS = 4000;   // the epilogue on a finished accumulator

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ uint32_t mbar_test(uint64_t *bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done;
}

__device__ __forceinline__ uint32_t mbar_test_sleep(uint64_t *bar, uint32_t parity, uint32_t hint_ns)
{
    // the thread may be suspended until the phase completes or about hint_ns have passed
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns) : "memory");
    return done;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for the phase of parity `parity` of *bar: false (and the block's abort flag and *err set) when it
// has not completed after limit_ns of wall time, or when another thread of the block has aborted. HINT_NS is the
// suspend-time hint of each poll (0: poll without one).
template <uint32_t HINT_NS>
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort, int *err,
                                          uint64_t limit_ns = WAIT_NS)
{
    if (mbar_test(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 1;; ++it) {
        if (HINT_NS ? mbar_test_sleep(bar, parity, HINT_NS) : mbar_test(bar, parity)) return true;
        if ((it & 255u) == 0) {
            if (*abort) return false;
            if (global_ns() - t0 > limit_ns) break;
        }
    }
    *abort = 1;
    if (err) atomicAdd(err, 1);
    return false;
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    // sm_100 shared-memory matrix descriptor: start address, leading (K) and stride (M/N) byte offsets in 16-byte
    // units, version 1 at bit 46, no swizzle
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mma_f16kind(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 :: "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_u32(bar)) : "memory");
}

// 16 consecutive accumulator columns of this thread's TMEM lane, without waiting
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// bytes = 4, 8 or 16 (dst and src aligned to it); the copy of an invalid element reads nothing and zero-fills the
// destination
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, int bytes, bool valid)
{
    if (bytes == 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
    else if (bytes == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" :: "r"(dst), "l"(src), "r"(valid ? 8 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

struct TcArgs {
    const float2 *__restrict__ d;
    int B, Pf, Qf, Qfp, S, nunits, nis;
    const double *__restrict__ ux;
    const double *__restrict__ uy;
    const float4 *__restrict__ seeds;      // the ramp seeds per tile and subaperture: float16 one (or null), split float16 two
    double spx, spy, a0, a1, fc2;
    const double *__restrict__ ucx;
    const double *__restrict__ ucy;
    const double *__restrict__ rc;
    const float *__restrict__ w;
    float2 *tiles;
    float2 *img;
    const int2 *__restrict__ first;
    int nx, ny, ox, oy;
    float scale;
    int *err;
    const int *amax;
    int interleave;                        // the order of the producer warps' items (final_tc_kernel)
    int nwi;                               // producer items per stage
    int seg, nsg;                          // final subapertures per accumulation (even unless all), accumulations per unit
    unsigned test_wait_ns;                 // tests only: the issuers' wait on a barrier nothing completes (0: none)
    int wexp;                              // the weights' power of two (FinalLaunch::wexp)
};

// The power of two s that brings samples whose components are at most *amax (a float's bits; null: unknown) to
// below 2^13 in magnitude, weighted by at most 2^wexp, so that d s times a ramp and a weight stays inside float16's range
// (65504).
__device__ __forceinline__ float operand_scale(const int *amax, int wexp)
{
    // (with the exponent taken from the float's bits the kernel of 107,520 float16 tiles of 36 x 71 takes 11.98 ms for 11.67)
    if (!amax) return 1.f;
    const float m = __int_as_float(*amax);
    if (!(m > 0.f) || !isfinite(m)) return 1.f;
    int ex;
    frexpf(m, &ex);                                             // m < 2^ex
    return ldexpf(1.f, min(max(13 - ex - wexp, -120), 120));    // it and its inverse normal float32 numbers
}

// The operands' arithmetic: float16, or x = hi + lo in bfloat16 (16 bits) or in float16 (22 bits).
enum Operands { OP_F16 = 0, OP_BF16X2 = 1, OP_F16X2 = 2 };

// 8 values -> 16 bytes of operand: float16, or the high parts (and the low parts in lo)
template <int OP>
__device__ __forceinline__ void pack8(const float *v, uint4 &hi, uint4 &lo)
{
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        l[e] = 0;
        if (OP == OP_BF16X2) {
            const __nv_bfloat162 x = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
            const float r0 = v[2 * e] - __low2float(x), r1 = v[2 * e + 1] - __high2float(x);
            const __nv_bfloat162 y = __floats2bfloat162_rn(r0, r1);
            h[e] = *reinterpret_cast<const uint32_t *>(&x);
            l[e] = *reinterpret_cast<const uint32_t *>(&y);
        } else {
            const __half2 x = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
            h[e] = *reinterpret_cast<const uint32_t *>(&x);
            if (OP == OP_F16X2) {
                const float2 f = __half22float2(x);
                const __half2 y = __floats2half2_rn(v[2 * e] - f.x, v[2 * e + 1] - f.y);
                l[e] = *reinterpret_cast<const uint32_t *>(&y);
            }
        }
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ uint4 flip_sign(uint4 v)
{
    const uint32_t sg = 0x80008000u;
    return make_uint4(v.x ^ sg, v.y ^ sg, v.z ^ sg, v.w ^ sg);
}

// Loader warps (6, or 6 and 7). Of the folded forms one warp's copies bound the stages (a subaperture of 33 x 37 took 700 ns,
// the producers 500), so two take turns: 2,048 x 2,048 pixels 637 -> 512 us in the float32 form and 367 -> 268 us in
// float16, 1,499 x 701 at T = 16 837 -> 754 and 573 -> 483 us. Two items of T = 32 in float16 per producer warp take longer
// than their copies, and the block with a 20th warp runs them slower, with one loader at work or two (107,520 tiles of
// 36 x 71: 10.75 ms with one, 12.1 with two; 900 of 72 x 96: 268 and 272 us); from three on two gain again (2,400 of
// 82 x 126: 985 -> 951 us).
template <int OP, bool WEIGHTED, int MAXWI, int TT> __host__ __device__ constexpr int loaders()
{
    return OP == OP_BF16X2 || WEIGHTED || (OP == OP_F16 && TT == 32 && MAXWI == 2) ? 1 : 2;
}

// Threads of a block.
template <int OP, bool WEIGHTED, int MAXWI, int TT> __host__ __device__ constexpr int block_threads()
{
    return (NEPI + NISS + loaders<OP, WEIGHTED, MAXWI, TT>() + NPW) * 32;
}

// Tiles per unit: 128 operand rows hold 2 TT rows per tile, twice that when split.
template <int OP, int TT> __host__ __device__ constexpr int unit_tiles() { return OP == OP_F16 ? 64 / TT : 32 / TT; }

// The tile of slot ts of this block's local unit ul (>= B when none).
template <int OP, int TT>
__device__ __forceinline__ int unit_tile(int ul, int ts)
{
    return unit_tiles<OP, TT>() * ((int)blockIdx.x + ul * (int)gridDim.x) + ts;
}

// The pixels of one T = 32 tile from P0 = D'[0:32, :] and P1 = D'[32:64, :] (rows of 64 + 1 floats in shared
// memory): thread t of the 128 epilogue threads takes row i = t / 4 and eight consecutive columns.
__device__ __forceinline__ void tile_pixels(const TcArgs &a, int tile, const float *P0, const float *P1, int t,
                                            float scale)
{
    constexpr int TT = 32;
    const int i = t >> 2, jb = (t & 3) * 8;
    const double cx = a.ucx[tile], cy = a.ucy[tile];
    const float f = (float)(a.fc2 / (2.0 * a.rc[tile]));
    const float dx = ((float)i - 0.5f * (TT - 1)) * (float)a.spx;
    const int2 f0 = a.img ? a.first[tile] : make_int2(0, 0);
    const int x = f0.x + i - a.ox;
    float2 outv[8];
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
        const int j = jb + jj;
        const float re = P0[i * 65 + j] - P1[i * 65 + j + 32];
        const float im = P0[i * 65 + j + 32] + P1[i * 65 + j];
        const float dy = ((float)j - 0.5f * (TT - 1)) * (float)a.spy;
        const float los = (float)cx * dx + (float)cy * dy;
        const float qc = (dx * dx + dy * dy - los * los) * f;
        const float2 e = cis_cycles(qc);
        const float2 o = cmul(make_float2(re, im), e);
        outv[jj] = make_float2(o.x * scale, o.y * scale);
    }
    if (a.img) {
        if (x >= 0 && x < a.nx) {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
                const int y = f0.y + jb + jj - a.oy;
                if (y >= 0 && y < a.ny) a.img[(size_t)x * a.ny + y] = outv[jj];
            }
        }
    } else {
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) a.tiles[((size_t)tile * TT + i) * TT + jb + jj] = outv[jj];
    }
}

// The pixels of one T = 16 tile: lane l < 16 of the warp holds accumulator row l (Ar row i = l) at the tile's 32
// columns (Br then Bi: v0 = D[i][j], v1 = D[i][j + 16]), lane l + 16 row Ai (v0 = D[i + 16][j], v1 = D[i + 16][j + 16]);
// re = D[i][j] - D[i + 16][j + 16], im = D[i][j + 16] + D[i + 16][j]. Lanes 0..15 write row i's 16 pixels.
__device__ __forceinline__ void tile16_pixels(const TcArgs &a, int tile, const float *v0, const float *v1, int lane,
                                              float scale)
{
    constexpr int TT = 16;
    float re[16], im[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float d11 = __shfl_down_sync(0xffffffffu, v1[j], 16), d10 = __shfl_down_sync(0xffffffffu, v0[j], 16);
        re[j] = v0[j] - d11;
        im[j] = v1[j] + d10;
    }
    if (lane >= 16 || tile >= a.B) return;
    const int i = lane;
    const double cx = a.ucx[tile], cy = a.ucy[tile];
    const float f = (float)(a.fc2 / (2.0 * a.rc[tile]));
    const float dx = ((float)i - 0.5f * (TT - 1)) * (float)a.spx;
    const int2 f0 = a.img ? a.first[tile] : make_int2(0, 0);
    const int x = f0.x + i - a.ox;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float dy = ((float)j - 0.5f * (TT - 1)) * (float)a.spy;
        const float los = (float)cx * dx + (float)cy * dy;
        const float qc = (dx * dx + dy * dy - los * los) * f;
        const float2 o = cmul(make_float2(re[j], im[j]), cis_cycles(qc));
        const float2 ov = make_float2(o.x * scale, o.y * scale);
        if (a.img) {
            const int y = f0.y + j - a.oy;
            if (x >= 0 && x < a.nx && y >= 0 && y < a.ny) a.img[(size_t)x * a.ny + y] = ov;
        } else {
            a.tiles[((size_t)tile * TT + i) * TT + j] = ov;
        }
    }
}

// The pixels of one tile of the folded operands from its accumulator P (2 TT rows of TT + 1 floats in shared memory; with
// h = TT / 2 and r, s < h, rows r, h + r, TT + r, TT + h + r: the sums with dr cos, di cos, dr sin, di sin of row r's ramp;
// columns s, h + s: with the cosine and sine of column s's). Rows r and TT - 1 - r (sg = +-1) and columns s and TT - 1 - s
// (sj = +-1) are the four sign combinations of d (cx + i sg sx) (cy + i sj sy). Thread t of 2 TT h / 8 takes row pair
// t / (TT / 4) and two neighbouring column pairs: 8 pixels, whose quadratic phases are equal in twos.
template <int TT>
__device__ __forceinline__ void tile_fold(const TcArgs &a, int tile, const float *P, int t, float scale)
{
    constexpr int h = TT / 2, W = TT + 1;
    const int r = t / (TT / 4), s0 = 2 * (t % (TT / 4));
    const double cx = a.ucx[tile], cy = a.ucy[tile];
    const float f = (float)(a.fc2 / (2.0 * a.rc[tile]));
    const float dx = ((float)r - 0.5f * (TT - 1)) * (float)a.spx;
    const int2 f0 = a.img ? a.first[tile] : make_int2(0, 0);
    const float *p0 = P + r * W + s0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int s = s0 + k;
        const float ccr = p0[k], csr = p0[h + k], cci = p0[h * W + k], csi = p0[h * W + h + k];
        const float scr = p0[TT * W + k], ssr = p0[TT * W + h + k];
        const float sci = p0[(TT + h) * W + k], ssi = p0[(TT + h) * W + h + k];
        const float dy = ((float)s - 0.5f * (TT - 1)) * (float)a.spy;
#pragma unroll
        for (int opp = 0; opp < 2; ++opp) {                    // sg == sj, then sg == -sj
            const float los = opp ? (float)cx * dx - (float)cy * dy : (float)cx * dx + (float)cy * dy;
            const float2 e = cis_cycles((dx * dx + dy * dy - los * los) * f);
            const float er = opp ? ccr + ssr : ccr - ssr, ei = opp ? cci + ssi : cci - ssi;
            const float dr = opp ? csi - sci : csi + sci, di = opp ? csr - scr : csr + scr;
#pragma unroll
            for (int neg = 0; neg < 2; ++neg) {                 // sj = +1, then -1
                const int j = neg ? TT - 1 - s : s, i = (neg != 0) != (opp != 0) ? TT - 1 - r : r;
                const float2 o = cmul(make_float2(neg ? er + dr : er - dr, neg ? ei - di : ei + di), e);
                const float2 ov = make_float2(o.x * scale, o.y * scale);
                if (a.img) {
                    const int x = f0.x + i - a.ox, y = f0.y + j - a.oy;
                    if (x >= 0 && x < a.nx && y >= 0 && y < a.ny) a.img[(size_t)x * a.ny + y] = ov;
                } else {
                    a.tiles[((size_t)tile * TT + i) * TT + j] = ov;
                }
            }
        }
    }
}

template <int OP, bool WEIGHTED, int MAXWI, int TT>
__global__ void __launch_bounds__(block_threads<OP, WEIGHTED, MAXWI, TT>(), 1) final_tc_kernel(const TcArgs a)
{
    constexpr int NLD = loaders<OP, WEIGHTED, MAXWI, TT>(), PW0 = NEPI + NISS + NLD;
    constexpr int NTHREADS = block_threads<OP, WEIGHTED, MAXWI, TT>();
    constexpr bool BF = OP == OP_BF16X2, X2 = OP == OP_F16X2, FOLD = !BF && !WEIGHTED;
    constexpr int NB = FOLD ? 64 : 128;                         // operand rows of B': the accumulator's columns
    constexpr int NTS = unit_tiles<OP, TT>();                   // tiles per unit
    extern __shared__ __align__(1024) unsigned char smem[];
    const int ng = a.Qfp / 8;                                   // core matrices along K per operand
    const uint32_t H = 64u * a.Qfp * 2u;                        // 64 operand rows
    const uint32_t HS = 2u * TT * a.Qfp * 2u;                   // one part (hi or lo) of a tile's operand rows, 2 TT rows
    const uint32_t HB = FOLD ? HS / 2 : HS;                     // a part of a tile's rows of B'
    const uint32_t stagebytes = FOLD ? 3u * H : 4u * H;         // A' (128 rows), B' (NB rows)
    float *sP = reinterpret_cast<float *>(smem + (size_t)a.S * stagebytes);             // [2][32][65] or [2][64][33]
    // the loader's ring: per slot and tile slot, the subaperture's Qfp samples (zero past Qf), ux, uy and the
    // three weights (split float16: the seeds of both ramps and the steps of the TT / 2 row pairs of each); tsb bytes
    unsigned char *ring = reinterpret_cast<unsigned char *>(sP + (FOLD ? 2 * 64 * 33 : 2 * 32 * 65));
    const uint32_t tsb = 8u * a.Qfp + 32u + (X2 ? 8u * TT : 0u), slotbytes = (uint32_t)NTS * tsb;
    uint64_t *bars = reinterpret_cast<uint64_t *>(ring + (size_t)LS * slotbytes);
    uint64_t *full = bars, *empty = bars + a.S, *accf = bars + 2 * a.S, *acce = accf + 2, *drain = acce + 2;
    uint64_t *lfull = drain + 2, *lempty = lfull + LS;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    __shared__ uint64_t s_never;                                // a barrier nothing arrives on (the tests' stuck wait)

    const int t = threadIdx.x, warp = t / 32, lane = t % 32;
    const int nis = a.nis;
    // this block's units: blockIdx.x + ul gridDim.x
    const int nul = a.nunits > (int)blockIdx.x ? (a.nunits - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (t == 0) {
        s_abort = 0;
        for (int s = 0; s < a.S; ++s) {
            mbar_init(&full[s], NPW);
            mbar_init(&empty[s], 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(&accf[k], (uint32_t)nis);
            mbar_init(&acce[k], NEPI);
            mbar_init(&drain[k], 1);
        }
        for (int k = 0; k < LS; ++k) {
            // the loader's 32 threads, once their copies have landed (split float16: and their steps are written)
            mbar_init(&lfull[k], X2 ? 64 : 32);
            mbar_init(&lempty[k], NPW);
        }
        mbar_init(&s_never, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (X2) {                                                   // whole groups past Qf are not written: zero once
        for (uint32_t i = (uint32_t)t * 16u; i < (uint32_t)a.S * stagebytes; i += NTHREADS * 16u)
            *reinterpret_cast<uint4 *>(smem + i) = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == NEPI) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&s_tmem)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t smem0 = smem_u32(smem);

    if (warp >= NEPI + NISS && warp < PW0) {
        // ------------------------------------------------------------------ loader
        // Stages every final subaperture of this block's units LS - 1 ahead of the producers: per tile slot the
        // Qfp samples (8 bytes each, zero past Qf and for a tile past the last), ux, uy and the weights, by cp.async
        // into ring slot it % LS; the copies' completion arrives on lfull (each thread's, .noinc), the producers'
        // reads of the slot on lempty. The next unit's samples and geometry are prefetched into L2 a unit ahead.
        const int nts = NTS;
        const int ntot = nul * a.Pf;
        const size_t nbp = (size_t)a.B * a.Pf;
        const bool fs = OP == OP_F16 && a.seeds;                // stage the float32 seeds in place of ux, uy
        auto prefetch_unit = [&](int ul) {
            if (ul >= nul) return;
            for (int ts = 0; ts < nts; ++ts) {
                const int tile = unit_tile<OP, TT>(ul, ts);
                if (tile >= a.B) break;
                const char *dbeg = reinterpret_cast<const char *>(a.d + (size_t)tile * a.Pf * a.Qf);
                const int dbytes = a.Pf * a.Qf * (int)sizeof(float2);
                for (int o = lane * 128; o < dbytes; o += 32 * 128)
                    asm volatile("prefetch.global.L2 [%0];" :: "l"(dbeg + o));
                const char *src = X2   ? reinterpret_cast<const char *>(a.seeds + 2 * (size_t)tile * a.Pf)
                                  : fs ? reinterpret_cast<const char *>(a.seeds + (size_t)tile * a.Pf)
                                       : reinterpret_cast<const char *>((lane < 16 ? a.ux : a.uy) + (size_t)tile * a.Pf);
                const int ub = a.Pf * (X2 ? 32 : fs ? 16 : 8);
                for (int o = (lane & 15) * 128; o < ub; o += 16 * 128)
                    asm volatile("prefetch.global.L2 [%0];" :: "l"(src + o));
            }
        };
        // loader k takes every NLD-th subaperture from the k-th on: ul, p its unit and subaperture
        const int k0 = warp - (NEPI + NISS);
        int ul = k0 / a.Pf, p = k0 % a.Pf;
        // split float16: lane l computes the step of row pair r of operand xop of tile slot xts, whose slope it reads
        // a subaperture ahead
        const int xts = X2 ? lane / TT : 0, xop = (lane % TT) / (TT / 2), xr = lane % (TT / 2);
        float2 slope = make_float2(0.f, 0.f);
        auto fetch_slope = [&](int fu, int fp) {
            const int tile = fu < nul ? unit_tile<OP, TT>(fu, xts) : a.B;
            slope = make_float2(0.f, 0.f);
            if (tile < a.B)
                slope = *(reinterpret_cast<const float2 *>(a.seeds + 2 * ((size_t)tile * a.Pf + fp) + xop) + 1);
        };
        if (X2) fetch_slope(ul, p);
        for (int it = k0; it < ntot; it += NLD) {
            const int ls = it % LS;
            if (it >= LS && !mbar_wait<PRODUCER_HINT_NS>(&lempty[ls], (uint32_t)((it / LS - 1) & 1), &s_abort, a.err))
                break;
            if (p == 0) prefetch_unit(ul + 1);
            const uint32_t sl = smem_u32(ring) + (uint32_t)ls * slotbytes;
            for (int ts = 0; ts < nts; ++ts) {
                const int tile = unit_tile<OP, TT>(ul, ts);
                const bool tv = tile < a.B;
                const size_t bp = tv ? (size_t)tile * a.Pf + p : 0;
                const float2 *src = a.d + bp * a.Qf;
                const uint32_t dst = sl + (uint32_t)ts * tsb;
                for (int q = lane; q < a.Qfp; q += 32) {
                    const bool v = tv && q < a.Qf;
                    cp_async(dst + 8u * q, v ? (const void *)(src + q) : (const void *)a.d, 8, v);
                }
                const uint32_t gd = dst + 8u * a.Qfp;
                if (X2) {
                    if (lane < 2) cp_async(gd + 16u * lane, (const void *)(a.seeds + 2 * bp + lane), 16, tv);
                } else if (fs) {
                    if (lane == 0) cp_async(gd, (const void *)(a.seeds + bp), 16, tv);
                } else if (lane < 2) cp_async(gd + 8u * lane, (const void *)((lane ? a.uy : a.ux) + bp), 8, tv);
                if (WEIGHTED && lane >= 2 && lane < 5)
                    cp_async(gd + 16u + 4u * (lane - 2), (const void *)(a.w + (size_t)(lane - 2) * nbp + bp), 4, tv);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(smem_u32(&lfull[ls])) : "memory");
            for (p += NLD; p >= a.Pf; p -= a.Pf) ++ul;
            if (X2) {
                const float m = (float)(2 * xr - (TT - 1));
                float c = m * slope.x;                          // exact; the low part then moves it by a rounding
                c = (c - rintf(c)) + m * slope.y;
                float sn, cs;
                sincospif(-2.f * c, &sn, &cs);
                *reinterpret_cast<float2 *>(ring + (size_t)ls * slotbytes + (uint32_t)xts * tsb + 8u * a.Qfp + 32u +
                                            8u * (uint32_t)(xop * (TT / 2) + xr)) = make_float2(cs, sn);
                mbar_arrive(&lfull[ls]);
                fetch_slope(ul, p);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (X2 && warp >= PW0) {
        // ------------------------------------------------------------------ producers, split float16
        // Items, lanes and rows as below. Here the items (twice the conversions and stores) alternate A, the heavier,
        // and B, and are dealt to the warps in turn from a start that moves by one more than their count per stage, so
        // that the warps' loads even out over a few stages (a fixed set of items per warp and stage was 1.4 times slower
        // at 40 x 46). With fewer items than warps some have none in a subaperture: they wait and arrive with the others
        // all the same. A parity wait tells a phase from its neighbours only: a warp that skipped one could test a slot
        // or a stage two phases ahead of its barrier (and pass), and one that waited without arriving could be passed
        // by two phases (and wait for ever). With the waits left out where there was no item 4,096 tiles of 40 x 46 took 512 us,
        // with them 533; one arrival a warp instead of one an item 754 -> 714 us (4,320 of 48 x 97 at T = 16).
        const int pw = warp - PW0;
        constexpr int GPI = 64 / TT;
        const int ngr = (a.Qf + 7) / 8, hg = (ngr + GPI - 1) / GPI, ntot = nul * a.Pf;
        const int r = lane % (TT / 2), sub = lane / (TT / 2);
        uint32_t roff[4];
        {
            const int rows[4] = {r, r + TT / 2, r + TT, r + TT + TT / 2};
#pragma unroll
            for (int k = 0; k < 4; ++k) roff[k] = (uint32_t)(((rows[k] >> 3) * ng) * 128 + (rows[k] & 7) * 16);
        }
        const float dscale = operand_scale(a.amax, a.wexp), m = (float)(2 * r - (TT - 1));
        const int rs = a.S / nis, turn = (a.nwi + 1) % NPW;
        int ps0 = 0, ps1 = 0, p = 0, first = pw;
        uint32_t pp0 = 0, pp1 = 0;
        for (int it = 0; it < ntot; ++it) {
            const int ls = it % LS, kq = nis == 2 ? (p & 1) : 0, stg = kq + nis * (kq ? ps1 : ps0);
            if (!mbar_wait<PRODUCER_HINT_NS>(&lfull[ls], (uint32_t)((it / LS) & 1), &s_abort, a.err)) break;
            if (!mbar_wait<PRODUCER_HINT_NS>(&empty[stg], (kq ? pp1 : pp0) ^ 1u, &s_abort, a.err)) break;
            for (int item = first; item < a.nwi; item += NPW) {
                const int q = item >> 1, ts = NTS == 1 ? 0 : q / hg, g = GPI * (NTS == 1 ? q : q - ts * hg) + sub;
                const bool isA = (item & 1) == 0;
                if (g < ngr) {
                    const unsigned char *tsp = ring + (size_t)ls * slotbytes + (uint32_t)ts * tsb;
                    // the ramp at sample 8 g: -(m Y + 8 g m V) cycles from the plan's seeds, whose high parts times m
                    // and 8 g m are exact
                    const float4 sd = *reinterpret_cast<const float4 *>(tsp + 8 * a.Qfp + (isA ? 0 : 16));
                    const float n8 = m * (8.f * (float)g);
                    float c0 = m * sd.x, c1 = n8 * sd.z;
                    c0 -= rintf(c0);
                    c1 -= rintf(c1);
                    float2 wv = cis_cycles(-((c0 + c1) + fmaf(m, sd.y, n8 * sd.w)));
                    const float2 st = *reinterpret_cast<const float2 *>(tsp + 8 * a.Qfp + 32 + 8 * ((isA ? 0 : TT / 2) + r));
                    const uint32_t part = isA ? HS : HB;
                    unsigned char *ob = smem + (size_t)stg * stagebytes + (isA ? 0u : 2u * H) + (uint32_t)ts * (2u * part) + (uint32_t)g * 128u;
                    uint4 h, l;
                    if (isA) {
                        wv.x *= dscale;
                        wv.y *= dscale;
                        const float4 *dq = reinterpret_cast<const float4 *>(tsp + 64 * g);
                        float r1[8], i1[8], r2[8], i2[8];
#pragma unroll
                        for (int e2 = 0; e2 < 4; ++e2) {
                            const float4 dd = dq[e2];
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                const int e = 2 * e2 + hh;
                                const float dr = hh ? dd.z : dd.x, di = hh ? dd.w : dd.y;
                                r1[e] = dr * wv.x; i1[e] = di * wv.x;
                                r2[e] = dr * wv.y; i2[e] = di * wv.y;
                                wv = cmul(wv, st);
                            }
                        }
                        pack8<OP>(r1, h, l);
                        *reinterpret_cast<uint4 *>(ob + roff[0]) = h;
                        *reinterpret_cast<uint4 *>(ob + HS + roff[0]) = l;
                        pack8<OP>(i1, h, l);
                        *reinterpret_cast<uint4 *>(ob + roff[1]) = h;
                        *reinterpret_cast<uint4 *>(ob + HS + roff[1]) = l;
                        pack8<OP>(r2, h, l);
                        *reinterpret_cast<uint4 *>(ob + roff[2]) = h;
                        *reinterpret_cast<uint4 *>(ob + HS + roff[2]) = l;
                        pack8<OP>(i2, h, l);
                        *reinterpret_cast<uint4 *>(ob + roff[3]) = h;
                        *reinterpret_cast<uint4 *>(ob + HS + roff[3]) = l;
                    } else {
                        float r1[8], i1[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            r1[e] = wv.x;
                            i1[e] = wv.y;
                            wv = cmul(wv, st);
                        }
                        pack8<OP>(r1, h, l);
                        *reinterpret_cast<uint4 *>(ob + roff[0]) = h;
                        *reinterpret_cast<uint4 *>(ob + HB + roff[0]) = l;
                        pack8<OP>(i1, h, l);
                        *reinterpret_cast<uint4 *>(ob + roff[1]) = h;
                        *reinterpret_cast<uint4 *>(ob + HB + roff[1]) = l;
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[stg]);
                mbar_arrive(&lempty[ls]);
            }
            first -= turn;
            if (first < 0) first += NPW;
            if (kq) {
                if (++ps1 == rs) { ps1 = 0; pp1 ^= 1u; }
            } else if (++ps0 == rs) {
                ps0 = 0;
                pp0 ^= 1u;
            }
            if (++p == a.Pf) p = 0;
        }
    } else if (warp >= PW0) {
        // ------------------------------------------------------------------ producers
        // Warp items: (tile slot ts, operand A or B, pair of 8-sample groups gp). Lane l of the warp takes pixel
        // row pair r = l % 16 (rows r and 31 - r, whose offsets are dl and -dl, so that their ramps are complex
        // conjugates and one recurrence serves both) and group g = 2 gp + l / 16. Folded, an A item writes dr and di times
        // the ramp's cosine and sine, a B item its cosine and sine. Otherwise an A item writes Ar, Ai of rows r and
        // 31 - r (d times the ramp and d times its conjugate), a B item Br, Bi of row r and, without weights, row
        // 31 - r from row r's words (the same real part, the imaginary part's sign flipped).
        const int pw = warp - PW0;
        constexpr int GPI = 64 / TT;                            // 8-sample groups per item: a lane per row pair
        const int hg = (ng + GPI - 1) / GPI;
        const int nts = NTS;
        const int nwi = nts * 2 * hg;
        const int ntot = nul * a.Pf;
        const int r = lane % (TT / 2), sub = lane / (TT / 2);
        // byte offsets (without the group) of rows r, r + TT, TT - 1 - r, 2 TT - 1 - r within a tile's 2 TT rows
        uint32_t roff[4];
        {
            const int rows[4] = {r, FOLD ? r + TT / 2 : r + TT, FOLD ? r + TT : TT - 1 - r, FOLD ? r + TT + TT / 2 : 2 * TT - 1 - r};
#pragma unroll
            for (int k = 0; k < 4; ++k) roff[k] = (uint32_t)(((rows[k] >> 3) * ng) * 128 + (rows[k] & 7) * 16);
        }
        // this warp's items (the same in every stage): tile slot, operand (0 = A), pair of groups; -1 = none
        int it_ts[MAXWI], it_op[MAXWI], it_gp[MAXWI];
#pragma unroll
        for (int k = 0; k < MAXWI; ++k) {
            if (a.interleave) {
                // A items first, then B items, dealt out to the warps forwards and backwards in turn, so that
                // with an even count per warp each warp builds as many A items (the heavier) as B items
                const int j = (k & 1) ? k * NPW + (NPW - 1 - pw) : k * NPW + pw;
                const int half = nwi / 2;
                it_ts[k] = j < nwi ? (j % half) / hg : -1;
                it_op[k] = j >= half ? 1 : 0;
                it_gp[k] = (j % half) % hg;
            } else {
                const int wi = pw + k * NPW;
                it_ts[k] = wi < nwi ? wi / (2 * hg) : -1;
                it_op[k] = (wi / hg) & 1;
                it_gp[k] = wi % hg;
            }
        }
        const float sp32x = (float)a.spx, sp32y = (float)a.spy;
        // the float16 operands carry d scaled by a power of two that keeps them inside the format's range
        const float dscale = BF ? 1.f : operand_scale(a.amax, a.wexp);
        // issuer k's stages are k + nis s for s < S / nis, filled and consumed in that issuer's order (one
        // consumer per stage: no wait can run two phases ahead); (ps_k, pp_k) is issuer k's next slot and parity
        const int rs = a.S / nis;
        int ps0 = 0, ps1 = 0;
        uint32_t pp0 = 0, pp1 = 0;
        int p = 0;
        for (int it = 0; it < ntot; ++it) {
            const int ls = it % LS;
            const int kq = nis == 2 ? (p & 1) : 0;
            const int stg = kq + nis * (kq ? ps1 : ps0);
            if (!mbar_wait<PRODUCER_HINT_NS>(&lfull[ls], (uint32_t)((it / LS) & 1), &s_abort, a.err)) break;
            if (!mbar_wait<PRODUCER_HINT_NS>(&empty[stg], (kq ? pp1 : pp0) ^ 1u, &s_abort, a.err)) break;
            const unsigned char *slotb = ring + (size_t)ls * slotbytes;
            unsigned char *sbase = smem + (size_t)stg * stagebytes;
#pragma unroll
            for (int k = 0; k < MAXWI; ++k) {
                if (it_ts[k] < 0) break;
                const int ts = it_ts[k], op = it_op[k];
                const int g = GPI * it_gp[k] + sub;
                if (g >= ng) continue;
                const unsigned char *tsp = slotb + (uint32_t)ts * tsb;
                const float *gw = reinterpret_cast<const float *>(tsp + 8 * a.Qfp + 16);   // the weights
                const bool isA = op == 0;
                const float dlf = ((float)r - 0.5f * (TT - 1)) * (isA ? sp32x : sp32y);      // r < TT / 2: dl < 0
                // the ramp of row offset dl = m sp / 2 (m = 2 r - (TT - 1)) at sample q: -u dl (a0 + a1 q) cycles,
                // seeded at q = 8 g with step -u dl a1
                float2 wv, st;
                if (!BF && a.seeds) {
                    // float32 from the plan's seeds (Y = frac(u sp a0 / 2), V = u sp a1 / 2): m Y carries the
                    // phase modulo 1 exactly as m u sp a0 / 2 does, to float32's rounding of Y and V
                    const float4 sd = *reinterpret_cast<const float4 *>(tsp + 8 * a.Qfp);
                    const float Y = isA ? sd.x : sd.z, V = isA ? sd.y : sd.w;
                    const float m = (float)(2 * r - (TT - 1)), mv = m * V;
                    wv = cis_cycles(-fmaf(m, Y, mv * (8.f * (float)g)));
                    st = cis_cycles(-mv);
                } else {
                    const double u = *reinterpret_cast<const double *>(tsp + 8 * a.Qfp + (isA ? 0 : 8));
                    const double dl = ((double)r - 0.5 * (TT - 1)) * (isA ? a.spx : a.spy);
                    const double ud = -(u * dl);
                    wv = cis_cycles_d(ud * fma(a.a1, 8.0 * g, a.a0));
                    st = cis_cycles_d(ud * a.a1);
                }
                if (isA) { wv.x *= dscale; wv.y *= dscale; }
                float w1 = 1.f, w2 = 1.f;                       // the weights of rows r and 31 - r
                if (WEIGHTED) {
                    if (isA) { w1 = gw[0] + gw[1] * dlf; w2 = gw[0] - gw[1] * dlf; }
                    else { w1 = 1.f + gw[2] * dlf; w2 = 1.f - gw[2] * dlf; }
                }
                // operand base: A' or B'; half: bfloat16 hi (lo one half further), float16 the tile slot's; group g
                unsigned char *ob = sbase + (isA ? 0u : 2u * H) + (BF ? 0u : (uint32_t)ts * (isA ? HS : HB)) + (uint32_t)g * 128u;
                float r1[8], i1[8], r2[8], i2[8];
                if (isA) {
                    const float4 *dq = reinterpret_cast<const float4 *>(tsp + 64 * g);
#pragma unroll
                    for (int e2 = 0; e2 < 4; ++e2) {
                        const float4 dd = dq[e2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int e = 2 * e2 + h;
                            const float dr = h ? dd.z : dd.x, di = h ? dd.w : dd.y;
                            const float p1 = dr * wv.x, p2 = di * wv.y, p3 = dr * wv.y, p4 = di * wv.x;
                            if (FOLD) {
                                r1[e] = p1; i1[e] = p4; r2[e] = p3; i2[e] = p2;
                                wv = cmul(wv, st);
                                continue;
                            }
                            r1[e] = (p1 - p2) * w1; i1[e] = (p3 + p4) * w1;       // d x
                            r2[e] = (p1 + p2) * w2; i2[e] = (p4 - p3) * w2;       // d conj(x)
                            wv = cmul(wv, st);
                        }
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        r1[e] = wv.x * w1; i1[e] = wv.y * w1;
                        r2[e] = WEIGHTED ? wv.x * w2 : 0.f;
                        i2[e] = WEIGHTED ? -wv.y * w2 : 0.f;
                        wv = cmul(wv, st);
                    }
                }
                uint4 h, l;
                const bool mirror = !isA && !WEIGHTED && !FOLD, half = !isA && FOLD;
                pack8<OP>(r1, h, l);
                *reinterpret_cast<uint4 *>(ob + roff[0]) = h;
                if (BF) *reinterpret_cast<uint4 *>(ob + H + roff[0]) = l;
                if (mirror) {
                    *reinterpret_cast<uint4 *>(ob + roff[2]) = h;
                    if (BF) *reinterpret_cast<uint4 *>(ob + H + roff[2]) = l;
                }
                pack8<OP>(i1, h, l);
                *reinterpret_cast<uint4 *>(ob + roff[1]) = h;
                if (BF) *reinterpret_cast<uint4 *>(ob + H + roff[1]) = l;
                if (mirror) {
                    *reinterpret_cast<uint4 *>(ob + roff[3]) = flip_sign(h);
                    if (BF) *reinterpret_cast<uint4 *>(ob + H + roff[3]) = flip_sign(l);
                } else if (!half) {
                    pack8<OP>(r2, h, l);
                    *reinterpret_cast<uint4 *>(ob + roff[2]) = h;
                    if (BF) *reinterpret_cast<uint4 *>(ob + H + roff[2]) = l;
                    pack8<OP>(i2, h, l);
                    *reinterpret_cast<uint4 *>(ob + roff[3]) = h;
                    if (BF) *reinterpret_cast<uint4 *>(ob + H + roff[3]) = l;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[stg]);
                mbar_arrive(&lempty[ls]);
            }
            if (kq) {
                if (++ps1 == rs) { ps1 = 0; pp1 ^= 1u; }
            } else if (++ps0 == rs) {
                ps0 = 0;
                pp0 ^= 1u;
            }
            if (++p == a.Pf) p = 0;
        }
    } else if (warp >= NEPI) {
        // ------------------------------------------------------------------ MMA issue
        const int k = warp - NEPI;
        if (lane == 0 && k < nis) {
            const uint32_t idesc = (1u << 4) | ((BF ? 1u : 0u) << 7) | ((BF ? 1u : 0u) << 10) | (((uint32_t)NB >> 3) << 17) |
                                   ((128u >> 4) << 24);
            const uint32_t lbo = 128, sbo = (uint32_t)ng * 128;
            const int nks = a.Qfp / 16;
            // descriptors of stage 0's A' and B'; stage s adds s stagebytes, K step ks adds 256 bytes (16 units)
            const uint64_t da0 = smem_desc(smem0, lbo, sbo), db0 = smem_desc(smem0 + 2u * H, lbo, sbo);
            const uint64_t dstage = (uint64_t)(stagebytes >> 4);
            const int rs = a.S / nis;
            int slot = 0;                                       // this issuer's stages: k + nis slot
            uint32_t par = 0;
            // tests of the failure report: a wait that runs out before any MMA, as a stuck pipeline's would
            const bool stuck = a.test_wait_ns &&
                               !mbar_wait<ISSUER_HINT_NS>(&s_never, 0, &s_abort, a.err, a.test_wait_ns);
            // an accumulation j (segment sg of unit ul) goes into this issuer's accumulator j mod 2
            int sg = 0;
            for (int j = 0, nj = stuck ? 0 : nul * a.nsg; j < nj; ++j) {
                const int ab = j & 1;
                if (!mbar_wait<ISSUER_HINT_NS>(&acce[ab], (uint32_t)(((j >> 1) & 1) ^ 1), &s_abort, a.err)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t dt = tmem + (uint32_t)((k * 2 + ab) * 128);
                bool ok = true;
                uint32_t accum = 0;
                const int p1 = min(a.Pf, (sg + 1) * a.seg);
                for (int p = sg * a.seg + k; p < p1; p += nis) {
                    const int stg = k + nis * slot;
                    if (!mbar_wait<ISSUER_HINT_NS>(&full[stg], par, &s_abort, a.err)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = da0 + dstage * (uint64_t)stg, db = db0 + dstage * (uint64_t)stg;
                    for (int ks = 0; ks < nks; ++ks) {
                        mma_f16kind(dt, da + 16u * ks, db + 16u * ks, idesc, accum);
                        accum = 1u;
                    }
                    mma_commit(&empty[stg]);
                    if (++slot == rs) { slot = 0; par ^= 1u; }
                }
                if (!ok) break;
                mma_commit(&accf[ab]);
                if (++sg == a.nsg) sg = 0;
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue (warps 0..3)
        float *P0 = sP, *P1 = sP + 32 * 65;
        const float oscale = a.scale / (BF ? 1.f : operand_scale(a.amax, a.wexp));
        // after a failed wait a warp keeps stepping through the units (and the epilogue's named barriers, which all
        // four warps must reach) without waiting, reading or writing
        bool live = true;
        int j = 0;                                              // accumulations read
        for (int ul = 0; ul < nul; ++ul) {
            const uint32_t lanes = (uint32_t)(32 * warp) << 16;
            float *mine = (warp & 1) ? P1 : P0;                 // accumulator rows 32..63 (mod 64) are the Ai rows
            if (OP == OP_F16X2) {
                // The tensor core's float32 sums truncate: a chain of n of them loses about n 3e-8 of the result. So a
                // unit is accumulated in segments, added here in float32 with rounding. This thread's accumulator row,
                // hi and lo columns summed:
                constexpr int NV = TT;
                float v[NV];
#pragma unroll
                for (int i = 0; i < NV; ++i) v[i] = 0.f;
                const int c0 = TT == 32 ? 0 : 32 * (warp >> 1);
                for (int sg = 0; sg < a.nsg; ++sg, ++j) {
                    const int ab = j & 1, na = min(nis, a.Pf - sg * a.seg);   // issuers with a stage in the segment
                    if (live) live = mbar_wait<EPILOGUE_HINT_NS>(&accf[ab], (uint32_t)((j >> 1) & 1), &s_abort, a.err);
                    live = __all_sync(0xffffffffu, live);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (!live) continue;
                    for (int k = 0; k < na; ++k) {
                        const uint32_t base = tmem + lanes + (uint32_t)((k * 2 + ab) * 128 + c0);
#pragma unroll
                        for (int c = 0; c < NV; c += 16) {
                            uint32_t q0[16], q1[16];
                            tmem_ld16(base + (uint32_t)c, q0);
                            tmem_ld16(base + (uint32_t)(NV + c), q1);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; ++i) v[c + i] += __uint_as_float(q0[i]) + __uint_as_float(q1[i]);
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[ab]);
                }
                if (TT == 32) {
                    // warps 0, 1: the hi rows; then warps 2, 3 add the lo rows
                    float *part = sP + ((warp & 1) * 32 + lane) * (TT + 1);
                    if (live && warp < 2) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) part[i] = v[i];
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (live && warp >= 2) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) part[i] += v[i];
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (live) tile_fold<TT>(a, unit_tile<OP, TT>(ul, 0), sP, t, oscale);
                } else {
                    // tile slot ts = warp / 2: the hi rows in the even warp's lanes, the lo rows in the odd one's
                    const int ts = warp >> 1, tile = unit_tile<OP, TT>(ul, ts);
                    float *part = sP + ts * (32 * (TT + 1)) + lane * (TT + 1);
                    if (live && (warp & 1)) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) part[i] = v[i];
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (live && !(warp & 1)) {
#pragma unroll
                        for (int i = 0; i < NV; ++i) part[i] += v[i];
                        __syncwarp();
                        if (tile < a.B) tile_fold<TT>(a, tile, sP + ts * (32 * (TT + 1)), lane, oscale);
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                continue;
            }
            const int ab = ul & 1;
            if (live) live = mbar_wait<EPILOGUE_HINT_NS>(&accf[ab], (uint32_t)((ul >> 1) & 1), &s_abort, a.err);
            live = __all_sync(0xffffffffu, live);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the sum over the issuers' accumulators of columns [c0, c0 + 16), plus [c0 + c1, c0 + c1 + 16) if c1
            auto gather = [&](int c0, int c1, float *v) {
                uint32_t q0[16], q1[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.f;
                for (int k = 0; k < nis; ++k) {
                    const uint32_t base = tmem + lanes + (uint32_t)((k * 2 + ab) * 128);
                    tmem_ld16(base + (uint32_t)c0, q0);
                    if (c1) tmem_ld16(base + (uint32_t)(c0 + c1), q1);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(q0[j]) + (c1 ? __uint_as_float(q1[j]) : 0.f);
                }
            };
            if (OP == OP_BF16X2) {
                // warps 0, 1: hi rows (hi hi + hi lo); then warps 2, 3 add the lo rows (lo hi + lo lo)
                float v[16];
                if (live && warp < 2) {
#pragma unroll
                    for (int c0 = 0; c0 < 64; c0 += 16) {
                        gather(c0, 64, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) mine[lane * 65 + c0 + j] = v[j];
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[ab]);
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (live && warp >= 2) {
#pragma unroll
                    for (int c0 = 0; c0 < 64; c0 += 16) {
                        gather(c0, 64, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) mine[lane * 65 + c0 + j] += v[j];
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[ab]);
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (live) tile_pixels(a, unit_tile<OP, TT>(ul, 0), P0, P1, t, oscale);
                asm volatile("bar.sync 1, 128;" ::: "memory");
            } else if (FOLD && TT == 16) {
                // tile slot ts = warp: accumulator rows [32 ts, 32 ts + 32) (this warp's lane quarter) at columns
                // [16 ts, 16 ts + 16)
                if (live) {
                    float v[16], *part = sP + warp * (32 * (TT + 1));
                    gather(16 * warp, 0, v);
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[ab]);
                    const int tile = unit_tile<OP, TT>(ul, warp);
#pragma unroll
                    for (int i = 0; i < 16; ++i) part[lane * (TT + 1) + i] = v[i];
                    __syncwarp();
                    if (tile < a.B) tile_fold<TT>(a, tile, part, lane, oscale);
                    __syncwarp();
                }
            } else if (FOLD) {
                // tile slot ts: accumulator rows [64 ts, 64 ts + 64) and columns [32 ts, 32 ts + 32), read by warps 2 ts and
                // 2 ts + 1
                const int ts = warp >> 1;
                if (live) {
                    float v[16], *part = sP + (ts * 64 + (warp & 1) * 32 + lane) * (TT + 1);
#pragma unroll
                    for (int c0 = 0; c0 < 32; c0 += 16) {
                        gather(32 * ts + c0, 0, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) part[c0 + i] = v[i];
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[ab]);
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                for (int k = 0; k < 2; ++k) {
                    const int tile = unit_tile<OP, TT>(ul, k);
                    if (live && tile < a.B) tile_fold<TT>(a, tile, sP + k * 64 * (TT + 1), t, oscale);
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            } else if (TT == 16) {
                // tile slot ts = warp: accumulator rows [32 ts, 32 ts + 32) (this warp's lane quarter) at columns
                // [32 ts, 32 ts + 32)
                if (live) {
                    float v0[16], v1[16];
                    gather(32 * warp, 0, v0);
                    gather(32 * warp + 16, 0, v1);
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[ab]);
                    tile16_pixels(a, unit_tile<OP, TT>(ul, warp), v0, v1, lane, oscale);
                }
            } else {
                // tile slot ts: accumulator rows and columns [64 ts, 64 ts + 64), read by warps 2 ts and 2 ts + 1
                for (int ts = 0; ts < 2; ++ts) {
                    if (live && (warp >> 1) == ts) {
                        float v[16];
#pragma unroll
                        for (int c0 = 0; c0 < 64; c0 += 16) {
                            gather(64 * ts + c0, 0, v);
#pragma unroll
                            for (int j = 0; j < 16; ++j) mine[lane * 65 + c0 + j] = v[j];
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&acce[ab]);
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    const int tile = unit_tile<OP, TT>(ul, ts);
                    if (live && tile < a.B) tile_pixels(a, tile, P0, P1, t, oscale);
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
            }
        }
    }

    // teardown: every role is done (or aborted); each issuer drains its MMAs before the accumulators are freed
    __syncthreads();
    if (warp >= NEPI && warp < NEPI + NISS && lane == 0) {
        // a commit on a fresh barrier arrives once every earlier MMA of this thread has completed
        uint64_t *dr = &drain[warp - NEPI];
        mma_commit(dr);
        const uint64_t t0 = global_ns();
        bool drained = false;
        while (!(drained = mbar_test(dr, 0)) && global_ns() - t0 < WAIT_NS) {
        }
        if (!drained && a.err) atomicAdd(a.err, 1);              // an MMA still running: reported
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == NEPI) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TMEM_COLS));
}

__global__ void final_seeds_kernel(const double *__restrict__ ux, const double *__restrict__ uy, long n, double spx,
                                   double spy, double a0, double a1, float4 *__restrict__ out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double yx = 0.5 * ux[i] * spx * a0, yy = 0.5 * uy[i] * spy * a0;
        out[i] = make_float4((float)(yx - floor(yx)), (float)(0.5 * ux[i] * spx * a1), (float)(yy - floor(yy)),
                             (float)(0.5 * uy[i] * spy * a1));
    }
}

// The split float16 form's seeds of one ramp: Y = frac(u sp a0 / 2) and V = u sp a1 / 2 as hi + lo, Y's high part of 18
// bits (times a row's m, |m| < 32, exact) and V's of 11 (times 8 g m, below 2^13, exact).
__device__ __forceinline__ float4 split_seed(double u, double sp, double a0, double a1)
{
    const double y = 0.5 * u * sp * a0, V = 0.5 * u * sp * a1, Y = y - floor(y);
    const float yh = (float)(rint(Y * 262144.0) / 262144.0), vf = (float)V, t = vf * 8193.f, vh = t - (t - vf);
    return make_float4(yh, (float)(Y - (double)yh), vh, (float)(V - (double)vh));
}

__global__ void final_seeds2_kernel(const double *__restrict__ ux, const double *__restrict__ uy, long n, double spx,
                                    double spy, double a0, double a1, float4 *__restrict__ out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        out[2 * i] = split_seed(ux[i], spx, a0, a1);
        out[2 * i + 1] = split_seed(uy[i], spy, a0, a1);
    }
}

}  // namespace

cudaError_t launch_final_seeds2(const double *ux, const double *uy, long n, double spx, double spy, double a0,
                                double a1, float4 *out, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const long nb = (n + 255) / 256;
    final_seeds2_kernel<<<(int)(nb < 4096 ? nb : 4096), 256, 0, s>>>(ux, uy, n, spx, spy, a0, a1, out);
    return cudaGetLastError();
}

cudaError_t launch_final_seeds(const double *ux, const double *uy, long n, double spx, double spy, double a0,
                               double a1, float4 *out, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const long nb = (n + 255) / 256;
    final_seeds_kernel<<<(int)(nb < 4096 ? nb : 4096), 256, 0, s>>>(ux, uy, n, spx, spy, a0, a1, out);
    return cudaGetLastError();
}

namespace {

struct TcShape { int nts, nwi, maxwi, S; size_t smem; };

// The unit and the ring of a final stage's shape (op: Operands); false with *why for shapes the kernel does not cover.
bool tc_shape(int op, bool weighted, int T, int Pf, int Qf, size_t maxsmem, TcShape *o, const char **why)
{
    const bool split = op != OP_F16;
    if (T != 32 && (T != 16 || op == OP_BF16X2)) {
        *why = "the tensor-core final stage takes T = 32, or T = 16 (float16 or split float16)";
        return false;
    }
    // warp items per stage: (tile slots) x (A, B) x (pairs of 8-sample groups) over the NPW producer warps
    const int Qfp = (Qf + 15) & ~15, gpi = 64 / T, hg = ((op == OP_F16X2 ? (Qf + 7) / 8 : Qfp / 8) + gpi - 1) / gpi;
    o->nts = (split ? 32 : 64) / T;
    o->nwi = o->nts * 2 * hg;
    o->maxwi = (o->nwi + NPW - 1) / NPW;
    if (o->maxwi > 4) { *why = "more than 256 frequency samples per final tile"; return false; }
    const int nis = Pf >= NISS ? NISS : 1;
    const size_t stage = (size_t)4 * 64 * Qfp * 2;
    const size_t slotbytes = (size_t)o->nts * (8 * Qfp + 32 + (op == OP_F16X2 ? 8 * T : 0));
    const size_t fixed = (size_t)2 * 32 * 65 * 4 + (size_t)LS * slotbytes + (size_t)(2 * 4 + 6 + 2 * LS) * 8;
    const size_t avail = maxsmem - 1024;                        // static shared memory and slack
    // stages: a multiple of the issuers (each owns S / nis of them)
    int S = 4;
    while (S > 2 && ((size_t)S * stage + fixed > avail || S % nis)) --S;
    if ((size_t)S * stage + fixed > avail) {
        *why = "a final subaperture's operands do not fit shared memory (Qf too large for the tensor-core stage)";
        return false;
    }
    o->S = S;
    o->smem = (size_t)S * stage + fixed;
    if (op != OP_BF16X2 && !weighted) {                         // folded operands: three quarters of a stage (what fits is
        const size_t st3 = stage / 4 * 3, fx3 = fixed + 2 * 64 * 4 + (2 * FS - 8) * 8;   // decided above, as before)
        for (S = FS; S > 2 && ((size_t)S * st3 + fx3 > avail || S % nis); --S) {}
        o->S = S;
        o->smem = (size_t)S * st3 + fx3;
    }
    return true;
}

size_t max_smem()
{
    int dev = 0, v = 227 * 1024;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return (size_t)v;
}

}  // namespace

bool final_tc32_supported(int T, int B, int Pf, int Qf)
{
    const char *why = nullptr;
    TcShape o;
    return (long long)B * Pf < (1LL << 31) && tc_shape(OP_F16X2, false, T, Pf, Qf, max_smem(), &o, &why);
}

cudaError_t launch_final_tc(const FinalLaunch &F, int mode, cudaStream_t s, const char **why)
{
    *why = nullptr;
    const int op = mode == 0 ? OP_F16X2 : (mode == 2 ? OP_BF16X2 : OP_F16);
    TcShape o;
    if (!tc_shape(op, F.w != nullptr, F.T, F.Pf, F.Qf, max_smem(), &o, why)) return cudaErrorNotSupported;
    if (F.B <= 0) return cudaSuccess;
    if ((long long)F.B * F.Pf >= (1LL << 31)) { *why = "more than 2^31 final tile subapertures"; return cudaErrorNotSupported; }
    TcArgs a;
    a.d = F.d; a.B = F.B; a.Pf = F.Pf; a.Qf = F.Qf; a.Qfp = (F.Qf + 15) & ~15;
    a.nunits = (F.B + o.nts - 1) / o.nts;
    a.nis = F.Pf >= NISS ? NISS : 1;
    a.nwi = o.nwi; a.S = o.S;
    // when every producer warp gets the same even number of items they are interleaved (as many A items, the heavier,
    // as B items on each warp: 3 % faster at 47 x 91 in float16; 1 % slower at 38 x 71, whose count is uneven)
    a.interleave = o.nwi % (2 * NPW) == 0 ? 1 : 0;
    // split float16: accumulations of about 24 steps (an even count of subapertures for two issuers)
    const int per = std::max(1, 24 / (a.Qfp / 16));
    a.seg = op == OP_F16X2 ? std::min(F.Pf, a.nis * per) : F.Pf;
    a.nsg = (F.Pf + a.seg - 1) / a.seg;
    a.ux = F.ux; a.uy = F.uy; a.seeds = F.seeds; a.spx = F.spx; a.spy = F.spy; a.a0 = F.a0; a.a1 = F.a1; a.fc2 = F.fc2;
    a.ucx = F.ucx; a.ucy = F.ucy; a.rc = F.rc; a.w = F.w; a.tiles = F.tiles; a.img = F.img; a.first = F.first;
    a.nx = F.nx; a.ny = F.ny; a.ox = F.ox; a.oy = F.oy; a.scale = F.scale; a.err = F.err; a.amax = F.amax; a.wexp = F.w ? F.wexp : 0;
    a.test_wait_ns = F.test_wait_ns;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int grid = a.nunits < nsm ? a.nunits : nsm;
    auto run = [&](auto kern, int threads) -> cudaError_t {
        cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)o.smem);
        if (r != cudaSuccess) return r;
        kern<<<grid, threads, o.smem, s>>>(a);
        return cudaGetLastError();
    };
#define FFBP_TC_ONE(OP, W, MW, TT) run(final_tc_kernel<OP, W, MW, TT>, block_threads<OP, W, MW, TT>())
    if (op == OP_F16X2) {
        // weighted tiles: a pulse's weight has no bound that float16's range could be held to
        if (a.w || !a.seeds) { *why = "the split float16 final stage takes the plan's seeds and no aperture weights"; return cudaErrorNotSupported; }
        return F.T == 16 ? FFBP_TC_ONE(OP_F16X2, false, 1, 16) : FFBP_TC_ONE(OP_F16X2, false, 1, 32);
    }
#define FFBP_TC_RUN(MW)                                                                                         \
    (op == OP_BF16X2 ? (a.w ? FFBP_TC_ONE(OP_BF16X2, true, MW, 32) : FFBP_TC_ONE(OP_BF16X2, false, MW, 32))          \
     : F.T == 16     ? (a.w ? FFBP_TC_ONE(OP_F16, true, MW, 16) : FFBP_TC_ONE(OP_F16, false, MW, 16))                \
                     : (a.w ? FFBP_TC_ONE(OP_F16, true, MW, 32) : FFBP_TC_ONE(OP_F16, false, MW, 32)))
    return o.maxwi <= 1 ? FFBP_TC_RUN(1) : o.maxwi <= 2 ? FFBP_TC_RUN(2) : FFBP_TC_RUN(4);
#undef FFBP_TC_RUN
#undef FFBP_TC_ONE
}

}  // namespace ffbp
