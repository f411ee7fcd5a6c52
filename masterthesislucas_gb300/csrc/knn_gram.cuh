// Candidate filter of the exact kNN on the tensor cores.
//
// The distances that define the neighbours (FP32, the dimensions in order) are
// a few operations a pair on the FP32 pipe; a matrix product gives them
// approximately at some fifty times the rate:
//     a_ij = |x_i|^2 + |x_j|^2 - 2 x_i . x_j,
// with x split into bfloat16 high and low parts and the products high-high,
// high-low and low-high accumulated in FP32 (high-high alone when every input
// is a bfloat16 number, as 8-bit pixels / 256 are).  With a bound E on
// |a_ij - d_ij|, the k-th smallest d of a row is at most (its k-th smallest a)
// + E, so every neighbour has a_ij <= (k-th smallest a) + 2 E.  The pairs that
// pass, some 120 of 20,000 for k = 90, get their defining distance and are
// ordered by (distance, index): the result is exact, whatever a_ij is within E.
//
// E, from nu_i = |x_i| and the largest nu:
// * the parts dropped: |l_i . l_j| + 2 |r| |x| <= 3 2^-18 nu_i nu_j (bfloat16
//   rounds to 2^-9, the second part's remainder to 2^-18);
// * the accumulation: an MMA step adds 16 products to the accumulator; a step
//   may lose 2^-20 of |x_i| |x_j| here, four times what FP32 sums that truncate
//   after aligning to the largest term would;
// * the norms and the final sum, FP32: 2^-21 (nu_i^2 + nu_j^2);
// * d_ij itself: (dim + 3) roundings, relative (its terms are positive).
// Rows with more candidates than the list holds (many equal distances, or
// distances small against the norms) flag their block of query rows, which
// k_knn then computes in full, and so does a non-finite or huge input or a
// bounded wait that gives up: all blocks.
#pragma once

#include "common.cuh"
#include "tcgen05.cuh"

namespace tc {
namespace {

constexpr int kGramRows = 128, kGramCols = 256;  // tile of a CTA (one accumulator: 256 tensor-memory columns)
constexpr int kGramK = 64;                       // dimensions per stage
constexpr int kGramStages = 4;
constexpr int kGramA = kGramRows * kGramK * 2, kGramB = kGramCols * kGramK * 2;
constexpr int kGramSmem = kGramStages * (kGramA + kGramB) + 1024;
constexpr int kGramThreads = 192;  // a producer warp, an MMA warp, four epilogue warps
constexpr int kCand = 384;         // candidates a row may have
constexpr int kSelT = 128;         // threads of the selection
constexpr int kSelGroups = 256;    // groups of a row whose smallest values bound it (at most; more than k are needed)
constexpr float kGramHuge = 1.0e15f;

struct GramStat {
    uint32_t bad;      // a non-finite or huge input, or a wait that gave up
    uint32_t any_lo;   // some input has a low part
    uint32_t nu_max;   // bits of the largest norm
    uint32_t nflagged; // query blocks for k_knn (their list follows the flags)
};

__host__ __device__ inline int64_t gram_block_bytes(int dimp) { return (int64_t)dimp / 8 * 4096; }

// Inputs as BF16 high and low parts in blocks of 256 rows, each block in the
// MMA's K-major layout without swizzle (8-row x 16-byte core matrices, 128
// bytes apart along the rows, 4096 along K), so that a stage is one or a few
// contiguous pieces; squared norms; a warp per row.  Rows past n are zero with
// an infinite norm.
__global__ void __launch_bounds__(256)
    k_gram_split(const float* __restrict__ x, int64_t n, int dim, int dimp, uint8_t* __restrict__ hi,
                 uint8_t* __restrict__ lo, float* __restrict__ s, GramStat* __restrict__ st)
{
    const int lane = threadIdx.x & 31;
    const int64_t r = blockIdx.x * 8ll + (threadIdx.x >> 5);
    const int64_t at = (r >> 8) * gram_block_bytes(dimp) + ((r & 255) >> 3) * 128 + (r & 7) * 16;
    double sum = 0.0;
    bool bad = false, low = false;
    for (int k8 = lane; k8 < dimp / 8; k8 += 32) {
        uint32_t hw[4], lw[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t h2 = 0, l2 = 0;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int k = 8 * k8 + 2 * j + e;
                const float v = r < n && k < dim ? x[r * dim + k] : 0.f;
                bad |= !(fabsf(v) <= kGramHuge);
                const __nv_bfloat16 h = __float2bfloat16_rn(v);
                const float rest = v - __bfloat162float(h);
                low |= rest != 0.f;
                sum = fma((double)v, (double)v, sum);
                h2 |= (uint32_t)__bfloat16_as_ushort(h) << (16 * e);
                l2 |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(rest)) << (16 * e);
            }
            hw[j] = h2;
            lw[j] = l2;
        }
        *reinterpret_cast<uint4*>(hi + at + k8 * 4096ll) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        *reinterpret_cast<uint4*>(lo + at + k8 * 4096ll) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
    }
    sum = warp_sum(sum);
    bad = __any_sync(0xffffffffu, bad);
    low = __any_sync(0xffffffffu, low);
    if (lane == 0) {
        s[r] = r < n ? (float)sum : INFINITY;
        if (bad) atomicOr(&st->bad, 1u);
        if (low) atomicOr(&st->any_lo, 1u);
        // rounded up; norms are not negative, so their bits order as they do
        if (!bad) atomicMax(&st->nu_max, __float_as_uint(sqrtf((float)sum) * (1.0f + 1e-6f)));
    }
}

// a_ij for the 128-row blocks [rb0, rb0 + nrb) against every column, tile after
// tile (row blocks first) and column after column in a tile, which is how a
// warp's lanes hold them (a row's own order would take a line per lane and
// store); and the smallest of every four columns, pitch npad / 4.
// Bound by the operands' way from L2 (a 128 x 256 tile reads 48 KB per 64
// dimensions) and, for few dimensions, by writing a_ij.  One CTA per SM walks
// the tiles; the accumulators alternate, so a tile is written out while the
// next one is multiplied.  20,224 x 20,224 x 784, high parts only: 819 us in all.
__global__ void __launch_bounds__(kGramThreads, 1)
    k_gram(const uint8_t* __restrict__ hi, const uint8_t* __restrict__ lo, const float* __restrict__ s, int64_t n,
           int64_t npad, int dimp, int64_t rb0, int nrb, float* __restrict__ out, float* __restrict__ gmin,
           GramStat* __restrict__ st)
{
    using namespace tcm;
    constexpr uint32_t IDESC = idesc_bf16(kGramRows, kGramCols);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[kGramStages], empty[kGramStages], tfull[2], tempty[2];
    __shared__ __align__(16) float s_norm[4][kGramCols];
    __shared__ uint32_t s_tmem;
    __shared__ volatile uint32_t s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t bb = gram_block_bytes(dimp);
    const int64_t ntiles = (npad / kGramCols) * nrb;
    if (tid == 0) {
        for (int i = 0; i < kGramStages; i++) {
            mbar_init(saddr(full + i), 1);
            mbar_init(saddr(empty + i), 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(saddr(tfull + i), 1);
            mbar_init(saddr(tempty + i), 4);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&s_tmem)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int npass = st->any_lo ? 3 : 1, chunks = (dimp + kGramK - 1) / kGramK, k8s = dimp / 8;
    auto stage_a = [&](uint32_t i) { return smem + (i % kGramStages) * (kGramA + kGramB); };
    auto stage_b = [&](uint32_t i) { return stage_a(i) + kGramA; };
    // false when the wait gave up here or elsewhere in the CTA
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (!s_abort && mbar_wait(saddr(bar), parity)) return true;
        s_abort = 1;
        return false;
    };
    uint32_t it = 0;  // stages issued (producer) or consumed (MMA)
    if (warp == 0 && lane == 0) {
        for (int64_t t = blockIdx.x; t < ntiles && !s_abort; t += gridDim.x) {
            const int64_t cb = t / nrb, rb = rb0 + t % nrb;
            for (int p = 0; p < npass; p++) {
                const uint8_t* a = (p == 2 ? lo : hi) + (rb >> 1) * bb + (rb & 1) * 2048;
                const uint8_t* b = (p == 1 ? lo : hi) + cb * bb;
                for (int c = 0; c < chunks; c++, it++) {
                    const uint32_t st_i = it % kGramStages;
                    if (it >= (uint32_t)kGramStages && !wait(empty + st_i, ((it / kGramStages) - 1) & 1)) break;
                    const int nk = min(kGramK / 8, k8s - c * (kGramK / 8));
                    const uint32_t bar = saddr(full + st_i), da = saddr(stage_a(it)), db = saddr(stage_b(it));
                    mbar_expect_tx(bar, (uint32_t)nk * (2048 + 4096));
                    for (int k = 0; k < nk; k++)
                        bulk_g2s(da + k * 2048, a + (int64_t)(c * (kGramK / 8) + k) * 4096, 2048, bar);
                    bulk_g2s(db, b + (int64_t)c * (kGramK / 8) * 4096, (uint32_t)nk * 4096, bar);
                }
                if (s_abort) break;
            }
        }
        // an abandoned walk: the copies in flight land before the CTA leaves
        if (s_abort)
            for (uint32_t i = it >= (uint32_t)kGramStages ? it - kGramStages : 0; i < it; i++)
                mbar_wait(saddr(full + i % kGramStages), (i / kGramStages) & 1);
    } else if (warp == 1 && lane == 0) {
        uint32_t tile = 0;
        for (int64_t t = blockIdx.x; t < ntiles && !s_abort; t += gridDim.x, tile++) {
            const uint32_t buf = tile & 1;
            if (tile >= 2 && !wait(tempty + buf, ((tile >> 1) - 1) & 1)) break;
            tc_fence_after();
            uint32_t acc = 0;
            for (int p = 0; p < npass && !s_abort; p++) {
                for (int c = 0; c < chunks; c++, it++) {
                    const uint32_t st_i = it % kGramStages;
                    if (!wait(full + st_i, (it / kGramStages) & 1)) break;
                    tc_fence_after();
                    const int nk = min(kGramK / 8, k8s - c * (kGramK / 8));
                    const uint32_t da = saddr(stage_a(it)), db = saddr(stage_b(it));
                    for (int k = 0; k < nk; k += 2) {
                        mma_bf16(tmem + buf * kGramCols, sdesc(da + k * 2048, 2048, 128), sdesc(db + k * 4096, 4096, 128),
                                 IDESC, acc);
                        acc = 1;
                    }
                    mma_commit(saddr(empty + st_i));
                }
            }
            mma_commit(saddr(tfull + buf));
        }
        // an abandoned walk: the MMAs in flight finish (a commit covers all of them) before the memory is freed
        if (s_abort && it > 0) mbar_wait(saddr(empty + (it - 1) % kGramStages), ((it - 1) / kGramStages) & 1);
    } else if (warp >= 2) {
        const int q = warp & 3;  // the tensor-memory lanes this warp may read: rows 32 q on
        uint32_t tile = 0;
        for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x, tile++) {
            const uint32_t buf = tile & 1;
            const int64_t cb = t / nrb, rl = t % nrb;
            const int64_t lrow = rl * kGramRows + q * 32 + lane, row = rb0 * kGramRows + lrow;
            const float si = s[row];
            // the columns' norms, while the tile is multiplied
            __syncwarp();
#pragma unroll
            for (int c = lane; c < kGramCols / 4; c += 32)
                reinterpret_cast<float4*>(s_norm[q])[c] = __ldg(reinterpret_cast<const float4*>(s + cb * kGramCols) + c);
            __syncwarp();
            bool ok = wait(tfull + buf, (tile >> 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const float4* sj = reinterpret_cast<const float4*>(s_norm[q]);
            float* o = out + (cb * nrb + rl) * (kGramRows * kGramCols) + q * 32 + lane;
            float4* om = reinterpret_cast<float4*>(gmin + (lrow * npad + cb * kGramCols) / 4);
            const uint32_t trow = tmem + buf * kGramCols + ((uint32_t)(q * 32) << 16);
            for (int c = 0; c < kGramCols / 32; c++) {
                float g[32];
                tmem_ld32(trow + 32 * c, g);
                if (row < n) {
                    float mn[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 v = sj[8 * c + j];
                        const float4 a =
                            make_float4(fmaf(-2.f, g[4 * j], si + v.x), fmaf(-2.f, g[4 * j + 1], si + v.y),
                                        fmaf(-2.f, g[4 * j + 2], si + v.z), fmaf(-2.f, g[4 * j + 3], si + v.w));
                        float* oc = o + (32 * c + 4 * j) * kGramRows;
                        oc[0] = a.x;
                        oc[kGramRows] = a.y;
                        oc[2 * kGramRows] = a.z;
                        oc[3 * kGramRows] = a.w;
                        mn[j] = fminf(fminf(a.x, a.y), fminf(a.z, a.w));
                    }
                    om[2 * c] = make_float4(mn[0], mn[1], mn[2], mn[3]);
                    om[2 * c + 1] = make_float4(mn[4], mn[5], mn[6], mn[7]);
                }
                __syncwarp();  // the next load takes the warp as a whole, also where its rows end
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(saddr(tempty + buf));
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_abort) atomicOr(&st->bad, 1u);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// The neighbours of one row: a block each.  The smallest values of a_ij in
// kSelGroups groups of the row give the bound: the (k + 1)-th smallest of them
// is no smaller than the k-th smallest a_ij of another point, and lets some
// 20 % more pass.  Only the fours whose smallest passes are read.  The listed
// pairs' distances are summed as k_knn sums them, a thread per pair; a warp
// brings its 32 rows' next 32 dimensions into shared memory in whole lines (a
// thread reading its own row takes a line per lane and load).  Ranked by
// counting.  Shared memory bounds it at many dimensions (some 100 accesses of
// 128 bytes per 32 dimensions of 32 candidates): 20,000 x 784, k = 90: 1.9 ms;
// at few, reading a_ij did: all of 20,000 x 4 took 1.65 ms with a_ij read twice
// in full, 1.13 with the fours.
constexpr int kSelPitch = 36;  // floats of a staged row: 32 dimensions, its 16-byte pieces in different banks

template <bool kVec>
__global__ void __launch_bounds__(kSelT, 8)
    k_knn_select(const float* __restrict__ x, int64_t n, int dim, int dimp, int k, const float* __restrict__ gram,
                 const float* __restrict__ gmin, int64_t npad, int64_t nrb, int64_t row0, const float* __restrict__ s,
                 const GramStat* __restrict__ st, float* __restrict__ out_d, int32_t* __restrict__ out_i,
                 uint32_t* __restrict__ qflag, int qrows)
{
    extern __shared__ __align__(16) float s_row[];  // [dim, rounded up to 32], zeros past dim
    __shared__ __align__(16) float s_stage[kSelT / 32][32 * kSelPitch];
    __shared__ __align__(16) float s_min[kSelGroups];
    __shared__ uint32_t s_cnt, s_fours;
    __shared__ int32_t s_cand[kCand];
    __shared__ unsigned long long s_key[kCand];
    int32_t* s_four = reinterpret_cast<int32_t*>(s_key);  // before the keys
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t i = row0 + blockIdx.x;
    if (st->bad) return;  // k_knn computes all rows
    const float4* m4 = reinterpret_cast<const float4*>(gmin + blockIdx.x * (npad / 4));
    // a_ij of column j: g[(j / 256) nrb 32768 + (j mod 256) 128]
    const float* g = gram + (int64_t)(blockIdx.x / kGramRows) * (kGramRows * kGramCols) + blockIdx.x % kGramRows;
    const int nm = (int)(npad / 16);
    // group 2 tid holds the first halves of this thread's pieces, 2 tid + 1 the second halves
    float2 mn = make_float2(INFINITY, INFINITY);
#pragma unroll 4
    for (int v = tid; v < nm; v += kSelT) {
        const float4 a = m4[v];
        mn.x = fminf(mn.x, fminf(a.x, a.y));
        mn.y = fminf(mn.y, fminf(a.z, a.w));
    }
    *reinterpret_cast<float2*>(s_min + 2 * tid) = mn;
    if (tid == 0) s_cnt = s_fours = 0;
    for (int d = tid; d < ((dim + 31) & ~31); d += kSelT) s_row[d] = d < dim ? x[i * dim + d] : 0.f;
    __syncthreads();
    // the (k + 1)-th smallest, rounded up to its leading 20 bits: every warp searches its bits from the top
    float thr;
    {
        uint32_t key[kSelGroups / 32];
#pragma unroll
        for (int u = 0; u < kSelGroups / 32; u++)
            key[u] = __float_as_uint(fmaxf(s_min[32 * u + lane], 0.f));  // a_ij below zero count as zero
        uint32_t pre = 0;
#pragma unroll 1
        for (uint32_t bit = 1u << 30; bit >= 1u << 12; bit >>= 1) {
            const uint32_t top = pre | (bit - 1u);  // the largest value without this bit
            int c = 0;
#pragma unroll
            for (int u = 0; u < kSelGroups / 32; u++) c += key[u] <= top;
            if (__reduce_add_sync(0xffffffffu, c) <= k) pre |= bit;
        }
        const float bound = __uint_as_float(pre | 0xFFFu);
        // E as at the top of this file, every factor rounded up
        const float nu = sqrtf(s[i]) * (1.0f + 1e-6f), num = __uint_as_float(st->nu_max);
        const float steps = (float)((st->any_lo ? 3 : 1) * (dimp / 16) + 8);
        const float e = nu * num * (2.1f * steps * 0x1p-20f + (st->any_lo ? 0x1p-15f : 0.f)) +
                        0x1p-21f * (nu * nu + num * num) + 1e-30f;
        const float gam = 1.1f * 0x1p-24f * (float)(dim + 8);
        thr = ((bound + e) * (1.0f + 3.0f * gam) + e) * (1.0f + 1e-6f);
    }
    if (!(thr < INFINITY)) {  // fewer than k + 1 groups of the row hold a point
        if (tid == 0) qflag[i / qrows] = 1u;
        return;
    }
    // the fours with a small enough value, then their values
    auto four = [&](float smallest, int v) {
        if (!(smallest <= thr)) return;
        const uint32_t c = atomicAdd(&s_fours, 1u);
        if (c < (uint32_t)kCand) s_four[c] = v;
    };
#pragma unroll 4
    for (int v = tid; v < nm; v += kSelT) {
        const float4 a = m4[v];
        four(a.x, 4 * v);
        four(a.y, 4 * v + 1);
        four(a.z, 4 * v + 2);
        four(a.w, 4 * v + 3);
    }
    __syncthreads();
    const int nf = (int)s_fours;
    for (int f = tid; f < min(nf, kCand); f += kSelT) {
        const int v = s_four[f];
        const float* a = g + (int64_t)(v >> 6) * nrb * (kGramRows * kGramCols) + (v & 63) * (4 * kGramRows);
        const float av[4] = {a[0], a[kGramRows], a[2 * kGramRows], a[3 * kGramRows]};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (av[j] <= thr && 4ll * v + j != i) {
                const uint32_t c = atomicAdd(&s_cnt, 1u);
                if (c < (uint32_t)kCand) s_cand[c] = 4 * v + j;
            }
        }
    }
    __syncthreads();
    const int m = (int)s_cnt;
    if (nf > kCand || m > kCand) {
        if (tid == 0) qflag[i / qrows] = 1u;
        return;
    }
    for (int c0 = 32 * warp; c0 < m; c0 += kSelT) {
        const int c = c0 + lane;
        const int32_t j = s_cand[c < m ? c : c0];
        float d = 0.f;
        if (kVec) {
            float* stage = s_stage[warp];
            const float* y = x + (int64_t)j * dim;
            // row r of the stage is lane r's: eight lanes bring 128 bytes of it, four rows at a time
            const int piece = lane & 7;
            const float* rows[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
                rows[u] = reinterpret_cast<const float*>(
                              __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(y), 4 * u + (lane >> 3))) +
                          4 * piece;
            float4 next[8];
            auto load = [&](int t0) {
#pragma unroll
                for (int u = 0; u < 8; u++)
                    next[u] = t0 + 4 * piece < dim ? *reinterpret_cast<const float4*>(rows[u] + t0)
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
            };
            load(0);
            for (int t0 = 0; t0 < dim; t0 += 32) {
#pragma unroll
                for (int u = 0; u < 8; u++)
                    *reinterpret_cast<float4*>(stage + (4 * u + (lane >> 3)) * kSelPitch + 4 * piece) = next[u];
                __syncwarp();
                load(t0 + 32);
#pragma unroll
                for (int t = 0; t < 32; t += 4) {  // dimensions past the end add (0 - 0)^2
                    const float4 b = *reinterpret_cast<const float4*>(stage + lane * kSelPitch + t);
                    const float4 a = *reinterpret_cast<const float4*>(s_row + t0 + t);
                    const float d0 = a.x - b.x, d1 = a.y - b.y, d2 = a.z - b.z, d3 = a.w - b.w;
                    d = fmaf(d0, d0, d);
                    d = fmaf(d1, d1, d);
                    d = fmaf(d2, d2, d);
                    d = fmaf(d3, d3, d);
                }
                __syncwarp();
            }
        } else {
            const float* y = x + (int64_t)j * dim;
#pragma unroll 4
            for (int t = 0; t < dim; t++) {
                const float d0 = s_row[t] - y[t];
                d = fmaf(d0, d0, d);
            }
        }
        if (c < m) s_key[c] = (unsigned long long)__float_as_uint(d) << 32 | (uint32_t)j;
    }
    __syncthreads();
    for (int c = tid; c < m; c += kSelT) {
        const unsigned long long key = s_key[c];
        int rank = 0;
        for (int t = 0; t < m; t++) rank += s_key[t] < key;
        if (rank < k) {
            out_d[i * k + rank] = __uint_as_float((uint32_t)(key >> 32));
            out_i[i * k + rank] = (int32_t)(uint32_t)key;
        }
    }
}

// the flagged query blocks in order (all of them when *bad), one block
__global__ void __launch_bounds__(1024) k_knn_flagged(const uint32_t* __restrict__ qflag, int64_t qblocks,
                                                      GramStat* __restrict__ st, uint32_t* __restrict__ list)
{
    uint32_t base = 0;
    const bool all = st->bad != 0;
    for (int64_t q0 = 0; q0 < qblocks; q0 += blockDim.x) {
        const int64_t q = q0 + threadIdx.x;
        const uint32_t f = q < qblocks && (all || qflag[q]) ? 1u : 0u;
        uint32_t tot;
        const uint32_t at = base + block_exclusive_scan(f, tot);
        if (f) list[at] = (uint32_t)q;
        base += tot;
    }
    if (threadIdx.x == 0) st->nflagged = base;
}

}  // namespace
}  // namespace tc
