// The t-SNE affinity matrix P on the GPU: exact k nearest neighbours, the
// per-point Gaussian bandwidth calibrated to a perplexity, and the symmetric
// CSR matrix (P + P^T) / (2N).
//
// The reference builds P offline with openTSNE (MnistLoader.ipynb cell 14:
// PerplexityBasedNN with k = 3 * perplexity, symmetrize=True, written with
// mmwrite) and reads it into CSR in TSNE::setupEfficientPmatrix
// (src/nBodyInstances/tsne.h:462-520: rows sorted, columns sorted within a
// row).  openTSNE is not available, so this file restates the published
// algorithm; every operation is defined so that the CPU restatement in the
// oracle (orc_knn, orc_perplexity, orc_symmetrize) gives the same bits:
// * distances: d_ij = sum_t (x_it - x_jt)^2 in FP32, t = 0..dim-1 in order,
//   each step one fused multiply-add; neighbours ordered by (d, j), self
//   excluded;
// * bandwidths: per row a bisection on beta (start 1, doubling until
//   bracketed) of H = log(s) + beta * sum_j d'_j w_j / s with
//   w_j = exp(-beta d'_j), d'_j = d_j - d_min, s = sum_j w_j (FP64, j in
//   order), stopping when |H - log(perplexity)| < tol; p_j = w_j / s;
// * exp and log in FP64 written here from the mathematics (a two-constant
//   reduction by ln 2 with a degree-13 Taylor polynomial; the atanh series of
//   log m on [sqrt(1/2), sqrt(2))), so no vendor math routine is involved;
// * symmetrisation: each stored p_ij contributes p_ij / (2N) to (i, j) and to
//   (j, i); the (at most two) contributions to an entry are added.
// This file is compiled without FMA contraction: the fused operations above
// are the explicit fma / fmaf calls.
#include <mutex>

#include "common.cuh"
#include "knn_gram.cuh"

namespace tc {
namespace {

// sizes the tensor-core filter takes (tc_knn_device) and its scratch for a_ij
#ifndef TC_KNN_GRAM_MIN_N
#define TC_KNN_GRAM_MIN_N 1024
#endif
constexpr int64_t kGramMinN = TC_KNN_GRAM_MIN_N;
constexpr int kGramMaxDim = 4096;
constexpr int64_t kGramBytes = 256ll << 20;

// ------------------------------------------------------------------ exp, log
constexpr double kLn2Hi = 0x1.62e42fee00000p-1;   // ln 2 to 32 significant bits
constexpr double kLn2Lo = 0x1.a39ef35793c76p-33;  // ln 2 - kLn2Hi
constexpr double kInvLn2 = 0x1.71547652b82fep+0;
constexpr double kSqrt2 = 1.4142135623730951;

__device__ inline double scale2(double v, int k)
{
    // v * 2^k for k >= -1100 (exact until the result is subnormal)
    if (k < -1000) {
        v *= 0x1p-600;
        k += 600;
    }
    return v * __longlong_as_double((long long)(k + 1023) << 52);
}

__device__ inline double aff_exp(double x)
{
    // outside [-745, 709] (below the smallest subnormal, NaN; overflow) by selection, so that loops over it interleave
    const double out = x > 709.0 ? INFINITY : 0.0;
    const bool in = x > -745.0 && x <= 709.0;
    x = in ? x : 0.0;
    const double kf = floor(x * kInvLn2 + 0.5);
    const int k = (int)kf;
    double r = fma(-kf, kLn2Hi, x);
    r = fma(-kf, kLn2Lo, r);
    // e^r = sum_n r^n / n!, n <= 13, |r| <= ln(2) / 2
    double q = 0x1.6124613a86d09p-33;
    q = fma(q, r, 0x1.1eed8eff8d898p-29);
    q = fma(q, r, 0x1.ae64567f544e4p-26);
    q = fma(q, r, 0x1.27e4fb7789f5cp-22);
    q = fma(q, r, 0x1.71de3a556c734p-19);
    q = fma(q, r, 0x1.a01a01a01a01ap-16);
    q = fma(q, r, 0x1.a01a01a01a01ap-13);
    q = fma(q, r, 0x1.6c16c16c16c17p-10);
    q = fma(q, r, 0x1.1111111111111p-7);
    q = fma(q, r, 0x1.5555555555555p-5);
    q = fma(q, r, 0x1.5555555555555p-3);
    q = fma(q, r, 0.5);
    q = fma(q, r, 1.0);
    q = fma(q, r, 1.0);
    return in ? scale2(q, k) : out;
}

// natural log of a positive normal double
__device__ inline double aff_log(double x)
{
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7FF) - 1023;
    b = (b & 0x000FFFFFFFFFFFFFull) | 0x3FF0000000000000ull;
    double m = __longlong_as_double((long long)b);  // x = m 2^e, m in [1, 2)
    if (m > kSqrt2) {
        m *= 0.5;
        e += 1;
    }
    // log m = 2 atanh(z), z = (m - 1) / (m + 1), |z| <= 0.1716
    const double z = (m - 1.0) / (m + 1.0);
    const double z2 = z * z;
    double q = 0.037037037037037035;  // 1/27
    q = fma(q, z2, 0.04);
    q = fma(q, z2, 0.043478260869565216);
    q = fma(q, z2, 0.047619047619047616);
    q = fma(q, z2, 0.05263157894736842);
    q = fma(q, z2, 0.058823529411764705);
    q = fma(q, z2, 0.06666666666666667);
    q = fma(q, z2, 0.07692307692307693);
    q = fma(q, z2, 0.09090909090909091);
    q = fma(q, z2, 0.1111111111111111);
    q = fma(q, z2, 0.14285714285714285);
    q = fma(q, z2, 0.2);
    q = fma(q, z2, 0.3333333333333333);
    const double lm = 2.0 * fma(z * z2, q, z);
    const double ed = (double)e;
    return fma(ed, kLn2Hi, fma(ed, kLn2Lo, lm));
}

// ------------------------------------------------------------------ kNN
// Every pair costs two FP32 operations a dimension (a difference and a fused
// multiply-add, in the definition's order), so the FP32 pipe bounds the kernel
// (15.6 ms at 20,000 x 784) and the rest is kept off it:
// * A thread accumulates a 4 x 8 block of distances, two candidates to a
//   packed FP32x2 operand: 32 packed instructions a dimension against 3
//   16-byte shared loads.
// * kKC dimensions of the tile's rows are staged transposed in shared memory,
//   the next kKC fetched into registers meanwhile.
// * The (query block, candidate tile) units are dealt to the blocks in equal
//   contiguous runs: a block may start and end inside a query block's row of
//   tiles, and then leaves a partial neighbour list.  k_knn_merge joins the
//   partial lists of every query row.  One block per 64 queries instead left
//   a third of the SMs idle in the second wave.
// A list entry is the 64-bit key (distance bits, index): distances are never
// negative, so integer order is (distance, index) order, and NaNs sort last.
// 20,000 x 784, k = 90, all query blocks: 70.0 ms before (4 x 4 blocks of
// scalar operations, a block per 64 queries), 22.8 ms now.  Inputs that the
// tensor-core filter takes (knn_gram.cuh) come here only where it gave up.  8 x 8 blocks need fewer shared loads
// but leave 8 or 12 warps an SM instead of 16: 23.9 and 25.4 ms.
constexpr int kQ = 64;        // query rows per block
constexpr int kC = 128;       // candidates per tile
constexpr int kKC = 16;       // dimensions per staged chunk
constexpr int kKnnT = 256;    // threads
constexpr int kMaxK = 128;    // longest neighbour list
constexpr int kTilePad = 4;   // floats between the rows of a distance tile
constexpr int kStageFloats = 2 * kKC * (kQ + kC);
constexpr int kTileFloats = kQ * (kC + kTilePad);
// the distance tile takes the staging buffers' place once its last chunk is used
constexpr size_t kKnnStatic = 4 * (size_t)(kStageFloats > kTileFloats ? kStageFloats : kTileFloats);
constexpr size_t kKnnMaxDyn = kKnnStatic + (size_t)kQ * kMaxK * 8;
typedef unsigned long long u64;

// packed FP32 operations that keep subnormals, as fmaf does
__device__ __forceinline__ u64 x2_sub(u64 a, u64 b)
{
    u64 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 x2_fma(u64 a, u64 b, u64 c)
{
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 x2_pack(float a, float b)
{
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void x2_unpack(u64 v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

// unit u of `units` belongs to run owner(u): run b holds [b units / runs, (b + 1) units / runs)
__host__ __device__ inline int64_t knn_owner(int64_t u, int64_t units, int64_t runs)
{
    return ((u + 1) * runs - 1) / units;
}

// The units of the listed query blocks (all of them without a list) and the
// runs they are dealt to.  With a list the runs are at most kListRuns a query
// block, which bounds the partial lists that a row's merge holds.
constexpr int kListRuns = 14;
struct KnnRuns {
    int64_t units, runs;
    __host__ __device__ KnnRuns(int64_t qblocks, int64_t ctiles, int64_t max_runs, const uint32_t* nlist)
    {
        const int64_t q = nlist ? (int64_t)*nlist : qblocks;
        units = q * ctiles;
        runs = units < max_runs ? units : max_runs;
        if (nlist && runs > kListRuns * q) runs = kListRuns * q;
    }
};

// one key into a row's sorted list (k keys, unused ones all-ones), by a warp
__device__ __forceinline__ void knn_insert(u64* __restrict__ list, int k, u64 key, int lane)
{
    u64 own[kMaxK / 32], prev[kMaxK / 32];
    int pos = 0;
#pragma unroll
    for (int u = 0; u < kMaxK / 32; u++) {
        const int e = lane + 32 * u;
        own[u] = e < k ? list[e] : ~0ull;
        prev[u] = e > 0 && e < k ? list[e - 1] : 0ull;
        pos += __popc(__ballot_sync(0xffffffffu, own[u] < key));
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kMaxK / 32; u++) {
        const int e = lane + 32 * u;
        if (e < k && e >= pos) list[e] = e == pos ? key : prev[u];
    }
    __syncwarp();
}

template <bool kVec>
__global__ void __launch_bounds__(kKnnT, 2)
    k_knn(const float* __restrict__ x, int64_t n, int dim, int k, int64_t ctiles, int64_t qblocks,
          const uint32_t* __restrict__ list, const uint32_t* __restrict__ nlist, u64* __restrict__ part,
          float* __restrict__ out_d, int32_t* __restrict__ out_i)
{
    extern __shared__ __align__(16) uint8_t dyn[];
    float* stage = reinterpret_cast<float*>(dyn);          // [2][kKC][kQ + kC]
    float* tile = stage;                                   // [kQ][kC + kTilePad]
    u64* lists = reinterpret_cast<u64*>(dyn + kKnnStatic); // [kQ][k]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ty = tid >> 4, tx = tid & 15;  // queries 4 ty + a; candidates 4 tx + b and 64 + 4 tx + b
    constexpr int kRows = kQ + kC;
    constexpr int kLoads = kRows * (kKC / 4) / kKnnT;  // 16-byte pieces a thread fetches per chunk
    const KnnRuns kr(qblocks, ctiles, gridDim.x, nlist);
    const int64_t units = kr.units, runs = kr.runs, run = blockIdx.x;
    if (run >= runs) return;
    auto qblock = [&](int64_t o) { return list ? (int64_t)list[o] : o; };
    const int64_t u0 = run * units / runs, u1 = (run + 1) * units / runs;
    const int chunks = (dim + kKC - 1) / kKC;
    float4 pre[kLoads];
    // piece i of a chunk: row (i mod kRows) of the tile, dimensions 4 (i / kRows) on; a warp's pieces are 32
    // different rows, so their transposed stores hit 32 banks
    auto fetch = [&](int64_t q0, int64_t c0, int t0) {
#pragma unroll
        for (int j = 0; j < kLoads; j++) {
            const int i = tid + j * kKnnT, r = i % kRows, t = t0 + 4 * (i / kRows);
            const int64_t row = r < kQ ? q0 + r : c0 + (r - kQ);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);  // rows and dimensions past the end add (0 - 0)^2
            if (row < n) {
                const float* src = x + row * dim + t;
                if (kVec) {
                    if (t < dim) v = *reinterpret_cast<const float4*>(src);
                } else {
                    if (t < dim) v.x = src[0];
                    if (t + 1 < dim) v.y = src[1];
                    if (t + 2 < dim) v.z = src[2];
                    if (t + 3 < dim) v.w = src[3];
                }
            }
            pre[j] = v;
        }
    };
    auto store = [&](float* s) {
#pragma unroll
        for (int j = 0; j < kLoads; j++) {
            const int i = tid + j * kKnnT, r = i % kRows, t = 4 * (i / kRows);
            s[t * kRows + r] = pre[j].x;
            s[(t + 1) * kRows + r] = pre[j].y;
            s[(t + 2) * kRows + r] = pre[j].z;
            s[(t + 3) * kRows + r] = pre[j].w;
        }
    };
    if (u0 < u1) fetch(qblock(u0 / ctiles) * kQ, u0 % ctiles * kC, 0);
    for (int64_t u = u0; u < u1; u++) {
        const int64_t o = u / ctiles, q0 = qblock(o) * kQ, c0 = u % ctiles * kC;
        if (u == u0 || u % ctiles == 0)
            for (int e = tid; e < kQ * k; e += kKnnT) lists[e] = ~0ull;
        u64 acc[4][4];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = 0ull;
        for (int c = 0; c < chunks; c++) {
            float* s = stage + (c & 1) * kKC * kRows;
            store(s);
            __syncthreads();
            if (c + 1 < chunks)
                fetch(q0, c0, (c + 1) * kKC);
            else if (u + 1 < u1)
                fetch(qblock((u + 1) / ctiles) * kQ, (u + 1) % ctiles * kC, 0);
#pragma unroll
            for (int t = 0; t < kKC; t++) {
                const float4 q = *reinterpret_cast<const float4*>(s + t * kRows + 4 * ty);
                const ulonglong2 ca = *reinterpret_cast<const ulonglong2*>(s + t * kRows + kQ + 4 * tx);
                const ulonglong2 cb = *reinterpret_cast<const ulonglong2*>(s + t * kRows + kQ + 64 + 4 * tx);
                const u64 q2[4] = {x2_pack(q.x, q.x), x2_pack(q.y, q.y), x2_pack(q.z, q.z), x2_pack(q.w, q.w)};
                const u64 c2[4] = {ca.x, ca.y, cb.x, cb.y};
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        const u64 df = x2_sub(q2[a], c2[b]);
                        acc[a][b] = x2_fma(df, df, acc[a][b]);
                    }
            }
        }
        __syncthreads();  // the last chunk is read: the tile may overwrite the staging buffers
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b += 2) {
                float4 v;
                x2_unpack(acc[a][b], v.x, v.y);
                x2_unpack(acc[a][b + 1], v.z, v.w);
                *reinterpret_cast<float4*>(tile + (4 * ty + a) * (kC + kTilePad) + 32 * b + 4 * tx) = v;
            }
        __syncthreads();
        // fold the tile into the lists: warp w owns rows w, w + 8, ...
        for (int r = warp; r < kQ; r += kKnnT / 32) {
            const int64_t qi = q0 + r;
            if (qi >= n) break;
            u64* list = lists + r * k;
#pragma unroll
            for (int h = 0; h < kC / 32; h++) {
                const int64_t cj = c0 + 32 * h + lane;
                const u64 key = (u64)__float_as_uint(tile[r * (kC + kTilePad) + 32 * h + lane]) << 32 | (uint32_t)cj;
                uint32_t m = __ballot_sync(0xffffffffu, cj < n && cj != qi && key < list[k - 1]);
                while (m) {
                    const int src = __ffs(m) - 1;
                    m &= m - 1u;
                    const u64 kv = __shfl_sync(0xffffffffu, key, src);
                    if (kv < list[k - 1]) knn_insert(list, k, kv, lane);
                }
            }
        }
        __syncthreads();
        if (u + 1 == u1 || (u + 1) % ctiles == 0) {
            if (out_d) {  // a single candidate tile: the lists are whole
                for (int e = tid; e < kQ * k && q0 + e / k < n; e += kKnnT) {
                    out_d[q0 * k + e] = __uint_as_float((uint32_t)(lists[e] >> 32));
                    out_i[q0 * k + e] = (int32_t)(uint32_t)lists[e];
                }
            } else {
                // runs and query blocks both grow along the units: their sum numbers the partial lists
                u64* dst = part + (run + o) * (int64_t)(kQ * k);
                for (int e = tid; e < kQ * k; e += kKnnT) dst[e] = lists[e];
            }
            __syncthreads();
        }
    }
}

// A warp per query row joins the row's partial lists (of the runs that hold
// its query block's units): an entry's place is its own index plus, for every
// other list, the number of that list's smaller entries.
constexpr int kMergeWarps = 4;
constexpr size_t kMergeMaxDyn = (size_t)kMergeWarps * (kListRuns + 2) * kMaxK * 8;
__global__ void __launch_bounds__(32 * kMergeWarps)
    k_knn_merge(const u64* __restrict__ part, int64_t n, int k, int64_t ctiles, int64_t qblocks, int64_t max_runs,
                const uint32_t* __restrict__ list, const uint32_t* __restrict__ nlist, int maxseg,
                float* __restrict__ out_d, int32_t* __restrict__ out_i)
{
    extern __shared__ __align__(16) uint8_t dyn[];
    const int lane = threadIdx.x & 31;
    u64* sl = reinterpret_cast<u64*>(dyn) + (size_t)(threadIdx.x >> 5) * maxseg * k;
    const KnnRuns kr(qblocks, ctiles, max_runs, nlist);
    const int64_t units = kr.units, runs = kr.runs;
    const int64_t at = blockIdx.x * (int64_t)kMergeWarps + (threadIdx.x >> 5), o = at / kQ;
    if (o * ctiles >= units) return;
    const int64_t row = (list ? (int64_t)list[o] : o) * kQ + at % kQ;
    if (row >= n) return;
    const int64_t b0 = knn_owner(o * ctiles, units, runs), b1 = knn_owner((o + 1) * ctiles - 1, units, runs);
    const int nseg = (int)(b1 - b0 + 1) < maxseg ? (int)(b1 - b0 + 1) : maxseg;
    for (int sg = 0; sg < nseg; sg++) {
        const u64* src = part + (b0 + sg + o) * (int64_t)(kQ * k) + (row % kQ) * k;
        for (int e = lane; e < k; e += 32) sl[sg * k + e] = src[e];
    }
    __syncwarp();
    for (int e = lane; e < nseg * k; e += 32) {
        const u64 key = sl[e];
        if (key == ~0ull) continue;
        const int sg = e / k;
        int place = e - sg * k;
        for (int l = 0; l < nseg && place < k; l++) {
            if (l == sg) continue;
            int lo = 0, hi = k;  // the first entry of list l not below key
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (sl[l * k + mid] < key) lo = mid + 1;
                else hi = mid;
            }
            place += lo;
        }
        if (place < k) {
            out_d[row * k + place] = __uint_as_float((uint32_t)(key >> 32));
            out_i[row * k + place] = (int32_t)(uint32_t)key;
        }
    }
}

// ------------------------------------------------------------------ bandwidths
// FP64 issues at 1/64 of the FP32 rate and an evaluation of a row's entropy H
// takes 24 FP64 operations a neighbour, so a bisection step is decided by the
// cheapest evaluation that is certain to decide as the FP64 one does:
// * FP32.  With all w <= 1, one w = 1 and <x> <= H <= ln k for x = beta d', the
//   roundings of x (5 2^-24 x), of the exponential (2^-22), of the k-term sums
//   and of the logarithm move H by less than
//   (11 <x^2> + (2 ln k + 1) (k + 10)) 2^-24 < 1.6e-4 at k = 128 (<x^2> <= 0.55 k).
// * FP32 with x to FP64 accuracy, an exponential good to 2.5e-7 and compensated
//   sums.  Relative errors delta of the w move H by at most delta (1 + sd(x)),
//   sd(x) <= 3.5 at k = 128: 1.4e-6 with the products' roundings; the logarithm
//   (an ulp), the quotient and the sums of the last line 1.6e-6.
// * FP64, as the definition says, where neither decides.
// The steps are the same, to the bit.
constexpr int kScreenK = 128;
constexpr float kScreenErr = 2.0e-4f, kScreenErr2 = 3.5e-6f;

// exp(-x) of x = p + e >= 0, |e| tiny, to 2.5e-7: reduction by ln 2 in two parts, the exponential series to r^7
__device__ __forceinline__ float screen_exp(float p, float e)
{
    const float t = rintf(fminf(p, 150.0f) * 1.44269504f);  // beyond 150 the result is zero
    float r = fmaf(t, -0x1.62e4p-1f, p);                    // ln 2 to 15 bits: t times it is exact
    r = fmaf(t, -0x1.7f7d1cp-20f, r) + e;
    float q = -1.0f / 5040.0f;
    q = fmaf(q, r, 1.0f / 720.0f);
    q = fmaf(q, r, -1.0f / 120.0f);
    q = fmaf(q, r, 1.0f / 24.0f);
    q = fmaf(q, r, -1.0f / 6.0f);
    q = fmaf(q, r, 0.5f);
    q = fmaf(q, r, -1.0f);
    q = fmaf(q, r, 1.0f);
    // 2^-t in two factors (t up to 217)
    const int ti = (int)t, h = ti >> 1;
    return p > 150.0f ? 0.0f : q * __int_as_float((127 - h) << 23) * __int_as_float((127 - (ti - h)) << 23);
}

// a / s by its correctly rounded reciprocal y: the quotient's remainder is exact in a fused operation and the
// correction rounds as the division does (P. Markstein, 1990); far from the subnormal range only
__device__ __forceinline__ double quotient(double a, double s, double y)
{
    if (!(a > 1e-280 && s < 1e280)) return a / s;
    const double q = a * y;
    return fma(fma(-q, s, a), y, q);
}

// kPerpLanes lanes share a row: they take its neighbours in turn, and for an
// FP64 evaluation two of them then run the sums of w and of d' w, each a chain
// in the order that defines the rows, over the staged terms.  20,000 rows of
// 90: 4.24 ms with a thread per row and every step in FP64, 2.0 ms with the
// first screen, 1.4 ms with the row's lanes (at 85 % of the FP64 pipe), 0.63 ms
// with the second screen.
constexpr int kPerpLanes = 8;
constexpr int kPerpThreads = 64;
constexpr int kPerpChunk = 64;  // neighbours staged at a time

__global__ void __launch_bounds__(kPerpThreads)
    k_perplexity(const float* __restrict__ dist, int64_t n, int k, double perplexity, int max_iter, double tol,
                 double* __restrict__ p)
{
    constexpr int kRows = kPerpThreads / kPerpLanes;
    // (w, d') of a row's chunk; the odd row length spreads the rows over the banks
    __shared__ double2 s_term[kRows][kPerpChunk + 1];
    const int sub = threadIdx.x % kPerpLanes, group = threadIdx.x / kPerpLanes;
    double2* term = s_term[group];
    const double log_perp = aff_log(perplexity);
    const float screen = (float)tol + kScreenErr;
    // a warp's rows go through the loops together, finished ones idling
    for (int64_t i0 = blockIdx.x * (int64_t)kRows; i0 < n; i0 += (int64_t)gridDim.x * kRows) {
        const bool valid = i0 + group < n;
        const int64_t i = valid ? i0 + group : n - 1;
        const float* d = dist + i * k;
        const float dmin = d[0];
        // sum of w_j = exp(-beta d'_j) in lane 0, of d'_j w_j in lane 1; out: the w_j are kept in the row of p
        auto sums = [&](double beta, bool on, double* out) {
            double chain = 0.0;
            for (int j0 = 0; j0 < k; j0 += kPerpChunk) {
                const int m = on ? min(k - j0, kPerpChunk) : 0;
#pragma unroll 2
                for (int j = sub; j < m; j += kPerpLanes) {
                    const double dj = (double)d[j0 + j] - (double)dmin;
                    const double w = aff_exp(-dj * beta);
                    term[j] = make_double2(w, dj);
                    if (out) out[j0 + j] = w;
                }
                __syncwarp();
                if (sub < 2) {
#pragma unroll 8
                    for (int j = 0; j < m; j++) {
                        const double2 t = term[j];
                        chain = fma(sub == 0 ? 1.0 : t.y, t.x, chain);  // fma(1, w, s) rounds as s + w
                    }
                }
                __syncwarp();
            }
            return chain;
        };
        // the screens' error bounds are for rows whose first entry is the smallest, as kNN rows are
        bool ordered = k <= kScreenK;
        for (int j = sub; j < k; j += kPerpLanes) ordered = ordered && d[j] >= dmin;
        const uint32_t groups = __ballot_sync(0xffffffffu, ordered);
        const uint32_t own = ((1u << kPerpLanes) - 1u) << (threadIdx.x % 32 / kPerpLanes * kPerpLanes);
        const bool screened = (groups & own) == own;
        double beta = 1.0, lo = 0.0, hi = INFINITY;
        bool active = valid;
        for (int it = 0; it < max_iter && __any_sync(0xffffffffu, active); it++) {
            double diff = 0.0;
            bool exact = active;
            if (k <= kScreenK) {
                const float b = (float)beta;
                float s = 0.f, sd = 0.f;
                for (int j = sub; j < k; j += kPerpLanes) {
                    const float dj = d[j] - dmin;
                    const float w = __expf(-dj * b);
                    s += w;
                    sd = fmaf(dj, w, sd);
                }
#pragma unroll
                for (int o = 1; o < kPerpLanes; o <<= 1) {
                    s += __shfl_xor_sync(0xffffffffu, s, o);
                    sd += __shfl_xor_sync(0xffffffffu, sd, o);
                }
                const float quick = __logf(s) + b * sd / s - (float)log_perp;
                if (screened && fabsf(quick) > screen) {  // false for NaN
                    exact = false;
                    diff = (double)quick;
                }
            }
            if (k <= kScreenK && __any_sync(0xffffffffu, exact)) {
                const float b = (float)beta, bl = (float)(beta - (double)b);
                float s = 0.f, sd = 0.f, cs = 0.f, cd = 0.f;  // sums and their compensations
                for (int j = sub; j < k; j += kPerpLanes) {
                    const float dj = d[j] - dmin, dl = (d[j] - dj) - dmin;  // d' exactly, as a sum (T. Dekker)
                    const float p0 = dj * b;
                    const float w = screen_exp(p0, fmaf(dj, b, -p0) + fmaf(dj, bl, dl * b));
                    const float y = w - cs, t = s + y;
                    cs = (t - s) - y;
                    s = t;
                    const float yd = dj * w - cd, td = sd + yd;
                    cd = (td - sd) - yd;
                    sd = td;
                }
                double s64 = (double)s - (double)cs, d64 = (double)sd - (double)cd;
#pragma unroll
                for (int o = 1; o < kPerpLanes; o <<= 1) {
                    s64 += __shfl_xor_sync(0xffffffffu, s64, o);
                    d64 += __shfl_xor_sync(0xffffffffu, d64, o);
                }
                const float sf = (float)s64;
                const float close = logf(sf) + b * ((float)d64 / sf) - (float)log_perp;
                // beta and the sums in the normal range, where the error bounds hold
                if (exact && screened && b > 1e-30f && b < 1e30f && d64 * beta > 1e-3) {
                    if (fabsf(close) > (float)tol + kScreenErr2) {
                        exact = false;
                        diff = (double)close;
                    } else if (fabsf(close) + kScreenErr2 < (float)tol) {
                        exact = active = false;
                    }
                }
            }
            if (__any_sync(0xffffffffu, exact)) {
                const double chain = sums(beta, exact, nullptr);
                const double s = __shfl_sync(0xffffffffu, chain, 0, kPerpLanes);
                const double sd = __shfl_sync(0xffffffffu, chain, 1, kPerpLanes);
                if (exact) {
                    const double h = aff_log(s) + beta * sd / s;
                    diff = h - log_perp;
                    if (fabs(diff) < tol) active = false;
                }
            }
            if (active) {
                if (diff > 0.0) {
                    lo = beta;
                    beta = isinf(hi) ? beta * 2.0 : (lo + hi) * 0.5;
                } else {
                    hi = beta;
                    beta = (lo + hi) * 0.5;
                }
            }
        }
        double* row = p + i * k;
        const double s = __shfl_sync(0xffffffffu, sums(beta, valid, row), 0, kPerpLanes);
        const double y = 1.0 / s;
        for (int j = sub; valid && j < k; j += kPerpLanes) row[j] = quotient(row[j], s, y);
    }
}

// ------------------------------------------------------------------ symmetrisation
// entry e < nk: (i, j) with value p_ij / (2N); entry nk + e: its transpose (j, i)
__global__ void k_sym_entries(const int32_t* __restrict__ idx, const double* __restrict__ p, int64_t n, int k,
                              double c, uint32_t* __restrict__ col_key, uint32_t* __restrict__ row,
                              double* __restrict__ v)
{
    const int64_t nk = n * k;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nk; e += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t i = (uint32_t)(e / k), j = (uint32_t)idx[e];
        const double w = p[e] * c;
        col_key[e] = j;
        row[e] = i;
        v[e] = w;
        col_key[nk + e] = i;
        row[nk + e] = j;
        v[nk + e] = w;
    }
}

__global__ void k_gather_u32(const uint32_t* __restrict__ in, const uint32_t* __restrict__ perm, int64_t m,
                             uint32_t* __restrict__ out)
{
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x)
        out[e] = in[perm[e]];
}

// sorted position q holds entry ord[q] = perm1[perm2[q]] (rows sorted, columns
// within a row); flag the first entry of each (row, col)
__global__ void k_sym_flags(const uint32_t* __restrict__ perm1, const uint32_t* __restrict__ perm2, int64_t m,
                            const uint32_t* __restrict__ row, const uint32_t* __restrict__ col_key,
                            uint32_t* __restrict__ ord, uint32_t* __restrict__ flag)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m; q += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t e = perm1[perm2[q]];
        ord[q] = e;
        bool first = q == 0;
        if (!first) {
            const uint32_t f = perm1[perm2[q - 1]];
            first = row[f] != row[e] || col_key[f] != col_key[e];
        }
        flag[q] = first ? 1u : 0u;
    }
}

// pos: exclusive scan of the flags (pos[m] = the number of distinct entries)
__global__ void k_sym_write(const uint32_t* __restrict__ ord, const uint32_t* __restrict__ flag,
                            const uint32_t* __restrict__ pos, int64_t m, int64_t n, const uint32_t* __restrict__ row,
                            const uint32_t* __restrict__ col_key, const double* __restrict__ v,
                            uint32_t* __restrict__ row_ptr, uint32_t* __restrict__ col, double* __restrict__ val)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m; q += (int64_t)gridDim.x * blockDim.x) {
        if (!flag[q]) continue;
        const uint32_t e = ord[q], u = pos[q];
        double s = v[e];
        if (q + 1 < m && !flag[q + 1]) s = s + v[ord[q + 1]];  // the transposed contribution to the same entry
        col[u] = col_key[e];
        val[u] = s;
        if (q == 0 || row[ord[q - 1]] != row[e]) row_ptr[row[e]] = u;
        if (u + 1 == pos[m]) row_ptr[n] = pos[m];
    }
}

}  // namespace
}  // namespace tc

using namespace tc;

// The kNN's scratch comes from a memory pool of its own, which keeps up to 64 MB between calls: the device's default
// pool gives everything back at each synchronisation, and allocating anew took more than a small call's kernels (1,024 x 2,
// k = 1: 266 us a call, 60 with the pool; 150 before the kNN had scratch).  nullptr: the default pool.
constexpr size_t kKnnPoolKeep = 64ull << 20;
static cudaMemPool_t knn_pool()
{
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> g(mu);
    if (!pools[dev]) {
        cudaMemPoolProps p = {};
        p.allocType = cudaMemAllocationTypePinned;
        p.location.type = cudaMemLocationTypeDevice;
        p.location.id = dev;
        uint64_t keep = kKnnPoolKeep;
        // (no stream's work: allowed while this or another thread captures)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (cudaMemPoolCreate(&pools[dev], &p) != cudaSuccess ||
            cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            pools[dev] = nullptr;
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    return pools[dev];
}

static cudaError_t knn_alloc(void** p, size_t bytes, cudaStream_t s)
{
    // more than the pool keeps: the default pool, whose memory the symmetrisation after it takes over
    const cudaMemPool_t pool = bytes > kKnnPoolKeep ? nullptr : knn_pool();
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

extern "C" int tc_knn_device(const float* d_x, int64_t n, int dim, int k, float* d_dist, int32_t* d_idx, void* stream)
{
    if (!d_x || !d_dist || !d_idx || n < 2 || dim < 1 || k < 1 || k > kMaxK || k >= n || n > 0x7FFFFFFF) {
        tc_set_error("tc_knn_device: invalid arguments (need 1 <= k <= %d, k < n)", kMaxK);
        return TC_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t qblocks = (n + kQ - 1) / kQ, ctiles = (n + kC - 1) / kC;
    // two resident blocks per SM (registers and shared memory), each one run of units
    const int64_t max_runs = 2 * (int64_t)sm_count();
    const int64_t runs = KnnRuns(qblocks, ctiles, max_runs, nullptr).runs;
    // 16-byte loads: every row starts on a 16-byte boundary
    const bool vec = dim % 4 == 0 && (reinterpret_cast<uintptr_t>(d_x) & 15) == 0;
    // the filter on the tensor cores wherever its bound holds: a row's bound needs more than k groups of eight columns
    // (1,024 points have 128; a row that finds too few goes to k_knn), its inputs 16 KB of shared memory.  It is the
    // faster one over all of that range, k = 90, against k_knn alone: 1,024 x 4: 91 us, 295; 2,000 x 32: 111, 573;
    // 20,000 x 128: 1.28 ms, 6.70; 20,000 x 784: 3.0, 23.2 (4.6 when the inputs have low parts); 70,000 x 784: 22.2,
    // 254.9
    bool gram = n >= kGramMinN && dim <= kGramMaxDim;
    auto kernel = vec ? k_knn<true> : k_knn<false>;
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    // scratch: partial lists; for the filter the split inputs, norms, status, flags and list of query blocks, and
    // a_ij of as many query rows as kGramBytes holds (at least one tile of rows)
    const int dimp = (dim + 15) & ~15;
    const int64_t npad = (n + kGramCols - 1) / kGramCols * kGramCols, rblocks = (n + kGramRows - 1) / kGramRows;
    int64_t rb_chunk = kGramBytes / (npad * 4 * kGramRows);
    rb_chunk = rb_chunk < 1 ? 1 : rb_chunk > rblocks ? rblocks : rb_chunk;
    const size_t b_part = up((size_t)(runs + qblocks) * kQ * k * 8), b_half = up((size_t)npad * dimp * 2),
                 b_norm = up((size_t)npad * 4), b_flag = up(sizeof(GramStat) + (size_t)qblocks * 4),
                 b_list = up((size_t)qblocks * 4);
    const size_t b_fixed = b_part + 2 * b_half + b_norm + b_flag + b_list, rb_bytes = (size_t)kGramRows * npad * 5;
    // up to 12,288 points, where allocating the scratch anew costs more than shorter launches do, no more than the pool
    // keeps, as long as a launch has two tiles for nearly every multiprocessor (10,000 x 2, k = 1: 890 us -> 303)
    const int64_t rb_pool = b_fixed + 512 < kKnnPoolKeep ? (int64_t)((kKnnPoolKeep - b_fixed - 512) / rb_bytes) : 0;
    if (n <= 12288 && rb_pool < rb_chunk && rb_pool * (npad / kGramCols) >= 2 * sm_count() - 64) rb_chunk = rb_pool;
    const size_t b_gram = up((size_t)rb_chunk * kGramRows * npad * 4), b_gmin = b_gram / 4;
    void* buf_p = nullptr;
    if (gram && knn_alloc(&buf_p, b_fixed + b_gram + b_gmin, s) != cudaSuccess) {
        cudaGetLastError();  // no room for the filter's scratch: every query block by k_knn
        gram = false;
    }
    const bool whole = ctiles == 1;  // no partial lists, no scratch
    if (!gram && !whole) TC_CUDA_TRY(knn_alloc(&buf_p, b_part, s));
    uint8_t* buf = static_cast<uint8_t*>(buf_p);
    // runs that share a query block: each holds at least units / runs of its ctiles units
    int64_t maxseg = gram ? kListRuns + 2 : runs / qblocks + 2;
    if (maxseg > ctiles) maxseg = ctiles;
    const size_t dyn = kKnnStatic + (size_t)kQ * k * 8, mdyn = (size_t)kMergeWarps * maxseg * k * 8;
    if (mdyn > kMergeMaxDyn) {  // up to 400 runs (200 multiprocessors) a row lies in at most 16
        tc_set_error("tc_knn_device: more runs a query block than the merge holds");
        if (buf_p) cudaFreeAsync(buf_p, s);
        return TC_ERR_STATE;
    }
    u64* part = reinterpret_cast<u64*>(buf);
    uint32_t *list = nullptr, *nlist = nullptr;
    // the limits of every k, not this one's: calls of other threads set them too
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKnnMaxDyn);
    if (e == cudaSuccess && !whole)
        e = cudaFuncSetAttribute(k_knn_merge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMergeMaxDyn);
    if (gram && e == cudaSuccess) {
        uint8_t *hi = buf + b_part, *lo = hi + b_half;
        float* norm = reinterpret_cast<float*>(lo + b_half);
        GramStat* st = reinterpret_cast<GramStat*>(reinterpret_cast<uint8_t*>(norm) + b_norm);
        uint32_t* qflag = reinterpret_cast<uint32_t*>(st + 1);
        list = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(st) + b_flag);
        nlist = &st->nflagged;
        float* a = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(list) + b_list);
        float* gmin = a + b_gram / 4;
        const size_t sdyn = (size_t)((dim + 31) & ~31) * 4;
        auto select = vec ? k_knn_select<true> : k_knn_select<false>;
        e = cudaFuncSetAttribute(k_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSmem);
        if (e == cudaSuccess) e = cudaMemsetAsync(st, 0, b_flag, s);
        if (e == cudaSuccess) {
            k_gram_split<<<(unsigned)(npad / 8), 256, 0, s>>>(d_x, n, dim, dimp, hi, lo, norm, st);
            for (int64_t rb = 0; rb < rblocks; rb += rb_chunk) {
                const int64_t nrb = rblocks - rb < rb_chunk ? rblocks - rb : rb_chunk;
                const int64_t tiles = nrb * (npad / kGramCols), row0 = rb * kGramRows;
                const int64_t rows = n - row0 < nrb * kGramRows ? n - row0 : nrb * kGramRows;
                k_gram<<<(unsigned)(tiles < sm_count() ? tiles : sm_count()), kGramThreads, kGramSmem, s>>>(
                    hi, lo, norm, n, npad, dimp, rb, (int)nrb, a, gmin, st);
                select<<<(unsigned)rows, kSelT, sdyn, s>>>(d_x, n, dim, dimp, k, a, gmin, npad, nrb, row0, norm, st, d_dist,
                                                          d_idx, qflag, kQ);
            }
            k_knn_flagged<<<1, 1024, 0, s>>>(qflag, qblocks, st, list);
        }
    }
    if (e == cudaSuccess) {
        kernel<<<(unsigned)runs, kKnnT, dyn, s>>>(d_x, n, dim, k, ctiles, qblocks, list, nlist, part,
                                                  whole ? d_dist : nullptr, d_idx);
        if (!whole) k_knn_merge<<<(unsigned)(qblocks * (kQ / kMergeWarps)), 32 * kMergeWarps, mdyn, s>>>(
            part, n, k, ctiles, qblocks, runs, list, nlist, (int)maxseg, d_dist, d_idx);
        e = cudaGetLastError();
    }
    const cudaError_t ef = buf ? cudaFreeAsync(buf, s) : cudaSuccess;
    if (e != cudaSuccess) return tc_cuda_fail(e, "tc_knn_device");
    TC_CUDA_TRY(ef);
    return TC_OK;
}

extern "C" int tc_perplexity_device(const float* d_dist, int64_t n, int k, double perplexity, int max_iter, double tol,
                                    double* d_p, void* stream)
{
    if (!d_dist || !d_p || n < 1 || k < 1 || !(perplexity > 1.0) || max_iter < 1 || !(tol > 0.0)) {
        tc_set_error("tc_perplexity_device: invalid arguments (perplexity must exceed 1)");
        return TC_ERR_INVALID;
    }
    k_perplexity<<<grid_for(n * kPerpLanes, kPerpThreads), kPerpThreads, 0, (cudaStream_t)stream>>>(d_dist, n, k, perplexity, max_iter, tol, d_p);
    TC_CUDA_TRY(cudaGetLastError());
    return TC_OK;
}

extern "C" int tc_symmetrize_device(const int32_t* d_idx, const double* d_p, int64_t n, int k, uint32_t* d_row_ptr,
                                    uint32_t* d_col, double* d_val, int64_t* nnz, void* stream)
{
    const int64_t m = 2 * n * (int64_t)k;
    if (!d_idx || !d_p || !d_row_ptr || !d_col || !d_val || !nnz || n < 2 || k < 1 || m >= 0xFFFFFFFFll) {
        tc_set_error("tc_symmetrize_device: invalid arguments");
        return TC_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t tw = radix_tmp_words(m) > scan_tmp_words(m) ? radix_tmp_words(m) : scan_tmp_words(m);
    // scratch (32-bit words): values (2m); column keys, rows, the two sorts' keys and permutations, their
    // alternates and the sorted order (9 arrays of m); flags (m); positions (m + 1); sort/scan temporaries
    const size_t words = (size_t)m * 2 + (size_t)m * 9 + (size_t)m + (size_t)(m + 2) + (size_t)tw;
    void* buf = nullptr;
    TC_CUDA_TRY(cudaMallocAsync(&buf, words * 4 + 64, s));
    uint32_t* w = static_cast<uint32_t*>(buf);
    double* v = reinterpret_cast<double*>(w);
    uint32_t* colk = w + 2 * m;
    uint32_t* row = colk + m;
    uint32_t* k1 = row + m;
    uint32_t* p1 = k1 + m;
    uint32_t* k2 = p1 + m;
    uint32_t* p2 = k2 + m;
    uint32_t* ak = p2 + m;
    uint32_t* av = ak + m;
    uint32_t* ord = av + m;
    uint32_t* flag = ord + m;
    uint32_t* pos = flag + m;
    uint32_t* tmp = pos + (m + 2) - (m & 1);  // 8-byte aligned; ends before w + words
    int rc = TC_OK;
    const double c = 1.0 / (2.0 * (double)n);
    k_sym_entries<<<grid_for(n * k, 256), 256, 0, s>>>(d_idx, d_p, n, k, c, colk, row, v);
    // stable sort by column, then stable by row: rows sorted, columns sorted within a row
    cudaError_t e = cudaMemcpyAsync(k1, colk, (size_t)m * 4, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) rc = radix_sort_u32(k1, p1, ak, av, m, tmp, s, nullptr, 0);
    if (e == cudaSuccess && rc == TC_OK) {
        k_gather_u32<<<grid_for(m, 256), 256, 0, s>>>(row, p1, m, k2);
        rc = radix_sort_u32(k2, p2, ak, av, m, tmp, s, nullptr, 0);
    }
    if (e == cudaSuccess && rc == TC_OK) {
        k_sym_flags<<<grid_for(m, 256), 256, 0, s>>>(p1, p2, m, row, colk, ord, flag);
        rc = exclusive_scan_u32(flag, pos, m, tmp, s);
    }
    if (e == cudaSuccess && rc == TC_OK) {
        k_sym_write<<<grid_for(m, 256), 256, 0, s>>>(ord, flag, pos, m, n, row, colk, v, d_row_ptr, d_col, d_val);
        uint32_t cnt = 0;
        e = cudaMemcpyAsync(&cnt, pos + m, 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        *nnz = cnt;
    }
    const cudaError_t ef = cudaFreeAsync(buf, s);
    if (e != cudaSuccess) return tc_cuda_fail(e, "tc_symmetrize_device");
    if (rc) return rc;
    if (ef != cudaSuccess) return tc_cuda_fail(ef, "cudaFreeAsync");
    TC_CUDA_TRY(cudaGetLastError());
    return TC_OK;
}
