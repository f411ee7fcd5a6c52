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
#include "common.cuh"

namespace tc {
namespace {

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
// 20,000 x 784, k = 90: 70.0 ms before (4 x 4 blocks of scalar operations, a
// block per 64 queries), 22.8 ms now.  8 x 8 blocks need fewer shared loads
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
    k_knn(const float* __restrict__ x, int64_t n, int dim, int k, int64_t ctiles, int64_t units, u64* __restrict__ part)
{
    extern __shared__ __align__(16) uint8_t dyn[];
    float* stage = reinterpret_cast<float*>(dyn);          // [2][kKC][kQ + kC]
    float* tile = stage;                                   // [kQ][kC + kTilePad]
    u64* lists = reinterpret_cast<u64*>(dyn + kKnnStatic); // [kQ][k]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ty = tid >> 4, tx = tid & 15;  // queries 4 ty + a; candidates 4 tx + b and 64 + 4 tx + b
    constexpr int kRows = kQ + kC;
    constexpr int kLoads = kRows * (kKC / 4) / kKnnT;  // 16-byte pieces a thread fetches per chunk
    const int64_t runs = gridDim.x, run = blockIdx.x;
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
    if (u0 < u1) fetch(u0 / ctiles * kQ, u0 % ctiles * kC, 0);
    for (int64_t u = u0; u < u1; u++) {
        const int64_t qb = u / ctiles, q0 = qb * kQ, c0 = u % ctiles * kC;
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
                fetch((u + 1) / ctiles * kQ, (u + 1) % ctiles * kC, 0);
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
            // runs and query blocks both grow along the units: run + query block numbers the partial lists
            u64* dst = part + (run + qb) * (int64_t)(kQ * k);
            for (int e = tid; e < kQ * k; e += kKnnT) dst[e] = lists[e];
            __syncthreads();
        }
    }
}

// A warp per query row joins the row's partial lists (of the runs that hold
// its query block's units): an entry's place is its own index plus, for every
// other list, the number of that list's smaller entries.
constexpr int kMergeWarps = 4;
__global__ void __launch_bounds__(32 * kMergeWarps)
    k_knn_merge(const u64* __restrict__ part, int64_t n, int k, int64_t ctiles, int64_t units, int64_t runs,
                int maxseg, float* __restrict__ out_d, int32_t* __restrict__ out_i)
{
    extern __shared__ __align__(16) uint8_t dyn[];
    const int lane = threadIdx.x & 31;
    u64* sl = reinterpret_cast<u64*>(dyn) + (size_t)(threadIdx.x >> 5) * maxseg * k;
    const int64_t row = blockIdx.x * (int64_t)kMergeWarps + (threadIdx.x >> 5);
    if (row >= n) return;
    const int64_t qb = row / kQ;
    const int64_t b0 = knn_owner(qb * ctiles, units, runs), b1 = knn_owner((qb + 1) * ctiles - 1, units, runs);
    const int nseg = (int)(b1 - b0 + 1) < maxseg ? (int)(b1 - b0 + 1) : maxseg;
    for (int sg = 0; sg < nseg; sg++) {
        const u64* src = part + (b0 + sg + qb) * (int64_t)(kQ * k) + (row % kQ) * k;
        for (int e = lane; e < k; e += 32) sl[sg * k + e] = src[e];
    }
    __syncwarp();
    for (int e = lane; e < nseg * k; e += 32) {
        const u64 key = sl[e];
        if (key == ~0ull) continue;
        const int sg = e / k;
        int place = e - sg * k;
        for (int o = 0; o < nseg && place < k; o++) {
            if (o == sg) continue;
            int lo = 0, hi = k;  // the first entry of list o not below key
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (sl[o * k + mid] < key) lo = mid + 1;
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
// The entropy of one row in FP32.  It decides a bisection step wherever it is
// farther from the target than its error: with all w <= 1 and one w = 1, and
// <x> <= H <= ln k for x = beta d', the roundings of x (5 2^-24 x), of the
// exponential (2^-22), of the k-term sums and of the logarithm move H by less
// than (11 <x^2> + (2 ln k + 1) (k + 10)) 2^-24 < 1.6e-4 at k = 128, where
// <x^2> <= 0.55 k.
constexpr int kScreenK = 128;
constexpr float kScreenErr = 2.0e-4f;

__device__ inline float entropy_f32(const float* __restrict__ d, int k, float beta)
{
    const float dmin = d[0];
    float s = 0.f, sd = 0.f;
#pragma unroll 4
    for (int j = 0; j < k; j++) {
        const float dj = d[j] - dmin;
        const float w = __expf(-dj * beta);
        s += w;
        sd = fmaf(dj, w, sd);
    }
    return __logf(s) + beta * sd / s;
}

// A thread per row (the sums' order is part of the result).  FP64 issues at
// 1/64 of the FP32 rate and an evaluation takes 24 FP64 operations a
// neighbour, so only the steps that FP32 cannot decide, the last five or six of
// some 22, are evaluated in FP64: the same steps, to the bit.  20,000 rows of
// 90: 4.24 ms with every step in FP64, 2.0 ms now.  Small blocks spread few
// rows over the SMs.
constexpr int kPerpThreads = 64;

__global__ void __launch_bounds__(kPerpThreads)
    k_perplexity(const float* __restrict__ dist, int64_t n, int k, double perplexity, int max_iter, double tol,
                 double* __restrict__ p)
{
    const double log_perp = aff_log(perplexity);
    const float screen = (float)tol + kScreenErr;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float* d = dist + i * k;
        const double dmin = (double)d[0];
        double beta = 1.0, lo = 0.0, hi = INFINITY;
        for (int it = 0; it < max_iter; it++) {
            double diff;
            const float quick = k <= kScreenK ? entropy_f32(d, k, (float)beta) - (float)log_perp : 0.f;
            if (fabsf(quick) > screen) {  // false for NaN
                diff = (double)quick;
            } else {
                double s = 0.0, sd = 0.0;
#pragma unroll 4
                for (int j = 0; j < k; j++) {
                    const double dj = (double)d[j] - dmin;
                    const double w = aff_exp(-dj * beta);
                    s += w;
                    sd = fma(dj, w, sd);
                }
                const double h = aff_log(s) + beta * sd / s;
                diff = h - log_perp;
                if (fabs(diff) < tol) break;
            }
            if (diff > 0.0) {
                lo = beta;
                beta = isinf(hi) ? beta * 2.0 : (lo + hi) * 0.5;
            } else {
                hi = beta;
                beta = (lo + hi) * 0.5;
            }
        }
        double s = 0.0;
#pragma unroll 4
        for (int j = 0; j < k; j++) {
            const double w = aff_exp(-((double)d[j] - dmin) * beta);
            s += w;
            p[i * k + j] = w;
        }
        for (int j = 0; j < k; j++) p[i * k + j] = p[i * k + j] / s;
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

extern "C" int tc_knn_device(const float* d_x, int64_t n, int dim, int k, float* d_dist, int32_t* d_idx, void* stream)
{
    if (!d_x || !d_dist || !d_idx || n < 2 || dim < 1 || k < 1 || k > kMaxK || k >= n || n > 0x7FFFFFFF) {
        tc_set_error("tc_knn_device: invalid arguments (need 1 <= k <= %d, k < n)", kMaxK);
        return TC_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t qblocks = (n + kQ - 1) / kQ, ctiles = (n + kC - 1) / kC, units = qblocks * ctiles;
    // two resident blocks per SM (registers and shared memory), each one run of units
    const int64_t runs = units < 2 * (int64_t)sm_count() ? units : 2 * (int64_t)sm_count();
    // runs that share a query block: each holds at least units / runs of its ctiles units
    const int64_t maxseg = runs / qblocks + 2 < ctiles ? runs / qblocks + 2 : ctiles;
    const size_t dyn = kKnnStatic + (size_t)kQ * k * 8, mdyn = (size_t)kMergeWarps * maxseg * k * 8;
    // 16-byte loads: every row starts on a 16-byte boundary
    const bool vec = dim % 4 == 0 && (reinterpret_cast<uintptr_t>(d_x) & 15) == 0;
    auto kernel = vec ? k_knn<true> : k_knn<false>;
    TC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    TC_CUDA_TRY(cudaFuncSetAttribute(k_knn_merge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mdyn));
    void* part = nullptr;
    TC_CUDA_TRY(cudaMallocAsync(&part, (size_t)(runs + qblocks) * kQ * k * 8, s));
    kernel<<<(unsigned)runs, kKnnT, dyn, s>>>(d_x, n, dim, k, ctiles, units, static_cast<u64*>(part));
    k_knn_merge<<<(unsigned)((n + kMergeWarps - 1) / kMergeWarps), 32 * kMergeWarps, mdyn, s>>>(
        static_cast<const u64*>(part), n, k, ctiles, units, runs, (int)maxseg, d_dist, d_idx);
    const cudaError_t e = cudaGetLastError(), ef = cudaFreeAsync(part, s);
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
    k_perplexity<<<grid_for(n, kPerpThreads), kPerpThreads, 0, (cudaStream_t)stream>>>(d_dist, n, k, perplexity, max_iter, tol, d_p);
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
    const size_t words = (size_t)m * 2 + (size_t)m * 9 + (size_t)m + (size_t)(m + 1) + (size_t)tw;
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
    uint32_t* tmp = pos + (m + 1);  // ends at w + words
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
