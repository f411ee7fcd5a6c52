// Tree construction, bit-exact to NBodySolverFMM_SYM_MORTON::updateTree
// (src/nbodysolvers/cpu/nBodySolverFMM_SYM_MORTON.h:79-95):
//   createMortonCode (:538-561)  -> k_morton_fast + k_morton_exact (FP32
//                                   where its floor provably agrees, else FP64)
//   integer_sort (:89)           -> radix_sort_u32   (stable on input order)
//   createLeafNodes (:328-379)   -> k_gather_bounds + k_leaf_moments
//   bottomUpNodeConstruction (:381-470) -> k_bottom_up, one launch per level
// Leaf moments are summed sequentially in sorted order by one thread per
// leaf and internal nodes combine children in the reference's j = 3..0 order,
// so COM, M0 and M2 come out bit-identical to the reference's FP64 values.
// The order-p path (FP32 only) builds its records in tree_p.cu instead.
// Alongside the FP64 node record the kernels write the compute copies in
// cell-relative coordinates (COM minus the ideal cell centre), which keep
// FP32 differences accurate to a fraction of the cell size.
#include <cmath>

#include "state.cuh"

namespace tc {
namespace {

// one coordinate of createMortonCode (:545-549): (uint32)clamp(((p - min)/L) * 65536, 0, 65535).
// FP64 division runs at 1/64 of the FP32 rate on GB300, so the quotient is
// first formed as (p - min) * (65536/L), within 2 ulp of the exact product;
// only when that lands within 1e-9 of an integer can the floor differ from
// the reference's, and then the reference's own division decides.
__device__ inline uint32_t morton_coord(double p, double nm, double L, double s65536)
{
    const double a = p + nm;
    double v = a * s65536;
    const double f = v - floor(v);
    if (f < 1e-9 || f > 1.0 - 1e-9) v = (a / (L)) * 65536.0;
    v = (v < 0.0) ? 0.0 : v;             // glm::max(v, 0)
    v = (65535.0 < v) ? 65535.0 : v;     // glm::min(v, 65535)
    return (uint32_t)v;
}

// IEEE double as an integer with the same order (for box tests on the integer pipe)
__device__ inline long long dorder(double v)
{
    const long long b = __double_as_longlong(v);
    return b >= 0 ? b : (long long)(0x8000000000000000ull - (unsigned long long)b);
}

// v rounded to the nearest float (ties to even) with integer operations: the
// FP64 -> FP32 conversion instruction shares GB300's narrow FP64 pipe.
// Results below the smallest normal float flush to a signed zero.
__device__ inline float f32_rn(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
    const int e = (int)((b >> 52) & 0x7FFull);
    const unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    if (e == 0x7FF) return m ? __uint_as_float(0x7FC00000u) : __uint_as_float(sign | 0x7F800000u);
    const int ef = e - 1023 + 127;
    if (ef <= 0) return __uint_as_float(sign);
    if (ef >= 255) return __uint_as_float(sign | 0x7F800000u);
    unsigned long long r = m >> 29;
    const unsigned long long rem = m & ((1ull << 29) - 1ull);
    if (rem > (1ull << 28) || (rem == (1ull << 28) && (r & 1ull))) r++;
    // a mantissa carry (r = 2^23) moves into the exponent, as rounding does
    const uint32_t bits = ((uint32_t)ef << 23) + (uint32_t)r;
    return __uint_as_float(sign | (bits < 0x7F800000u ? bits : 0x7F800000u));
}

// createMortonCode's quantisation, fast form.  FP64 runs at 1/64 of the FP32
// rate on GB300, so the quotient ((p - min) / L) * 65536 is first formed in
// FP32 from the FP64 difference: fl32(fl32(p - min) * fl32(65536 / L)) is
// within 3 * 2^-24 relative (<= 0.012 absolute below 65536) of the
// reference's FP64 value, so its floor is the reference's whenever its
// fraction lies in [1/64, 63/64).  Points with a coordinate closer than that
// to a cell edge are queued, and k_morton_exact recomputes them with the
// reference's FP64 arithmetic.  Each block queues into its own region of
// morton_region(n, grid) entries (shared-memory counter, no global atomics).
// The box test compares the doubles' order-preserving integer images.
constexpr int kMortonThreads = 256;

__host__ __device__ inline int64_t morton_region(int64_t n, int64_t grid)
{
    const int64_t per = grid * kMortonThreads;
    return ((n + per - 1) / per) * kMortonThreads;
}

__global__ void __launch_bounds__(kMortonThreads)
    k_morton_fast(const double2* __restrict__ pos, int64_t n, double minx, double miny, double maxx, double maxy,
                  float s65536, uint32_t* __restrict__ codes, uint32_t* __restrict__ err,
                  uint32_t* __restrict__ queue, uint32_t* __restrict__ qcount)
{
    __shared__ uint32_t s_count;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    uint32_t* region = queue + (int64_t)blockIdx.x * morton_region(n, gridDim.x);
    const long long kx0 = dorder(minx), kx1 = dorder(maxx), ky0 = dorder(miny), ky1 = dorder(maxy);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 p = pos[i];
        const long long kx = dorder(p.x), ky = dorder(p.y);
        // NaN images lie outside every finite box
        if (!(kx >= kx0 && kx <= kx1 && ky >= ky0 && ky <= ky1)) atomicOr(err, 1u);
        const float vx = f32_rn(p.x - minx) * s65536, vy = f32_rn(p.y - miny) * s65536;
        bool exact = false;
        uint32_t q[2];
        const float v2[2] = {vx, vy};
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const float v = v2[c];
            if (v >= 65535.0f + 1.0f / 64.0f) {
                q[c] = 65535u;  // the reference's clamp whatever the last bits
            } else {
                const float f = v - floorf(v);
                exact |= !(f >= 1.0f / 64.0f && f < 63.0f / 64.0f);
                q[c] = v > 0.0f ? (uint32_t)v : 0u;
            }
        }
        if (exact)
            region[atomicAdd(&s_count, 1u)] = (uint32_t)i;
        else
            codes[i] = (spread16(q[1]) << 1) | spread16(q[0]);
    }
    __syncthreads();
    if (threadIdx.x == 0) qcount[blockIdx.x] = s_count;
}

// what the tree build clears and tabulates before its leaves, done by k_morton_exact (as clears and a launch of their
// own they were four operations): the leaves' first and end indices, the large leaves' counters, the cell centres
// relative to the box corner, (i + 0.5) h for i < w
struct TreePrep {
    uint32_t* first;
    uint32_t* endp;
    int64_t nleaf;
    uint32_t* big;  // kBigLeaves words, may be null
    double* off;    // may be null
    int w;
    double h;
};

// the queued points of k_morton_fast, in the reference's FP64 arithmetic: block
// b of the same grid takes region b
__global__ void __launch_bounds__(kMortonThreads)
    k_morton_exact(const double2* __restrict__ pos, int64_t n, double minx, double miny, double L,
                   const uint32_t* __restrict__ queue, const uint32_t* __restrict__ qcount,
                   uint32_t* __restrict__ codes, TreePrep prep)
{
    const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = id; i < prep.nleaf; i += step) {
        prep.first[i] = 0;
        prep.endp[i] = 0;
    }
    if (prep.big && id < kBigLeaves) prep.big[id] = 0;
    for (int64_t i = id; prep.off && i < prep.w; i += step) prep.off[i] = ((double)i + 0.5) * prep.h;
    const double nmx = -minx, nmy = -miny;
    const double s65536 = 65536.0 / L;
    const uint32_t* region = queue + (int64_t)blockIdx.x * morton_region(n, gridDim.x);
    const uint32_t nq = qcount[blockIdx.x];
    for (uint32_t k = threadIdx.x; k < nq; k += blockDim.x) {
        const uint32_t i = region[k];
        const double2 p = pos[i];
        codes[i] = (spread16(morton_coord(p.y, nmy, L, s65536)) << 1) | spread16(morton_coord(p.x, nmx, L, s65536));
    }
}

template <typename real>
__global__ void k_gather_bounds(const uint32_t* __restrict__ codes, const uint32_t* __restrict__ perm,
                                const double2* __restrict__ pos_in, int64_t n, int depth, double minx, double miny,
                                double h, double2* __restrict__ pos64, real* __restrict__ prel,
                                uint32_t* __restrict__ first, uint32_t* __restrict__ endp)
{
    const int shift = 32 - 2 * depth;
    const uint32_t li = level_index(depth);
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        uint32_t leaf = depth ? (codes[k] >> shift) : 0u;
        double2 p = pos_in[perm[k]];
        pos64[k] = p;
        uint32_t ix = compact16(leaf), iy = compact16(leaf >> 1);
        double cx = minx + ((double)ix + 0.5) * h;
        double cy = miny + ((double)iy + 0.5) * h;
        prel[2 * k] = (real)(p.x - cx);
        prel[2 * k + 1] = (real)(p.y - cy);
        if (k == 0 || (depth ? (codes[k - 1] >> shift) : 0u) != leaf) first[li + leaf] = (uint32_t)k;
        if (k == n - 1 || (depth ? (codes[k + 1] >> shift) : 0u) != leaf) endp[li + leaf] = (uint32_t)(k + 1);
    }
}

// k_gather_bounds for FP32 compute copies: p - centre as (p - min) - (i + 0.5) h
// from the offset table (two FP64 additions per coordinate; the difference is
// the FP64 one to within its last bits, far below FP32 resolution)
__global__ void k_gather_bounds_f32(const uint32_t* __restrict__ codes, const uint32_t* __restrict__ perm,
                                    const double2* __restrict__ pos_in, int64_t n, int depth, double minx,
                                    double miny, const double* __restrict__ off, double2* __restrict__ pos64,
                                    float2* __restrict__ prel, uint32_t* __restrict__ first,
                                    uint32_t* __restrict__ endp)
{
    const int shift = 32 - 2 * depth;
    const uint32_t li = level_index(depth);
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t leaf = depth ? (codes[k] >> shift) : 0u;
        const double2 p = pos_in[perm[k]];
        pos64[k] = p;
        const uint32_t ix = compact16(leaf), iy = compact16(leaf >> 1);
        prel[k] = make_float2(f32_rn((p.x - minx) - off[ix]), f32_rn((p.y - miny) - off[iy]));
        if (k == 0 || (depth ? (codes[k - 1] >> shift) : 0u) != leaf) first[li + leaf] = (uint32_t)k;
        if (k == n - 1 || (depth ? (codes[k + 1] >> shift) : 0u) != leaf) endp[li + leaf] = (uint32_t)(k + 1);
    }
}

template <typename real>
__device__ inline void write_compute(int64_t node, double comx, double comy, double m0, double m2xx, double m2xy,
                                     double m2yy, double cx, double cy, real* comrel, real* m0r, real* m2t)
{
    comrel[2 * node] = (real)(comx - cx);
    comrel[2 * node + 1] = (real)(comy - cy);
    m0r[node] = (real)m0;
    double inv = m0 > 0.0 ? 1.0 / m0 : 0.0;
    m2t[3 * node] = (real)(inv * m2xx);
    m2t[3 * node + 1] = (real)(inv * m2xy);
    m2t[3 * node + 2] = (real)(inv * m2yy);
}

// createLeafNodes, second loop (:355-377) plus the first-occupant box (:343-350).
// The reference adds a leaf's particles one after the other in FP64, and its
// sums are reproduced bit for bit, so each sum is a chain of dependent
// additions.  kMomLanes lanes share a leaf: they load and multiply kMomChunk
// particles at a time in parallel, and one lane each runs the chains of x, y
// (then of xx, xy, yy) over the staged terms, so that a particle costs one
// FP64 warp instruction per loop and not eight (FP64 issues at 1/64 of the
// FP32 rate, as much for one lane as for 32).  The next chunk is loaded while
// the chains run.  What is left is the chain of the largest leaf: one draw of
// 200,003 particles of two disks in 4,096 leaves (largest 6,400; it follows the
// draw's outermost particles): 2,386 us with a thread per leaf, 736 us now.
constexpr int kMomLanes = 8;
constexpr int kMomChunk = 32;
constexpr int kMomThreads = 128;

template <typename real>
__global__ void __launch_bounds__(kMomThreads)
    k_leaf_moments(const double2* __restrict__ pos64, int depth, double minx, double miny, double h,
                   uint32_t* __restrict__ count, const uint32_t* __restrict__ first, double2* __restrict__ com64,
                   double* __restrict__ m0, double* __restrict__ m2, double2* __restrict__ bbc,
                   double* __restrict__ bblen, real* __restrict__ comrel, real* __restrict__ m0r,
                   real* __restrict__ m2t)
{
    constexpr int kPer = kMomChunk / kMomLanes;  // particles a lane loads per chunk
    constexpr int kGroups = kMomThreads / kMomLanes;
    // a group's staged terms; the odd row length spreads the groups over the banks
    __shared__ double s_term[kGroups][3 * kMomChunk + 1];
    const int sub = threadIdx.x % kMomLanes, group = threadIdx.x / kMomLanes;
    double* term = s_term[group];
    const uint32_t li = level_index(depth);
    const int64_t nl = (int64_t)1 << (2 * depth);
    // a warp's groups take neighbouring leaves and leave the loops together
    for (int64_t i0 = blockIdx.x * (int64_t)kGroups; i0 < nl; i0 += (int64_t)gridDim.x * kGroups) {
        const int64_t i = i0 + group;
        const int64_t node = li + i;
        const uint32_t f = i < nl ? first[node] : 0u;
        const uint32_t c = i < nl ? count[node] - f : 0u;  // count holds the end index here
        const uint32_t cmax = __reduce_max_sync(0xffffffffu, c);
        double2 q[kPer] = {};
        auto load = [&](uint32_t p0) {
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                const uint32_t p = p0 + u * kMomLanes + sub;
                if (p < c) q[u] = pos64[f + p];
            }
        };
        double chain = 0.0;
        load(0);
        for (uint32_t p0 = 0; p0 < cmax; p0 += kMomChunk) {
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                term[u * kMomLanes + sub] = q[u].x;
                term[kMomChunk + u * kMomLanes + sub] = q[u].y;
            }
            __syncwarp();
            load(p0 + kMomChunk);
            if (sub < 2) {
                const uint32_t m = c > p0 ? min(c - p0, (uint32_t)kMomChunk) : 0u;
                const double* t = term + sub * kMomChunk;
#pragma unroll 8
                for (uint32_t k = 0; k < m; k++) chain += t[k];
            }
            __syncwarp();
        }
        const double M0 = (double)c;
        chain /= M0;
        const double sx = __shfl_sync(0xffffffffu, chain, 0, kMomLanes);
        const double sy = __shfl_sync(0xffffffffu, chain, 1, kMomLanes);
        chain = 0.0;
        load(0);
        for (uint32_t p0 = 0; p0 < cmax; p0 += kMomChunk) {
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                const double rx = q[u].x - sx, ry = q[u].y - sy;
                term[u * kMomLanes + sub] = rx * rx;
                term[kMomChunk + u * kMomLanes + sub] = rx * ry;
                term[2 * kMomChunk + u * kMomLanes + sub] = ry * ry;
            }
            __syncwarp();
            load(p0 + kMomChunk);
            if (sub < 3) {
                const uint32_t m = c > p0 ? min(c - p0, (uint32_t)kMomChunk) : 0u;
                const double* t = term + sub * kMomChunk;
#pragma unroll 8
                for (uint32_t k = 0; k < m; k++) chain += t[k];
            }
            __syncwarp();
        }
        const double a = __shfl_sync(0xffffffffu, chain, 0, kMomLanes);
        const double b = __shfl_sync(0xffffffffu, chain, 1, kMomLanes);
        const double d = __shfl_sync(0xffffffffu, chain, 2, kMomLanes);
        if (sub != 0 || i >= nl) continue;
        count[node] = c;
        const uint32_t ix = compact16((uint32_t)i), iy = compact16((uint32_t)i >> 1);
        const double cx = minx + ((double)ix + 0.5) * h;
        const double cy = miny + ((double)iy + 0.5) * h;
        if (c == 0) {
            com64[node] = make_double2(0.0, 0.0);
            m0[node] = 0.0;
            m2[3 * node] = m2[3 * node + 1] = m2[3 * node + 2] = 0.0;
            bbc[node] = make_double2(0.0, 0.0);
            bblen[node] = 0.0;
            write_compute<real>(node, cx, cy, 0.0, 0.0, 0.0, 0.0, cx, cy, comrel, m0r, m2t);
            continue;
        }
        com64[node] = make_double2(sx, sy);
        m0[node] = M0;
        m2[3 * node] = a;
        m2[3 * node + 1] = b;
        m2[3 * node + 2] = d;
        // BBcentre = minPos + h * g + 0.5 * h (:345)
        bbc[node] = make_double2(minx + h * (double)ix + 0.5 * h, miny + h * (double)iy + 0.5 * h);
        bblen[node] = h;
        write_compute<real>(node, sx, sy, M0, a, b, d, cx, cy, comrel, m0r, m2t);
    }
}

// the arrays of the reference's node records and their compute copies
template <typename real>
struct NodeRecords {
    uint32_t* count;
    uint32_t* first;
    double2* com64;
    double* m0;
    double* m2;
    double2* bbc;
    double* bblen;
    real* comrel;
    real* m0r;
    real* m2t;
};

// bottomUpNodeConstruction (:381-470) for node i of level l
template <typename real>
__device__ __forceinline__ void bottom_up_node(int l, int64_t i, double minx, double miny, double hl, const NodeRecords<real>& t)
{
    const int64_t node = level_index(l) + i;
    const int64_t fc = level_index(l + 1) + 4 * i;
    uint32_t cnt = 0;
    int low = -1;  // the lowest non-empty child, whose box and first particle the reference's loop leaves
    double cx = 0.0, cy = 0.0, M0 = 0.0;
    for (int j = 3; j >= 0; j--) {
        const int64_t ch = fc + j;
        const uint32_t cc = t.count[ch];
        if (cc == 0) continue;
        low = j;
        cnt += cc;
        const double cm = t.m0[ch];
        const double2 cc2 = t.com64[ch];
        cx += cm * cc2.x;
        cy += cm * cc2.y;
        M0 += cm;
    }
    const uint32_t ix = compact16((uint32_t)i), iy = compact16((uint32_t)i >> 1);
    const double ccx = minx + ((double)ix + 0.5) * hl;
    const double ccy = miny + ((double)iy + 0.5) * hl;
    t.count[node] = cnt;
    if (cnt == 0) {
        t.first[node] = 0;
        t.com64[node] = make_double2(0.0, 0.0);
        t.m0[node] = 0.0;
        t.m2[3 * node] = t.m2[3 * node + 1] = t.m2[3 * node + 2] = 0.0;
        t.bbc[node] = make_double2(0.0, 0.0);
        t.bblen[node] = 0.0;
        write_compute<real>(node, ccx, ccy, 0.0, 0.0, 0.0, 0.0, ccx, ccy, t.comrel, t.m0r, t.m2t);
        return;
    }
    const double clen = t.bblen[fc + low];
    const double2 cb = t.bbc[fc + low];
    t.first[node] = t.first[fc + low];
    cx /= M0;
    cy /= M0;
    double a = 0.0, b = 0.0, d = 0.0;
    for (int j = 0; j < 4; j++) {
        const int64_t ch = fc + j;
        const double cm = t.m0[ch];
        if (cm == 0.0) continue;
        const double2 cc2 = t.com64[ch];
        const double rx = cc2.x - cx, ry = cc2.y - cy;
        a += rx * rx;
        b += rx * ry;
        d += ry * ry;
        a += t.m2[3 * ch];
        b += t.m2[3 * ch + 1];
        d += t.m2[3 * ch + 2];
    }
    t.com64[node] = make_double2(cx, cy);
    t.m0[node] = M0;
    t.m2[3 * node] = a;
    t.m2[3 * node + 1] = b;
    t.m2[3 * node + 2] = d;
    t.bbc[node] = make_double2(((low & 1) ? -0.5 : 0.5) * clen + cb.x, ((low & 2) ? -0.5 : 0.5) * clen + cb.y);
    t.bblen[node] = 2.0 * clen;
    write_compute<real>(node, cx, cy, M0, a, b, d, ccx, ccy, t.comrel, t.m0r, t.m2t);
}

template <typename real>
__global__ void k_bottom_up(int l, double minx, double miny, double hl, NodeRecords<real> t)
{
    const int64_t nl = (int64_t)1 << (2 * l);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nl; i += (int64_t)gridDim.x * blockDim.x)
        bottom_up_node<real>(l, i, minx, miny, hl, t);
}

// levels l0 (kTopBottomUp at most: 64 nodes) .. 0 in one block, a barrier between levels: launched by themselves they
// are 9 us each of latency
constexpr int kTopBottomUp = 3;
template <typename real>
__global__ void __launch_bounds__(64) k_bottom_up_top(int l0, double minx, double miny, double L, NodeRecords<real> t)
{
    for (int l = l0; l >= 0; l--) {
        if ((int64_t)threadIdx.x < ((int64_t)1 << (2 * l)))
            bottom_up_node<real>(l, threadIdx.x, minx, miny, L / (double)(1u << l), t);
        __syncthreads();
    }
}

template <typename real>
NodeRecords<real> node_records(Handle& h)
{
    return {P<uint32_t>(h.count), P<uint32_t>(h.first), P<double2>(h.com64), P<double>(h.m0), P<double>(h.m2),
            P<double2>(h.bbc), P<double>(h.bblen), P<real>(h.comrel), P<real>(h.m0r), P<real>(h.m2t)};
}

}  // namespace

// ---------------------------------------------------------------- active nodes
// The order-p passes over a level (M2M, M2L, L2L, P2M, lists) visit only its
// non-empty nodes: on clustered inputs most cells of the deep levels are empty
// (about 9 of 10 leaves at depth 11 for two 4M-particle disks), and a thread
// per cell would leave most lanes idle.
__global__ void k_act_flag(const uint32_t* __restrict__ count, int64_t nn, uint32_t* __restrict__ flag)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= nn; i += (int64_t)gridDim.x * blockDim.x)
        flag[i] = i < nn && count[i] != 0;
}

__global__ void k_act_scatter(const uint32_t* __restrict__ count, int64_t nn, const uint32_t* __restrict__ pos,
                              uint32_t* __restrict__ act)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x)
        if (count[i] != 0) act[pos[i]] = (uint32_t)i;
}

// the same in one block, kActChunk nodes at a time: 5,461 nodes 6 us, against 3, 5 and 3 in three launches
constexpr int kActThreads = 1024, kActItems = 8, kActChunk = kActThreads * kActItems;
constexpr int64_t kActBlock = 4 * kActChunk;
__global__ void __launch_bounds__(kActThreads)
    k_act_block(const uint32_t* __restrict__ count, int64_t nn, uint32_t* __restrict__ pos, uint32_t* __restrict__ act)
{
    uint32_t carry = 0;
    for (int64_t base = 0; base < nn; base += kActChunk) {
        const int64_t i0 = base + (int64_t)threadIdx.x * kActItems;
        uint32_t flags = 0;
#pragma unroll
        for (int i = 0; i < kActItems; i++) flags |= (i0 + i < nn && count[i0 + i] != 0 ? 1u : 0u) << i;
        uint32_t tot;
        uint32_t at = carry + block_exclusive_scan(__popc(flags), tot);
#pragma unroll
        for (int i = 0; i < kActItems; i++) {
            if (i0 + i >= nn) break;
            pos[i0 + i] = at;
            if (flags >> i & 1u) act[at++] = (uint32_t)(i0 + i);
        }
        carry += tot;
    }
    if (threadIdx.x == 0) pos[nn] = pos[nn + 1] = carry;
}

int build_active(Handle& h)
{
    cudaStream_t s = h.stream;
    const int64_t nn = h.nnodes;
    int rc;
    if ((rc = ensure(h.act, (nn + 1) * 4)) || (rc = ensure(h.act_pos, (nn + 2) * 4)) ||
        (rc = ensure(h.tmp, scan_tmp_words(nn + 1) * 4)))
        return rc;
    uint32_t* act = P<uint32_t>(h.act);
    uint32_t* pos = P<uint32_t>(h.act_pos);
    if (nn <= kActBlock) {
        k_act_block<<<1, kActThreads, 0, s>>>(P<uint32_t>(h.count), nn, pos, act);
        h.launches++;
        TC_CUDA_TRY(cudaGetLastError());
        return TC_OK;
    }
    k_act_flag<<<grid_for(nn + 1, 256), 256, 0, s>>>(P<uint32_t>(h.count), nn, act);
    if ((rc = exclusive_scan_u32(act, pos, nn + 1, P<uint32_t>(h.tmp), s))) return rc;
    k_act_scatter<<<grid_for(nn, 256), 256, 0, s>>>(P<uint32_t>(h.count), nn, pos, act);
    h.launches += 2;
    TC_CUDA_TRY(cudaGetLastError());
    return TC_OK;
}

int build_tree(Handle& h, const double* d_pos, int64_t n, double minx, double miny, double maxx, double maxy)
{
    cudaStream_t s = h.stream;
    const double nmx = -minx, nmy = -miny;
    const double ax = maxx + nmx, ay = maxy + nmy;
    const double L = (ax < ay) ? ay : ax;  // compMax(maxPos - minPos) (:84-85)
    if (!(L > 0.0) || !std::isfinite(L)) {
        tc_set_error("bounding box must have a positive finite extent (got %g)", L);
        return TC_ERR_INVALID;
    }
    int depth = h.cfg.depth;
    if (depth < 0) {
        uint32_t d = 0;
        tc_get_depth(h.cfg.max_children, n, &d);
        depth = (int)d;
    }
    if (depth > 15) {
        tc_set_error("tree depth %d exceeds the 15 levels that 32-bit Morton codes resolve", depth);
        return TC_ERR_INVALID;
    }
    int64_t nn = 0;
    tc_node_count((uint32_t)depth, &nn);
    h.depth = depth;
    h.n = n;
    h.nnodes = nn;
    h.minx = minx;
    h.miny = miny;
    h.L = L;
    h.tree_ready = false;
    const bool f64 = h.cfg.precision == TC_PREC_FP64;
    const size_t rs = f64 ? 8 : 4;
    int rc = 0;
    if ((rc = ensure(h.codes, n * 4)) || (rc = ensure(h.perm, n * 4)) || (rc = ensure(h.alt_keys, n * 4)) ||
        (rc = ensure(h.alt_vals, n * 4)) || (rc = ensure(h.pos64, n * 16)) || (rc = ensure(h.prel, n * 2 * rs)) ||
        (rc = ensure(h.count, nn * 4)) || (rc = ensure(h.first, nn * 4)) || (rc = ensure(h.com64, nn * 16)) ||
        (rc = ensure(h.m0, nn * 8)) || (rc = ensure(h.m2, nn * 24)) || (rc = ensure(h.bbc, nn * 16)) ||
        (rc = ensure(h.bblen, nn * 8)) || (rc = ensure(h.comrel, nn * 2 * rs)) || (rc = ensure(h.m0r, nn * rs)) ||
        (rc = ensure(h.m2t, nn * 3 * rs)) || (rc = ensure(h.tmp, radix_tmp_words(n) * 4)) ||
        (rc = ensure(h.err, 64)))
        return rc;

    if ((rc = record(h, 0))) return rc;
    TC_CUDA_TRY(cudaMemsetAsync(h.err.p, 0, sizeof(uint32_t), s));
    // order p in FP32: the physics-mode moments of tree_p.cu.  Codes, permutation and topology are the
    // reference's on every path: FP64 Morton quantisation and a sort over all 32 code bits, whose tie
    // order (stable) fixes the in-leaf order the reference's unstable sort leaves undefined.
    const bool physics = h.cfg.order && !f64;
    // codes by the FP32 fast path; points near a cell edge queued per block for the FP64 path
    const int mgrid = grid_for(n, kMortonThreads);
    if ((rc = ensure(h.mqueue, (size_t)(mgrid * morton_region(n, mgrid) + mgrid) * 4))) return rc;
    uint32_t* mq = P<uint32_t>(h.mqueue);
    uint32_t* mcount = mq + mgrid * morton_region(n, mgrid);
    k_morton_fast<<<mgrid, kMortonThreads, 0, s>>>((const double2*)d_pos, n, minx, miny, maxx, maxy,
                                                   (float)(65536.0 / L), P<uint32_t>(h.codes), P<uint32_t>(h.err), mq,
                                                   mcount);
    const uint32_t li = level_index(depth);
    const int64_t nleaf = (int64_t)1 << (2 * depth);
    const double hleaf = L / (double)(1u << depth);
    const int w = 1 << depth;
    if (!f64 && (rc = ensure(h.celloff, (size_t)w * 8))) return rc;
    if (physics && (rc = ensure(h.bigleaf, (size_t)bigleaf_words(n) * 4))) return rc;
    // a tree of many more leaves than points is cleared faster by itself than by the points' few blocks: 2,000 points,
    // a whole update by the blocks and by clears: 33 leaves a point 202 and 209 us, 131: 257 and 258, 524: 332 and 318
    const bool sparse = nleaf > 128 * n;
    if (sparse) {
        TC_CUDA_TRY(cudaMemsetAsync(P<uint32_t>(h.count) + li, 0, nleaf * 4, s));
        TC_CUDA_TRY(cudaMemsetAsync(P<uint32_t>(h.first) + li, 0, nleaf * 4, s));
    }
    const TreePrep prep{P<uint32_t>(h.first) + li, P<uint32_t>(h.count) + li, sparse ? 0 : nleaf,
                        physics ? P<uint32_t>(h.bigleaf) : nullptr, f64 ? nullptr : P<double>(h.celloff), w, hleaf};
    k_morton_exact<<<mgrid, kMortonThreads, 0, s>>>((const double2*)d_pos, n, minx, miny, L, mq, mcount,
                                                    P<uint32_t>(h.codes), prep);
    h.launches += 2;
    TC_CUDA_TRY(cudaGetLastError());
    rc = radix_sort_u32(P<uint32_t>(h.codes), P<uint32_t>(h.perm), P<uint32_t>(h.alt_keys), P<uint32_t>(h.alt_vals), n,
                        P<uint32_t>(h.tmp), s, &h.launches, 0);
    if (rc || (rc = record(h, 1))) return rc;
    if (f64) {
        k_gather_bounds<double><<<grid_for(n, 256), 256, 0, s>>>(P<uint32_t>(h.codes), P<uint32_t>(h.perm),
                                                                 (const double2*)d_pos, n, depth, minx, miny, hleaf,
                                                                 P<double2>(h.pos64), P<double>(h.prel),
                                                                 P<uint32_t>(h.first), P<uint32_t>(h.count));
        k_leaf_moments<double><<<grid_for(nleaf * kMomLanes, kMomThreads), kMomThreads, 0, s>>>(
            P<double2>(h.pos64), depth, minx, miny, hleaf, P<uint32_t>(h.count), P<uint32_t>(h.first),
            P<double2>(h.com64), P<double>(h.m0), P<double>(h.m2), P<double2>(h.bbc), P<double>(h.bblen),
            P<double>(h.comrel), P<double>(h.m0r), P<double>(h.m2t));
    } else {
        k_gather_bounds_f32<<<grid_for(n, 256), 256, 0, s>>>(P<uint32_t>(h.codes), P<uint32_t>(h.perm),
                                                             (const double2*)d_pos, n, depth, minx, miny,
                                                             P<double>(h.celloff), P<double2>(h.pos64),
                                                             P<float2>(h.prel), P<uint32_t>(h.first),
                                                             P<uint32_t>(h.count));
        if (physics) {
            if ((rc = build_records_p(h, hleaf))) return rc;
        } else {
            k_leaf_moments<float><<<grid_for(nleaf * kMomLanes, kMomThreads), kMomThreads, 0, s>>>(
                P<double2>(h.pos64), depth, minx, miny, hleaf, P<uint32_t>(h.count), P<uint32_t>(h.first),
                P<double2>(h.com64), P<double>(h.m0), P<double>(h.m2), P<double2>(h.bbc), P<double>(h.bblen),
                P<float>(h.comrel), P<float>(h.m0r), P<float>(h.m2t));
        }
    }
    h.launches += physics ? 1 : 2;
    if (!physics && depth > 0) {
        const int top = depth - 1 < kTopBottomUp ? depth - 1 : kTopBottomUp;
        for (int l = depth - 1; l > top; l--) {
            const double hl = L / (double)(1u << l);
            const int64_t nl = (int64_t)1 << (2 * l);
            if (f64)
                k_bottom_up<double><<<grid_for(nl, 64), 64, 0, s>>>(l, minx, miny, hl, node_records<double>(h));
            else
                k_bottom_up<float><<<grid_for(nl, 64), 64, 0, s>>>(l, minx, miny, hl, node_records<float>(h));
        }
        if (f64)
            k_bottom_up_top<double><<<1, 64, 0, s>>>(top, minx, miny, L, node_records<double>(h));
        else
            k_bottom_up_top<float><<<1, 64, 0, s>>>(top, minx, miny, L, node_records<float>(h));
        h.launches += depth - top;
    }
    TC_CUDA_TRY(cudaGetLastError());
    if (h.cfg.order && (rc = build_active(h))) return rc;
    // order-p multipoles belong to the tree: the list builder's controller reads them
    if (h.cfg.order && !h.split_mu && (rc = build_multipoles(h))) return rc;
    if ((rc = record(h, 2))) return rc;
    h.tree_ready = true;
    return TC_OK;
}

}  // namespace tc
