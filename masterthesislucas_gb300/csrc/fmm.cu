// Force evaluation of the symmetric Morton FMM at the reference's fixed
// order: multipoles M0 + M2 about the centre of mass, local expansion C1, C2,
// C3 (src/nbodysolvers/cpu/nBodySolverFMM_SYM_MORTON.h:622-836), evaluated
// sink by sink from the interaction lists built in lists.cu.
//
// The reference applies each symmetric kernel to both nodes of a pair; here
// each direction is evaluated by its own sink, so nothing is accumulated by
// atomics and results are deterministic:
//   k_m2l     one warp per node A: C(A) += M2L(B -> A) for B in nn(A)
//             (kernelNN, :622-723; the MA0 factor that applyForces later
//             divides out (:488-492) is never applied)
//   k_leaf_local, k_leaf_near  one block per non-empty leaf S, per 32 sinks of S:
//             C_S = own C(S) + every ancestor's C shifted to com_S
//                   (applyForces' L2L chain, :482-519, composed per leaf)
//                 + P2L from points t of partners T < S with pass(t, S)
//                   (kernelPN second half, :764-814)
//             g_s = L2P(C_S) (:521-534)
//                 + self P2P over S (the j >= i loop of :176-192)
//                 + for T > S: M2P(T) if pass(s, T) else P2P over T
//                 + for T < S: P2P from the t in T with !pass(t, S)
// where pass(x, B) is the point-node MAC of traverse_SYM_PN (:272-313),
// |x - com_B|^2 > (L_B / theta)^2, evaluated in FP64 like the reference.  For
// a leaf pair the reference tests the points of the first node of the pair
// (the lower Morton index) against the second, which is what fixes the roles
// above.  Geometry is in cell-relative coordinates: offsets between cells are
// integer multiples of the cell size, so FP32 differences lose nothing to the
// absolute position magnitude.
#include <cmath>

#include "kernels.cuh"
#include "state.cuh"

namespace tc {
namespace {

// C1 of a source with mass m0 and normalised second moment T = M2/M0 (:638-655)
template <typename real>
__device__ inline void far_c1(real Rx, real Ry, real m0, real Txx, real Txy, real Tyy, real D1, real D2, real D3,
                              real& ox, real& oy)
{
    real S1 = Txx + Tyy;
    real S2 = Rx * Rx * Txx + real(2) * Rx * Ry * Txy + Ry * Ry * Tyy;
    real S3x = Rx * Txx + Ry * Txy;
    real S3y = Rx * Txy + Ry * Tyy;
    real base = D1 + real(0.5) * S1 * D2 + real(0.5) * S2 * D3;
    ox = m0 * (Rx * base + S3x * D2);
    oy = m0 * (Ry * base + S3y * D2);
}

// C2 and C3 of a monopole of mass m at offset R (:657-697)
template <typename real>
__device__ inline void add_c2c3(real Rx, real Ry, real m, real D1, real D2, real D3, real* C)
{
    C[L_C2XX] += m * (D1 + Rx * Rx * D2);
    C[L_C2XY] += m * (Rx * Ry * D2);
    C[L_C2YY] += m * (D1 + Ry * Ry * D2);
    C[L_C3XXX] += m * (real(3) * Rx * D2 + Rx * Rx * Rx * D3);
    C[L_C3XXY] += m * (Ry * D2 + Rx * Rx * Ry * D3);
    C[L_C3XYY] += m * (Rx * D2 + Rx * Ry * Ry * D3);
    C[L_C3YYY] += m * (real(3) * Ry * D2 + Ry * Ry * Ry * D3);
}

// evaluate C1 + d.C2 + 1/2 d.(d.C3) (the L2P / L2L C1 formula, :501-531)
template <typename real>
__device__ inline void eval_c1(const real* C, real dx, real dy, real& gx, real& gy)
{
    real txx = dx * C[L_C3XXX] + dy * C[L_C3XXY];
    real txy = dx * C[L_C3XXY] + dy * C[L_C3XYY];
    real tyy = dx * C[L_C3XYY] + dy * C[L_C3YYY];
    gx = C[L_C1X] + (dx * C[L_C2XX] + dy * C[L_C2XY]) + real(0.5) * (dx * txx + dy * txy);
    gy = C[L_C1Y] + (dx * C[L_C2XY] + dy * C[L_C2YY]) + real(0.5) * (dx * txy + dy * tyy);
}

// L2L shift of an expansion by d, added into acc (:497-516)
template <typename real>
__device__ inline void add_shifted(const real* C, real dx, real dy, real* acc)
{
    real gx, gy;
    eval_c1(C, dx, dy, gx, gy);
    acc[L_C1X] += gx;
    acc[L_C1Y] += gy;
    acc[L_C2XX] += C[L_C2XX] + dx * C[L_C3XXX] + dy * C[L_C3XXY];
    acc[L_C2XY] += C[L_C2XY] + dx * C[L_C3XXY] + dy * C[L_C3XYY];
    acc[L_C2YY] += C[L_C2YY] + dx * C[L_C3XYY] + dy * C[L_C3YYY];
    acc[L_C3XXX] += C[L_C3XXX];
    acc[L_C3XXY] += C[L_C3XXY];
    acc[L_C3XYY] += C[L_C3XYY];
    acc[L_C3YYY] += C[L_C3YYY];
}

struct Geo {
    int depth;
    double inv_theta;
    double theta;
    double h_leaf;     // leaf cell size
    double far;        // largest coordinate of the box: cell centres are rounded by 2^-53 of it
    int variant;       // 1: the non-symmetric FMM_MORTON leaf stage
};

// box / 2^l, exactly
__device__ __forceinline__ float level_size(float box, int l) { return box * __int_as_float((127 - l) << 23); }
__device__ __forceinline__ double level_size(double box, int l)
{
    return box * __longlong_as_double((long long)(1023 - l) << 52);
}

// all levels from 1 on in one launch (nodes n0 .. n1 of the level-dense numbering): they do not depend on one another
template <typename real, typename K>
__global__ void __launch_bounds__(128) k_m2l(K ker, int64_t n0, int64_t n1, real box, LevelLists lists,
                                             const real* __restrict__ comrel, const real* __restrict__ m0r,
                                             const real* __restrict__ m2t, real* __restrict__ loc,
                                             double* __restrict__ zpart)
{
    const int lane = threadIdx.x & 31;
    const int64_t wstride = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t na = n0 + blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); na < n1; na += wstride) {
        const int l = level_of((uint32_t)na);
        const uint32_t li = level_index(l);
        const int64_t nl = (int64_t)1 << (2 * l), a = na - li;
        const real hl = level_size(box, l);
        const uint32_t* nn_ptr = lists.ptr[l];
        const uint32_t* nn_idx = lists.idx[l];
        const uint32_t b0 = nn_ptr[a], b1 = nn_ptr[list_end(nl, a)];
        if (b0 == b1) {
            if (lane < L_NCOEF) loc[na * L_NCOEF + lane] = real(0);
            if (lane == 0) zpart[na] = 0.0;
            continue;
        }
        const int iax = (int)compact16((uint32_t)a), iay = (int)compact16((uint32_t)a >> 1);
        const real cax = comrel[2 * na], cay = comrel[2 * na + 1];
        real C[L_NCOEF];
#pragma unroll
        for (int c = 0; c < L_NCOEF; c++) C[c] = real(0);
        real z = real(0);
        for (uint32_t e = b0 + lane; e < b1; e += 32) {
            const uint32_t b = nn_idx[e];
            const int64_t nb = li + b;
            const int ibx = (int)compact16(b), iby = (int)compact16(b >> 1);
            const real Rx = real(iax - ibx) * hl + (cax - comrel[2 * nb]);
            const real Ry = real(iay - iby) * hl + (cay - comrel[2 * nb + 1]);
            real D1, D2, D3, t;
            ker.far(Rx * Rx + Ry * Ry, D1, D2, D3, t);
            const real mb = m0r[nb];
            real c1x, c1y;
            far_c1(Rx, Ry, mb, m2t[3 * nb], m2t[3 * nb + 1], m2t[3 * nb + 2], D1, D2, D3, c1x, c1y);
            C[L_C1X] += c1x;
            C[L_C1Y] += c1y;
            add_c2c3(Rx, Ry, mb, D1, D2, D3, C);
            z += mb * t;
        }
#pragma unroll
        for (int c = 0; c < L_NCOEF; c++) C[c] = warp_sum(C[c]);
        double zz = warp_sum((double)z) * (double)m0r[na];
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < L_NCOEF; c++) loc[na * L_NCOEF + c] = C[c];
            zpart[na] = zz;
        }
    }
}

// point-node MAC of the non-symmetric solver's traverseBHMP
// (nBodySolverFMM_MORTON.h:201-204): L_B / |x - com_B| < theta
__device__ inline bool pn_pass_m(double2 x, double2 com, double len, double theta)
{
    double dx = x.x - com.x, dy = x.y - com.y;
    return len / sqrt(dx * dx + dy * dy) < theta;
}

// point-node MAC of traverse_SYM_PN, exactly as the reference evaluates it
__device__ inline bool pn_pass(double2 x, double2 com, double len, double inv_theta)
{
    double dx = x.x - com.x, dy = x.y - com.y;
    double dist = dx * dx + dy * dy;
    double thr = len * inv_theta;
    return dist > thr * thr;
}

// The point-node MAC from the FP32 offset R = x - com_B (threshold thr =
// L_B / theta, the same for every non-empty leaf), decided in FP64 by exact()
// only where the FP32 squared distance is too close to the threshold: at the
// threshold R is off by at most a few 2^-24 (thr + 3 h), which moves |R|^2 by
// less than an eighth of the band (and by the rounding of the cells' centres,
// the band's second part).  FP64 runs at 1/64 of the FP32 rate, and
// the test is made for every particle and partner leaf.  (Squares below 1e-30
// are left to FP64: near the end of the normal range the band says nothing.)
template <typename real>
struct PointMac {
    real thr2, band;
    __device__ PointMac(real thr, real h, real far)
        : thr2(thr * thr),
          band(thr2 > real(1e-30) ? real(3.2e-6) * thr * (thr + real(3) * h) + real(0x1p-49) * thr * far
                                  : real(INFINITY))
    {
    }
    template <typename F>
    __device__ __forceinline__ bool pass(real Rx, real Ry, F&& exact) const
    {
        if (sizeof(real) == 4) {
            const real diff = (Rx * Rx + Ry * Ry) - thr2;
            if (fabs(diff) > band) return diff > real(0);
        }
        return exact();
    }
};

constexpr int kLeafWarps = 4;

// 32 entries of a near list, one per lane: leaf, first particle, count and the
// offset (cell of S - cell of the entry) h
template <typename real>
struct NearBatch {
    uint32_t ti, f, c;
    real ox, oy;
    __device__ __forceinline__ void load(const uint32_t* __restrict__ near_idx, const uint32_t* __restrict__ first,
                                         const uint32_t* __restrict__ count, uint32_t li, uint32_t e, uint32_t e1,
                                         int isx, int isy, real h)
    {
        ti = f = c = 0;
        ox = oy = real(0);
        if (e >= e1) return;
        ti = near_idx[e];
        f = first[li + ti];
        c = count[li + ti];
        ox = real(isx - (int)compact16(ti)) * h;
        oy = real(isy - (int)compact16(ti >> 1)) * h;
    }
    __device__ __forceinline__ NearBatch at(int k) const
    {
        NearBatch b;
        b.ti = __shfl_sync(0xffffffffu, ti, k);
        b.f = __shfl_sync(0xffffffffu, f, k);
        b.c = __shfl_sync(0xffffffffu, c, k);
        b.ox = __shfl_sync(0xffffffffu, ox, k);
        b.oy = __shfl_sync(0xffffffffu, oy, k);
        return b;
    }
};

// phase A, per non-empty leaf S: the final local expansion of S at com_S (own
// M2L + shifted ancestors + P2L from the passing points of partners T < S),
// and the number of 32-sink chunks of S.  A block takes kLeafWarps leaves, a
// warp each; a leaf of more than kLeafLocalBlock particles, which lies in a
// dense region, takes a block of its own: a warp alone was a
// serial chain of up to 10^5 points there (one draw of 200,003 particles of
// two disks: 947 us, 174 us now).  The points of 32 partners are one flat range
// dealt 32 at a time, so that partners of a few points fill the lanes too.
// Where the line lies, at 32, 64 and 256: 200,000 uniform particles, leaves of
// 64: 38, 29 and 28 us; 100,000 of twenty clusters: 91, 97 and 115; the disks
// with leaves of 256, whose outer leaves hold 32 to 64: 307, 642 and 905.
constexpr uint32_t kLeafLocalBlock = 64;

template <typename real, typename K>
__global__ void __launch_bounds__(32 * kLeafWarps)
    k_leaf_local(K ker, Geo geo, const uint32_t* __restrict__ count, const uint32_t* __restrict__ first,
                 const double2* __restrict__ com64, const double* __restrict__ bblen, const real* __restrict__ comrel,
                 const real* __restrict__ m0r, const real* __restrict__ loc, const uint32_t* __restrict__ near_ptr,
                 const uint32_t* __restrict__ near_idx, const double2* __restrict__ pos64,
                 const real* __restrict__ prel, real* __restrict__ locfin, double* __restrict__ zloc,
                 uint32_t* __restrict__ nchunk, unsigned long long* __restrict__ counters)
{
    __shared__ real s_part[kLeafWarps][L_NCOEF];
    __shared__ double s_z[kLeafWarps];
    uint32_t n_p2l = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int dep = geo.depth;
    const uint32_t li = level_index(dep);
    const int64_t nl = (int64_t)1 << (2 * dep);
    const real h = (real)geo.h_leaf;
    const PointMac<real> mac((real)(geo.h_leaf * geo.inv_theta), h, (real)geo.far);
    const double inv_theta = geo.inv_theta;
    // leaf si by nv warps, this one taking runs v, v + nv, ... of its partners' points; C and z are the warp's sums
    auto leaf = [&](int64_t si, int v, int nv, real (&C)[L_NCOEF], double& z) {
        const int64_t S = li + si;
        const int isx = (int)compact16((uint32_t)si), isy = (int)compact16((uint32_t)si >> 1);
        const real csx = comrel[2 * S], csy = comrel[2 * S + 1];
        const real mS = m0r[S];
        const uint32_t e0 = near_ptr[si], e1 = near_ptr[list_end(nl, si)];
#pragma unroll
        for (int c = 0; c < L_NCOEF; c++) C[c] = real(0);
        real zA = real(0);
        if (v == 0 && lane <= dep) {
            // lane k shifts the expansion of the ancestor at level k (k == dep is S)
            const int k = lane;
            const uint32_t ai = (uint32_t)((uint64_t)si >> (2 * (dep - k)));
            const int64_t A = level_index(k) + ai;
            real CA[L_NCOEF];
#pragma unroll
            for (int c = 0; c < L_NCOEF; c++) CA[c] = loc[A * L_NCOEF + c];
            const real scale = (real)(1 << (dep - k));
            const real iax = (real)compact16(ai), iay = (real)compact16(ai >> 1);
            // com_S - com_A = (cell centre offset) + (relative COMs)
            const real dx = h * (((real)isx + real(0.5)) - (iax + real(0.5)) * scale) + (csx - comrel[2 * A]);
            const real dy = h * (((real)isy + real(0.5)) - (iay + real(0.5)) * scale) + (csy - comrel[2 * A + 1]);
            add_shifted(CA, dx, dy, C);
        }
        // partners T < S: lists are in ascending order, so they come first (the non-symmetric solver has no P2L here)
        for (uint32_t eb = e0; eb < e1 && !geo.variant; eb += 32) {
            NearBatch<real> batch;
            batch.load(near_idx, first, count, li, eb + lane, e1, isx, isy, h);
            const uint32_t nt = __popc(__ballot_sync(0xffffffffu, eb + lane < e1 && batch.ti < (uint32_t)si));
            const uint32_t mc = (uint32_t)lane < nt ? batch.c : 0u;
            uint32_t inc = mc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            const uint32_t ex = inc - mc, tot = __shfl_sync(0xffffffffu, inc, 31);
            for (uint32_t base = 32u * (uint32_t)v; base < tot; base += 32u * (uint32_t)nv) {
                // position q belongs to the last entry that starts at or before it (every entry is a non-empty leaf)
                const uint32_t q = base + lane;
                const uint32_t before = __popc(__ballot_sync(0xffffffffu, (uint32_t)lane < nt && ex < base));
                const uint32_t d = ex - base;
                const uint32_t bits = __reduce_or_sync(0xffffffffu, ((uint32_t)lane < nt && d < 32u) ? 1u << d : 0u);
                const int k = (int)(before + __popc(bits & (0xffffffffu >> (31 - lane)))) - 1;
                const NearBatch<real> T = batch.at(k);
                const uint32_t exT = __shfl_sync(0xffffffffu, ex, k);
                if (q >= tot) continue;
                const uint32_t t = T.f + (q - exT);
                // R' = com_S - x_t
                const real Rx = T.ox + (csx - prel[2 * t]);
                const real Ry = T.oy + (csy - prel[2 * t + 1]);
                if (!mac.pass(Rx, Ry, [&] { return pn_pass(pos64[t], com64[S], bblen[S], inv_theta); }))
                    continue;
                real D1, D2, D3, tt;
                ker.far(Rx * Rx + Ry * Ry, D1, D2, D3, tt);
                C[L_C1X] += Rx * D1;
                C[L_C1Y] += Ry * D1;
                add_c2c3(Rx, Ry, real(1), D1, D2, D3, C);
                zA += mS * tt;
                n_p2l++;
            }
            if (nt < 32u) break;
        }
#pragma unroll
        for (int c = 0; c < L_NCOEF; c++) C[c] = warp_sum(C[c]);
        z = (double)warp_sum(zA);
    };
    for (int64_t s0 = blockIdx.x * (int64_t)kLeafWarps; s0 < nl; s0 += (int64_t)gridDim.x * kLeafWarps) {
        real C[L_NCOEF];
        double z;
        const int64_t own = s0 + w;
        const uint32_t cO = own < nl ? count[li + own] : 0u;
        if (own < nl) {
            if (lane == 0) nchunk[own] = (cO + 31u) / 32u;
            if (cO == 0) {
                if (lane == 0) zloc[own] = 0.0;
            } else if (cO <= kLeafLocalBlock) {
                leaf(own, 0, 1, C, z);
                if (lane == 0) {
#pragma unroll
                    for (int c = 0; c < L_NCOEF; c++) locfin[own * L_NCOEF + c] = C[c];
                    zloc[own] = z;
                }
            }
        }
    }
    for (int64_t si = blockIdx.x; si < nl; si += gridDim.x) {
        if (count[li + si] <= kLeafLocalBlock) continue;  // the same in the whole block
        real C[L_NCOEF];
        double z;
        leaf(si, w, kLeafWarps, C, z);
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < L_NCOEF; c++) s_part[w][c] = C[c];
            s_z[w] = z;
        }
        __syncthreads();
        if (threadIdx.x < L_NCOEF) {
            real sum = s_part[0][threadIdx.x];
#pragma unroll
            for (int i = 1; i < kLeafWarps; i++) sum += s_part[i][threadIdx.x];
            locfin[si * L_NCOEF + threadIdx.x] = sum;
        }
        if (threadIdx.x == 0) {
            double sum = s_z[0];
#pragma unroll
            for (int i = 1; i < kLeafWarps; i++) sum += s_z[i];
            zloc[si] = sum;
        }
        __syncthreads();
    }
    const unsigned long long c = warp_sum((unsigned long long)n_p2l);
    if (lane == 0 && c) atomicAdd(counters + 2, c);
}

// sources a warp of phase B stages before it evaluates them (a multiple of 8
// per lane of a sink, for 1 to 32 lanes)
constexpr int kLeafBuf = 256;

// the staged sources of one warp in the sink leaf's frame: FP32 two per
// 16-byte slot for the packed loop, FP64 one per slot
template <typename K>
__device__ __forceinline__ void leaf_stage(float* buf, uint32_t q, float x, float y)
{
    buf[(q >> 1) * 4 + (q & 1)] = x;
    buf[(q >> 1) * 4 + 2 + (q & 1)] = y;
}
template <typename K>
__device__ __forceinline__ void leaf_stage(double* buf, uint32_t q, double x, double y)
{
    buf[2 * q] = x;
    buf[2 * q + 1] = y;
}
__device__ __forceinline__ float2 leaf_staged(const float* buf, uint32_t q)
{
    return make_float2(buf[(q >> 1) * 4 + (q & 1)], buf[(q >> 1) * 4 + 2 + (q & 1)]);
}
__device__ __forceinline__ double2 leaf_staged(const double* buf, uint32_t q)
{
    return make_double2(buf[2 * q], buf[2 * q + 1]);
}

// the sink (px, py) against its lane's share of n staged sources (g lanes a sink, this one the r-th)
template <typename K>
__device__ __forceinline__ void leaf_eval(const K& ker, const float* buf, uint32_t n8, uint32_t r, uint32_t g,
                                          float px, float py, float& gx, float& gy, float& zs)
{
    unsigned long long ax = 0ull, ay = 0ull, az = 0ull;
    p2p_slots(ker, reinterpret_cast<const float4*>(buf), n8 / 2, r, g, px, py, ax, ay, az);
    gx += K::kSign * f2_total(ax);
    gy += K::kSign * f2_total(ay);
    zs += K::kSign * f2_total(az);
}
template <typename K>
__device__ __forceinline__ void leaf_eval(const K& ker, const double* buf, uint32_t n, uint32_t r, uint32_t g,
                                          double px, double py, double& gx, double& gy, double& zs)
{
    for (uint32_t j = r; j < n; j += g) {
        const double2 s = leaf_staged(buf, j);
        const double Rx = px - s.x, Ry = py - s.y;
        double D1, t;
        ker.near(Rx * Rx + Ry * Ry, D1, t);
        gx += D1 * Rx;
        gy += D1 * Ry;
        zs += t;
    }
}

// phase B, one block per work item (leaf S, chunk of up to 32 sinks of S).
// The P2P pairs bound it.  The block's warps take the 32-point runs of each
// partner in turn, every warp with all of the item's sinks (a sink of an item
// of m sinks gets g = 2^floor(log2(32/m)) of a warp's lanes, which split the
// sources), and stage the points that interact directly, shifted into S's
// frame, until kLeafBuf of them can be evaluated at once; runs that only some
// of the sinks see are evaluated by themselves.  The warps' sums are added in
// warp order.  The same draw of 200,003 particles of two disks, theta 0.5:
// 2,805 us with a warp per item and one source at a time, 1,546 us now.
template <typename real, typename K>
__global__ void __launch_bounds__(32 * kLeafWarps)
    k_leaf_near(K ker, Geo geo, const uint32_t* __restrict__ count, const uint32_t* __restrict__ first,
                const double2* __restrict__ com64, const double* __restrict__ bblen, const real* __restrict__ comrel,
                const real* __restrict__ m0r, const real* __restrict__ m2t, const real* __restrict__ locfin,
                const uint32_t* __restrict__ near_ptr, const uint32_t* __restrict__ near_idx,
                const uint32_t* __restrict__ chunk_ptr, const double2* __restrict__ pos64,
                const real* __restrict__ prel, const uint32_t* __restrict__ perm, double* __restrict__ grad,
                int accumulate, int scatter, double* __restrict__ zwork, unsigned long long* __restrict__ counters)
{
    __shared__ __align__(16) real s_src[kLeafWarps][2 * kLeafBuf];
    __shared__ real s_part[kLeafWarps][3][32];
    uint32_t n_pp = 0, n_m2p = 0;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    real* buf = s_src[w];
    const int dep = geo.depth;
    const uint32_t li = level_index(dep);
    const int64_t nl = (int64_t)1 << (2 * dep);
    const real h = (real)geo.h_leaf;
    const PointMac<real> mac((real)(geo.h_leaf * geo.inv_theta), h, (real)geo.far);
    const double inv_theta = geo.inv_theta;
    const uint32_t nwork = chunk_ptr[nl];
    for (uint32_t wi = blockIdx.x; wi < nwork; wi += gridDim.x) {
        // leaf of this work item: last si with chunk_ptr[si] <= wi
        int64_t lo = 0, hi = nl;
        while (hi - lo > 1) {
            const int64_t mid = (lo + hi) >> 1;
            if (chunk_ptr[mid] <= wi) lo = mid; else hi = mid;
        }
        const int64_t si = lo;
        const int64_t S = li + si;
        const uint32_t fS = first[S];
        const uint32_t c0 = (wi - chunk_ptr[si]) * 32u;
        const uint32_t m = min(32u, count[S] - c0);
        const int isx = (int)compact16((uint32_t)si), isy = (int)compact16((uint32_t)si >> 1);
        const real csx = comrel[2 * S], csy = comrel[2 * S + 1];
        const uint32_t e0 = near_ptr[si], e1 = near_ptr[list_end(nl, si)];
        const uint32_t lg = 5u - (32u - __clz(m - 1u));  // log2 g, g * m <= 32
        const uint32_t g = 1u << lg, r = lane & (g - 1u), sk = lane >> lg;
        const bool act = sk < m;
        const uint32_t sl = c0 + (act ? sk : 0u);
        const uint32_t s = fS + sl;
        const real px = prel[2 * s], py = prel[2 * s + 1];
        real gx = real(0), gy = real(0), zs = real(0);
        uint32_t fill = 0;
        // evaluates the staged sources for the sinks of the lanes in `sees`
        auto flush = [&](bool sees) {
            if (fill == 0) return;
            uint32_t n = fill;
            if (sizeof(real) == 4) {
                n = (fill + 8u * g - 1u) / (8u * g) * (8u * g);
                for (uint32_t q = fill + lane; q < n; q += 32u) leaf_stage<K>(buf, q, (real)kFarAway, (real)kFarAway);
            }
            __syncwarp();
            if (sees) {
                leaf_eval(ker, buf, n, r, g, px, py, gx, gy, zs);
                if (r == 0) n_pp += fill;
            }
            __syncwarp();
            fill = 0;
        };
        // a run of up to 32 points of a partner: those with `take`, in the sink leaf's frame
        auto append = [&](bool take, real x, real y) {
            const uint32_t bal = __ballot_sync(0xffffffffu, take);
            if (take) leaf_stage<K>(buf, fill + __popc(bal & ((1u << lane) - 1u)), x, y);
            fill += __popc(bal);
        };
        for (uint32_t eb = e0; eb < e1; eb += 32) {
            NearBatch<real> batch;
            batch.load(near_idx, first, count, li, eb + lane, e1, isx, isy, h);
            const int nt = (int)min(32u, e1 - eb);
            for (int k = 0; k < nt; k++) {
                const uint32_t q1 = 32u * ((w + (uint32_t)k) % kLeafWarps);  // this warp's first run
                const NearBatch<real> T = batch.at(k);
                if (q1 > 0 && q1 >= T.c) continue;
                const int64_t nT = li + T.ti;
                bool direct = act;
                if (geo.variant || T.ti > (uint32_t)si) {
                    // symmetric: S is the first node of the pair and each sink is tested against T; non-symmetric:
                    // every sink tests every partner T, S itself included (traverseBHMP, :199-232)
                    const real Rx = (T.ox + px) - comrel[2 * nT], Ry = (T.oy + py) - comrel[2 * nT + 1];
                    const bool pass = act && mac.pass(Rx, Ry, [&] {
                        return geo.variant ? pn_pass_m(pos64[s], com64[nT], bblen[nT], geo.theta)
                                           : pn_pass(pos64[s], com64[nT], bblen[nT], inv_theta);
                    });
                    if (pass && q1 == 0 && r == 0) {
                        real D1, D2, D3, t;
                        ker.far(Rx * Rx + Ry * Ry, D1, D2, D3, t);
                        const real mT = m0r[nT];
                        real c1x, c1y;
                        far_c1(Rx, Ry, mT, m2t[3 * nT], m2t[3 * nT + 1], m2t[3 * nT + 2], D1, D2, D3, c1x, c1y);
                        gx += c1x;
                        gy += c1y;
                        zs += mT * t;
                        n_m2p++;
                    }
                    direct = act && !pass;
                }
                if (!__any_sync(0xffffffffu, direct)) continue;
                const bool all = __all_sync(0xffffffffu, direct || !act);
                const bool tested = !geo.variant && T.ti < (uint32_t)si;  // S is the second node of the pair
                if (!all) flush(act);
                for (uint32_t q0 = q1; q0 < T.c; q0 += 32u * kLeafWarps) {
                    const uint32_t q = q0 + lane;
                    real x = real(0), y = real(0);
                    bool take = q < T.c;
                    if (take) {
                        const uint32_t t = T.f + q;
                        const real tx = prel[2 * t], ty = prel[2 * t + 1];
                        // only the points of T that fail the MAC against S interact with the sinks directly
                        if (tested)
                            take = !mac.pass(T.ox + (csx - tx), T.oy + (csy - ty), [&] {
                                return pn_pass(pos64[t], com64[S], bblen[S], inv_theta);
                            });
                        x = tx - T.ox;
                        y = ty - T.oy;
                    }
                    if (T.ti == (uint32_t)si && q0 == c0) {
                        // the sinks themselves: each against the others, one at a time
                        flush(all ? act : direct);
                        append(take, x, y);
                        __syncwarp();
                        if (direct) {
                            for (uint32_t j = r; j < m; j += g) {
                                if (j == sk) continue;
                                const auto src = leaf_staged(buf, j);
                                const real Rx = px - src.x, Ry = py - src.y;
                                real D1, t;
                                ker.near(Rx * Rx + Ry * Ry, D1, t);
                                gx += D1 * Rx;
                                gy += D1 * Ry;
                                zs += t;
                            }
                            if (r == 0) n_pp += m - 1u;
                        }
                        __syncwarp();
                        fill = 0;
                        continue;
                    }
                    append(take, x, y);
                    if (fill > kLeafBuf - 32) flush(all ? act : direct);
                }
                if (!all) flush(direct);
            }
        }
        flush(act);
        for (uint32_t o = g >> 1; o > 0; o >>= 1) {
            gx += __shfl_xor_sync(0xffffffffu, gx, o);
            gy += __shfl_xor_sync(0xffffffffu, gy, o);
        }
        s_part[w][0][lane] = gx;
        s_part[w][1][lane] = gy;
        s_part[w][2][lane] = act ? zs : real(0);
        __syncthreads();
        if (w == 0) {
            real C[L_NCOEF];
#pragma unroll
            for (int c = 0; c < L_NCOEF; c++) C[c] = locfin[si * L_NCOEF + c];
            eval_c1(C, px - csx, py - csy, gx, gy);
            real z = real(0);
#pragma unroll
            for (int i = 0; i < kLeafWarps; i++) {
                gx += s_part[i][0][lane];
                gy += s_part[i][1][lane];
                z += s_part[i][2][lane];
            }
            if (act && r == 0) {
                const int64_t o = scatter ? (int64_t)perm[s] : (int64_t)s;
                double ox2 = (double)gx, oy2 = (double)gy;
                if (accumulate) {
                    ox2 += grad[2 * o];
                    oy2 += grad[2 * o + 1];
                }
                grad[2 * o] = ox2;
                grad[2 * o + 1] = oy2;
            }
            const double zz = warp_sum((double)z);
            if (lane == 0) zwork[wi] = zz;
        }
        __syncthreads();
    }
    const unsigned long long a = warp_sum((unsigned long long)n_pp);
    const unsigned long long b = warp_sum((unsigned long long)n_m2p);
    if (lane == 0 && (a | b)) {
        atomicAdd(counters + 0, a);
        atomicAdd(counters + 1, b);
    }
}

// deterministic sum of the Z partials: per node (M2L), per leaf (P2L) and
// per work item (near field; the count is read from the chunk offsets)
__global__ void k_sum_z(const double* __restrict__ a, int64_t na, const double* __restrict__ b, int64_t nb,
                        const double* __restrict__ c, const uint32_t* __restrict__ nc, double* __restrict__ out,
                        int accumulate)
{
    __shared__ double ws[32];
    double s = 0.0;
    const int64_t ncv = *nc;
    for (int64_t i = threadIdx.x; i < na; i += blockDim.x) s += a[i];
    for (int64_t i = threadIdx.x; i < nb; i += blockDim.x) s += b[i];
    for (int64_t i = threadIdx.x; i < ncv; i += blockDim.x) s += c[i];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? ws[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) *out = accumulate ? *out + v : v;
    }
}

// final local expansion of every node (what applyForces leaves in the
// reference's node C fields): leaves from the leaf kernel, internal nodes by
// composing the shifted expansions of their ancestors
template <typename real>
__global__ void k_final_locals(int dep, double L, const uint32_t* __restrict__ count,
                               const real* __restrict__ comrel, const real* __restrict__ loc,
                               const real* __restrict__ locfin, double* __restrict__ out, int64_t nn)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nn; k += (int64_t)gridDim.x * blockDim.x) {
        int l = 0;
        while (l < dep && (int64_t)level_index(l + 1) <= k) l++;
        const uint32_t i = (uint32_t)(k - level_index(l));
        real C[L_NCOEF];
#pragma unroll
        for (int c = 0; c < L_NCOEF; c++) C[c] = real(0);
        if (count[k] != 0) {
            if (l == dep) {
                for (int c = 0; c < L_NCOEF; c++) C[c] = locfin[(int64_t)i * L_NCOEF + c];
            } else {
                const real h = (real)(L / (double)(1u << l));
                const real ix = (real)compact16(i), iy = (real)compact16(i >> 1);
                for (int a = 0; a <= l; a++) {
                    const uint32_t ai = i >> (2 * (l - a));
                    const int64_t A = level_index(a) + ai;
                    real CA[L_NCOEF];
                    for (int c = 0; c < L_NCOEF; c++) CA[c] = loc[A * L_NCOEF + c];
                    const real scale = (real)(1 << (l - a));
                    const real dx = h * ((ix + real(0.5)) - ((real)compact16(ai) + real(0.5)) * scale) +
                                    (comrel[2 * k] - comrel[2 * A]);
                    const real dy = h * ((iy + real(0.5)) - ((real)compact16(ai >> 1) + real(0.5)) * scale) +
                                    (comrel[2 * k + 1] - comrel[2 * A + 1]);
                    add_shifted(CA, dx, dy, C);
                }
            }
        }
        for (int c = 0; c < L_NCOEF; c++) out[k * L_NCOEF + c] = (double)C[c];
    }
}

template <typename real, typename K>
int solve_t(Handle& h, K ker, double* d_grad, int accumulate, int scatter, double* d_total)
{
    cudaStream_t s = h.stream;
    const int dep = h.depth;
    const int64_t nn = h.nnodes;
    const int64_t nleaf = (int64_t)1 << (2 * dep);
    int rc;
    if ((rc = ensure(h.loc, nn * L_NCOEF * sizeof(real))) || (rc = ensure(h.locfin, nleaf * L_NCOEF * sizeof(real))) ||
        (rc = ensure(h.zpart, nn * 8 + 64)))
        return rc;
    if ((rc = ensure(h.counters, 64)) || (rc = record(h, 4))) return rc;
    TC_CUDA_TRY(cudaMemsetAsync(h.counters.p, 0, 64, s));
    double* zp = P<double>(h.zpart);
    real* loc = P<real>(h.loc);
    // the root has no M2L partners
    TC_CUDA_TRY(cudaMemsetAsync(loc, 0, L_NCOEF * sizeof(real), s));
    TC_CUDA_TRY(cudaMemsetAsync(zp, 0, 8, s));
    const uint32_t* ptr = P<uint32_t>(h.ptr_pool);
    const uint32_t* idx = P<uint32_t>(h.idx_pool);
    if (dep > 0) {
        k_m2l<real, K><<<grid_for((nn - 1) * 32, 128, sm_count() * 64), 128, 0, s>>>(
            ker, 1, nn, (real)h.L, level_lists(h), P<real>(h.comrel), P<real>(h.m0r), P<real>(h.m2t), loc, zp);
        h.launches++;
    }
    Geo geo;
    geo.depth = dep;
    geo.inv_theta = 1.0 / h.cfg.theta;
    geo.theta = h.cfg.theta;
    geo.h_leaf = h.L / (double)(1u << dep);
    geo.far = std::fmax(std::fmax(std::fabs(h.minx), std::fabs(h.minx + h.L)),
                        std::fmax(std::fabs(h.miny), std::fabs(h.miny + h.L)));
    geo.variant = h.variant;
    // work items of the near field: 32-sink chunks of the non-empty leaves
    const int64_t wmax = h.n / 32 + (h.n < nleaf ? h.n : nleaf) + 1;
    if ((rc = ensure(h.chunk, (nleaf + 1) * 4)) || (rc = ensure(h.zwork, wmax * 8)) ||
        (rc = ensure(h.zloc, nleaf * 8)) || (rc = ensure(h.cnt_tmp, nleaf * 4 + 64)) ||
        (rc = ensure(h.tmp, scan_tmp_words(nleaf) * 4)))
        return rc;
    uint32_t* nchunk = P<uint32_t>(h.cnt_tmp);
    uint32_t* chunk_ptr = P<uint32_t>(h.chunk);
    k_leaf_local<real, K><<<(unsigned)(nleaf < sm_count() * 256 ? nleaf : sm_count() * 256), 32 * kLeafWarps, 0, s>>>(
        ker, geo, P<uint32_t>(h.count), P<uint32_t>(h.first), P<double2>(h.com64), P<double>(h.bblen),
        P<real>(h.comrel), P<real>(h.m0r), loc, ptr + h.lists.near_ptr_off[dep], idx + h.lists.near_idx_off[dep],
        P<double2>(h.pos64), P<real>(h.prel), P<real>(h.locfin), P<double>(h.zloc), nchunk,
        P<unsigned long long>(h.counters));
    if ((rc = exclusive_scan_u32(nchunk, chunk_ptr, nleaf, P<uint32_t>(h.tmp), s))) return rc;
    if ((rc = record(h, 5))) return rc;
    k_leaf_near<real, K><<<(unsigned)(wmax < sm_count() * 256 ? wmax : sm_count() * 256), 32 * kLeafWarps, 0, s>>>(
        ker, geo, P<uint32_t>(h.count), P<uint32_t>(h.first), P<double2>(h.com64), P<double>(h.bblen),
        P<real>(h.comrel), P<real>(h.m0r), P<real>(h.m2t), P<real>(h.locfin), ptr + h.lists.near_ptr_off[dep],
        idx + h.lists.near_idx_off[dep], chunk_ptr, P<double2>(h.pos64), P<real>(h.prel), P<uint32_t>(h.perm),
        d_grad, accumulate, scatter, P<double>(h.zwork), P<unsigned long long>(h.counters));
    if ((rc = record(h, 6))) return rc;
    k_sum_z<<<1, 1024, 0, s>>>(zp, nn, P<double>(h.zloc), nleaf, P<double>(h.zwork), chunk_ptr + nleaf, d_total, 1);
    h.launches += 6;
    TC_CUDA_TRY(cudaGetLastError());
    return record(h, 7);
}

}  // namespace

int dump_final_locals(Handle& h, std::vector<double>& out)
{
    out.clear();
    if (!h.loc.p || !h.locfin.p) return TC_OK;
    const int64_t nn = h.nnodes;
    Buf tmp;
    int rc = ensure(tmp, nn * L_NCOEF * 8);
    if (rc) return rc;
    if (h.cfg.precision == TC_PREC_FP64)
        k_final_locals<double><<<grid_for(nn, 128), 128, 0, h.stream>>>(h.depth, h.L, P<uint32_t>(h.count),
                                                                       P<double>(h.comrel), P<double>(h.loc),
                                                                       P<double>(h.locfin), P<double>(tmp), nn);
    else
        k_final_locals<float><<<grid_for(nn, 128), 128, 0, h.stream>>>(h.depth, h.L, P<uint32_t>(h.count),
                                                                      P<float>(h.comrel), P<float>(h.loc),
                                                                      P<float>(h.locfin), P<double>(tmp), nn);
    out.resize(nn * L_NCOEF);
    cudaError_t e = cudaMemcpyAsync(out.data(), tmp.p, nn * L_NCOEF * 8, cudaMemcpyDeviceToHost, h.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h.stream);
    release(tmp);
    if (e != cudaSuccess) return tc_cuda_fail(e, "dump_final_locals");
    return TC_OK;
}

int solve_fmm(Handle& h, double* d_grad, double* d_total, int accumulate, int scatter)
{
    const double eps2 = h.cfg.softening * h.cfg.softening;
    if (h.cfg.precision == TC_PREC_FP64) {
        if (h.cfg.kernel == TC_KERNEL_GRAVITY) return solve_t<double>(h, KGrav<double>{eps2}, d_grad, accumulate, scatter, d_total);
        return solve_t<double>(h, KTsne<double>{}, d_grad, accumulate, scatter, d_total);
    }
    if (h.cfg.kernel == TC_KERNEL_GRAVITY) return solve_t<float>(h, KGrav<float>{(float)eps2}, d_grad, accumulate, scatter, d_total);
    return solve_t<float>(h, KTsne<float>{}, d_grad, accumulate, scatter, d_total);
}

}  // namespace tc
