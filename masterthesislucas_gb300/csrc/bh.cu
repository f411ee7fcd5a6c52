// Barnes-Hut on the GPU with the reference's own tree: NBodySolverBH + QuadTree
// (src/nbodysolvers/cpu/nBodySolverBH.h:33-116, src/trees/cpu/quadtree.h:29-172).
//
// Tree (level-synchronous, device):
//   root box [lo, lo + D + 1e-4]^2 (D = largest extent, quadtree.h:29-53); a
//   node with more than maxChildren occupants splits at mid = lo + (hi.x-lo.x)/2
//   on both axes (:104-107) into HH, HL, LH, LL (:109-134), each child keeping
//   its parent's occupant order.  Per level: classify the points of splitting
//   nodes, four scans give each point its slot in the stable quadrant
//   partition of its node, children are appended in HH, HL, LH, LL order.
// Masses and COMs (quadtree.h:137-172) are rebuilt bottom-up with the
// reference's types: float totalMass, FP64 COM, and the child COM seen by the
// parent through std::pair<float, glm::vec2>, i.e. rounded to float.
// Traversal (nBodySolverBH.h:56-89): per point, depth-first in the
// children order with the MAC l/|x - com| < theta; a node with at most one
// child is treated as a leaf (PP over all its occupants).  In FP64 the
// result is the reference's, bit for bit (same operations, same order).
//
// Trees of up to kPathLevels levels (all but clusters of nearly coincident
// points) are built by one sort instead: a point's quadrants level by level
// are a key, the key order is the depth-first order, and a node is a run of
// keys with a common prefix.  Nodes are numbered depth first, so the
// traversal needs no stack: the next node is the following one, or the one
// after the subtree.  It visits the nodes a warp at a time, the warp's 32
// points being neighbours in key order.  65,536 points of a Gaussian mixture,
// leaves of 16, theta 0.5: 190 launches and 10 host round trips before,
// 16 and one now; traversal 3,546 us with a thread per point in input order and
// the MAC in FP64, 234 us now.  Deeper trees take the level-synchronous
// build and the per-point traversal, which know no depth limit.
//
// The multipole variant (NBodySolverBHMP + QuadTreeMultiPole,
// src/nbodysolvers/cpu/nBodySolverBHMP.h:17-135,
// src/trees/cpu/quadtreemultipole.h:31-289) uses the same tree with FP64
// masses and COMs and a quadrupole sum_c [M_c (dc dc^T) + Q_c]; an accepted
// node contributes the FMM kernels' C1 (monopole + quadrupole).
#include <map>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "kernels.cuh"
#include "state.cuh"

namespace tc {
namespace {

struct Quad {
    double x, y, z, w;  // xx, xy, yx, yy
};

struct BHNodes {
    double2* lo;
    double2* hi;
    uint32_t* start;
    uint32_t* count;
    uint32_t* first_child;  // index of the first child, valid when nchild > 0
    uint32_t* nchild;
    float* mass;
    double2* com;   // full-precision COM (the node's own member)
    float2* comf;   // the COM its parent sees (float)
    double* m64;    // multipole variant: FP64 mass
    Quad* quad;     // multipole variant: quadrupole
};

// QuadTreeMultiPole::createTree's moments for one level (children done)
__global__ void k_bhmp_moments(uint32_t lvl_begin, uint32_t lvl_end, BHNodes t, const double2* __restrict__ pos,
                               const uint32_t* __restrict__ order)
{
    for (uint32_t k = lvl_begin + blockIdx.x * blockDim.x + threadIdx.x; k < lvl_end; k += gridDim.x * blockDim.x) {
        double m = 0.0, cx = 0.0, cy = 0.0;
        Quad q = {0.0, 0.0, 0.0, 0.0};
        if (t.nchild[k] == 0) {
            for (uint32_t i = t.start[k]; i < t.start[k] + t.count[k]; i++) {
                const double2 p = pos[order[i]];
                m += 1.0;
                cx += 1.0 * p.x;
                cy += 1.0 * p.y;
            }
            cx /= m;
            cy /= m;
            for (uint32_t i = t.start[k]; i < t.start[k] + t.count[k]; i++) {
                const double2 p = pos[order[i]];
                const double rx = p.x - cx, ry = p.y - cy;
                q.x += rx * rx;
                q.y += rx * ry;
                q.z += ry * rx;
                q.w += ry * ry;
            }
        } else {
            const uint32_t f = t.first_child[k], e = f + t.nchild[k];
            for (uint32_t c = f; c < e; c++) {
                const double mc = t.m64[c];
                const double2 cc = t.com[c];
                m += mc;
                cx += mc * cc.x;
                cy += mc * cc.y;
            }
            cx /= m;
            cy /= m;
            for (uint32_t c = f; c < e; c++) {
                const double mc = t.m64[c];
                const double2 cc = t.com[c];
                const double rx = cc.x - cx, ry = cc.y - cy;
                const Quad qc = t.quad[c];
                q.x += mc * (rx * rx);
                q.y += mc * (rx * ry);
                q.z += mc * (ry * rx);
                q.w += mc * (ry * ry);
                q.x += qc.x;
                q.y += qc.y;
                q.z += qc.z;
                q.w += qc.w;
            }
        }
        t.m64[k] = m;
        t.com[k] = make_double2(cx, cy);
        t.quad[k] = q;
    }
}

// C1 of a source of mass m and quadrupole Q at offset R (the FMM kernels' far
// field, nBodySolverBHMP.h:111-126)
template <typename real>
__device__ inline void bh_far_c1(real Rx, real Ry, real m, Quad Q, real D1, real D2, real D3, real& ox, real& oy)
{
    const double inv = 1.0 / (double)m;
    const real Txx = (real)(inv * Q.x), Txy = (real)(inv * Q.y), Tyx = (real)(inv * Q.z), Tyy = (real)(inv * Q.w);
    const real S1 = Txx + Tyy;
    const real S2 = (Rx * Rx * Txx) + (Rx * Ry * Txy) + (Ry * Rx * Tyx) + (Ry * Ry * Tyy);
    const real S3x = Rx * Txx + Ry * Txy;
    const real S3y = Rx * Tyx + Ry * Tyy;
    const real base = D1 + real(0.5) * S1 * D2 + real(0.5) * S2 * D3;
    ox = m * (Rx * base + S3x * D2);
    oy = m * (Ry * base + S3y * D2);
}

__global__ void k_bh_root(const double* __restrict__ keys, uint32_t n, BHNodes t)
{
    // keys: order-preserving images of min x, min y, max x, max y
    const unsigned long long* k = reinterpret_cast<const unsigned long long*>(keys);
    const double lx = bbox_unkey(k[0]), ly = bbox_unkey(k[1]);
    const double hx = bbox_unkey(k[2]), hy = bbox_unkey(k[3]);
    const double ax = hx - lx, ay = hy - ly;
    const double ld = (ax < ay) ? ay : ax;  // std::max(a, b)
    t.lo[0] = make_double2(lx, ly);
    t.hi[0] = make_double2(lx + ld + 0.0001, ly + ld + 0.0001);
    t.start[0] = 0;
    t.count[0] = n;
    t.nchild[0] = 0;
    t.first_child[0] = 0;
}

__device__ inline int quadrant(double x, double y, double2 lo, double2 hi)
{
    const double l = (hi.x - lo.x) / 2.0;
    const double mx = lo.x + l, my = lo.y + l;
    if (x >= mx && y >= my) return 0;  // HH
    if (x >= mx && y < my) return 1;   // HL
    if (x < mx && y >= my) return 2;   // LH
    return 3;                          // LL
}

// points of splitting nodes of this level: quadrant indicators
__global__ void k_bh_classify(const double2* __restrict__ pos, const uint32_t* __restrict__ order,
                              const uint32_t* __restrict__ node_of, uint32_t n, uint32_t lvl_begin, uint32_t lvl_end,
                              BHNodes t, int maxc, uint32_t* __restrict__ ind /* 4 x n */, uint8_t* __restrict__ q)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t nd = node_of[i];
        int qq = 4;
        if (nd >= lvl_begin && nd < lvl_end && t.count[nd] > (uint32_t)maxc) {
            const double2 p = pos[order[i]];
            qq = quadrant(p.x, p.y, t.lo[nd], t.hi[nd]);
        }
        q[i] = (uint8_t)qq;
        for (int k = 0; k < 4; k++) ind[(size_t)k * n + i] = (qq == k);
    }
}

// per splitting node of the level: number of non-empty children (for the child scan)
__global__ void k_bh_nchild(uint32_t lvl_begin, uint32_t lvl_end, BHNodes t, int maxc,
                            const uint32_t* __restrict__ pre /* 4 x (n+1) */, uint32_t n, uint32_t* __restrict__ nc)
{
    for (uint32_t k = lvl_begin + blockIdx.x * blockDim.x + threadIdx.x; k < lvl_end; k += gridDim.x * blockDim.x) {
        uint32_t c = 0;
        if (t.count[k] > (uint32_t)maxc) {
            const uint32_t s = t.start[k], e = s + t.count[k];
            for (int qd = 0; qd < 4; qd++) c += (pre[(size_t)qd * (n + 1) + e] - pre[(size_t)qd * (n + 1) + s]) > 0;
        }
        nc[k - lvl_begin] = c;
    }
}

// create the children of the splitting nodes (appended at child_base + offset)
__global__ void k_bh_children(uint32_t lvl_begin, uint32_t lvl_end, BHNodes t, int maxc,
                              const uint32_t* __restrict__ pre, uint32_t n, const uint32_t* __restrict__ coff,
                              uint32_t child_base)
{
    for (uint32_t k = lvl_begin + blockIdx.x * blockDim.x + threadIdx.x; k < lvl_end; k += gridDim.x * blockDim.x) {
        if (t.count[k] <= (uint32_t)maxc) {
            t.nchild[k] = 0;
            continue;
        }
        const uint32_t s = t.start[k], e = s + t.count[k];
        const double2 lo = t.lo[k], hi = t.hi[k];
        const double l = (hi.x - lo.x) / 2.0;
        const double mx = lo.x + l, my = lo.y + l;
        const double2 clo[4] = {make_double2(mx, my), make_double2(mx, lo.y), make_double2(lo.x, my), lo};
        const double2 chi[4] = {hi, make_double2(hi.x, my), make_double2(mx, hi.y), make_double2(mx, my)};
        uint32_t c = child_base + coff[k - lvl_begin];
        t.first_child[k] = c;
        uint32_t nc = 0, off = s;
        for (int qd = 0; qd < 4; qd++) {
            const uint32_t cnt = pre[(size_t)qd * (n + 1) + e] - pre[(size_t)qd * (n + 1) + s];
            if (cnt == 0) continue;
            t.lo[c] = clo[qd];
            t.hi[c] = chi[qd];
            t.start[c] = off;
            t.count[c] = cnt;
            t.nchild[c] = 0;
            t.first_child[c] = 0;
            off += cnt;
            c++;
            nc++;
        }
        t.nchild[k] = nc;
    }
}

// stable partition of each splitting node's occupants by quadrant
__global__ void k_bh_scatter(const uint32_t* __restrict__ order, const uint32_t* __restrict__ node_of,
                             const uint8_t* __restrict__ q, uint32_t n, BHNodes t,
                             const uint32_t* __restrict__ pre, uint32_t* __restrict__ order2,
                             uint32_t* __restrict__ node_of2)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int qq = q[i];
        const uint32_t nd = node_of[i];
        if (qq == 4) {
            order2[i] = order[i];
            node_of2[i] = nd;
            continue;
        }
        const uint32_t s = t.start[nd], e = s + t.count[nd];
        uint32_t dst = s, child = t.first_child[nd];
        for (int k = 0; k < qq; k++) {
            const uint32_t cnt = pre[(size_t)k * (n + 1) + e] - pre[(size_t)k * (n + 1) + s];
            dst += cnt;
            child += cnt > 0;
        }
        dst += pre[(size_t)qq * (n + 1) + i] - pre[(size_t)qq * (n + 1) + s];
        order2[dst] = order[i];
        node_of2[dst] = child;
    }
}

// createTree's mass/COM for the nodes of one level (children already done)
__global__ void k_bh_mass(uint32_t lvl_begin, uint32_t lvl_end, BHNodes t, const double2* __restrict__ pos,
                          const uint32_t* __restrict__ order)
{
    for (uint32_t k = lvl_begin + blockIdx.x * blockDim.x + threadIdx.x; k < lvl_end; k += gridDim.x * blockDim.x) {
        float tm = 0.0f;
        double cx = 0.0, cy = 0.0;
        if (t.nchild[k] == 0) {
            for (uint32_t i = t.start[k]; i < t.start[k] + t.count[k]; i++) {
                tm = (float)((double)tm + 1.0);
                const double2 p = pos[order[i]];
                cx += 1.0 * p.x;
                cy += 1.0 * p.y;
            }
        } else {
            for (uint32_t c = t.first_child[k]; c < t.first_child[k] + t.nchild[k]; c++) {
                const double m = (double)t.mass[c];
                tm = (float)((double)tm + m);
                const float2 cc = t.comf[c];
                cx += m * (double)cc.x;
                cy += m * (double)cc.y;
            }
        }
        cx /= (double)tm;
        cy /= (double)tm;
        t.mass[k] = tm;
        t.com[k] = make_double2(cx, cy);
        t.comf[k] = make_float2((float)cx, (float)cy);
    }
}

constexpr int kBHStack = 128;

// traverseBH (nBodySolverBH.h:56-89) per point, depth first in children order
template <typename real, typename K, bool MP>
__global__ void __launch_bounds__(128) k_bh_traverse(K ker, const double2* __restrict__ pos, uint32_t n, BHNodes t,
                                                     const uint32_t* __restrict__ order, double theta,
                                                     double* __restrict__ grad, double* __restrict__ zrow,
                                                     uint32_t* __restrict__ err)
{
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const double2 x = pos[p];
        real gx = 0, gy = 0, z = 0;
        uint32_t stack[kBHStack];
        int sp = 0;
        stack[sp++] = 0;
        while (sp > 0) {
            const uint32_t nd = stack[--sp];
            const double l = t.hi[nd].x - t.lo[nd].x;
            const double2 c = t.com[nd];
            const double dx = x.x - c.x, dy = x.y - c.y;
            const double len = sqrt(dx * dx + dy * dy);
            if (l / len < theta) {
                if constexpr (MP) {
                    const real tm = (real)t.m64[nd];
                    real D1, D2, D3, tt;
                    ker.far((real)(dx * dx + dy * dy), D1, D2, D3, tt);
                    real cx1, cy1;
                    bh_far_c1<real>((real)dx, (real)dy, tm, t.quad[nd], D1, D2, D3, cx1, cy1);
                    z += tm * tt;
                    gx += cx1;
                    gy += cy1;
                } else {
                    const real tm = (real)t.mass[nd];
                    real D1, tt;
                    ker.near((real)(dx * dx + dy * dy), D1, tt);
                    z += tm * tt;
                    gx += tm * D1 * (real)dx;
                    gy += tm * D1 * (real)dy;
                }
            } else if (t.nchild[nd] <= 1) {
                for (uint32_t i = t.start[nd]; i < t.start[nd] + t.count[nd]; i++) {
                    const uint32_t o = order[i];
                    if (o == p) continue;
                    const double2 q = pos[o];
                    const double ex = x.x - q.x, ey = x.y - q.y;
                    real D1, tt;
                    ker.near((real)(ex * ex + ey * ey), D1, tt);
                    z += tt;
                    gx += D1 * (real)ex;
                    gy += D1 * (real)ey;
                }
            } else {
                const uint32_t f = t.first_child[nd], nc = t.nchild[nd];
                if (sp + (int)nc > kBHStack) {
                    atomicOr(err, 2u);  // stack exhausted: report, stop this point
                    break;
                }
                for (int c = (int)nc - 1; c >= 0; c--) stack[sp++] = f + (uint32_t)c;
            }
        }
        grad[2 * p] = (double)gx;
        grad[2 * p + 1] = (double)gy;
        zrow[p] = (double)z;
    }
}

// ---------------------------------------------------------------- path keys
constexpr int kPathLevels = 16;
// largest maxChildren of the sorted build, whose leaves are ordered by counting (a point against its leaf's others)
constexpr int kPathMaxLeaf = 256;

// sorted-build node records, depth-first order
struct PathNodes {
    uint32_t* start;    // occupants [start, end) in tree order
    uint32_t* end;
    uint32_t* skip;     // the node after the subtree
    uint32_t* parent;
    uint32_t* nchild;
    uint32_t* arrived;  // children done (bottom-up pass)
    double* len;        // box length
    float* mass;        // monopole variant: the reference's float mass and the COM its parent sees
    float2* comf;
    double2* com;
    double* m64;        // multipole variant
    Quad* quad;
    float4* rec;        // [2 i]: COM relative to the root corner, high and low parts (x, y, x, y; path_split);
                        // [2 i + 1]: l / theta, mass, leaf flag, unused
    float4* mom;        // multipole variant, FP32: quadrupole / mass
};

__device__ __forceinline__ void root_box(const double* keys, double2& lo, double& hix)
{
    const unsigned long long* k = reinterpret_cast<const unsigned long long*>(keys);
    const double lx = bbox_unkey(k[0]), ly = bbox_unkey(k[1]);
    const double ax = bbox_unkey(k[2]) - lx, ay = bbox_unkey(k[3]) - ly;
    const double ld = (ax < ay) ? ay : ax;  // std::max(a, b)
    lo = make_double2(lx, ly);
    hix = lx + ld + 0.0001;
}

// the points' extent is at most 2^E
__device__ __forceinline__ int root_exponent(const double* keys)
{
    const unsigned long long* k = reinterpret_cast<const unsigned long long*>(keys);
    return ilogb(fmax(fmax(bbox_unkey(k[2]) - bbox_unkey(k[0]), bbox_unkey(k[3]) - bbox_unkey(k[1])), 1e-300)) + 1;
}

// Coordinates relative to the root corner as FP32 pairs: highs on the grid 2^(E - 24), so that the difference of two is
// exact, and the rest.
struct PathSplit {
    double snap;  // adding and subtracting it rounds to the grid
    __device__ explicit PathSplit(const double* keys) : snap(ldexp(1.5, root_exponent(keys) + 28)) {}
    __device__ __forceinline__ float4 operator()(double x, double y) const
    {
        const double hx = (x + snap) - snap, hy = (y + snap) - snap;
        return make_float4((float)hx, (float)hy, (float)(x - hx), (float)(y - hy));
    }
};

// a - b of two such pairs, rounded once, and the square of its length with the roundings' share (10 of the traversal's
// 234 us)
struct PathDiff {
    float2 d;
    float d2;
    __device__ __forceinline__ PathDiff(float4 a, float4 b)
    {
        const float sx = a.x - b.x, sy = a.y - b.y;  // exact
        const float tx = a.z - b.z, ty = a.w - b.w;  // at most the grid's step, as a non-zero s is at least
        d = make_float2(sx + tx, sy + ty);
        const float rx = tx - (d.x - sx), ry = ty - (d.y - sy);
        const float c = d.x * rx + d.y * ry;
        d2 = d.x * d.x + (d.y * d.y + (c + c));
    }
};

// squared distances below this are taken in FP64: the pairs' own error, 2^(E - 48), could exceed 2^-28 of the distance
__device__ __forceinline__ float path_close2(const double* keys)
{
    return fmaxf((float)ldexp(1.0, 2 * (root_exponent(keys) - 20)), 1e-30f);
}

// one level down: the box of quadrant qd (quadtree.h:104-134; the upper y edge is never read)
__device__ __forceinline__ void child_box(int qd, double2& lo, double& hix)
{
    const double l = (hix - lo.x) / 2.0;
    const double mx = lo.x + l, my = lo.y + l;
    if (qd < 2) lo.x = mx; else hix = mx;
    if ((qd & 1) == 0) lo.y = my;
}

__global__ void k_path_keys(const double2* __restrict__ pos, uint32_t n, const double* __restrict__ bbox,
                            uint32_t* __restrict__ keys)
{
    double2 rlo;
    double rhi;
    root_box(bbox, rlo, rhi);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double2 p = pos[i];
        double2 lo = rlo;
        double hix = rhi;
        uint32_t key = 0;
        for (int l = 0; l < kPathLevels; l++) {
            const int qd = quadrant(p.x, p.y, lo, make_double2(hix, 0.0));
            child_box(qd, lo, hix);
            key = key << 2 | (uint32_t)qd;
        }
        keys[i] = key;
    }
}

// leading quadrants two keys share
__device__ __forceinline__ int common_levels(uint32_t a, uint32_t b)
{
    return a == b ? kPathLevels : __clz((int)(a ^ b)) >> 1;
}

// first index in [a, b) whose key's leading l quadrants are not below those of key (above: beyond those of key)
__device__ __forceinline__ uint32_t path_bound(const uint32_t* __restrict__ keys, uint32_t a, uint32_t b, uint32_t key,
                                               int l, bool above)
{
    const int sh = 2 * (kPathLevels - l);
    const uint64_t v = ((uint64_t)key >> sh) + (above ? 1u : 0u);
    while (a < b) {
        const uint32_t mid = (a + b) >> 1;
        if (((uint64_t)keys[mid] >> sh) < v) a = mid + 1;
        else b = mid;
    }
    return a;
}

// per sorted point: the level of its leaf (the first with at most maxc occupants), the nodes that begin at it, and its
// place in the leaf (the reference keeps a node's occupants in input order).  A leaf of more than maxc points at
// level kPathLevels sets *deep.
__global__ void k_path_leaves(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ perm, uint32_t n,
                              uint32_t maxc, const double2* __restrict__ pos, const double* __restrict__ bbox,
                              uint8_t* __restrict__ depth, uint32_t* __restrict__ nbegin,
                              uint32_t* __restrict__ order, double2* __restrict__ psort, float4* __restrict__ prel,
                              uint32_t* __restrict__ deep)
{
    double2 rlo;
    double rhi;
    root_box(bbox, rlo, rhi);
    const PathSplit split(bbox);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t key = keys[i];
        uint32_t a = 0, b = n;
        int l = 0;
        while (b - a > maxc && l < kPathLevels) {
            l++;
            a = path_bound(keys, a, i, key, l, false);
            b = path_bound(keys, i, b, key, l, true);
        }
        if (b - a > maxc) {
            atomicOr(deep, 1u);
            b = a;  // no place in the leaf is needed: the build is given up
        }
        const int shared = i ? common_levels(keys[i - 1], key) : -1;
        depth[i] = (uint8_t)l;
        nbegin[i] = l > shared ? (uint32_t)(l - shared) : 0u;
        const uint32_t o = perm[i];
        uint32_t r = a;
        for (uint32_t j = a; j < b; j++) r += perm[j] < o;
        if (a == b) r = i;
        const double2 p = pos[o];
        order[r] = o;
        psort[r] = p;
        prel[r] = split(p.x - rlo.x, p.y - rlo.y);
    }
}

// the nodes that begin at each sorted point, numbered from base[i] on by level
__global__ void k_path_nodes(const uint32_t* __restrict__ keys, const uint8_t* __restrict__ depth,
                             const uint32_t* __restrict__ base, uint32_t n, const double* __restrict__ bbox,
                             PathNodes t)
{
    double2 rlo;
    double rhi;
    root_box(bbox, rlo, rhi);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t key = keys[i], b0 = base[i];
        const int nl = (int)(base[i + 1] - b0);
        if (nl == 0) continue;
        const int l1 = depth[i], l0 = l1 - nl + 1;
        // ends from the leaf up: a node's subtree holds its first child's
        uint32_t e = i + 1;
        for (int l = l1; l >= l0; l--) {
            const uint32_t nd = b0 + (uint32_t)(l - l0);
            e = path_bound(keys, e, n, key, l, true);
            t.start[nd] = i;
            t.end[nd] = e;
            t.skip[nd] = base[e];
            uint32_t par = nd - 1;
            if (l == l0 && l > 0) {
                // the level l - 1 node that holds i begins earlier
                const uint32_t p0 = path_bound(keys, 0, i, key, l - 1, false);
                par = base[p0] + (base[p0 + 1] - base[p0]) - 1u - (uint32_t)(depth[p0] - (l - 1));
            }
            t.parent[nd] = par;
            if (l > 0) atomicAdd(&t.nchild[par], 1u);
        }
        double2 lo = rlo;
        double hix = rhi;
        for (int l = 0;; l++) {
            if (l >= l0) t.len[b0 + (uint32_t)(l - l0)] = hix - lo.x;
            if (l == l1) break;
            child_box((int)(key >> (2 * (kPathLevels - 1 - l)) & 3u), lo, hix);
        }
    }
}

// masses, COMs and quadrupoles bottom up with the reference's types and orders (k_bh_mass, k_bhmp_moments): a thread
// per leaf, and the last child to arrive goes on with the parent
template <bool MP>
__global__ void k_path_moments(uint32_t total, PathNodes t, const double2* __restrict__ psort,
                               const double* __restrict__ bbox, double theta)
{
    double2 rlo;
    double rhi;
    root_box(bbox, rlo, rhi);
    const PathSplit split(bbox);
    for (uint32_t leaf = blockIdx.x * blockDim.x + threadIdx.x; leaf < total; leaf += gridDim.x * blockDim.x) {
        if (t.nchild[leaf] != 0) continue;
        uint32_t nd = leaf;
        while (true) {
            double cx = 0.0, cy = 0.0, m = 0.0;
            const uint32_t nch = t.nchild[nd], e = t.skip[nd];
            if constexpr (MP) {
                Quad q = {0.0, 0.0, 0.0, 0.0};
                if (nch == 0) {
                    for (uint32_t i = t.start[nd]; i < t.end[nd]; i++) {
                        const double2 p = psort[i];
                        m += 1.0;
                        cx += 1.0 * p.x;
                        cy += 1.0 * p.y;
                    }
                    cx /= m;
                    cy /= m;
                    for (uint32_t i = t.start[nd]; i < t.end[nd]; i++) {
                        const double2 p = psort[i];
                        const double rx = p.x - cx, ry = p.y - cy;
                        q.x += rx * rx;
                        q.y += rx * ry;
                        q.z += ry * rx;
                        q.w += ry * ry;
                    }
                } else {
                    for (uint32_t c = nd + 1; c != e; c = t.skip[c]) {
                        const double mc = __ldcg(t.m64 + c);
                        const double2 cc = __ldcg(t.com + c);
                        m += mc;
                        cx += mc * cc.x;
                        cy += mc * cc.y;
                    }
                    cx /= m;
                    cy /= m;
                    for (uint32_t c = nd + 1; c != e; c = t.skip[c]) {
                        const double mc = __ldcg(t.m64 + c);
                        const double2 cc = __ldcg(t.com + c);
                        const double rx = cc.x - cx, ry = cc.y - cy;
                        const double* qc = reinterpret_cast<const double*>(t.quad + c);
                        q.x += mc * (rx * rx);
                        q.y += mc * (rx * ry);
                        q.z += mc * (ry * rx);
                        q.w += mc * (ry * ry);
                        q.x += __ldcg(qc);
                        q.y += __ldcg(qc + 1);
                        q.z += __ldcg(qc + 2);
                        q.w += __ldcg(qc + 3);
                    }
                }
                t.m64[nd] = m;
                t.com[nd] = make_double2(cx, cy);
                t.quad[nd] = q;
                const double inv = 1.0 / (double)(float)m;
                t.mom[nd] = make_float4((float)(inv * q.x), (float)(inv * q.y), (float)(inv * q.z), (float)(inv * q.w));
            } else {
                float tm = 0.0f;
                if (nch == 0) {
                    for (uint32_t i = t.start[nd]; i < t.end[nd]; i++) {
                        tm = (float)((double)tm + 1.0);
                        const double2 p = psort[i];
                        cx += 1.0 * p.x;
                        cy += 1.0 * p.y;
                    }
                } else {
                    for (uint32_t c = nd + 1; c != e; c = t.skip[c]) {
                        const double mc = (double)__ldcg(t.mass + c);
                        tm = (float)((double)tm + mc);
                        const float2 cc = __ldcg(t.comf + c);
                        cx += mc * (double)cc.x;
                        cy += mc * (double)cc.y;
                    }
                }
                cx /= (double)tm;
                cy /= (double)tm;
                t.mass[nd] = tm;
                t.com[nd] = make_double2(cx, cy);
                t.comf[nd] = make_float2((float)cx, (float)cy);
                m = (double)tm;
            }
            t.rec[2 * (size_t)nd] = split(cx - rlo.x, cy - rlo.y);
            t.rec[2 * (size_t)nd + 1] = make_float4((float)(t.len[nd] / theta), (float)m, nch <= 1 ? 1.0f : 0.0f, 0.0f);
            if (nd == 0) break;
            const uint32_t par = t.parent[nd];
            __threadfence();
            if (atomicAdd(&t.arrived[par], 1u) + 1u < t.nchild[par]) break;
            __threadfence();
            nd = par;
        }
    }
}

constexpr int kPathThreads = 64;  // few points leave few warps: small blocks spread them evenly

// traverseBH, a warp per 32 points neighbouring in tree order: the warp walks the nodes depth first, going into a
// node while any of its points opens it; a point that has accepted a node sits out the subtree.  Each point meets
// its nodes in the order it would alone.  The MAC is decided in FP32 and, within 1e-5 of its threshold (the FP32
// square is good to 2e-7), as the reference decides it.  FP32 forces take offset and square as good as the FP64 ones
// rounded (path_close2: the FP64 ones where the pairs are too few bits).
template <typename real, typename K, bool MP>
__global__ void __launch_bounds__(kPathThreads) k_path_traverse(K ker, uint32_t n, uint32_t total, PathNodes t,
                                                       const double2* __restrict__ psort,
                                                       const float4* __restrict__ prel,
                                                       const uint32_t* __restrict__ order,
                                                       const double* __restrict__ bbox, double theta,
                                                       double* __restrict__ grad, double* __restrict__ zrow)
{
    constexpr bool kF32 = sizeof(real) == 4;
    const float close2 = path_close2(bbox);
    for (uint32_t p0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; p0 < n; p0 += gridDim.x * blockDim.x) {
        const uint32_t i = p0 + (threadIdx.x & 31);
        const bool valid = i < n;
        const float4 xs = valid ? prel[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const double2 x = valid ? psort[i] : make_double2(0.0, 0.0);
        real gx = 0, gy = 0, z = 0;
        uint32_t resume = valid ? 0u : total;  // nodes before this one are not this point's
        for (uint32_t nd = 0; nd < total;) {
            const float4 c = t.rec[2 * (size_t)nd], r = t.rec[2 * (size_t)nd + 1];
            const uint32_t skip = t.skip[nd];
            const bool on = nd >= resume;
            const PathDiff diff(xs, c);
            const float2 d = diff.d;
            const float d2 = diff.d2, thr2 = r.x * r.x;
            const bool apart = d2 >= close2;  // false for NaN (highs that overflow)
            bool pass = d2 > thr2;
            if (on && !(fabsf(d2 - thr2) > 1e-5f * thr2 && thr2 > 1e-30f && apart)) {
                const double2 com = t.com[nd];
                const double ex = x.x - com.x, ey = x.y - com.y;
                pass = t.len[nd] / sqrt(ex * ex + ey * ey) < theta;
            }
            if (on && pass) {
                resume = skip;
                if (kF32 && apart) {
                    if constexpr (MP) {
                        const float4 q = t.mom[nd];
                        real D1, D2, D3, tt;
                        ker.far(d2, D1, D2, D3, tt);
                        const real S2 = (d.x * d.x * q.x) + (d.x * d.y * q.y) + (d.y * d.x * q.z) + (d.y * d.y * q.w);
                        const real base = D1 + real(0.5) * (q.x + q.w) * D2 + real(0.5) * S2 * D3;
                        z += r.y * tt;
                        gx += r.y * (d.x * base + (d.x * q.x + d.y * q.y) * D2);
                        gy += r.y * (d.y * base + (d.x * q.z + d.y * q.w) * D2);
                    } else {
                        real D1, tt;
                        ker.near(d2, D1, tt);
                        z += r.y * tt;
                        gx += r.y * D1 * d.x;
                        gy += r.y * D1 * d.y;
                    }
                } else {
                    const double2 com = t.com[nd];
                    const double dx = x.x - com.x, dy = x.y - com.y;
                    if constexpr (MP) {
                        const real tm = (real)t.m64[nd];
                        real D1, D2, D3, tt;
                        ker.far((real)(dx * dx + dy * dy), D1, D2, D3, tt);
                        real cx1, cy1;
                        bh_far_c1<real>((real)dx, (real)dy, tm, t.quad[nd], D1, D2, D3, cx1, cy1);
                        z += tm * tt;
                        gx += cx1;
                        gy += cy1;
                    } else {
                        const real tm = (real)t.mass[nd];
                        real D1, tt;
                        ker.near((real)(dx * dx + dy * dy), D1, tt);
                        z += tm * tt;
                        gx += tm * D1 * (real)dx;
                        gy += tm * D1 * (real)dy;
                    }
                }
            }
            const bool open = on && !pass;
            const bool any = __any_sync(0xffffffffu, open);
            if (any && r.z == 0.0f) {
                nd++;
                continue;
            }
            if (any) {
                const uint32_t e = t.end[nd];
                if constexpr (kF32) {
                    // summed by themselves first: fewer roundings against the running sums
                    real lx = 0, ly = 0, lz = 0;
                    bool near = false;
#pragma unroll 4
                    for (uint32_t j = t.start[nd]; j < e; j++) {
                        const PathDiff f(xs, prel[j]);
                        real D1, tt;
                        ker.near(f.d2, D1, tt);
                        const bool ok = f.d2 >= close2, use = open && ok;
                        near |= open && !ok && j != i;
                        lz += use ? tt : real(0);
                        lx += use ? D1 * f.d.x : real(0);
                        ly += use ? D1 * f.d.y : real(0);
                    }
                    if (near) {
                        for (uint32_t j = t.start[nd]; j < e; j++) {
                            if (PathDiff(xs, prel[j]).d2 >= close2 || j == i) continue;
                            const double2 q = psort[j];
                            const double ex = x.x - q.x, ey = x.y - q.y;
                            real D1, tt;
                            ker.near((real)(ex * ex + ey * ey), D1, tt);
                            lz += tt;
                            lx += D1 * (real)ex;
                            ly += D1 * (real)ey;
                        }
                    }
                    gx += lx;
                    gy += ly;
                    z += lz;
                } else if (open) {
                    for (uint32_t j = t.start[nd]; j < e; j++) {
                        if (j == i) continue;
                        const double2 q = psort[j];
                        const double ex = x.x - q.x, ey = x.y - q.y;
                        real D1, tt;
                        ker.near((real)(ex * ex + ey * ey), D1, tt);
                        z += tt;
                        gx += D1 * (real)ex;
                        gy += D1 * (real)ey;
                    }
                }
            }
            nd = skip;
        }
        if (valid) {
            const uint32_t o = order[i];
            grad[2 * (size_t)o] = (double)gx;
            grad[2 * (size_t)o + 1] = (double)gy;
            zrow[o] = (double)z;
        }
    }
}

// Scratch of one call, carved from a per-device workspace that persists
// between calls and only grows (calls on one device are serialised by its
// mutex), so that repeated solves allocate nothing after the first.
struct BHWork {
    std::mutex mu;
    Buf slot[64];
    cudaEvent_t done = nullptr;  // recorded after each call's last use of the workspace
    bool recorded = false;
};

// records the workspace's completion event on every exit of a call
struct WorkRelease {
    BHWork& w;
    cudaStream_t s;
    ~WorkRelease()
    {
        if (w.done && cudaEventRecord(w.done, s) == cudaSuccess) w.recorded = true;
    }
};

__global__ void k_bh_iota(uint32_t* __restrict__ order, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) order[i] = i;
}

BHWork& bh_work(int dev)
{
    static std::mutex m;
    static std::map<int, std::unique_ptr<BHWork>> w;
    std::lock_guard<std::mutex> g(m);
    auto& p = w[dev];
    if (!p) p.reset(new BHWork());
    return *p;
}

struct DevBuf {
    void* p = nullptr;
};

thread_local BHWork* g_work = nullptr;
thread_local int g_slot = 0;

template <typename T>
int dalloc(DevBuf& b, size_t count)
{
    if (!g_work || g_slot >= 64) {
        tc_set_error("bh: workspace slots exhausted");
        return TC_ERR_STATE;
    }
    Buf& w = g_work->slot[g_slot++];
    int rc = ensure(w, count * sizeof(T) + 16);
    if (rc) return rc;
    b.p = w.p;
    return TC_OK;
}

}  // namespace



}  // namespace tc

using namespace tc;

namespace tc {
namespace {

// launches the traversal of either tree; F(ker, real(), mp) does the launch
template <typename F>
void bh_dispatch(int kernel, double softening, int precision, bool mp, F&& f)
{
    const double e2 = softening * softening;
    auto with_mp = [&](auto ker, auto zero) {
        if (mp) f(ker, zero, std::true_type());
        else f(ker, zero, std::false_type());
    };
    if (precision == TC_PREC_FP64) {
        if (kernel == TC_KERNEL_GRAVITY) with_mp(KGrav<double>{e2}, 0.0);
        else with_mp(KTsne<double>{}, 0.0);
    } else {
        if (kernel == TC_KERNEL_GRAVITY) with_mp(KGrav<float>{(float)e2}, 0.0f);
        else with_mp(KTsne<float>{}, 0.0f);
    }
}

// Builds the tree by sorting path keys and walks it.  1: the tree is not one for it (deeper than kPathLevels, or more
// nodes than the level-synchronous build would accept, which then refuses it); nothing has been written that the
// caller sees.
int bh_path_solve(int kernel, double softening, int max_children, double theta, int precision, const double2* pos,
                  uint32_t n, double* d_grad_xy, double* zrow, cudaStream_t s, bool mp, const double* bbox,
                  uint32_t* err, size_t cap)
{
    int rc;
    DevBuf b_keys, b_perm, b_akeys, b_avals, b_tmp, b_depth, b_nbegin, b_base, b_order, b_psort, b_prel;
    const int64_t tw = radix_tmp_words(n) > scan_tmp_words(n) ? radix_tmp_words(n) : scan_tmp_words(n);
    if ((rc = dalloc<uint32_t>(b_keys, n)) || (rc = dalloc<uint32_t>(b_perm, n)) ||
        (rc = dalloc<uint32_t>(b_akeys, n)) || (rc = dalloc<uint32_t>(b_avals, n)) ||
        (rc = dalloc<uint32_t>(b_tmp, (size_t)tw)) || (rc = dalloc<uint8_t>(b_depth, n)) ||
        (rc = dalloc<uint32_t>(b_nbegin, n)) || (rc = dalloc<uint32_t>(b_base, (size_t)n + 1)) ||
        (rc = dalloc<uint32_t>(b_order, n)) || (rc = dalloc<double2>(b_psort, n)) || (rc = dalloc<float4>(b_prel, n)))
        return rc;
    uint32_t *keys = (uint32_t*)b_keys.p, *perm = (uint32_t*)b_perm.p, *base = (uint32_t*)b_base.p;
    uint32_t* order = (uint32_t*)b_order.p;
    double2* psort = (double2*)b_psort.p;
    float4* prel = (float4*)b_prel.p;
    k_path_keys<<<grid_for(n, 128), 128, 0, s>>>(pos, n, bbox, keys);
    if ((rc = radix_sort_u32(keys, perm, (uint32_t*)b_akeys.p, (uint32_t*)b_avals.p, n, (uint32_t*)b_tmp.p, s, nullptr)))
        return rc;
    k_path_leaves<<<grid_for(n, 128), 128, 0, s>>>(keys, perm, n, (uint32_t)max_children, pos, bbox,
                                                   (uint8_t*)b_depth.p, (uint32_t*)b_nbegin.p, order, psort, prel,
                                                   err + 1);
    if ((rc = exclusive_scan_u32((uint32_t*)b_nbegin.p, base, n, (uint32_t*)b_tmp.p, s))) return rc;
    uint32_t total = 0, flags[2] = {0, 0};
    TC_CUDA_TRY(cudaMemcpyAsync(&total, base + n, 4, cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaMemcpyAsync(flags, err, 8, cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaStreamSynchronize(s));
    if (flags[0]) {
        tc_set_error("tc_bh_solve_device: positions contain NaN or infinity");
        return TC_ERR_INVALID;
    }
    if (flags[1] || total > cap) return 1;
    // sized by the points, so that the workspace does not grow with every tree
    const size_t nn = total > n ? total : n;
    DevBuf b_start, b_end, b_skip, b_parent, b_cnt, b_len, b_mass, b_comf, b_com, b_m64, b_quad, b_rec, b_mom;
    if ((rc = dalloc<uint32_t>(b_start, nn)) || (rc = dalloc<uint32_t>(b_end, nn)) ||
        (rc = dalloc<uint32_t>(b_skip, nn)) || (rc = dalloc<uint32_t>(b_parent, nn)) ||
        (rc = dalloc<uint32_t>(b_cnt, 2 * nn)) || (rc = dalloc<double>(b_len, nn)) ||
        (rc = dalloc<double2>(b_com, nn)) || (rc = dalloc<float4>(b_rec, 2 * nn)))
        return rc;
    if (mp && ((rc = dalloc<double>(b_m64, nn)) || (rc = dalloc<Quad>(b_quad, nn)) ||
               (rc = dalloc<float4>(b_mom, nn))))
        return rc;
    if (!mp && ((rc = dalloc<float>(b_mass, nn)) || (rc = dalloc<float2>(b_comf, nn)))) return rc;
    uint32_t* cnt = (uint32_t*)b_cnt.p;
    PathNodes t{(uint32_t*)b_start.p, (uint32_t*)b_end.p, (uint32_t*)b_skip.p, (uint32_t*)b_parent.p, cnt, cnt + total,
                (double*)b_len.p, (float*)b_mass.p, (float2*)b_comf.p, (double2*)b_com.p, (double*)b_m64.p,
                (Quad*)b_quad.p, (float4*)b_rec.p, (float4*)b_mom.p};
    TC_CUDA_TRY(cudaMemsetAsync(cnt, 0, (size_t)2 * total * 4, s));
    k_path_nodes<<<grid_for(n, 128), 128, 0, s>>>(keys, (const uint8_t*)b_depth.p, base, n, bbox, t);
    if (mp)
        k_path_moments<true><<<grid_for(total, 128), 128, 0, s>>>(total, t, psort, bbox, theta);
    else
        k_path_moments<false><<<grid_for(total, 128), 128, 0, s>>>(total, t, psort, bbox, theta);
    bh_dispatch(kernel, softening, precision, mp, [&](auto ker, auto zero, auto m) {
        k_path_traverse<decltype(zero), decltype(ker), decltype(m)::value>
            <<<grid_for(n, kPathThreads, 1 << 20), kPathThreads, 0, s>>>(ker, n, total, t, psort, prel, order, bbox,
                                                                        theta, d_grad_xy, zrow);
    });
    TC_CUDA_TRY(cudaGetLastError());
    return TC_OK;
}

// The tree of any depth, level by level, and the per-point traversal
int bh_level_solve(int kernel, double softening, int max_children, double theta, int precision, const double* d_pos_xy,
                   uint32_t n, double* d_grad_xy, double* zrow, cudaStream_t s, bool mp, const double* bbox,
                   uint32_t* err, size_t cap)
{
    int rc;
    DevBuf b_lo, b_hi, b_start, b_count, b_fc, b_nc, b_mass, b_com, b_comf, b_order, b_order2, b_nodeof, b_nodeof2,
        b_q, b_ind, b_pre, b_nck, b_coff, b_tmp;
    if ((rc = dalloc<double2>(b_lo, cap)) || (rc = dalloc<double2>(b_hi, cap)) || (rc = dalloc<uint32_t>(b_start, cap)) ||
        (rc = dalloc<uint32_t>(b_count, cap)) || (rc = dalloc<uint32_t>(b_fc, cap)) ||
        (rc = dalloc<uint32_t>(b_nc, cap)) || (rc = dalloc<float>(b_mass, cap)) || (rc = dalloc<double2>(b_com, cap)) ||
        (rc = dalloc<float2>(b_comf, cap)) || (rc = dalloc<uint32_t>(b_order, n)) ||
        (rc = dalloc<uint32_t>(b_order2, n)) || (rc = dalloc<uint32_t>(b_nodeof, n)) ||
        (rc = dalloc<uint32_t>(b_nodeof2, n)) || (rc = dalloc<uint8_t>(b_q, n)) ||
        (rc = dalloc<uint32_t>(b_ind, (size_t)4 * n)) || (rc = dalloc<uint32_t>(b_pre, (size_t)4 * (n + 1))) ||
        (rc = dalloc<uint32_t>(b_nck, cap)) || (rc = dalloc<uint32_t>(b_coff, cap + 1)) ||
        (rc = dalloc<uint32_t>(b_tmp, (size_t)(scan_tmp_words((int64_t)cap + n) + 2 * scan_tmp_words(n)))))
        return rc;
    DevBuf b_m64, b_quad;
    if (mp && ((rc = dalloc<double>(b_m64, cap)) || (rc = dalloc<Quad>(b_quad, cap)))) return rc;
    BHNodes t{(double2*)b_lo.p, (double2*)b_hi.p, (uint32_t*)b_start.p, (uint32_t*)b_count.p, (uint32_t*)b_fc.p,
              (uint32_t*)b_nc.p, (float*)b_mass.p, (double2*)b_com.p, (float2*)b_comf.p, (double*)b_m64.p,
              (Quad*)b_quad.p};
    uint32_t* order = (uint32_t*)b_order.p;
    uint32_t* order2 = (uint32_t*)b_order2.p;
    uint32_t* node_of = (uint32_t*)b_nodeof.p;
    uint32_t* node_of2 = (uint32_t*)b_nodeof2.p;
    uint32_t* ind = (uint32_t*)b_ind.p;
    uint32_t* pre = (uint32_t*)b_pre.p;
    TC_CUDA_TRY(cudaMemsetAsync(node_of, 0, (size_t)n * 4, s));
    k_bh_iota<<<grid_for(n, 256), 256, 0, s>>>(order, n);
    k_bh_root<<<1, 1, 0, s>>>(bbox, n, t);
    std::vector<uint32_t> level_begin = {0}, level_end = {1};
    uint32_t total_nodes = 1;
    const int grid = grid_for(n, 256);
    for (int lvl = 0; lvl < 64; lvl++) {
        const uint32_t lb = level_begin.back(), le = level_end.back();
        k_bh_classify<<<grid, 256, 0, s>>>((const double2*)d_pos_xy, order, node_of, n, lb, le, t, max_children, ind,
                                           (uint8_t*)b_q.p);
        for (int k = 0; k < 4; k += 2)
            if ((rc = exclusive_scan2_u32(ind + (size_t)k * n, pre + (size_t)k * (n + 1), ind + (size_t)(k + 1) * n,
                                          pre + (size_t)(k + 1) * (n + 1), n, (uint32_t*)b_tmp.p, s)))
                return rc;
        k_bh_nchild<<<grid_for(le - lb, 256), 256, 0, s>>>(lb, le, t, max_children, pre, n, (uint32_t*)b_nck.p);
        if ((rc = exclusive_scan_u32((uint32_t*)b_nck.p, (uint32_t*)b_coff.p, le - lb, (uint32_t*)b_tmp.p, s))) return rc;
        uint32_t nnew = 0;
        TC_CUDA_TRY(cudaMemcpyAsync(&nnew, (uint32_t*)b_coff.p + (le - lb), 4, cudaMemcpyDeviceToHost, s));
        TC_CUDA_TRY(cudaStreamSynchronize(s));
        if (total_nodes + nnew > cap) {
            tc_set_error("tc_bh_solve_device: node capacity exceeded (coincident points?)");
            return TC_ERR_INVALID;
        }
        k_bh_children<<<grid_for(le - lb, 256), 256, 0, s>>>(lb, le, t, max_children, pre, n, (uint32_t*)b_coff.p,
                                                            total_nodes);
        if (nnew == 0) break;
        k_bh_scatter<<<grid, 256, 0, s>>>(order, node_of, (const uint8_t*)b_q.p, n, t, pre, order2, node_of2);
        std::swap(order, order2);
        std::swap(node_of, node_of2);
        level_begin.push_back(total_nodes);
        total_nodes += nnew;
        level_end.push_back(total_nodes);
        if (lvl == 63) {
            tc_set_error("tc_bh_solve_device: tree deeper than 64 levels (coincident points?)");
            return TC_ERR_INVALID;
        }
    }
    for (int l = (int)level_begin.size() - 1; l >= 0; l--) {
        if (mp)
            k_bhmp_moments<<<grid_for(level_end[l] - level_begin[l], 128), 128, 0, s>>>(
                level_begin[l], level_end[l], t, (const double2*)d_pos_xy, order);
        else
            k_bh_mass<<<grid_for(level_end[l] - level_begin[l], 128), 128, 0, s>>>(level_begin[l], level_end[l], t,
                                                                                   (const double2*)d_pos_xy, order);
    }
    const double2* pos = (const double2*)d_pos_xy;
    bh_dispatch(kernel, softening, precision, mp, [&](auto ker, auto zero, auto m) {
        k_bh_traverse<decltype(zero), decltype(ker), decltype(m)::value>
            <<<grid_for(n, 128), 128, 0, s>>>(ker, pos, n, t, order, theta, d_grad_xy, zrow, err);
    });
    TC_CUDA_TRY(cudaGetLastError());
    return TC_OK;
}

int bh_check(int kernel, int max_children, double theta, const double* pos_xy, int64_t n, const double* grad_xy)
{
    if (!pos_xy || !grad_xy || n <= 0 || n > (1 << 30) || max_children <= 0 || !(theta > 0.0) ||
        (kernel != TC_KERNEL_TSNE && kernel != TC_KERNEL_GRAVITY)) {
        tc_set_error("tc_bh_solve_device: invalid arguments");
        return TC_ERR_INVALID;
    }
    return TC_OK;
}

int bh_solve_impl(int kernel, double softening, int max_children, double theta, int precision,
                  const double* d_pos_xy, int64_t n64, double* d_grad_xy, double* d_total, void* stream, bool mp)
{
    if (const int bad = bh_check(kernel, max_children, theta, d_pos_xy, n64, d_grad_xy)) return bad;
    const uint32_t n = (uint32_t)n64;
    cudaStream_t s = (cudaStream_t)stream;
    int rc = TC_OK;
    int dev = 0;
    TC_CUDA_TRY(cudaGetDevice(&dev));
    BHWork& work = bh_work(dev);
    std::lock_guard<std::mutex> work_lock(work.mu);
    if (!work.done) TC_CUDA_TRY(cudaEventCreateWithFlags(&work.done, cudaEventDisableTiming));
    // the previous call's kernels (possibly on another stream) finish first
    if (work.recorded) TC_CUDA_TRY(cudaStreamWaitEvent(s, work.done, 0));
    WorkRelease release_on_exit{work, s};
    g_work = &work;
    g_slot = 0;
    // node capacity (splits past it are refused, not written)
    const size_t cap = (size_t)4 * n + 64;
    DevBuf b_bbox, b_zrow, b_err, b_sum;
    if ((rc = dalloc<double>(b_bbox, 4)) || (rc = dalloc<double>(b_zrow, n)) || (rc = dalloc<uint32_t>(b_err, 4)) ||
        (rc = dalloc<double>(b_sum, sum_tmp_doubles())))
        return rc;
    const double* bbox = (const double*)b_bbox.p;
    double* zrow = (double*)b_zrow.p;
    uint32_t* err = (uint32_t*)b_err.p;
    TC_CUDA_TRY(cudaMemsetAsync(b_err.p, 0, 16, s));
    if ((rc = bbox_keys(d_pos_xy, n64, (double*)b_bbox.p, (uint32_t*)b_err.p, s))) return rc;
    const int first_slot = g_slot;
    rc = max_children <= kPathMaxLeaf ? bh_path_solve(kernel, softening, max_children, theta, precision,
                                                      (const double2*)d_pos_xy, n, d_grad_xy, zrow, s, mp, bbox, err, cap)
                                      : 1;
    if (rc == 1) {
        g_slot = first_slot;  // the same scratch, laid out anew (its kernels are done)
        rc = bh_level_solve(kernel, softening, max_children, theta, precision, d_pos_xy, n, d_grad_xy, zrow, s, mp, bbox,
                            err, cap);
    }
    if (rc) return rc;
    if (d_total && (rc = sum_f64(zrow, n, nullptr, nullptr, d_total, 0, (double*)b_sum.p, s)))
        return rc;
    uint32_t herr = 0;
    TC_CUDA_TRY(cudaMemcpyAsync(&herr, b_err.p, 4, cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr) {
        tc_set_error("tc_bh_solve_device: traversal stack exhausted");
        return TC_ERR_INVALID;
    }
    return TC_OK;
}

}  // namespace
}  // namespace tc

extern "C" int tc_bh_solve_device(int kernel, double softening, int max_children, double theta, int precision,
                                  const double* d_pos_xy, int64_t n64, double* d_grad_xy, double* d_total,
                                  void* stream)
{
    return bh_solve_impl(kernel, softening, max_children, theta, precision, d_pos_xy, n64, d_grad_xy, d_total, stream,
                         false);
}

extern "C" int tc_bhmp_solve_device(int kernel, double softening, int max_children, double theta, int precision,
                                    const double* d_pos_xy, int64_t n64, double* d_grad_xy, double* d_total,
                                    void* stream)
{
    return bh_solve_impl(kernel, softening, max_children, theta, precision, d_pos_xy, n64, d_grad_xy, d_total, stream,
                         true);
}

static int bh_solve_host(int kernel, double softening, int max_children, double theta, int precision,
                         const double* pos_xy, int64_t n, double* grad_xy, double* total, bool mp)
{
    if (!pos_xy || !grad_xy || n <= 0) {
        tc_set_error("tc_bh_solve: invalid arguments");
        return TC_ERR_INVALID;
    }
    int rc = tc::bh_check(kernel, max_children, theta, pos_xy, n, grad_xy);
    if (rc) return rc;
    tc::HostStage st;
    if ((rc = st.open((size_t)n * 16, (size_t)n * 16 + 64))) return rc;
    double *d_total = static_cast<double*>(st.out()), *d_grad = d_total + 8;
    TC_CUDA_TRY(cudaMemcpyAsync(st.in(), pos_xy, (size_t)n * 16, cudaMemcpyHostToDevice, st.stream()));
    rc = tc::bh_solve_impl(kernel, softening, max_children, theta, precision, static_cast<const double*>(st.in()), n,
                           d_grad, d_total, st.stream(), mp);
    if (rc) return rc;
    TC_CUDA_TRY(cudaMemcpyAsync(grad_xy, d_grad, (size_t)n * 16, cudaMemcpyDeviceToHost, st.stream()));
    if (total) TC_CUDA_TRY(cudaMemcpyAsync(total, d_total, 8, cudaMemcpyDeviceToHost, st.stream()));
    TC_CUDA_TRY(cudaStreamSynchronize(st.stream()));
    return TC_OK;
}

extern "C" int tc_bh_solve(int kernel, double softening, int max_children, double theta, int precision,
                           const double* pos_xy, int64_t n, double* grad_xy, double* total)
{
    return bh_solve_host(kernel, softening, max_children, theta, precision, pos_xy, n, grad_xy, total, false);
}

extern "C" int tc_bhmp_solve(int kernel, double softening, int max_children, double theta, int precision,
                             const double* pos_xy, int64_t n, double* grad_xy, double* total)
{
    return bh_solve_host(kernel, softening, max_children, theta, precision, pos_xy, n, grad_xy, total, true);
}
