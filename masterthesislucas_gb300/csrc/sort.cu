// Stable LSD radix sort of (u32 key, u32 value): passes of 8 bits.  Up to
// kLookBack keys one kernel counts the digits of all passes, and a pass is then
// one kernel, in which every tile ranks its keys, stages itself digit-sorted in
// shared memory, finds its digits' offsets by looking back over the tiles
// before it (their digit counts, or running sums once they have them) and
// writes each digit run contiguously; with more keys a pass counts and scans
// its tiles' digits first.  Keys are ranked in their input order with warp
// match-any groups against warp-private digit counters.  Up to kSmallSort keys
// one block sorts in shared memory.  Stability makes ties between equal Morton
// codes keep input order, which defines the permutation where the reference's
// unstable integer_sort (nBodySolverFMM_SYM_MORTON.h:89) does not.
//
// What bounds it: launches for few keys (a histogram, one to three scan
// kernels and a scatter per pass were 12 to 20 launches; 2,000 keys: 39 us then,
// 15 in one block), memory and the ranking for many.
#include "common.cuh"

namespace tc {
namespace {

constexpr int RT = 256;           // threads per tile
#ifndef TC_SORT_RI
#define TC_SORT_RI 8
#endif
constexpr int RI = TC_SORT_RI;    // keys per thread
constexpr int RTILE = RT * RI;    // keys per tile
constexpr int RADIX = 256;
constexpr int NW = RT / 32;
constexpr int kMaxPass = 4;
// the most keys whose tiles look back; above, a pass counts its tiles' digits and scans the counts first.  A block
// that looks back holds its SM while the sums pass through the tiles in flight, a window per round trip to L2: 65,536
// keys: 8.5 us a pass against 14 with a histogram and a scan; 1M: 23 and 25; 3.6M: 48 and 39; 4M: 58 and 55
constexpr int64_t kLookBack = (int64_t)1 << 20;
// a tile's word for a digit: 0 not there yet, the tile's own count, or the count of all tiles up to it (top two bits)
enum : uint32_t { kOwn = 1u << 30, kUpTo = 2u << 30, kValue = (1u << 30) - 1u };
// looks at words that are not there yet, before a block counts for itself (about a second or two)
#ifndef TC_SORT_POLLS
#define TC_SORT_POLLS (1u << 22)
#endif
constexpr uint32_t kMaxPolls = TC_SORT_POLLS;

// scratch: [0, 4) tile tickets of the passes, [8, 8 + 4 * 256) digit counts of the passes, then per pass nb * 256
// words of the tiles
constexpr int kHistAt = 8, kTilesAt = kHistAt + kMaxPass * RADIX;

__global__ void __launch_bounds__(RT) k_radix_hist(const uint32_t* __restrict__ keys, int64_t n, int lo_bit, int npass,
                                                   uint32_t* __restrict__ scratch)
{
    // two copies (even and odd warps) halve the collisions of clustered keys' top digits
    __shared__ uint32_t h[2][kMaxPass][RADIX];
    for (int i = threadIdx.x; i < 2 * kMaxPass * RADIX; i += RT) (&h[0][0][0])[i] = 0;
    __syncthreads();
    uint32_t(*own)[RADIX] = h[(threadIdx.x >> 5) & 1];
    for (int64_t base = blockIdx.x * (int64_t)RTILE; base < n; base += (int64_t)gridDim.x * RTILE) {
        uint32_t k[RI];
#pragma unroll
        for (int r = 0; r < RI; r++) {
            const int64_t p = base + (int64_t)r * RT + threadIdx.x;
            k[r] = p < n ? keys[p] : 0u;
        }
#pragma unroll
        for (int r = 0; r < RI; r++) {
            if (base + (int64_t)r * RT + threadIdx.x >= n) continue;
            for (int p = 0; p < npass; p++) atomicAdd(&own[p][(k[r] >> (lo_bit + 8 * p)) & 255u], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npass * RADIX; i += RT) {
        const uint32_t c = (&h[0][0][0])[i] + (&h[1][0][0])[i];
        if (c) atomicAdd(scratch + kHistAt + i, c);
    }
}

// digit counts of every tile, digit-major
__global__ void __launch_bounds__(RT) k_radix_tile_hist(const uint32_t* __restrict__ keys, int64_t n, int shift,
                                                        uint32_t* __restrict__ hist, int nblocks)
{
    __shared__ uint32_t h[RADIX];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RTILE;
    uint32_t k[RI];
#pragma unroll
    for (int r = 0; r < RI; r++) {
        const int64_t p = base + (int64_t)r * RT + threadIdx.x;
        k[r] = p < n ? keys[p] : 0u;
    }
#pragma unroll
    for (int r = 0; r < RI; r++)
        if (base + (int64_t)r * RT + threadIdx.x < n) atomicAdd(&h[(k[r] >> shift) & 255u], 1u);
    __syncthreads();
    hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// one pass over all tiles.  kLook: blocks take tiles in the order they start, so the tiles a block waits for are
// running, and scratch is the sort's; otherwise offs holds the scanned counts of k_radix_tile_hist
template <bool kLook>
__global__ void __launch_bounds__(RT) k_radix_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                   uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, int64_t n,
                                                   int shift, int pass, uint32_t* scratch,
                                                   const uint32_t* __restrict__ offs, int nblocks, int iota_vals)
{
    __shared__ uint32_t s_keys[RTILE];
    __shared__ uint32_t s_vals[RTILE];
    __shared__ uint32_t s_wh[NW][RADIX];  // per warp: digit counts, then the warp's offset within the digit
    __shared__ uint32_t s_start[RADIX];
    __shared__ uint32_t s_gofs[RADIX];
    __shared__ uint32_t s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    if (tid == 0) s_tile = kLook ? atomicAdd(scratch + pass, 1u) : blockIdx.x;
    for (int i = tid; i < NW * RADIX; i += RT) (&s_wh[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    volatile uint32_t* tiles = scratch + kTilesAt + (int64_t)pass * nblocks * RADIX;
    // the digit's count over all tiles, or this tile's global start of it
    const uint32_t hist = kLook ? scratch[kHistAt + pass * RADIX + tid] : offs[(int64_t)tid * nblocks + tile];
    uint32_t key[RI], val[RI], rank[RI], dig[RI];
    const int64_t base = tile * RTILE + (int64_t)warp * (32 * RI);
    uint32_t* wh = s_wh[warp];
    // warp w ranks the tile's w-th run of RT * RI / NW consecutive keys, 32 at a time, against its own counters:
    // warps cover the tile in input order, so (warp, row, lane) order is input order and the sort is stable.
    // All of the warp's loads first (independent, in flight together), then the ranking.
#pragma unroll
    for (int r = 0; r < RI; r++) {
        const int64_t p = base + r * 32 + lane;
        const bool valid = p < n;
        key[r] = valid ? kin[p] : 0u;
        val[r] = valid ? (iota_vals ? (uint32_t)p : vin[p]) : 0u;
    }
#pragma unroll
    for (int r = 0; r < RI; r++) {
        const uint32_t d = base + r * 32 + lane < n ? ((key[r] >> shift) & 255u) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = d < 256u ? wh[d] : 0u;
        __syncwarp();
        if (d < 256u && lane == (uint32_t)(__ffs(peers) - 1)) wh[d] = before + __popc(peers);
        __syncwarp();
        rank[r] = before + __popc(peers & lt_mask);
        dig[r] = d;
    }
    __syncthreads();
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
        const uint32_t c = s_wh[w][tid];
        s_wh[w][tid] = run;
        run += c;
    }
    // thread d: this tile's count of digit d, then the count of the tiles before it
    if (kLook) tiles[tile * RADIX + tid] = run | (tile == 0 ? kUpTo : kOwn);
    uint32_t tot;
    const uint32_t digit_start = kLook ? block_exclusive_scan(hist, tot) : hist;
    const uint32_t st = block_exclusive_scan(run, tot);
    s_start[tid] = st;
    __syncthreads();
    // the tile's own order does not wait for the others
#pragma unroll
    for (int r = 0; r < RI; r++) {
        if (dig[r] < 256u) {
            const uint32_t idx = s_start[dig[r]] + wh[dig[r]] + rank[r];
            s_keys[idx] = key[r];
            s_vals[idx] = val[r];
        }
    }
    // eight tiles at a time (one at a time: 14 us more a pass at 4M keys)
    constexpr int kWindow = 8;
    uint32_t before = 0, polls = 0;
    bool lost = false, found = !kLook || tile == 0;
    for (int64_t t = tile - 1; !found && !lost;) {
        uint32_t v[kWindow];
#pragma unroll
        for (int u = 0; u < kWindow; u++) v[u] = t >= u ? tiles[(t - u) * RADIX + tid] : kUpTo;
        int u = 0;
#pragma unroll
        for (int w = 0; w < kWindow; w++) {
            if (u != w || found || v[w] == 0) continue;  // stop at the first that is not there yet
            before += v[w] & kValue;
            found = (v[w] & kUpTo) != 0;
            u = w + 1;
        }
        t -= u;
        if (u == 0) lost = ++polls > kMaxPolls;
    }
    auto publish = [&] {
        if (kLook && tile > 0) tiles[tile * RADIX + tid] = (before + run) | kUpTo;
    };
    if (!lost) publish();
    s_gofs[tid] = digit_start + before - st;  // global position of tile slot j of digit d: s_gofs[d] + j (mod 2^32)
    // a wait that ran out: the block counts the digits of the tiles before it itself (up to kLookBack keys, which no
    // block of this pass writes), so the sort is complete however long a tile stalls
    if (__syncthreads_or(lost)) {
        uint32_t* cnt = s_wh[0];
        cnt[tid] = 0;
        __syncthreads();
        for (int64_t p = tid; p < tile * RTILE; p += RT) atomicAdd(&cnt[(kin[p] >> shift) & 255u], 1u);
        __syncthreads();
        before = cnt[tid];
        publish();
        s_gofs[tid] = digit_start + before - st;
        __syncthreads();
    }
    const int64_t rem = n - tile * RTILE;
    const int cnt = rem < RTILE ? (int)rem : RTILE;
#pragma unroll
    for (int r = 0; r < RI; r++) {
        const int j = r * RT + tid;
        if (j < cnt) {
            const uint32_t k = s_keys[j];
            const uint32_t o = s_gofs[(k >> shift) & 255u] + (uint32_t)j;
            kout[o] = k;
            vout[o] = s_vals[j];
        }
    }
}

// few keys: all passes in one block
constexpr int ST = 512, SI = 8, SNW = ST / 32;
constexpr int kSmallSort = ST * SI;
__global__ void __launch_bounds__(ST) k_radix_small(const uint32_t* kin, uint32_t* kout, uint32_t* vout, int n, int lo_bit, int npass)
{
    __shared__ uint32_t s_keys[kSmallSort];
    __shared__ uint16_t s_vals[kSmallSort];
    __shared__ uint16_t s_wh[SNW][RADIX];
    __shared__ uint32_t s_start[ST];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const int base = warp * (32 * SI);
    uint32_t key[SI], val[SI];
#pragma unroll
    for (int r = 0; r < SI; r++) {
        const int p = base + r * 32 + lane;
        key[r] = p < n ? kin[p] : 0u;
        val[r] = (uint32_t)p;
    }
    for (int pass = 0; pass < npass; pass++) {
        const int shift = lo_bit + 8 * pass;
        for (int i = tid; i < SNW * RADIX; i += ST) (&s_wh[0][0])[i] = 0;
        __syncthreads();
        uint16_t* wh = s_wh[warp];
        uint32_t rank[SI], dig[SI];
#pragma unroll
        for (int r = 0; r < SI; r++) {
            const uint32_t d = base + r * 32 + lane < n ? ((key[r] >> shift) & 255u) : 256u;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const uint32_t before = d < 256u ? wh[d] : 0u;
            __syncwarp();
            if (d < 256u && lane == __ffs(peers) - 1) wh[d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
            rank[r] = before + __popc(peers & lt_mask);
            dig[r] = d;
        }
        __syncthreads();
        uint32_t run = 0;
        if (tid < RADIX) {
#pragma unroll
            for (int w = 0; w < SNW; w++) {
                const uint32_t c = s_wh[w][tid];
                s_wh[w][tid] = (uint16_t)run;
                run += c;
            }
        }
        uint32_t tot;
        s_start[tid] = block_exclusive_scan(run, tot);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SI; r++) {
            if (dig[r] < 256u) {
                const uint32_t idx = s_start[dig[r]] + wh[dig[r]] + rank[r];
                s_keys[idx] = key[r];
                s_vals[idx] = (uint16_t)val[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SI; r++) {
            const int p = base + r * 32 + lane;
            if (p < n) {
                key[r] = s_keys[p];
                val[r] = s_vals[p];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < SI; r++) {
        const int p = base + r * 32 + lane;
        if (p < n) {
            kout[p] = key[r];
            vout[p] = val[r];
        }
    }
}

}  // namespace

int64_t radix_tmp_words(int64_t n)
{
    const int64_t nb = (n + RTILE - 1) / RTILE, h = nb * RADIX;
    return n <= kLookBack ? kTilesAt + kMaxPass * h + 8 : 2 * (h + 1) + scan_tmp_words(h) + 8;
}

int radix_sort_u32(uint32_t* keys, uint32_t* vals, uint32_t* alt_keys, uint32_t* alt_vals, int64_t n,
                   uint32_t* tmp, cudaStream_t s, int* launches, int lo_bit)
{
    if (n <= 0) return TC_OK;
    const int npass = (32 - lo_bit + 7) / 8;
    // an odd number of passes starts from the alternate buffers (the keys are
    // there), so that the result always lands in keys / vals
    uint32_t *ki = keys, *vi = vals, *ko = alt_keys, *vo = alt_vals;
    if (npass & 1) {
        ki = alt_keys;
        vi = alt_vals;
        ko = keys;
        vo = vals;
    }
    if (n <= kSmallSort) {
        k_radix_small<<<1, ST, 0, s>>>(ki, keys, vals, (int)n, lo_bit, npass);
        if (launches) *launches += 1;
        TC_CUDA_TRY(cudaGetLastError());
        return TC_OK;
    }
    const int nb = (int)((n + RTILE - 1) / RTILE);
    const int64_t h = (int64_t)nb * RADIX;
    const bool look = n <= kLookBack;
    uint32_t *hist = tmp, *offs = tmp + (h + 1), *stmp = offs + (h + 1);
    if (look) {
        TC_CUDA_TRY(cudaMemsetAsync(tmp, 0, (size_t)(kTilesAt + npass * h) * 4, s));
        k_radix_hist<<<grid_for(n, RTILE, sm_count() * 4), RT, 0, s>>>(ki, n, lo_bit, npass, tmp);
        if (launches) *launches += 1;
    }
    for (int pass = 0; pass < npass; pass++) {
        const int shift = lo_bit + 8 * pass;
        if (look) {
            k_radix_pass<true><<<nb, RT, 0, s>>>(ki, vi, ko, vo, n, shift, pass, tmp, nullptr, nb, pass == 0);
        } else {
            k_radix_tile_hist<<<nb, RT, 0, s>>>(ki, n, shift, hist, nb);
            int rc = exclusive_scan_u32(hist, offs, h, stmp, s);
            if (rc) return rc;
            k_radix_pass<false><<<nb, RT, 0, s>>>(ki, vi, ko, vo, n, shift, pass, nullptr, offs, nb, pass == 0);
        }
        if (launches) *launches += look ? 1 : 4;
        uint32_t* t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    TC_CUDA_TRY(cudaGetLastError());
    return TC_OK;
}

}  // namespace tc
