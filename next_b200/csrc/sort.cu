// Stable LSD radix sort of (uint64 key, uint32 value) pairs, 8-bit digits.  Up
// to 16,384 pairs one block or one cluster does all passes (kSmallSorts).  Above,
// one count of all digits over the keys (made with the keys in a tree build),
// then one "onesweep" pass per digit.  A onesweep pass works on tiles of pairs (see Layout):
//   1. load the tile, count its digits per warp (ballot peer masks, kept in
//      shared memory for the ranking; one shared add per digit group) and
//      publish the per-digit tile counts in a status array (flag + count
//      packed in one 32-bit word);
//   2. scan the counts and rank and scatter the tile into shared memory in
//      digit order;
//   3. add up the counts of the tiles before it -- all at once where there are
//      at most as many tiles as SMs, else by a decoupled look-back over 8 tiles
//      at a time that was started before the ranking -- and write the tile
//      out, each digit run to its global offset,
// so a pass reads and writes every pair exactly once.  Tiles are numbered
// in the order blocks start (an atomic ticket), so every tile a block waits
// on is already running; each wait is still bounded and raises
// NEXT_DEVERR_SORT_TIMEOUT instead of spinning forever.
//
// Memory bound: per pass 12 B read + 12 B written per pair.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.cuh"
#include "sort_digits.cuh"

namespace nb {

namespace {

constexpr int kRadix = 256;
constexpr int kHistThreads = 256;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1;
constexpr int kSpinLimit = 1 << 20;
constexpr int kLookWindow = 8;   // earlier tiles whose status one look-back step reads

// Digit counts of all passes.  Four keys per thread and round, their loads in
// flight together; small sorts get a block per 1,024 keys.
__global__ void __launch_bounds__(kHistThreads)
histogram_kernel(const uint64_t* __restrict__ keys, int64_t n, int key_bits, uint32_t* __restrict__ hist) {
    const int passes = (key_bits + 7) / 8;
    __shared__ uint32_t local[8 * kRadix];
    for (int i = threadIdx.x; i < passes * kRadix; i += kHistThreads) local[i] = 0;
    __syncthreads();
    const int64_t stride = static_cast<int64_t>(gridDim.x) * kHistThreads;
    for (int64_t i = blockIdx.x * (int64_t)kHistThreads + threadIdx.x; i < n; i += 4 * stride) {
        uint64_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < n) k[u] = keys[i + u * stride];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < n) count_digits(k[u], key_bits, local);
    }
    __syncthreads();
    add_digit_counts<kHistThreads>(local, passes, hist);
}

template <int THREADS, int ITEMS>
struct SortSmemT {
    uint32_t warp_hist[THREADS / 32][kRadix];
    uint32_t global_delta[kRadix];
    uint32_t warp_total[kRadix / 32];
    uint64_t keys[THREADS * ITEMS];
    uint32_t vals[THREADS * ITEMS];
    uint32_t peers[ITEMS][THREADS];   // the count pass's peer masks, reused by the ranking
    int tile;
};

// Lanes of the warp whose 8-bit digit equals this lane's: eight ballots,
// one per digit bit (cheaper than a match-any on this part).  Written as one
// volatile block that is also ordered with memory accesses, so the compiler
// neither hoists the bit tests of all items nor keeps them in registers.
__device__ __forceinline__ uint32_t digit_peers(int dig) {
    uint32_t peers;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 t, m, r;\n\t" "mov.u32 r, 0xffffffff;\n\t"
        "and.b32 t, %1, 1;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 2;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 4;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 8;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 16;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 32;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 64;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "and.b32 t, %1, 128;\n\t" "setp.ne.u32 p, t, 0;\n\t" "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t" "@!p not.b32 m, m;\n\t" "and.b32 r, r, m;\n\t"
        "mov.u32 %0, r;\n\t}"
        : "=r"(peers) : "r"(dig) : "memory");
    return peers;
}

// Tile loads into registers: item k of lane l of warp w is pair
// tile_base + (w * kItems + k) * 32 + l; pairs past n are padding keys that
// rank after every real key of the tile and are never written out.
template <int THREADS, int ITEMS>
__device__ __forceinline__ void load_tile(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                          int64_t n, int tile, int w, int lane, uint64_t (&key)[ITEMS],
                                          uint32_t (&val)[ITEMS]) {
    const int64_t warp_base = static_cast<int64_t>(tile) * (THREADS * ITEMS) + static_cast<int64_t>(w) * ITEMS * 32;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int64_t g = warp_base + k * 32 + lane;
        if (g < n) { key[k] = keys_in[g]; val[k] = vals_in[g]; }
        else { key[k] = ~0ull; val[k] = 0u; }
    }
}

// Four digits' status words of one tile, past L1 (another block may be about to write them).
__device__ __forceinline__ uint4 load_status(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// Persistent: a block takes tiles by ticket until none is left.  Once a
// tile's pairs sit ranked in shared memory, the block takes its next ticket
// and loads that tile into the registers the ranking has freed, so the load
// runs while this tile waits on its look-back and writes itself out.
template <int THREADS, int ITEMS, int MINB, bool DIRECT>
__global__ void __launch_bounds__(THREADS, MINB)
onesweep_kernel(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int64_t n, int shift,
                uint32_t dmask, const uint32_t* __restrict__ hist, uint32_t* status, unsigned int* tile_ticket,
                int* err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortSmemT<THREADS, ITEMS>& S = *reinterpret_cast<SortSmemT<THREADS, ITEMS>*>(smem_raw);
    constexpr int kWarps = THREADS / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int d = threadIdx.x;                 // the thread's digit, below kRadix
    const int ntiles = static_cast<int>((n + (THREADS * ITEMS) - 1) / (THREADS * ITEMS));
    if (threadIdx.x == 0) S.tile = static_cast<int>(atomicAdd(tile_ticket, 1u));
    // first output position of each digit: the pass's counts, scanned over the digits
    uint32_t digit_first = 0;
    {
        const uint32_t c = d < kRadix ? hist[d] : 0u;
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (d < kRadix && lane == 31) S.warp_total[w] = inc;
        __syncthreads();
        digit_first = inc - c;
        for (int ww = 0; ww < w && ww < kRadix / 32; ++ww) digit_first += S.warp_total[ww];
    }
    int tile = S.tile;
    // Digits are re-extracted from the keys where needed: holding them (or
    // anything derived from them) across the passes costs more registers.
    uint64_t key[ITEMS];
    uint32_t val[ITEMS];
    if (tile < ntiles) load_tile<THREADS, ITEMS>(keys_in, vals_in, n, tile, w, lane, key, val);
    while (tile < ntiles) {
        const int64_t tile_base = static_cast<int64_t>(tile) * (THREADS * ITEMS);
        for (int i = threadIdx.x; i < kWarps * kRadix; i += THREADS) (&S.warp_hist[0][0])[i] = 0;
        __syncthreads();
        // Per-warp digit counts first (fire-and-forget shared adds by each digit's
        // lowest lane), so the tile's counts are published before the ranking.
        const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int dk = static_cast<int>((key[k] >> shift) & dmask);
            const uint32_t peers = digit_peers(dk);
            S.peers[k][threadIdx.x] = peers;
            if ((peers & lt) == 0) atomicAdd(&S.warp_hist[w][dk], static_cast<uint32_t>(__popc(peers)));
        }
        __syncthreads();
        // Per digit d: exclusive prefix over warps and the tile count, published
        // at once; the first look-back window is read now and consumed after the
        // local scan and the ranking, which do not need it.
        uint32_t count = 0;
        volatile uint32_t* vstat = status;
        uint32_t win[kLookWindow];
        if (d < kRadix) {
            for (int ww = 0; ww < kWarps; ++ww) {
                const uint32_t c = S.warp_hist[ww][d];
                S.warp_hist[ww][d] = count;
                count += c;
            }
            if (!DIRECT && tile == 0) vstat[d] = kFlagInc | count;
            else vstat[static_cast<int64_t>(tile) * kRadix + d] = kFlagAgg | count;
            if (!DIRECT) {
#pragma unroll
                for (int j = 0; j < kLookWindow; ++j)
                    win[j] = tile - 1 - j >= 0 ? vstat[static_cast<int64_t>(tile - 1 - j) * kRadix + d]
                                               : static_cast<uint32_t>(kFlagInc);
            }
        }
        // Exclusive scan of the tile counts over digits: warp scans + warp totals.
        uint32_t inc = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (d < kRadix && lane == 31) S.warp_total[w] = inc;
        __syncthreads();
        uint32_t tile_start = inc - count;
        if (d < kRadix) {
            for (int ww = 0; ww < w; ++ww) tile_start += S.warp_total[ww];
            // warp_hist[w][d] becomes the first local slot of warp w's digit-d keys
            for (int ww = 0; ww < kWarps; ++ww) S.warp_hist[ww][d] += tile_start;
        }
        __syncthreads();
        // Warp-level multisplit in item order (stable: item k of every lane
        // precedes item k+1, lanes in order within an item), scattering each key
        // to its local slot as it is ranked.
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int dk = static_cast<int>((key[k] >> shift) & dmask);
            const uint32_t peers = S.peers[k][threadIdx.x];
            const uint32_t base = S.warp_hist[w][dk];
            const uint32_t pos = base + __popc(peers & lt);
            __syncwarp();
            if ((peers & lt) == 0) S.warp_hist[w][dk] = base + __popc(peers);
            S.keys[pos] = key[k];
            S.vals[pos] = val[k];
            __syncwarp();
        }
        // the tile is ranked in shared memory: take the next ticket and start
        // loading that tile into the registers it has freed
        if (threadIdx.x == 0) S.tile = static_cast<int>(atomicAdd(tile_ticket, 1u));
        __syncthreads();
        const int next = S.tile;
        if (next < ntiles) load_tile<THREADS, ITEMS>(keys_in, vals_in, n, next, w, lane, key, val);
        // Decoupled look-back for digit d over the earlier tiles, a window of
        // statuses per step: entries are taken in order, an entry without a
        // flag yet is re-read alone (bounded), the first inclusive one ends it.
        uint32_t excl = 0;
        if (DIRECT) {
            // the counts of all earlier tiles, summed at once: 64 threads take four digits each of every
            // (THREADS / 64)-th tile, four tiles' loads in flight, and the block adds up their shares
            constexpr int kGroups = THREADS / 64;
            uint4* part = reinterpret_cast<uint4*>(&S.warp_hist[0][0]);      // free once the tile is ranked
            const int g = threadIdx.x >> 6, c4 = threadIdx.x & 63;
            const uint4* st4 = reinterpret_cast<const uint4*>(status) + c4;
            uint4 sum = make_uint4(0, 0, 0, 0);
            bool timed_out = false;
            for (int t0 = g; t0 < tile; t0 += 4 * kGroups) {
                uint4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    v[j] = t0 + j * kGroups < tile ? load_status(st4 + (t0 + j * kGroups) * (kRadix / 4))
                                                   : make_uint4(kFlagAgg, kFlagAgg, kFlagAgg, kFlagAgg);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int spins = 0;
                    while ((v[j].x & v[j].y & v[j].z & v[j].w & kFlagAgg) == 0) {
                        if (++spins > kSpinLimit) { timed_out = true; break; }
                        v[j] = load_status(st4 + (t0 + j * kGroups) * (kRadix / 4));
                    }
                    sum.x += v[j].x & kCountMask; sum.y += v[j].y & kCountMask;
                    sum.z += v[j].z & kCountMask; sum.w += v[j].w & kCountMask;
                }
            }
            if (timed_out) raise_error(err, kErrSort);
            part[g * 64 + c4] = sum;
            __syncthreads();
            if (d < kRadix)
                for (int k = 0; k < kGroups; ++k) excl += (&S.warp_hist[0][0])[k * kRadix + d];
        } else if (d < kRadix && tile > 0) {
            int pred = tile - 1;
            bool done = false, timed_out = false;
            while (!done) {
#pragma unroll
                for (int j = 0; j < kLookWindow; ++j) {
                    if (done) break;
                    uint32_t v = win[j];
                    int spins = 0;
                    while ((v & (kFlagAgg | kFlagInc)) == 0) {
                        if (++spins > kSpinLimit) { timed_out = true; break; }
                        v = vstat[static_cast<int64_t>(pred - j) * kRadix + d];
                    }
                    excl += v & kCountMask;
                    done = (v & kFlagInc) || timed_out || pred - j == 0;
                }
                if (done) break;
                pred -= kLookWindow;
#pragma unroll
                for (int j = 0; j < kLookWindow; ++j)
                    win[j] = pred - j >= 0 ? vstat[static_cast<int64_t>(pred - j) * kRadix + d]
                                           : static_cast<uint32_t>(kFlagInc);
            }
            if (timed_out) raise_error(err, kErrSort);
            vstat[static_cast<int64_t>(tile) * kRadix + d] = kFlagInc | ((excl + count) & kCountMask);
        }
        // global position of local slot i with digit d: global_delta[d] + i
        if (d < kRadix) S.global_delta[d] = digit_first + excl - tile_start;
        __syncthreads();
        const int64_t valid = n - tile_base < (THREADS * ITEMS) ? n - tile_base : (THREADS * ITEMS);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int i = k * THREADS + threadIdx.x;
            if (i < valid) {
                const uint64_t kk = S.keys[i];
                const int dd = static_cast<int>((kk >> shift) & dmask);
                const uint32_t gpos = S.global_delta[dd] + static_cast<uint32_t>(i);
                if (gpos >= n) { raise_error(err, kErrIndex); continue; }
                keys_out[gpos] = kk;
                vals_out[gpos] = S.vals[i];
            }
        }
        __syncthreads();          // shared memory is reused by the next tile
        tile = next;
    }
}

// A sort of at most THREADS x ITEMS pairs in one block: every pass on the pairs
// in shared memory, by the same counts and ranking as above, without the
// counts in global memory and their clearing.  In place or not: all pairs are
// read before the first is written.
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS)
one_block_kernel(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out, uint32_t* vals_out, int n,
                 int key_bits) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortSmemT<THREADS, ITEMS>& S = *reinterpret_cast<SortSmemT<THREADS, ITEMS>*>(smem_raw);
    constexpr int kWarps = THREADS / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int d = threadIdx.x;
    const uint32_t lt = (1u << lane) - 1u;
    uint64_t key[ITEMS];
    uint32_t val[ITEMS];
    load_tile<THREADS, ITEMS>(keys_in, vals_in, n, 0, w, lane, key, val);   // the padding stays behind every pair
    for (int p = 0; 8 * p < key_bits; ++p) {
        const int shift = 8 * p;
        const uint32_t dmask = pass_mask(key_bits, p);
        for (int i = threadIdx.x; i < kWarps * kRadix; i += THREADS) (&S.warp_hist[0][0])[i] = 0;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int dk = static_cast<int>((key[k] >> shift) & dmask);
            const uint32_t peers = digit_peers(dk);
            S.peers[k][threadIdx.x] = peers;
            if ((peers & lt) == 0) atomicAdd(&S.warp_hist[w][dk], static_cast<uint32_t>(__popc(peers)));
        }
        __syncthreads();
        uint32_t count = 0;
        uint32_t c[kWarps];
        if (d < kRadix) {
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) c[ww] = S.warp_hist[ww][d];
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) count += c[ww];
        }
        uint32_t inc = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (d < kRadix && lane == 31) S.warp_total[w] = inc;
        __syncthreads();
        if (d < kRadix) {
            uint32_t start = inc - count;
            for (int ww = 0; ww < w; ++ww) start += S.warp_total[ww];
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) { S.warp_hist[ww][d] = start; start += c[ww]; }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int dk = static_cast<int>((key[k] >> shift) & dmask);
            const uint32_t peers = S.peers[k][threadIdx.x];
            const uint32_t base = S.warp_hist[w][dk];
            const uint32_t pos = base + __popc(peers & lt);
            __syncwarp();
            if ((peers & lt) == 0) S.warp_hist[w][dk] = base + __popc(peers);
            S.keys[pos] = key[k];
            S.vals[pos] = val[k];
            __syncwarp();
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int i = (w * ITEMS + k) * 32 + lane;
            key[k] = S.keys[i];
            val[k] = S.vals[i];
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = (w * ITEMS + k) * 32 + lane;
        if (i < n) { keys_out[i] = key[k]; vals_out[i] = val[k]; }
    }
}

struct SmallSort {
    int pairs;
    cudaError_t (*launch)(int n, const uint64_t* ki, const uint32_t* vi, uint64_t* ko, uint32_t* vo, int key_bits,
                          cudaStream_t st);
    cudaError_t (*prepare)();
};

template <int THREADS, int ITEMS>
constexpr SmallSort one_block() {
    return {THREADS * ITEMS,
            [](int n, const uint64_t* ki, const uint32_t* vi, uint64_t* ko, uint32_t* vo, int key_bits, cudaStream_t st) {
                one_block_kernel<THREADS, ITEMS><<<1, THREADS, sizeof(SortSmemT<THREADS, ITEMS>), st>>>(ki, vi, ko, vo, n,
                                                                                                       key_bits);
                return cudaGetLastError();
            },
            []() {
                return cudaFuncSetAttribute(one_block_kernel<THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(sizeof(SortSmemT<THREADS, ITEMS>)));
            }};
}

// A sort of at most C x THREADS x ITEMS pairs by one cluster of C blocks: a
// block holds a tile of the pairs in registers; a pass exchanges the tiles'
// digit counts through the cluster's shared memory, so every block knows the
// next position of each of its pairs, and sends them to the shared memory of
// the blocks that hold those positions.  Bound by those scattered stores and
// the two cluster barriers of a pass: a pair goes as one 16-byte store (as two,
// 16,384 pairs 26.9 us against 24.8 us).
template <int THREADS, int ITEMS>
struct ClusterSmemT {
    uint32_t warp_hist[THREADS / 32][kRadix];
    uint32_t count[kRadix];           // the tile's, read by the other blocks
    uint32_t warp_total[kRadix / 32];
    ulonglong2 pairs[THREADS * ITEMS];   // key and value, written by the other blocks
    uint32_t peers[ITEMS][THREADS];
};

template <int C, int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS)
cluster_sort_kernel(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out, uint32_t* vals_out, int n,
                    int key_bits) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Smem = ClusterSmemT<THREADS, ITEMS>;
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    constexpr int kWarps = THREADS / 32, kTile = THREADS * ITEMS;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank());
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int d = threadIdx.x;
    const uint32_t lt = (1u << lane) - 1u;
    uint64_t key[ITEMS];
    uint32_t val[ITEMS];
    load_tile<THREADS, ITEMS>(keys_in, vals_in, n, rank, w, lane, key, val);   // the padding stays behind every pair
    for (int p = 0; 8 * p < key_bits; ++p) {
        const int shift = 8 * p;
        const uint32_t dmask = pass_mask(key_bits, p);
        for (int i = threadIdx.x; i < kWarps * kRadix; i += THREADS) (&S.warp_hist[0][0])[i] = 0;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int dk = static_cast<int>((key[k] >> shift) & dmask);
            const uint32_t peers = digit_peers(dk);
            S.peers[k][threadIdx.x] = peers;
            if ((peers & lt) == 0) atomicAdd(&S.warp_hist[w][dk], static_cast<uint32_t>(__popc(peers)));
        }
        __syncthreads();
        uint32_t c[kWarps], mine = 0;
        if (d < kRadix) {
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) c[ww] = S.warp_hist[ww][d];
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) mine += c[ww];
            S.count[d] = mine;
        }
        cluster.sync();
        // per digit: the pairs of the tiles before this one, and of all tiles
        uint32_t before = 0, all = 0;
        if (d < kRadix) {
            uint32_t v[C];
#pragma unroll
            for (int b = 0; b < C; ++b) v[b] = *cluster.map_shared_rank(&S.count[d], b);
#pragma unroll
            for (int b = 0; b < C; ++b) {
                before += b < rank ? v[b] : 0u;
                all += v[b];
            }
        }
        uint32_t inc = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (d < kRadix && lane == 31) S.warp_total[w] = inc;
        __syncthreads();
        if (d < kRadix) {
            uint32_t start = inc - all + before;
            for (int ww = 0; ww < w; ++ww) start += S.warp_total[ww];
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) { S.warp_hist[ww][d] = start; start += c[ww]; }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int dk = static_cast<int>((key[k] >> shift) & dmask);
            const uint32_t peers = S.peers[k][threadIdx.x];
            const uint32_t base = S.warp_hist[w][dk];
            const uint32_t pos = base + __popc(peers & lt);          // below C x kTile
            __syncwarp();
            if ((peers & lt) == 0) S.warp_hist[w][dk] = base + __popc(peers);
            cluster.map_shared_rank(&S, pos / kTile)->pairs[pos % kTile] = make_ulonglong2(key[k], val[k]);
            __syncwarp();
        }
        cluster.sync();               // every pair has arrived, and every count has been read
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int i = (w * ITEMS + k) * 32 + lane;
            const ulonglong2 kv = S.pairs[i];
            key[k] = kv.x;
            val[k] = static_cast<uint32_t>(kv.y);
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = rank * kTile + (w * ITEMS + k) * 32 + lane;
        if (i < n) { keys_out[i] = key[k]; vals_out[i] = val[k]; }
    }
}

template <int C, int THREADS, int ITEMS>
constexpr SmallSort cluster_sort() {
    return {C * THREADS * ITEMS,
            [](int n, const uint64_t* ki, const uint32_t* vi, uint64_t* ko, uint32_t* vo, int key_bits, cudaStream_t st) {
                cudaLaunchAttribute attr{};
                attr.id = cudaLaunchAttributeClusterDimension;
                attr.val.clusterDim.x = C;
                attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3(C);
                cfg.blockDim = dim3(THREADS);
                cfg.dynamicSmemBytes = sizeof(ClusterSmemT<THREADS, ITEMS>);
                cfg.stream = st;
                cfg.attrs = &attr;
                cfg.numAttrs = 1;
                return cudaLaunchKernelEx(&cfg, cluster_sort_kernel<C, THREADS, ITEMS>, ki, vi, ko, vo, n, key_bits);
            },
            []() {
                return cudaFuncSetAttribute(cluster_sort_kernel<C, THREADS, ITEMS>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(sizeof(ClusterSmemT<THREADS, ITEMS>)));
            }};
}

// Small sorts, by size: one block up to 2,048 pairs, a cluster of four or eight
// blocks (which every GPU of this kind can launch) up to 16,384.  They need no
// counts in global memory, no clearing of them and one launch, where the passes
// above are a launch of two to six microseconds each.  Sort of a tree build,
// 30 to 39 key bits / 63 bits: 1,024 bodies 19 -> 10 / 14 us, 2,048 21 -> 12.5 / 20
// us, 4,096 22.5 -> 14.6 / 29 (in one block) -> 22.6 us, 8,192 21 -> 16 / 52 -> 26.5 us,
// 16,384 27 -> 24.5 / 52 -> 35 us; by the entry point for device buffers, 63 bits,
// host call included, 75-79 -> 34, 36, 46, 45 and 58 us.  From there on tiles on more
// SMs win: 32,768 bodies 31 us against 35 us by a cluster of eight.  Sixteen
// blocks per cluster measured 24.8 us at 16,384 and 19 us at 8,192.
constexpr SmallSort kSmallSorts[] = {one_block<256, 4>(), one_block<512, 4>(), cluster_sort<4, 256, 4>(),
                                     cluster_sort<8, 256, 4>(), cluster_sort<8, 512, 4>()};
constexpr int64_t kSmallPairs = 16384;

cudaError_t sort_small(const uint64_t* ki, const uint32_t* vi, uint64_t* ko, uint32_t* vo, int64_t n, int key_bits,
                       cudaStream_t st) {
    for (const SmallSort& s : kSmallSorts)
        if (n <= s.pairs) {
            count_launches(1);
            return s.launch(static_cast<int>(n), ki, vi, ko, vo, key_bits, st);
        }
    return cudaErrorInvalidValue;
}

// Tile layouts.  Up to 148 x 512 x 15 = 1,136,640 pairs the smallest layout is
// taken that gives every SM at most one tile: a pass then lasts one tile, and a
// tile sums the counts of all earlier ones at once (DIRECT) instead of
// following a chain of look-backs.  Above that, tiles of 256 x 15, three blocks
// per SM, whose phases overlap, with the look-back.  Whole sorts of 63-bit keys
// by the entry point for device buffers, host call included, against 256 x 8
// up to 262,144 pairs and 256 x 15 above: 262,144 pairs 117 -> 106 us, 1,048,576
// 164 -> 143 us.  A pass is bound there by the ballots and the
// ranking of an SM's own tile.
struct Layout {
    int pairs;                 // per tile
    void (*launch)(int64_t n, const uint64_t* ki, const uint32_t* vi, uint64_t* ko, uint32_t* vo, int shift,
                   uint32_t dmask, const uint32_t* hist, uint32_t* status, unsigned int* ticket, int* err,
                   cudaStream_t st);
    cudaError_t (*prepare)();
};

// Blocks of one pass: no more than fit on the device at once, each taking
// tiles until none is left.
template <int THREADS, int ITEMS, int MINB, bool DIRECT>
unsigned onesweep_grid(int64_t tiles) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, onesweep_kernel<THREADS, ITEMS, MINB, DIRECT>, THREADS,
                                                      sizeof(SortSmemT<THREADS, ITEMS>)) != cudaSuccess ||
        per_sm < 1 || sms < 1)
        return static_cast<unsigned>(tiles);
    const int64_t resident = static_cast<int64_t>(per_sm) * sms;
    return static_cast<unsigned>(tiles < resident ? tiles : resident);
}

template <int THREADS, int ITEMS, int MINB, bool DIRECT>
constexpr Layout layout() {
    return {THREADS * ITEMS,
            [](int64_t n, const uint64_t* ki, const uint32_t* vi, uint64_t* ko, uint32_t* vo, int shift, uint32_t dmask,
               const uint32_t* hist, uint32_t* status, unsigned int* ticket, int* err, cudaStream_t st) {
                const int64_t tiles = (n + THREADS * ITEMS - 1) / (THREADS * ITEMS);
                onesweep_kernel<THREADS, ITEMS, MINB, DIRECT>
                    <<<onesweep_grid<THREADS, ITEMS, MINB, DIRECT>(tiles), THREADS, sizeof(SortSmemT<THREADS, ITEMS>), st>>>(
                        ki, vi, ko, vo, n, shift, dmask, hist, status, ticket, err);
            },
            []() {
                return cudaFuncSetAttribute(onesweep_kernel<THREADS, ITEMS, MINB, DIRECT>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(sizeof(SortSmemT<THREADS, ITEMS>)));
            }};
}

constexpr Layout kOneTile[] = {layout<256, 4, 1, true>(), layout<256, 8, 1, true>(), layout<512, 8, 1, true>(),
                               layout<512, 15, 1, true>()};
constexpr Layout kManyTiles = layout<256, NB_SORT_ITEMS, 3, false>();
constexpr int64_t kOneTileBlocks = 148;    // this GPU's SMs; a fixed table, right (if not the fastest) on any number

const Layout& layout_for(int64_t n) {
    for (const Layout& l : kOneTile)
        if (n <= kOneTileBlocks * l.pairs) return l;
    return kManyTiles;
}

int64_t tiles_for(int64_t n) { return (n + layout_for(n).pairs - 1) / layout_for(n).pairs; }

}  // namespace

static_assert(kSortTile == kManyTiles.pairs, "tile size shared with the scratch-size formula");
static_assert(kSortFixedWords % 4 == 0, "statuses are read as 16-byte vectors");

// Scratch words for sorts of up to n pairs: digit counts (8 x 256), tile tickets
// (8), status (8 x tiles x 256) for the layout with the most tiles any such sort
// can use.
size_t sort_scratch_words(int64_t n) {
    const int64_t one = (n + kOneTile[0].pairs - 1) / kOneTile[0].pairs;
    const size_t few = static_cast<size_t>(kSortFixedWords + 8 * kRadix * (one < kOneTileBlocks ? one : kOneTileBlocks));
    const size_t many = static_cast<size_t>(sort_scratch_words_for(n));
    return few > many ? few : many;
}

cudaError_t sort_prepare() {
    cudaError_t e = kManyTiles.prepare();
    for (const Layout& l : kOneTile)
        if (e == cudaSuccess) e = l.prepare();
    for (const SmallSort& b : kSmallSorts)
        if (e == cudaSuccess) e = b.prepare();
    return e;
}

bool sort_counts_digits(int64_t n) { return n > kSmallPairs; }

// Clears the scratch of a sort of n pairs; the digit counts (the scratch's
// first 8 x 256 words) can be added to from then on.
cudaError_t sort_begin(int64_t n, int key_bits, uint32_t* scratch, cudaStream_t st) {
    if (!sort_counts_digits(n)) return cudaSuccess;
    const size_t words = static_cast<size_t>(kSortFixedWords + ((key_bits + 7) / 8) * tiles_for(n) * kRadix);
    return cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * words, st);
}

cudaError_t sort_count(const uint64_t* keys, int64_t n, int key_bits, uint32_t* scratch, cudaStream_t st) {
    int64_t blocks = (n + kHistThreads * 4 - 1) / (kHistThreads * 4);
    if (blocks > 592) blocks = 592;
    histogram_kernel<<<static_cast<unsigned>(blocks), kHistThreads, 0, st>>>(keys, n, key_bits, scratch);
    count_launches(1);
    return cudaGetLastError();
}

// The passes of a counted sort, from (keys_in, vals_in), which are left
// untouched unless they are also the other half of the ping-pong, to
// (keys_out, vals_out): the passes alternate between the outputs and
// (alt_keys, alt_vals), starting on whichever side makes the last pass land
// in the outputs.
cudaError_t sort_passes(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out, uint32_t* vals_out,
                        uint64_t* alt_keys, uint32_t* alt_vals, int64_t n, int key_bits, uint32_t* scratch, int* err,
                        cudaStream_t st) {
    const int passes = (key_bits + 7) / 8;
    const Layout& l = layout_for(n);
    const int64_t tiles = tiles_for(n);
    unsigned int* tickets = scratch + 8 * kRadix;
    uint32_t* status = scratch + kSortFixedWords;              // read 16 bytes at a time
    const uint64_t* src_k = keys_in;
    const uint32_t* src_v = vals_in;
    for (int p = 0; p < passes; ++p) {
        const bool to_out = ((passes - 1 - p) & 1) == 0;
        uint64_t* dst_k = to_out ? keys_out : alt_keys;
        uint32_t* dst_v = to_out ? vals_out : alt_vals;
        l.launch(n, src_k, src_v, dst_k, dst_v, 8 * p, pass_mask(key_bits, p), scratch + p * kRadix,
                 status + static_cast<int64_t>(p) * tiles * kRadix, tickets + p, err, st);
        src_k = dst_k;
        src_v = dst_v;
    }
    count_launches(passes);
    return cudaGetLastError();
}

// Sorts (keys, vals) of length n using (alt_keys, alt_vals) as the other
// half of the ping-pong.  The result lands in (keys, vals) when the number
// of passes is even, else in (alt_keys, alt_vals); *in_alt tells which.
// scratch holds sort_scratch_words(n) words.
cudaError_t radix_sort_pairs(uint64_t* keys, uint32_t* vals, uint64_t* alt_keys, uint32_t* alt_vals,
                             int64_t n, int key_bits, uint32_t* scratch, bool counted, int* err, bool* in_alt,
                             cudaStream_t st) {
    *in_alt = false;
    if (n <= 1) return cudaSuccess;
    if (!sort_counts_digits(n)) return sort_small(keys, vals, keys, vals, n, key_bits, st);
    cudaError_t e = cudaSuccess;
    if (!counted) {
        e = sort_begin(n, key_bits, scratch, st);
        if (e == cudaSuccess) e = sort_count(keys, n, key_bits, scratch, st);
        if (e != cudaSuccess) return e;
    }
    *in_alt = (((key_bits + 7) / 8) & 1) != 0;
    return *in_alt ? sort_passes(keys, vals, alt_keys, alt_vals, keys, vals, n, key_bits, scratch, err, st)
                   : sort_passes(keys, vals, keys, vals, alt_keys, alt_vals, n, key_bits, scratch, err, st);
}

// Sorts n pairs from (keys_in, vals_in) into (keys_out, vals_out), never
// writing the inputs.  scratch holds sort_scratch_words(n) words, err one word.
cudaError_t radix_sort_pairs_to(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                                uint32_t* vals_out, uint64_t* alt_keys, uint32_t* alt_vals, int64_t n, int key_bits,
                                uint32_t* scratch, int* err, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (n == 1) {
        cudaError_t e = cudaMemcpyAsync(keys_out, keys_in, sizeof(uint64_t), cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(vals_out, vals_in, sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
        return e;
    }
    if (!sort_counts_digits(n)) return sort_small(keys_in, vals_in, keys_out, vals_out, n, key_bits, st);
    cudaError_t e = sort_begin(n, key_bits, scratch, st);
    if (e == cudaSuccess) e = sort_count(keys_in, n, key_bits, scratch, st);
    if (e != cudaSuccess) return e;
    return sort_passes(keys_in, vals_in, keys_out, vals_out, alt_keys, alt_vals, n, key_bits, scratch, err, st);
}

}  // namespace nb
