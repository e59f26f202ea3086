// Octree build from sorted octant keys, and the upward (moment) pass.
//
// A cell at level l is a run of sorted keys sharing their first l octant
// digits.  With d[s] = shared-prefix level of keys s-1 and s (-1 where a
// system starts), position s starts exactly the cells of levels > d[s]; the
// cell (l, s) holds more than B bodies iff the next B keys all share l
// digits with their predecessor, i.e. l <= min(d[s+1..s+B]).  So the
// internal cells (more than B bodies, above the deepest level) starting at s
// are the levels d[s]+1 .. min(min(d[s+1..s+B]), levels-1): counted per
// position, scanned, and materialised in one pass each -- no level-by-level
// loop.  For B = 1 this is exactly the tree the reference's one-body-per-
// leaf insertion builds (src/gravity/octree.h:69-87).
//
// Numbering: internal cells get a depth-first id q (position, then level);
// nodes are laid out sibling-contiguous (children of a node consecutive, in
// octant order, system roots first) for the walks.
//
// Child bounds: one thread per internal cell runs the eight lower-bound
// searches for the cell's end and child starts together.
//
// Upward pass, two launches and no per-level loop: one thread per leaf
// computes the leaf's moments and counts itself in at its parent; parents
// whose children are all leaves are then complete and go on a ready list.
// The second launch runs one thread per ready parent: it combines the
// children and climbs, an atomic arrival counter at each parent electing the
// last child's thread to combine all children in octant order
// (deterministic) and climb on.  With accurate physics a leaf's bodies and a
// cell's children are each read in one pass (moments about the first one,
// shifted to the centre of mass by the parallel-axis rule); the reference's
// physics keeps its own two-pass order for bit-exact moments.
//
// Built with -fmad=false: every FP64 + and * rounds separately, so the
// reference-mode moments repeat src/gravity/octree.h:92-127 bit for bit.
#include "common.cuh"
#include "kernels.cuh"
#include "scan.cuh"
#include "softening.cuh"

namespace nb {

namespace {

// Words of Tree::work, zeroed at the start of every build: two tile tickets,
// the ready-list length, the deepest leaf level, the group walk's queue and
// blocks per SM, then the look-back statuses of the two scans.
constexpr int kWorkCells = 0, kWorkChildren = 1, kWorkReady = 2, kWorkDeepest = 3,
              kWorkStatus = kTreeWorkQueue + kTreeWorkWalk;
static_assert(kTreeWorkQueue == 4, "the queue's word");

// Internal cells per position, their ids and records, in one pass: d[s] for a
// tile of positions and the leaf_cap behind it (in shared memory), the counts,
// their scan over the tile and the tiles before it, and the cells themselves.
// work[kWorkDeepest] gets the deepest leaf level (one below the deepest
// internal cell) of the build, or kDepthOverfull if a cell at the last key
// level holds more than leaf_cap.
//
// Six launches (d, counts, three of a scan, cells) took 2.5-3 us each on small
// systems and re-read their arrays on large ones.  With the child counts' scan
// below in one launch too (five before): build 0.138 -> 0.123 ms at 16,384
// bodies, 0.246 -> 0.228 ms at 1,048,576, 2.79 -> 2.71 ms at 16.7 M.
constexpr int kCellThreads = 256, kCellItems = 4, kCellTile = kCellThreads * kCellItems;
constexpr int kMaxLeafCap = 64;

__global__ void __launch_bounds__(kCellThreads)
cells_kernel(const uint64_t* __restrict__ keys, int64_t n, int base, int levels, int leaf_cap, Tree t, int* err) {
    __shared__ int8_t d[kCellTile + kMaxLeafCap + 1];
    __shared__ unsigned long long before;
    __shared__ int ticket;
    __shared__ unsigned deepest;
    if (threadIdx.x == 0) {
        ticket = static_cast<int>(atomicAdd(t.work + kWorkCells, 1ull));
        deepest = 0;
    }
    __syncthreads();
    const int tile = ticket;
    const int64_t s0 = static_cast<int64_t>(tile) * kCellTile;
    // positions past the last body get -1: no run of equal prefixes crosses the end
    for (int p = threadIdx.x; p <= kCellTile + leaf_cap; p += kCellThreads) {
        const int64_t s = s0 + p;
        d[p] = static_cast<int8_t>(s == 0 || s >= n ? -1 : shared_levels(keys[s - 1], keys[s], base, levels));
    }
    __syncthreads();
    // the thread's positions p0 .. p0 + 3; window of position p0 + i: p0 + i + 1 .. p0 + i + leaf_cap
    const int p0 = threadIdx.x * kCellItems;
    int own[kCellItems], cnt[kCellItems];
#pragma unroll
    for (int i = 0; i < kCellItems; ++i) own[i] = d[p0 + i];
    int win[kCellItems];
    if (leaf_cap >= kCellItems) {
        int core = 127;                                    // what all four windows share
        for (int p = p0 + kCellItems; p <= p0 + leaf_cap; ++p) core = min(core, static_cast<int>(d[p]));
#pragma unroll
        for (int i = 0; i < kCellItems; ++i) {
            win[i] = core;
#pragma unroll
            for (int k = 1; k < kCellItems; ++k) {
                if (k > i) win[i] = min(win[i], own[k]);
                if (k <= i) win[i] = min(win[i], static_cast<int>(d[p0 + leaf_cap + k]));
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < kCellItems; ++i) {
            win[i] = 127;
            for (int j = 1; j <= leaf_cap; ++j) win[i] = min(win[i], static_cast<int>(d[p0 + i + j]));
        }
    }
    unsigned deep = 0;
    unsigned long long mine = 0;
#pragma unroll
    for (int i = 0; i < kCellItems; ++i) {
        const int top = min(win[i], levels - 1);
        cnt[i] = s0 + p0 + i < n ? max(0, top - own[i]) : 0;
        mine += static_cast<unsigned>(cnt[i]);
        if (cnt[i] > 0) deep = max(deep, static_cast<unsigned>(top + 1));
        if (s0 + p0 + i < n && win[i] >= levels) deep = kDepthOverfull;
    }
    deep = __reduce_max_sync(0xffffffffu, deep);
    if ((threadIdx.x & 31) == 0 && deep) atomicMax(&deepest, deep);
    unsigned long long sum;
    const unsigned long long ex = block_exclusive<kCellThreads>(mine, &sum);
    if (threadIdx.x < 32) {
        const unsigned long long b = look_back(t.work + kWorkStatus, tile, sum, err);
        if (threadIdx.x == 0) before = b;
    }
    __syncthreads();
    int64_t q = static_cast<int64_t>(before + ex);
    int first[kCellItems];
#pragma unroll
    for (int i = 0; i < kCellItems; ++i) { first[i] = static_cast<int>(q); q += cnt[i]; }
    const int64_t s = s0 + p0;
    if (s + kCellItems <= n) {
        *reinterpret_cast<int4*>(t.nint + s) = make_int4(first[0], first[1], first[2], first[3]);
        *reinterpret_cast<char4*>(t.dlev + s) = make_char4(own[0], own[1], own[2], own[3]);
    } else {
#pragma unroll
        for (int i = 0; i < kCellItems; ++i)
            if (s + i < n) { t.nint[s + i] = first[i]; t.dlev[s + i] = static_cast<int8_t>(own[i]); }
    }
#pragma unroll
    for (int i = 0; i < kCellItems; ++i) {
        for (int k = 0; k < cnt[i]; ++k) {
            const int64_t c = static_cast<int64_t>(first[i]) + k;
            if (c >= t.cap_int) { raise_error(err, kErrTree); break; }
            t.int_start[c] = static_cast<int32_t>(s + i);
            t.int_level[c] = static_cast<int8_t>(own[i] + 1 + k);
        }
    }
    if (threadIdx.x == 0) {
        // skipped where it cannot raise the value: one hot address
        unsigned long long* all = t.work + kWorkDeepest;
        if (deepest > *reinterpret_cast<volatile unsigned long long*>(all))
            atomicMax(all, static_cast<unsigned long long>(deepest));
        if (s0 + kCellTile >= n) {
            t.nint[n] = static_cast<int32_t>(before + sum);
            t.counts[0] = static_cast<int64_t>(before + sum);
        }
    }
}

// Walk groups from the children of one cell holding more than G bodies:
// the bodies of consecutive children of at most G bodies are cut into runs
// of G in key order (a child that does not fit tops the current run up to G
// and starts the next one with the rest of its bodies), so most groups fill
// a warp; a child of more than G bodies that is a leaf (deepest level) is
// cut into chunks of G.  emit(start, count) is called per group; returns
// the count.
template <typename F>
__device__ int pack_groups(const int32_t* b, int level, int levels, int leaf_cap, int group_cap, F emit) {
    int ng = 0, run_start = -1, run_cnt = 0;
    for (int c = 0; c < 8; ++c) {
        const int cnt = b[c + 1] - b[c];
        if (cnt == 0) continue;
        if (cnt <= group_cap) {
            if (run_start >= 0 && run_cnt + cnt <= group_cap) {
                run_cnt += cnt;
            } else if (run_start >= 0) {
                // top the run up to group_cap with the first bodies of this
                // child and go on with the rest of it: full warps
                const int take = group_cap - run_cnt;
                emit(run_start, group_cap); ++ng;
                run_start = b[c] + take; run_cnt = cnt - take;
            } else {
                run_start = b[c]; run_cnt = cnt;
            }
        } else {
            if (run_start >= 0) { emit(run_start, run_cnt); ++ng; run_start = -1; run_cnt = 0; }
            const bool leaf = !(cnt > leaf_cap && level + 1 < levels);
            if (leaf)
                for (int o = 0; o < cnt; o += group_cap) { emit(b[c] + o, min(group_cap, cnt - o)); ++ng; }
        }
    }
    if (run_start >= 0) { emit(run_start, run_cnt); ++ng; }
    return ng;
}

// Child boundaries of every internal cell (l, s): the cell ends at the first
// key above its prefix, and child c starts at the first key >= prefix | c at
// level l+1.  All eight are lower bounds over the same range [s, system end),
// run together with one shared step sequence (the range halves every step
// whatever the comparisons give), so a thread has eight independent loads in
// flight per step and no divergence.  The counts of children and walk groups
// are scanned here too (tiles of cells by ticket, look-back between them); the
// last tile checks the totals.
//
// Bound by the instructions of a thread's searches (keys in shared memory
// changed nothing at up to 22,000 bodies): reading dlev as 16-byte vectors,
// tested four bytes at a time, and 32-bit positions instead of a byte at a time
// and 64-bit ones took the build from 0.076 to 0.072 ms at 1,024 bodies, 0.109
// to 0.106 ms at 16,384, 0.215 to 0.210 ms at 1,048,576, and 0.548 to 0.522 ms
// with as many one-body leaves.
constexpr int kEndScan = 128;
// The child bounds of cell q, stored, and its counts of children and groups.
__device__ __forceinline__ void find_children(const uint64_t* __restrict__ keys, int64_t n,
                                              const int32_t* __restrict__ sysid, const int64_t* __restrict__ offsets,
                                              int base, int levels, int leaf_cap, int group_cap, int64_t q, Tree& t,
                                              int* err, int* nchild, int* ngroups) {
    const int s = t.int_start[q];
    const int l = t.int_level[q];
    if (s < 0 || s >= n || l < 0 || l >= levels) { raise_error(err, kErrIndex); return; }
    const int64_t hi = offsets ? offsets[(sysid ? sysid[s] : 0) + 1] : n;
    const uint64_t ks = keys[s];
    const int sh = base - 3 * l;                       // bits below level l's digits
    const uint64_t low = (sh >= 64) ? ~0ull : ((1ull << sh) - 1ull);
    const uint64_t prefix = ks & ~low;
    const int csh = sh - 3;
    uint64_t v[8];
    v[0] = (prefix | low) + 1ull;                      // end of the cell
#pragma unroll
    for (int c = 1; c < 8; ++c) v[c] = prefix | (static_cast<uint64_t>(c) << csh);
    // A small cell's end is the first p > s whose key shares fewer than l
    // digits with its predecessor (dlev[p] < l): found by reading dlev forward,
    // 32 aligned bytes per round trip, for some kEndScan positions; the
    // children's searches then run over the cell only.
    const int hi32 = static_cast<int>(hi);
    int e = -1;
    {
        const int lim = min(hi32, s + 1 + kEndScan);
        const unsigned l4 = 0x01010101u * static_cast<unsigned>(l);
        for (int w0 = (s + 1) & ~15; w0 < lim && e < 0; w0 += 32) {
            uint4 v2[2];
#pragma unroll
            for (int j = 0; j < 2; ++j)
                v2[j] = w0 + 16 * j < lim ? *reinterpret_cast<const uint4*>(t.dlev + w0 + 16 * j) : make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                const uint4& q4 = v2[j >> 2];
                const unsigned word = (j & 3) == 0 ? q4.x : (j & 3) == 1 ? q4.y : (j & 3) == 2 ? q4.z : q4.w;
                // the top bit of each byte below l: bytes and l are at most 21, and a system's start
                // (-1) is never inside the range
                unsigned less = ~((word | 0x80808080u) - l4) & 0x80808080u;
                const int p = w0 + 4 * j;
                if (p <= s) less = s + 1 - p >= 4 ? 0u : less & (~0u << 8 * (s + 1 - p));
                if (less) e = p + ((__ffs(static_cast<int>(less)) - 1) >> 3);
            }
        }
        if (e > lim || (e < 0 && lim == hi32)) e = lim == hi32 ? hi32 : -1;
    }
    int pos[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) pos[c] = s;
    int len = (e >= 0 ? e : hi32) - s;
    while (len > 1) {
        const int half = len >> 1;
#pragma unroll
        for (int c = 0; c < 8; ++c) pos[c] = __ldg(keys + pos[c] + half) < v[c] ? pos[c] + half : pos[c];
        len -= half;
    }
    int32_t b[9];
    b[0] = s;
#pragma unroll
    for (int c = 1; c < 8; ++c) b[c] = pos[c] + (__ldg(keys + pos[c]) < v[c] ? 1 : 0);
    b[8] = e >= 0 ? e : pos[0] + (__ldg(keys + pos[0]) < v[0] ? 1 : 0);
    for (int c = 0; c < 8; ++c) *nchild += b[c + 1] > b[c];
    if (b[8] - b[0] > group_cap)
        *ngroups = pack_groups(b, l, levels, leaf_cap, group_cap, [](int, int) {});
    for (int c = 0; c < 9; ++c) t.int_bounds[9 * q + c] = b[c];
}

constexpr int kChildThreads = 256;
__global__ void __launch_bounds__(kChildThreads)
internal_kernel(const uint64_t* __restrict__ keys, int64_t n, const int32_t* __restrict__ sysid,
                const int64_t* __restrict__ offsets, int nsys, int base, int levels, int leaf_cap, int group_cap,
                int64_t status_at, Tree t, int* err) {
    // the whole block leaves or none of it: other blocks of this launch may be raising bits, and a block that
    // only some of its threads left would take its tiles from a ticket that nobody writes
    if (__syncthreads_or(*err & kErrAbort)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            t.counts[1] = t.counts[2] = nsys;
            t.counts[3] = static_cast<int64_t>(t.work[kWorkDeepest]);
        }
        return;
    }
    __shared__ unsigned long long before;
    __shared__ int ticket;
    const int64_t m = t.counts[0] < t.cap_int ? t.counts[0] : t.cap_int;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) ticket = static_cast<int>(atomicAdd(t.work + kWorkChildren, 1ull));
        __syncthreads();
        const int tile = ticket;
        const int64_t q0 = static_cast<int64_t>(tile) * kChildThreads;
        if (q0 >= m && tile > 0) break;
        const int64_t q = q0 + threadIdx.x;
        int nchild = 0, ngroups = 0;
        if (q < m)
            find_children(keys, n, sysid, offsets, base, levels, leaf_cap, group_cap, q, t, err, &nchild, &ngroups);
        unsigned long long sum;
        const unsigned long long ex = block_exclusive<kChildThreads>(
            static_cast<unsigned long long>(nchild) | (static_cast<unsigned long long>(ngroups) << 32), &sum);
        if (threadIdx.x < 32) {
            const unsigned long long b = look_back(t.work + status_at, tile, sum, err);
            if (threadIdx.x == 0) before = b;
        }
        __syncthreads();
        if (q < m) t.int_packed[q] = static_cast<int64_t>(before + ex);
        if (threadIdx.x == 0 && q0 + kChildThreads >= m) {
            const unsigned long long all = before + sum;
            t.int_packed[m] = static_cast<int64_t>(all);
            const int64_t nodes = nsys + static_cast<int64_t>(all & 0xffffffffull);
            const int64_t groups = nsys + static_cast<int64_t>(all >> 32);
            if (nodes > t.cap_node || groups > t.cap_group) raise_error(err, kErrTree);
            t.counts[1] = nodes < t.cap_node ? nodes : t.cap_node;
            t.counts[2] = groups < t.cap_group ? groups : t.cap_group;
            t.counts[3] = static_cast<int64_t>(t.work[kWorkDeepest]);
        }
    }
}

// Geometric centre of the level-l cell holding `key` (the reference's child
// centre rule, src/gravity/octree.h:56-64).
__device__ double3 cell_centre(uint64_t key, int level, double4 cube, int base) {
    double cx = cube.x, cy = cube.y, cz = cube.z, h = cube.w;
    for (int l = 1; l <= level; ++l) {
        const int d = key_digit(key, l, base);
        const double hs = h * 0.5;
        cx = cx + ((d & 1) ? hs : -hs);
        cy = cy + ((d & 2) ? hs : -hs);
        cz = cz + ((d & 4) ? hs : -hs);
        h = hs;
    }
    return make_double3(cx, cy, cz);
}

__global__ void children_kernel(const uint64_t* __restrict__ keys, const int8_t* __restrict__ dlev,
                                const int32_t* __restrict__ int_base, const int32_t* __restrict__ sysid,
                                const int64_t* __restrict__ offsets, const double4* __restrict__ cubes, int64_t n,
                                int nsys, int base, int levels, int leaf_cap, int group_cap, bool accurate, Tree t,
                                int* err) {
    if (*err & kErrAbort) return;
    // the system roots: leaves here, internal ones by their cell below
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsys; s += gridDim.x * blockDim.x) {
        const int64_t b = offsets ? offsets[s] : 0;
        const int64_t e = offsets ? offsets[s + 1] : n;
        const int cnt = static_cast<int>(e - b);
        if (cnt <= leaf_cap) {
            t.link[s] = make_int2(static_cast<int>(b), -cnt);
            t.parent[s] = -1;
            t.level[s] = 0;
        }
        t.groups[s] = make_int4(static_cast<int>(b), cnt <= group_cap ? cnt : 0, s, 0);
    }
    const int64_t m = t.counts[0];
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m; q += (int64_t)gridDim.x * blockDim.x) {
        const int l = t.int_level[q];
        const int s = t.int_start[q];
        int32_t b[9];
        for (int c = 0; c < 9; ++c) b[c] = t.int_bounds[9 * q + c];
        const int64_t pk = t.int_packed[q], nx = t.int_packed[q + 1];
        const int fc = nsys + static_cast<int>(pk & 0xffffffffll);
        const int nc = static_cast<int>((nx & 0xffffffffll) - (pk & 0xffffffffll));
        const int fg = nsys + static_cast<int>(pk >> 32);
        const int sys = sysid ? sysid[s] : 0;
        // the cell's centre (accurate physics) and half-width, for the upward pass
        const double4 cube = cubes[sys];
        double4 cell = make_double4(0.0, 0.0, 0.0, ldexp(cube.w, -l));
        if (accurate) {
            const double3 g = cell_centre(keys[s], l, cube, base);
            cell.x = g.x; cell.y = g.y; cell.z = g.z;
        }
        t.cell[q] = cell;
        if (l == 0) {
            t.link[sys] = make_int2(fc, nc);
            t.climb[q] = make_int4(sys, fc, nc, -1);
            t.parent[sys] = -1;
            t.level[sys] = 0;
        }
        // every child's records are loaded before the first store (the tree's
        // arrays may alias as far as the compiler knows, so loads after a
        // store would each wait for it), and checked before any store
        int64_t q2c[8], p2c[8], n2c[8];
        bool bad = fc + nc > t.cap_node;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int cs = b[c], cnt = b[c + 1] - b[c];
            q2c[c] = -1; p2c[c] = 0; n2c[c] = 0;
            if (cnt > leaf_cap && l + 1 < levels) {
                const int64_t q2 = static_cast<int64_t>(int_base[cs]) + (l + 1 - dlev[cs] - 1);
                q2c[c] = q2;
                if (q2 <= q || q2 >= m) bad = true;
                else { p2c[c] = t.int_packed[q2]; n2c[c] = t.int_packed[q2 + 1]; }
            }
        }
        if (bad) { raise_error(err, kErrIndex); return; }
        int k = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int cs = b[c], cnt = b[c + 1] - b[c];
            if (cnt == 0) continue;
            const int nid = fc + k++;
            t.parent[nid] = static_cast<int32_t>(q);
            t.level[nid] = static_cast<int8_t>(l + 1);
            if (q2c[c] >= 0) {
                const int64_t q2 = q2c[c];
                const int fc2 = nsys + static_cast<int>(p2c[c] & 0xffffffffll);
                const int nc2 = static_cast<int>((n2c[c] & 0xffffffffll) - (p2c[c] & 0xffffffffll));
                t.link[nid] = make_int2(fc2, nc2);
                t.climb[q2] = make_int4(nid, fc2, nc2, static_cast<int>(q));
            } else {
                t.link[nid] = make_int2(cs, -cnt);
            }
        }
        if (b[8] - b[0] > group_cap) {
            int g = fg;
            int4* groups = t.groups;
            const int64_t gcap = t.cap_group;
            pack_groups(b, l, levels, leaf_cap, group_cap, [&](int gs, int gc) {
                if (g < gcap) groups[g] = make_int4(gs, gc, sys, 0);
                ++g;
            });
        }
    }
}

// ---- moments ---------------------------------------------------------------

__device__ __forceinline__ double4 ldcg4(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldcg(q), b = __ldcg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ double4 ldg4(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldg(q), b = __ldg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

struct Mom {
    double m, cx, cy, cz, q[6];
};

__device__ __forceinline__ void store_moments(Tree& t, int nid, int2 link, const Mom& a, double half, double rcrit,
                                              double G, bool accurate) {
    t.com[nid] = make_double4(a.cx, a.cy, a.cz, a.m);
    double2* q64 = reinterpret_cast<double2*>(t.quad64 + 8 * static_cast<int64_t>(nid));
    q64[0] = make_double2(a.q[0], a.q[1]);
    q64[1] = make_double2(a.q[2], a.q[3]);
    q64[2] = make_double2(a.q[4], a.q[5]);
    q64[3] = make_double2(half, rcrit);
    if (accurate) {
        const float r2 = a.m > 0.0 ? static_cast<float>(rcrit * rcrit) : -1.0f;
        t.box[nid] = make_float4(static_cast<float>(a.cx), static_cast<float>(a.cy), static_cast<float>(a.cz), r2);
        // stored negated (-G Q): the walk's quadrupole terms then need no negation
        t.quad32[2 * static_cast<int64_t>(nid)] =
            make_float4(static_cast<float>(-G * a.q[0]), static_cast<float>(-G * a.q[1]),
                        static_cast<float>(-G * a.q[2]), static_cast<float>(-G * a.q[3]));
        t.quad32[2 * static_cast<int64_t>(nid) + 1] =
            make_float4(static_cast<float>(-G * a.q[4]), static_cast<float>(-G * a.q[5]), static_cast<float>(G * a.m), 0.0f);
    } else {
        // what the reference's softening of this node has that no target changes: a cube root and,
        // for the dark bodies of the one mass, a power, once per node instead of once per interaction
        const double dark = *t.dark_mass;
        t.soft[2 * static_cast<int64_t>(nid)] = make_double2(half, __hiloint2double(link.y, link.x));
        t.soft[2 * static_cast<int64_t>(nid) + 1] =
            make_double2(softening_base(half, a.m), dark == dark ? softening_dark(half, a.m, dark) : 0.0);
    }
}

// Reference rules (src/gravity/octree.h:104-126) over a list of (m, x, y, z)
// children in octant order; `size` is the cell's half-width.
template <typename Get>
__device__ Mom combine_ref(int count, double size, Get get) {
    Mom a{};
    double m = 0, cx = 0, cy = 0, cz = 0;
    for (int k = 0; k < count; ++k) {
        const double4 c = get(k);
        if (c.w == 0) continue;
        m += c.w;
        cx += c.x * c.w; cy += c.y * c.w; cz += c.z * c.w;
    }
    if (m > 0) { cx /= m; cy /= m; cz /= m; }
    for (int k = 0; k < count; ++k) {
        const double4 c = get(k);
        if (c.w == 0) continue;
        const double rx = c.x - cx, ry = c.y - cy, rz = c.z - cz;
        const double r2 = rx * rx + ry * ry + rz * rz + (size * size * 0.01);
        const double mc = c.w;
        a.q[0] += mc * (3.0 * rx * rx - r2);
        a.q[1] += mc * (3.0 * ry * ry - r2);
        a.q[2] += mc * (3.0 * rz * rz - r2);
        a.q[3] += mc * (3.0 * rx * ry);
        a.q[4] += mc * (3.0 * rx * rz);
        a.q[5] += mc * (3.0 * ry * rz);
    }
    a.m = m; a.cx = cx; a.cy = cy; a.cz = cz;
    return a;
}

// The same over the (up to 8) children of a cell, held in registers.
__device__ __forceinline__ Mom combine_ref8(int count, double size, const double4 (&c)[8]) {
    Mom a{};
    double m = 0, cx = 0, cy = 0, cz = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k >= count || c[k].w == 0) continue;
        m += c[k].w;
        cx += c[k].x * c[k].w; cy += c[k].y * c[k].w; cz += c[k].z * c[k].w;
    }
    if (m > 0) { cx /= m; cy /= m; cz /= m; }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k >= count || c[k].w == 0) continue;
        const double rx = c[k].x - cx, ry = c[k].y - cy, rz = c[k].z - cz;
        const double r2 = rx * rx + ry * ry + rz * rz + (size * size * 0.01);
        const double mc = c[k].w;
        a.q[0] += mc * (3.0 * rx * rx - r2);
        a.q[1] += mc * (3.0 * ry * ry - r2);
        a.q[2] += mc * (3.0 * rz * rz - r2);
        a.q[3] += mc * (3.0 * rx * ry);
        a.q[4] += mc * (3.0 * rx * rz);
        a.q[5] += mc * (3.0 * ry * rz);
    }
    a.m = m; a.cx = cx; a.cy = cy; a.cz = cz;
    return a;
}

__device__ __forceinline__ double rcrit_of(const Mom& a, double3 g, double half, double theta) {
    double ox = a.cx - g.x, oy = a.cy - g.y, oz = a.cz - g.z;
    if (!(a.m > 0)) { ox = oy = oz = 0.0; }
    return 2.0 * half / theta + sqrt(ox * ox + oy * oy + oz * oz);
}

__device__ __forceinline__ int arrive_acq_rel(int32_t* counter) {
    int old;
    asm volatile("atom.add.acq_rel.gpu.s32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
    return old;
}

// Moments of leaf n (bodies [first, first + cnt)), stored.
__device__ __forceinline__ void leaf_moments(const Bodies& bd, const uint64_t* __restrict__ keys,
                                             const int32_t* __restrict__ sysid, const double4* __restrict__ cubes,
                                             int base, const Params& P, Tree& t, bool accurate, int64_t n, int first,
                                             int cnt) {
    const int lvl = t.level[n];
    // an empty leaf can only be the root of an empty system (node id = system)
    const int sys = sysid ? (cnt > 0 ? sysid[first] : static_cast<int>(n)) : 0;
    const double4 cube = cubes[sys];
    const double half = ldexp(cube.w, -lvl);
    Mom a{};
    double rcrit = 0.0;
    if (!accurate) {
        if (cnt == 1) {
            a.m = bd.m[first]; a.cx = bd.x[first]; a.cy = bd.y[first]; a.cz = bd.z[first];
        } else if (cnt > 1) {
            a = combine_ref(cnt, half, [&](int k) {
                return make_double4(bd.x[first + k], bd.y[first + k], bd.z[first + k], bd.m[first + k]);
            });
        }
    } else {
        // one pass over the leaf's bodies: mass, first and second moments
        // about its first body (all of cell size, so no cancellation),
        // then shifted to the centre of mass
        const double3 g = cell_centre(cnt > 0 ? keys[first] : 0ull, lvl, cube, base);
        const double x0 = cnt > 0 ? bd.x[first] : 0.0, y0 = cnt > 0 ? bd.y[first] : 0.0,
                     z0 = cnt > 0 ? bd.z[first] : 0.0;
        double m = 0, sx = 0, sy = 0, sz = 0, sxx = 0, syy = 0, szz = 0, sxy = 0, sxz = 0, syz = 0;
        const auto add = [&](double mj, double xj, double yj, double zj) {
            const double dx = xj - x0, dy = yj - y0, dz = zj - z0;
            const double mx = mj * dx, my = mj * dy, mz = mj * dz;
            m += mj; sx += mx; sy += my; sz += mz;
            sxx += mx * dx; syy += my * dy; szz += mz * dz;
            sxy += mx * dy; sxz += mx * dz; syz += my * dz;
        };
        int j = first;
        // A bucket of the deepest level may hold any number of bodies: eight at a time, all loads before the first
        // sum, else the thread waits for one sector of four bodies after another, as long as the bucket's alignment
        // has it (build with a bucket of 3,900 bodies 681 us, of 3,950 434 us; now 385 and 435 us).
        for (; j + 8 <= first + cnt && cnt > kMaxLeafCap; j += 8) {
            double v[8][4];
#pragma unroll
            for (int k = 0; k < 8; ++k) { v[k][0] = bd.m[j + k]; v[k][1] = bd.x[j + k]; v[k][2] = bd.y[j + k]; v[k][3] = bd.z[j + k]; }
#pragma unroll
            for (int k = 0; k < 8; ++k) add(v[k][0], v[k][1], v[k][2], v[k][3]);
        }
        for (; j < first + cnt; ++j) add(bd.m[j], bd.x[j], bd.y[j], bd.z[j]);
        double cx, cy, cz;
        if (m > 0) {
            const double ox = sx / m, oy = sy / m, oz = sz / m;
            cx = x0 + ox; cy = y0 + oy; cz = z0 + oz;
            // second moments about the centre of mass
            const double qxx = sxx - sx * ox, qyy = syy - sy * oy, qzz = szz - sz * oz;
            const double tr = qxx + qyy + qzz;
            a.q[0] = 3.0 * qxx - tr; a.q[1] = 3.0 * qyy - tr; a.q[2] = 3.0 * qzz - tr;
            a.q[3] = 3.0 * (sxy - sx * oy); a.q[4] = 3.0 * (sxz - sx * oz); a.q[5] = 3.0 * (syz - sy * oz);
        } else {
            cx = g.x; cy = g.y; cz = g.z;
        }
        a.m = m; a.cx = cx; a.cy = cy; a.cz = cz;
        rcrit = rcrit_of(a, g, half, P.theta);
    }
    store_moments(t, static_cast<int>(n), make_int2(first, -cnt), a, half, rcrit, P.G, accurate);
}

// Moments of internal node rec.x from its children rec.y .. rec.y + nchild
// (all of them final), stored; cell = its geometric centre and half-width.
template <bool ACCURATE>
__device__ __forceinline__ void combine_children(const Params& P, Tree& t, const int4 rec, const double4 cell) {
    const int first = rec.y, count = rec.z;
    const double half = cell.w;
    Mom p{};
    double prc = 0.0;
    if (!ACCURATE) {
        // the children's masses and centres once, for both of the reference's passes
        double4 c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = k < count ? ldcg4(t.com + first + k) : make_double4(0.0, 0.0, 0.0, 0.0);
        p = combine_ref8(count, half, c);
    } else {
        // one pass over the children: mass, first and second moments of
        // their centres of mass about the first child's, their own
        // quadrupoles; then shifted to the parent's centre of mass
        // (parallel axes)
        double4 c[8];
        double2 cq[8][3];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k < count) {
                c[k] = ldcg4(t.com + first + k);
                const double2* q2 = reinterpret_cast<const double2*>(t.quad64 + 8 * static_cast<int64_t>(first + k));
#pragma unroll
                for (int f = 0; f < 3; ++f) cq[k][f] = __ldcg(q2 + f);
            }
        }
        const double4 c0 = c[0];
        double m = 0, sx = 0, sy = 0, sz = 0, sxx = 0, syy = 0, szz = 0, sxy = 0, sxz = 0, syz = 0;
        double qs[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k >= count) break;
            const double dx = c[k].x - c0.x, dy = c[k].y - c0.y, dz = c[k].z - c0.z;
            const double mx = c[k].w * dx, my = c[k].w * dy, mz = c[k].w * dz;
            m += c[k].w; sx += mx; sy += my; sz += mz;
            sxx += mx * dx; syy += my * dy; szz += mz * dz;
            sxy += mx * dy; sxz += mx * dz; syz += my * dz;
#pragma unroll
            for (int f = 0; f < 3; ++f) { qs[2 * f] += cq[k][f].x; qs[2 * f + 1] += cq[k][f].y; }
        }
        double cx, cy, cz;
        if (m > 0) {
            const double ox = sx / m, oy = sy / m, oz = sz / m;
            cx = c0.x + ox; cy = c0.y + oy; cz = c0.z + oz;
            const double qxx = sxx - sx * ox, qyy = syy - sy * oy, qzz = szz - sz * oz;
            const double tr = qxx + qyy + qzz;
            p.q[0] = qs[0] + (3.0 * qxx - tr); p.q[1] = qs[1] + (3.0 * qyy - tr);
            p.q[2] = qs[2] + (3.0 * qzz - tr); p.q[3] = qs[3] + 3.0 * (sxy - sx * oy);
            p.q[4] = qs[4] + 3.0 * (sxz - sx * oz); p.q[5] = qs[5] + 3.0 * (syz - sy * oz);
        } else {
            cx = cell.x; cy = cell.y; cz = cell.z;
            for (int f = 0; f < 6; ++f) p.q[f] = qs[f];
        }
        p.m = m; p.cx = cx; p.cy = cy; p.cz = cz;
        prc = rcrit_of(p, make_double3(cell.x, cell.y, cell.z), half, P.theta);
    }
    store_moments(t, rec.x, make_int2(first, count), p, half, prc, P.G, ACCURATE);
}

// A climb record is valid when it describes a node with 1-8 children inside
// the node array; false (and the index error raised) otherwise.
__device__ __forceinline__ bool climb_record_check(int64_t nodes, const int4& rec, int* err) {
    const int nc = rec.z;
    if (rec.x < 0 || rec.x >= nodes || nc < 1 || nc > 8 || rec.y < 0 || static_cast<int64_t>(rec.y) + nc > nodes) {
        raise_error(err, kErrIndex);
        return false;
    }
    return true;
}

// From internal id q, whose children are all final, upward: combine q's
// children and arrive at the parent; the last child's thread goes on there.
template <bool ACCURATE>
__device__ __forceinline__ void climb_from(int q, const Params& P, Tree& t, int64_t nodes, int64_t ninternal, int* err) {
    int4 rec = q < ninternal ? __ldg(t.climb + q) : make_int4(0, 0, 0, 0);
    double4 cell = q < ninternal ? ldg4(t.cell + q) : make_double4(0.0, 0.0, 0.0, 0.0);
    for (;;) {
        if (q >= ninternal) { raise_error(err, kErrIndex); break; }
        if (!climb_record_check(nodes, rec, err)) break;
        const int up = rec.w;
        const int4 cur = rec;
        const double4 here = cell;
        // the next level's record, loaded before this level's stores
        if (up >= 0 && up < ninternal) { rec = __ldg(t.climb + up); cell = ldg4(t.cell + up); }
        combine_children<ACCURATE>(P, t, cur, here);
        if (up < 0) break;
        if (up >= ninternal) { raise_error(err, kErrIndex); break; }
        // release this cell's moments / acquire its siblings'
        if (arrive_acq_rel(t.counter + up) != rec.z - 1) break;
        t.counter[up] = 0;                     // re-armed for the next build
        q = up;
    }
}

// Two launches.  Leaves: one thread per leaf computes its moments and counts
// itself in at its parent (a plain atomic: the climb launch that reads the
// moments comes after this one); a parent all of whose children are leaves
// is complete when its last leaf arrives, and goes on the ready list.
template <bool ACCURATE>
__global__ void __launch_bounds__(256, 3)
upward_leaves_kernel(Bodies bd, int64_t nbodies, const uint64_t* __restrict__ keys,
                     const int32_t* __restrict__ sysid, const double4* __restrict__ cubes, int base, Params P, Tree t,
                     int* err) {
    if (*err & kErrAbort) return;
    constexpr bool accurate = ACCURATE;
    const int64_t nodes = t.counts[1];
    const int64_t ninternal = t.counts[0];
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nodes;
         n += (int64_t)gridDim.x * blockDim.x) {
        const int2 lk = t.link[n];
        if (lk.y > 0) continue;
        if (lk.x < 0 || static_cast<int64_t>(lk.x) - lk.y > nbodies) { raise_error(err, kErrIndex); continue; }
        // the parent and its record before the moments' stores
        const int q = t.parent[n];
        const int4 rec = q >= 0 && q < ninternal ? __ldg(t.climb + q) : make_int4(0, 0, 0, 0);
        leaf_moments(bd, keys, sysid, cubes, base, P, t, accurate, n, lk.x, -lk.y);
        if (q < 0) continue;
        if (q >= ninternal) { raise_error(err, kErrIndex); continue; }
        if (!climb_record_check(nodes, rec, err)) continue;
        if (atomicAdd(t.counter + q, 1) == rec.z - 1) {
            t.counter[q] = 0;
            const unsigned long long slot = atomicAdd(t.work + kWorkReady, 1ull);
            if (slot < static_cast<unsigned long long>(t.cap_int)) t.ready[slot] = q;
            else raise_error(err, kErrIndex);
        }
    }
}

// Climb: one thread per ready parent combines its (leaf) children and
// climbs on; the parents' arrival counters already hold their leaf children.
//
// Bound by the longest chain of levels, each an arrival, a round trip for the
// children and the combination: all the children's records are in flight at
// once (247 registers, 126 in the reference's physics, in blocks of one warp;
// chunks of two or four children needed two to four round trips a level), and
// the cell's centre, half-width and parent come from the child-search pass instead of a descent
// from the key.  16,384 bodies: build 0.158 -> 0.134 ms; 65,536 bodies with one
// body per leaf 0.260 -> 0.223 ms; 1,048,576 such 0.67 -> 0.60 ms; 16.7 M bodies
// 2.86 -> 2.81 ms.
constexpr int kClimbThreads = 32;
template <bool ACCURATE>
__global__ void __launch_bounds__(kClimbThreads, 8)
upward_climb_kernel(Params P, Tree t, int* err) {
    if (*err & kErrAbort) return;
    const int64_t nodes = t.counts[1];
    const int64_t ninternal = t.counts[0];
    const int64_t listed = static_cast<int64_t>(t.work[kWorkReady]);
    const int64_t nready = listed < t.cap_int ? listed : t.cap_int;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nready;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int q = t.ready[i];
        if (q < 0) { raise_error(err, kErrIndex); continue; }
        climb_from<ACCURATE>(q, P, t, nodes, ninternal, err);
    }
}
}  // namespace

int64_t tree_work_words(int64_t n, int64_t cap_int) {
    return kWorkStatus + n / kCellTile + 1 + cap_int / kChildThreads + 1;
}

cudaError_t build_tree(const uint64_t* keys, int64_t n, const Bodies& bd, const int32_t* sysid,
                       const Systems& sys, const int64_t* d_offsets, const Params& P, Tree& t, int sm_count, int* err,
                       cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    const int leaf_cap = P.physics == NEXT_PHYSICS_REFERENCE ? 1 : P.leaf_cap;
    const int group_cap = P.group_cap < leaf_cap ? leaf_cap : P.group_cap;
    const int32_t* sid = sys.n > 1 ? sysid : nullptr;
    const int64_t* offs = sys.n > 1 ? d_offsets : nullptr;
    cudaError_t e = cudaMemsetAsync(t.work, 0, sizeof(unsigned long long) * tree_work_words(n, t.cap_int), st);
    if (e != cudaSuccess) return e;
    const unsigned tiles = static_cast<unsigned>((n + kCellTile - 1) / kCellTile);
    cells_kernel<<<tiles, kCellThreads, 0, st>>>(keys, n, sys.base, sys.levels, leaf_cap, t, err);
    const int64_t itiles = (t.cap_int + kChildThreads - 1) / kChildThreads;
    const int64_t resident = 4 * static_cast<int64_t>(sm_count);
    const int64_t status_at = kWorkStatus + n / kCellTile + 1;
    internal_kernel<<<static_cast<unsigned>(itiles < resident ? (itiles ? itiles : 1) : resident), kChildThreads, 0, st>>>(
        keys, n, sid, offs, sys.n, sys.base, sys.levels, leaf_cap, group_cap, status_at, t, err);
    const unsigned cblocks = static_cast<unsigned>((t.cap_int + threads - 1) / threads);
    children_kernel<<<cblocks < 4096u ? (cblocks ? cblocks : 1u) : 4096u, threads, 0, st>>>(
        keys, t.dlev, t.nint, sid, offs, sys.cube, n, sys.n, sys.base, sys.levels, leaf_cap, group_cap,
        P.physics == NEXT_PHYSICS_ACCURATE, t, err);
    const unsigned ublocks = static_cast<unsigned>((t.cap_node + threads - 1) / threads);
    Params Pu = P;
    const unsigned ugrid = ublocks < 8192u ? ublocks : 8192u;
    const bool acc = P.physics == NEXT_PHYSICS_ACCURATE;
    if (acc)
        upward_leaves_kernel<true><<<ugrid, threads, 0, st>>>(bd, n, keys, sid, sys.cube, sys.base, Pu, t, err);
    else
        upward_leaves_kernel<false><<<ugrid, threads, 0, st>>>(bd, n, keys, sid, sys.cube, sys.base, Pu, t, err);
    const int64_t cl = (t.cap_int + kClimbThreads - 1) / kClimbThreads;
    const unsigned cgrid = static_cast<unsigned>(cl < 8192 ? (cl ? cl : 1) : 8192);
    if (acc) upward_climb_kernel<true><<<cgrid, kClimbThreads, 0, st>>>(Pu, t, err);
    else upward_climb_kernel<false><<<cgrid, kClimbThreads, 0, st>>>(Pu, t, err);
    count_launches(5);
    return cudaGetLastError();
}

}  // namespace nb
