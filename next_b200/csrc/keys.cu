// Root cube and octant keys.
//
// Root cube: bounding box of the bodies, centre = box middle, half-width =
// half the largest extent (1 if that is <= 0) -- src/gravity/step.h:69-100.
// Octant key: the path the reference's insertion takes for a body, i.e. at
// every level the octant (x>cx) + 2(y>cy) + 4(z>cz) against the cell centre,
// then the child centre = centre +/- half of the half-width
// (src/gravity/octree.h:49-64).  Computing the descent with the same FP64
// operations makes the key's leading digits equal the reference tree path
// bit for bit, so a tree built from sorted keys has the reference topology.
//
// Memory bound: 24 B of positions read + 12 B of key/index written per body.
#include "box.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "sort_digits.cuh"

namespace nb {

namespace {

// One system: grid-wide reduction; the last block to finish folds the block
// partials and writes the cube, then re-arms the ticket for the next launch.
__global__ void __launch_bounds__(kBoxThreads)
root_cube_kernel(const double* __restrict__ x, const double* __restrict__ y,
                 const double* __restrict__ z, int64_t n, double* __restrict__ partial,
                 unsigned int* ticket, double4* cube) {
    double lo[3] = {1e30, 1e30, 1e30}, hi[3] = {-1e30, -1e30, -1e30};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double px = x[i], py = y[i], pz = z[i];
        lo[0] = fmin(lo[0], px); hi[0] = fmax(hi[0], px);
        lo[1] = fmin(lo[1], py); hi[1] = fmax(hi[1], py);
        lo[2] = fmin(lo[2], pz); hi[2] = fmax(hi[2], pz);
    }
    block_minmax3(lo, hi);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        for (int a = 0; a < 3; ++a) { partial[6 * blockIdx.x + a] = lo[a]; partial[6 * blockIdx.x + 3 + a] = hi[a]; }
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double l2[3] = {1e30, 1e30, 1e30}, h2[3] = {-1e30, -1e30, -1e30};
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int a = 0; a < 3; ++a) {
            l2[a] = fmin(l2[a], __ldcg(partial + 6 * b + a));
            h2[a] = fmax(h2[a], __ldcg(partial + 6 * b + 3 + a));
        }
    block_minmax3(l2, h2);
    if (threadIdx.x == 0) {
        *cube = cube_from_box(l2, h2);
        *ticket = 0u;
    }
}

// The descent itself: the reference's comparisons and centres, level by level.
__device__ __forceinline__ uint64_t descend(double px, double py, double pz, const double4& c, int levels) {
    double cx = c.x, cy = c.y, cz = c.z, h = c.w;
    uint64_t key = 0;
    for (int l = 1; l <= levels; ++l) {
        const bool bx = px > cx, by = py > cy, bz = pz > cz;
        key = (key << 3) | static_cast<uint64_t>(bx) | (static_cast<uint64_t>(by) << 1) |
              (static_cast<uint64_t>(bz) << 2);
        const double hs = h * 0.5;
        cx = cx + (bx ? hs : -hs);
        cy = cy + (by ? hs : -hs);
        cz = cz + (bz ? hs : -hs);
        h = hs;
    }
    return key;
}

// Bits of v (at most 11) moved three apart.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
    v = (v | (v << 16)) & 0x070000ffu;
    v = (v | (v << 8)) & 0x0700f00fu;
    v = (v | (v << 4)) & 0x430c30c3u;
    return (v | (v << 2)) & 0x49249249u;
}

// One axis by fixed point: the number u of the finest cell that holds p, when
// the descent is sure to agree.  Every centre the descent compares with is a
// cell boundary up to its roundings, each at most r = 2^-53 (|centre| + half)
// and at most 21 of them.  In units of the finest cell, 2 half / 2^levels,
// that is at most 2^(levels-53) 11 (|centre| + half) / half; computing y below
// adds at most 2^(levels-53) ((|centre| + half) / half + 6).  So a fraction of
// y further than 2^(levels-53) 32 ((|centre| + half) / half + 1) = `margin` from
// 0 and 1 decides every level.
__device__ __forceinline__ bool cell_number(double p, double lo, double scale, double margin, double cells,
                                            uint32_t* u) {
    const double y = (p - lo) * scale;
    const double f = floor(y);
    const double frac = y - f;
    *u = static_cast<uint32_t>(__double2ll_rz(f));
    return y >= 0.0 && y < cells && frac >= margin && frac <= 1.0 - margin;
}

// Two bodies per thread and round (more independent work in flight per thread).
// A body's cell number per axis gives its digits at once; the few bodies too
// near a cell boundary to be sure descend level by level.  The block also
// counts the digits of its keys for the sort that follows (hist), which saves
// that pass over the keys.
//
// The descent for every body was bound by its chain of FP64 steps: 418 us at 16.7 M
// bodies and 21 levels, 31 us at 1,048,576; this is 200 us and 15 us, where the
// 36 B per body take 91 us and 6 us.  Moving the pairs as 16-byte vectors
// changed nothing.
constexpr int kKeysPerThread = 2;
constexpr int kKeyThreads = 256;
constexpr int64_t kCountingBlocks = 740;    // 296 to 1,480 measured the same
__global__ void __launch_bounds__(kKeyThreads)
keys_kernel(const double* __restrict__ x, const double* __restrict__ y,
            const double* __restrict__ z, const int32_t* __restrict__ sysid, int64_t n,
            const double4* __restrict__ cubes, int base, int levels,
            uint64_t* __restrict__ keys, uint32_t* __restrict__ idx, int key_bits, uint32_t* __restrict__ hist) {
    __shared__ uint32_t local[8 * kSortRadix];
    const int passes = hist ? (key_bits + 7) / 8 : 0;
    for (int i = threadIdx.x; i < passes * kSortRadix; i += kKeyThreads) local[i] = 0;
    __syncthreads();
    const int64_t stride = static_cast<int64_t>(gridDim.x) * kKeyThreads * kKeysPerThread;
    const double cells = static_cast<double>(1u << levels);        // levels <= 21
    int held = -1;                                                 // the system the values below belong to
    double4 c = make_double4(0.0, 0.0, 0.0, 0.0);
    double scale = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
    for (int64_t i0 = (blockIdx.x * (int64_t)kKeyThreads + threadIdx.x) * kKeysPerThread; i0 < n; i0 += stride) {
#pragma unroll
        for (int u = 0; u < kKeysPerThread; ++u) {
            const int64_t i = i0 + u;
            if (i >= n) break;
            const int s = sysid ? sysid[i] : 0;
            const double px = x[i], py = y[i], pz = z[i];
            if (s != held) {
                held = s;
                c = cubes[s];
                scale = 0.5 * cells / c.w;
                const double unit = 32.0 * cells * 0x1p-53;
                mx = unit * ((fabs(c.x) + c.w) / c.w + 1.0);
                my = unit * ((fabs(c.y) + c.w) / c.w + 1.0);
                mz = unit * ((fabs(c.z) + c.w) / c.w + 1.0);
            }
            uint32_t ux, uy, uz;
            const bool sx = cell_number(px, c.x - c.w, scale, mx, cells, &ux);
            const bool sy = cell_number(py, c.y - c.w, scale, my, cells, &uy);
            const bool sz = cell_number(pz, c.z - c.w, scale, mz, cells, &uz);
            uint64_t digits;
            if (sx && sy && sz) {
                const uint32_t lo = spread3(ux & 0x3ffu) | (spread3(uy & 0x3ffu) << 1) | (spread3(uz & 0x3ffu) << 2);
                const uint64_t hx = spread3(ux >> 10), hy = spread3(uy >> 10), hz = spread3(uz >> 10);
                digits = lo | ((hx | (hy << 1) | (hz << 2)) << 30);
            } else {
                digits = descend(px, py, pz, c, levels);
            }
            const uint64_t key = (base < 64 ? (static_cast<uint64_t>(s) << base) : 0ull) | (digits << (base - 3 * levels));
            keys[i] = key;
            idx[i] = static_cast<uint32_t>(i);
            if (hist) count_digits(key, key_bits, local);
        }
    }
    if (hist) {
        __syncthreads();
        add_digit_counts<kKeyThreads>(local, passes, hist);
    }
}

}  // namespace

cudaError_t launch_root_cubes(const Bodies& b, const int32_t* sysid, int64_t n, const Systems& sys, double* partial,
                              int partial_blocks, unsigned int* ticket, cudaStream_t st) {
    if (sys.n != 1) return launch_system_boxes(b, sysid, n, sys, nullptr, nullptr, ticket, st);
    int blocks = static_cast<int>((n + kBoxThreads - 1) / kBoxThreads);
    if (blocks > partial_blocks) blocks = partial_blocks;
    if (blocks < 1) blocks = 1;
    root_cube_kernel<<<blocks, kBoxThreads, 0, st>>>(b.x, b.y, b.z, n, partial, ticket, sys.cube);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_keys(const Bodies& b, const int32_t* sysid, int64_t n, const Systems& sys,
                        uint64_t* keys, uint32_t* idx, int key_bits, uint32_t* hist, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    // with counts, fewer and longer blocks: each adds its counts to the sort's once
    const int64_t all = (n + kKeyThreads * kKeysPerThread - 1) / (kKeyThreads * kKeysPerThread);
    const unsigned blocks = static_cast<unsigned>(hist && all > kCountingBlocks ? kCountingBlocks : all);
    keys_kernel<<<blocks, kKeyThreads, 0, st>>>(b.x, b.y, b.z, sys.n > 1 ? sysid : nullptr, n, sys.cube, sys.base,
                                                sys.levels, keys, idx, key_bits, hist);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace nb
