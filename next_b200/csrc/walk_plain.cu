// Plain FP64 force walks: every body opens the tree by its own distance.
//
// Reference physics: one thread per target body (several lanes in small
// systems), depth-first over the tree in octant order 0..7 -- the order bhAccel
// recurses (src/gravity/octree.h:176-178) -- with a per-level (next sibling,
// end) stack instead of recursion, and bhAccel's arithmetic (octree.h:134-173,
// softening.h:21-35) operation for operation.  Accurate physics (Plummer
// softening, full-width opening test, corrected quadrupole): a warp, or eight
// lanes in small systems, per few bodies, one node per lane.
//
// Also: the FP64 direct-summation kernel used to state force errors.
//
// Built with -fmad=false so each + and * rounds on its own, matching the
// reference's x86-64 build (no FMA contraction); the accurate walk's sums use
// fma() explicitly.  cbrt and pow come from CUDA's math library; they may
// differ from the host libm in the last bit.
#include "common.cuh"
#include "fp64_math.cuh"
#include "kernels.cuh"
#include "softening.cuh"

namespace nb {

namespace {

// One accepted node in reference physics, from its separation, mass, softening
// base, dark-matter softening (-1 for bodies it does not apply to) and
// quadrupole: the two addends bhAccel accumulates (src/gravity/octree.h:138-172).
struct RefTerm {
    double mx, my, mz, qx, qy, qz;
};

__device__ __forceinline__ RefTerm ref_term(double nm, double dx, double dy, double dz, double r2, double base,
                                            double dark, const double2& qa, const double2& qb, const double2& qc) {
    const double eps = dmax_like_std(softening_at(base, sqrt(r2 + 1e-20)), dark);
    const double r2s = r2 + eps * eps;
    const double dinv = 1.0 / sqrt(r2s);
    const double inv3 = dinv * dinv * dinv;
    const double fac = 1.0 * nm * inv3;
    const double inv5 = inv3 * (dinv * dinv);
    const double inv7 = inv5 * (dinv * dinv);
    const double q = qa.x * dx * dx + qa.y * dy * dy + qb.x * dz * dz +
                     2.0 * (qb.y * dx * dy + qc.x * dx * dz + qc.y * dy * dz);
    const double qrx = 2.0 * (qa.x * dx + qb.y * dy + qc.x * dz);
    const double qry = 2.0 * (qb.y * dx + qa.y * dy + qc.y * dz);
    const double qrz = 2.0 * (qc.x * dx + qc.y * dy + qb.x * dz);
    RefTerm f;
    f.mx = dx * fac; f.my = dy * fac; f.mz = dz * fac;
    f.qx = 0.5 * (qrx * inv5 - 5.0 * q * inv7 * dx);
    f.qy = 0.5 * (qry * inv5 - 5.0 * q * inv7 * dy);
    f.qz = 0.5 * (qrz * inv5 - 5.0 * q * inv7 * dz);
    return f;
}

__device__ __forceinline__ void add_stats(unsigned long long* stats, unsigned long long pp, unsigned long long pc) {
    for (int o = 16; o > 0; o >>= 1) {
        pp += __shfl_xor_sync(0xffffffffu, pp, o);
        pc += __shfl_xor_sync(0xffffffffu, pc, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (pp) atomicAdd(stats + 0, pp);
        if (pc) atomicAdd(stats + 1, pc);
    }
}

// The reference's opening test, size / dist < theta with dist = sqrt(r2 + 1e-20) (octree.h:153): decided by
// the squares wherever they differ by more than the square root's and the division's rounding could hide, by
// the reference's own operations otherwise.
__device__ __forceinline__ bool ref_opens(const double4& c, double size, double xi, double yi, double zi, double theta,
                                          double theta2, bool squarable) {
    const double dx = c.x - xi, dy = c.y - yi, dz = c.z - zi;
    const double d2 = dx * dx + dy * dy + dz * dz + 1e-20;
    const double s2 = size * size, t2 = theta2 * d2;
    bool near = squarable && s2 > t2 * (1.0 + 1e-14);
    const bool far = squarable && s2 < t2 * (1.0 - 1e-14);
    if (!near && !far) near = !((size / sqrt(d2)) < theta);
    return near;
}

// A listed node's addends for a target at (xi, yi, zi).
__device__ __forceinline__ RefTerm ref_entry(const Tree& t, int64_t nd, bool leaf, double xi, double yi, double zi,
                                             double mi, bool dark, bool stored) {
    const double4 c = t.com[nd];
    const double2 soft = t.soft[2 * nd + 1];               // base and dark softening of the node
    double2 qa = make_double2(0.0, 0.0), qb = qa, qc = qa; // a body has no quadrupole
    const double2* q2 = reinterpret_cast<const double2*>(t.quad64 + 8 * nd);
    if (!leaf) { qa = q2[0]; qb = q2[1]; qc = q2[2]; }
    const double dx = c.x - xi, dy = c.y - yi, dz = c.z - zi;
    const double r2 = dx * dx + dy * dy + dz * dz;
    double sd = -1.0;
    if (dark) sd = stored ? soft.y : softening_dark(t.soft[2 * nd].x, c.w, mi);
    return ref_term(c.w, dx, dy, dz, r2, soft.x, sd, qa, qb, qc);
}

// What the softening of a bucket's bodies takes from their masses alone, computed when the mass changes (mostly
// once: the cube root and the power are most of a bucket's work otherwise).
struct BucketSoftening {
    double mass = -1.0, base = 0.0, dark = -1.0;
    __device__ __forceinline__ void of(double mj, double size, double mi, bool is_dark) {
        if (mj == mass) return;
        mass = mj;
        base = softening_base(size, mj);
        dark = is_dark ? softening_dark(size, mj, mi) : -1.0;
    }
};

// The bodies of a deepest-level bucket act as one-body leaves of its size; added one by one.
__device__ __forceinline__ void ref_bucket(const Bodies& bd, double size, const int2& lk, int64_t self, double xi, double yi,
                                           double zi, double mi, bool dark, double& ax, double& ay, double& az,
                                           unsigned& npp) {
    const double2 zero = make_double2(0.0, 0.0);
    BucketSoftening soft;
    for (int j = lk.x; j < lk.x - lk.y; ++j) {
        const double mj = bd.m[j];
        if (j == self || mj == 0.0) continue;
        const double ex = bd.x[j] - xi, ey = bd.y[j] - yi, ez = bd.z[j] - zi;
        const double e2 = ex * ex + ey * ey + ez * ez;
        soft.of(mj, size, mi, dark);
        const RefTerm f = ref_term(mj, ex, ey, ez, e2, soft.base, soft.dark, zero, zero, zero);
        ax += f.mx; ay += f.my; az += f.mz;
        ax += f.qx; ay += f.qy; az += f.qz;
        ++npp;
    }
}

// Reference physics, opening angles from kRefListTheta on.  The warp alternates
// between two phases: first every lane runs its own depth-first walk with the
// opening tests only, until it has a list of kRefList accepted nodes, stands
// before a bucket or its walk is over; then all lanes evaluate their lists in
// order, and the buckets, which neighbours mostly reach together.  The tests
// diverge but are cheap; the evaluation (two square roots, two divisions, the
// quadrupole) runs with nearly all lanes.
//
// Bound by FP64 latency: bhAccel's operations in bhAccel's order leave a chain
// of four roots and divisions per interaction and no fused multiply-adds.
// 1,048,576 bodies, a fifth of them dark matter: 5.81 -> 3.58 ms per walk (65,536
// bodies 1.05 -> 0.63 ms) against one loop that tested and evaluated a node per
// pass (13.7 of 32 lanes active) and took the node's cube root and the dark
// bodies' power anew in every interaction.  Lists of 8 and 6 blocks per SM (80
// registers) were the fastest of lists of 4-32 at 4-8 blocks; loading a sibling's
// record while its predecessor is tested, or evaluating two entries at once,
// cost more in registers than it hid (3.9-4.4 ms).  Buckets: 300,000 bodies with
// radii log-uniform over 2^-20 .. 1, 57 -> 24 ms against evaluating a bucket in the
// middle of the tests, with a cube root per body of it (the plain loop: 47 ms).
constexpr int kRefThreads = 128;
constexpr int kRefList = 8;
constexpr unsigned kRefLeaf = 0x80000000u;                         // list entry: the node is a single body

__global__ void __launch_bounds__(kRefThreads, 6)
walk_reference_kernel(Bodies bd, const int32_t* __restrict__ sysid, int64_t n, Tree t, Params P,
                      unsigned long long* stats, int* err) {
    if (__any_sync(0xffffffffu, *err & kErrAbort)) return;       // whole warps: other blocks may be raising bits
    __shared__ unsigned list[kRefList][kRefThreads];
    const int64_t nodes = t.counts[1];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool active = i < n && i >= P.own_lo && i < P.own_hi;
    const int64_t ii = active ? i : 0;
    const double xi = bd.x[ii], yi = bd.y[ii], zi = bd.z[ii], mi = bd.m[ii];
    const bool dark = bd.type[ii] == 1;
    // the mass whose dark-matter softening the upward pass stored per node
    const bool stored = dark && mi == *t.dark_mass;
    double ax = 0.0, ay = 0.0, az = 0.0;
    unsigned npp = 0, npc = 0;
    const double theta = P.theta, theta2 = theta * theta;
    int2 stack[kMaxLevel + 2];
    int sp = 0;
    int cur = sysid ? sysid[ii] : 0, end = active ? cur + 1 : cur;
    while (__any_sync(0xffffffffu, cur < end || sp > 0)) {
        int cnt = 0;
        while (cnt < kRefList) {
            while (cur >= end && sp > 0) {
                --sp;
                cur = stack[sp].x;
                end = stack[sp].y;
            }
            if (cur >= end) break;                                 // the walk is over
            const int k = cur++;
            if (k < 0 || k >= nodes) { raise_error(err, kErrIndex); cur = end; sp = 0; break; }
            const double4 c = t.com[k];
            const double2 head = t.soft[2 * static_cast<int64_t>(k)];    // half-width and link
            const double size = head.x;
            const int2 lk = make_int2(__double2loint(head.y), __double2hiint(head.y));
            if (c.w == 0.0) continue;
            const bool leaf = lk.y <= 0;
            if (leaf ? (lk.x < 0 || static_cast<int64_t>(lk.x) - lk.y > n) : (sp >= kMaxLevel + 1)) {
                raise_error(err, leaf ? kErrIndex : kErrStack);
                cur = end; sp = 0;
                break;
            }
            if (!leaf) {
                if (ref_opens(c, size, xi, yi, zi, theta, theta2, P.theta_squarable)) {
                    stack[sp++] = make_int2(cur, end);
                    cur = lk.x;
                    end = lk.x + lk.y;
                } else {
                    list[cnt++][threadIdx.x] = static_cast<unsigned>(k);
                }
            } else if (lk.y == -1) {
                if (lk.x != i) list[cnt++][threadIdx.x] = static_cast<unsigned>(k) | kRefLeaf;   // not its own leaf (octree.h:135)
            } else {
                --cur;                                             // a bucket: behind the listed nodes, with the other lanes' ones
                break;
            }
        }
        __syncwarp();
        for (int e = 0; e < cnt; ++e) {
            const unsigned entry = list[e][threadIdx.x];
            const bool leaf = entry & kRefLeaf;
            const RefTerm f = ref_entry(t, entry & ~kRefLeaf, leaf, xi, yi, zi, mi, dark, stored);
            ax += f.mx; ay += f.my; az += f.mz;
            ax += f.qx; ay += f.qy; az += f.qz;
            if (leaf) ++npp; else ++npc;
        }
        __syncwarp();
        if (cnt < kRefList && cur < end) {                         // stopped before a bucket
            const double2 head = t.soft[2 * static_cast<int64_t>(cur++)];
            ref_bucket(bd, head.x, make_int2(__double2loint(head.y), __double2hiint(head.y)), i, xi, yi, zi, mi, dark, ax, ay, az,
                       npp);
        }
        __syncwarp();
    }
    if (active) {
        bd.ax[i] = ax; bd.ay[i] = ay; bd.az[i] = az;
        if (bd.pot) bd.pot[i] = 0.0;
    }
    add_stats(stats, npp, npc);
}

// Reference physics, smaller opening angles: one loop that tests a node and, if
// it is accepted, evaluates it at once.  Lists set the lanes' places in the tree
// apart, and then a node is read by one lane instead of by all that need it: that
// costs the more, the more nodes a warp's bodies have in common.  Walks of Plummer
// spheres of 1,000,000 / 300,000 bodies, this loop against lists: theta 0.1 461 /
// 131 ms against 543 / 152, 0.2 67.3 / 21.0 against 72.7 / 22.8, 0.3 22.7 / 7.27 against 23.0 / 7.37,
// 0.4 9.60 / 3.18 against 9.40 / 3.08, 0.5 6.16 / 2.00 against 6.00 / 1.95.
constexpr double kRefListTheta = 0.4;

__global__ void __launch_bounds__(kRefThreads, 6)
walk_reference_small_theta_kernel(Bodies bd, const int32_t* __restrict__ sysid, int64_t n, Tree t, Params P,
                                  unsigned long long* stats, int* err) {
    if (__any_sync(0xffffffffu, *err & kErrAbort)) return;       // whole warps: other blocks may be raising bits
    const int64_t nodes = t.counts[1];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool active = i < n && i >= P.own_lo && i < P.own_hi;
    unsigned npp = 0, npc = 0;
    if (active) {
        const double xi = bd.x[i], yi = bd.y[i], zi = bd.z[i], mi = bd.m[i];
        const bool dark = bd.type[i] == 1;
        const bool stored = dark && mi == *t.dark_mass;
        const double theta = P.theta, theta2 = theta * theta;
        double ax = 0.0, ay = 0.0, az = 0.0;
        int2 stack[kMaxLevel + 2];
        int sp = 0;
        int cur = sysid ? sysid[i] : 0, end = cur + 1;
        for (;;) {
            if (cur >= end) {
                if (sp == 0) break;
                --sp;
                cur = stack[sp].x;
                end = stack[sp].y;
                continue;
            }
            const int k = cur++;
            if (k < 0 || k >= nodes) { raise_error(err, kErrIndex); break; }
            const double4 c = t.com[k];
            const double2 head = t.soft[2 * static_cast<int64_t>(k)];      // half-width and link
            const double2 soft = t.soft[2 * static_cast<int64_t>(k) + 1];  // softening base, of dark bodies
            const double2* q2 = reinterpret_cast<const double2*>(t.quad64 + 8 * static_cast<int64_t>(k));
            const double size = head.x;
            const int2 lk = make_int2(__double2loint(head.y), __double2hiint(head.y));
            if (c.w == 0.0) continue;
            const bool leaf = lk.y <= 0;
            if (leaf ? (lk.x < 0 || static_cast<int64_t>(lk.x) - lk.y > n) : (sp >= kMaxLevel + 1)) {
                raise_error(err, leaf ? kErrIndex : kErrStack);
                break;
            }
            if (leaf && lk.y == -1 && lk.x == i) continue;         // its own leaf (octree.h:135)
            if (leaf && lk.y < -1) {
                ref_bucket(bd, size, lk, i, xi, yi, zi, mi, dark, ax, ay, az, npp);
                continue;
            }
            if (!leaf && ref_opens(c, size, xi, yi, zi, theta, theta2, P.theta_squarable)) {
                stack[sp++] = make_int2(cur, end);
                cur = lk.x;
                end = lk.x + lk.y;
                continue;
            }
            double2 qa = make_double2(0.0, 0.0), qb = qa, qc = qa;
            if (!leaf) { qa = q2[0]; qb = q2[1]; qc = q2[2]; }
            const double dx = c.x - xi, dy = c.y - yi, dz = c.z - zi;
            const double r2 = dx * dx + dy * dy + dz * dz;
            double sd = -1.0;
            if (dark) sd = stored ? soft.y : softening_dark(size, c.w, mi);
            const RefTerm f = ref_term(c.w, dx, dy, dz, r2, soft.x, sd, qa, qb, qc);
            ax += f.mx; ay += f.my; az += f.mz;
            ax += f.qx; ay += f.qy; az += f.qz;
            if (leaf) ++npp; else ++npc;
        }
        bd.ax[i] = ax; bd.ay[i] = ay; bd.az[i] = az;
        if (bd.pot) bd.pot[i] = 0.0;
    }
    add_stats(stats, npp, npc);
}

// Reference physics with 8, 16 or 32 lanes per body, for small systems: the
// lanes test the siblings of an opened cell at once and evaluate as many
// accepted nodes at once as there are lanes; the addends go through shared
// memory to the lanes that own the sums and are added there one by one in
// depth-first order, so every bit is that of the walk above.
//
// Small systems are bound by the latency of one body's walk, a chain of some
// hundred tests and interactions of about a microsecond each, whatever the
// number of bodies.  Walk of 256 bodies 157 -> 45 us, 1,000 264 -> 54 us, 4,096
// 377 -> 93 us, 16,384 460 -> 187 us, 32,768 485 -> 364 us (Plummer spheres).
// More lanes are better while all warps are resident: 2,048 bodies 72 us with 32
// lanes, 86 with 16 and 108 with 8; 4,096 129, 100 and 121 us; 8,192 210, 179 and
// 141 us.  Eight lanes at 5, 6 and 7 blocks per SM (96, 80 and 72 registers):
// 8,192 bodies 135, 152 and 159 us, 14,000 218, 166 and 186, 16,384 236, 230 and
// 206, 40,960 491, 449 and 499 us.  Above 49,152 bodies (550 us against 562 us;
// 57,344: 575 us against 619 us) the walk above has warps enough and takes fewer
// instructions, which bind there.  Those comparisons were made with the buckets
// evaluated by every lane for itself; a bucket's bodies spread over the lanes
// need fewer registers, and all of these walks take 5-8% less (49,000 bodies
// 541 -> 506 us); with 5,000 of 20,000 bodies at one place 4.3 -> 0.73 ms.
//
// The numbers of lanes and blocks are a table for the 148 SMs of this GPU and
// all bodies of the launch; on another number of SMs, or where a rank walks only
// its share of the bodies, another entry may be the fastest.
//
// A sub-warp's walk: the group being tested, or what is left of one behind its
// first opened cell -- (first sibling, masks of accepted, opened, single-body
// and bucket siblings) -- with the levels above on a stack.  Accepted siblings
// before the next opened one join a ring of listed nodes.
constexpr int kWideRing = 64;
constexpr int64_t kWideMax = 49152;
template <int LANES>
struct WideShared {
    double term[6][33];                                            // mass and quadrupole addends per lane
    int2 stack[32 / LANES][kMaxLevel + 2];
    unsigned ring[32 / LANES][kWideRing];
};

template <int LANES, int MINB>
__global__ void __launch_bounds__(kRefThreads, MINB)
walk_reference_wide_kernel(Bodies bd, const int32_t* __restrict__ sysid, int64_t n, Tree t, Params P,
                           unsigned long long* stats, int* err) {
    if (__any_sync(0xffffffffu, *err & kErrAbort)) return;       // whole warps: other blocks may be raising bits
    __shared__ WideShared<LANES> shared[kRefThreads / 32];
    WideShared<LANES>& S = shared[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, sub = lane / LANES, sl = lane % LANES;
    const unsigned nodes = static_cast<unsigned>(t.counts[1]), nbodies = static_cast<unsigned>(n);
    const int64_t i = (blockIdx.x * static_cast<int64_t>(kRefThreads / 32) + (threadIdx.x >> 5)) * (32 / LANES) + sub;
    const bool active = i < n && i >= P.own_lo && i < P.own_hi;
    const int64_t ii = active ? i : 0;
    const int self = static_cast<int>(i);
    unsigned npp = 0, npc = 0;
    const double xi = bd.x[ii], yi = bd.y[ii], zi = bd.z[ii], mi = bd.m[ii];
    const bool dark = bd.type[ii] == 1;
    const bool stored = dark && mi == *t.dark_mass;
    const double theta = P.theta, theta2 = theta * theta;
    double sum = 0.0;                                              // lanes 0..2 of a body: x, y, z
    int first = sysid ? sysid[ii] : 0, count = active ? 1 : 0;     // siblings to test
    unsigned rest = 0;                                             // or masks of tested ones, 8 bits each:
    int sp = 0, head = 0, cnt = 0, bucket = -1;                    // accepted, opened, single bodies, buckets
    for (;;) {
        for (;;) {
            const bool open_work = (count > 0 || rest != 0 || sp > 0) && bucket < 0;
            if (!__any_sync(0xffffffffu, open_work && cnt < LANES)) break;
            const bool go = open_work && cnt <= kWideRing - 8;
            const bool fresh = go && count > 0;
            if (go && !fresh && rest == 0) {
                --sp;
                const int2 item = S.stack[sub][sp];
                first = item.x;
                rest = static_cast<unsigned>(item.y);
            }
            __syncwarp();
            bool accept = false, leaf = false, open = false, many = false;
            int2 lk = make_int2(0, 0);
            const int k = first + sl;
            if (fresh && sl < count) {
                if (static_cast<unsigned>(k) >= nodes) {
                    raise_error(err, kErrIndex);
                } else {
                    const double4 c = t.com[k];
                    const double2 nh = t.soft[2 * static_cast<int64_t>(k)];    // half-width and link
                    lk = make_int2(__double2loint(nh.y), __double2hiint(nh.y));
                    leaf = lk.y <= 0;
                    // children lie behind their parent in the tree, so a walk ends
                    if (leaf ? (lk.x < 0 || static_cast<unsigned>(lk.x) - static_cast<unsigned>(lk.y) > nbodies)
                             : (lk.x <= k || lk.y > 8)) {
                        if (c.w != 0.0) raise_error(err, kErrIndex);
                    } else if (c.w != 0.0) {
                        many = leaf && lk.y != -1;
                        open = many || (!leaf && ref_opens(c, nh.x, xi, yi, zi, theta, theta2, P.theta_squarable));
                        accept = !open && !(leaf && lk.x == self);    // not its own leaf (octree.h:135)
                    }
                }
            }
            const int shift = LANES * sub;
            const unsigned am = __ballot_sync(0xffffffffu, accept) >> shift & 0xffu;
            const unsigned om = __ballot_sync(0xffffffffu, open) >> shift & 0xffu;
            const unsigned lm = __ballot_sync(0xffffffffu, accept && leaf) >> shift & 0xffu;
            const unsigned bm = __ballot_sync(0xffffffffu, many) >> shift & 0xffu;
            if (fresh) { rest = am | om << 8 | lm << 16 | bm << 24; count = 0; }
            const unsigned acc = rest & 0xffu, opened = rest >> 8 & 0xffu;
            const int j = opened ? __ffs(static_cast<int>(opened)) - 1 : 8;
            const int2 lj = make_int2(__shfl_sync(0xffffffffu, lk.x, shift + (j & 7)),
                                      __shfl_sync(0xffffffffu, lk.y, shift + (j & 7)));
            if (go) {
                const unsigned pre = acc & ((1u << j) - 1u);
                if (pre >> sl & 1u)
                    S.ring[sub][(head + cnt + __popc(pre & ((1u << sl) - 1u))) % kWideRing] =
                        static_cast<unsigned>(k) | (rest >> (16 + sl) & 1u ? kRefLeaf : 0u);
                cnt += __popc(pre);
                if (j == 8) {
                    rest = 0;
                } else {
                    const unsigned later = 0xffu & ~((2u << j) - 1u);
                    const unsigned left = rest & (later | later << 8 | later << 16 | later << 24);
                    const bool is_bucket = rest >> (24 + j) & 1u;
                    const int nd = first + j;
                    if (left & 0xffffu) {
                        if (sp < kMaxLevel + 2) {
                            if (sl == 0) S.stack[sub][sp] = make_int2(first, static_cast<int>(left));
                            ++sp;
                        } else if (sl == 0) {
                            raise_error(err, kErrStack);
                        }
                    }
                    rest = 0;
                    if (is_bucket) {
                        bucket = nd;                               // its bodies follow the listed nodes
                    } else {
                        int2 ch = lj;
                        if (!fresh) {
                            const double2 nh = t.soft[2 * static_cast<int64_t>(nd)];
                            ch = make_int2(__double2loint(nh.y), __double2hiint(nh.y));
                        }
                        first = ch.x;
                        count = ch.y;
                    }
                }
            }
            __syncwarp();
        }
        const int take = min(cnt, LANES);
        if (!__any_sync(0xffffffffu, take > 0 || bucket >= 0)) break;
        if (sl < take) {
            const unsigned entry = S.ring[sub][(head + sl) % kWideRing];
            const bool leaf = entry & kRefLeaf;
            const RefTerm f = ref_entry(t, entry & ~kRefLeaf, leaf, xi, yi, zi, mi, dark, stored);
            S.term[0][lane] = f.mx; S.term[1][lane] = f.my; S.term[2][lane] = f.mz;
            S.term[3][lane] = f.qx; S.term[4][lane] = f.qy; S.term[5][lane] = f.qz;
            if (leaf) ++npp; else ++npc;
        }
        __syncwarp();
        if (sl < 3) {
            const double* m = &S.term[sl][sub * LANES];
            const double* q = &S.term[3 + sl][sub * LANES];
#pragma unroll
            for (int e = 0; e < LANES; ++e) {
                if (e < take) {
                    sum += m[e];
                    sum += q[e];
                }
            }
        }
        __syncwarp();
        head += take;
        cnt -= take;
        // Deepest-level buckets, behind their sub-warps' listed nodes: the bodies act as one-body leaves of that
        // size, as many at once as there are lanes.
        const bool at_bucket = bucket >= 0 && cnt == 0;
        if (__any_sync(0xffffffffu, at_bucket)) {
            double size = 0.0;
            int from = 0, bodies = 0;
            if (at_bucket) {
                const double2 nh = t.soft[2 * static_cast<int64_t>(bucket)];
                size = nh.x;
                from = __double2loint(nh.y);
                bodies = -__double2hiint(nh.y);
                bucket = -1;
            }
            const double2 zero = make_double2(0.0, 0.0);
            BucketSoftening soft;
            for (int o = 0; __any_sync(0xffffffffu, o < bodies); o += LANES) {
                const int b = from + o + sl;
                bool use = false;
                if (o + sl < bodies) {
                    const double mj = bd.m[b];
                    use = b != self && mj != 0.0;
                    if (use) {
                        const double ex = bd.x[b] - xi, ey = bd.y[b] - yi, ez = bd.z[b] - zi;
                        const double e2 = ex * ex + ey * ey + ez * ez;
                        soft.of(mj, size, mi, dark);
                        const RefTerm f = ref_term(mj, ex, ey, ez, e2, soft.base, soft.dark, zero, zero, zero);
                        S.term[0][lane] = f.mx; S.term[1][lane] = f.my; S.term[2][lane] = f.mz;
                        S.term[3][lane] = f.qx; S.term[4][lane] = f.qy; S.term[5][lane] = f.qz;
                        ++npp;
                    }
                }
                const unsigned used = __ballot_sync(0xffffffffu, use) >> (LANES * sub);
                __syncwarp();
                if (sl < 3) {
                    const double* m = &S.term[sl][sub * LANES];
                    const double* q = &S.term[3 + sl][sub * LANES];
#pragma unroll
                    for (int e = 0; e < LANES; ++e) {
                        if (used >> e & 1u) {
                            sum += m[e];
                            sum += q[e];
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    if (active) {
        if (sl < 3) (sl == 0 ? bd.ax : sl == 1 ? bd.ay : bd.az)[i] = sum;
        if (sl == 3 && bd.pot) bd.pot[i] = 0.0;
    }
    add_stats(stats, npp, npc);
}

// Accurate physics.  One warp walks the tree for W consecutive bodies (in key
// order, so they lie close together).  A stack entry is a node and the mask of
// the bodies that opened its parent; each round pops up to 32 nodes, one per
// lane, and every lane tests and evaluates its node against the masked bodies
// in turn, with the node's record in registers.  Each lane sums its own share
// of every body's force; the shares are folded once, at the end.
//
// A thread per body read every node's record through 32 scattered lanes (L1
// data wavefronts at 87-93% of their peak, 17 of 32 lanes active); here a record
// is read once for W bodies, mostly with its siblings beside it, and small
// systems have 1 / W of a warp per body instead of 1 / 32.  1,048,576 bodies
// (theta 0.5, one body per leaf): 21.7 -> 8.3 ms per walk, 16,384 bodies 1.95 ->
// 0.21 ms.  Bound by the issue of the FP64 chains and what surrounds them (62%
// of issue slots).  The targets' coordinates lie in shared memory and a node
// that gives no force is switched off by its inverse distance alone: with the
// coordinates in registers and a select per component the loop had room for
// four bodies (9.25 ms).  W = 7: the bodies of a warp open different cells, so a
// larger W spends more lanes on nodes few of them want (8: 8.4 ms, 9: 9.0 ms)
// and a smaller one reads and tests more nodes per body (6: 8.4 ms, 4: 9.1 ms);
// 128 registers, 4 blocks per SM (5: 9.3 ms and more).
constexpr int kPlainW = 7;
constexpr int kPlainWarps = 4;
constexpr int64_t kSmallSystem = 80;                     // systems of fewer bodies take the walk below
// Popping k nodes adds at most 7 k entries, and one node at a time never more
// than 7 per level: rounds are cut short so that 7 * kMaxLevel + 8 entries stay
// free for a walk that goes on one node at a time.
constexpr int kPlainStack = 640;
constexpr int kPlainReserve = 7 * kMaxLevel + 8;
constexpr int kPlainChunk = 16;                          // bodies of an opened leaf appended per lane and turn
constexpr int kPlainList = 32 + 32 * kPlainChunk;
struct PlainShared {
    int2 stack[kPlainStack];                             // node, mask of the bodies that opened its parent
    int2 list[kPlainList];                               // body, mask of the bodies that opened its leaf
    double pos[kPlainW][4];
};

// a target's coordinate, read where it is used: held in registers the targets would cost the loop its overlap
__device__ __forceinline__ double at(const double& v) { return *reinterpret_cast<const volatile double*>(&v); }

template <bool POT>
__global__ void __launch_bounds__(32 * kPlainWarps, 4)
walk_accurate_kernel(Bodies bd, const int64_t* __restrict__ offsets, int nsys, const double4* __restrict__ cubes,
                     int64_t n, Tree t, Params P,
                     unsigned long long* stats, int* err) {
    if (__any_sync(0xffffffffu, *err & kErrAbort)) return;       // whole warps: other blocks may be raising bits
    __shared__ PlainShared shared[kPlainWarps];
    PlainShared& S = shared[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t w = blockIdx.x * (int64_t)kPlainWarps + (threadIdx.x >> 5);
    unsigned npp = 0, npc = 0;
    // Bodies first .. first + W of one system, counted from the system's first body, so that a body's
    // sums do not depend on the systems around it: system s owns the warps from offsets[s] / W + s on.
    int sys = 0;
    int64_t first = w * kPlainW, last = n;
    if (offsets) {
        int top = nsys;
        while (top - sys > 1) {
            const int mid = (sys + top) >> 1;
            if (offsets[mid] / kPlainW + mid <= w) sys = mid;
            else top = mid;
        }
        first = offsets[sys] + (w - (offsets[sys] / kPlainW + sys)) * kPlainW;
        last = offsets[sys + 1] - offsets[sys] < kSmallSystem ? first : offsets[sys + 1];   // small: the walk below
    }
    // a warp with any body of this device's share computes all of its bodies (again so that a body's
    // sums do not depend on the share) and stores the share's
    unsigned bodies = 0, own = 0;
#pragma unroll
    for (int b = 0; b < kPlainW; ++b) {
        if (first + b >= last) continue;
        bodies |= 1u << b;
        if (first + b >= P.own_lo && first + b < P.own_hi) own |= 1u << b;
    }
    if (own) {                                           // warp-uniform
        const unsigned nodes = static_cast<unsigned>(t.counts[1]), nbodies = static_cast<unsigned>(n);
        // Lengths of a system far from 1 are scaled by a power of two, which rounds nothing, so that fifth
        // powers of distances stay in range.
        const int ex = static_cast<int>((__double_as_longlong(cubes[sys].w) >> 52) & 0x7ff) - 1023;
        const bool scaled = ex > 150 || ex < -150;
        const double S1 = scaled ? scalbn(1.0, -ex) : 1.0;
        const double eps2 = (P.eps * S1) * (P.eps * S1);
        double ax[kPlainW], ay[kPlainW], az[kPlainW], pot[kPlainW];
        int sp = 1, pn = 0;
#pragma unroll
        for (int b = 0; b < kPlainW; ++b) {
            const int64_t i = first + b < last ? first + b : first;
            if (lane == b) { S.pos[b][0] = bd.x[i] * S1; S.pos[b][1] = bd.y[i] * S1; S.pos[b][2] = bd.z[i] * S1; }
            ax[b] = ay[b] = az[b] = pot[b] = 0.0;
        }
        if (lane == 0) S.stack[0] = make_int2(sys, static_cast<int>(bodies));
        __syncwarp();
        while (sp > 0 || pn > 0) {
            const int room = (kPlainStack - kPlainReserve - sp) / 7;
            const int nb = min(min(sp, 32), max(room, 1));
            sp -= nb;
            const int2 entry = lane < nb ? S.stack[sp + lane] : make_int2(-1, 0);
            const int node = entry.x;
            unsigned mask = static_cast<unsigned>(entry.y);
            __syncwarp();
            int2 lk = make_int2(0, 0);
            double4 c = make_double4(0.0, 0.0, 0.0, 0.0);
            double2 qa = make_double2(0.0, 0.0), qb = qa, qc = qa, qd = qa;
            if (mask) {
                bool ok = static_cast<unsigned>(node) < nodes;
                if (ok) {
                    // the node's whole record in one round trip
                    lk = __ldg(t.link + node);
                    const double2* c2 = reinterpret_cast<const double2*>(t.com + node);
                    const double2 ca = __ldg(c2), cb = __ldg(c2 + 1);
                    const double2* q2 = reinterpret_cast<const double2*>(t.quad64 + 8 * static_cast<int64_t>(node));
                    qd = __ldg(q2 + 3);
                    if (P.quad) { qa = __ldg(q2); qb = __ldg(q2 + 1); qc = __ldg(q2 + 2); }
                    c = make_double4(ca.x, ca.y, cb.x, cb.y);
                    const unsigned e = static_cast<unsigned>(lk.x) + static_cast<unsigned>(lk.y > 0 ? lk.y : -lk.y);
                    ok = lk.x >= 0 && lk.y <= 8 && e <= (lk.y > 0 ? nodes : nbodies);
                }
                if (!ok) raise_error(err, kErrIndex);
                if (!ok || c.w == 0.0) mask = 0;
            }
            if (scaled) {                                 // warp-uniform
                c.x *= S1; c.y *= S1; c.z *= S1;
                qd.y *= S1;
                qa.x = qa.x * S1 * S1; qa.y = qa.y * S1 * S1; qb.x = qb.x * S1 * S1;
                qb.y = qb.y * S1 * S1; qc.x = qc.x * S1 * S1; qc.y = qc.y * S1 * S1;
            }
            const double rc2 = qd.y * qd.y;
            unsigned opened = 0;
            // no branch in this loop: the bodies' chains of dependent FP64 operations interleave
#pragma unroll
            for (int b = 0; b < kPlainW; ++b) {
                const bool mine = mask >> b & 1u;
                const double dx = c.x - at(S.pos[b][0]), dy = c.y - at(S.pos[b][1]), dz = c.z - at(S.pos[b][2]);
                const double r2 = dx * dx + dy * dy + dz * dz;
                const bool open = mine && r2 < rc2, use = mine && !open;
                opened |= static_cast<unsigned>(open) << b;
                const double r2s = away_from_ends(r2 + eps2);
                const double rinv = use ? rsqrt_fast(r2s) : 0.0;    // zero: no force from this node
                const double rinv2 = rinv * rinv;
                // a = rinv5 ((m r2 + 2.5 d.Q.d rinv2) d - Q d), times G at the end; Q = 0 in monopole walks
                const double qx = fma(qc.x, dz, fma(qb.y, dy, qa.x * dx));
                const double qy = fma(qc.y, dz, fma(qa.y, dy, qb.y * dx));
                const double qz = fma(qb.x, dz, fma(qc.y, dy, qc.x * dx));
                const double q = fma(dz, qz, fma(dy, qy, dx * qx));
                const double rinv5 = rinv * (rinv2 * rinv2);
                const double k = fma(2.5 * q, rinv2, c.w * r2s);
                ax[b] = fma(rinv5, fma(k, dx, -qx), ax[b]);
                ay[b] = fma(rinv5, fma(k, dy, -qy), ay[b]);
                az[b] = fma(rinv5, fma(k, dz, -qz), az[b]);
                if (POT) pot[b] -= fma(0.5 * q, rinv5, c.w * rinv);
            }
            npc += __popc(mask & ~opened & own);
            // children of opened cells -> stack
            const int push = opened && lk.y > 0 ? lk.y : 0;
            int off = 0, total = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t m = __ballot_sync(0xffffffffu, (push >> k) & 1);
                off += __popc(m & lt) << k;
                total += __popc(m) << k;
            }
            if (sp + total > kPlainStack) {              // only a broken tree gets here
                if (lane == 0) raise_error(err, kErrIndex);
                break;
            }
            if (total > 0) {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k < push) S.stack[sp + off + k] = make_int2(lk.x + k, static_cast<int>(opened));
            }
            sp += total;
            // bodies of opened leaves -> list, evaluated 32 at a time, the rest when the walk ends
            int remaining = opened && lk.y < 0 ? -lk.y : 0;
            int src = lk.x;
            for (bool more = __any_sync(0xffffffffu, remaining > 0) || (sp == 0 && pn > 0); more;) {
                const int take = min(remaining, kPlainChunk);
                int o2 = 0, tot = 0;
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const uint32_t m = __ballot_sync(0xffffffffu, (take >> k) & 1);
                    o2 += __popc(m & lt) << k;
                    tot += __popc(m) << k;
                }
                for (int k = 0; k < take; ++k) S.list[pn + o2 + k] = make_int2(src + k, static_cast<int>(opened));
                pn += tot;
                src += take;
                remaining -= take;
                more = __any_sync(0xffffffffu, remaining > 0);
                __syncwarp();
                while (pn >= 32 || (pn > 0 && sp == 0 && !more)) {
                    const int k = pn - 32 > 0 ? pn - 32 : 0;     // from the end: nothing moves
                    const int2 pe = k + lane < pn ? S.list[k + lane] : make_int2(-1, 0);
                    const int j = pe.x;
                    const unsigned jm = static_cast<unsigned>(pe.y);
                    pn = k;
                    double xj = 0.0, yj = 0.0, zj = 0.0, mj = 0.0;
                    if (jm) { xj = bd.x[j]; yj = bd.y[j]; zj = bd.z[j]; mj = bd.m[j]; }
                    if (scaled) { xj *= S1; yj *= S1; zj *= S1; }
#pragma unroll
                    for (int b = 0; b < kPlainW; ++b) {
                        if (!(jm >> b & 1u) || j == first + b) continue;
                        const double dx = xj - at(S.pos[b][0]), dy = yj - at(S.pos[b][1]), dz = zj - at(S.pos[b][2]);
                        const double rinv = rsqrt(dx * dx + dy * dy + dz * dz + eps2);
                        const double mr = mj * rinv, mr3 = mr * rinv * rinv;
                        ax[b] = fma(mr3, dx, ax[b]);
                        ay[b] = fma(mr3, dy, ay[b]);
                        az[b] = fma(mr3, dz, az[b]);
                        if (POT) pot[b] -= mr;
                        npp += own >> b & 1u;
                    }
                    __syncwarp();
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int b = 0; b < kPlainW; ++b) {
            for (int o = 16; o > 0; o >>= 1) {
                ax[b] += __shfl_xor_sync(0xffffffffu, ax[b], o);
                ay[b] += __shfl_xor_sync(0xffffffffu, ay[b], o);
                az[b] += __shfl_xor_sync(0xffffffffu, az[b], o);
                if (POT) pot[b] += __shfl_xor_sync(0xffffffffu, pot[b], o);
            }
            const int64_t i = first + b;
            if (lane == 0 && (own >> b & 1u)) {
                const double g = P.G * S1;
                bd.ax[i] = g * ax[b] * S1; bd.ay[i] = g * ay[b] * S1; bd.az[i] = g * az[b] * S1;
                if (POT) bd.pot[i] = g * pot[b];
            }
        }
    }
    add_stats(stats, npp, npc);
}

// The same for systems of fewer than kSmallSystem bodies, with eight lanes for W
// bodies: such a system's walk has few nodes at a time, and four of them share
// a warp (loops are the warp's, stacks and lists each group's own).
//
// A whole warp leaves most lanes idle there, and batches of many tiny systems
// were slower than by a thread per body: walk of 1,048,576 systems of 4 bodies
// 9.2 ms, here 2.8 ms (a thread per body 0.45 ms), 262,144 of 16 6.1 -> 2.2 (1.5) ms,
// 65,536 of 32 2.7 -> 1.45 (1.31) ms, of 64 5.8 -> 4.4 (4.7) ms, 40,000 of 100 6.1 -> 6.0
// (6.6) ms, 30,000 of 128 6.1 -> 7.0 (7.2) ms.  A small system on its own is bound by
// its rounds instead: 20 bodies 18 -> 21 (38) us, 50 20 -> 39 (88) us, which is why
// the line lies below the one of batches.  It is by a system's own size, so that
// a body's sums stay the same alone and in a batch.
constexpr int kSmallLanes = 8;
constexpr int kSmallStack = kPlainReserve + 7 * kSmallLanes;
constexpr int kSmallChunk = 4;                           // bodies of an opened leaf appended per lane and turn
constexpr int kSmallList = kSmallLanes + kSmallLanes * kSmallChunk;
struct SmallShared {
    int2 stack[kSmallStack];
    int2 list[kSmallList];
    double pos[kPlainW][4];
};

template <bool POT>
__global__ void __launch_bounds__(32 * kPlainWarps, 4)
walk_accurate_small_kernel(Bodies bd, const int64_t* __restrict__ offsets, int nsys, const double4* __restrict__ cubes,
                           int64_t n, Tree t, Params P, unsigned long long* stats, int* err) {
    if (__any_sync(0xffffffffu, *err & kErrAbort)) return;       // whole warps: other blocks may be raising bits
    __shared__ SmallShared shared[32 * kPlainWarps / kSmallLanes];
    SmallShared& S = shared[threadIdx.x / kSmallLanes];
    const int lane = threadIdx.x & 31, sl = lane % kSmallLanes, shift = lane - sl;
    const uint32_t lt = (1u << sl) - 1u;
    // the group's part of a ballot
    const auto mine_of = [&](bool v) { return __ballot_sync(0xffffffffu, v) >> shift & ((1u << kSmallLanes) - 1u); };
    const int64_t w = (blockIdx.x * static_cast<int64_t>(32 * kPlainWarps) + threadIdx.x) / kSmallLanes;
    unsigned npp = 0, npc = 0;
    int sys = 0;
    int64_t first = w * kPlainW, last = n;
    if (offsets) {
        int top = nsys;
        while (top - sys > 1) {
            const int mid = (sys + top) >> 1;
            if (offsets[mid] / kPlainW + mid <= w) sys = mid;
            else top = mid;
        }
        first = offsets[sys] + (w - (offsets[sys] / kPlainW + sys)) * kPlainW;
        last = offsets[sys + 1] - offsets[sys] < kSmallSystem ? offsets[sys + 1] : first;   // large: the walk above
    }
    unsigned bodies = 0, own = 0;
#pragma unroll
    for (int b = 0; b < kPlainW; ++b) {
        if (first + b >= last) continue;
        bodies |= 1u << b;
        if (first + b >= P.own_lo && first + b < P.own_hi) own |= 1u << b;
    }
    const unsigned nodes = static_cast<unsigned>(t.counts[1]), nbodies = static_cast<unsigned>(n);
    const int ex = static_cast<int>((__double_as_longlong(cubes[sys].w) >> 52) & 0x7ff) - 1023;
    const bool scaled = ex > 150 || ex < -150;
    const double S1 = scaled ? scalbn(1.0, -ex) : 1.0;
    const double eps2 = (P.eps * S1) * (P.eps * S1);
    double ax[kPlainW], ay[kPlainW], az[kPlainW], pot[kPlainW];
    int sp = own ? 1 : 0, pn = 0;
#pragma unroll
    for (int b = 0; b < kPlainW; ++b) {
        const int64_t i = own && first + b < last ? first + b : 0;
        if (sl == b) { S.pos[b][0] = bd.x[i] * S1; S.pos[b][1] = bd.y[i] * S1; S.pos[b][2] = bd.z[i] * S1; }
        ax[b] = ay[b] = az[b] = pot[b] = 0.0;
    }
    if (sl == 0) S.stack[0] = make_int2(sys, static_cast<int>(bodies));
    __syncwarp();
    while (__any_sync(0xffffffffu, sp > 0 || pn > 0)) {
        const int room = (kSmallStack - kPlainReserve - sp) / 7;
        const int nb = min(min(sp, kSmallLanes), max(room, 1));
        sp -= nb;
        const int2 entry = sl < nb ? S.stack[sp + sl] : make_int2(-1, 0);
        const int node = entry.x;
        unsigned mask = static_cast<unsigned>(entry.y);
        __syncwarp();
        int2 lk = make_int2(0, 0);
        double4 c = make_double4(0.0, 0.0, 0.0, 0.0);
        double2 qa = make_double2(0.0, 0.0), qb = qa, qc = qa, qd = qa;
        if (mask) {
            bool ok = static_cast<unsigned>(node) < nodes;
            if (ok) {
                lk = __ldg(t.link + node);
                const double2* c2 = reinterpret_cast<const double2*>(t.com + node);
                const double2 ca = __ldg(c2), cb = __ldg(c2 + 1);
                const double2* q2 = reinterpret_cast<const double2*>(t.quad64 + 8 * static_cast<int64_t>(node));
                qd = __ldg(q2 + 3);
                if (P.quad) { qa = __ldg(q2); qb = __ldg(q2 + 1); qc = __ldg(q2 + 2); }
                c = make_double4(ca.x, ca.y, cb.x, cb.y);
                const unsigned e = static_cast<unsigned>(lk.x) + static_cast<unsigned>(lk.y > 0 ? lk.y : -lk.y);
                ok = lk.x >= 0 && lk.y <= 8 && e <= (lk.y > 0 ? nodes : nbodies);
            }
            if (!ok) raise_error(err, kErrIndex);
            if (!ok || c.w == 0.0) mask = 0;
        }
        if (scaled) {
            c.x *= S1; c.y *= S1; c.z *= S1;
            qd.y *= S1;
            qa.x = qa.x * S1 * S1; qa.y = qa.y * S1 * S1; qb.x = qb.x * S1 * S1;
            qb.y = qb.y * S1 * S1; qc.x = qc.x * S1 * S1; qc.y = qc.y * S1 * S1;
        }
        const double rc2 = qd.y * qd.y;
        unsigned opened = 0;
#pragma unroll
        for (int b = 0; b < kPlainW; ++b) {
            const bool mine = mask >> b & 1u;
            const double dx = c.x - at(S.pos[b][0]), dy = c.y - at(S.pos[b][1]), dz = c.z - at(S.pos[b][2]);
            const double r2 = dx * dx + dy * dy + dz * dz;
            const bool open = mine && r2 < rc2, use = mine && !open;
            opened |= static_cast<unsigned>(open) << b;
            const double r2s = away_from_ends(r2 + eps2);
            const double rinv = use ? rsqrt_fast(r2s) : 0.0;
            const double rinv2 = rinv * rinv;
            const double qx = fma(qc.x, dz, fma(qb.y, dy, qa.x * dx));
            const double qy = fma(qc.y, dz, fma(qa.y, dy, qb.y * dx));
            const double qz = fma(qb.x, dz, fma(qc.y, dy, qc.x * dx));
            const double q = fma(dz, qz, fma(dy, qy, dx * qx));
            const double rinv5 = rinv * (rinv2 * rinv2);
            const double k = fma(2.5 * q, rinv2, c.w * r2s);
            ax[b] = fma(rinv5, fma(k, dx, -qx), ax[b]);
            ay[b] = fma(rinv5, fma(k, dy, -qy), ay[b]);
            az[b] = fma(rinv5, fma(k, dz, -qz), az[b]);
            if (POT) pot[b] -= fma(0.5 * q, rinv5, c.w * rinv);
        }
        npc += __popc(mask & ~opened & own);
        // children of opened cells -> stack
        const int push = opened && lk.y > 0 ? lk.y : 0;
        int off = 0, total = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t m = mine_of((push >> k) & 1);
            off += __popc(m & lt) << k;
            total += __popc(m) << k;
        }
        const bool broken = sp + total > kSmallStack;    // only a broken tree gets here
        if (broken) {
            if (sl == 0) raise_error(err, kErrIndex);
            sp = total = 0;
        } else if (total > 0) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < push) S.stack[sp + off + k] = make_int2(lk.x + k, static_cast<int>(opened));
        }
        sp += total;
        // bodies of opened leaves -> list, evaluated eight at a time, the rest when the walk ends
        int remaining = opened && lk.y < 0 && !broken ? -lk.y : 0;
        int src = lk.x;
        while (__any_sync(0xffffffffu, remaining > 0 || (sp == 0 && pn > 0))) {
            const int take = min(remaining, kSmallChunk);
            int o2 = 0, tot = 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint32_t m = mine_of((take >> k) & 1);
                o2 += __popc(m & lt) << k;
                tot += __popc(m) << k;
            }
            for (int k = 0; k < take; ++k) S.list[pn + o2 + k] = make_int2(src + k, static_cast<int>(opened));
            pn += tot;
            src += take;
            remaining -= take;
            const bool more = mine_of(remaining > 0) != 0;
            __syncwarp();
            for (;;) {
                const bool go = pn >= kSmallLanes || (pn > 0 && sp == 0 && !more);
                if (!__any_sync(0xffffffffu, go)) break;
                const int k = go ? max(pn - kSmallLanes, 0) : pn;        // from the end: nothing moves
                const int2 pe = k + sl < pn ? S.list[k + sl] : make_int2(-1, 0);
                const int j = pe.x;
                const unsigned jm = static_cast<unsigned>(pe.y);
                pn = k;
                double xj = 0.0, yj = 0.0, zj = 0.0, mj = 0.0;
                if (jm) { xj = bd.x[j]; yj = bd.y[j]; zj = bd.z[j]; mj = bd.m[j]; }
                if (scaled) { xj *= S1; yj *= S1; zj *= S1; }
#pragma unroll
                for (int b = 0; b < kPlainW; ++b) {
                    if (!(jm >> b & 1u) || j == first + b) continue;
                    const double dx = xj - at(S.pos[b][0]), dy = yj - at(S.pos[b][1]), dz = zj - at(S.pos[b][2]);
                    const double rinv = rsqrt(dx * dx + dy * dy + dz * dz + eps2);
                    const double mr = mj * rinv, mr3 = mr * rinv * rinv;
                    ax[b] = fma(mr3, dx, ax[b]);
                    ay[b] = fma(mr3, dy, ay[b]);
                    az[b] = fma(mr3, dz, az[b]);
                    if (POT) pot[b] -= mr;
                    npp += own >> b & 1u;
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int b = 0; b < kPlainW; ++b) {
        for (int o = kSmallLanes / 2; o > 0; o >>= 1) {
            ax[b] += __shfl_xor_sync(0xffffffffu, ax[b], o);
            ay[b] += __shfl_xor_sync(0xffffffffu, ay[b], o);
            az[b] += __shfl_xor_sync(0xffffffffu, az[b], o);
            if (POT) pot[b] += __shfl_xor_sync(0xffffffffu, pot[b], o);
        }
        const int64_t i = first + b;
        if (sl == 0 && (own >> b & 1u)) {
            const double g = P.G * S1;
            bd.ax[i] = g * ax[b] * S1; bd.ay[i] = g * ay[b] * S1; bd.az[i] = g * az[b] * S1;
            if (POT) bd.pot[i] = g * pot[b];
        }
    }
    add_stats(stats, npp, npc);
}

// FP64 direct summation: block (x = 128 targets, y = source slice).
constexpr int kDirectThreads = 128;

__global__ void __launch_bounds__(kDirectThreads)
direct_kernel(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
              const double* __restrict__ m, int64_t n, const int64_t* __restrict__ targets, int64_t k,
              double eps2, double G, double* __restrict__ partial) {
    __shared__ double4 src[kDirectThreads];
    const int64_t t = blockIdx.x * (int64_t)kDirectThreads + threadIdx.x;
    const int64_t slice = (n + gridDim.y - 1) / gridDim.y;
    const int64_t js = blockIdx.y * slice;
    const int64_t je = js + slice < n ? js + slice : n;
    const int64_t ti = t < k ? targets[t] : -1;
    const double xi = ti >= 0 ? x[ti] : 0.0, yi = ti >= 0 ? y[ti] : 0.0, zi = ti >= 0 ? z[ti] : 0.0;
    double ax = 0.0, ay = 0.0, az = 0.0, ph = 0.0;
    for (int64_t b = js; b < je; b += kDirectThreads) {
        const int64_t j = b + threadIdx.x;
        src[threadIdx.x] = j < je ? make_double4(x[j], y[j], z[j], m[j]) : make_double4(0, 0, 0, 0);
        __syncthreads();
        const int cnt = static_cast<int>(je - b < kDirectThreads ? je - b : kDirectThreads);
        for (int s = 0; s < cnt; ++s) {
            if (b + s == ti) continue;
            const double4 p = src[s];
            const double dx = p.x - xi, dy = p.y - yi, dz = p.z - zi;
            const double r2 = dx * dx + dy * dy + dz * dz + eps2;
            const double rinv = 1.0 / sqrt(r2);
            const double mr3 = G * p.w * rinv * rinv * rinv;
            ax += mr3 * dx; ay += mr3 * dy; az += mr3 * dz;
            ph -= G * p.w * rinv;
        }
        __syncthreads();
    }
    if (t < k) {
        double* o = partial + 4 * (blockIdx.y * k + t);
        o[0] = ax; o[1] = ay; o[2] = az; o[3] = ph;
    }
}

__global__ void direct_reduce_kernel(const double* __restrict__ partial, int64_t k, int slices,
                                     double* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= k) return;
    double s[4] = {0, 0, 0, 0};
    for (int sl = 0; sl < slices; ++sl)
        for (int c = 0; c < 4; ++c) s[c] += partial[4 * (sl * k + t) + c];
    for (int c = 0; c < 4; ++c) out[4 * t + c] = s[c];
}

// The device softening law on k (size, mass, dist) triples (test support).
__global__ void softening_kernel(const double* __restrict__ in, int64_t k, double* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < k) out[t] = softening_at(softening_base(in[t], in[k + t]), in[2 * k + t]);
}

// The walks' inverse square root on k values (test support).
__global__ void inverse_root_kernel(const double* __restrict__ in, int64_t k, double* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < k) out[t] = rsqrt_fast(away_from_ends(in[t]));
}

}  // namespace

cudaError_t launch_softening_eval(const double* in, int64_t k, double* out, cudaStream_t st) {
    if (k <= 0) return cudaSuccess;
    softening_kernel<<<static_cast<unsigned>((k + 127) / 128), 128, 0, st>>>(in, k, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_inverse_root_eval(const double* in, int64_t k, double* out, cudaStream_t st) {
    if (k <= 0) return cudaSuccess;
    inverse_root_kernel<<<static_cast<unsigned>((k + 127) / 128), 128, 0, st>>>(in, k, out);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_walk_plain(const Bodies& bd, const int32_t* sysid, const int64_t* d_offsets, const Systems& sys,
                              int64_t n, const Tree& t, const Params& P, bool potential, unsigned long long* stats, int* err,
                              cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int32_t* sid = sys.n > 1 ? sysid : nullptr;
    if (P.physics == NEXT_PHYSICS_ACCURATE) {
        const int64_t* offsets = sys.n > 1 ? d_offsets : nullptr;
        const int64_t chunks = (n + kPlainW - 1) / kPlainW + (sys.n > 1 ? sys.n : 0);    // of up to W bodies
        if (sys.smallest < kSmallSystem) {
            constexpr int per = 32 * kPlainWarps / kSmallLanes;
            auto kern = potential ? walk_accurate_small_kernel<true> : walk_accurate_small_kernel<false>;
            kern<<<static_cast<unsigned>((chunks + per - 1) / per), 32 * kPlainWarps, 0, st>>>(bd, offsets, sys.n, sys.cube, n, t,
                                                                                            P, stats, err);
        }
        if (sys.largest >= kSmallSystem) {
            auto kern = potential ? walk_accurate_kernel<true> : walk_accurate_kernel<false>;
            kern<<<static_cast<unsigned>((chunks + kPlainWarps - 1) / kPlainWarps), 32 * kPlainWarps, 0, st>>>(
                bd, offsets, sys.n, sys.cube, n, t, P, stats, err);
        }
        if (sys.smallest < kSmallSystem && sys.largest >= kSmallSystem) count_launches(1);
    } else if (n <= kWideMax) {
        // as many lanes, then as many registers, as leave every warp resident at once
        const int64_t block = 148 * (kRefThreads / 32);           // warps of one block per SM
        const int lanes = n <= 5 * block ? 32 : n <= 10 * block ? 16 : 8, per = kRefThreads / lanes;
        auto kern = lanes == 32      ? walk_reference_wide_kernel<32, 5>
                    : lanes == 16    ? walk_reference_wide_kernel<16, 5>
                    : n <= 20 * block ? walk_reference_wide_kernel<8, 5>
                    : n > 24 * block && n <= 28 * block ? walk_reference_wide_kernel<8, 7>
                                                        : walk_reference_wide_kernel<8, 6>;
        kern<<<static_cast<unsigned>((n + per - 1) / per), kRefThreads, 0, st>>>(bd, sid, n, t, P, stats, err);
    } else {
        const unsigned blocks = static_cast<unsigned>((n + kRefThreads - 1) / kRefThreads);
        auto kern = P.theta < kRefListTheta ? walk_reference_small_theta_kernel : walk_reference_kernel;
        kern<<<blocks, kRefThreads, 0, st>>>(bd, sid, n, t, P, stats, err);
    }
    count_launches(1);
    return cudaGetLastError();
}

int direct_slices(int64_t n, int64_t k) {
    const int64_t tblocks = (k + kDirectThreads - 1) / kDirectThreads;
    int64_t slices = (4 * 148 + tblocks - 1) / (tblocks > 0 ? tblocks : 1);
    if (slices < 1) slices = 1;
    if (slices > 256) slices = 256;
    if (slices > n) slices = n > 0 ? n : 1;
    return static_cast<int>(slices);
}

cudaError_t launch_direct(const Bodies& bd, int64_t n, const int64_t* targets, int64_t k, double eps, double G,
                          double* partial, int slices, double* out, cudaStream_t st) {
    if (k <= 0) return cudaSuccess;
    dim3 grid(static_cast<unsigned>((k + kDirectThreads - 1) / kDirectThreads), static_cast<unsigned>(slices));
    direct_kernel<<<grid, kDirectThreads, 0, st>>>(bd.x, bd.y, bd.z, bd.m, n, targets, k, eps * eps, G, partial);
    direct_reduce_kernel<<<static_cast<unsigned>((k + 127) / 128), 128, 0, st>>>(partial, k, slices, out);
    count_launches(2);
    return cudaGetLastError();
}

}  // namespace nb
