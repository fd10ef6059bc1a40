// gf_tree.cu — GPU octree that reproduces the reference's Barnes-Hut tree
// (cpp/nbody.cpp:76-256) and its refit (cpp/nbody.cpp:262-305).
//
// The reference partitions index ranges recursively: a particle goes to octant bit k of a
// cell when coordinate k is strictly greater than the cell centre, centres being computed
// in float64 by repeated halving (child = parent +- half/2). Partitions are stable, so
// inside every cell particles keep increasing index order; a cell is a leaf when it holds
// at most 8 particles or sits at depth 48; nodes are stored depth-first with `next` links.
//
// Here the same tree comes out of a sort:
//   1. float64 bbox -> root cube, same formula as cpp/nbody.cpp:218-219.
//   2. 63-bit Morton key per particle holding its octant at levels 1..21. Fast path: a
//      fixed-point grid position; when a coordinate lies within a rounding margin of a
//      cell wall the key is recomputed with the exact float64 centre chain, so every
//      octant decision equals the reference's `pos > c` test.
//   3. stable radix sort of (key, index): tree order = (octant path, index).
//   4. cells: 9 consecutive sorted keys sharing a level-d prefix <=> that cell holds > 8
//      particles, so each particle's leaf depth and the nodes that start at it follow from
//      common-prefix lengths of neighbouring keys; an exclusive scan numbers the nodes in
//      depth-first order, and `next` is the id of the first node starting after the cell.
//      Cells that still hold > 8 particles at level 21 get extension keys (levels 22..48,
//      exact chain) and are re-sorted in shared memory.
//   5. node emission, where a leaf's thread also puts its particles in index order (the
//      reference never partitions a leaf).
//   6. moments bottom-up in one launch (the last child to arrive completes its parent), float64
//      sums of the same terms as the reference (a parent's first four children and its last four
//      apart, then both), rounded to the same float32 node record.
#include <algorithm>
#include <cfloat>
#include <climits>

#include <cooperative_groups.h>

#include "gf_scan.cuh"
#include "gf_tree.cuh"

namespace gf {

namespace {

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------- bbox

// Order-preserving map of float64 values to int64 (and back): min / max of the images is the
// image of the min / max, so the reduction runs on the integer pipes instead of the narrow
// float64 one. Non-finite values are flagged separately.
__device__ __forceinline__ long long fkey(double v) {
    const long long b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double fkey_inv(long long k) { return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL)); }
__device__ __forceinline__ bool finite_bits(double v) {
    return ((__double_as_longlong(v) >> 52) & 0x7ff) != 0x7ff;
}

// Root cube of a bounding box tot = {lo x, y, z, hi x, y, z} (cpp/nbody.cpp:218-219) and the grid of
// the fast key path.
__device__ RootBox root_box(const double (&tot)[6], double theta) {
    RootBox R;
    double ext = 0;
    for (int a = 0; a < 3; ++a) {
        R.c[a] = __dmul_rn(0.5, __dadd_rn(tot[a], tot[3 + a]));
        ext = fmax(ext, __dsub_rn(tot[3 + a], tot[a]));
    }
    // 0.5 * max extent * 1.0001 + 1e-12 (cpp/nbody.cpp:219), unfused
    R.half = __dadd_rn(__dmul_rn(__dmul_rn(0.5, ext), 1.0001), 1e-12);
    R.open0 = __ddiv_rn(__dmul_rn(2.0, R.half), theta);
    // (theta infinite: a node's first term is scaled down from this one by its exponent, which 0 lacks)
    if (R.open0 == 0.0) R.open0 = ldexp(1.0, -900);
    double cmax = 0;
    for (int a = 0; a < 3; ++a) {
        R.lo[a] = __dsub_rn(R.c[a], R.half);
        cmax = fmax(cmax, fabs(R.c[a]));
    }
    R.inv_w = __ddiv_rn(2097152.0, __dmul_rn(2.0, R.half));
    // Rounding of the float64 centre chain (<= 21 roundings of <= 1/2 ulp(|c| + half)) plus
    // that of the fixed-point position stays below 2^-27 (|c|/half + 2) grid units; the
    // margin keeps a factor 8 on top.
    R.margin = ldexp(1.0, -24) * (cmax / R.half + 2.0);
    // the same test in 32.32 fixed point (scaling by 2^32 is exact): the fraction window
    // [m_lo, m_hi] of the truncated fixed-point position lies inside [margin, 1 - margin]
    R.inv_w32 = R.inv_w * 4294967296.0;
    const double ml = fmin(ceil(R.margin * 4294967296.0), 2147483648.0);
    R.m_lo = uint32_t(ml);
    R.m_hi = uint32_t(4294967295.0 - ml);
    return R;
}

// float64 bounding box -> root cube (cpp/nbody.cpp:210-219) in one launch: every block reduces
// its share of the positions and writes a partial; the last block to finish (arrival counter)
// reduces the partials and writes the root cube. min / max are exact, so the result does not
// depend on the order of the reductions.
__global__ void k_bbox(const double* __restrict__ pos, int n, double* __restrict__ part, RootBox* __restrict__ root,
                       double theta, uint32_t* status, int* __restrict__ done) {
    long long lo[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, hi[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    int bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double v = pos[3 * size_t(i) + a];
            bad |= finite_bits(v) ? 0 : 1;
            const long long k = fkey(v);
            lo[a] = min(lo[a], k);
            hi[a] = max(hi[a], k);
        }
    }
    __shared__ long long s[6][kThreads / 32];
    __shared__ int s_bad[kThreads / 32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_reduce = [&](long long* out, int* out_bad) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = min(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = max(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
            bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        }
        if (lane == 0) {
            for (int a = 0; a < 3; ++a) {
                s[a][warp] = lo[a];
                s[3 + a][warp] = hi[a];
            }
            s_bad[warp] = bad;
        }
        __syncthreads();
        if (threadIdx.x < 6) {
            long long v = s[threadIdx.x][0];
            for (int w = 1; w < kThreads / 32; ++w)
                v = threadIdx.x < 3 ? min(v, s[threadIdx.x][w]) : max(v, s[threadIdx.x][w]);
            out[threadIdx.x] = v;
        }
        if (threadIdx.x == 6) {
            int v = 0;
            for (int w = 0; w < kThreads / 32; ++w) v |= s_bad[w];
            *out_bad = v;
        }
    };
    long long* ipart = reinterpret_cast<long long*>(part);
    int dummy;
    block_reduce(ipart + 7 * size_t(blockIdx.x), &dummy);
    if (threadIdx.x == 6) ipart[7 * size_t(blockIdx.x) + 6] = dummy;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1) == int(gridDim.x) - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int a = 0; a < 3; ++a) {
        lo[a] = LLONG_MAX;
        hi[a] = LLONG_MIN;
    }
    bad = 0;
    for (int b = threadIdx.x; b < int(gridDim.x); b += blockDim.x) {
        for (int a = 0; a < 3; ++a) {
            lo[a] = min(lo[a], __ldcg(&ipart[7 * size_t(b) + a]));
            hi[a] = max(hi[a], __ldcg(&ipart[7 * size_t(b) + 3 + a]));
        }
        bad |= int(__ldcg(&ipart[7 * size_t(b) + 6]));
    }
    __shared__ long long itot[6];
    __shared__ int tot_bad;
    __syncthreads();
    block_reduce(itot, &tot_bad);
    __syncthreads();
    if (threadIdx.x != 0) return;
    double tot[6];
    for (int a = 0; a < 6; ++a) tot[a] = fkey_inv(itot[a]);
    if (tot_bad) raise_status(status, GF_ERR_NONFINITE);
    *root = root_box(tot, theta);
}

// ---------------------------------------------------------------------------- keys

__device__ __forceinline__ uint64_t part1by2(uint32_t v) {
    uint64_t x = v & 0x1fffffu;
    x = (x | (x << 32)) & 0x1f00000000ffffull;
    x = (x | (x << 16)) & 0x1f0000ff0000ffull;
    x = (x | (x << 8)) & 0x100f00f00f00f00full;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// Exact octant digits from the float64 centre chain (cpp/nbody.cpp:80, :92-96, :135-139).
// Levels 1..21 -> k0, 22..42 -> k1, 43..48 -> k2 (each left-aligned in its word).
__device__ void exact_keys(double x, double y, double z, const RootBox& R, int levels,
                           uint64_t& k0, uint64_t& k1, uint64_t& k2) {
    double cx = R.c[0], cy = R.c[1], cz = R.c[2], h = R.half;
    k0 = k1 = k2 = 0;
    for (int l = 1; l <= levels; ++l) {
        h = 0.5 * h;
        const unsigned o = unsigned(x > cx) | (unsigned(y > cy) << 1) | (unsigned(z > cz) << 2);
        cx = __dadd_rn(cx, (o & 1) ? h : -h);
        cy = __dadd_rn(cy, (o & 2) ? h : -h);
        cz = __dadd_rn(cz, (o & 4) ? h : -h);
        if (l <= 21)
            k0 = (k0 << 3) | o;
        else if (l <= 42)
            k1 = (k1 << 3) | o;
        else
            k2 = (k2 << 3) | o;
    }
    if (levels < 21) k0 <<= 3 * (21 - levels);
}

// Grid cell of coordinate a on the 2^21 grid, when the position lies at least `margin` grid
// units from every cell wall (else the exact path decides). 32.32 fixed point: u = (x - lo) *
// inv_w * 2^32 (the same rounding as without the 2^32), truncated; the integer part is the
// cell, the fraction is tested against a window no wider than [margin, 1 - margin]. One float64
// subtract, multiply and conversion per coordinate; the tests are integer.
__device__ __forceinline__ bool grid_coord(double x, int a, const RootBox& R, uint32_t& ic) {
    const double u = __dmul_rn(__dsub_rn(x, R.lo[a]), R.inv_w32);
    const long long ub = __double_as_longlong(u);
    if (ub < 0 || ub >= 0x4340000000000000LL) return false;  // outside [0, 2^53) (or NaN)
    const unsigned long long q = __double2ull_rz(u);
    ic = uint32_t(q >> 32);
    const uint32_t fr = uint32_t(q);
    return ic < 2097152u && fr >= R.m_lo && fr <= R.m_hi;
}

// The 63-bit Morton key: the octants of levels 1..21.
__device__ __forceinline__ uint64_t morton_key(double x, double y, double z, const RootBox& R) {
    uint32_t ix, iy, iz;
    uint64_t k;
    if (grid_coord(x, 0, R, ix) && grid_coord(y, 1, R, iy) && grid_coord(z, 2, R, iz)) {
        k = part1by2(ix) | (part1by2(iy) << 1) | (part1by2(iz) << 2);
    } else {
        uint64_t k1, k2;
        exact_keys(x, y, z, R, 21, k, k1, k2);
    }
    return k;
}

__global__ void k_keys(const double* __restrict__ pos, int n, const RootBox* __restrict__ rootp,
                       uint64_t* __restrict__ key, int* __restrict__ perm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const RootBox R = *rootp;
    key[i] = morton_key(pos[3 * size_t(i)], pos[3 * size_t(i) + 1], pos[3 * size_t(i) + 2], R);
    perm[i] = i;
}

// ---------------------------------------------------------------------------- small sets

// Bounding box, keys and their radix sort in one launch, for sets that fit the shared memory of one
// cluster: kSmallCtas blocks hold m consecutive positions each; 8-bit passes rank the keys
// as the one-sweep sort does (ballots per warp, warps in key order), add up the blocks' digit
// counts through distributed shared memory and scatter keys and indices straight into the block
// that holds their new position. Two cluster barriers a pass take the place of a launch, a digit
// histogram and a look-back. The launch's time grows with the keys per block (scattered remote
// stores), where the chain of 12 launches hardly changes: 25 us at 2k keys, 39 at 10k and 70 at 28k,
// against 75 for the chain's sort alone at 50k. Engine.gravity of 28,672 / 28,673 particles, the last count with
// this launch and the first with the chain: 325 / 352 us. (Blocks of 512 threads instead of 1024,
// whose barriers are longer: 2 % faster builds.)
static_assert(kKeyLevels == 21, "eight 8-bit passes over a 63-bit key");
constexpr int kSmallCtas = 8;
constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallItems = 7;                             // keys per thread at most
constexpr int kSmallMaxPer = kSmallThreads * kSmallItems;  // positions per block at most
constexpr int kSmallMax = kSmallCtas * kSmallMaxPer;        // 28,672 particles

// The keys are sorted by their top 40 bits first (13 octree levels). Keys that share those are mostly
// alone or in twos and threes, and a thread sorts such a run by insertion; a run of more than kSmallRun
// (coincident particles, cores 10^4 times smaller than the box) sends the whole set through all eight
// digits. Engine.gravity of a 2k / 10k / 24k cloud with eight passes 154 / 226 / 268 us, with five
// and the runs 150 / 217 / 253 (with four 148 / 213 / 246, but 385 instead of 325 us for a concentrated
// 28k set whose core then takes all twelve). Such a set pays for both sorts, 63 instead of 39 us at 10k:
// gravity of 10k / 28k particles in groups of 20 within 10^-6 396 / 469 us.
constexpr int kSmallTopPasses = 5, kSmallTopShift = 63 - 8 * kSmallTopPasses, kSmallRun = 16;

constexpr size_t small_sort_smem(int m) {
    return size_t(m) * 2 * (sizeof(uint64_t) + sizeof(int)) + sizeof(uint16_t) * kSmallWarps * 256;
}

__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallThreads)
    k_small_sort(const double* __restrict__ pos, int n, int m, unsigned div_m, double theta, RootBox* __restrict__ root,
                 uint64_t* __restrict__ key, int* __restrict__ perm, TreeCounts* __restrict__ counts, uint32_t* status) {
    extern __shared__ unsigned char smem_small[];
    uint64_t* kb = reinterpret_cast<uint64_t*>(smem_small);  // two buffers of m keys
    int* vb = reinterpret_cast<int*>(kb + 2 * m);            // two of m indices
    uint16_t* cnt = reinterpret_cast<uint16_t*>(vb + 2 * m);  // [warp][digit]
    __shared__ int s_tot[kSmallCtas][256], s_part[kSmallThreads / 256][256], s_base[256], s_wsum[kSmallWarps];
    __shared__ long long s_box[7], s_red[kSmallWarps][7];
    __shared__ RootBox s_root;
    __shared__ int s_found;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = lanemask_lt();
    const int first = rank * m;                   // this block's positions: [first, first + own)
    const int own = max(0, min(m, n - first));
    if (rank == 0)  // the build's counters start at zero (nothing uses them before the next launch)
        for (int t = tid; t < int(sizeof(TreeCounts) / sizeof(int)); t += kSmallThreads)
            reinterpret_cast<int*>(counts)[t] = 0;

    if (tid == 0) s_found = 0;
    // bounding box of the block's share, then of all blocks (exact: min and max of integer images)
    long long v[7] = {LLONG_MAX, LLONG_MAX, LLONG_MAX, LLONG_MIN, LLONG_MIN, LLONG_MIN, 0};
    for (int o = tid; o < own; o += kSmallThreads) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double x = pos[3 * size_t(first + o) + a];
            v[6] |= finite_bits(x) ? 0 : 1;
            const long long k = fkey(x);
            v[a] = min(v[a], k);
            v[3 + a] = max(v[3 + a], k);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            v[a] = min(v[a], __shfl_xor_sync(0xffffffffu, v[a], o));
            v[3 + a] = max(v[3 + a], __shfl_xor_sync(0xffffffffu, v[3 + a], o));
        }
        v[6] |= __shfl_xor_sync(0xffffffffu, v[6], o);
    }
    if (lane == 0)
        for (int a = 0; a < 7; ++a) s_red[warp][a] = v[a];
    __syncthreads();
    if (tid < 7) {
        long long x = s_red[0][tid];
        for (int w = 1; w < kSmallWarps; ++w) {
            const long long y = s_red[w][tid];
            x = tid < 3 ? min(x, y) : tid < 6 ? max(x, y) : x | y;
        }
        s_box[tid] = x;
    }
    cluster.sync();
    if (tid < 7) {
        long long x = *cluster.map_shared_rank(&s_box[tid], 0);
        for (int c = 1; c < kSmallCtas; ++c) {
            const long long y = *cluster.map_shared_rank(&s_box[tid], c);
            x = tid < 3 ? min(x, y) : tid < 6 ? max(x, y) : x | y;
        }
        s_red[0][tid] = x;
    }
    __syncthreads();
    if (tid == 0) {
        double tot[6];
        for (int a = 0; a < 6; ++a) tot[a] = fkey_inv(s_red[0][a]);
        s_root = root_box(tot, theta);
        if (rank == 0) {
            *root = s_root;
            if (s_red[0][6]) raise_status(status, GF_ERR_NONFINITE);
        }
    }
    __syncthreads();
    {
        const RootBox R = s_root;
        for (int o = tid; o < own; o += kSmallThreads) {
            const double* p = pos + 3 * size_t(first + o);
            kb[o] = morton_key(p[0], p[1], p[2], R);
            vb[o] = first + o;
        }
    }
    __syncthreads();

    const int items = (m + kSmallThreads - 1) / kSmallThreads;  // per thread, uniform over the cluster
    const int wbase = warp * 32 * items;                        // a warp's consecutive positions
    auto clear_counts = [&] {
        for (int t = lane; t < 128; t += 32) reinterpret_cast<unsigned*>(cnt + warp * 256)[t] = 0u;
        __syncwarp();
    };
    clear_counts();
    int cur = 0;  // buffer of the keys
    for (int pass = 0;; ++pass) {
        const uint64_t* ki = kb + cur * m;
        const int* vi = vb + cur * m;
        cur ^= 1;
        uint64_t* ko = kb + cur * m;
        int* vo = vb + cur * m;
        const int shift = pass < kSmallTopPasses ? kSmallTopShift + 8 * pass : 8 * (pass - kSmallTopPasses);
        uint64_t k[kSmallItems];
        int rk[kSmallItems];
#pragma unroll
        for (int s = 0; s < kSmallItems; ++s) {
            if (s >= items) break;
            const int o = wbase + 32 * s + lane;
            const bool ok = o < own;
            k[s] = ok ? ki[o] : 0ull;
            const unsigned d = unsigned(k[s] >> shift) & 255u;
            const unsigned peers = digit_peers(d, ok);
            const int before = ok ? cnt[warp * 256 + d] : 0;
            rk[s] = before + __popc(peers & lt);
            __syncwarp();
            if (ok && lane == __ffs(peers) - 1) cnt[warp * 256 + d] = uint16_t(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // two threads per digit: exclusive prefix over the warps; the block's count of every digit
        // goes to all blocks
        const int d = tid & 255, part = tid >> 8;
        constexpr int kParts = kSmallThreads / 256, kPart = kSmallWarps / kParts;
        int sum = 0;
#pragma unroll
        for (int w = 0; w < kPart; ++w) sum += cnt[(part * kPart + w) * 256 + d];
        s_part[part][d] = sum;
        __syncthreads();
        int run = 0, own_d = 0;
#pragma unroll
        for (int t = 0; t < kParts; ++t) {
            const int x = s_part[t][d];
            if (t < part) run += x;
            own_d += x;
        }
#pragma unroll
        for (int c = part; c < kSmallCtas; c += kParts) *cluster.map_shared_rank(&s_tot[rank][d], c) = own_d;
        auto counted = cluster.barrier_arrive();
#pragma unroll
        for (int w = 0; w < kPart; ++w) {
            const int c = cnt[(part * kPart + w) * 256 + d];
            cnt[(part * kPart + w) * 256 + d] = uint16_t(run);
            run += c;
        }
        cluster.barrier_wait(std::move(counted));
        // the digit's keys in all blocks, and in the blocks before this one
        int all = 0, prev = 0;
        if (tid < 256) {
#pragma unroll
            for (int c = 0; c < kSmallCtas; ++c) {
                const int x = s_tot[c][tid];
                all += x;
                if (c < rank) prev += x;
            }
        }
        int scan = warp_incl_scan(all);  // over the 256 digits: the first eight warps
        if (lane == 31) s_wsum[warp] = scan;
        __syncthreads();
        if (tid < 256) {
            int before = 0;
            for (int w = 0; w < warp; ++w) before += s_wsum[w];
            s_base[tid] = before + scan - all + prev;
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < kSmallItems; ++s) {
            if (s >= items) break;
            const int o = wbase + 32 * s + lane;
            if (o < own) {
                const unsigned dg = unsigned(k[s] >> shift) & 255u;
                const unsigned to = unsigned(s_base[dg] + int(cnt[warp * 256 + dg]) + rk[s]);
                const unsigned c = __umulhi(to, div_m);  // to / m
                const unsigned off = to - c * unsigned(m);
                *cluster.map_shared_rank(ko + off, c) = k[s];
                *cluster.map_shared_rank(vo + off, c) = vi[o];
            }
        }
        auto scattered = cluster.barrier_arrive();
        __syncwarp();
        clear_counts();
        cluster.barrier_wait(std::move(scattered));
        if (pass == kSmallTopPasses + 7) break;
        if (pass != kSmallTopPasses - 1) continue;
        // keys in order of their top bits: runs that share them are sorted in place, by the thread of
        // a run's first key, unless one is too long for that
        auto key_at = [&](int p) {
            const unsigned c = __umulhi(unsigned(p), div_m);
            return cluster.map_shared_rank(kb + cur * m + (p - int(c) * m), c);
        };
        auto val_at = [&](int p) {
            const unsigned c = __umulhi(unsigned(p), div_m);
            return cluster.map_shared_rank(vb + cur * m + (p - int(c) * m), c);
        };
        // four bits for each of this thread's keys: the length minus one of the run that starts there.
        // (The insertion goes by it: the key after a run belongs to the next run's thread, which may
        // be moving it.)
        static_assert(kSmallRun == 16 && kSmallItems <= 8, "four bits per key");
        unsigned lens = 0;
        int found = 0;  // 1: runs, 2: one too long
        for (int s = 0; s < items; ++s) {
            const int p = first + tid + kSmallThreads * s;
            if (p >= first + own) break;
            const uint64_t top = *key_at(p) >> kSmallTopShift;
            if (p > 0 && *key_at(p - 1) >> kSmallTopShift == top) continue;
            int len = 1;
            while (p + len < n && len <= kSmallRun && *key_at(p + len) >> kSmallTopShift == top) ++len;
            lens |= unsigned(min(len, kSmallRun) - 1) << (4 * s);
            found |= len > kSmallRun ? 2 : len > 1 ? 1 : 0;
        }
        found = __reduce_or_sync(0xffffffffu, unsigned(found));
        if (lane == 0 && found)
            for (int c = 0; c < kSmallCtas; ++c) atomicOr(cluster.map_shared_rank(&s_found, c), found);
        cluster.sync();
        found = s_found;
        if (found & 2) continue;  // all eight digits after all
        if (!found) break;
        for (int s = 0; lens; ++s, lens >>= 4) {
            const int p = first + tid + kSmallThreads * s;
            for (int e = p + 1; e <= p + int(lens & 15u); ++e) {  // insertion, stable
                const uint64_t k = *key_at(e);
                const int v = *val_at(e);
                int q = e;
                for (; q > p && *key_at(q - 1) > k; --q) {
                    *key_at(q) = *key_at(q - 1);
                    *val_at(q) = *val_at(q - 1);
                }
                if (q != e) *key_at(q) = k, *val_at(q) = v;
            }
        }
        cluster.sync();
        break;
    }
    for (int o = tid; o < own; o += kSmallThreads) {
        key[first + o] = kb[cur * m + o];
        perm[first + o] = vb[cur * m + o];
    }
}

// ---------------------------------------------------------------------------- prefixes

struct KeyView {
    const uint64_t* k0;
    const uint64_t* k1;  // null unless some level-21 cell holds > 8 particles
    const uint64_t* k2;
};

// Number of leading octree levels shared by sorted positions i and j (0..48).
__device__ __forceinline__ int cpl(const KeyView& K, int i, int j) {
    uint64_t a = K.k0[i], b = K.k0[j];
    if (a != b) return (__clzll(a ^ b) - 1) / 3;
    if (!K.k1) return 21;
    a = K.k1[i];
    b = K.k1[j];
    if (a != b) return 21 + (__clzll(a ^ b) - 1) / 3;
    a = K.k2[i];
    b = K.k2[j];
    if (a != b) return 42 + (__clzll(a ^ b) - 46) / 3;
    return 48;
}

__device__ __forceinline__ int digit(const KeyView& K, int i, int l) {
    if (l <= 21) return int((K.k0[i] >> (3 * (21 - l))) & 7);
    if (l <= 42) return int((K.k1[i] >> (3 * (42 - l))) & 7);
    return int((K.k2[i] >> (3 * (48 - l))) & 7);
}

// The nodes that start at each sorted position, numbered depth-first. A cell holding positions i and
// i + L (L = leaf capacity) holds more than L particles and must split, so position i's leaf depth
// is one more than the longest prefix among the pairs (j, j + L) around it, and the nodes of depths
// dsplit .. ldepth start at i, dsplit one more than the prefix shared with position i - 1.
struct StartScan {
    KeyView K;
    int n, L;
    int8_t* ldepth;
    int8_t* dsplit;
    int* nbase;    // first node id of each position
    int* owner;    // position of each node id below cap
    int cap;
    TreeCounts* cnt;
    __device__ int first(int i) const {
        int m = -1;
        for (int j = max(0, i - L); j <= i; ++j) {
            if (j + L >= n) break;
            const int c = cpl(K, j, j + L);
            m = max(m, c);
            if (j == i && c == 21 && !K.k1) cnt->deep = 1;
        }
        const int ds = i == 0 ? 0 : cpl(K, i - 1, i) + 1;
        ldepth[i] = int8_t(min(kDepthMax, m + 1));
        dsplit[i] = int8_t(min(ds, 127));
        return again(i);
    }
    __device__ int again(int i) const { return max(0, int(ldepth[i]) - int(dsplit[i]) + 1); }
    __device__ void put(int i, int v, int ex) const {
        nbase[i] = ex;
        for (int t = 0; t < v && ex + t < cap; ++t) owner[ex + t] = i;
    }
};

// first j > i with j == n or cpl(i, j) < d
__device__ int run_end(const KeyView& K, int n, int i, int d) {
    if (d == 0) return n;
    int j = i + 1;
    for (int t = 0; t < 9 && j < n; ++t, ++j)
        if (cpl(K, i, j) < d) return j;
    if (j >= n) return n;
    int lo = j, step = 16, hi;
    for (;;) {
        hi = lo + step;
        if (hi >= n) {
            hi = n;
            break;
        }
        if (cpl(K, i, hi) < d) break;
        lo = hi + 1;
        step *= 2;
    }
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cpl(K, i, mid) < d)
            hi = mid;
        else
            lo = mid + 1;
    }
    return lo;
}

// first j <= i with cpl(j, i) >= lev
__device__ int run_begin(const KeyView& K, int i, int lev) {
    int hi = i, step = 1, lo;
    for (;;) {
        lo = hi - step;
        if (lo < 0) {
            lo = -1;
            break;
        }
        if (cpl(K, lo, i) < lev) break;
        hi = lo;
        step *= 2;
    }
    int a = lo + 1, b = hi;
    while (a < b) {
        const int mid = (a + b) >> 1;
        if (cpl(K, mid, i) >= lev)
            b = mid;
        else
            a = mid + 1;
    }
    return b;
}

// ---------------------------------------------------------------------------- emit

// Node emission, one thread per node. Position i starts the nodes of depths ds[i] .. ld[i]
// (ids nbase[i] ..); the scan that numbers the nodes writes, for every node id, the position that
// starts it (k_node_owner again, after the node buffers have grown), and k_emit fills the node: the cube centre by the float64 halving chain from the root along
// i's octant digits (cpp/nbody.cpp:92-96), the particle range [i, end) with end the first
// position whose prefix leaves the node's, `next` = the first node starting at end, the leaf
// flag and the parent (the previous node of the chain, or the deepest node at depth d - 1 of
// the run containing i). Threads of consecutive ids take chains of similar depth, so a warp
// keeps most lanes busy (one thread per starting position left 5 of 32 busy).
// A leaf's thread also puts its particles in increasing index order (the reference's stable
// partitions never reorder a leaf), the nodes of each depth are counted for the breadth-first
// numbering, and that pass's look-back statuses are cleared.
__global__ void k_node_owner(int n, StartScan S) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) S.put(i, S.again(i), S.nbase[i]);
}

// Particle indices of a leaf into increasing order: up to kLeafMax of them by a sorting network in
// registers (Batcher's odd-even merge, 19 exchanges); leaves of more than 64 hold identical keys
// and are sorted already.
__device__ __forceinline__ void sort_leaf(int* p, int count) {
    if (count <= kLeafMax) {
        static_assert(kLeafMax == 8, "a network of 8");
        int v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) v[t] = t < count ? p[t] : INT_MAX;
        constexpr int kA[19] = {0, 2, 4, 6, 0, 1, 4, 5, 1, 5, 0, 1, 2, 3, 2, 3, 1, 3, 5};
        constexpr int kB[19] = {1, 3, 5, 7, 2, 3, 6, 7, 2, 6, 4, 5, 6, 7, 4, 5, 2, 4, 6};
#pragma unroll
        for (int c = 0; c < 19; ++c) {
            const int a = v[kA[c]], b = v[kB[c]];
            v[kA[c]] = min(a, b);
            v[kB[c]] = max(a, b);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (t < count) p[t] = v[t];
        return;
    }
    if (count > 64) return;
    for (int a = 1; a < count; ++a) {
        const int v = p[a];
        int b = a - 1;
        while (b >= 0 && p[b] > v) {
            p[b + 1] = p[b];
            --b;
        }
        p[b + 1] = v;
    }
}

__device__ __forceinline__ void emit_node(KeyView K, int n, int span, const RootBox* __restrict__ rootp,
                                          const int8_t* __restrict__ ldepth, const int8_t* __restrict__ dsplit,
                                          const int* __restrict__ nbase, const int* __restrict__ owner,
                                          const TreeCounts* cnt, int4* __restrict__ n_i4, double4* __restrict__ n_cd,
                                          float4* __restrict__ n_geo, int* __restrict__ n_parent,
                                          int* __restrict__ perm, int cap, int* s_depth) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    const int total = cnt->total_nodes;
    if (id >= span || id >= total || id >= cap) return;  // past cap: reported by k_node_cap_check
    const int i = owner[id];
    const int ds = dsplit[i], ld = ldepth[i];
    const int d = ds + (id - nbase[i]);
    const RootBox R = *rootp;
    double c[3] = {R.c[0], R.c[1], R.c[2]};
    double h = R.half;
    for (int l = 1; l <= d; ++l) {
        h = 0.5 * h;
        const int o = digit(K, i, l);
        c[0] = __dadd_rn(c[0], (o & 1) ? h : -h);
        c[1] = __dadd_rn(c[1], (o & 2) ? h : -h);
        c[2] = __dadd_rn(c[2], (o & 4) ? h : -h);
    }
    const int end = run_end(K, n, i, d);
    const int next = end < n ? nbase[end] : total;
    int parent;
    if (d == 0) {
        parent = -1;
    } else if (d > ds) {
        parent = id - 1;
    } else {
        const int s = run_begin(K, i, d - 1);
        parent = nbase[s] + (d - 1 - dsplit[s]);
    }
    n_i4[id] = make_int4(i, end - i, next, (d == ld ? 1 : 0) | (d << 8));
    n_cd[id] = make_double4(c[0], c[1], c[2], h);
    n_geo[id] = make_float4(float(c[0]), float(c[1]), float(c[2]), float(h));
    n_parent[id] = parent;
    atomicAdd(&s_depth[d], 1);
    if (d == ld) sort_leaf(perm + i, end - i);
}

__global__ void k_emit(KeyView K, int n, int span, const RootBox* __restrict__ rootp,
                       const int8_t* __restrict__ ldepth, const int8_t* __restrict__ dsplit,
                       const int* __restrict__ nbase, const int* __restrict__ owner,
                       TreeCounts* __restrict__ cnt, int4* __restrict__ n_i4,
                       double4* __restrict__ n_cd, float4* __restrict__ n_geo,
                       int* __restrict__ n_parent, int* __restrict__ perm, int cap,
                       unsigned* __restrict__ bfs_status, int status_words) {
    __shared__ int s_depth[kDepthMax + 1];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < status_words; t += gridDim.x * blockDim.x) bfs_status[t] = 0u;
    if (threadIdx.x <= kDepthMax) s_depth[threadIdx.x] = 0;
    __syncthreads();
    emit_node(K, n, span, rootp, ldepth, dsplit, nbase, owner, cnt, n_i4, n_cd, n_geo, n_parent, perm, cap, s_depth);
    __syncthreads();
    if (threadIdx.x <= kDepthMax && s_depth[threadIdx.x]) atomicAdd(&cnt->depth_nodes[threadIdx.x], s_depth[threadIdx.x]);
}

__global__ void k_node_cap_check(TreeCounts* cnt, int cap, uint32_t* status) {
    if (cnt->total_nodes > cap) {
        raise_status(status, GF_ERR_CAPACITY);
        cnt->total_nodes = 0;
    }
}

// Node kernels: launched over [0, span); the live node count is *nn_dev.
__device__ __forceinline__ int live_nodes(int span, const int* nn_dev) {
    return nn_dev ? min(span, *nn_dev) : span;
}

// Positions (and masses) in tree order: p4 = float32 position and mass, plo = the float32
// remainders. The build saves the float64 positions in tree order (xsave); a refit measures each
// particle's displacement since the build against them (xbuild, tree order: coalesced reads).
__global__ void k_gather(int n, const int* __restrict__ perm, const double* __restrict__ pos,
                         const double* __restrict__ mass, const double* __restrict__ xbuild,
                         float4* __restrict__ p4, float* __restrict__ pdisp, float4* __restrict__ plo,
                         int disp32 = 0, double* __restrict__ xsave = nullptr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = perm[i];
    const double x = pos[3 * size_t(j)], y = pos[3 * size_t(j) + 1], z = pos[3 * size_t(j) + 2];
    const double m = mass ? mass[j] : 1.0;
    const float fx = float(x), fy = float(y), fz = float(z);
    p4[i] = make_float4(fx, fy, fz, float(m));
    if (plo) plo[i] = make_float4(float(x - double(fx)), float(y - double(fy)), float(z - double(fz)), 0.f);
    if (xsave) {
        xsave[3 * size_t(i)] = x;
        xsave[3 * size_t(i) + 1] = y;
        xsave[3 * size_t(i) + 2] = z;
    }
    if (pdisp && disp32) {  // mixed form: float64 differences, float32 length
        const float dx = float(x - xbuild[3 * size_t(i)]), dy = float(y - xbuild[3 * size_t(i) + 1]),
                    dz = float(z - xbuild[3 * size_t(i) + 2]);
        pdisp[i] = m > 0 ? sqrtf(dx * dx + dy * dy + dz * dz) : 0.0f;
    } else if (pdisp) {  // refit: displacement since the build (cpp/nbody.cpp:273-275)
        const double dx = __dsub_rn(x, xbuild[3 * size_t(i)]);
        const double dy = __dsub_rn(y, xbuild[3 * size_t(i) + 1]);
        const double dz = __dsub_rn(z, xbuild[3 * size_t(i) + 2]);
        pdisp[i] = m > 0 ? float(__dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                                                      __dmul_rn(dz, dz))))
                         : 0.0f;
    }
}

// ---------------------------------------------------------------------------- moments

// Relative opening radius of a quadrupole node: the walk accepts the node for a group sphere
// (centre c, radius R) when |com - c| - R exceeds rho * (alpha * min |a_old|)^(-1/5), i.e. when
// the octupole-order estimate M b^3 / r^5 of the truncation error is at most alpha times the
// group's smallest previous acceleration (the relative criterion of Springel 2005, GADGET-2,
// to the next order). b bounds the distance of the node's mass from its centre of mass.
// rho = M^(1/5) b^(3/5) in logarithms, so no intermediate overflows in float32. The second
// radius, (M b^2)^(1/4), is the quadrupole-order one: beyond rho_q (alpha_q a_min)^(-1/4) the
// node's quadrupole term itself is below alpha_q a_min and the walk takes its monopole alone.
__device__ __forceinline__ float2 rel_radii(float m, float ox, float oy, float oz, float half) {
    if (!(m > 0.f)) return make_float2(0.f, 0.f);
    const float lm = log2f(m), lb = log2f(sqrtf(ox * ox + oy * oy + oz * oz) + 1.7320508f * half);
    return make_float2(exp2f(0.2f * lm + 0.6f * lb), exp2f(0.25f * lm + 0.5f * lb));
}

// Traceless quadrupole Q = sum m (3 d d - |d|^2 I) and trace T = sum m |d|^2 about a centre.
struct QuadSum {
    KahanF xx, yy, xy, xz, yz, tr;
    __device__ __forceinline__ void point(float m, float dx, float dy, float dz) {
        const float r2 = dx * dx + dy * dy + dz * dz;
        xx.add(m * (3.f * dx * dx - r2));
        yy.add(m * (3.f * dy * dy - r2));
        xy.add(3.f * m * dx * dy);
        xz.add(3.f * m * dx * dz);
        yz.add(3.f * m * dy * dz);
        tr.add(m * r2);
    }
};

// Mixed form: monopole and traceless quadrupole in one bottom-up pass, float32 with
// Kahan-compensated sums, directly in the breadth-first walk layout (the children of a node
// are contiguous there, in octant order, so a parent reads them with independent loads). A
// leaf sums its particles; the last child to finish a parent (arrival counter) combines the
// children's masses and centres, then their quadrupoles shifted by the parallel-axis term.
// open_r = 2 (half + displacement) / theta + |com - cell centre| in float32, and the relative
// opening radii. Used by the build (pdisp null: no displacement) and by the refit (pdisp: the
// displacement of each particle since the build). Thread per breadth-first node.
struct RefitBfsArgs {
    int span;
    const int* nn_dev;
    float theta;
    const int* wparent;
    const float4* wgeo;
    int* counter;
    float4* wa;   // com, m
    float4* wb;   // open_r, first, code, rho
    float4* wq;   // Qxx, Qyy, Qxy, Qxz
    float2* wt;   // Qyz, T
    float* wrq;   // quadrupole-order radius
    float* ndisp; // breadth-first
    const float4* p4;
    const float* pdisp;  // null: no displacement (the build)
};

// Writes node b's monopole, opening radii and displacement bound (g: its cell, loaded early).
__device__ __forceinline__ void finalize_bfs(const RefitBfsArgs& A, int b, const float4 g, float m, float cx,
                                             float cy, float cz, float dm) {
    A.wa[b] = make_float4(cx, cy, cz, m);
    const float ox = cx - g.x, oy = cy - g.y, oz = cz - g.z;
    A.wb[b].x = 2.f * (g.w + dm) / A.theta + sqrtf(ox * ox + oy * oy + oz * oz);
    const float2 rr = rel_radii(m, ox, oy, oz, g.w + dm);
    A.wb[b].w = rr.x;
    A.wrq[b] = rr.y;
    A.ndisp[b] = dm;
}

__device__ __forceinline__ float4 leaf_centre(const KahanF& M, const KahanF& sx, const KahanF& sy, const KahanF& sz) {
    const float inv = M.s > 0.f ? 1.f / M.s : 0.f;
    return make_float4(sx.s * inv, sy.s * inv, sz.s * inv, M.s);
}

// Compensated sum over the 8 lanes of an aligned lane group (all 32 lanes take part): Knuth's
// two-sum at each of the three butterfly steps, the rounding errors carried in a second float.
// Both lanes of a pair compute the same bits, so the 8 lanes end with identical values.
__device__ __forceinline__ float group8_sum(float v) {
    float s = v, e = 0.f;
#pragma unroll
    for (int off = 4; off; off >>= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, s, off);
        const float oe = __shfl_xor_sync(0xffffffffu, e, off);
        const float t = s + o;
        const float bp = t - s;
        const float err = (s - (t - bp)) + (o - bp);
        s = t;
        e = (e + oe) + err;
    }
    return s + e;
}

__device__ __forceinline__ float group8_max(float v) {
#pragma unroll
    for (int off = 4; off; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// The arrival of a finished node at its parent (arrival counter, parent's child count nc, loaded
// before the atomic). The counter is an acquire-release atomic: it publishes this thread's
// records of the node and, for the last child, makes its siblings' records visible. Returns
// whether this arrival completed the parent; the counter is then back at zero for the next pass.
__device__ __forceinline__ bool arrive(int* counter, int nc) {
    if (atom_add_acq_rel(counter, 1) != nc - 1) return false;
    *counter = 0;
    return true;
}

// Child range {first, count} of node b from its walk record (structure fields, constant here).
__device__ __forceinline__ int2 child_range(const float4* wb, int b) {
    const int* pbi = reinterpret_cast<const int*>(wb) + 4 * size_t(b);
    return make_int2(__ldg(pbi + 1), __ldg(pbi + 2));
}

// The climb of a warp's completed parents (p, child range pc; -1: none). Each round the four
// groups of 8 lanes take up to four of them (group k the one held by the k-th lane holding one).
// combine(q, first child, children, c), called by all lanes (q = -1 for a group without a parent),
// sums the children's records, lane c of a group child c, and its lane 0 writes the parent; then
// lane 0 arrives at the grandparent, and a completed grandparent goes back to the lane that held
// the parent. Each round serves at least one parent and a parent precedes its children in the
// layout, so the loop ends. kSingle: parents of one child are left to single(p, child), by each
// lane for itself, all of a warp's side by side.
template <bool kSingle, class Combine, class Single>
__device__ __forceinline__ void climb_parents(int p, int2 pc, const int* __restrict__ wparent, const float4* wb,
                                              int* counter, Combine combine, Single single) {
    const int lane = threadIdx.x & 31;
    const int grp = lane >> 3, c = lane & 7;
    for (;;) {
        if (kSingle && p >= 0 && pc.y == 1) {
            const int gp = __ldg(&wparent[p]);
            const int2 gc = gp >= 0 ? child_range(wb, gp) : make_int2(0, 0);
            single(p, pc.x);
            // (an only child: nobody else arrives at its parent)
            p = gp >= 0 && (gc.y == 1 || arrive(&counter[gp], gc.y)) ? gp : -1;
            pc = gc;
        }
        const bool shared = p >= 0 && !(kSingle && pc.y == 1);
        const unsigned pend = __ballot_sync(0xffffffffu, shared);
        if (pend == 0u) {
            if (kSingle && __any_sync(0xffffffffu, p >= 0)) continue;
            break;
        }
        unsigned rest = pend;  // the holders from the grp-th on (lowest lanes first)
        for (int k = 0; k < grp; ++k) rest &= rest - 1u;
        const int src = rest ? __ffs(int(rest)) - 1 : 0;
        int q = __shfl_sync(0xffffffffu, p, src);
        const int q0 = __shfl_sync(0xffffffffu, pc.x, src);
        const int qn = __shfl_sync(0xffffffffu, pc.y, src);
        if (!rest) q = -1;
        __syncwarp();  // orders the holder's acquiring arrival before its group's loads
        int gp = -1;
        int2 gc = make_int2(0, 0);
        if (q >= 0 && c == 0) {
            gp = __ldg(&wparent[q]);
            if (gp >= 0) gc = child_range(wb, gp);
        }
        combine(q, q0, qn, c);
        int np = -1;
        if (gp >= 0 && arrive(&counter[gp], gc.y)) np = gp;
        // back to the holders: the k-th holder (k < 4) was served by group k
        const int rank = __popc(pend & lanemask_lt());
        const int from = 8 * min(rank, 3);
        const int np_ = __shfl_sync(0xffffffffu, np, from);
        const int nc0_ = __shfl_sync(0xffffffffu, gc.x, from);
        const int nnc_ = __shfl_sync(0xffffffffu, gc.y, from);
        if (shared && rank < 4) {
            p = np_;
            pc = make_int2(nc0_, nnc_);
        }
    }
}

// Threads take the nodes from the end of the breadth-first layout (the deepest first), so the
// deep subtrees are summed and climbed by the first blocks and the last blocks hold the shallow
// nodes, whose climbs to the root are short. A leaf's thread sums its particles (sequential
// Kahan sums); a parent is combined by a group of 8 lanes of the warp whose lane completed it,
// lane c loading child c, so that all of a parent's records arrive with one memory latency and
// the sums are pairwise with compensation. 64 registers: 4 blocks per SM.
__global__ void __launch_bounds__(kThreads, 4) k_refit_bfs_quad32(RefitBfsArgs A) {
    const int b = live_nodes(A.span, A.nn_dev) - 1 - int(blockIdx.x * blockDim.x + threadIdx.x);
    int p = -1;  // a parent that this lane's arrival completed, its child range
    int2 pc = make_int2(0, 0);
    const float4 wb = b >= 0 ? A.wb[b] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int first = __float_as_int(wb.y), code = __float_as_int(wb.z);
    if (b >= 0 && code < 0) {  // a leaf (internal nodes are reached by the climb)
        const int cnt = -code;
        const float4 g = __ldg(&A.wgeo[b]);
        const int par = __ldg(&A.wparent[b]);
        const int2 cr = par >= 0 ? child_range(A.wb, par) : make_int2(0, 0);
        QuadSum S;
        if (cnt <= kLeafMax) {  // the leaf's particles loaded once, together (one memory latency)
            float4 pp[kLeafMax];
            float pd[kLeafMax];
#pragma unroll
            for (int t = 0; t < kLeafMax; ++t) {
                pp[t] = t < cnt ? A.p4[first + t] : make_float4(0.f, 0.f, 0.f, 0.f);
                pd[t] = t < cnt && A.pdisp ? A.pdisp[first + t] : 0.f;
            }
            KahanF M, sx, sy, sz;
            float dm = 0.f;
#pragma unroll
            for (int t = 0; t < kLeafMax; ++t) {
                if (t < cnt) {
                    M.add(pp[t].w);
                    sx.add(pp[t].w * pp[t].x);
                    sy.add(pp[t].w * pp[t].y);
                    sz.add(pp[t].w * pp[t].z);
                    dm = fmaxf(dm, pd[t]);
                }
            }
            const float4 c = leaf_centre(M, sx, sy, sz);
            finalize_bfs(A, b, g, c.w, c.x, c.y, c.z, dm);
#pragma unroll
            for (int t = 0; t < kLeafMax; ++t)
                if (t < cnt) S.point(pp[t].w, pp[t].x - c.x, pp[t].y - c.y, pp[t].z - c.z);
        } else {  // depth-48 leaves of coincident points
            KahanF M, sx, sy, sz;
            float dm = 0.f;
            for (int i = first; i < first + cnt; ++i) {
                const float4 q = A.p4[i];
                M.add(q.w);
                sx.add(q.w * q.x);
                sy.add(q.w * q.y);
                sz.add(q.w * q.z);
                if (A.pdisp) dm = fmaxf(dm, A.pdisp[i]);
            }
            const float4 c = leaf_centre(M, sx, sy, sz);
            finalize_bfs(A, b, g, c.w, c.x, c.y, c.z, dm);
            for (int i = first; i < first + cnt; ++i) {
                const float4 q = A.p4[i];
                S.point(q.w, q.x - c.x, q.y - c.y, q.z - c.z);
            }
        }
        A.wq[b] = make_float4(S.xx.s, S.yy.s, S.xy.s, S.xz.s);
        A.wt[b] = make_float2(S.yz.s, S.tr.s);
        if (par >= 0 && arrive(&A.counter[par], cr.y)) {
            p = par;
            pc = cr;
        }
    }
    climb_parents<false>(p, pc, A.wparent, A.wb, A.counter, [&](int q, int q0, int qn, int c) {
        float4 cm = make_float4(0.f, 0.f, 0.f, 0.f), qc = cm, g = cm;
        float2 yt = make_float2(0.f, 0.f);
        float dmc = 0.f;
        if (q >= 0) {
            if (c < qn) {
                cm = __ldcg(&A.wa[q0 + c]);
                dmc = __ldcg(&A.ndisp[q0 + c]);
                qc = __ldcg(&A.wq[q0 + c]);
                yt = __ldcg(&A.wt[q0 + c]);
            }
            if (c == 0) g = __ldg(&A.wgeo[q]);
        }
        // children past qn (and groups without a parent) add zeros
        const float M = group8_sum(cm.w);
        const float sx = group8_sum(cm.w * cm.x), sy = group8_sum(cm.w * cm.y), sz = group8_sum(cm.w * cm.z);
        const float dm = group8_max(dmc);
        const float inv = M > 0.f ? 1.f / M : 0.f;
        const float cx = sx * inv, cy = sy * inv, cz = sz * inv;
        const float dx = cm.x - cx, dy = cm.y - cy, dz = cm.z - cz;
        const float r2 = dx * dx + dy * dy + dz * dz, m = cm.w;
        const float xx = group8_sum(qc.x + m * (3.f * dx * dx - r2));
        const float yy = group8_sum(qc.y + m * (3.f * dy * dy - r2));
        const float xy = group8_sum(qc.z + 3.f * m * dx * dy);
        const float xz = group8_sum(qc.w + 3.f * m * dx * dz);
        const float yz = group8_sum(yt.x + 3.f * m * dy * dz);
        const float tr = group8_sum(yt.y + m * r2);
        if (q >= 0 && c == 0) {
            finalize_bfs(A, q, g, M, cx, cy, cz, dm);
            A.wq[q] = make_float4(xx, yy, xy, xz);
            A.wt[q] = make_float2(yz, tr);
        }
    }, [](int, int) {});
}

// Plain form (the reference's arithmetic): monopoles in float64 sums, rounded to the float32 node
// records (cpp/nbody.cpp:98-131; refit :285-303), in the same bottom-up pass over the breadth-first
// walk layout. Bound by the float64 pipe and, at small counts, by the chain of arrivals: a leaf's
// thread sums its particles (4 or 7 float64 instructions each), a parent is combined by 8 lanes, one
// child each. (One thread climbing per subtree and summing its children one after another kept 9 of
// 32 lanes active: build passes of 10k / 150k particles 64 / 123 us, now 43 / 77 us; refits of
// 200k 126 -> 72 us; gravity of the 4M cloud 7.07 -> 6.60 ms.)
struct Moments64Args {
    int span;
    const int* nn_dev;
    bool refit;
    float theta;
    const RootBox* root;    // open0: the root's 2 half / theta
    const int* wparent;
    const float4* wgeo;     // refit: float32 centre + half
    const int* dfs;         // build: depth-first id of a breadth-first node
    const double4* cd;      // build: float64 centre + half, depth-first
    int* counter;
    float4* wa;             // com, m
    float4* wb;             // open_r, first, code, 0
    float* ndisp;           // refit
    const int* perm;        // build: particles in float64
    const double* xbuild;
    const double* mass;
    const float4* p4;       // refit: the float32 copies
    const float* pdisp;
};

// 1/M of a node's mass (0 for a massless node).
__device__ __forceinline__ double inverse_mass(double M) {
    return in_inverse_range(M) ? inverse(M) : M > 0 ? __drcp_rn(M) : 0.0;
}

// open_r of a node whose centre of mass lies at squared distance o2 from its cell's centre.
__device__ __forceinline__ float open_radius(const Moments64Args& A, double half, double o2, float dm) {
    double first;
    if (!A.refit) {
        // 2 half / theta (cpp/nbody.cpp:104-106): half is the root's, halved depth times, so the
        // quotient is the root's scaled by the same power of two (both exponents drop alike)
        const double open0 = A.root->open0;
        const int drop = __double2hiint(A.root->half) - __double2hiint(half);
        first = __hiloint2double(__double2hiint(open0) - drop, __double2loint(open0));
    } else {  // cpp/nbody.cpp:301-303: the first term is evaluated in float32
        first = double(__fdiv_rn(__fmul_rn(2.0f, __fadd_rn(float(half), dm)), A.theta));
    }
    return float(first + root(o2));
}

// The centre and half of node b's cell, as the pass measures against them.
__device__ __forceinline__ double4 cell64(const Moments64Args& A, int b) {
    if (!A.refit) return A.cd[A.dfs[b]];
    const float4 g = __ldg(&A.wgeo[b]);
    return make_double4(double(g.x), double(g.y), double(g.z), double(g.w));
}

__global__ void __launch_bounds__(kThreads) k_moments64(Moments64Args A) {
    const int b = live_nodes(A.span, A.nn_dev) - 1 - int(blockIdx.x * blockDim.x + threadIdx.x);
    int p = -1;
    int2 pc = make_int2(0, 0);
    const float4 wb = b >= 0 ? A.wb[b] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int first = __float_as_int(wb.y), code = __float_as_int(wb.z);
    if (b >= 0 && code < 0) {  // a leaf: its particles in order (cpp/nbody.cpp:124-131, refit :285-289)
        const double4 g = cell64(A, b);
        const int par = __ldg(&A.wparent[b]);
        const int2 cr = par >= 0 ? child_range(A.wb, par) : make_int2(0, 0);
        double M = 0, sx = 0, sy = 0, sz = 0;
        float dm = 0.f;
        for (int base = 0; base < -code; base += kLeafMax) {  // once, but for leaves at the depth limit
            double4 pm[kLeafMax];
            float pd[kLeafMax];
#pragma unroll
            for (int t = 0; t < kLeafMax; ++t) {  // loaded together
                pm[t] = make_double4(0.0, 0.0, 0.0, 0.0);
                pd[t] = 0.f;
                if (base + t < -code) {
                    const int i = first + base + t;
                    if (!A.refit) {
                        pm[t] = make_double4(A.xbuild[3 * size_t(i)], A.xbuild[3 * size_t(i) + 1],
                                             A.xbuild[3 * size_t(i) + 2], A.mass ? A.mass[A.perm[i]] : 1.0);
                    } else {
                        const float4 q = A.p4[i];
                        pm[t] = make_double4(double(q.x), double(q.y), double(q.z), double(q.w));
                        pd[t] = A.pdisp[i];
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < kLeafMax; ++t) {
                if (base + t < -code) {
                    M += pm[t].w;
                    if (A.refit) {  // (exact products: fused or not, the same sums)
                        sx = fma(pm[t].w, pm[t].x, sx);
                        sy = fma(pm[t].w, pm[t].y, sy);
                        sz = fma(pm[t].w, pm[t].z, sz);
                    } else {
                        sx = __dadd_rn(sx, __dmul_rn(pm[t].w, pm[t].x));
                        sy = __dadd_rn(sy, __dmul_rn(pm[t].w, pm[t].y));
                        sz = __dadd_rn(sz, __dmul_rn(pm[t].w, pm[t].z));
                    }
                    dm = fmaxf(dm, pd[t]);
                }
            }
        }
        const double inv = inverse_mass(M);
        const double mx = sx * inv, my = sy * inv, mz = sz * inv;
        A.wa[b] = make_float4(float(mx), float(my), float(mz), float(M));
        const double ox = mx - g.x, oy = my - g.y, oz = mz - g.z;
        A.wb[b].x = open_radius(A, g.w, fma(ox, ox, fma(oy, oy, oz * oz)), dm);
        if (A.refit) A.ndisp[b] = dm;
        if (par >= 0 && arrive(&A.counter[par], cr.y)) {
            p = par;
            pc = cr;
        }
    }
    climb_parents<true>(p, pc, A.wparent, A.wb, A.counter, [&](int q, int q0, int qn, int c) {
        // Lane c: quantity c & 3 (0 the mass, 1..3 mass times coordinate) of the children 4 (c >> 2)
        // .. + 3, so that one instruction serves all four sums (the products of float32 values are
        // exact in float64: a fused multiply-add rounds as the reference's product and sum).
        const int quantity = c & 3, k0 = c & 4;
        const float* w = reinterpret_cast<const float*>(A.wa);
        float cm[4], cx[4], dm = 0.f;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            cm[t] = cx[t] = 0.f;
            if (q >= 0 && k0 + t < qn) {
                const size_t r = 4 * size_t(q0 + k0 + t);
                cm[t] = __ldcg(w + r + 3);
                cx[t] = quantity ? __ldcg(w + r + (quantity - 1)) : 1.f;
                if (A.refit) dm = fmaxf(dm, __ldcg(&A.ndisp[q0 + k0 + t]));
            }
        }
        double4 g = make_double4(0.0, 0.0, 0.0, 0.0);
        if (q >= 0) g = cell64(A, q);
        double s = 0.0;
#pragma unroll
        for (int t = 0; t < 4; ++t) s = fma(double(cm[t]), double(cx[t]), s);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        dm = fmaxf(dm, __shfl_xor_sync(0xffffffffu, dm, 4));
        const double M = __shfl_sync(0xffffffffu, s, 0, 8);
        const double com = __dmul_rn(s, inverse_mass(M));  // lanes 1..3
        const double o = __dsub_rn(com, quantity == 1 ? g.x : quantity == 2 ? g.y : g.z);
        const double oo = o * o;
        const double o2 = __shfl_sync(0xffffffffu, oo, 1, 8) + __shfl_sync(0xffffffffu, oo, 2, 8) +
                          __shfl_sync(0xffffffffu, oo, 3, 8);
        if (q >= 0 && c < 4) reinterpret_cast<float*>(A.wa)[4 * size_t(q) + (c ? c - 1 : 3)] = float(c ? com : M);
        if (q >= 0 && c == 0) {
            A.wb[q].x = open_radius(A, g.w, o2, dm);
            if (A.refit) A.ndisp[q] = dm;
        }
        __syncwarp();  // the group's writes before its lane 0 arrives at the grandparent
    }, [&](int p, int child) {
        // One of a chain of cells with one child each, as above coincident or tightly grouped particles, with
        // combine's operations. (A combine of eight lanes serves four of a warp's up to 32 chains at
        // a time: gravity of 2,000 particles in coincident groups of 20 1455 us instead of 375, the pass
        // 1203 instead of 120; of 28k in groups 10^-6 wide 544 instead of 469.)
        const float4 r = __ldcg(&A.wa[child]);
        const float dm = A.refit ? __ldcg(&A.ndisp[child]) : 0.f;
        const double4 g = cell64(A, p);
        const double M = fma(double(r.w), 1.0, 0.0), inv = inverse_mass(M);
        const double mx = __dmul_rn(fma(double(r.w), double(r.x), 0.0), inv);
        const double my = __dmul_rn(fma(double(r.w), double(r.y), 0.0), inv);
        const double mz = __dmul_rn(fma(double(r.w), double(r.z), 0.0), inv);
        const double ox = __dsub_rn(mx, g.x), oy = __dsub_rn(my, g.y), oz = __dsub_rn(mz, g.z);
        A.wa[p] = make_float4(float(mx), float(my), float(mz), float(M));
        A.wb[p].x = open_radius(
            A, g.w, __dadd_rn(__dadd_rn(__dmul_rn(ox, ox), __dmul_rn(oy, oy)), __dmul_rn(oz, oz)), dm);
        if (A.refit) A.ndisp[p] = dm;
    });
}

// ---------------------------------------------------------------------------- groups + layout

// Walk groups: the shallowest nodes holding at most gmax particles, in depth-first order. The same
// pass counts every node's children and clears its arrival counter.
struct GroupScan {
    const int* nn_dev;
    int span, gmax;
    const int4* n_i4;
    const int* parent;
    int* nchild;
    int* counter;
    int* groups;
    __device__ int first(int k) const {
        if (k >= live_nodes(span, nn_dev)) return 0;  // past the live nodes (the scan covers span)
        const int4 q = n_i4[k];
        int c = 0;
        if (!(q.w & 1)) {
            for (int ch = k + 1; ch < q.z && c < 8; ch = n_i4[ch].z) ++c;  // <= 8 children
        }
        nchild[k] = c;
        counter[k] = 0;
        return again(k);
    }
    __device__ int again(int k) const {
        if (k >= live_nodes(span, nn_dev)) return 0;
        const int4 q = n_i4[k];
        const bool candidate = q.y <= gmax || (q.w & 1);
        const int p = parent[k];
        return candidate && (p < 0 || n_i4[p].y > gmax) ? 1 : 0;
    }
    __device__ void put(int k, int v, int ex) const {
        if (v) groups[ex] = k;
    }
};

// Breadth-first numbering: a stable counting sort by depth (the nodes per depth are counted by the
// emission). One sweep like a pass of the radix sort, over kDepthBins digits: tiles in ticket
// order, a thread per depth adds up the tiles before its own by look-back. bfs[k] = rank of node
// k, dfs[rank] = k.
constexpr int kBfsThreads = 256, kBfsItems = 4, kBfsTile = kBfsThreads * kBfsItems;
constexpr int kBfsWarps = kBfsThreads / 32;
constexpr int kDepthBins = 64;
constexpr unsigned kBfsOwn = 1u << 30, kBfsAll = 2u << 30, kBfsValue = (1u << 30) - 1;
constexpr long kBfsSpinMax = 1l << 20;  // bounded waits (a waited-on tile is always running)

__global__ void __launch_bounds__(kBfsThreads) k_bfs_rank(int span, TreeCounts* cnt, const int4* __restrict__ n_i4,
                                                          unsigned* __restrict__ status, int* __restrict__ bfs,
                                                          int* __restrict__ dfs, uint32_t* err) {
    __shared__ int s_cnt[kBfsWarps][kDepthBins];
    __shared__ int s_base[kDepthBins];
    __shared__ int s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = lanemask_lt();
    if (tid == 0) s_tile = atomicAdd(&cnt->bfs_ticket, 1);
    for (int t = tid; t < kBfsWarps * kDepthBins; t += kBfsThreads) (&s_cnt[0][0])[t] = 0;
    __syncthreads();
    const int nodes = live_nodes(span, &cnt->total_nodes);
    const int tile = s_tile;
    const int base = tile * kBfsTile + warp * 32 * kBfsItems;
    if (tile * kBfsTile >= nodes) return;  // nothing here, and no later tile waits for it
    int d[kBfsItems], rk[kBfsItems];
#pragma unroll
    for (int s = 0; s < kBfsItems; ++s) {
        const int k = base + 32 * s + lane;
        d[s] = k < nodes ? n_i4[k].w >> 8 : kDepthBins;
    }
#pragma unroll
    for (int s = 0; s < kBfsItems; ++s) {
        const bool ok = d[s] < kDepthBins;
        const unsigned peers = __match_any_sync(0xffffffffu, d[s]);
        const int before = ok ? s_cnt[warp][d[s]] : 0;
        rk[s] = before + __popc(peers & lt);
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) s_cnt[warp][d[s]] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    if (tid < kDepthBins) {
        int run = 0;
        for (int w = 0; w < kBfsWarps; ++w) {
            const int c = s_cnt[w][tid];
            s_cnt[w][tid] = run;
            run += c;
        }
        int shallower = 0;  // nodes of smaller depths
        for (int t = 0; t < tid && t <= kDepthMax; ++t) shallower += cnt->depth_nodes[t];
        unsigned* mine = status + size_t(tile) * kDepthBins + tid;
        int excl = 0;
        if (tile == 0) {
            st_relaxed(mine, kBfsAll | unsigned(run));
        } else {
            st_relaxed(mine, kBfsOwn | unsigned(run));
            long polls = 0;
            for (int j = tile - 1; j >= 0;) {
                const unsigned w = ld_relaxed(status + size_t(j) * kDepthBins + tid);
                if ((w & ~kBfsValue) == 0u) {  // not there yet
                    if (++polls < kBfsSpinMax) continue;
                    raise_status(err, GF_ERR_TIMEOUT);
                    break;
                }
                excl += int(w & kBfsValue);
                if (w & kBfsAll) break;
                --j;
            }
            st_relaxed(mine, kBfsAll | unsigned(excl + run));
        }
        s_base[tid] = shallower + excl;
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kBfsItems; ++s) {
        const int k = base + 32 * s + lane;
        if (k < nodes) {
            const int b = s_base[d[s]] + s_cnt[warp][d[s]] + rk[s];
            bfs[k] = b;
            dfs[b] = k;
        }
    }
}

// The structure of the breadth-first layout (the moments passes write the rest afterwards).
__global__ void k_walk_fill(int nn, const int4* __restrict__ n_i4, const int* __restrict__ nchild,
                            const int* __restrict__ bfs, const float4* __restrict__ geo, float4* __restrict__ wb,
                            float4* __restrict__ wgeo, int* __restrict__ leaf_of,
                            const int* __restrict__ parent, int* __restrict__ wparent, const int* __restrict__ nn_dev) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= live_nodes(nn, nn_dev)) return;
    const int4 q = n_i4[k];
    const int b = bfs[k];
    int first, code;
    if (q.w & 1) {
        first = q.x;
        code = -q.y;
        if (leaf_of)
            for (int i = q.x; i < q.x + q.y; ++i) leaf_of[i] = b;
    } else {
        first = bfs[k + 1];
        code = nchild[k];
    }
    wb[b] = make_float4(0.f, __int_as_float(first), __int_as_float(code), 0.f);
    wgeo[b] = geo[k];
    wparent[b] = parent[k] < 0 ? -1 : bfs[parent[k]];
}

// ---------------------------------------------------------------------------- deep cells

// Positions of cells that still hold > 8 particles at level 21 get extension keys.
// Extension keys are read (by cpl and digit) only at positions whose level-21 key equals a
// neighbour's in sorted order, so the others are skipped: they hold stale words that nothing
// reads. Shared positions outside deep runs get zeros.
__global__ void k_deep_keys(int n, const uint64_t* __restrict__ k0, const int* __restrict__ perm,
                            const double* __restrict__ pos, const RootBox* __restrict__ rootp,
                            uint64_t* __restrict__ k1, uint64_t* __restrict__ k2,
                            int* __restrict__ starts, int* __restrict__ nstarts, int L) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t ki = k0[i];
    if (!((i > 0 && k0[i - 1] == ki) || (i + 1 < n && k0[i + 1] == ki))) return;
    bool deep = false;
    for (int j = max(0, i - L); j <= i && !deep; ++j)
        deep = j + L < n && k0[j] == k0[j + L];
    uint64_t a = 0, b = 0;
    if (deep) {
        const RootBox R = *rootp;
        const int p = perm[i];
        uint64_t c0;
        exact_keys(pos[3 * size_t(p)], pos[3 * size_t(p) + 1], pos[3 * size_t(p) + 2], R, kDepthMax, c0, a, b);
        if (i == 0 || k0[i - 1] != k0[i]) starts[atomicAdd(nstarts, 1)] = i;
    }
    k1[i] = a;
    k2[i] = b;
}

// One block per deep run: stable sort of (k1, k2) inside the run (ties keep index order).
__global__ void k_deep_sort(int n, const uint64_t* __restrict__ k0, uint64_t* __restrict__ k1,
                            uint64_t* __restrict__ k2, int* __restrict__ perm,
                            const int* __restrict__ starts, const int* __restrict__ nstarts,
                            uint32_t* status) {
    extern __shared__ unsigned char smem[];
    uint64_t* s1 = reinterpret_cast<uint64_t*>(smem);
    uint64_t* s2 = s1 + kDeepRunMax;
    int* sp = reinterpret_cast<int*>(s2 + kDeepRunMax);
    for (int r = blockIdx.x; r < *nstarts; r += gridDim.x) {
        const int b = starts[r];
        __shared__ int s_len;
        if (threadIdx.x == 0) {
            int e = b + 1;
            while (e < n && k0[e] == k0[b]) ++e;
            s_len = e - b;
        }
        __syncthreads();
        const int len = s_len;
        if (len > kDeepRunMax) {
            // sorted already when every extension key is equal (coincident particles)
            bool sorted = true;
            for (int i = b + 1 + threadIdx.x; i < b + len; i += blockDim.x)
                if (k1[i] < k1[i - 1] || (k1[i] == k1[i - 1] && k2[i] < k2[i - 1])) sorted = false;
            if (__syncthreads_or(!sorted) && threadIdx.x == 0) raise_status(status, GF_ERR_DEEP_CELL);
            __syncthreads();
            continue;
        }
        int P = 1;
        while (P < len) P <<= 1;
        for (int t = threadIdx.x; t < P; t += blockDim.x) {
            if (t < len) {
                s1[t] = k1[b + t];
                s2[t] = k2[b + t];
                sp[t] = perm[b + t];
            } else {
                s1[t] = ~0ull;
                s2[t] = ~0ull;
                sp[t] = 0x7fffffff;
            }
        }
        __syncthreads();
        for (int size = 2; size <= P; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = threadIdx.x; t < P; t += blockDim.x) {
                    const int u = t ^ stride;
                    if (u > t) {
                        const bool up = (t & size) == 0;
                        const bool gt = s1[t] > s1[u] || (s1[t] == s1[u] && (s2[t] > s2[u] ||
                                                          (s2[t] == s2[u] && sp[t] > sp[u])));
                        if (gt == up) {
                            uint64_t x = s1[t]; s1[t] = s1[u]; s1[u] = x;
                            x = s2[t]; s2[t] = s2[u]; s2[u] = x;
                            const int y = sp[t]; sp[t] = sp[u]; sp[u] = y;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int t = threadIdx.x; t < len; t += blockDim.x) {
            k1[b + t] = s1[t];
            k2[b + t] = s2[t];
            perm[b + t] = sp[t];
        }
        __syncthreads();
    }
}

}  // namespace

// ------------------------------------------------------------------------------- host side

static Octree g_tree;
Octree& gravity_tree() { return g_tree; }
static Octree* g_last_walked = nullptr;
Octree*& last_walked() { return g_last_walked; }

void Octree::reserve_graph_build() {
    if (!valid || n <= 0) throw Error(GF_ERR_ARG, "a captured rebuild needs a regular build first");
    key1.get<uint64_t>(n);
    key2.get<uint64_t>(n);
    pdisp.get<float>(n);
    node_owner.get<int>(node_cap);
    work.get<int4>(std::max(size_t(node_cap), size_t(n)) + 1);
    sphere.get<float4>(std::max(size_t(node_cap), size_t(n)) + 1);
    if (quad) item_gam.get<float2>(std::max(size_t(node_cap), size_t(n)) + 1);
    gweight.get<int>(std::max(node_cap, 1));
    gflag.get<int>(std::max(node_cap, 1));
    gscan.get<int>(std::max(node_cap, 1));
    reserve_scan_sort(std::max(n, node_cap), &scratch);
    deep_sort_attr();
}

void Octree::deep_sort_attr() {
    static bool attr = false;
    if (!attr) {
        const size_t sm = size_t(kDeepRunMax) * (2 * sizeof(uint64_t) + sizeof(int));
        GF_CUDA(cudaFuncSetAttribute(k_deep_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
        attr = true;
    }
}

void Octree::small_sort(const double* pos, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        GF_CUDA(cudaFuncSetAttribute(k_small_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(small_sort_smem(kSmallMaxPer))));
        attr = true;
    }
    const int m = std::max(2, div_up(n, kSmallCtas));  // at least 2: the reciprocal then has 32 bits
    // floor(t / m) = mulhi(t, div_m) for every t below kSmallMax: t m < 2^32
    const unsigned div_m = unsigned((0x100000000ull + m - 1) / m);
    k_small_sort<<<kSmallCtas, kSmallThreads, small_sort_smem(m), s>>>(
        pos, n, m, div_m, double(theta_f), root.as<RootBox>(), key.as<uint64_t>(), perm.as<int>(),
        counts.as<TreeCounts>(), ctx().d_status);
    GF_CHECK_LAUNCH();
}

void Octree::build(int n_, const double* pos, const double* mass, double theta, cudaStream_t s, bool graph_safe) {
    Context& C = ctx();
    ProfScope ps(want_knn ? kStKnnTree : kStTreeBuild, s);
    if (graph_safe && (!valid || n != n_ || node_cap <= 0))
        throw Error(GF_ERR_ARG, "a captured rebuild needs a regular build of the same particle set first");
    n = n_;
    theta_f = float(theta);
    if (!graph_safe) valid = false;
    if (!h_counts) GF_CUDA(cudaMallocHost(&h_counts, sizeof(TreeCounts)));
    TreeCounts* cnt = counts.get<TreeCounts>(1);
    RootBox* R = root.get<RootBox>(1);
    const int grid = div_up(n, kThreads);
    uint64_t* k0 = key.get<uint64_t>(n);
    int* pm = perm.get<int>(n);
    key_alt.get<uint64_t>(n);
    perm_alt.get<int>(n);
    const int nparts = std::min(4 * C.sms, std::max(1, grid));
    int* nb = nbase.get<int>(std::max(size_t(n) + 1, size_t(nparts) * 14 + 16));
    if (n <= kSmallMax) {
        ProfScope pso(want_knn ? kStCount : kStTreeSort, s);
        small_sort(pos, s);
    } else {
        GF_CUDA(cudaMemsetAsync(cnt, 0, sizeof(TreeCounts), s));
        double* part = reinterpret_cast<double*>(nb);  // bbox partials, consumed before the scan
        k_bbox<<<nparts, kThreads, 0, s>>>(pos, n, part, R, double(theta_f), C.d_status, &cnt->bbox_done);
        GF_CHECK_LAUNCH();
        k_keys<<<grid, kThreads, 0, s>>>(pos, n, R, k0, pm);
        GF_CHECK_LAUNCH();
        ProfScope pso(want_knn ? kStCount : kStTreeSort, s);
        radix_sort_pairs(k0, pm, key_alt.as<uint64_t>(), perm_alt.as<int>(), n, 0, 63, s, &scratch);
    }

    // The owners' bound is the buffer's own size: node_cap is raised before the node buffers grow, and
    // a growth that fails leaves it above what they hold.
    StartScan starts{KeyView{k0, nullptr, nullptr}, n, leaf_max, ldepth.get<int8_t>(n), dsplit.get<int8_t>(n), nb,
                     node_owner.as<int>(), int(std::min(size_t(node_cap), node_owner.holds<int>())), cnt};
    // Deep cells (> 8 particles in one level-21 cell) need extension keys. A regular build
    // finds out on the host; a captured one always computes them (zero outside deep runs,
    // where they leave every common-prefix length the tree uses unchanged).
    bool deep = graph_safe;
    if (!graph_safe) {
        scan_with(starts, n, &cnt->total_nodes, s, &scratch);
        GF_CUDA(cudaMemcpyAsync(h_counts, cnt, sizeof(TreeCounts), cudaMemcpyDeviceToHost, s));
        GF_CUDA(cudaStreamSynchronize(s));
        deep = h_counts->deep != 0;
    }
    if (deep) {
        uint64_t* e1 = key1.get<uint64_t>(n);
        uint64_t* e2 = key2.get<uint64_t>(n);
        int* run_starts = reinterpret_cast<int*>(key_alt.as<uint64_t>());  // scratch
        int* nst = &cnt->deep_runs;
        k_deep_keys<<<grid, kThreads, 0, s>>>(n, k0, pm, pos, R, e1, e2, run_starts, nst, leaf_max);
        GF_CHECK_LAUNCH();
        deep_sort_attr();
        const size_t sm = size_t(kDeepRunMax) * (2 * sizeof(uint64_t) + sizeof(int));
        k_deep_sort<<<2 * C.sms, 512, sm, s>>>(n, k0, e1, e2, pm, run_starts, nst, C.d_status);
        GF_CHECK_LAUNCH();
        starts.K = KeyView{k0, e1, e2};
        scan_with(starts, n, &cnt->total_nodes, s, &scratch);
        if (!graph_safe) {
            GF_CUDA(cudaMemcpyAsync(h_counts, cnt, sizeof(TreeCounts), cudaMemcpyDeviceToHost, s));
            GF_CUDA(cudaStreamSynchronize(s));
        }
    }
    const KeyView K = starts.K;
    if (!graph_safe) {
        nn = h_counts->total_nodes;
        // headroom: later synchronisation-free rebuilds (captured or not) build inside it
        // (a tree within an eighth of the capacity would keep asking for regular builds: outgrowing)
        if (nn > node_cap - node_cap / 8) node_cap = nn + nn / 2 + 1024;
    }
    const int cap = node_cap;
    // node kernels cover [0, span) and read the live count on the device
    const int span = graph_safe ? cap : nn;
    const int* nn_dev = &cnt->total_nodes;
    const int ngrid = div_up(span, kThreads);
    const int bfs_tiles = div_up(span, kBfsTile);

    int4* i4 = n_i4.get<int4>(cap);
    double4* cd = n_cd.get<double4>(cap);
    float4* geo = n_geo.get<float4>(cap);
    int* par = n_parent.get<int>(cap);
    {
        ProfScope pse(want_knn ? kStCount : kStTreeEmit, s);
        int* own = node_owner.get<int>(cap);
        if (cap > starts.cap) {  // the buffers have grown since the scan
            starts.owner = own;
            starts.cap = cap;
            k_node_owner<<<grid, kThreads, 0, s>>>(n, starts);
            GF_CHECK_LAUNCH();
        }
        k_emit<<<ngrid, kThreads, 0, s>>>(K, n, span, R, starts.ldepth, starts.dsplit, nb, own, cnt, i4, cd, geo, par,
                                          pm, cap, bfs_status.get<unsigned>(size_t(div_up(cap, kBfsTile)) * kDepthBins),
                                          bfs_tiles * kDepthBins);
        GF_CHECK_LAUNCH();
    }
    if (graph_safe) {  // more nodes than the buffers hold: flag, and leave an empty tree
        k_node_cap_check<<<1, 1, 0, s>>>(cnt, cap, C.d_status);
        GF_CHECK_LAUNCH();
    }
    float4* pp = p4.get<float4>(n);
    double* xb = xbuild.get<double>(3 * size_t(n));
    k_gather<<<grid, kThreads, 0, s>>>(n, pm, pos, mass, nullptr, pp, nullptr,
                                       want_knn ? plo.get<float4>(n) : nullptr, 0, xb);
    GF_CHECK_LAUNCH();

    int* nch = n_nchild.get<int>(cap);
    scan_with(GroupScan{nn_dev, span, group_max, i4, par, nch, n_counter.get<int>(cap), groups.get<int>(cap)}, span,
              &cnt->num_groups, s, &scratch);
    int* bfs = n_bfs.get<int>(cap);
    k_bfs_rank<<<bfs_tiles, kBfsThreads, 0, s>>>(span, cnt, i4, bfs_status.as<unsigned>(), bfs, bfs_val.get<int>(cap),
                                                 C.d_status);
    GF_CHECK_LAUNCH();
    k_walk_fill<<<ngrid, kThreads, 0, s>>>(span, i4, nch, bfs, geo, w_b.get<float4>(cap), w_geo.get<float4>(cap),
                                           want_knn ? leaf_of.get<int>(n) : nullptr, par, w_parent.get<int>(cap),
                                           nn_dev);
    GF_CHECK_LAUNCH();
    if (!want_knn) {  // (a neighbour-search tree needs geometry only)
        w_a.get<float4>(cap);
        n_disp.get<float>(cap);
        if (quad) {
            w_q.get<float4>(cap);
            w_t.get<float2>(cap);
            w_rq.get<float>(cap);
        }
        ProfScope psm(kStTreeMoments, s);
        moments(mass, false, span, s);
    }
    valid = true;
    if (!graph_safe) {
        live_pending = false;  // the host knows the node count, and the buffers have room for it
    } else if (!g_no_alloc) {  // outside a capture: the live node count, for outgrowing()
        if (!h_live) GF_CUDA(cudaMallocHost(&h_live, sizeof(int)));
        if (!live_ev) GF_CUDA(cudaEventCreateWithFlags(&live_ev, cudaEventDisableTiming));
        GF_CUDA(cudaMemcpyAsync(h_live, &cnt->total_nodes, sizeof(int), cudaMemcpyDeviceToHost, s));
        GF_CUDA(cudaEventRecord(live_ev, s));
        live_pending = true;
    }
}

bool Octree::outgrowing() {
    if (!live_pending) return false;
    const cudaError_t e = cudaEventQuery(live_ev);
    if (e == cudaErrorNotReady) {
        (void)cudaGetLastError();  // not an error: the copy is still on its way
        return false;
    }
    GF_CUDA(e);
    live_pending = false;
    return *h_live > node_cap - node_cap / 8;
}

// Node kernels cover node_cap and read the live node count on the device, so a refit stays
// valid after a rebuild inside a captured graph (whose node count the host never sees).
void Octree::refit(const double* pos, const double* mass, cudaStream_t s, cudaStream_t s_moments,
                   cudaEvent_t gathered) {
    ProfScope ps(kStTreeRefit, s);
    const int grid = div_up(n, kThreads);
    const int span = std::max(node_cap, nn);
    float4* pp = p4.as<float4>();
    float* pd = pdisp.get<float>(n);
    k_gather<<<grid, kThreads, 0, s>>>(n, perm.as<int>(), pos, mass, xbuild.as<double>(), pp, pd,
                                       want_knn ? plo.get<float4>(n) : nullptr, quad ? 1 : 0);
    GF_CHECK_LAUNCH();
    if (s_moments) {  // the moments on their own stream, after the gather
        GF_CUDA(cudaEventRecord(gathered, s));
        GF_CUDA(cudaStreamWaitEvent(s_moments, gathered, 0));
        s = s_moments;
    }
    moments(mass, true, span, s);
}

// The bottom-up moments pass of a build or a refit, straight into the breadth-first walk layout.
// (The arrival counters are zero: the group scan clears them in a build, and each pass leaves them so.)
void Octree::moments(const double* mass, bool refit, int span, cudaStream_t s) {
    const int* nn_dev = &counts.as<TreeCounts>()->total_nodes;
    const int ngrid = div_up(span, kThreads);
    if (quad) {
        RefitBfsArgs A{span, nn_dev, theta_f, w_parent.as<int>(), w_geo.as<float4>(), n_counter.as<int>(),
                       w_a.as<float4>(), w_b.as<float4>(), w_q.as<float4>(), w_t.as<float2>(), w_rq.as<float>(),
                       n_disp.as<float>(), p4.as<float4>(), refit ? pdisp.as<float>() : nullptr};
        k_refit_bfs_quad32<<<ngrid, kThreads, 0, s>>>(A);
    } else {
        Moments64Args A{span, nn_dev, refit, theta_f, root.as<RootBox>(), w_parent.as<int>(), w_geo.as<float4>(),
                        bfs_val.as<int>(), n_cd.as<double4>(), n_counter.as<int>(), w_a.as<float4>(),
                        w_b.as<float4>(), n_disp.as<float>(), perm.as<int>(), xbuild.as<double>(), mass,
                        p4.as<float4>(), refit ? pdisp.as<float>() : nullptr};
        k_moments64<<<ngrid, kThreads, 0, s>>>(A);
    }
    GF_CHECK_LAUNCH();
}

}  // namespace gf
