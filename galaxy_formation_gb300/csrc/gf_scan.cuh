// gf_scan.cuh — device-wide exclusive scan of int32 values that a functor computes and consumes, so
// that flags and scanned values need no arrays and no launches of their own.
//
// The functor F has three device members:
//   int first(int i)   the value of entry i, called once per entry (it may store what put needs);
//   int again(int i)   the same value later, from what first left (launches of two passes);
//   void put(int i, int v, int ex)   entry i's value and the sum of the values before it.
//
// Small inputs: one cluster launch, the values in registers between the passes and the blocks'
// sums exchanged through distributed shared memory. Larger ones: tile sums, then each tile adds up
// the sums before its own (up to kScanDirectTiles tiles) or reads them scanned (one launch more).
//
// Small tree builds are bound by the number of launches: with flags and values computed inside the
// scans, the leaf sort inside the node emission and one counting pass for the breadth-first order,
// a regular build went from 22 launches to 8 and Engine.gravity of 2k / 10k / 40k particles from
// 225 / 302 / 411 to 168 / 240 / 349 us.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>
#include <utility>

#include "gf_common.cuh"

namespace gf {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;       // entries per thread of a tile
constexpr int kScanSmallItems = 1;  // while that makes at most kScanDirectTiles tiles (524,288 entries)
constexpr int kScanSmallTile = kScanThreads * kScanSmallItems;
// Tiles up to which each block of the second launch adds up the sums before its own (a few KB of L2
// reads per block).
constexpr int kScanDirectTiles = 2048;
// One cluster launch up to this many entries: 1024 threads x kScanRows entries in each of 8 blocks
// (with two rows, 16,384: gravity of 31k particles 292 us, with four 305; up to 24k no difference).
constexpr int kScanCtas = 8;
constexpr int kScanClusterThreads = 1024;
constexpr int kScanRows = 2;
constexpr int kScanClusterMax = kScanCtas * kScanClusterThreads * kScanRows;

__device__ __forceinline__ int block_excl_scan(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    int incl = warp_incl_scan(v);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nw ? s_warp[lane] : 0;
        int wi = warp_incl_scan(w);
        if (lane < nw) s_warp[lane] = wi - w;
        if (lane == nw - 1) s_warp[32] = wi;
    }
    __syncthreads();
    const int r = incl - v + s_warp[warp];
    if (total) *total = s_warp[32];
    __syncthreads();
    return r;
}

template <class F>
__global__ void __cluster_dims__(kScanCtas, 1, 1) __launch_bounds__(kScanClusterThreads)
    k_scan_cluster(F f, int n, int m, int* __restrict__ total) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // Another block's shared memory may be written only once that block runs: every block says so here
    // and waits for the others before its first remote store, with its own values read in between.
    auto running = cluster.barrier_arrive();
    __shared__ int s_warp[33], s_sums[kScanCtas];
    const int rank = int(cluster.block_rank());
    const int lo = rank * m, hi = min(n, lo + m);
    int v[kScanRows], ex[kScanRows];
    int sum = 0;
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {  // rows of consecutive entries
        const int i = lo + r * kScanClusterThreads + int(threadIdx.x);
        v[r] = 0;
        ex[r] = 0;
        if (lo + r * kScanClusterThreads >= hi) continue;  // uniform over the block
        if (i < hi) v[r] = f.first(i);
        int row;
        ex[r] = sum + block_excl_scan(v[r], s_warp, &row);
        sum += row;
    }
    cluster.barrier_wait(std::move(running));
    if (threadIdx.x < kScanCtas) *cluster.map_shared_rank(&s_sums[rank], int(threadIdx.x)) = sum;
    cluster.sync();
    int before = 0, all = 0;
#pragma unroll
    for (int c = 0; c < kScanCtas; ++c) {
        all += s_sums[c];
        if (c < rank) before += s_sums[c];
    }
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
        const int i = lo + r * kScanClusterThreads + int(threadIdx.x);
        if (i < hi) f.put(i, v[r], before + ex[r]);
    }
    if (total && rank == 0 && threadIdx.x == 0) *total = all;
}

template <class F, int kItems>
__global__ void k_scan_tile_sums(F f, int n, int* __restrict__ sums) {
    __shared__ int s_warp[33];
    const int base = blockIdx.x * kScanThreads * kItems;
    int acc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = base + k * kScanThreads + threadIdx.x;
        if (i < n) acc += f.first(i);
    }
    int tot;
    block_excl_scan(acc, s_warp, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// offs: the tile sums, or (SCANNED) their exclusive scan; the last block writes the total of the
// former.
template <class F, int kItems, bool SCANNED>
__global__ void k_scan_tiles(F f, int n, const int* __restrict__ offs, int* __restrict__ total) {
    __shared__ int s_warp[33];
    int prefix;
    if (SCANNED) {
        prefix = offs[blockIdx.x];
    } else {
        int before = 0;
        for (int t = threadIdx.x; t < int(blockIdx.x); t += kScanThreads) before += offs[t];
        block_excl_scan(before, s_warp, &prefix);
    }
    const int base = (blockIdx.x * kScanThreads + threadIdx.x) * kItems;
    int v[kItems];
    int acc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        v[k] = (base + k < n) ? f.again(base + k) : 0;
        acc += v[k];
    }
    int tile_total;
    int ex = block_excl_scan(acc, s_warp, &tile_total) + prefix;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        if (base + k < n) f.put(base + k, v[k], ex);
        ex += v[k];
    }
    if (!SCANNED && total && threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) *total = prefix + tile_total;
}

// Exclusive scan of `cnt` tile sums in place, total to *total (gf_core.cu).
void scan_sums(int* sums, int cnt, int* total, cudaStream_t s);
int* scan_scratch(int n, ScanScratch* sc);

template <class F>
void scan_with(const F& f, int n, int* total, cudaStream_t s, ScanScratch* sc) {
    if (n <= 0) {
        if (total) GF_CUDA(cudaMemsetAsync(total, 0, sizeof(int), s));
        return;
    }
    if (n <= kScanClusterMax) {
        k_scan_cluster<F><<<kScanCtas, kScanClusterThreads, 0, s>>>(f, n, div_up(n, kScanCtas), total);
        GF_CHECK_LAUNCH();
        return;
    }
    // The values of a tree build's scans are chains of loads (nine key pairs, up to eight children), so
    // threads with fewer entries finish sooner: the tile sums of the node starts / groups of 200k
    // particles 17.2 / 19.6 us with eight entries per thread, 5.5 / 6.6 with one; gravity of 100k
    // particles 438 -> 414 us (four 426, two 416).
    int* sums = scan_scratch(n, sc);
    auto go = [&](auto items) {
        constexpr int kItems = decltype(items)::value;
        const int tiles = div_up(n, kScanThreads * kItems);
        k_scan_tile_sums<F, kItems><<<tiles, kScanThreads, 0, s>>>(f, n, sums);
        GF_CHECK_LAUNCH();
        if (tiles <= kScanDirectTiles) {
            k_scan_tiles<F, kItems, false><<<tiles, kScanThreads, 0, s>>>(f, n, sums, total);
        } else if constexpr (kItems == kScanItems) {  // (the small tiles are taken while they are that few)
            scan_sums(sums, tiles, total, s);
            k_scan_tiles<F, kItems, true><<<tiles, kScanThreads, 0, s>>>(f, n, sums, nullptr);
        }
        GF_CHECK_LAUNCH();
    };
    if (div_up(n, kScanSmallTile) <= kScanDirectTiles)
        go(std::integral_constant<int, kScanSmallItems>{});
    else
        go(std::integral_constant<int, kScanItems>{});
}

}  // namespace gf
