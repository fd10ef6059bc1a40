// gf_direct.cu — exact float64 direct sum (cpp/nbody.cpp:428-441): the oracle of every
// Barnes-Hut error report. One thread per target, sources staged through shared memory in
// tiles (x, y, z, m). Same pair formula as the reference:
//   a_i += m_j d / (r2 sqrt(r2)),  r2 = |d|^2 + eps^2,  d = x_j - x_i.
//
// Bound by the float64 pipe (2 lanes per SM and clock): 17 float64 instructions per pair, the
// power -3/2 from the hardware's approximate inverse root and its series, against 38 with a
// square root and a division. The blocks of a cluster share a block of targets, each taking a part
// of the sources, so that a few thousand targets still reach every SM; their sums meet in
// distributed shared memory, in rank order. 20,001 particles: 37.0 ms with one block per 256
// targets (79 of them on 152 SMs), 13.4 ms now (10.8 ms at the pipe's nominal rate); 300k: 2.81 s
// (2.83 s with one part, so eight parts at every size; four: 14.9 ms at 20,001, 305 instead of
// 173 us at 2,000; blocks of 128 targets: 314 us there).
#include <cooperative_groups.h>

#include "gf_common.cuh"

namespace gf {

namespace {

constexpr int kDirThreads = 64;
constexpr int kDirParts = 8;  // blocks per cluster: source parts

// m r2^(-3/2). The seed y of 1/sqrt(r2) has e = 1 - r2 y^2 of about 2^-20, and (1 - e)^(-3/2) =
// 1 + 3/2 e + 15/8 e^2 + ...: the next term is below rounding. (The mass comes last: with an infinite one
// the series' corrections would cancel.)
__device__ __forceinline__ double pair_factor(double r2, double m) {
    if (exponent_of(r2) - 423u < 1200u) {  // 2^-600 <= r2 < 2^600: r2^(-3/2) is a normal number
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
        const double e = fma(-(r2 * y), y, 1.0);
        const double g = y * y * y;
        return m * fma(g * e, fma(1.875, e, 1.5), g);
    }
    return m / (r2 * sqrt(r2));
}

__global__ void __cluster_dims__(kDirParts, 1, 1) __launch_bounds__(kDirThreads) k_direct(int n, const double* __restrict__ pos,
                                                        const double* __restrict__ mass, int nt,
                                                        const int64_t* __restrict__ targets,
                                                        double* __restrict__ acc, double eps2) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double4_32a src[kDirThreads];
    __shared__ double part_sum[3][kDirThreads];
    const int rank = int(cluster.block_rank());
    const int t = (blockIdx.x / kDirParts) * kDirThreads + threadIdx.x;
    const bool ok = t < nt;
    const int64_t i = ok ? (targets ? targets[t] : t) : 0;
    const double xi = ok ? pos[3 * i] : 0, yi = ok ? pos[3 * i + 1] : 0, zi = ok ? pos[3 * i + 2] : 0;
    double ax = 0, ay = 0, az = 0;
    const int tiles = (n + kDirThreads - 1) / kDirThreads;
    const int tile1 = int((long long)tiles * (rank + 1) / kDirParts);
    for (int tile = int((long long)tiles * rank / kDirParts); tile < tile1; ++tile) {
        const int base = tile * kDirThreads;
        const int j = base + threadIdx.x;
        __syncthreads();
        src[threadIdx.x] = j < n ? double4_32a{pos[3 * size_t(j)], pos[3 * size_t(j) + 1], pos[3 * size_t(j) + 2], mass[j]}
                                 : double4_32a{0, 0, 0, 0};
        __syncthreads();
        const int cnt = min(kDirThreads, n - base);
#pragma unroll 4
        for (int q = 0; q < cnt; ++q) {
            const double4_32a s = src[q];
            const double dx = s.x - xi, dy = s.y - yi, dz = s.z - zi;
            const double f = pair_factor(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))), s.w);
            ax = fma(f, dx, ax);
            ay = fma(f, dy, ay);
            az = fma(f, dz, az);
        }
    }
    part_sum[0][threadIdx.x] = ax;
    part_sum[1][threadIdx.x] = ay;
    part_sum[2][threadIdx.x] = az;
    cluster.sync();
    if (rank == 0) {
        for (int c = 1; c < kDirParts; ++c) {
            ax += *cluster.map_shared_rank(&part_sum[0][threadIdx.x], c);
            ay += *cluster.map_shared_rank(&part_sum[1][threadIdx.x], c);
            az += *cluster.map_shared_rank(&part_sum[2][threadIdx.x], c);
        }
    }
    cluster.sync();  // the other blocks' shared memory stays until it has been read
    if (ok && rank == 0) {
        acc[3 * size_t(t)] = ax;
        acc[3 * size_t(t) + 1] = ay;
        acc[3 * size_t(t) + 2] = az;
    }
}

}  // namespace

void direct_sum(int n, const double* pos, const double* mass, int nt, const int64_t* targets,
                double* acc, double eps, cudaStream_t s) {
    if (nt <= 0) return;
    k_direct<<<div_up(nt, kDirThreads) * kDirParts, kDirThreads, 0, s>>>(n, pos, mass, nt, targets, acc, eps * eps);
    GF_CHECK_LAUNCH();
}

}  // namespace gf
