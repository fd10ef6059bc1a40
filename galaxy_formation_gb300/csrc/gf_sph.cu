// gf_sph.cu — SPH on the GPU (galaxy_formation/sph.py).
//
//   kernel / kernel_grad ..... sph.py:31-54, float64
//   sph_forces ............... sph.py:57-106: density pass with the equation of state of each
//                              particle (P/rho^2, sound speed), then the force pass (pressure,
//                              Monaghan-Gingold viscosity on approaching pairs, du/dt, Courant
//                              step); a few lanes per particle, float64.
//   knn_from_candidates ...... sph.py:109-135: one warp per particle, float64 distances,
//                              bitonic sort of the (<= 64) candidates in shared memory.
//   exact k nearest .......... replaces cKDTree(p).query(p, k) (sph.py:165-166):
//                              octree of the points (same builder as gravity); one warp per
//                              one to three consecutive queries walks it with a radius each,
//                              collecting the points within each radius (float32 distances
//                              from hi/lo split coordinates) until the count lies in
//                              [k, 128] — the radius iteration, Newton steps on
//                              count ~ R^3 from a guess (2.5 x the previous h, 1.06 x the
//                              learned guess of the k-th-neighbour distance, a rank of the
//                              distances to the points next to the query in the tree's
//                              order, or the leaf's cell density). The collected points are
//                              sorted, the k nearest plus near-ties at the boundary are re-measured
//                              in float64 and sorted again, so the result is the exact
//                              float64 kNN.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <string>
#include <type_traits>

#include "gf_mlp.cuh"
#include "gf_sph.cuh"
#include "gf_tree.cuh"

namespace gf {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr int kThreads = 256;

// sph.py:31-40
__device__ __forceinline__ double w_m4(double r, double h) {
    const double q = r / h;
    const double s = 1.0 / (kPi * h * h * h);
    if (q < 1.0) return s * (1 - 1.5 * q * q + 0.75 * q * q * q);
    if (q < 2.0) {
        const double t = 2 - q;
        return s * 0.25 * t * t * t;
    }
    return 0.0;
}

// sph.py:43-54
__device__ __forceinline__ double dw_m4(double r, double h) {
    const double q = r / h;
    const double s = 1.0 / (kPi * h * h * h * h);
    double g;
    if (q < 1.0) {
        g = s * (-3 * q + 2.25 * q * q);
    } else if (q < 2.0) {
        const double t = 2 - q;
        g = -s * 0.75 * t * t;
    } else {
        return 0.0;
    }
    return g / fmax(r, 1e-30);
}

__global__ void k_sph_kernel(int n, const double* __restrict__ r, const double* __restrict__ h,
                             double* __restrict__ w, double* __restrict__ dw) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (w) w[i] = w_m4(r[i], h[i]);
    if (dw) dw[i] = dw_m4(r[i], h[i]);
}

// ---- sph_forces in float64 ---------------------------------------------------------------
//
// Bound by the float64 pipe (2 lanes per SM and clock on this GPU), so the pair terms are written
// for few float64 instructions: about 17 in the density pass and 49 in the force pass, against
// 30 and 100 with a division and a square root per factor. (At 500k gas the pipe is 85 % busy.)
//   * 1/r by a seed and one step of third order, r = r^2 (1/r); 1/x the same way (inv_root,
//     inverse): the error of the seed cubed is below rounding.
//   * the kernel's two branches are one polynomial whose coefficients are picked by integer
//     compares on q's upper word.
//   * per-particle factors (1/h, the kernel's normalisation, P/rho^2, scaled sound speed) are
//     computed once per particle, and the two quotients of the viscosity share one inverse.
// kLanes lanes share a particle's row: without them a lone warp works through 32 neighbours one
// after another, and small sets leave most of the chip idle.

// The kernel gradient's normalisation -3 / (4 pi h^4) (sph.py:43-54). It stays finite where h^4
// underflows (h below 2e-77): it is multiplied by shapes that are zero outside the support.
__device__ __forceinline__ double grad_norm(double h) { return -0.75 / fmax(kPi * h * h * h * h, 4.2e-309); }

// 1/h for q = r (1/h), finite for any h but 0: a particle's own q is 0 also where h is subnormal.
__device__ __forceinline__ double inv_length(double h) {
    const double y = 1.0 / h;
    return h != 0.0 && fabs(y) > DBL_MAX ? copysign(DBL_MAX, y) : y;
}

// Threads per block: small blocks even out the last wave of the small launches.
template <int kLanes>
constexpr int kSphThreads = kLanes >= 4 ? 64 : 128;

// Neighbour data of a pair term. PackedSrc: one 128-byte record per particle, a line per
// neighbour: {x, y, z, m}, {vx, vy, vz, h/20}, {s, 1/h, s P/rho^2, 5 alpha c}, {rho, c} with s =
// -3 / (4 pi h^4).
struct PairEos {
    double s, inv_h, sp, ca;
};
struct alignas(128) SphRec {
    double4_32a xm, vh, eos, rc;
};
struct PackedSrc {
    const SphRec* rec;
    __device__ __forceinline__ double4_32a xm(int64_t j) const { return rec[j].xm; }
    __device__ __forceinline__ double4_32a vh(int64_t j) const { return rec[j].vh; }
    __device__ __forceinline__ PairEos eos(int64_t j) const {
        const double4_32a e = rec[j].eos;
        return PairEos{e.x, e.y, e.z, e.w};
    }
    __device__ __forceinline__ double rho(int64_t j) const { return rec[j].rc.x; }
    __device__ __forceinline__ double sound(int64_t j) const { return rec[j].rc.y; }
};
// PlainSrc: the caller's arrays and two scratch arrays (the entry point that may not allocate);
// a neighbour's 1/h is then formed per pair.
struct PlainSrc {
    const double* pos;
    const double* vel;
    const double* mass;
    const double* h;
    const double* rho_;
    const double* pr2;
    const double* cs;
    double ha;  // 5 alpha
    __device__ __forceinline__ double4_32a xm(int64_t j) const {
        return double4_32a{pos[3 * j], pos[3 * j + 1], pos[3 * j + 2], mass[j]};
    }
    __device__ __forceinline__ double4_32a vh(int64_t j) const {
        return double4_32a{vel[3 * j], vel[3 * j + 1], vel[3 * j + 2], 0.05 * h[j]};
    }
    __device__ __forceinline__ PairEos eos(int64_t j) const {
        const double s4 = grad_norm(h[j]);
        return PairEos{s4, 1.0 / h[j], s4 * pr2[j], ha * cs[j]};
    }
    __device__ __forceinline__ double rho(int64_t j) const { return rho_[j]; }
    __device__ __forceinline__ double sound(int64_t j) const { return cs[j]; }
};

// q < 1 and q < 2 on the upper word of a float64. Negative values (a negative h) are below both, as for
// the comparison of the values; a NaN of either sign and -infinity are below neither.
__device__ __forceinline__ bool below_word(double q, int word) {
    const int w = __double2hiint(q);
    return w < word && unsigned(w) < 0xfff00000u;
}
__device__ __forceinline__ bool below_1(double q) { return below_word(q, 0x3ff00000); }
__device__ __forceinline__ bool below_2(double q) { return below_word(q, 0x40000000); }

// M4 kernel without its 1/(pi h^3) (sph.py:31-40): 1 - 3/2 q^2 + 3/4 q^3, or (2 - q)^3 / 4
__device__ __forceinline__ double w_shape64(double q) {
    const bool in = below_1(q);
    const double x = in ? q : 2.0 - q;
    const double w = fma(x * x, fma(in ? 0.75 : 0.25, x, in ? -1.5 : 0.0), in ? 1.0 : 0.0);
    return below_2(q) ? w : 0.0;
}

// -4/3 dW/dq without its 1/(pi h^4) (sph.py:43-54): q (4 - 3 q), or (2 - q)^2 (0 outside the support,
// also where q is infinite)
__device__ __forceinline__ double dw_shape64(double q) {
    const bool in = below_1(q);
    const double l = fma(in ? -3.0 : -1.0, q, in ? 4.0 : 2.0);
    const double p = (in ? q : l) * l;
    return below_2(q) ? p : 0.0;
}

template <int kLanes>
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
    for (int o = kLanes / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double nan64() { return __longlong_as_double(0x7ff8000000000000ll); }

__global__ void k_sph_pack(int n, const double* __restrict__ pos, const double* __restrict__ vel,
                           const double* __restrict__ mass, const double* __restrict__ h, SphRec* __restrict__ rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rec[i].xm = double4_32a{pos[3 * size_t(i)], pos[3 * size_t(i) + 1], pos[3 * size_t(i) + 2], mass[i]};
    rec[i].vh = double4_32a{vel[3 * size_t(i)], vel[3 * size_t(i) + 1], vel[3 * size_t(i) + 2], 0.05 * h[i]};
}

// A neighbour row from the caller may hold an index outside [0, n): such a particle gets NaN
// outputs and GF_ERR_ARG is raised (status may be null), instead of a read out of bounds.

// pass 1 (sph.py:63-71): rho_i = sum_j m_j W(r_ij, h_i), the particle itself included; then the
// equation of state of the particle (the per-j factors of sph.py:88-89), into its record
// (PackedSrc) or pr2 / cs.
template <class Idx, int kLanes, class Src>
__global__ void __launch_bounds__(kSphThreads<kLanes>) k_sph_density(int n, int k, int ld, Src src, const int* __restrict__ order,
                                                          const Idx* __restrict__ nb, const double* __restrict__ h,
                                                          const double* __restrict__ u, double gamma, double ha,
                                                          double* __restrict__ rho, SphRec* rec, double* pr2,
                                                          double* cs, Subset sub, uint32_t* status) {
    const int s = threadIdx.x % kLanes;
    int i = 0;
    const bool on = subset_item(sub, (blockIdx.x * kSphThreads<kLanes> + threadIdx.x) / kLanes, n, order, i);
    bool ok = true;
    double sum = 0.0, hi = 1.0;
    if (on) {
        const double4_32a p = src.xm(i);
        hi = h[i];
        const double inv_h = inv_length(hi);
        const Idx* row = nb + size_t(i) * ld;
#pragma unroll 4
        for (int jj = s; jj < k; jj += kLanes) {
            int64_t j = row[jj];
            if (j < 0 || j >= n) {
                ok = false;
                j = i;
            }
            const double4_32a q = src.xm(j);
            const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double r = j != i ? root(r2) : r2;  // r2 of itself: 0, or NaN of such a position
            sum = fma(q.w, w_shape64(r * inv_h), sum);
        }
    }
    sum = lanes_sum<kLanes>(sum);
    if (kLanes > 1) {
        ok = (__ballot_sync(0xffffffffu, !ok) >> (threadIdx.x & 31 & ~(kLanes - 1)) & ((1u << kLanes) - 1u)) == 0u;
        // the rest is a few divisions per particle: by full warps of one particle per thread (at four
        // lanes per particle it took a third of the pass)
        __shared__ double s_sum[kSphThreads<kLanes> / kLanes];
        __shared__ int s_i[kSphThreads<kLanes> / kLanes];  // INT_MIN: none; ~i: a bad row
        if (s == 0) {
            s_sum[threadIdx.x / kLanes] = sum;
            s_i[threadIdx.x / kLanes] = !on ? INT_MIN : ok ? i : ~i;
        }
        __syncthreads();
        if (threadIdx.x >= kSphThreads<kLanes> / kLanes) return;
        i = s_i[threadIdx.x];
        if (i == INT_MIN) return;
        ok = i >= 0;
        if (!ok) i = ~i;
        sum = s_sum[threadIdx.x];
        hi = h[i];
    } else if (!on) {
        return;
    }
    if (!ok) raise_status(status, GF_ERR_ARG);
    const double d = !ok ? nan64() : sum == 0.0 ? 0.0 : sum * (1.0 / (kPi * hi * hi * hi));
    const double P = (gamma - 1) * d * u[i];
    const double pr = P / (d * d), c = sqrt(gamma * (gamma - 1) * u[i]);
    rho[i] = d;
    if (rec) {
        const double s4 = grad_norm(hi);
        rec[i].eos = double4_32a{s4, 1.0 / hi, s4 * pr, ha * c};
        rec[i].rc = double4_32a{d, c, 0.0, 0.0};
    } else {
        pr2[i] = pr;
        cs[i] = c;
    }
}

// pass 2 (sph.py:72-106)
template <class Idx, int kLanes, class Src>
__global__ void __launch_bounds__(kSphThreads<kLanes>) k_sph_force(int n, int k, int ld, Src src, const int* __restrict__ order,
                                                        const Idx* __restrict__ nb, const double* __restrict__ h,
                                                        double alpha, double beta, double* __restrict__ acc,
                                                        double* __restrict__ dudt, double* __restrict__ dt_i,
                                                        float* __restrict__ divv, Subset sub, uint32_t* status) {
    const int s = threadIdx.x % kLanes;
    int i = 0;
    const bool on = subset_item(sub, (blockIdx.x * kSphThreads<kLanes> + threadIdx.x) / kLanes, n, order, i);
    bool ok = true;
    // Sums over the row: the acceleration; dw = sum m v.d P_i / r and hv = sum m v.d V / r, which
    // give du/dt (pressure and viscous part) and the velocity divergence; the most negative mu / 10, and whose.
    // With P the kernel gradient's shape (times s), A = s P/rho^2 and half_visc half the pair's
    // viscosity: V = half_visc (s_i P_i + s_j P_j), and the pair's force is m (A_i P_i + A_j P_j + V) d / r.
    double ax = 0, ay = 0, az = 0, dw = 0, hv = 0, mu_min = -0.0;
    int j_min = -1;
    PairEos ei{0, 0, 0, 0};
    if (on) {
        const double4_32a p = src.xm(i), v = src.vh(i);
        ei = src.eos(i);
        const double rhoi = src.rho(i), beta100 = 100.0 * beta;
        const Idx* row = nb + size_t(i) * ld;
        for (int jj = s; jj < k; jj += kLanes) {
            const int64_t j = row[jj];
            if (j == i) continue;
            if (j < 0 || j >= n) {
                ok = false;
                continue;
            }
            const double4_32a q = src.xm(j), w = src.vh(j);
            const PairEos ej = src.eos(j);
            const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            double r, inv_r;
            inv_root(r2, r, inv_r);
            const double Pi = dw_shape64(r * ei.inv_h), Pj = dw_shape64(r * ej.inv_h);
            const double vr = (v.x - w.x) * dx + (v.y - w.y) * dy + (v.z - w.z) * dz;
            const double m = q.w * inv_r, mv = m * vr;
            double f = fma(ej.sp, Pj, ei.sp * Pi);
            dw = fma(mv, Pi, dw);
            if (vr < 0) {
                // mu = hb vr / (r^2 + 0.01 hb^2), visc = (-alpha c mu + beta mu^2) / rho with the means
                // hb, c and rho of the pair; hs = 0.1 hb and x = mu / 10 save two products
                const double hs = v.w + w.w, num = hs * vr;
                const double den = fma(hs, hs, r2), rs = rhoi + src.rho(j);
                const double prod = den * rs;
                double x, xr;  // mu / 10, and that over rs
                if (in_inverse_range(prod)) {
                    xr = num * inverse(prod);
                    x = xr * rs;
                } else {
                    x = num / den;
                    xr = x / rs;
                }
                const double half_visc = fma(beta100, x, -(ei.ca + ej.ca)) * xr;
                // Of negative numbers the smallest has the largest bits: from those of -0 on, up to those of
                // -inf. Positive values (a negative hb) and NaN of either sign lie outside.
                const uint64_t xb = uint64_t(__double_as_longlong(x));
                if (xb > uint64_t(__double_as_longlong(mu_min)) && xb <= 0xfff0000000000000ull) mu_min = x, j_min = int(j);
                const double V = half_visc * fma(ej.s, Pj, ei.s * Pi);
                f += V;
                hv = fma(mv, V, hv);
            }
            const double mf = m * f;
            ax = fma(-mf, dx, ax);
            ay = fma(-mf, dy, ay);
            az = fma(-mf, dz, az);
        }
    }
    ax = lanes_sum<kLanes>(ax);
    ay = lanes_sum<kLanes>(ay);
    az = lanes_sum<kLanes>(az);
    dw = lanes_sum<kLanes>(dw);
    hv = lanes_sum<kLanes>(hv);
    double du = fma(0.5, hv, ei.sp * dw);
    const double dv = ei.s * dw;
#pragma unroll
    for (int o = kLanes / 2; o; o >>= 1) {  // by their bits, as above
        const double m2 = __shfl_xor_sync(0xffffffffu, mu_min, o);
        const int j2 = __shfl_xor_sync(0xffffffffu, j_min, o);
        if (uint64_t(__double_as_longlong(m2)) > uint64_t(__double_as_longlong(mu_min))) mu_min = m2, j_min = j2;
    }
    if (kLanes > 1) {
        const unsigned bad = __ballot_sync(0xffffffffu, !ok) >> (threadIdx.x & 31 & ~(kLanes - 1));
        ok = (bad & ((1u << kLanes) - 1u)) == 0u;
    }
    if (!on || s != 0) return;
    if (fabs(ei.sp) > DBL_MAX || ei.sp != ei.sp) {  // no number times an empty sum: a particle alone is not heated
        const Idx* row = nb + size_t(i) * ld;
        bool alone = true;
        for (int jj = 0; jj < k; ++jj) alone = alone && row[jj] == i;
        if (alone) du = 0.0;
    }
    if (!ok) {
        raise_status(status, GF_ERR_ARG);
        ax = ay = az = du = nan64();
    }
    acc[3 * size_t(i)] = ax;
    acc[3 * size_t(i) + 1] = ay;
    acc[3 * size_t(i) + 2] = az;
    dudt[i] = du;
    // The mu that sets the Courant step once more, with its own division: with the pair term's shared
    // inverse the step's mean error against 64 bits is 1.17e-16, from here 1.01e-16 (with a division per
    // factor in every pair it was 1.08e-16). Keeping track of the pair and this take 2 to 7 % of the pass
    // (28.6 -> 30.7 us for 5k gas, 492 -> 514 for 150k, 1499 -> 1521 for 500k).
    mu_min = -0.0;
    if (j_min >= 0) {
        const double4_32a p = src.xm(i), v = src.vh(i), q = src.xm(j_min), w = src.vh(j_min);
        const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
        const double vr = (v.x - w.x) * dx + (v.y - w.y) * dy + (v.z - w.z) * dz;
        const double hb = 0.5 * (h[i] + h[j_min]);
        mu_min = hb * vr / fma(0.01 * hb, hb, dx * dx + dy * dy + dz * dz);
    }
    const double c = src.sound(i);
    dt_i[i] = ok ? 0.3 * h[i] / (c + 1.2 * (alpha * c - beta * mu_min) + 1e-30) : nan64();
    if (divv) divv[i] = ok ? float(-dv / src.rho(i)) : __int_as_float(0x7fc00000);  // SPH velocity divergence
                                                                                  // (a feature of the h guess)
}

// --------------------------------------------------------------- knn_from_candidates

constexpr int kCandWarps = 8;

__global__ void __launch_bounds__(kCandWarps * 32) k_knn_cand(
    int n, int m, const double* __restrict__ pos, const int64_t* __restrict__ cand, int k,
    int64_t* __restrict__ nb, double* __restrict__ dist, int* __restrict__ all_ok) {
    __shared__ unsigned long long s_key[kCandWarps][64];
    __shared__ int s_tag[kCandWarps][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long* key = s_key[w];
    int* tag = s_tag[w];
    const int nwarps = gridDim.x * kCandWarps;
    for (int i = blockIdx.x * kCandWarps + w; i < n; i += nwarps) {
        const double xi = pos[3 * size_t(i)], yi = pos[3 * size_t(i) + 1], zi = pos[3 * size_t(i) + 2];
        int valid = 0;
        for (int jj = lane; jj < 64; jj += 32) {
            double d2 = INFINITY;
            if (jj < m) {
                const int64_t j = cand[size_t(i) * m + jj];
                if (j >= 0) {
                    const double dx = xi - pos[3 * j], dy = yi - pos[3 * j + 1], dz = zi - pos[3 * j + 2];
                    d2 = dx * dx + dy * dy + dz * dz;
                    ++valid;
                }
            }
            key[jj] = (unsigned long long)__double_as_longlong(d2);
            tag[jj] = jj;
        }
        valid = warp_sum(valid);
        __syncwarp();
        if (valid < k) {  // sph.py:128-130: not enough candidates, row untouched
            if (lane == 0) *all_ok = 0;
            continue;
        }
        warp_bitonic(key, tag, 64);
        for (int t = lane; t < k; t += 32) {
            nb[size_t(i) * k + t] = cand[size_t(i) * m + tag[t]];
            dist[size_t(i) * k + t] = sqrt(__longlong_as_double((long long)key[t]));
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------ exact kNN

constexpr int kKnnOneQuery = 8 * 1024, kKnnTwoQueries = 64 * 1024;  // most queries with one / two per warp
// Leaf capacity of the neighbour-search tree. The search is exact for any tree; 16 walks
// fewer levels per query (7 % faster on the 1M disk) but its coarser leaf counts make the
// learned guess's features less informative, so the reference's 8 is kept.
constexpr int kKnnLeaf = kLeafMax;
constexpr int kKnnStack = 512;
constexpr int kKnnCap = 128;

// A collected point: (float32 squared distance bits << 32) | tree position. The bits of a
// non-negative float order like the float, so sorting the keys orders by distance, then index.
__device__ __forceinline__ unsigned long long knn_key(float d2, int j) {
    return ((unsigned long long)__float_as_uint(d2) << 32) | unsigned(j);
}
__device__ __forceinline__ float key_d2(unsigned long long k) { return __uint_as_float(unsigned(k >> 32)); }
__device__ __forceinline__ int key_idx(unsigned long long k) { return int(unsigned(k)); }

// A query of a neighbour walk: position (hi / lo) with the radius and its square, in shared memory
// (registers for two to four of them spilled at four blocks per SM).
struct KnnQuery {
    float4 h;  // x y z of the position's high parts, radius
    float4 l;  // low parts, squared radius
    float lo, hi;  // bracket of the radius iteration
};

// Shared memory of a warp that serves kQ queries. The sort's counters and the float64 near-ties
// reuse the walk's stack: a query is finished after its walk.
template <int kQ>
struct KnnSmem {
    union {
        int stack[kKnnStack];
        struct {
            unsigned long long dd[64];  // float64 squared distances as bit patterns
            int di[64];
            int first[kSortBuckets + 4];  // of the sort: a bucket's count, then its first key
        };
    };
    unsigned long long key[kQ][kKnnCap];  // the collected points of the warp's queries
    int seg[32];                // opened leaves of a round: first particle minus first slot
    KnnQuery q[kQ];
    int cnt[kQ];                // points of the last walk
};

struct KnnArgs {
    int n, k, nn;
    const float4* wb;
    const float4* wgeo;
    const float4* p4;
    const float4* plo;
    const int* perm;
    const int* leaf_of;
    const double* pos;      // caller order
    const float* r_guess;   // caller order, optional
    int64_t* nb;            // (n, k) caller order, or null
    double* dist;           // (n, k), or null
    int* nb32;              // (n, ld32) caller order, or null
    int ld32;
    double* dsel;           // distance of neighbour `dsel_col` (n,), or null
    int dsel_col;
    int* dsel_idx;          // instead of dsel (float32 order): that neighbour's caller index, whose
                            // float64 distance the caller measures a thread per query (-1: failed)
    float* dfar;            // distance of the k-th nearest in float32 (n,), or null
    uint32_t* status;
    unsigned long long* iters;
    const int* wparent;     // breadth-first parent of each node (-1 for the root)
    int window_rank;        // without r_guess: start at this rank of the distances to the points
                            // next to the query in tree order (0: at the leaf's cell density)
    int exact_order;        // 1: float64 re-sort of the k nearest; 0: float32 order, float64
                            //    only to settle the neighbour at dsel_col (the h boundary)
};

// Collects, for each of the warp's (up to) kQ queries that is on, the points within its radius
// into S.key[i] (the first kKnnCap of them) and their number into S.cnt[i]. One walk serves all: a
// node is opened when it meets any of the spheres (a test against the queries' bounding box and
// largest radius opens far too much where consecutive queries lie in cells apart: 10 ms instead of
// 2 for the 1M disk's gas), and each point of an opened leaf is tested against every query. A query
// with more than `enough` (>= kKnnCap) points is done with this radius: its sphere opens no further
// nodes (S.cnt[i] then is only known to exceed that). Returns false on stack overflow. The queries of a
// warp are neighbours in the tree's order (often in one leaf), so their walks share most nodes.
template <int kQ>
__device__ bool knn_collect(const KnnArgs& A, KnnSmem<kQ>& S, unsigned live, int leaf, int enough) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    int cnt[kQ] = {};
    // start at the smallest ancestor of the leaf whose cube contains every sphere that is on
    // (every point within a radius then lies in that subtree)
    int start = leaf;
    for (int up = 0; start > 0 && up < 64; ++up) {
        const float4 g = A.wgeo[start];
        const int parent = A.wparent[start];
        const float pad = 2e-6f * (fabsf(g.x) + fabsf(g.y) + fabsf(g.z) + g.w) + 1e-30f;
        bool inside = true;
#pragma unroll
        for (int i = 0; i < kQ; ++i) {
            if (!(live >> i & 1u)) continue;
            const float4 qh = S.q[i].h, ql = S.q[i].l;
            const float lim = g.w - qh.w - pad;
            inside = inside && fabsf((qh.x - g.x) + ql.x) <= lim && fabsf((qh.y - g.y) + ql.y) <= lim &&
                     fabsf((qh.z - g.z) + ql.z) <= lim;
        }
        if (inside) break;
        start = parent;
    }
    if (start < 0) start = 0;
    int sp = 1;
    if (lane == 0) S.stack[0] = (start << 4) | 1;
    __syncwarp();
    for (int rounds = 0; sp > 0; ++rounds) {
        if (rounds > A.nn) return false;  // each node is popped at most once
        int node[1];
        pop_round<1>(S.stack, sp, node);
        bool open = false;
        int first = 0, code = 0;
        if (node[0] >= 0) {
            const float4 g = A.wgeo[node[0]], b = A.wb[node[0]];
            first = __float_as_int(b.y);
            code = __float_as_int(b.z);
            // distance from each query to the cell cube, padded for float32 rounding
            const float lim = g.w + 2e-6f * (fabsf(g.x) + fabsf(g.y) + fabsf(g.z) + g.w) + 1e-30f;
#pragma unroll
            for (int i = 0; i < kQ; ++i) {
                if (!(live >> i & 1u)) continue;
                const float4 qh = S.q[i].h, ql = S.q[i].l;
                const float ex = fmaxf(fabsf((g.x - qh.x) - ql.x) - lim, 0.f);
                const float ey = fmaxf(fabsf((g.y - qh.y) - ql.y) - lim, 0.f);
                const float ez = fmaxf(fabsf((g.z - qh.z) - ql.z) - lim, 0.f);
                open = open || ex * ex + ey * ey + ez * ez <= ql.w;
            }
        }
        const bool inner = open && code > 0;
        const unsigned om = __ballot_sync(0xffffffffu, inner);
        const int npush = __popc(om);
        if (sp + npush > kKnnStack) return false;
        if (inner) S.stack[sp + __popc(om & lt)] = (first << 4) | code;
        sp += npush;
        // particles of the opened leaves, concatenated in lane order and tested 32 at a time: lane l
        // takes offset o = base + l
        const bool leaf_open = open && code < 0;
        const unsigned lm = __ballot_sync(0xffffffffu, leaf_open);
        if (lm) {
            const int lc = leaf_open ? -code : 0;
            const int lincl = warp_incl_scan(lc);
            const int lexcl = lincl - lc;
            const int ltot = __shfl_sync(0xffffffffu, lincl, 31);
            if (leaf_open) S.seg[__popc(lm & lt)] = first - lexcl;
            __syncwarp();
            int before = -1;
            for (int base = 0; base < ltot; base += 32) {
                const int o = base + lane;
                const unsigned marks = segment_marks(leaf_open, lexcl, base);
                const int src = before + __popc(marks & (lt | (1u << lane)));
                before += __popc(marks);
                float4 ph = make_float4(0.f, 0.f, 0.f, 0.f), pl = ph;
                int j = 0;
                if (o < ltot) {
                    j = S.seg[src] + o;
                    ph = A.p4[j];
                    pl = A.plo[j];
                }
#pragma unroll
                for (int i = 0; i < kQ; ++i) {
                    if (!(live >> i & 1u)) continue;
                    const float4 qh = S.q[i].h, ql = S.q[i].l;
                    const float dx = (ph.x - qh.x) + (pl.x - ql.x);
                    const float dy = (ph.y - qh.y) + (pl.y - ql.y);
                    const float dz = (ph.z - qh.z) + (pl.z - ql.z);
                    const float d2 = dx * dx + dy * dy + dz * dz;
                    const bool hit = o < ltot && d2 <= ql.w;
                    const unsigned hm = __ballot_sync(0xffffffffu, hit);
                    if (hit) {
                        const int slot = cnt[i] + __popc(hm & lt);
                        if (slot < kKnnCap) S.key[i][slot] = knn_key(d2, j);
                    }
                    cnt[i] += __popc(hm);
                }
            }
            unsigned full = 0;
#pragma unroll
            for (int i = 0; i < kQ; ++i) full |= cnt[i] > enough ? 1u << i : 0u;
            live &= ~full;
            if (!live) break;
        }
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < kQ; ++i)
        if (lane == i) S.cnt[i] = cnt[i];
    __syncwarp();
    return true;
}

// Sorts the cnt (<= kKnnCap) keys of a query within the squared radius 1 / inv_R2, ascending, by
// buckets of their distance (distance_bucket): a key's place is its bucket's first one plus the
// smaller keys of that bucket (two or three). About 130 warp instructions for 64 keys and 210 for 128, where the bitonic
// network takes 300 and 780. Distances piled up in one bucket take the network.
__device__ __forceinline__ void knn_sort(unsigned long long* key, int* first, int cnt, float inv_R2) {
    constexpr int kPer = kKnnCap / 32;
    const int lane = threadIdx.x & 31;
    clear_buckets(first);
    __syncwarp();
    unsigned long long K[kPer];
    int at[kPer];  // bucket << 8 | place in it
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        at[t] = -1;
        if (32 * t >= cnt) break;  // warp-uniform
        if (32 * t + lane < cnt) {
            K[t] = key[32 * t + lane];
            const int b = distance_bucket(key_d2(K[t]) * inv_R2);
            at[t] = b << 8 | atomicAdd(first + b, 1);
        }
    }
    __syncwarp();
    if (bucket_starts(first, cnt) > 12) {
        int P = 64;
        while (P < cnt) P <<= 1;
        for (int t = cnt + lane; t < P; t += 32) key[t] = ~0ull;
        __syncwarp();
        warp_sort_u64(key, P);
        return;
    }
    int b0[kPer], b1[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        b0[t] = b1[t] = 0;
        if (32 * t >= cnt) break;
        if (at[t] >= 0) {
            b0[t] = first[at[t] >> 8];
            b1[t] = first[(at[t] >> 8) + 1];
            key[b0[t] + (at[t] & 255)] = K[t];
        }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        if (32 * t >= cnt) break;
        int r = b0[t];
        for (int m = b0[t]; m < b1[t]; ++m) r += key[m] < K[t] ? 1 : 0;
        at[t] = at[t] >= 0 ? r : -1;
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        if (32 * t >= cnt) break;
        if (at[t] >= 0) key[at[t]] = K[t];
    }
    __syncwarp();
}

// Sorts the cnt (<= kKnnCap) collected points of query q (tree position), re-measures the
// k nearest and the float32 near-ties in float64 and writes the k nearest (ascending, ties by
// index) in the caller's order.
__device__ __forceinline__ double d2_f64(const KnnArgs& A, int pi, int pj) {
    const double dx = A.pos[3 * size_t(pi)] - A.pos[3 * size_t(pj)];
    const double dy = A.pos[3 * size_t(pi) + 1] - A.pos[3 * size_t(pj) + 1];
    const double dz = A.pos[3 * size_t(pi) + 2] - A.pos[3 * size_t(pj) + 2];
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

template <int kQ>
__device__ void knn_finish(const KnnArgs& A, KnnSmem<kQ>& S, unsigned long long* key, int cnt, float R2, int q) {
    unsigned long long* dd = S.dd;
    int* di = S.di;
    const int lane = threadIdx.x & 31;
    const int k = A.k;
    const int oq = A.perm[q];
    knn_sort(key, S.first, cnt, 1.0f / R2);
    const int pi = oq;
    if (!A.exact_order) {
        // Float32 order: the k nearest as a set (only pairs tied to float32 rounding can
        // swap). The neighbour at dsel_col fixes h: the entries within float32 rounding of
        // it are re-measured in float64 and the dsel_col-th smallest is taken.
        const int c = A.dsel_col;
        const float dc = key_d2(key[c]);
        const float lo = dc * (1.0f - 2e-5f), hi = dc * (1.0f + 2e-5f);
        int below = 0, inband = 0;
        for (int t = lane; t < cnt; t += 32) {
            const float v = key_d2(key[t]);
            below += v < lo;
            inband += v >= lo && v <= hi;
        }
        below = __reduce_add_sync(0xffffffffu, below);
        inband = __reduce_add_sync(0xffffffffu, inband);
        double best = 0.0;
        int selc = -1;  // caller index of the entry that fixes h
        if (inband == 1) {  // no float32 near-tie: entry c itself, measured in float64
            selc = A.perm[key_idx(key[c])];
            if (!A.dsel_idx) best = d2_f64(A, pi, selc);
        } else {
            const int rank_need = c - below;  // rank of the wanted entry among the ambiguous ones
            for (int t = lane; t < 64; t += 32) {
                double v = INFINITY;
                int tag = 0x7fffffff;
                const float vf = t < cnt ? key_d2(key[t]) : INFINITY;
                if (t < cnt && vf >= lo && vf <= hi) {
                    const int j = key_idx(key[t]);
                    v = d2_f64(A, pi, A.perm[j]);
                    tag = j;
                }
                dd[t] = (unsigned long long)__double_as_longlong(v);
                di[t] = tag;
            }
            __syncwarp();
            warp_bitonic(dd, di, 64);
            best = __longlong_as_double((long long)dd[max(0, rank_need)]);
            selc = A.perm[di[max(0, rank_need)]];
            // the tied entries [below, below + inband) take the float64 order (ties by tree
            // position), so the first c + 1 entries are the exact set the smoothing length is
            // measured on; their float32 distance bits stay (all within the band)
            if (below + inband <= 64)
                for (int t = lane; t < inband; t += 32)
                    key[below + t] = (key[below + t] & 0xffffffff00000000ull) | unsigned(di[t]);
            __syncwarp();
        }
        for (int t = lane; t < k; t += 32) {
            const int pj = A.perm[key_idx(key[t])];
            if (A.nb32) A.nb32[size_t(oq) * A.ld32 + t] = pj;
            if (A.nb) A.nb[size_t(oq) * k + t] = pj;
        }
        if (A.dsel_idx) {
            if (lane == 0) A.dsel_idx[oq] = selc;
        } else if (A.dsel && lane == 0) {
            A.dsel[oq] = __dsqrt_rn(best);
        }
        if (A.dfar && lane == 0) A.dfar[oq] = sqrtf(key_d2(key[k - 1]));
        __syncwarp();
        return;
    }
    // the k nearest and everything within float32 rounding of the k-th distance
    const float thr = key_d2(key[k - 1]) * (1.0f + 2e-5f);
    int m = 0;
    for (int t = lane; t < cnt; t += 32) m += key_d2(key[t]) <= thr;
    m = min(64, __reduce_add_sync(0xffffffffu, m));
    for (int t = lane; t < 64; t += 32) {
        double v = INFINITY;
        int tag = 0x7fffffff;
        if (t < m) {
            const int pj = A.perm[key_idx(key[t])];
            v = d2_f64(A, pi, pj);
            tag = pj;
        }
        dd[t] = (unsigned long long)__double_as_longlong(v);
        di[t] = tag;
    }
    __syncwarp();
    warp_bitonic(dd, di, 64);
    for (int t = lane; t < k; t += 32) {
        const double dt = __longlong_as_double((long long)dd[t]);
        if (A.nb) A.nb[size_t(oq) * k + t] = di[t];
        if (A.dist) A.dist[size_t(oq) * k + t] = __dsqrt_rn(dt);
        if (A.nb32) A.nb32[size_t(oq) * A.ld32 + t] = di[t];
        if (A.dsel && t == A.dsel_col) A.dsel[oq] = __dsqrt_rn(dt);
        if (A.dfar && t == k - 1) A.dfar[oq] = sqrtf(float(dt));
    }
    __syncwarp();
}

__device__ void knn_fail_output(const KnnArgs& A, int q, bool stack) {
    const int lane = threadIdx.x & 31;
    const int oq = A.perm[q];
    if (lane == 0) raise_status(A.status, stack ? GF_ERR_WALK_STACK : GF_ERR_KNN);
    for (int t = lane; t < A.k; t += 32) {
        if (A.nb) A.nb[size_t(oq) * A.k + t] = -1;
        if (A.dist) A.dist[size_t(oq) * A.k + t] = INFINITY;
        if (A.nb32) A.nb32[size_t(oq) * A.ld32 + t] = -1;
    }
    if (A.dsel && lane == 0) A.dsel[oq] = INFINITY;
    if (A.dsel_idx && lane == 0) A.dsel_idx[oq] = -1;
}

// Radius from the density of the query's leaf cell.
__device__ __forceinline__ float knn_cell_radius(const KnnArgs& A, int q) {
    const int lf = A.leaf_of[q];
    const float half = A.wgeo[lf].w;
    const int c = max(1, -__float_as_int(A.wb[lf].z));
    return 2.0f * half * cbrtf(float(A.k) / float(c));
}

// A radius that encloses at least `rank` of kPer * 32 points, kPer per lane, given as the upper
// kKnnRankBits bits of their float32 squared distances (their order is the bits' order; all ones:
// no point): bisection on those bits, each step one compare per point and one warp sum. The
// radius is the upper edge of the bucket that reaches the rank.
constexpr int kKnnRankBits = 12;  // exponent and 4 bits of mantissa: 6 % in d^2, 3 % in the radius
constexpr int kKnnRankShift = 31 - kKnnRankBits;  // the sign bit is 0

template <int kPer>
__device__ __forceinline__ float knn_rank_radius(const unsigned (&b)[kPer], int rank) {
    unsigned lo = 0, hi = (1u << kKnnRankBits) - 1u;
    while (lo < hi) {
        const unsigned mid = (lo + hi) >> 1;
        int c = 0;
#pragma unroll
        for (int t = 0; t < kPer; ++t) c += b[t] <= mid ? 1 : 0;
        if (__reduce_add_sync(0xffffffffu, c) >= rank)
            hi = mid;
        else
            lo = mid + 1;
    }
    // padded so that a distance tied with the edge to rounding is inside
    return sqrtf(__uint_as_float((lo + 1) << kKnnRankShift)) * 1.0001f;
}

// Starting radius of a query without a previous h: the kKnnWindow points around its warp's queries
// in tree order hold most of the nearest ones, so the radius that encloses window_rank of them
// encloses about k of all points. The first search of the 1M disk's 500k gas is bound by the
// points its spheres collect: from the leaf's cell density, whose one to eight points say little,
// spheres held hundreds to thousands of them (8.70 ms); from here, with collections that stop at the
// cap, 2.64 ms (1.51 ms with a previous h).
constexpr int kKnnWindow = 128;

__device__ __forceinline__ float knn_window_radius(const KnnArgs& A, int q0, const KnnQuery& Q) {
    constexpr int kPer = kKnnWindow / 32;
    const int lane = threadIdx.x & 31;
    const int w0 = max(0, min(q0 - kKnnWindow / 2 + 1, A.n - kKnnWindow));
    unsigned b[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
        const int j = w0 + 32 * t + lane;
        b[t] = 0xffffffffu;
        if (j < A.n) {
            const float4 ph = A.p4[j], pl = A.plo[j];
            const float dx = (ph.x - Q.h.x) + (pl.x - Q.l.x);
            const float dy = (ph.y - Q.h.y) + (pl.y - Q.l.y);
            const float dz = (ph.z - Q.h.z) + (pl.z - Q.l.z);
            b[t] = __float_as_uint(dx * dx + dy * dy + dz * dz) >> kKnnRankShift;
        }
    }
    return knn_rank_radius<kPer>(b, min(A.window_rank, min(A.n, kKnnWindow)));
}

// Next radius of a query whose sphere holds more than kKnnCap points (key: kKnnCap of them): the
// sphere around k + kKnnShrink of those, or smaller than R by what one point too many implies.
constexpr int kKnnShrink = 8;

__device__ __forceinline__ float knn_shrunk_radius(const unsigned long long* key, int k, float R) {
    constexpr int kPer = kKnnCap / 32;
    const int lane = threadIdx.x & 31;
    unsigned b[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) b[t] = unsigned(key[32 * t + lane] >> 32) >> kKnnRankShift;
    return fminf(knn_rank_radius<kPer>(b, k + kKnnShrink), 0.9f * R);
}

// Walks of a search that stop at kKnnCap points. A radius from the points of such a walk may be as
// little as a tenth smaller (the first points met can all lie at the rim), so a start far too large, the
// previous h of a set that has collapsed since, could use up all the walks: from then on a walk counts
// every point in the sphere, and the count itself gives the step.
constexpr int kKnnStopWalks = 12;

// Radius step of the count-to-k iteration: Newton on count ~ R^3 below k and, with the whole count
// (counted), above the cap; else a rank of the collected distances; bisection once it is bracketed.
__device__ __forceinline__ float knn_next_radius(float R, int cnt, bool counted, int k, const unsigned long long* key,
                                                 float& lo, float& hi) {
    if (cnt < k)
        lo = R;
    else
        hi = R;
    if (lo > 0.f && hi < INFINITY) return 0.5f * (lo + hi);
    if (cnt < k) return R * (cnt >= 4 ? cbrtf(1.3f * float(k) / float(cnt)) : 2.0f);
    if (counted) return R * cbrtf(0.75f * float(kKnnCap) / float(cnt));
    return knn_shrunk_radius(key, k, R);
}

// One warp per kQ consecutive queries (tree order): one walk from the smallest ancestor cell that
// contains all their spheres collects for all of them; each iterates its radius on its own, and
// those still searching walk again together. Bound by instruction issue (about 70 % of the slots).
// 32 warps per SM at 64 registers (24 at 80: 15 % slower; 40 at 48, spilling: 12 %). Of the time of a
// pair of queries 30 % went to node rounds of 28 nodes, 32 % to finishing (the sort), 20 % to points,
// 8 % to the ascent; with three queries to a walk, rounds of one node per lane instead of two and
// the sort by buckets the search of 500k gas takes 1.51 ms with a previous h (2.07 before) and 2.64
// ms without one (3.20).
template <int kQ, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, 32 / kWarps) k_knn(KnnArgs A) {
    __shared__ __align__(16) KnnSmem<kQ> smem_all[kWarps];
    KnnSmem<kQ>& S = smem_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int k = A.k;
    const int cap = kKnnCap;  // count window [k, cap]
    const int nwarps = gridDim.x * kWarps;
    auto set_radius = [&](int i, float R) {
        if (!(R > 0.f) || !isfinite(R)) R = 1e-3f;
        if (lane == 0) S.q[i].h.w = R, S.q[i].l.w = R * R;
    };
    for (int q0 = kQ * (blockIdx.x * kWarps + (threadIdx.x >> 5)); q0 < A.n; q0 += kQ * nwarps) {
        const int nq = min(kQ, A.n - q0);
        const bool window = !A.r_guess && A.window_rank > 0;
        unsigned on = (1u << nq) - 1u, windowed = window ? on : 0u;  // bits of the queries
        int total = 0, walks = 0;
        if (lane < nq) {
            S.q[lane].h = A.p4[q0 + lane];
            S.q[lane].l = A.plo[q0 + lane];
            S.q[lane].lo = 0.f;
            S.q[lane].hi = INFINITY;
        }
        __syncwarp();
        for (int i = 0; i < nq; ++i)
            set_radius(i, window      ? knn_window_radius(A, q0, S.q[i])
                          : A.r_guess ? A.r_guess[A.perm[q0 + i]]
                                      : knn_cell_radius(A, q0 + i));
        __syncwarp();
        while (on) {
            const bool counted = walks >= kKnnStopWalks;
            const bool ok_walk =
                knn_collect<kQ>(A, S, on, A.leaf_of[q0 + __ffs(on) - 1], counted ? INT_MAX : kKnnCap);
            total += __popc(on);
            ++walks;
            for (int i = 0; i < nq; ++i) {
                if (!(on >> i & 1u)) continue;
                const int cnt = S.cnt[i];
                const float R = S.q[i].h.w;
                if (ok_walk && cnt >= k && cnt <= cap) {
                    knn_finish<kQ>(A, S, S.key[i], cnt, S.q[i].l.w, q0 + i);
                    on &= ~(1u << i);
                } else if (ok_walk && walks < 48) {
                    float lo = S.q[i].lo, hi = S.q[i].hi;
                    const float next = knn_next_radius(R, cnt, counted, k, S.key[i], lo, hi);
                    __syncwarp();
                    if (lane == 0) {
                        S.q[i].lo = lo;
                        S.q[i].hi = hi;
                        S.q[i].h.w = next;
                        S.q[i].l.w = next * next;
                    }
                } else if (windowed >> i & 1u) {  // once more, from the cell density
                    if (lane == 0) {
                        S.q[i].lo = 0.f;
                        S.q[i].hi = INFINITY;
                    }
                    set_radius(i, knn_cell_radius(A, q0 + i));
                } else {
                    knn_fail_output(A, q0 + i, !ok_walk);
                    on &= ~(1u << i);
                }
            }
            if (walks == 48 || !ok_walk) windowed = 0, walks = 0;
            __syncwarp();
        }
        if (lane == 0 && A.iters) atomicAdd(A.iters, (unsigned long long)total);
        __syncwarp();
    }
}

}  // namespace

// ------------------------------------------------------------------------------- host

void sph_kernel_values(int n, const double* r, const double* h, double* w, double* dw, cudaStream_t s) {
    if (n <= 0) return;
    k_sph_kernel<<<div_up(n, kThreads), kThreads, 0, s>>>(n, r, h, w, dw);
    GF_CHECK_LAUNCH();
}

// The two float64 passes with L lanes per particle, on any neighbour source. timed: as stages of the
// profiler, which creates events and keeps them.
template <class Idx, int L, class Src>
void sph_launch(int n, int k, int ld, const Src& src, const int* order, const Idx* nb, const double* h,
                const double* u, double gamma, double alpha, double beta, double* rho, SphRec* rec, double* pr2,
                double* cs, double* acc, double* dudt, double* dt_i, cudaStream_t s, float* divv, Subset sub,
                uint32_t* status, bool timed) {
    constexpr int threads = kSphThreads<L>;
    const int grid = div_up((long long)n * L, threads);
    {
        ProfScope ps(timed ? kStSphDensity : -1, s);
        k_sph_density<Idx, L><<<grid, threads, 0, s>>>(n, k, ld, src, order, nb, h, u, gamma, 5.0 * alpha, rho, rec,
                                                        pr2, cs, sub, status);
        GF_CHECK_LAUNCH();
    }
    ProfScope ps(timed ? kStSphForce : -1, s);
    k_sph_force<Idx, L><<<grid, threads, 0, s>>>(n, k, ld, src, order, nb, h, alpha, beta, acc, dudt, dt_i, divv,
                                                  sub, status);
    GF_CHECK_LAUNCH();
}

// Lanes per particle by the particles of a launch: one thread each fills the chip (and needs no
// reduction) from some hundred thousand on; below, more lanes shorten the chain of neighbours, and a
// subset of unknown size takes four. Density + force in us with 1 / 2 / 4 / 8 lanes (before: a thread
// per particle with a division and a square root per factor):
//     5k gas   118 /   70 /   47 /   45   (329)        150k    718 /  673 /  698 /  785   (1361)
//    20k       171 /  135 /  115 /  123                250k   1140 / 1134 / 1199 / 1356
//   100k       534 /  476 /  472 /  534                500k   2048 / 2135 / 2262 / 2573   (4141)
constexpr int kSphEightLanes = 8 * 1024, kSphFourLanes = 128 * 1024, kSphTwoLanes = 256 * 1024;

template <class Idx>
void sph_forces(SphScratch& S, int n, int k, int ld, const int* order, const double* pos, const double* vel,
                const double* mass, const Idx* nb, const double* h, const double* u, double gamma, double alpha,
                double beta, double* rho, double* acc, double* dudt, double* dt_i, cudaStream_t s, float* divv,
                Subset sub) {
    if (n <= 0) return;
    SphRec* rec = S.rec.get<SphRec>(n);
    k_sph_pack<<<div_up(n, kThreads), kThreads, 0, s>>>(n, pos, vel, mass, h, rec);
    GF_CHECK_LAUNCH();
    auto go = [&](auto lanes) {
        sph_launch<Idx, decltype(lanes)::value>(n, k, ld, PackedSrc{rec}, order, nb, h, u, gamma, alpha, beta, rho,
                                                rec, nullptr, nullptr, acc, dudt, dt_i, s, divv, sub, ctx().d_status,
                                                true);
    };
    if (!sub.idx && n <= kSphEightLanes)
        go(std::integral_constant<int, 8>());
    else if (sub.idx || n <= kSphFourLanes)
        go(std::integral_constant<int, 4>());
    else if (n <= kSphTwoLanes)
        go(std::integral_constant<int, 2>());
    else
        go(std::integral_constant<int, 1>());
}
template void sph_forces<int64_t>(SphScratch&, int, int, int, const int*, const double*, const double*, const double*,
                                  const int64_t*, const double*, const double*, double, double, double,
                                  double*, double*, double*, double*, cudaStream_t, float*, Subset);
template void sph_forces<int>(SphScratch&, int, int, int, const int*, const double*, const double*, const double*,
                              const int*, const double*, const double*, double, double, double,
                              double*, double*, double*, double*, cudaStream_t, float*, Subset);

void knn_from_candidates(int n, int m, const double* pos, const int64_t* cand, int k, int64_t* nb,
                         double* dist, int* d_ok, cudaStream_t s) {
    if (n <= 0) return;
    const int blocks = std::min(div_up(n, kCandWarps), 8 * ctx().sms);
    k_knn_cand<<<blocks, kCandWarps * 32, 0, s>>>(n, m, pos, cand, k, nb, dist, d_ok);
    GF_CHECK_LAUNCH();
}

// Features of the smoothing-length guess, per gas particle (caller order):
// (log cell density of its leaf, log previous h, leaf count, previous velocity divergence).
// Features of the learned guess: log cell density, log previous h, leaf count, velocity
// divergence. A particle without a previous h (the first search of a particle set) gets, in
// its place, the h that its cell density implies (the search radius of the cell-density start
// over 2.5: a function of the first feature, cold_log_h) and a divergence of 0.
__global__ void k_hfeatures(int n, int k, const int* __restrict__ perm, const int* __restrict__ leaf_of,
                            const float4* __restrict__ wb, const float4* __restrict__ wgeo, const int* __restrict__ gidx,
                            const double* __restrict__ hprev, const float* __restrict__ divv, float* __restrict__ X) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int i = perm[q];
    const int lf = leaf_of[q];
    const float c = float(max(1, -__float_as_int(wb[lf].z)));
    const float side = 2.f * wgeo[lf].w;
    const int g = gidx ? gidx[i] : i;
    const double hp = hprev ? hprev[g] : 0.0;
    const float f0 = logf(c / fmaxf(side * side * side, 1e-30f));
    X[4 * size_t(i) + 0] = f0;
    X[4 * size_t(i) + 1] = hp > 0 ? float(log(hp)) : cold_log_h(f0, k);
    X[4 * size_t(i) + 2] = c;
    X[4 * size_t(i) + 3] = hp > 0 && divv ? divv[g] : 0.f;
}

// The learned guess predicts the log distance of the k-th nearest; the search starts a little
// outside it, so that nearly every first sphere holds the k nearest and rarely more than 64
// points (one sort of 64 keys instead of 128).
constexpr float kFarMargin = 1.06f;

__global__ void k_guess_from_logdk(int n, const float* __restrict__ Y, float* __restrict__ rg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) rg[i] = kFarMargin * expf(Y[i]);
}

// Rank of the window distances that a search without a previous h starts at: 3/4 of k, since the
// window misses a part of the sphere (36 for the 48 nearest: 34 and 38 are 0.5 % and 3 % slower,
// 46 15 %), but for the smaller k at least 24 or k itself: any count from k to the cap settles a query,
// and rank k makes sure of it. Searches of a 200k cloud for 1 / 4 / 16 neighbours 424 / 553 / 707 us; with
// rank 24 807 / 821 / 833; from the leaf's cell density 475 / 559 / 852.
static int knn_window_rank(int k) { return std::max(std::min(24, k), (3 * k + 3) / 4); }

void knn_exact(Octree& T, int n, const double* pos, int k, const float* r_guess, int64_t* nb,
               double* dist, unsigned long long* d_iters, cudaStream_t s, int* nb32, int ld32,
               double* dsel, int dsel_col, const HGuess* hg, bool same_set, int* dsel_idx, bool cell_start) {
    if (n <= 0) return;
    // same_set (the caller's point set drifted since the last search): the synchronisation-free
    // rebuild inside the node buffers of the last regular build (no host round trip in the middle
    // of the hydro chain), unless the last tree came close to filling them
    const bool same = same_set && T.valid && T.n == n && T.want_knn && T.leaf_max == kKnnLeaf && !T.outgrowing();
    T.want_knn = true;
    T.leaf_max = kKnnLeaf;
    if (same) {
        T.reserve_graph_build();
        T.build(n, pos, nullptr, 0.7, s, true);
    } else {
        T.build(n, pos, nullptr, 0.7, s);
    }
    if (hg && hg->X) {  // features for the learned guess (and for training pairs)
        k_hfeatures<<<div_up(n, kThreads), kThreads, 0, s>>>(n, k, T.perm.as<int>(), T.leaf_of.as<int>(),
                                                             T.w_b.as<float4>(), T.w_geo.as<float4>(), hg->gidx,
                                                             hg->hprev, hg->divv, hg->X);
        GF_CHECK_LAUNCH();
        if (hg->use_mlp) {
            mlp().predict(n, hg->X, hg->Y, s);
            k_guess_from_logdk<<<div_up(n, kThreads), kThreads, 0, s>>>(n, hg->Y, hg->rg);
            GF_CHECK_LAUNCH();
            r_guess = hg->rg;
        }
    }
    KnnArgs A{};
    A.n = n;
    A.k = k;
    A.nn = std::max(T.nn, T.node_cap);  // bounds the walk rounds (the live count is on the device)
    A.wb = T.w_b.as<float4>();
    A.wgeo = T.w_geo.as<float4>();
    A.p4 = T.p4.as<float4>();
    A.plo = T.plo.as<float4>();
    A.perm = T.perm.as<int>();
    A.leaf_of = T.leaf_of.as<int>();
    A.pos = pos;
    A.r_guess = r_guess;
    A.nb = nb;
    A.dist = dist;
    A.nb32 = nb32;
    A.ld32 = ld32;
    A.dsel = dsel;
    A.dsel_col = dsel_col;
    A.dsel_idx = dsel_col >= 0 ? dsel_idx : nullptr;
    A.dfar = hg ? hg->dk : nullptr;
    A.exact_order = (nb != nullptr || dist != nullptr || dsel_col < 0) ? 1 : 0;
    A.status = ctx().d_status;
    A.iters = d_iters;
    A.wparent = T.w_parent.as<int>();
    A.window_rank = cell_start ? 0 : knn_window_rank(k);
    ProfScope ps(kStKnn, s);
    // Queries per warp: more of them share a walk, as long as their warps still fill the chip. First /
    // later search in us with 1, 2, 3, 4 per warp (a Plummer-like cloud):
    //     5k   83 /  54    124 /   66    148 /   81    193 /  100
    //    10k  128 /  76    153 /   68    192 /   76    221 /   95
    //    40k  313 / 189    299 /  165    354 /  151    505 /  162
    //    80k  581 / 349    551 /  286    487 /  254    499 /  257
    //   320k 2040 / 1288  1775 / 1193   1662 / 1082   1716 /  941
    // (1M disk, 500k gas: 2 2854 / 1716, 3 2638 / 1509, 4 2853 / 1622).
    auto go = [&](auto queries) {
        constexpr int kQ = decltype(queries)::value, kWarps = kQ <= 2 ? 8 : 4;  // 48 KB of shared memory a block
        k_knn<kQ, kWarps><<<std::min(div_up(n, kQ * kWarps), 16 * 8 / kWarps * ctx().sms), kWarps * 32, 0, s>>>(A);
    };
    if (n <= kKnnOneQuery)
        go(std::integral_constant<int, 1>{});
    else if (n <= kKnnTwoQueries)
        go(std::integral_constant<int, 2>{});
    else
        go(std::integral_constant<int, 3>{});
    GF_CHECK_LAUNCH();
}

}  // namespace gf

// ---------------------------------------------------------------------------------------
// sph_forces without any device allocation.
//
// Some callers cannot call cudaMalloc: hosts whose own memory pool owns the whole GPU (an
// extra allocation fails or fragments their pool), and step loops that must not allocate
// because cudaMalloc / cudaFree synchronise the device. gf_sph_forces_noalloc_dev serves
// them: the caller passes inputs and outputs in device memory as for gf_sph_forces_dev, and
// the per-particle scratch (P / rho^2 and the sound speed, 16 bytes per particle) lives in
// the fixed array below instead of a growing allocation. The array holds
// GF_SPH_NOALLOC_MAX_N particles (4 MiB); every GPU that loads the library keeps it until
// the process exits.
//
// In host code `g_sph_noalloc_scratch` names a host-side stand-in, not device memory: the
// device address is fetched with cudaGetSymbolAddress once per device (with that device
// current) by the first call on that device, and passed to the kernels. The cached address
// belongs to the device's context of that moment: after cudaDeviceReset (or a reset of the
// primary context) the array is loaded anew elsewhere and the cache is stale, so a process
// that resets a device must not call this entry point on it afterwards.

namespace gf {
namespace {

constexpr int kNoallocMaxN = GF_SPH_NOALLOC_MAX_N;
constexpr int kNoallocMaxDevices = 64;

static __device__ __align__(256) double g_sph_noalloc_scratch[2 * size_t(kNoallocMaxN)];

std::mutex g_noalloc_mu;
double* g_noalloc_ptr[kNoallocMaxDevices] = {};

// Device address of g_sph_noalloc_scratch on the current device (set up on first use).
cudaError_t noalloc_scratch(double** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kNoallocMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_sph_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}

int noalloc_fail(int code, const std::string& msg) {
    Context& c = ctx();
    c.last_status = code;
    c.last_error = msg;
    return code;
}

}  // namespace

}  // namespace gf

extern "C" int gf_sph_forces_noalloc_dev(int n, int k, const double* pos, const double* vel,
                                         const double* mass, const int64_t* nb, const double* h,
                                         const double* u, double gamma, double alpha, double beta,
                                         double* rho, double* acc, double* dudt, double* dt_i,
                                         void* stream) {
    using namespace gf;
    Context& c = ctx();
    c.last_status = 0;
    c.last_error.clear();
    if (n < 0 || k < 0) return noalloc_fail(GF_ERR_ARG, "gf_sph_forces_noalloc_dev: negative size");
    if (n > kNoallocMaxN) {
        char buf[160];
        snprintf(buf, sizeof buf, "gf_sph_forces_noalloc_dev: n = %d exceeds the fixed scratch of %d particles",
                 n, kNoallocMaxN);
        return noalloc_fail(GF_ERR_CAPACITY, buf);
    }
    if (n == 0) return GF_OK;
    if (!(pos && vel && mass && nb && h && u && rho && acc && dudt && dt_i))
        return noalloc_fail(GF_ERR_ARG, "gf_sph_forces_noalloc_dev: null array");
    double* scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess)
        return noalloc_fail(GF_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    // P / rho^2 and the sound speed are written for every particle before they are read,
    // so nothing left by an earlier call needs clearing.
    double* pr2 = scratch;
    double* cs = scratch + kNoallocMaxN;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    try {
        sph_launch<int64_t, 4>(n, k, k, PlainSrc{pos, vel, mass, h, rho, pr2, cs, 5.0 * alpha}, nullptr, nb, h, u,
                               gamma, alpha, beta, rho, nullptr, pr2, cs, acc, dudt, dt_i, s, nullptr, Subset(),
                               nullptr, false);
    } catch (const Error& err) {
        return noalloc_fail(err.code, err.what());
    }
    return GF_OK;
}
