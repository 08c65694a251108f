// Clebsch-Gordan tensor products of spherical-expansion blocks: the real CG
// coefficients (host) and the coupling kernel behind
// featomic_b200_cg_coefficients / featomic_b200_cg_product.
//
// Follows python/featomic/featomic/clebsch_gordan/_coefficients.py:
// complex CG coefficients (the `wigners` package there, Racah's closed form
// here), turned real with the real<->complex harmonic transforms of
// _coefficients.py:336-384 (U(l) on m1 and m2, U(lambda)^H on mu) and the real
// or imaginary part kept by the parity of l1 + l2 + lambda
// (_coefficients.py:137-224); the product of two blocks is
// out[s, mu, p * n2 + q] = sum_{m1 m2} C[m1, m2, mu] a[s, m1, p] b[s, m2, q]
// (_coefficients.py:628-709, properties p-major as
// _utils.py:_compute_labels_full_cartesian_product).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "../../include/featomic_b200.h"
#include "clebsch_gordan.hpp"
#include "engine.hpp"

namespace fb200 {

namespace {

long double factorial(int n) {
    long double f = 1.0L;
    for (int k = 2; k <= n; k++) f *= (long double)k;
    return f;
}

// <j1 m1 j2 m2 | J M> by Racah's formula (Racah 1942; e.g. Varshalovich et
// al., "Quantum Theory of Angular Momentum", 8.2.1 eq. 3), Condon-Shortley
// phase convention.
long double complex_cg(int j1, int m1, int j2, int m2, int J, int M) {
    if (m1 + m2 != M || std::abs(m1) > j1 || std::abs(m2) > j2 || std::abs(M) > J) return 0.0L;
    if (J < std::abs(j1 - j2) || J > j1 + j2) return 0.0L;
    const long double pre = std::sqrt((2.0L * J + 1.0L) * factorial(J + j1 - j2) * factorial(J - j1 + j2) *
                                      factorial(j1 + j2 - J) / factorial(j1 + j2 + J + 1));
    const long double norm = std::sqrt(factorial(J + M) * factorial(J - M) * factorial(j1 - m1) *
                                       factorial(j1 + m1) * factorial(j2 - m2) * factorial(j2 + m2));
    long double sum = 0.0L;
    const int kmin = std::max({0, j2 - J - m1, j1 - J + m2});
    const int kmax = std::min({j1 + j2 - J, j1 - m1, j2 + m2});
    for (int k = kmin; k <= kmax; k++) {
        const long double d = factorial(k) * factorial(j1 + j2 - J - k) * factorial(j1 - m1 - k) *
                              factorial(j2 + m2 - k) * factorial(J - j2 + m1 + k) * factorial(J - j1 - m2 + k);
        sum += ((k & 1) ? -1.0L : 1.0L) / d;
    }
    return pre * norm * sum;
}

using cplx = std::complex<long double>;

// U(l)[l + m, l + m'] with complex Y = U . real Y (real harmonics in
// featomic's m order -l..l, _coefficients.py:336-369).
std::vector<cplx> real_to_complex(int l) {
    const int M = 2 * l + 1;
    std::vector<cplx> u((size_t)M * M, cplx(0, 0));
    const long double r = 1.0L / std::sqrt(2.0L);
    for (int m = -l; m <= l; m++) {
        const long double sign = (m & 1) ? -1.0L : 1.0L;
        if (m < 0) {
            u[(size_t)(l + m) * M + (l + m)] = cplx(0, -r);
            u[(size_t)(l + m) * M + (l - m)] = cplx(0, r * sign);
        } else if (m == 0) {
            u[(size_t)l * M + l] = cplx(1, 0);
        } else {
            u[(size_t)(l + m) * M + (l - m)] = cplx(r, 0);
            u[(size_t)(l + m) * M + (l + m)] = cplx(r * sign, 0);
        }
    }
    return u;
}

}  // namespace

// Real CG coefficients, dense [2 l1 + 1][2 l2 + 1][2 lambda + 1].
std::vector<double> real_cg_coefficients(int l1, int l2, int lambda) {
    if (l1 < 0 || l2 < 0 || lambda < 0) throw invalid_parameter("angular orders must be non-negative");
    if (lambda < std::abs(l1 - l2) || lambda > l1 + l2)
        throw invalid_parameter("lambda = " + std::to_string(lambda) + " can not couple l1 = " + std::to_string(l1) +
                                " and l2 = " + std::to_string(l2));
    if (l1 + l2 > 40) throw invalid_parameter("angular orders above 40 are not supported");
    const int A = 2 * l1 + 1, B = 2 * l2 + 1, C = 2 * lambda + 1;
    std::vector<cplx> cg((size_t)A * B * C);
    for (int a = 0; a < A; a++)
        for (int b = 0; b < B; b++)
            for (int c = 0; c < C; c++)
                cg[((size_t)a * B + b) * C + c] = cplx(complex_cg(l1, a - l1, l2, b - l2, lambda, c - lambda), 0);
    const auto u1 = real_to_complex(l1), u2 = real_to_complex(l2), ul = real_to_complex(lambda);
    // x1[a', b, c] = sum_a U1[a', a] cg[a, b, c]
    std::vector<cplx> x1((size_t)A * B * C, cplx(0, 0)), x2((size_t)A * B * C, cplx(0, 0));
    for (int ap = 0; ap < A; ap++)
        for (int a = 0; a < A; a++) {
            const cplx u = u1[(size_t)ap * A + a];
            if (u == cplx(0, 0)) continue;
            for (size_t bc = 0; bc < (size_t)B * C; bc++) x1[(size_t)ap * B * C + bc] += u * cg[(size_t)a * B * C + bc];
        }
    // x2[a, b', c] = sum_b U2[b', b] x1[a, b, c]
    for (int a = 0; a < A; a++)
        for (int bp = 0; bp < B; bp++)
            for (int b = 0; b < B; b++) {
                const cplx u = u2[(size_t)bp * B + b];
                if (u == cplx(0, 0)) continue;
                for (int c = 0; c < C; c++) x2[((size_t)a * B + bp) * C + c] += u * x1[((size_t)a * B + b) * C + c];
            }
    // real[a, b, c'] = sum_c x2[a, b, c] conj(U_lambda)[c', c]  (x2 @ U_lambda^H)
    const bool even = ((l1 + l2 + lambda) & 1) == 0;
    std::vector<double> out((size_t)A * B * C);
    for (size_t ab = 0; ab < (size_t)A * B; ab++)
        for (int cp = 0; cp < C; cp++) {
            cplx s(0, 0);
            for (int c = 0; c < C; c++) s += x2[ab * C + c] * std::conj(ul[(size_t)cp * C + c]);
            out[ab * C + cp] = (double)(even ? s.real() : s.imag());
        }
    return out;
}

namespace {

struct DeviceCgTask {
    const void* first;
    const void* second;
    void* output;
    int64_t n_samples;
    int64_t block_start;  // first CTA of this task
    int64_t out_stride;   // elements between (sample, mu) rows of the output
    int32_t n_first, n_second, lambda;
    int32_t m1_count, m2_count;
    int32_t entries;      // offset of the task's (mu-sorted) coefficient list
    int32_t mu_offsets;   // offset of its [2 lambda + 2] per-mu starts
    int32_t vector;       // rows of `second` / `output` take 4-wide vector accesses
    int32_t vector_first; // rows of `first` take 8-wide vector loads
};

struct CgEntry {
    int16_t m1, m2;
    float pad;
    double value;
};

constexpr int CG_THREADS = 256;
constexpr int CG_PV = 8;  // first-block properties per thread
constexpr int CG_QV = 4;  // second-block properties per thread

__device__ inline void load4(const float* p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
}
__device__ inline void load4(const double* p, double (&x)[4]) {
    const double2 u = reinterpret_cast<const double2*>(p)[0], v = reinterpret_cast<const double2*>(p)[1];
    x[0] = u.x, x[1] = u.y, x[2] = v.x, x[3] = v.y;
}
__device__ inline void load8(const float* p, float (&x)[8]) {
    const float4 u = reinterpret_cast<const float4*>(p)[0], v = reinterpret_cast<const float4*>(p)[1];
    x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w, x[4] = v.x, x[5] = v.y, x[6] = v.z, x[7] = v.w;
}
__device__ inline void load8(const double* p, double (&x)[8]) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 u = reinterpret_cast<const double2*>(p)[k];
        x[2 * k] = u.x, x[2 * k + 1] = u.y;
    }
}
__device__ inline void store4(float* p, const float (&x)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ inline void store4(double* p, const double (&x)[4]) {
    reinterpret_cast<double2*>(p)[0] = make_double2(x[0], x[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(x[2], x[3]);
}

// One thread per (sample, 8 first-block properties, 4 second-block
// properties) of one task: each coefficient and first-block value is loaded
// once for 4 or 32 products, the first-block row (8 wide), the second-block
// row and the output row (4 wide) are vector accesses when the task allows, and every output value is written
// once.  Each output is sum_k (C_k * a[m1_k]) * b[m2_k] over the task's
// non-zero coefficients of that mu, in the table order.
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
cg_product_kernel(const DeviceCgTask* __restrict__ tasks, int n_tasks, const CgEntry* __restrict__ entries,
                  const int32_t* __restrict__ mu_starts) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (tasks[mid].block_start <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const DeviceCgTask t = tasks[lo];
    const int nqt = (t.n_second + CG_QV - 1) / CG_QV, npt = (t.n_first + CG_PV - 1) / CG_PV;
    const int64_t tiles = (int64_t)npt * nqt;
    const int64_t item = ((int64_t)blockIdx.x - t.block_start) * CG_THREADS + threadIdx.x;
    if (item >= t.n_samples * tiles) return;
    const int64_t s = item / tiles;
    const int64_t r = item - s * tiles;
    const int pt = (int)(r / nqt), qt = (int)(r - (int64_t)pt * nqt);
    const int p0 = pt * CG_PV, q0 = qt * CG_QV;
    const int np = min(CG_PV, t.n_first - p0), nq = min(CG_QV, t.n_second - q0);
    const T* __restrict__ a = static_cast<const T*>(t.first) + s * t.m1_count * t.n_first + p0;
    const T* __restrict__ b = static_cast<const T*>(t.second) + s * t.m2_count * t.n_second + q0;
    T* __restrict__ out = static_cast<T*>(t.output) + s * (2 * t.lambda + 1) * t.out_stride +
                          (int64_t)p0 * t.n_second + q0;
    const bool vec = t.vector && nq == CG_QV;
    const bool vec_first = CG_PV == 8 && t.vector_first && np == CG_PV;
    const int32_t* starts = mu_starts + t.mu_offsets;
    const CgEntry* e = entries + t.entries;
    for (int mu = 0; mu <= 2 * t.lambda; mu++) {
        T acc[CG_PV][CG_QV];
#pragma unroll
        for (int i = 0; i < CG_PV; i++)
#pragma unroll
            for (int j = 0; j < CG_QV; j++) acc[i][j] = T(0);
        for (int k = starts[mu]; k < starts[mu + 1]; k++) {
            const CgEntry c = e[k];
            const T* brow = b + (int64_t)c.m2 * t.n_second;
            T bv[CG_QV];
            if (vec) {
                load4(brow, bv);
            } else {
#pragma unroll
                for (int j = 0; j < CG_QV; j++) bv[j] = j < nq ? brow[j] : T(0);
            }
            T av[CG_PV];
            if (vec_first) {
                load8(a + (int64_t)c.m1 * t.n_first, av);
            } else {
#pragma unroll
                for (int i = 0; i < CG_PV; i++) av[i] = i < np ? a[(int64_t)c.m1 * t.n_first + i] : T(0);
            }
#pragma unroll
            for (int i = 0; i < CG_PV; i++) {
                const T ca = T(c.value) * av[i];
#pragma unroll
                for (int j = 0; j < CG_QV; j++) acc[i][j] += ca * bv[j];
            }
        }
        T* orow = out + mu * t.out_stride;
#pragma unroll
        for (int i = 0; i < CG_PV; i++) {
            if (i >= np) break;
            if (vec) {
                store4(orow + (int64_t)i * t.n_second, acc[i]);
            } else {
#pragma unroll
                for (int j = 0; j < CG_QV; j++)
                    if (j < nq) orow[(int64_t)i * t.n_second + j] = acc[i][j];
            }
        }
    }
}

// ---- FP64 products on the tensor cores ---------------------------------------
//
// For one output row (lambda, mu) the product is a matrix product over m1,
//   out[p, q] = sum_m1 a[m1, p] D[m1, q],   D[m1, q] = sum_m2 C[m1, m2, mu] b[m2, q],
// and a real Clebsch-Gordan coefficient has at most two m2 for given m1 and
// mu (|m2| = ||mu| +- |m1||, one sign of each).  A warp owns up to 32 x 32
// properties of one sample and walks over the output rows of one block pair,
// every lambda: both blocks' rows are read once into shared memory, each lane
// makes its elements of D from two products, and DMMAs (8 x 8 x 4) do the
// rest, 512-byte streaming stores per 8 x 8 tile.
//
// Bound by the HBM stream of the output.  Every (l1 <= l2 <= 4, lambda) block of 2000
// centres with 32 x 32 properties (6.47 GB written): 1.08 ms = 5.98 TB/s, 0.91
// of the measured copy; 1.12 ms with 100 rows to a warp, 1.24 ms without the
// streaming hint.  The thread-per-8 x 4 kernel above takes 1.78 ms on it: six
// 16-byte loads for 32 multiply-adds keep its L1 busier than its FP64 pipe
// (fused multiply-adds alone gave 2 %).

struct CgCoef {  // the two terms of D[m1, :] of one output row
    double v0, v1;
    int32_t m0, m1;  // offsets of their m2 rows in shared memory
    int32_t pad[2];
};

struct CgRow {
    double* out;       // (sample 0, mu) row of the task's output
    int64_t stride;    // elements between samples
    int32_t table;     // first of the row's [m1 padded to 4] CgCoef
    int32_t pad;
};

struct DeviceCgGroup {
    const double* first;
    const double* second;
    int64_t n_samples;
    int64_t warp_start;  // first warp of this group
    int32_t n_first, n_second, m1_count, m2_count;
    int32_t row_begin, row_end;
    int32_t p_blocks, q_blocks;  // tiles of a sample
    int32_t p_size, q_size;      // their sizes: multiples of 8, at most 32
    int32_t vector;      // 16-byte stores
};

constexpr int CG_MMA_WARPS = 4;
constexpr int CG_GROUP_ROWS = 12;  // output rows of a warp: at least this many, where the block pair has them
constexpr int CG_PITCH = 36;  // doubles; 4 (mod 16): fragment loads hit every bank once

__device__ __forceinline__ void cg_dmma(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

__device__ __forceinline__ void cg_cp8(double* dst, const double* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}

__global__ void __launch_bounds__(32 * CG_MMA_WARPS, 4)
cg_product_mma_kernel(const DeviceCgGroup* __restrict__ groups, int n_groups, const CgRow* __restrict__ rows,
                      const CgCoef* __restrict__ table, int warp_doubles) {
    extern __shared__ __align__(16) double cg_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * CG_MMA_WARPS + warp;
    int lo = 0, hi = n_groups - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (groups[mid].warp_start <= w) lo = mid; else hi = mid - 1;
    }
    const DeviceCgGroup g = groups[lo];
    const int64_t item = w - g.warp_start;
    const int blocks = g.p_blocks * g.q_blocks;
    if (item >= g.n_samples * blocks) return;
    const int64_t s = item / blocks;
    const int tile = (int)(item - s * blocks);
    const int p0 = g.p_size * (tile / g.q_blocks), q0 = g.q_size * (tile % g.q_blocks);
    const int np = min(g.p_size, g.n_first - p0), nq = min(g.q_size, g.n_second - q0);
    const int mt = (np + 7) / 8, nt = (nq + 7) / 8, ksteps = (g.m1_count + 3) / 4;
    double* As = cg_smem + warp * warp_doubles;      // [4 ksteps][pitch], zero outside the block
    double* Bs = As + 4 * ksteps * CG_PITCH;         // [m2][pitch]
    const double* a = g.first + s * g.m1_count * g.n_first + p0;
    const double* b = g.second + s * g.m2_count * g.n_second + q0;
    for (int m = 0; m < 4 * ksteps; m++) {
        const bool ok = m < g.m1_count && lane < np;
        cg_cp8(As + m * CG_PITCH + lane, a + (ok ? (int64_t)m * g.n_first + lane : 0), ok);
    }
    for (int m = 0; m < g.m2_count; m++) {
        const bool ok = lane < nq;
        cg_cp8(Bs + m * CG_PITCH + lane, b + (ok ? (int64_t)m * g.n_second + lane : 0), ok);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // zeros of the padding and of D would turn an infinity or a NaN of the
    // inputs into NaNs of rows that it does not couple to: such a sample is
    // summed over its non-zero coefficients instead
    bool finite = true;
    for (int m = 0; m < g.m1_count; m++) finite &= lane >= np || isfinite(As[m * CG_PITCH + lane]);
    for (int m = 0; m < g.m2_count; m++) finite &= lane >= nq || isfinite(Bs[m * CG_PITCH + lane]);
    if (!__all_sync(0xffffffffu, finite)) {
        for (int r = g.row_begin; r < g.row_end; r++) {
            const CgRow row = rows[r];
            for (int x = lane; x < np * nq; x += 32) {
                const int p = x / nq, q = x - p * nq;
                double sum = 0.0;
                for (int m = 0; m < g.m1_count; m++) {
                    const CgCoef c = table[row.table + m];
                    const double f = As[m * CG_PITCH + p];
                    if (c.v0 != 0.0) sum = fma(c.v0 * f, Bs[c.m0 + q], sum);
                    if (c.v1 != 0.0) sum = fma(c.v1 * f, Bs[c.m1 + q], sum);
                }
                row.out[s * row.stride + (int64_t)(p0 + p) * g.n_second + q0 + q] = sum;
            }
        }
        return;
    }
    const int k = lane & 3, n = lane >> 2;
    const double* A0 = As + k * CG_PITCH + n;
    const double* B0 = Bs + n;
    for (int r = g.row_begin; r < g.row_end; r++) {
        const CgRow row = rows[r];
        const CgCoef* coef = table + row.table + k;
        double acc[4][4][2];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
        for (int ks = 0; ks < ksteps; ks++) {
            const double2 v = *reinterpret_cast<const double2*>(&coef[4 * ks].v0);
            const int2 m = *reinterpret_cast<const int2*>(&coef[4 * ks].m0);
            double d[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < nt) d[j] = fma(v.y, B0[m.y + 8 * j], v.x * B0[m.x + 8 * j]);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (i < mt) {
                    const double x = A0[4 * ks * CG_PITCH + 8 * i];
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (j < nt) cg_dmma(acc[i][j], x, d[j]);
                }
            }
        }
        double* out = row.out + s * row.stride + (int64_t)(p0 + n) * g.n_second + q0 + 2 * k;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (8 * i + n >= np) continue;
            double* o = out + (int64_t)8 * i * g.n_second;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int q = 8 * j + 2 * k;
                if (g.vector && q + 1 < nq) {
                    __stcs(reinterpret_cast<double2*>(o + 8 * j), make_double2(acc[i][j][0], acc[i][j][1]));
                } else {
                    if (q < nq) o[8 * j] = acc[i][j][0];
                    if (q + 1 < nq) o[8 * j + 1] = acc[i][j][1];
                }
            }
        }
    }
}

struct DeviceCoupleTask {
    const void* input;
    void* output;
    int64_t n_outer, n_inner;
    int64_t block_start;
    int32_t m1_count, m2_count, lambda;
    int32_t entries, mu_offsets;
};

// Coupling of two spherical axes of one array: one thread per (outer,
// inner) index, out[o, mu, i] = sum_k C_k * x[o, m1_k, m2_k, i] over the
// non-zero coefficients of mu in table order; loads and stores coalesced
// along the inner index.
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
cg_couple_kernel(const DeviceCoupleTask* __restrict__ tasks, int n_tasks, const CgEntry* __restrict__ entries,
                 const int32_t* __restrict__ mu_starts) {
    int lo = 0, hi = n_tasks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (tasks[mid].block_start <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const DeviceCoupleTask t = tasks[lo];
    const int64_t item = ((int64_t)blockIdx.x - t.block_start) * CG_THREADS + threadIdx.x;
    if (item >= t.n_outer * t.n_inner) return;
    const int64_t o = item / t.n_inner, i = item - o * t.n_inner;
    const T* __restrict__ x = static_cast<const T*>(t.input) + o * t.m1_count * t.m2_count * t.n_inner + i;
    T* __restrict__ out = static_cast<T*>(t.output) + o * (2 * t.lambda + 1) * t.n_inner + i;
    const int32_t* starts = mu_starts + t.mu_offsets;
    const CgEntry* e = entries + t.entries;
    for (int mu = 0; mu <= 2 * t.lambda; mu++) {
        T acc = T(0);
        for (int k = starts[mu]; k < starts[mu + 1]; k++) {
            const CgEntry c = e[k];
            acc += T(c.value) * x[((int64_t)c.m1 * t.m2_count + c.m2) * t.n_inner];
        }
        out[mu * t.n_inner] = acc;
    }
}

// Non-zero real CG coefficients of (l1, l2, lambda), grouped by mu, cached.
struct SparseCg {
    std::vector<CgEntry> entries;
    std::vector<int32_t> mu_starts;  // [2 lambda + 2], relative to entries
};

const SparseCg& sparse_cg(int l1, int l2, int lambda) {
    static std::mutex mutex;
    static std::map<std::tuple<int, int, int>, SparseCg> cache;
    std::lock_guard<std::mutex> lock(mutex);
    auto it = cache.find({l1, l2, lambda});
    if (it != cache.end()) return it->second;
    const auto dense = real_cg_coefficients(l1, l2, lambda);
    const int A = 2 * l1 + 1, B = 2 * l2 + 1, C = 2 * lambda + 1;
    SparseCg sp;
    sp.mu_starts.push_back(0);
    for (int c = 0; c < C; c++) {
        for (int a = 0; a < A; a++)
            for (int b = 0; b < B; b++) {
                const double v = dense[((size_t)a * B + b) * C + c];
                if (std::fabs(v) > 1e-15) sp.entries.push_back(CgEntry{(int16_t)a, (int16_t)b, 0.0f, v});
            }
        sp.mu_starts.push_back((int32_t)sp.entries.size());
    }
    return cache.emplace(std::make_tuple(l1, l2, lambda), std::move(sp)).first->second;
}

int64_t cg_table_rows(int l1, int lambda) { return (int64_t)(2 * lambda + 1) * ((2 * l1 + 1 + 3) / 4 * 4); }

// The table of one (l1, l2, lambda) for the tensor-core kernel: per mu and m1
// (padded to a multiple of 4) its two terms; false when an m1 has more.
bool cg_coef_rows(const SparseCg& sp, int l1, int lambda, std::vector<CgCoef>& table) {
    const int pad = (2 * l1 + 1 + 3) / 4 * 4;
    const size_t base = table.size();
    table.resize(base + (size_t)cg_table_rows(l1, lambda), CgCoef{});
    for (int mu = 0; mu <= 2 * lambda; mu++)
        for (int e = sp.mu_starts[mu]; e < sp.mu_starts[mu + 1]; e++) {
            const CgEntry& x = sp.entries[e];
            CgCoef& c = table[base + (size_t)mu * pad + x.m1];
            if (c.v0 == 0.0) {
                c.v0 = x.value;
                c.m0 = x.m2 * CG_PITCH;
            } else if (c.v1 == 0.0) {
                c.v1 = x.value;
                c.m1 = x.m2 * CG_PITCH;
            } else {
                return false;
            }
        }
    return true;
}

bool cg_vector_stores(const featomic_b200_cg_task_t& t) {
    const int64_t stride = t.output_stride == 0 ? (int64_t)t.n_first * t.n_second : t.output_stride;
    return t.n_second % 2 == 0 && stride % 2 == 0 && reinterpret_cast<uintptr_t>(t.output) % 16 == 0;
}

// Whether the tensor cores are worth it: all tasks of more than 16 properties on
// a side (with two or fewer 8-wide tiles a side the row loop's own work is not
// covered by the DMMAs; 2000 centres, l <= 4: 24 x 24 properties, l <= 3, 0.33
// against 0.58 ms; 16 x 16 0.63 against 0.56 ms; 8 x 8 0.53 against 0.30 ms), and
// enough output for their tables.  Those are larger than the thread kernel's
// lists, are made and copied by the host (l <= 6: 456 KB, 107 us of a call of 350),
// and pay when the device has work to cover it with: 2500 times their size in
// outputs that take 16-byte stores (l <= 2, 32 x 32 properties, 30 samples 42.7
// against 45.8 us with the tables, 300 samples 66.9 and 46.7; l <= 6, 30 samples
// 350 and 457, 100 samples 541 and 456); the thread kernel is slower with others,
// for which 1000 times are enough (17 x 17, l <= 6: 100 samples 400 and 458, 300
// samples 882 and 595), and 60 times tables of up to 16 KB (20 x 33, l <= 2: 10
// samples 54 and 46).
bool cg_product_mma_pays(const featomic_b200_cg_task_t* tasks, size_t n_tasks) {
    std::vector<uint64_t> orders;
    int64_t out = 0;
    bool vector = true;
    for (size_t i = 0; i < n_tasks; i++) {
        const auto& t = tasks[i];
        const int64_t items = t.n_samples * (int64_t)t.n_first * t.n_second;
        if (items == 0) continue;
        if (t.n_first <= 16 || t.n_second <= 16) return false;
        out += items * (2 * t.lambda + 1) * (int64_t)sizeof(double);
        vector = vector && cg_vector_stores(t);
        orders.push_back((uint64_t)t.l1 << 40 | (uint64_t)t.l2 << 20 | (uint64_t)t.lambda);
    }
    std::sort(orders.begin(), orders.end());
    orders.erase(std::unique(orders.begin(), orders.end()), orders.end());
    int64_t table = 0;
    for (uint64_t o : orders) table += cg_table_rows((int)(o >> 40), (int)(o & 0xfffff)) * (int64_t)sizeof(CgCoef);
    const int64_t times = vector ? 2500 : table > 16 * 1024 ? 1000 : 60;
    return out >= times * (table + 6000);  // 6000: what the other host work of a call is worth
}

// FP64 products on the tensor cores; false (nothing launched) when one of the
// tasks does not fit the kernel.
bool cg_product_mma(const featomic_b200_cg_task_t* tasks, size_t n_tasks, cudaStream_t stream) {
    std::vector<DeviceCgGroup> groups;
    std::vector<CgRow> rows;
    std::vector<CgCoef> table;
    std::map<std::tuple<int, int, int>, int32_t> known;
    int64_t warps = 0;
    size_t warp_doubles = 0;
    for (size_t i = 0; i < n_tasks; i++) {
        const auto& t = tasks[i];
        const int64_t pq = (int64_t)t.n_first * t.n_second;
        if (t.n_samples * pq == 0) continue;
        const int64_t stride = t.output_stride == 0 ? pq : t.output_stride;
        auto at = known.find({t.l1, t.l2, t.lambda});
        if (at == known.end()) {
            const int32_t start = (int32_t)table.size();
            if (!cg_coef_rows(sparse_cg(t.l1, t.l2, t.lambda), t.l1, t.lambda, table)) return false;
            at = known.emplace(std::make_tuple(t.l1, t.l2, t.lambda), start).first;
        }
        const bool vector = cg_vector_stores(t);
        const int pad = (2 * t.l1 + 1 + 3) / 4 * 4;
        bool joins = false;
        if (!groups.empty()) {
            const DeviceCgGroup& g = groups.back();
            joins = g.first == t.first && g.second == t.second && g.n_samples == t.n_samples && g.n_first == t.n_first &&
                    g.n_second == t.n_second && g.m1_count == 2 * t.l1 + 1 && g.m2_count == 2 * t.l2 + 1 &&
                    g.vector == (int)vector && g.row_end - g.row_begin < CG_GROUP_ROWS;
        }
        if (!joins) {
            DeviceCgGroup g{};
            g.first = static_cast<const double*>(t.first);
            g.second = static_cast<const double*>(t.second);
            g.n_samples = t.n_samples;
            g.warp_start = warps;
            g.n_first = t.n_first;
            g.n_second = t.n_second;
            g.m1_count = 2 * t.l1 + 1;
            g.m2_count = 2 * t.l2 + 1;
            g.row_begin = g.row_end = (int32_t)rows.size();
            g.p_blocks = (t.n_first + 31) / 32;
            g.q_blocks = (t.n_second + 31) / 32;
            g.p_size = ((t.n_first + g.p_blocks - 1) / g.p_blocks + 7) / 8 * 8;
            g.q_size = ((t.n_second + g.q_blocks - 1) / g.q_blocks + 7) / 8 * 8;
            g.vector = vector;
            warps += t.n_samples * g.p_blocks * g.q_blocks;
            warp_doubles = std::max(warp_doubles, (size_t)(pad + g.m2_count) * CG_PITCH);
            groups.push_back(g);
        }
        for (int mu = 0; mu <= 2 * t.lambda; mu++)
            rows.push_back(CgRow{static_cast<double*>(t.output) + mu * stride, (2 * t.lambda + 1) * stride,
                                 at->second + mu * pad, 0});
        groups.back().row_end = (int32_t)rows.size();
    }
    if (groups.empty()) return true;
    const size_t smem = CG_MMA_WARPS * warp_doubles * sizeof(double);
    const int64_t blocks = (warps + CG_MMA_WARPS - 1) / CG_MMA_WARPS;
    if (smem > 200 * 1024 || blocks > 0x7fffffffLL) return false;
    const size_t gb = (groups.size() * sizeof(DeviceCgGroup) + 31) / 32 * 32, rb = (rows.size() * sizeof(CgRow) + 31) / 32 * 32,
                 tb = table.size() * sizeof(CgCoef);
    std::vector<unsigned char> host(gb + rb + tb, 0);
    std::memcpy(host.data(), groups.data(), groups.size() * sizeof(DeviceCgGroup));
    std::memcpy(host.data() + gb, rows.data(), rows.size() * sizeof(CgRow));
    std::memcpy(host.data() + gb + rb, table.data(), tb);
    unsigned char* buffer = nullptr;
    CUDA_CHECK(cudaMallocAsync(reinterpret_cast<void**>(&buffer), host.size(), stream));
    // staged before the call returns (pageable source)
    CUDA_CHECK(cudaMemcpyAsync(buffer, host.data(), host.size(), cudaMemcpyHostToDevice, stream));
    allow_shared_memory(cg_product_mma_kernel, smem);
    cg_product_mma_kernel<<<(unsigned)blocks, 32 * CG_MMA_WARPS, smem, stream>>>(
        reinterpret_cast<const DeviceCgGroup*>(buffer), (int)groups.size(), reinterpret_cast<const CgRow*>(buffer + gb),
        reinterpret_cast<const CgCoef*>(buffer + gb + rb), (int)warp_doubles);
    CUDA_CHECK(cudaGetLastError());
    CUDA_CHECK(cudaFreeAsync(buffer, stream));
    return true;
}

}  // namespace

void cg_product(const featomic_b200_cg_task_t* tasks, size_t n_tasks, int precision, cudaStream_t stream) {
    if (precision != 32 && precision != 64) throw invalid_parameter("precision must be 32 or 64");
    for (size_t i = 0; i < n_tasks; i++) {
        const auto& t = tasks[i];
        if (t.n_samples < 0 || t.n_first < 0 || t.n_second < 0)
            throw invalid_parameter("negative size in Clebsch-Gordan task " + std::to_string(i));
        const int64_t pq = (int64_t)t.n_first * t.n_second;
        if (t.n_samples * pq == 0) continue;
        if (!t.first || !t.second || !t.output)
            throw invalid_parameter("NULL array in Clebsch-Gordan task " + std::to_string(i));
        sparse_cg(t.l1, t.l2, t.lambda);  // rejects impossible orders
        if (t.output_stride != 0 && t.output_stride < pq)
            throw invalid_parameter("output_stride of Clebsch-Gordan task " + std::to_string(i) +
                                    " is smaller than n_first * n_second");
    }
    if (precision == 64 && cg_product_mma_pays(tasks, n_tasks) && cg_product_mma(tasks, n_tasks, stream)) return;
    std::vector<DeviceCgTask> dev;
    std::vector<CgEntry> entries;
    std::vector<int32_t> mu_starts;
    int64_t blocks = 0;
    for (size_t i = 0; i < n_tasks; i++) {
        const auto& t = tasks[i];
        const int64_t items = t.n_samples * (int64_t)t.n_first * t.n_second;
        if (items == 0) continue;
        const SparseCg& sp = sparse_cg(t.l1, t.l2, t.lambda);
        DeviceCgTask d;
        d.first = t.first;
        d.second = t.second;
        d.output = t.output;
        d.n_samples = t.n_samples;
        d.block_start = blocks;
        const int64_t pq = (int64_t)t.n_first * t.n_second;
        d.out_stride = t.output_stride == 0 ? pq : t.output_stride;
        d.n_first = t.n_first;
        d.n_second = t.n_second;
        d.lambda = t.lambda;
        d.m1_count = 2 * t.l1 + 1;
        d.m2_count = 2 * t.l2 + 1;
        d.entries = (int32_t)entries.size();
        d.mu_offsets = (int32_t)mu_starts.size();
        const size_t align = 4 * (precision == 64 ? sizeof(double) : sizeof(float));
        d.vector = t.n_second % CG_QV == 0 && d.out_stride % CG_QV == 0 && reinterpret_cast<uintptr_t>(t.second) % std::min<size_t>(align, 16) == 0 &&
                   reinterpret_cast<uintptr_t>(t.output) % std::min<size_t>(align, 16) == 0;
        d.vector_first = t.n_first % CG_PV == 0 && reinterpret_cast<uintptr_t>(t.first) % 16 == 0;
        entries.insert(entries.end(), sp.entries.begin(), sp.entries.end());
        mu_starts.insert(mu_starts.end(), sp.mu_starts.begin(), sp.mu_starts.end());
        dev.push_back(d);
        const int64_t threads = t.n_samples * ((t.n_first + CG_PV - 1) / CG_PV) * ((t.n_second + CG_QV - 1) / CG_QV);
        blocks += (threads + CG_THREADS - 1) / CG_THREADS;
    }
    if (dev.empty()) return;
    if (blocks > 0x7fffffffLL) throw invalid_parameter("Clebsch-Gordan product too large for one launch");
    // one device buffer for the three tables, released in stream order
    const size_t tb = dev.size() * sizeof(DeviceCgTask);
    const size_t eb = std::max<size_t>(entries.size(), 1) * sizeof(CgEntry);
    const size_t mb = mu_starts.size() * sizeof(int32_t);
    const size_t e_off = (tb + 15) / 16 * 16, m_off = e_off + (eb + 15) / 16 * 16, total = m_off + mb;
    std::vector<unsigned char> host(total, 0);
    std::memcpy(host.data(), dev.data(), tb);
    if (!entries.empty()) std::memcpy(host.data() + e_off, entries.data(), entries.size() * sizeof(CgEntry));
    std::memcpy(host.data() + m_off, mu_starts.data(), mb);
    unsigned char* buffer = nullptr;
    CUDA_CHECK(cudaMallocAsync(reinterpret_cast<void**>(&buffer), total, stream));
    // a copy from pageable host memory returns once the source has been
    // staged, so `host` may be released when this function returns
    CUDA_CHECK(cudaMemcpyAsync(buffer, host.data(), total, cudaMemcpyHostToDevice, stream));
    const auto* d_tasks = reinterpret_cast<const DeviceCgTask*>(buffer);
    const auto* d_entries = reinterpret_cast<const CgEntry*>(buffer + e_off);
    const auto* d_mu = reinterpret_cast<const int32_t*>(buffer + m_off);
    if (precision == 64)
        cg_product_kernel<double><<<(unsigned)blocks, CG_THREADS, 0, stream>>>(d_tasks, (int)dev.size(), d_entries, d_mu);
    else
        cg_product_kernel<float><<<(unsigned)blocks, CG_THREADS, 0, stream>>>(d_tasks, (int)dev.size(), d_entries, d_mu);
    CUDA_CHECK(cudaGetLastError());
    CUDA_CHECK(cudaFreeAsync(buffer, stream));
}

void cg_couple(const featomic_b200_cg_couple_task_t* tasks, size_t n_tasks, int precision, cudaStream_t stream) {
    if (precision != 32 && precision != 64) throw invalid_parameter("precision must be 32 or 64");
    std::vector<DeviceCoupleTask> dev;
    std::vector<CgEntry> entries;
    std::vector<int32_t> mu_starts;
    int64_t blocks = 0;
    for (size_t i = 0; i < n_tasks; i++) {
        const auto& t = tasks[i];
        if (t.n_outer < 0 || t.n_inner < 0)
            throw invalid_parameter("negative size in Clebsch-Gordan coupling task " + std::to_string(i));
        const int64_t items = t.n_outer * t.n_inner;
        const SparseCg& sp = sparse_cg(t.l1, t.l2, t.lambda);
        if (items == 0) continue;
        if (!t.input || !t.output)
            throw invalid_parameter("NULL array in Clebsch-Gordan coupling task " + std::to_string(i));
        DeviceCoupleTask d;
        d.input = t.input;
        d.output = t.output;
        d.n_outer = t.n_outer;
        d.n_inner = t.n_inner;
        d.block_start = blocks;
        d.m1_count = 2 * t.l1 + 1;
        d.m2_count = 2 * t.l2 + 1;
        d.lambda = t.lambda;
        d.entries = (int32_t)entries.size();
        d.mu_offsets = (int32_t)mu_starts.size();
        entries.insert(entries.end(), sp.entries.begin(), sp.entries.end());
        mu_starts.insert(mu_starts.end(), sp.mu_starts.begin(), sp.mu_starts.end());
        dev.push_back(d);
        blocks += (items + CG_THREADS - 1) / CG_THREADS;
    }
    if (dev.empty()) return;
    if (blocks > 0x7fffffffLL) throw invalid_parameter("Clebsch-Gordan coupling too large for one launch");
    const size_t tb = dev.size() * sizeof(DeviceCoupleTask);
    const size_t eb = std::max<size_t>(entries.size(), 1) * sizeof(CgEntry);
    const size_t mb = mu_starts.size() * sizeof(int32_t);
    const size_t e_off = (tb + 15) / 16 * 16, m_off = e_off + (eb + 15) / 16 * 16, total = m_off + mb;
    std::vector<unsigned char> host(total, 0);
    std::memcpy(host.data(), dev.data(), tb);
    if (!entries.empty()) std::memcpy(host.data() + e_off, entries.data(), entries.size() * sizeof(CgEntry));
    std::memcpy(host.data() + m_off, mu_starts.data(), mb);
    unsigned char* buffer = nullptr;
    CUDA_CHECK(cudaMallocAsync(reinterpret_cast<void**>(&buffer), total, stream));
    // staged before the call returns (pageable source), as above
    CUDA_CHECK(cudaMemcpyAsync(buffer, host.data(), total, cudaMemcpyHostToDevice, stream));
    const auto* d_tasks = reinterpret_cast<const DeviceCoupleTask*>(buffer);
    const auto* d_entries = reinterpret_cast<const CgEntry*>(buffer + e_off);
    const auto* d_mu = reinterpret_cast<const int32_t*>(buffer + m_off);
    if (precision == 64)
        cg_couple_kernel<double><<<(unsigned)blocks, CG_THREADS, 0, stream>>>(d_tasks, (int)dev.size(), d_entries, d_mu);
    else
        cg_couple_kernel<float><<<(unsigned)blocks, CG_THREADS, 0, stream>>>(d_tasks, (int)dev.size(), d_entries, d_mu);
    CUDA_CHECK(cudaGetLastError());
    CUDA_CHECK(cudaFreeAsync(buffer, stream));
}

}  // namespace fb200
