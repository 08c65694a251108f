// Per-centre contractions of the dense power spectrum with a warp per centre,
// straight from global memory to matrix instructions (larger bases in FP32 are in
// dense_mma.cu):
//
//   values  P_l = X_l^T X_l, X_l[m][(s, n)] = c[s][l m][n]
//           P_ab[l][n1][n2] = scale(l, a != b) P_l[(a, n1), (b, n2)]
//           (featomic/src/calculators/soap/power_spectrum.rs:529-780)
//   dL/dc   of a loss whose dL/dP row belongs to the centre's species (the
//           weights of a linear model): D_l[(a, n)][(c, m)] =
//           sum_(b, q) G'_l[(a, n), (b, q)] X_l[(c, m)][(b, q)], one left
//           operand for all centres c of the species
//
// A product of one centre is 32 x 32 x 13 at most, far below a tcgen05 tile:
// dense_mma.cu puts four centres on the diagonal of a 128 x 128 tile, and
// spends its time on building operands in shared memory and waiting for the
// round's MMAs.  Here the fragment layout of mma.sync (FP32: m16n8k8 TF32
// with operands split into hi + lo, three products; FP64: m8n8k4) is the
// layout of the coefficients in memory: a fragment of X_l is four rows m of
// eight consecutive (s, n), one coalesced load per element, and is the left
// and the right operand of P_l at once.  The kernels are bound by the latency of
// those loads: a warp's steps follow one another, at a third of the warps that an
// SM holds (65 to 128 registers).
#include <algorithm>
#include <type_traits>

#include "dense.hpp"

namespace fb200 {

namespace {

constexpr int DW_WARPS = 8;

// power spectrum normalisation 1 / ((-1)^l sqrt(2l + 1)), times sqrt(2) for
// two different neighbour species: [l] same species, [32 + l] mixed
template <typename T>
__device__ __forceinline__ void fill_scales(T* table) {
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        const int l = i & 31;
        const double s = sqrt((double)(2 * l + 1));
        table[i] = (T)(((i >= 32) ? 1.4142135623730951 : 1.0) * (1.0 / ((l % 2 == 0) ? s : -s)));
    }
}

__device__ __forceinline__ int key_of(int a, int b, int S) { return a * S - a * (a - 1) / 2 + (b - a); }

__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    lo = __float_as_uint(x - __uint_as_float(hi));
}

// rows g and g + 8 of a 16 x 8 tile: (c0, c1) and (c2, c3)
__device__ __forceinline__ void mma_tf32(float (&top)[2], float (&bottom)[2], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(top[0]), "+f"(top[1]), "+f"(bottom[0]), "+f"(bottom[1])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

__device__ __forceinline__ void store2(float* p, float x, float y) { __stcs(reinterpret_cast<float2*>(p), make_float2(x, y)); }
__device__ __forceinline__ void store2(double* p, double x, double y) { __stcs(reinterpret_cast<double2*>(p), make_double2(x, y)); }

// acc (4 x 4 tiles of 8 x 8, lane: row lane / 4, columns 2 (lane % 4) + {0, 1})
// += the products of four m: x, y [column tile] hold rows m = lane % 4 at column
// lane / 4.  Tile (i, j) is computed when bit 4 i + j of `need` is set.
__device__ __forceinline__ void step(double (&acc)[4][4][2], const double (&x)[4], const double (&y)[4], unsigned need) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (need & (1u << (4 * i + j))) mma_f64(acc[i][j], x[i], y[j]);
}

// One step of m (8 in FP32, 4 in FP64) of the upper tiles (i <= j < NT) of
// P = X^T X: x [tile] holds rows m = lane % 4 (and + 4) at column lane / 4.
template <int NT>
__device__ __forceinline__ void step_upper(float (&acc)[NT + 1][NT][2], const float (&x)[NT][2]) {
    uint32_t h[NT + 1][2], l[NT + 1][2];
    h[NT][0] = h[NT][1] = l[NT][0] = l[NT][1] = 0;
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) split(x[j][e], h[j][e], l[j][e]);
#pragma unroll
    for (int i = 0; i < NT; i += 2)
#pragma unroll
        for (int j = i; j < NT; j++) {
            mma_tf32(acc[i][j], acc[i + 1][j], h[i][0], h[i + 1][0], h[i][1], h[i + 1][1], h[j][0], h[j][1]);
            mma_tf32(acc[i][j], acc[i + 1][j], h[i][0], h[i + 1][0], h[i][1], h[i + 1][1], l[j][0], l[j][1]);
            mma_tf32(acc[i][j], acc[i + 1][j], l[i][0], l[i + 1][0], l[i][1], l[i + 1][1], h[j][0], h[j][1]);
        }
}
template <int NT>
__device__ __forceinline__ void step_upper(double (&acc)[NT + 1][NT][2], const double (&x)[NT][1]) {
#pragma unroll
    for (int i = 0; i < NT; i++)
#pragma unroll
        for (int j = i; j < NT; j++) mma_f64(acc[i][j], x[i][0], x[j][0]);
}

// ... and of four m of D^T X + X^T D
template <int NT>
__device__ __forceinline__ void step_upper2(double (&acc)[NT][NT][2], const double (&x)[NT], const double (&d)[NT]) {
#pragma unroll
    for (int i = 0; i < NT; i++)
#pragma unroll
        for (int j = i; j < NT; j++) {
            mma_f64(acc[i][j], x[i], d[j]);
            mma_f64(acc[i][j], d[i], x[j]);
        }
}

// nmax <= 8 and NT <= 4 species: a tile is one species pair (nmax < 8 padded
// with zeros), and everything that depends on the species is known to the
// compiler.  Bound by load latency (10 of 15 stall cycles an instruction at 21
// warps per SM, DRAM half busy, 1.4 of 4 instructions a cycle): 20 000 atoms, 4
// species, lmax 6, nmax 8 (125 MB read, 358 written) 0.109 ms = 4.4 TB/s, 0.232
// with four centres on a tcgen05 tile; with the species found at run time 0.174.
// FP64, 2000 atoms: 17 us, 52 with a CTA per centre.
// `energy`: with a linear model's weights [species][keys][props], the centre's
// energy sum_P w P from the values on their way out (134 128 atoms: 0.72 ms;
// 1.49 + 0.53 with a kernel that read them back): a lane's ten products of an l
// and parity in T, their sums over l and lanes in FP64 (one sum of 140 terms in
// FP32 was twice as far from the exact one as the 256-thread sums before it).
template <typename T, bool ENERGY, int NT, bool N8>
__global__ void __launch_bounds__(32 * DW_WARPS, 3)
dense_contraction_tiles(DenseArgs<T> a, const T* __restrict__ weights, T* __restrict__ energy) {
    constexpr int E = sizeof(T) == 4 ? 2 : 1, STEP = 4 * E;
    __shared__ T scales[64];
    fill_scales(scales);
    __syncthreads();
    const int lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    const int64_t c = (int64_t)blockIdx.x * DW_WARPS + (threadIdx.x >> 5);
    if (c >= a.n_atoms) return;
    const int N = N8 ? 8 : a.nmax, K = a.K, P = (int)a.n_props;
    const int64_t first = N * g + 2 * t;  // this lane's two values of a tile
    const bool row = N8 || g < N, two = N8 || (row && (N & 1) == 0 && 2 * t < N), one = !N8 && !two && row;
    const T* X = a.coef + c * NT * (int64_t)K + N * t + (row ? g : 0);
    T* out = a.values + c * (NT * (NT + 1) / 2) * (int64_t)P + first;
    const T* w = ENERGY ? weights + (int64_t)a.atom_species[c] * (NT * (NT + 1) / 2) * P + first : nullptr;
    double sum = 0.0;
#pragma unroll 1
    for (int l = 0; l <= a.lmax; l++) {
        const int M = 2 * l + 1;
        T part[2] = {T(0), T(0)};  // of the energy
        T acc[NT + 1][NT][2];
#pragma unroll
        for (int i = 0; i <= NT; i++)
#pragma unroll
            for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = T(0);
#pragma unroll 1
        for (int m0 = 0; m0 < M; m0 += STEP) {
            T x[NT][E];
#pragma unroll
            for (int e = 0; e < E; e++) {
                const bool ok = m0 + t + 4 * e < M && row;
#pragma unroll
                for (int i = 0; i < NT; i++) x[i][e] = ok ? __ldg(X + i * K + N * (m0 + 4 * e)) : T(0);
            }
            step_upper<NT>(acc, x);
        }
        X += N * M;
        const T same = scales[l], other = scales[32 + l];
        int key = 0;
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int j = i; j < NT; j++, key++) {
                const T scale = i != j ? other : same;
                const T v0 = acc[i][j][0] * scale, v1 = acc[i][j][1] * scale;
                if (two) {
                    store2(out + key * P, v0, v1);
                    if (ENERGY) {
                        part[0] += v0 * w[key * P];
                        part[1] += v1 * w[key * P + 1];
                    }
                } else if (one) {
                    if (2 * t < N) {
                        out[key * P] = v0;
                        if (ENERGY) part[0] += v0 * w[key * P];
                    }
                    if (2 * t + 1 < N) {
                        out[key * P + 1] = v1;
                        if (ENERGY) part[1] += v1 * w[key * P + 1];
                    }
                }
            }
        out += N * N;
        if (ENERGY) {
            w += N * N;
            sum += (double)part[0] + (double)part[1];
        }
    }
    if (ENERGY) {
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) energy[c] = (T)sum;
    }
}

// Tangent of the power spectrum, dP = dX^T X + X^T dX, by the same tiles: a
// warp per centre (the CUDA-core kernel with a warp per species pair reads
// four coefficients for two multiply-adds).  FP32 coefficients are multiplied
// and summed in FP64 as well: TF32 operands split into hi + lo, as for the
// values, are four times as far from the exact products as the CUDA cores'
// FP32 multiply-adds (2.1e-7 against 5.3e-8 of the norm).  Bound by its stores
// and the load latency of a warp's serial steps.  1500 atoms, 3 species,
// lmax 6, nmax 8, FP32: 13 us (57 on the CUDA cores, 12 with TF32).
template <typename T, int NT, bool N8>
__global__ void __launch_bounds__(32 * DW_WARPS, 2)
dense_tangent_tiles(DenseArgs<T> a, const T* __restrict__ tcoef, T* __restrict__ tvalues) {
    __shared__ double scales[64];
    fill_scales(scales);
    __syncthreads();
    const int lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    const int64_t c = (int64_t)blockIdx.x * DW_WARPS + (threadIdx.x >> 5);
    if (c >= a.n_atoms) return;
    const int N = N8 ? 8 : a.nmax, K = a.K, P = (int)a.n_props;
    const bool row = N8 || g < N, two = N8 || (row && (N & 1) == 0 && 2 * t < N), one = !N8 && !two && row;
    int64_t at = c * NT * (int64_t)K + N * t + (row ? g : 0);
    T* out = tvalues + c * (NT * (NT + 1) / 2) * (int64_t)P + N * g + 2 * t;
#pragma unroll 1
    for (int l = 0; l <= a.lmax; l++) {
        const int M = 2 * l + 1;
        double acc[NT][NT][2];
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 1
        for (int m0 = 0; m0 < M; m0 += 4) {
            double x[NT], d[NT];
            const bool ok = m0 + t < M && row;
#pragma unroll
            for (int i = 0; i < NT; i++) {
                x[i] = ok ? (double)__ldg(a.coef + at + i * K + N * m0) : 0.0;
                d[i] = ok ? (double)__ldg(tcoef + at + i * K + N * m0) : 0.0;
            }
            step_upper2<NT>(acc, x, d);
        }
        at += N * M;
        const double same = scales[l], other = scales[32 + l];
        int key = 0;
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int j = i; j < NT; j++, key++) {
                const double scale = i != j ? other : same;
                const T v0 = (T)(acc[i][j][0] * scale), v1 = (T)(acc[i][j][1] * scale);
                if (two) {
                    store2(out + key * P, v0, v1);
                } else if (one) {
                    if (2 * t < N) out[key * P] = v0;
                    if (2 * t + 1 < N) out[key * P + 1] = v1;
                }
            }
        out += N * N;
    }
}

// The values in FP64 for any nmax and number of species, by blocks of 32 x 32
// (s, n); dense_contraction_by_warp says where.  What depends on a row or column
// alone is found once per block: an offset among the values is a row's term plus
// a column's.
__global__ void __launch_bounds__(32 * DW_WARPS, 2) dense_contraction_warp(DenseArgs<double> a) {
    __shared__ double scales[64];
    fill_scales(scales);
    __syncthreads();
    const int lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    const int64_t c = (int64_t)blockIdx.x * DW_WARPS + (threadIdx.x >> 5);
    if (c >= a.n_atoms) return;
    const int S = a.n_species, N = a.nmax, K = a.K, SN = S * N, NN = N * N, P = (int)a.n_props;
    const int64_t KP = (int64_t)a.n_keys * P;
    const double* X = a.coef + c * S * (int64_t)K;
    double* out_c = a.values + c * KP;
    const bool pairs = (N & 1) == 0;  // two neighbouring columns are of one species, and 2-element aligned
    for (int r0 = 0; r0 < SN; r0 += 32) {
        // columns from the row block's first species on
        for (int q0 = r0 / N * N / 32 * 32; q0 < SN; q0 += 32) {
            const bool diagonal = q0 == r0;
            // tiles with a column species not below every row species
            unsigned need = 0;
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int first = r0 + 8 * i, last = min(q0 + 8 * j + 7, SN - 1);
                    if (first < SN && q0 + 8 * j < SN && last / N >= first / N) need |= 1u << (4 * i + j);
                }
            // -1: past the last (s, n)
            int x_at[4], y_at[4], row_at[4], column_at[4];
            // per tile 4 i + j and value e of the lane, bit 16 e + 4 i + j
            unsigned write = 0, equal = 0, crosses = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int r = r0 + 8 * i + g, q = q0 + 8 * i + g, s1 = r / N, n1 = r - s1 * N;
                x_at[i] = r < SN ? s1 * K + n1 : -1;
                y_at[i] = q < SN ? q / N * K + q % N : -1;
                row_at[i] = (key_of(s1, s1, S) - s1) * P + n1 * N;
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int c2 = q0 + 8 * j + 2 * t + e, s2 = c2 / N;
                        if ((need & (1u << (4 * i + j))) && r < SN && c2 < SN && s1 <= s2) write |= 1u << (16 * e + 4 * i + j);
                        if (s1 == s2) equal |= 1u << (16 * e + 4 * i + j);
                    }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int c2 = q0 + 8 * j + 2 * t, s2 = c2 / N;
                column_at[j] = s2 * P + c2 - s2 * N;
                if ((c2 + 1) / N != s2) crosses |= 1u << j;
            }
#pragma unroll 1
            for (int l = 0; l <= a.lmax; l++) {
                const int M = 2 * l + 1;
                double acc[4][4][2];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 1
                for (int m0 = 0; m0 < M; m0 += 4) {
                    double x[4], y[4];
                    const int m = m0 + t;
                    const double* row = X + (l * l + m) * N;
                    const bool ok = m < M;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        x[i] = ok && x_at[i] >= 0 ? __ldg(row + x_at[i]) : 0.0;
                        if (!diagonal) y[i] = ok && y_at[i] >= 0 ? __ldg(row + y_at[i]) : 0.0;
                    }
                    if (diagonal) step(acc, x, x, need);
                    else step(acc, x, y, need);
                }
                const double same = scales[l], other = scales[32 + l];
                double* out = out_c + l * NN;
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int at = row_at[i] + column_at[j];
                        const double scale0 = equal & (1u << (4 * i + j)) ? same : other;
                        const double v0 = acc[i][j][0] * scale0;
                        if (pairs) {
                            if (!(write & (1u << (4 * i + j)))) continue;
                            store2(out + at, v0, acc[i][j][1] * scale0);
                        } else {
                            if (write & (1u << (4 * i + j))) out[at] = v0;
                            if (write & (1u << (16 + 4 * i + j)))
                                out[at + (crosses & (1u << j) ? P - N + 1 : 1)] =
                                    acc[i][j][1] * (equal & (1u << (16 + 4 * i + j)) ? same : other);
                        }
                    }
            }
        }
    }
}

// dL/dc in FP64 (nmax <= 8, NT <= 4 species), a warp per centre:
//   D_l[(a, n)][m] = sum_(b, q) G'_l[(a, n), (b, q)] X_l[m][(b, q)]
// by 8 x 8 tiles over (a; eight m), with the scale of the species pair in the
// right operand.  MMA slot k = t of the two steps of a species is q = 2 t and
// 2 t + 1.  Bound by the loads of G (read once straight and once transposed):
// L1 77 % busy, 12 of 17 stall cycles an instruction wait for a load (4000
// atoms).  2000 atoms, 4 species, lmax 6: 37 us, 98 with a CTA per centre and its
// rows staged in shared memory.
template <int NT, bool N8>
__global__ void __launch_bounds__(32 * DW_WARPS, 2) dense_grad_coef_tiles(DenseArgs<double> a) {
    __shared__ double scales[64];
    fill_scales(scales);
    __syncthreads();
    const int lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    const int64_t c = (int64_t)blockIdx.x * DW_WARPS + (threadIdx.x >> 5);
    if (c >= a.n_atoms) return;
    const int N = N8 ? 8 : a.nmax, K = a.K, P = (int)a.n_props, NN = N * N;
    const double* G = a.grad_values + (a.grad_species ? (int64_t)a.grad_species[c] : c) * (NT * (NT + 1) / 2) * P;
    const double* X = a.coef + c * NT * (int64_t)K;
    double* out = a.grad_coef + c * NT * (int64_t)K;
    const bool row = N8 || g < N;
    const bool k_ok[2] = {N8 || 2 * t < N, N8 || 2 * t + 1 < N};
    for (int l = 0; l <= a.lmax; l++, G += NN) {
        const int M = 2 * l + 1;
        const double same = scales[l], other = scales[32 + l];
        for (int m0 = 0; m0 < M; m0 += 8) {
            // right operand: (l m) = m0 + g, (b, q)
            double xs[NT][2], xo[NT][2];
            const bool m_ok = m0 + g < M;
#pragma unroll
            for (int b = 0; b < NT; b++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const double v = m_ok && k_ok[e] ? __ldg(X + b * K + (l * l + m0 + g) * N + 2 * t + e) : 0.0;
                    xs[b][e] = v * same;
                    xo[b][e] = v * other;
                }
            double acc[NT][2];
#pragma unroll
            for (int i = 0; i < NT; i++) acc[i][0] = acc[i][1] = 0.0;
#pragma unroll
            for (int i = 0; i < NT; i++)
#pragma unroll
                for (int b = 0; b < NT; b++) {
                    const double* gk = G + (i < b ? i * NT - i * (i - 1) / 2 + b - i : b * NT - b * (b - 1) / 2 + i - b) * P;
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const bool ok = row && k_ok[e];
                        const int q = 2 * t + e;
                        double v = 0.0;
                        if (i <= b) v = ok ? __ldg(gk + g * N + q) : 0.0;
                        if (i >= b) v += ok ? __ldg(gk + q * N + g) : 0.0;
                        mma_f64(acc[i], v, i == b ? xs[b][e] : xo[b][e]);
                    }
                }
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int m = m0 + 2 * t + e;
                if (m >= M || !row) continue;
#pragma unroll
                for (int i = 0; i < NT; i++) out[i * K + (l * l + m) * N + g] = acc[i][e];
            }
        }
    }
}

// dL/dc for rows of dL/dP by species (nmax even, S nmax <= 32).  A CTA owns
// up to DG_CENTRES centres of one species; per l the left operand G'_l (32 x
// 32, split into hi and lo) is built in shared memory and kept in each warp's
// registers, and the warps take the columns (c, m), eight at a time.  MMA
// slots k = t and t + 4 are (b, q) = 2 t and 2 t + 1, so that both operands
// are read in pairs.  Bound by load latency and its 116 registers (15 warps per
// SM, 1.7 of 4 instructions a cycle, DRAM a quarter busy).  134 128 atoms, 4
// species, lmax 6, nmax 8 (841 MB read and written): 0.74 to 0.83 ms; 2.95 with an
// operand per centre on tcgen05 tiles.
constexpr int DG_CENTRES = 64;
constexpr int DG_PITCH = 40;  // floats; rows 4 g apart hit banks 8 bytes apart

__global__ void __launch_bounds__(32 * DW_WARPS) dense_grad_coef_species(DenseArgs<float> a, const int32_t* __restrict__ order,
                                                                        const int32_t* __restrict__ tiles) {
    __shared__ float hi[32 * DG_PITCH], lo[32 * DG_PITCH];
    __shared__ float scales[64];
    __shared__ int32_t centres[DG_CENTRES];
    fill_scales(scales);
    const int species = tiles[3 * blockIdx.x], first = tiles[3 * blockIdx.x + 1], count = tiles[3 * blockIdx.x + 2];
    for (int i = threadIdx.x; i < count; i += blockDim.x) centres[i] = order[first + i];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    const int S = a.n_species, N = a.nmax, K = a.K, SN = S * N, NN = N * N;
    const float* G = a.grad_values + (int64_t)species * a.n_keys * a.n_props;
    int k_offset[4];  // (b, q) of this lane's pair of every k step, in a centre's coefficients
    int row_offset[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int r = 8 * k + 2 * t, ro = 8 * k + g;
        k_offset[k] = r < SN ? (r / N) * K + r - (r / N) * N : -1;
        row_offset[k] = ro < SN ? (ro / N) * K + ro - (ro / N) * N : -1;
    }
    for (int l = 0; l <= a.lmax; l++) {
        const int M = 2 * l + 1;
        __syncthreads();
        for (int i = threadIdx.x; i < 32 * 32; i += blockDim.x) {
            const int r = i >> 5, k = i & 31;
            float v = 0.0f;
            if (r < SN && k < SN) {
                const int sa = r / N, n = r - sa * N, sb = k / N, q = k - sb * N;
                const float* gl = G + (int64_t)key_of(min(sa, sb), max(sa, sb), S) * a.n_props + l * NN;
                if (sa < sb) v = gl[n * N + q];
                else if (sa > sb) v = gl[q * N + n];
                else v = gl[n * N + q] + gl[q * N + n];
                v *= scales[(sa != sb ? 32 : 0) + l];
            }
            uint32_t h, w;
            split(v, h, w);
            hi[r * DG_PITCH + k] = __uint_as_float(h);
            lo[r * DG_PITCH + k] = __uint_as_float(w);
        }
        __syncthreads();
        uint32_t ah[2][4][4], al[2][4][4];  // [16-row tile][k step][fragment]
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int at = (16 * i + 8 * e + g) * DG_PITCH + 8 * k + 2 * t;
                    const float2 h = *reinterpret_cast<const float2*>(hi + at), w = *reinterpret_cast<const float2*>(lo + at);
                    ah[i][k][e] = __float_as_uint(h.x);
                    ah[i][k][2 + e] = __float_as_uint(h.y);
                    al[i][k][e] = __float_as_uint(w.x);
                    al[i][k][2 + e] = __float_as_uint(w.y);
                }
        const int columns = count * M;
        for (int j = 8 * warp; j < columns; j += 8 * DW_WARPS) {
            // right operand: column j + g
            const int col = j + g, ci = col / M;
            const bool ok = col < columns;
            const float* x = ok ? a.coef + centres[ci] * (int64_t)(S * K) + (int64_t)(l * l + col - ci * M) * N : nullptr;
            float acc[4][2];
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = 0.0f;
            float2 v[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[k] = ok && k_offset[k] >= 0 ? __ldg(reinterpret_cast<const float2*>(x + k_offset[k])) : make_float2(0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t bh[2], bl[2];
                split(v[k].x, bh[0], bl[0]);
                split(v[k].y, bh[1], bl[1]);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint32_t(&h)[4] = ah[i][k];
                    const uint32_t(&w)[4] = al[i][k];
                    mma_tf32(acc[2 * i], acc[2 * i + 1], h[0], h[1], h[2], h[3], bh[0], bh[1]);
                    mma_tf32(acc[2 * i], acc[2 * i + 1], h[0], h[1], h[2], h[3], bl[0], bl[1]);
                    mma_tf32(acc[2 * i], acc[2 * i + 1], w[0], w[1], w[2], w[3], bh[0], bh[1]);
                }
            }
            // columns 2 t, 2 t + 1: their centres and m
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int oc = j + 2 * t + e, oi = oc / M;
                if (oc >= columns) continue;
                float* out = a.grad_coef + centres[oi] * (int64_t)(S * K) + (int64_t)(l * l + oc - oi * M) * N;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (row_offset[i] >= 0) out[row_offset[i]] = acc[i][e];
            }
        }
    }
}

// a tile per species pair
template <typename T>
bool dense_tiles(const DenseArgs<T>& a) {
    return a.nmax <= 8 && a.n_species <= 4;
}

}  // namespace

template <typename T>
bool dense_contraction_by_warp(const DenseArgs<T>& a) {
    // two values are stored at a time, and the FP32 forms have one rule
    if ((uintptr_t)a.values % 16 != 0 || a.lmax >= 32) return false;
    if constexpr (sizeof(T) == 4) {
        // FP32 as the CUDA cores' contraction where that is asked for, and from
        // l = 16 on; larger bases keep the tcgen05 tiles, or the CUDA cores
        // (a warp per centre lost to tcgen05 with more than 32 (s, n): 8000
        // atoms, 6 species, nmax 8 271 against 224 us, 16 species 441 against
        // 308, 300 atoms 99 against 26)
        return dense_mma_enabled() && a.lmax < 16 && dense_tiles(a);
    }
    // FP64.  A warp walks over all of a centre's l one after the other, which
    // takes enough centres to hide: the tiles lose to the four warps a centre of
    // dense.cu with l > 8 and few centres (30 atoms, 4 species, lmax 12 34
    // against 26 us, 3000 atoms 81 against 222), the blocks of 32 with fewer
    // than some 1000 centres (300 atoms, 10 species, nmax 14 222 against 85 us).
    // Blocks also lose to them with many idle rows or odd 8-byte accesses (8000
    // atoms, 5 species, nmax 8 306 against 267; nmax 5 460 against 253), and win
    // with full ones (8000 atoms, 4 species, nmax 16 218 against 464) and where a
    // centre's coefficients do not fit dense.cu's 48 KB (1200 atoms, 12 species,
    // lmax 9 319 against 622).
    if (dense_tiles(a)) return a.lmax <= 8 || a.n_atoms >= 2000;
    const int SN = a.n_species * a.nmax, blocks = (SN + 31) / 32;
    const bool full = a.nmax % 8 == 0 && 5 * SN >= 4 * 32 * blocks;
    const bool staged = a.nmax <= 16 && sizeof(T) * (size_t)a.n_species * a.K <= 48 * 1024;
    return a.n_atoms >= 1200 && (full || !staged);
}
template bool dense_contraction_by_warp<float>(const DenseArgs<float>&);
template bool dense_contraction_by_warp<double>(const DenseArgs<double>&);

template <typename T>
void launch_dense_contraction_warp(const DenseArgs<T>& a, cudaStream_t stream) {
    const unsigned blocks = (unsigned)((a.n_atoms + DW_WARPS - 1) / DW_WARPS);
    auto run = [&](auto kernel) { kernel<<<blocks, 32 * DW_WARPS, 0, stream>>>(a, a.energy_weights, a.energy); };
    auto tiles = [&](auto energy, auto n8) {
        constexpr bool EN = decltype(energy)::value, N8 = decltype(n8)::value;
        switch (a.n_species) {
            case 1: run(dense_contraction_tiles<T, EN, 1, N8>); break;
            case 2: run(dense_contraction_tiles<T, EN, 2, N8>); break;
            case 3: run(dense_contraction_tiles<T, EN, 3, N8>); break;
            default: run(dense_contraction_tiles<T, EN, 4, N8>); break;
        }
    };
    if (dense_tiles(a)) {
        if (a.nmax == 8) a.energy ? tiles(std::true_type(), std::true_type()) : tiles(std::false_type(), std::true_type());
        else a.energy ? tiles(std::true_type(), std::false_type()) : tiles(std::false_type(), std::false_type());
    } else {
        if constexpr (sizeof(T) == 8) dense_contraction_warp<<<blocks, 32 * DW_WARPS, 0, stream>>>(a);
    }
    CUDA_CHECK(cudaGetLastError());
}

template void launch_dense_contraction_warp<float>(const DenseArgs<float>&, cudaStream_t);
template void launch_dense_contraction_warp<double>(const DenseArgs<double>&, cudaStream_t);

template <typename T>
bool dense_tangent_by_warp(const DenseArgs<T>& a, const T* tvalues) {
    // the l of a centre come one after the other: with l > 8 and few centres the
    // CUDA cores' warp per species pair is faster (a whole JVP of 30 atoms, 4
    // species, nmax 5, lmax 9: 100 against 111 us; 600 atoms, lmax 12: 181 and 206)
    return (sizeof(T) == 8 || dense_mma_enabled()) && dense_tiles(a) && a.lmax < 32 &&
           (a.lmax <= 8 || a.n_atoms >= 2000) && (uintptr_t)tvalues % (2 * sizeof(T)) == 0;
}

template <typename T>
void launch_dense_tangent_warp(const DenseArgs<T>& a, const T* tcoef, T* tvalues, cudaStream_t stream) {
    const unsigned blocks = (unsigned)((a.n_atoms + DW_WARPS - 1) / DW_WARPS);
    auto run = [&](auto kernel) { kernel<<<blocks, 32 * DW_WARPS, 0, stream>>>(a, tcoef, tvalues); };
    auto tiles = [&](auto n8) {
        constexpr bool N8 = decltype(n8)::value;
        switch (a.n_species) {
            case 1: run(dense_tangent_tiles<T, 1, N8>); break;
            case 2: run(dense_tangent_tiles<T, 2, N8>); break;
            case 3: run(dense_tangent_tiles<T, 3, N8>); break;
            default: run(dense_tangent_tiles<T, 4, N8>); break;
        }
    };
    if (a.nmax == 8) tiles(std::true_type());
    else tiles(std::false_type());
    CUDA_CHECK(cudaGetLastError());
}

template bool dense_tangent_by_warp<float>(const DenseArgs<float>&, const float*);
template bool dense_tangent_by_warp<double>(const DenseArgs<double>&, const double*);
template void launch_dense_tangent_warp<float>(const DenseArgs<float>&, const float*, float*, cudaStream_t);
template void launch_dense_tangent_warp<double>(const DenseArgs<double>&, const double*, double*, cudaStream_t);

bool dense_grad_coef_by_warp(const DenseArgs<double>& a) { return a.nmax <= 8 && a.n_species <= 4 && a.lmax < 32; }

void launch_dense_grad_coef_warp(const DenseArgs<double>& a, cudaStream_t stream) {
    const unsigned blocks = (unsigned)((a.n_atoms + DW_WARPS - 1) / DW_WARPS);
    auto tiles = [&](auto n8) {
        constexpr bool N8 = decltype(n8)::value;
        switch (a.n_species) {
            case 1: dense_grad_coef_tiles<1, N8><<<blocks, 32 * DW_WARPS, 0, stream>>>(a); break;
            case 2: dense_grad_coef_tiles<2, N8><<<blocks, 32 * DW_WARPS, 0, stream>>>(a); break;
            case 3: dense_grad_coef_tiles<3, N8><<<blocks, 32 * DW_WARPS, 0, stream>>>(a); break;
            default: dense_grad_coef_tiles<4, N8><<<blocks, 32 * DW_WARPS, 0, stream>>>(a); break;
        }
    };
    if (a.nmax == 8) tiles(std::true_type());
    else tiles(std::false_type());
    CUDA_CHECK(cudaGetLastError());
}

bool dense_grad_coef_species_supported(const DenseArgs<float>& a) {
    // pairs of radial functions are read as 8 bytes
    return a.species_order && a.species_tiles && a.n_species_tiles > 0 && a.nmax % 2 == 0 && a.n_species * a.nmax <= 32 &&
           a.lmax < 32 && (uintptr_t)a.coef % 8 == 0;
}

void launch_dense_grad_coef_species(const DenseArgs<float>& a, cudaStream_t stream) {
    dense_grad_coef_species<<<(unsigned)a.n_species_tiles, 32 * DW_WARPS, 0, stream>>>(a, a.species_order, a.species_tiles);
    CUDA_CHECK(cudaGetLastError());
}

std::vector<int32_t> dense_species_tiles(const std::vector<int32_t>& species, int n_species, std::vector<int32_t>& order) {
    std::vector<int32_t> start(n_species + 1, 0), tiles;
    for (int32_t s : species) start[s + 1]++;
    for (int s = 0; s < n_species; s++) start[s + 1] += start[s];
    order.resize(species.size());
    std::vector<int32_t> next(start.begin(), start.end() - 1);
    for (size_t i = 0; i < species.size(); i++) order[next[species[i]]++] = (int32_t)i;
    for (int s = 0; s < n_species; s++)
        for (int32_t at = start[s]; at < start[s + 1]; at += DG_CENTRES)
            tiles.insert(tiles.end(), {s, at, std::min(DG_CENTRES, start[s + 1] - at)});
    return tiles;
}

}  // namespace fb200
