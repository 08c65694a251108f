// Forward-mode derivative of the expansion coefficients along a displacement
// of positions and cells, with one CTA per centre (the layout of
// centre_expansion.cuh): a direction of pair (i, j) adds
//   (+-1)^l [ (f' R_ln + f R'_ln) Y_lm (u . delta) + f / r R_ln (dY_lm . delta) ],
//   delta = t[j] - t[i] + shift . T_cell[system]
// (featomic/src/calculators/soap/spherical_expansion_pair.rs:323-422, the sign
// for a reversed pair) to its (centre, species).  One warp makes Y_lm (u .
// delta) and f / r dY_lm . delta, a lane per direction; the other the spline's
// weights; both then the spline rows and the sums over directions.  Nothing
// per pair goes to memory, where the general path writes pair records with
// derivatives and a tangent per (pair, l, m) and reads both again.  Bound by
// the latency of its load and recursion chains: 127 registers and the shared
// memory leave 14 warps per SM, which issue 1.3 of 4 instructions a cycle.  FP32,
// lmax 6, nmax 8: 1500 atoms of 3 species 53 to 64 us (188 us by pair records);
// with the power spectrum's tangent 6000 atoms of 4 species 240 us (1033), FP64
// 514 (1558).  dense_tangent_by_centre below says where it is used.
#include "centre_expansion.cuh"
#include "dense.hpp"

namespace fb200 {

namespace {

template <typename T>
struct TangentLayout {
    int yp, nr, rp;
    size_t weights, rows, bytes;
    __host__ __device__ TangentLayout(int lmax, int nmax, int levels) {
        constexpr int W = 16 / (int)sizeof(T);
        yp = ((lmax + 1) * (lmax + 1)) | 1;
        nr = (nmax + W - 1) / W * W;
        rp = (lmax + 1) * nr;
        // [chunk][R, P][rp], [chunk][2][yp], [chunk][f, f'], [chunk][levels][8], [chunk][levels]
        weights = (sizeof(T) * (size_t)CE_CHUNK * (2 * rp + 2 * yp + 2) + 15) / 16 * 16;
        rows = weights + sizeof(T) * (size_t)CE_CHUNK * levels * 8;
        bytes = rows + sizeof(int) * (size_t)CE_CHUNK * levels;
    }
};

template <typename T, int NCAP>
__global__ void __launch_bounds__(CE_THREADS) centre_tangent_kernel(DenseArgs<T> a, const T* __restrict__ tpos,
                                                                   const T* __restrict__ tcell, T* __restrict__ tcoef) {
    extern __shared__ __align__(16) unsigned char ct_smem[];
    constexpr int W = 16 / (int)sizeof(T);
    constexpr int ROUNDS = ((CE_LMAX + 1) * (CE_LMAX + 1) + CE_THREADS - 1) / CE_THREADS;
    using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    const DeviceSplineT<T>& spline = a.tab.spline;
    const int L = a.lmax, L2 = (L + 1) * (L + 1), N = a.nmax, S = a.n_species, levels = spline.levels;
    const TangentLayout<T> lay(L, N, levels);
    T* Rs = reinterpret_cast<T*>(ct_smem);
    T* Ys = Rs + CE_CHUNK * 2 * lay.rp;
    T* Fs = Ys + CE_CHUNK * 2 * lay.yp;
    T* Hs = reinterpret_cast<T*>(ct_smem + lay.weights);
    int* Ks = reinterpret_cast<int*>(ct_smem + lay.rows);
    const int64_t c = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t d0 = a.seg_offset[c * S], d1 = a.seg_offset[(c + 1) * S];
    T acc[ROUNDS][NCAP];
    int row[ROUNDS];
#pragma unroll
    for (int x = 0; x < ROUNDS; x++) {
        const int lm = threadIdx.x + x * CE_THREADS;
        int l = 0;
        while ((l + 1) * (l + 1) <= lm) l++;
        row[x] = min(l, L) * lay.nr;
#pragma unroll
        for (int n = 0; n < NCAP; n++) acc[x][n] = T(0);
    }
    auto sum_row = [&](const T* R, const T* Y, int x) {
        const int lm = min(threadIdx.x + x * CE_THREADS, L2 - 1);
        const T along = Y[lm], across = Y[lay.yp + lm];
#pragma unroll
        for (int n = 0; n < NCAP; n += W) {
            if (n < lay.nr) {
                const V v = *reinterpret_cast<const V*>(R + row[x] + n), p = *reinterpret_cast<const V*>(R + lay.rp + row[x] + n);
#pragma unroll
                for (int e = 0; e < W; e++)
                    acc[x][n + e] += along * reinterpret_cast<const T*>(&p)[e] + across * reinterpret_cast<const T*>(&v)[e];
            }
        }
    };
    int t = 0;
    int64_t end = a.seg_offset[c * S + 1];
    auto next_species = [&]() {
#pragma unroll
        for (int x = 0; x < ROUNDS; x++) {
            const int lm = threadIdx.x + x * CE_THREADS;
            if (lm < L2) {
                T* out = tcoef + ((c * S + t) * L2 + lm) * N;
                if (lay.nr == N && (uintptr_t)tcoef % 16 == 0) {
#pragma unroll
                    for (int n = 0; n < NCAP; n += W) {
                        V v;
#pragma unroll
                        for (int e = 0; e < W; e++) reinterpret_cast<T*>(&v)[e] = acc[x][n + e];
                        if (n < N) *reinterpret_cast<V*>(out + n) = v;
                    }
                } else {
#pragma unroll
                    for (int n = 0; n < NCAP; n++)
                        if (n < N) out[n] = acc[x][n];
                }
            }
#pragma unroll
            for (int n = 0; n < NCAP; n++) acc[x][n] = T(0);
        }
        t++;
        if (t < S) end = a.seg_offset[c * S + t + 1];
    };
    if (lay.nr != N)
        for (int w = threadIdx.x; w < CE_CHUNK * 2 * lay.rp; w += CE_THREADS) Rs[w] = T(0);
    for (int64_t dc = d0; dc < d1; dc += CE_CHUNK) {
        const int nd = (int)min((int64_t)CE_CHUNK, d1 - dc);
        __syncthreads();
        if (lane < nd) {
            const int32_t code = a.dir_code[dc + lane];
            const int64_t p = code >> 1;
            const double r = a.pairs.distance[p];
            if (warp == 1) {
                for (int v = 0; v < levels; v++) {
                    double2 knot, next;
                    const int k = level_interval(spline, v, r, knot, next);
                    const soap::HermiteWeights h = soap::hermite_weights(knot.x, next.x, r);
                    T* o = Hs + (lane * levels + v) * 8;
                    o[0] = (T)h.h00;
                    o[1] = (T)(h.h10 * h.delta);
                    o[2] = (T)h.h01;
                    o[3] = (T)(h.h11 * h.delta);
                    o[4] = (T)(h.d00 * h.dxdt);
                    o[5] = (T)h.d10;
                    o[6] = (T)(h.d01 * h.dxdt);
                    o[7] = (T)h.d11;
                    Ks[lane * levels + v] = k * spline.quad_pitch[v];
                }
            } else {
                const double v0 = a.pairs.vector[3 * p], v1 = a.pairs.vector[3 * p + 1], v2 = a.pairs.vector[3 * p + 2];
                double u0 = v0 / r, u1 = v1 / r, u2 = v2 / r;
                if (r < 1e-6) {
                    u0 = 0.0;
                    u1 = 0.0;
                    u2 = 1.0;
                }
                double fc, dfc;
                soap::cutoff_function(a.cut.smoothing, a.cut.rc, a.cut.width, r, &fc, &dfc);
                double sc = 1.0, dsc = 0.0;
                if (a.cut.scaling) soap::willatt2018(a.cut.scale, a.cut.rate, a.cut.exponent, r, &sc, &dsc);
                const T f = (T)(sc * fc);
                Fs[2 * lane] = f;
                Fs[2 * lane + 1] = (T)(dfc * sc + fc * dsc);
                const int i = a.pairs.first[p], j = a.pairs.second[p];
                T d[3];
#pragma unroll
                for (int x = 0; x < 3; x++) d[x] = tpos[3 * (int64_t)j + x] - tpos[3 * (int64_t)i + x];
                if (tcell) {
                    // system of the pair: the last system that starts at or before atom i
                    int64_t lo = 0, hi = a.n_systems - 1;
                    while (lo < hi) {
                        const int64_t mid = (lo + hi + 1) >> 1;
                        if (a.atom_offset[mid] <= i) lo = mid;
                        else hi = mid - 1;
                    }
                    const T* U = tcell + 9 * lo;
#pragma unroll
                    for (int x = 0; x < 3; x++)
                        d[x] += (T)a.pairs.shift[3 * p] * U[x] + (T)a.pairs.shift[3 * p + 1] * U[3 + x] +
                                (T)a.pairs.shift[3 * p + 2] * U[6 + x];
                }
                const T ud = (T)u0 * d[0] + (T)u1 * d[1] + (T)u2 * d[2], f_over_r = f / (T)r;
                T* Y = Ys + lane * 2 * lay.yp;
                T* Z = Y + lay.yp;
                const bool inv = code & 1;
                T along = ud, across = f_over_r;
                ylm_rows<T, CE_LMAX, true>(
                    a.tab.ylm_const, (T)u0, (T)u1, (T)u2,
                    [&](int l) {
                        const bool flip = inv && (l & 1);
                        along = flip ? -ud : ud;
                        across = flip ? -f_over_r : f_over_r;
                    },
                    [&](int l, int m, T yp, T ym, const T* gp, const T* gm) {
                        Y[l * l + l + m] = along * yp;
                        Z[l * l + l + m] = across * (gp[0] * d[0] + gp[1] * d[1] + gp[2] * d[2]);
                        if (m > 0) {
                            Y[l * l + l - m] = along * ym;
                            Z[l * l + l - m] = across * (gm[0] * d[0] + gm[1] * d[1] + gm[2] * d[2]);
                        }
                    });
            }
        }
        __syncthreads();
        // R_nl and f' R_nl + f dR_nl of every direction, a thread per (l, n)
        for (int w = threadIdx.x; w < (L + 1) * N; w += CE_THREADS) {
            const int l = w / N, n = w - l * N, level = spline.level_of[l];
            const T* quads = spline.quads + 4 * (spline.first_quad[l] + n);
            T* R = Rs + l * lay.nr + n;
#pragma unroll 4
            for (int q = 0; q < nd; q++) {
                T h[4], g[4], x[4];
                load_quad(Hs + (q * levels + level) * 8, h);
                load_quad(Hs + (q * levels + level) * 8 + 4, g);
                load_quad_global(quads + 4 * Ks[q * levels + level], x);
                const T value = h[0] * x[0] + h[1] * x[1] + h[2] * x[2] + h[3] * x[3];
                const T slope = g[0] * x[0] + g[1] * x[1] + g[2] * x[2] + g[3] * x[3];
                R[q * 2 * lay.rp] = value;
                R[(q * 2 + 1) * lay.rp] = Fs[2 * q + 1] * value + Fs[2 * q] * slope;
            }
        }
        __syncthreads();
        for (int q = 0; q < nd;) {
            while (end <= dc + q) next_species();
            const int qe = (int)min((int64_t)nd, end - dc);
            const T* R = Rs + q * 2 * lay.rp;
            const T* Y = Ys + q * 2 * lay.yp;
#pragma unroll 4
            for (; q < qe; q++) {
                sum_row(R, Y, 0);
                if (ROUNDS > 1 && L2 > CE_THREADS) sum_row(R, Y, ROUNDS - 1);
                R += 2 * lay.rp;
                Y += 2 * lay.yp;
            }
        }
    }
    while (t < S) next_species();
}

}  // namespace

// Few directions: one launch instead of three, whatever the basis (500 atoms with
// 38 directions 1.0 to 2.4 times as fast).  Many: the pair records' kernels have
// a thread for every (pair, l, m), and a row of few coefficients does not hide
// this kernel's chain of recursions and barriers.  `work` grows with the sums of
// a direction; 4000 to 8000 atoms with 38 directions, pair records / by centre:
//   FP32  lmax 1, nmax 4 (work 32) 85 / 116 us; 2, 4 (72) 0.9 times as fast;
//         1, 16 (80) 1.02 to 1.07 times; 3, 4 (128) 1.2 to 1.3
//   FP64  lmax 1, nmax 4 (32) 119 / 233 us; 3, 4 (128) 232 / 278; 2, 12 (144) 0.92;
//         2, 16 (180) 1.1 to 1.3; 3, 8 (192) 1.1; 4, 4 (200) 1.2
// With 11 directions a centre, a third of a chunk, FP64 turns at about 250 (lmax
// 4, nmax 4 0.87 to 0.94, nmax 8 1.27).  Layouts of more than 112 KB (FP64, lmax 8,
// nmax 15 and 16) leave one CTA of two warps per SM (0.9 to 0.97).
template <typename T>
bool dense_tangent_by_centre(const DenseTables<T>& tables, int64_t n_atoms, int64_t n_pairs) {
    if (!centre_expansion_supported(tables)) return false;
    constexpr bool F32 = sizeof(T) == 4;
    if (2 * n_pairs <= (F32 ? 40000 : 24000)) return true;
    const int L = tables.ylm_const.lmax, N = tables.spline.nmax, work = (L + 1) * (L + 1) * (N + 4);
    if (work < (F32 ? 76 : 2 * n_pairs < 16 * n_atoms ? 250 : 175)) return false;
    return TangentLayout<T>(L, N, tables.spline.levels).bytes <= 112 * 1024;
}

template bool dense_tangent_by_centre<float>(const DenseTables<float>&, int64_t, int64_t);
template bool dense_tangent_by_centre<double>(const DenseTables<double>&, int64_t, int64_t);

template <typename T>
void launch_dense_tangent_by_centre(const DenseArgs<T>& a, const T* tpos, const T* tcell, T* tcoef, cudaStream_t stream) {
    const TangentLayout<T> lay(a.lmax, a.nmax, a.tab.spline.levels);
    auto run = [&](auto kernel) {
        allow_shared_memory(kernel, lay.bytes);
        kernel<<<(unsigned)a.n_atoms, CE_THREADS, lay.bytes, stream>>>(a, tpos, tcell, tcoef);
    };
    if (a.nmax <= 8) run(centre_tangent_kernel<T, 8>);
    else run(centre_tangent_kernel<T, 16>);
    CUDA_CHECK(cudaGetLastError());
}

template void launch_dense_tangent_by_centre<float>(const DenseArgs<float>&, const float*, const float*, float*, cudaStream_t);
template void launch_dense_tangent_by_centre<double>(const DenseArgs<double>&, const double*, const double*, double*,
                                                     cudaStream_t);

}  // namespace fb200
