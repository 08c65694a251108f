// Values of the spherical expansion with one CTA per centre: the dense forms
// (FP32, FP64) and the drop-in without gradients.
//
//   c[centre][s][l m n] = sum over the directions d of (centre, s) in pair
//   order of (+-1)^l f(r_d) Y_lm(u_d) R_nl(r_d), plus the centre's own density
//   (featomic/src/calculators/soap/spherical_expansion.rs:101-358,
//   spherical_expansion_pair.rs:130-163)
//
// Two warps own all directions of the centre (sorted by neighbour species),
// 32 at a time: one warp evaluates the cutoff and Y_lm, a lane per direction
// with the Legendre rows in registers, the other the spline R_nl, into shared
// memory; then a thread per (l, m) sums all its radial functions over the
// directions and writes them out where the species changes.  Nothing per pair
// goes to memory.
//
// A (centre, species) segment holds 5 to 20 directions, so that a CTA per
// segment leaves most of its lanes idle, and records per pair are written
// once and read twice.  A direction's terms are evaluated for both atoms of a
// pair instead; channels with the same knots (all of them, or two groups) share
// the interval search and the Hermite weights (with seven of each per
// direction they were a quarter of the instructions and half of the time).
// Bound by the latency of its chain of loads and recursions: 20 000 atoms in FP32
// issue 1.9 of 4 instructions a cycle at 19 warps per SM (96 registers, shared
// memory), 4.2 of 9 stall cycles an instruction wait for a load.  FP32, lmax 6,
// nmax 8: 20 000 atoms with 52 directions 0.30 ms (pair records and an expansion
// kernel: 0.80 ms), 134 128 atoms of molecules 1.02 to 1.12 ms (2.88); FP64 values
// of 16 600 atoms of molecules 0.36 ms (1.71 with a CTA per segment).  Small bases
// of many atoms gain least: FP64, 8000 atoms, nmax 4, lmax 3 93 us (71 by pair
// records).
//
// The sums use the operations of pair_features_kernel / se_accumulate_kernel
// in their order; without FMA contraction the results are bit-identical.
#pragma once

#include "engine.hpp"
#include "pair_math.cuh"
#include "soap_math.cuh"

namespace fb200 {

// internal linkage: the kernel is compiled with FMA contraction for the dense
// forms and without it for the drop-in
namespace {

constexpr int CE_CHUNK = 32;
constexpr int CE_THREADS = 64;
constexpr int CE_LMAX = YlmConst<double>::LCAP;

template <typename T>
struct CentreArgs {
    int64_t n_centres;
    int n_species;
    const int32_t* centre_species;  // [n_centres]
    const int64_t* seg_offset;      // [n_centres * S + 1]
    const int32_t* dir_code;        // pair << 1 | reversed
    const double* distance;         // of the pairs
    const double* vector;
    DeviceSplineT<T> spline;
    YlmConst<T> ylm;
    CutoffParams cut;
    const T* self_contribution;
    T* coef;  // [n_centres][S][(lmax + 1)^2][nmax]
};

// The interval of a level's knots that holds r (the largest knot <= r, as
// soap::spline_interval finds it): from the interval at the start of r's bin
template <typename T>
__device__ __forceinline__ int level_interval(const DeviceSplineT<T>& S, int level, double r, double2& knot, double2& next) {
    int k = __ldg(S.lut + level * S.lut_bins + min(max((int)(r * S.lut_scale), 0), S.lut_bins - 1));
    const double2* knots = S.knots + S.first_knot[level];
    knot = __ldg(knots + k);
    next = __ldg(knots + k + 1);
    while (k > 0 && knot.x > r) {
        next = knot;
        knot = __ldg(knots + --k);
    }
    while (k < S.level_knots[level] - 2 && next.x <= r) {
        knot = next;
        k++;
        next = __ldg(knots + k + 1);
    }
    return k;
}

// Hermite weights of values and (scaled) derivatives at both ends.  FP64: the
// operations of soap::hermite_weights; FP32: a multiplication by 1 / width in
// place of the division, still in FP64.
template <typename T>
__device__ __forceinline__ void spline_weights(double2 knot, double2 next, double r, T (&o)[4]) {
    if constexpr (sizeof(T) == 8) {
        const soap::HermiteWeights h = soap::hermite_weights(knot.x, next.x, r);
        o[0] = h.h00;
        o[1] = h.h10 * h.delta;
        o[2] = h.h01;
        o[3] = h.h11 * h.delta;
    } else {
        const double delta = next.x - knot.x, t = (r - knot.x) * knot.y, t2 = t * t, t3 = t2 * t;
        const double h01 = 3.0 * t2 - 2.0 * t3, h11 = t3 - t2;
        o[0] = (T)(1.0 - h01);
        o[1] = (T)((h11 - t2 + t) * delta);
        o[2] = (T)h01;
        o[3] = (T)(h11 * delta);
    }
}

__device__ __forceinline__ void load_quad(const float* p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
}
__device__ __forceinline__ void load_quad(const double* p, double (&x)[4]) {
    const double2 u = *reinterpret_cast<const double2*>(p), v = *(reinterpret_cast<const double2*>(p) + 1);
    x[0] = u.x, x[1] = u.y, x[2] = v.x, x[3] = v.y;
}
__device__ __forceinline__ void store_quad(float* p, const float (&x)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ void store_quad(double* p, const double (&x)[4]) {
    reinterpret_cast<double2*>(p)[0] = make_double2(x[0], x[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(x[2], x[3]);
}
__device__ __forceinline__ void load_quad_global(const float* p, float (&x)[4]) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
}
__device__ __forceinline__ void load_quad_global(const double* p, double (&x)[4]) {
    const double2 u = __ldg(reinterpret_cast<const double2*>(p)), v = __ldg(reinterpret_cast<const double2*>(p) + 1);
    x[0] = u.x, x[1] = u.y, x[2] = v.x, x[3] = v.y;
}

// sum + a b, the product rounded by itself: the sums of the pair records'
// kernels, whose adjoints see the same coefficients to the last bit
__device__ __forceinline__ float add_product(float sum, float a, float b) { return __fadd_rn(sum, __fmul_rn(a, b)); }
__device__ __forceinline__ double add_product(double sum, double a, double b) { return sum + a * b; }

// Shared memory of a chunk: R rows of nr (whole 16-byte groups, the padding
// zero), the Hermite weights and spline rows, and Y rows of an odd pitch
// (written by a lane per direction)
template <typename T>
struct CentreLayout {
    int yp, nr, rp;
    size_t bytes;
    __host__ __device__ CentreLayout(int lmax, int nmax, int levels) {
        constexpr int W = 16 / (int)sizeof(T);
        yp = ((lmax + 1) * (lmax + 1)) | 1;
        nr = (nmax + W - 1) / W * W;
        rp = (lmax + 1) * nr;
        bytes = sizeof(T) * (size_t)CE_CHUNK * (rp + yp + 4 * levels) + sizeof(int) * (size_t)CE_CHUNK * levels;
    }
};

template <typename T, int NCAP>
__global__ void __launch_bounds__(CE_THREADS) centre_expansion_kernel(CentreArgs<T> a) {
    extern __shared__ __align__(16) unsigned char ce_smem[];
    constexpr int W = 16 / (int)sizeof(T);
    constexpr int ROUNDS = ((CE_LMAX + 1) * (CE_LMAX + 1) + CE_THREADS - 1) / CE_THREADS;
    using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    const int L = a.ylm.lmax, L2 = (L + 1) * (L + 1), N = a.spline.nmax, S = a.n_species;
    const int levels = a.spline.levels;
    const CentreLayout<T> lay(L, N, levels);
    T* Rs = reinterpret_cast<T*>(ce_smem);        // [chunk][rp]
    T* Hs = Rs + CE_CHUNK * lay.rp;               // [chunk][levels][4] Hermite weights
    T* Ys = Hs + CE_CHUNK * 4 * levels;           // [chunk][yp]
    int* Ks = reinterpret_cast<int*>(Ys + CE_CHUNK * lay.yp);  // [chunk][levels] rows of `quads`
    const int64_t c = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t d0 = a.seg_offset[c * S], d1 = a.seg_offset[(c + 1) * S];
    const int tc = a.centre_species[c];

    // this thread's (l, m) and, for lmax 8, a second one
    T acc[ROUNDS][NCAP];
    int row[ROUNDS];  // offset of the row's l in R
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
        const int lm = threadIdx.x + x * CE_THREADS;
        const T y = Y[min(lm, L2 - 1)];
#pragma unroll
        for (int n = 0; n < NCAP; n += W) {
            if (n < lay.nr) {
                const V v = *reinterpret_cast<const V*>(R + row[x] + n);
#pragma unroll
                for (int e = 0; e < W; e++) acc[x][n + e] = add_product(acc[x][n + e], y, reinterpret_cast<const T*>(&v)[e]);
            }
        }
    };
    int t = 0;
    int64_t end = a.seg_offset[c * S + 1];
    // the sums of species t into its coefficients, and the next species
    auto next_species = [&]() {
#pragma unroll
        for (int x = 0; x < ROUNDS; x++) {
            const int lm = threadIdx.x + x * CE_THREADS;
            if (lm < L2) {
                const bool self = t == tc && lm == 0;
                T* out = a.coef + ((c * S + t) * L2 + lm) * N;
                if (self) {
#pragma unroll
                    for (int n = 0; n < NCAP; n++)
                        if (n < N) acc[x][n] = a.self_contribution[n] + acc[x][n];
                }
                if (lay.nr == N) {
                    // 16-byte stores: a row is whole groups, and rows of
                    // neighbouring threads are adjacent (4-byte stores of the
                    // same rows kept the L2 busy for two thirds of the kernel)
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

    // the lane's direction of the next chunk, read one chunk ahead
    int code = 0;
    double r = 0.0, v0 = 0.0, v1 = 0.0, v2 = 0.0;
    auto fetch = [&](int64_t d) {
        if (d >= d1) return;
        code = a.dir_code[d];
        const int64_t p = code >> 1;
        r = a.distance[p];
        if (warp == 0) {
            v0 = a.vector[3 * p];
            v1 = a.vector[3 * p + 1];
            v2 = a.vector[3 * p + 2];
        }
    };
    fetch(d0 + lane);
    if (lay.nr != N)
        for (int w = threadIdx.x; w < CE_CHUNK * lay.rp; w += CE_THREADS) Rs[w] = T(0);
    for (int64_t dc = d0; dc < d1; dc += CE_CHUNK) {
        const int nd = (int)min((int64_t)CE_CHUNK, d1 - dc);
        __syncthreads();
        if (lane < nd) {
            if (warp == 1) {
                // the spline's interval and weights, once per level
                for (int v = 0; v < levels; v++) {
                    double2 knot, next;
                    const int k = level_interval(a.spline, v, r, knot, next);
                    T h[4];
                    spline_weights(knot, next, r, h);
                    store_quad(Hs + 4 * (lane * levels + v), h);
                    Ks[lane * levels + v] = k * a.spline.quad_pitch[v];
                }
            }
            if (warp == 0) {
                double u0, u1, u2;
                if constexpr (sizeof(T) == 4) {
                    const double rinv = 1.0 / r;
                    u0 = v0 * rinv;
                    u1 = v1 * rinv;
                    u2 = v2 * rinv;
                } else {
                    u0 = v0 / r;
                    u1 = v1 / r;
                    u2 = v2 / r;
                }
                if (r < 1e-6) {
                    // coincident atoms: spherical_expansion_pair.rs:337-339
                    u0 = 0.0;
                    u1 = 0.0;
                    u2 = 1.0;
                }
                double fc, dfc;
                soap::cutoff_function(a.cut.smoothing, a.cut.rc, a.cut.width, r, &fc, &dfc);
                double sc = 1.0, dsc = 0.0;
                if (a.cut.scaling) soap::willatt2018(a.cut.scale, a.cut.rate, a.cut.exponent, r, &sc, &dsc);
                const T f = (T)(sc * fc);
                T* Y = Ys + lane * lay.yp;
                // (-1)^l of a reversed pair, exact
                T fl = f;
                const bool inv = code & 1;
                ylm_rows<T, CE_LMAX, false>(
                    a.ylm, (T)u0, (T)u1, (T)u2, [&](int l) { fl = (inv && (l & 1)) ? -f : f; },
                    [&](int l, int m, T yp, T ym, const T*, const T*) {
                        Y[l * l + l + m] = fl * yp;
                        if (m > 0) Y[l * l + l - m] = fl * ym;
                    });
            }
        }
        __syncthreads();
        fetch(dc + CE_CHUNK + lane);
        // R_nl of every (direction, l, n): a thread per (l, n), whose loads of
        // one direction are contiguous (a lane that reads its own direction's
        // rows touches a line per access)
        for (int w = threadIdx.x; w < (L + 1) * N; w += CE_THREADS) {
            const int l = w / N, n = w - l * N, level = a.spline.level_of[l];
            const T* quads = a.spline.quads + 4 * (a.spline.first_quad[l] + n);
            T* R = Rs + l * lay.nr + n;
#pragma unroll 4
            for (int q = 0; q < nd; q++) {
                T h[4], x[4];
                load_quad(Hs + 4 * (q * levels + level), h);
                load_quad_global(quads + 4 * Ks[q * levels + level], x);
                R[q * lay.rp] = h[0] * x[0] + h[1] * x[1] + h[2] * x[2] + h[3] * x[3];
            }
        }
        __syncthreads();
        for (int q = 0; q < nd;) {
            while (end <= dc + q) next_species();  // segments that end here, empty ones among them
            const int qe = (int)min((int64_t)nd, end - dc);
            const T* R = Rs + q * lay.rp;
            const T* Y = Ys + q * lay.yp;
#pragma unroll 4
            for (; q < qe; q++) {
                sum_row(R, Y, 0);
                if (ROUNDS > 1 && L2 > CE_THREADS) sum_row(R, Y, ROUNDS - 1);
                R += lay.rp;
                Y += lay.yp;
            }
        }
    }
    while (t < S) next_species();
}

template <typename T>
void launch_centre_expansion(const CentreArgs<T>& a, cudaStream_t stream) {
    if (a.n_centres == 0) return;
    const CentreLayout<T> lay(a.ylm.lmax, a.spline.nmax, a.spline.levels);
    auto run = [&](auto kernel) {
        allow_shared_memory(kernel, lay.bytes);
        kernel<<<(unsigned)a.n_centres, CE_THREADS, lay.bytes, stream>>>(a);
    };
    if (a.spline.nmax <= 8) run(centre_expansion_kernel<T, 8>);
    else run(centre_expansion_kernel<T, 16>);
    CUDA_CHECK(cudaGetLastError());
}

}  // namespace

}  // namespace fb200
