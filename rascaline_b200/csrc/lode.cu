// LODE spherical expansion (featomic/src/calculators/lode/spherical_expansion.rs)
// on the GPU.  For every periodic system:
//
//   host    k-vectors of the cell inside the k_cutoff ball (one of each +-k
//           pair) and the density's Fourier transform f(k); the radial integral
//           R_nl(|k|) per k-vector where it is analytic
//   kernel  lode_projection_kernel: R_nl(|k|) from its spline, T[k][(l m n)] =
//           R_nl(|k|) Y_lm(k^), the even l first, then the odd l
//   kernel  lode_phases_kernel: cos(k.r_i), sin(k.r_i) for every atom and k
//   kernel  lode_type_sums_kernel: the same summed over the atoms of each type
//   kernel  lode_gemm_kernel: values (rows: centre i towards neighbour type t)
//           and positions gradients (rows: centre i, atom j, neighbour type
//           t, component x) as products [rows][k] x T[k][(l m n)] on the FP64
//           tensor cores, with the structure factor S_i^t(k) or the pair
//           factor of (i, j), times 4 pi / V f(k), made on the way into
//           shared memory
//
// The sums over k run by fours (a tensor-core step) inside each split of the
// k-vectors, then over the splits: not featomic's order, and the same from call
// to call.  The sign (-1)^{l/2}, (-1)^{(l+1)/2} is applied at the end, which is
// exact, then the central-atom and k = 0 terms in featomic's order.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <map>
#include <set>

#include "lode.hpp"
#include "pair_math.cuh"
#include "soap_math.cuh"

namespace fb200 {

// ---------------------------------------------------------------------------
// host math
// ---------------------------------------------------------------------------
namespace {
constexpr double EULER_GAMMA = 0.5772156649015329;
}

// E1(x) = int_x^inf e^-t / t dt: power series -gamma - ln x - sum (-x)^k /
// (k k!) for x <= 1 (Abramowitz & Stegun 5.1.11), continued fraction
// e^-x / (x + 1 - 1 / (x + 3 - 4 / (x + 5 - ...))) evaluated by the modified
// Lentz method beyond (A&S 5.1.22)
double exp1(double x) {
    if (x == 0.0) return INFINITY;
    if (!(x > 0.0)) return NAN;
    if (x <= 1.0) {
        double term = 1.0, sum = 0.0;
        for (int k = 1; k < 200; k++) {
            term *= -x / (double)k;
            const double add = term / (double)k;
            sum += add;
            if (std::fabs(add) <= 1e-17 * std::fabs(sum)) break;
        }
        return -EULER_GAMMA - std::log(x) - sum;
    }
    const double tiny = 1e-300;
    double b = x + 1.0, c = 1.0 / tiny, d = 1.0 / b, h = d;
    for (int i = 1; i < 10000; i++) {
        const double a = -(double)i * (double)i;
        b += 2.0;
        d = 1.0 / (a * d + b);
        c = b + a / c;
        const double del = c * d;
        h *= del;
        if (std::fabs(del - 1.0) < 1e-16) break;
    }
    return h * std::exp(-x);
}

// Ei(x) = -E1(-x) for x < 0; power series gamma + ln x + sum x^k / (k k!)
// for 0 < x <= 40, asymptotic e^x / x sum k! / x^k beyond
double expi(double x) {
    if (x == 0.0) return -INFINITY;
    if (x < 0.0) return -exp1(-x);
    if (x <= 40.0) {
        double term = 1.0, sum = 0.0;
        for (int k = 1; k < 500; k++) {
            term *= x / (double)k;
            const double add = term / (double)k;
            sum += add;
            if (std::fabs(add) <= 1e-17 * std::fabs(sum)) break;
        }
        return EULER_GAMMA + std::log(x) + sum;
    }
    double term = 1.0, sum = 1.0;
    for (int k = 1; k <= 20; k++) {
        term *= (double)k / x;
        sum += term;
    }
    return std::exp(x) / x * sum;
}

// 2F1(1, b; c; z) = sum_k (b)_k / (c)_k z^k, every term positive for
// b, c > 0 and 0 <= z < 1
double hyp2f1_one(double b, double c, double z) {
    double term = 1.0, sum = 1.0;
    for (int k = 0; k < 2000000; k++) {
        term *= (b + (double)k) / (c + (double)k) * z;
        sum += term;
        if (term <= 1e-17 * sum) break;
    }
    return sum;
}

// math/k_vectors.rs:19-87: the reciprocal cell 2 pi (H^T)^-1, lattice points
// (n1, n2, n3) in featomic's order with |k| < k_cutoff, n1 > 0, or n1 = 0 and
// n2 > 0, or n1 = n2 = 0 and n3 > 0
KVectors compute_k_vectors(const double cell[9], double k_cutoff) {
    // inverse of the transposed cell (rows of `cell` are the cell vectors)
    const double* H = cell;
    double T[9] = {H[0], H[3], H[6], H[1], H[4], H[7], H[2], H[5], H[8]};
    const double det = T[0] * (T[4] * T[8] - T[5] * T[7]) - T[1] * (T[3] * T[8] - T[5] * T[6]) +
                       T[2] * (T[3] * T[7] - T[4] * T[6]);
    if (det == 0.0) throw invalid_parameter("LODE can only be used with periodic systems");
    double inv[9] = {(T[4] * T[8] - T[5] * T[7]) / det, (T[2] * T[7] - T[1] * T[8]) / det,
                     (T[1] * T[5] - T[2] * T[4]) / det, (T[5] * T[6] - T[3] * T[8]) / det,
                     (T[0] * T[8] - T[2] * T[6]) / det, (T[2] * T[3] - T[0] * T[5]) / det,
                     (T[3] * T[7] - T[4] * T[6]) / det, (T[1] * T[6] - T[0] * T[7]) / det,
                     (T[0] * T[4] - T[1] * T[3]) / det};
    double R[9];
    for (int k = 0; k < 9; k++) R[k] = 2.0 * M_PI * inv[k];
    const double* b1 = R;
    const double* b2 = R + 3;
    const double* b3 = R + 6;
    auto dot = [](const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; };
    const double m00 = dot(b1, b1), m11 = dot(b2, b2), m22 = dot(b3, b3);
    const double m01 = dot(b1, b2), m02 = dot(b1, b3), m12 = dot(b2, b3);
    const double volume = R[0] * (R[4] * R[8] - R[5] * R[7]) - R[1] * (R[3] * R[8] - R[5] * R[6]) +
                          R[2] * (R[3] * R[7] - R[4] * R[6]);
    const long n1_max = (long)(std::sqrt(m11 * m22 - m12 * m12) / volume * k_cutoff);
    const long n2_max = (long)(std::sqrt(m22 * m00 - m02 * m02) / volume * k_cutoff);
    const long n3_max = (long)(std::sqrt(m00 * m11 - m01 * m01) / volume * k_cutoff);
    const double cutoff2 = k_cutoff * k_cutoff;
    KVectors out;
    auto add = [&](long n1, long n2, long n3) {
        double k[3];
        for (int x = 0; x < 3; x++) k[x] = (double)n1 * b1[x] + (double)n2 * b2[x] + (double)n3 * b3[x];
        const double n2k = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
        if (n2k < cutoff2) {
            const double norm = std::sqrt(n2k);
            out.norm.push_back(norm);
            for (int x = 0; x < 3; x++) out.direction.push_back(k[x] / norm);
        }
    };
    for (long n3 = 1; n3 <= n3_max; n3++) add(0, 0, n3);
    for (long n2 = 1; n2 <= n2_max; n2++)
        for (long n3 = -n3_max; n3 <= n3_max; n3++) add(0, n2, n3);
    for (long n1 = 1; n1 <= n1_max; n1++)
        for (long n2 = -n2_max; n2 <= n2_max; n2++)
            for (long n3 = -n3_max; n3 <= n3_max; n3++) add(n1, n2, n3);
    return out;
}

namespace {

// lode/radial_integral/gto.rs:62-131 before the orthonormalisation:
// sqrt(pi / 2) sigma_n^{n+3} sqrt2^n (k sigma_n / sqrt2)^l G(a, b, -k^2 sigma_n^2 / 2)
// with G = Gamma(a) / Gamma(b) 1F1(a, b, z), a = (n + l + 3) / 2, b = l + 3/2,
// and its derivative in k
void lode_radial_raw(const LodeTables& t, int l, double k, double* values, double* grads) {
    const double global = std::sqrt(M_PI) / M_SQRT2;
    const int N = t.h.nmax();
    for (int n = 0; n < N; n++) {
        const double sigma = t.widths[n];
        const double ksig = k * sigma / M_SQRT2;
        const double factor = global * soap::powi(sigma, n + 3) * soap::powi(M_SQRT2, n) * soap::powi(ksig, l);
        const double kns2 = -k * sigma * sigma;
        const double z = 0.5 * k * kns2;
        const double a = 0.5 * (double)(n + l + 3), b = (double)l + 1.5;
        const double ratio = soap::gamma_fn(a) / soap::gamma_fn(b);
        values[n] = ratio * soap::hyp1f1(a, b, z);
        if (grads) grads[n] = ratio * (a / b * soap::hyp1f1(a + 1.0, b + 1.0, z));
        values[n] *= factor;
        if (grads) {
            grads[n] *= kns2 * factor;
            grads[n] += (double)l / k * values[n];
        }
    }
    // at k = 0 the expression above is 0 / 0 for the gradients: zero except
    // for l = 1 (gto.rs:107-124)
    if (k == 0.0 && grads) {
        for (int n = 0; n < N; n++) grads[n] = 0.0;
        if (l == 1) {
            for (int n = 0; n < N; n++) {
                const double sigma = t.widths[n];
                const double a = 0.5 * (double)(n + l) + 1.5, b = 2.5;
                const double factor = global * soap::powi(sigma, n + l + 3) * soap::powi(M_SQRT2, n - l);
                grads[n] = soap::gamma_fn(a) / soap::gamma_fn(b) * factor;
            }
        }
    }
}

void orthonormalize(const LodeTables& t, double* v) {
    const int N = t.h.nmax();
    double tmp[64];
    for (int k = 0; k < N; k++) {
        double s = 0.0;
        for (int n = 0; n < N; n++) s += v[n] * t.ortho[(size_t)k * N + n];
        tmp[k] = s;
    }
    for (int k = 0; k < N; k++) v[k] = tmp[k];
}

}  // namespace

void LodeTables::radial(int l, double k, double* v, double* g) const {
    const int N = h.nmax();
    if (!positions.empty()) {
        const double* pos = positions.data() + knot_offset[l];
        const int count = knot_count[l];
        const int kk = soap::spline_interval(pos, count, k);
        const soap::HermiteWeights w = soap::hermite_weights(pos[kk], pos[kk + 1], k);
        const double* pv = values.data() + ((size_t)knot_offset[l] + kk) * N;
        const double* pd = derivs.data() + ((size_t)knot_offset[l] + kk) * N;
        for (int n = 0; n < N; n++) {
            v[n] = soap::hermite_value(w, pv[n], pd[n], pv[N + n], pd[N + n]);
            if (g) g[n] = soap::hermite_derivative(w, pv[n], pd[n], pv[N + n], pd[N + n]);
        }
        return;
    }
    lode_radial_raw(*this, l, k, v, g);
    orthonormalize(*this, v);
    if (g) orthonormalize(*this, g);
}

// lode/spherical_expansion.rs:276-335
double LodeTables::density_fourier(double k) const {
    const int p = h.exponent;
    const double s2 = h.smearing * h.smearing;
    if (p == 0) return std::pow(4.0 * M_PI * s2, 0.75) * std::exp(-0.5 * k * k * s2);
    if (p == 1) {
        const double k2 = k * k;
        return 4.0 * M_PI * (std::exp(-0.5 * k2 * s2) / k2);
    }
    const double p_eff = 3.0 - (double)p;
    const double factor = std::pow(M_PI, 1.5) * std::pow(2.0 * s2, 0.5 * p_eff) / soap::gamma_fn(0.5 * (double)p);
    const double x = 0.5 * (k * k) * s2;
    const double sqrt_pi = std::sqrt(M_PI);
    double value = 0.0;
    switch (p) {
    case 2: value = std::sqrt(M_PI / x) * std::erfc(std::sqrt(x)); break;
    case 3: value = -expi(-x); break;
    case 4: value = 2.0 * (std::exp(-x) - std::sqrt(M_PI * x) * std::erfc(std::sqrt(x))); break;
    case 5: value = std::exp(-x) + x * expi(-x); break;
    case 6:
        value = ((2.0 - 4.0 * x) * std::exp(-x) + 4.0 * sqrt_pi * std::pow(x, 1.5) * std::erfc(std::sqrt(x))) / 3.0;
        break;
    case 7: value = (1.0 - x) * std::exp(-x) / 2.0 - x * x / 2.0 * expi(-x); break;
    case 8:
        value = -2.0 / 15.0 * ((-3.0 + 2.0 * x - 4.0 * x * x) * std::exp(-x) +
                               4.0 * sqrt_pi * std::pow(x, 2.5) * std::erfc(std::sqrt(x)));
        break;
    case 9: value = (x * x - x + 2.0) * std::exp(-x) / 6.0 + x * x * x / 6.0 * expi(-x); break;
    default: throw invalid_parameter("potential_exponent = " + std::to_string(p) + " is not implemented");
    }
    return factor * value;
}

LodeTables build_lode_tables(const LodeHypers& h) {
    LodeTables t;
    t.h = h;
    const int N = h.nmax();
    t.widths = gto_basis_widths(N, h.radius);
    t.ortho = gto_basis_orthonormalization(N, h.radius);
    if (h.splined) {
        // one spline per angular channel over [0, k_cutoff] (radial_integral/
        // spline.rs:28-68, featomic/src/math/splines.rs:79-193)
        std::vector<double> pos, val, der;
        for (int l = 0; l <= h.max_angular; l++) {
            build_spline_knots([&](double k, double* v, double* g) {
                lode_radial_raw(t, l, k, v, g);
                orthonormalize(t, v);
                orthonormalize(t, g);
            }, h.k_cutoff, N, N, h.spline_accuracy, pos, val, der);
            t.knot_offset.push_back((int32_t)t.positions.size());
            t.knot_count.push_back((int32_t)pos.size());
            t.positions.insert(t.positions.end(), pos.begin(), pos.end());
            t.values.insert(t.values.end(), val.begin(), val.end());
            t.derivs.insert(t.derivs.end(), der.begin(), der.end());
        }
    }
    // central-atom contribution <n 0 0> (gto.rs:133-181), from the analytic
    // expressions whether or not the integral is splined
    std::vector<double> c(N);
    const double s = h.smearing, p = (double)h.exponent;
    for (int n = 0; n < N; n++) {
        const double n_eff = 0.5 * (3.0 + (double)n);
        if (h.exponent == 0) {
            const double factor = std::pow(M_PI, -0.25) / std::pow(s * s, 0.75);
            const double alpha = 0.5 * (1.0 / (s * s) + 1.0 / (t.widths[n] * t.widths[n]));
            c[n] = factor * soap::gamma_fn(n_eff) / std::pow(alpha, n_eff);
        } else {
            const double factor = 2.0 * std::sqrt(4.0 * M_PI) / soap::gamma_fn(p / 2.0) / p;
            const double q = s / t.widths[n];
            const double hyparg = 1.0 / (1.0 + q * q);
            c[n] = factor * std::pow(2.0, (1.0 + (double)n - p) / 2.0) * soap::powi(s, 3 + n - h.exponent) *
                   soap::gamma_fn(n_eff) * hyp2f1_one(n_eff, (p + 2.0) / 2.0, hyparg) * std::pow(hyparg, n_eff);
        }
    }
    orthonormalize(t, c.data());
    t.center = c;
    // k = 0 term (spherical_expansion.rs:337-376): factor times R_n0(0)
    double factor = 0.0;
    if (h.exponent == 0) {
        const double s2 = s * s;
        factor = std::pow(2.0 * M_PI * s2, 1.5) / std::pow(M_PI * s2, 0.75) / std::sqrt(4.0 * M_PI);
    } else if (h.exponent > 3) {
        const double p_eff = 3.0 - p;
        factor = 0.5 * M_PI * std::pow(2.0, p_eff) / soap::gamma_fn(0.5 * p) * std::pow(2.0, (p - 1.0) / 2.0) / -p_eff *
                 std::pow(s, -p_eff) / std::pow(s, 2.0 * p - 6.0);
    }
    std::vector<double> r0(N);
    t.radial(0, 0.0, r0.data(), nullptr);
    t.k0.resize(N);
    for (int n = 0; n < N; n++) t.k0[n] = factor * r0[n];
    return t;
}

}  // namespace fb200

namespace fb200 {

namespace {

constexpr int LODE_KB = 16;       // k-vectors per step of the product, and the padding of their number
constexpr int LODE_ROWS = 64;     // rows of one tile of the product
constexpr int LODE_THREADS = 128;
constexpr int LODE_LDA = LODE_KB + 4;  // pitch = 4 (mod 16) doubles: fragment loads hit every bank once

// Columns of T and of the product: the even l, then (from `odd0`) the odd l,
// each in (l, m, n) order and padded to 16 bytes
struct LodeColumns {
    int n_even, n_odd, odd0, ld;
};

LodeColumns lode_columns(int L, int N) {
    LodeColumns c{};
    for (int l = 0; l <= L; l++) (l & 1 ? c.n_odd : c.n_even) += (2 * l + 1) * N;
    c.odd0 = (c.n_even + 1) & ~1;
    c.ld = c.odd0 + ((c.n_odd + 1) & ~1);
    return c;
}

// (l, m) rows of one parity before channel l: sum of 2 l' + 1 over l' = l - 2, l - 4, ...
__host__ __device__ inline int lode_lm_before(int l) { return l * (l - 1) / 2; }

__device__ inline double lode_phase(int l) {
    // spherical_expansion.rs:667-671
    return (l % 2 == 0) ? ((l / 2) % 2 == 0 ? 1.0 : -1.0) : (((l + 1) / 2) % 2 == 0 ? 1.0 : -1.0);
}

// T[k][column] = R_nl(|k|) Y_lm(k^) (spherical_expansion.rs:226-274) for `kc`
// k-vectors per CTA, zero for the padding of their number: a thread per (k, m)
// for the Legendre columns and harmonics, a thread per (k, l) for the spline
// of the radial integral (`radial` holds it when there is no spline), then
// every thread writes columns.  One thread per k-vector, as it was, left the
// chip to 36 CTAs and the radial integrals to the host: 65 us for 4522
// k-vectors, and 14 us now, with 2 MB less to copy up.
__global__ void __launch_bounds__(128) lode_projection_kernel(int K, int Kp, int kc, int N, LodeColumns cols,
                                                              const double* __restrict__ dir,
                                                              const double* __restrict__ norm,
                                                              const double* __restrict__ radial, DeviceRadial spline,
                                                              DeviceYlm ylm, double* __restrict__ T) {
    extern __shared__ double proj_smem[];
    const int L = ylm.lmax, L1 = L + 1, L2 = L1 * L1, NP = L1 * (L + 2) / 2;
    double* P = proj_smem;               // [kc][NP]
    double* Y = P + kc * NP;             // [kc][L2]
    double* R = Y + kc * L2;             // [kc][L1][N]
    const int k0 = blockIdx.x * kc;
    for (int w = threadIdx.x; w < 2 * kc * L1; w += blockDim.x) {
        const bool column = w < kc * L1;
        const int v = column ? w : w - kc * L1;
        const int q = v / L1, j = v - q * L1, k = k0 + q;
        if (k >= K) continue;
        if (column) {
            ylm_legendre_column(ylm, ylm_angles(dir[3 * k], dir[3 * k + 1], dir[3 * k + 2]), j, P + q * NP);
        } else if (radial == nullptr) {
            radial_spline_compute(spline, j, norm[k], R + (q * L1 + j) * N, nullptr);
        } else {
            for (int n = 0; n < N; n++) R[(q * L1 + j) * N + n] = radial[((size_t)k * L1 + j) * N + n];
        }
    }
    __syncthreads();
    for (int w = threadIdx.x; w < kc * L1; w += blockDim.x) {
        const int q = w / L1, m = w - q * L1, k = k0 + q;
        if (k >= K) continue;
        ylm_column_outputs(ylm, ylm_angles(dir[3 * k], dir[3 * k + 1], dir[3 * k + 2]), m, P + q * NP, Y + q * L2,
                           (double*)nullptr, (double*)nullptr, (double*)nullptr);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < cols.ld; c += blockDim.x) {
        const bool odd = c >= cols.odd0;
        const int pos = odd ? c - cols.odd0 : c;
        const bool pad = pos >= (odd ? cols.n_odd : cols.n_even);
        const int row = pos / N, n = pos - row * N;
        int l = odd ? 1 : 0;
        while (lode_lm_before(l + 2) <= row) l += 2;
        const int lm = l * l + row - lode_lm_before(l);
        for (int q = 0; q < kc; q++) {
            const int k = k0 + q;
            if (k >= Kp) break;
            T[(size_t)k * cols.ld + c] = (pad || k >= K) ? 0.0 : R[(q * L1 + l) * N + n] * Y[q * L2 + lm];
        }
    }
}

// cos and sin of k.r for every (atom, k) (spherical_expansion.rs:92-111),
// k.r = (|k| k^) . r in featomic's order; zero for the padding of k
__global__ void lode_phases_kernel(int n_atoms, int K, int Kp, const double* __restrict__ positions,
                                   const double* __restrict__ kvec, double* __restrict__ C, double* __restrict__ S) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n_atoms * Kp) return;
    const int i = (int)(idx / Kp), k = (int)(idx - (int64_t)i * Kp);
    double sn = 0.0, cs = 0.0;
    if (k < K) {
        const double* p = positions + 3 * i;
        const double* q = kvec + 3 * k;
        sincos(q[0] * p[0] + q[1] * p[1] + q[2] * p[2], &sn, &cs);
    }
    C[idx] = cs;
    S[idx] = sn;
}

// 4 pi / V f(k) times the sums of cos(k.r_j), sin(k.r_j) over the atoms j of
// each type (spherical_expansion.rs:125-141), from the atoms sorted by type:
// CTA (32 k-vectors, type) with eight atoms in flight per k-vector, added in
// a fixed order.  (A thread per (type, k) that walked over every atom took
// 134 us for 1000 atoms and 4522 k-vectors, this takes 13 us.)
__global__ void __launch_bounds__(256) lode_type_sums_kernel(int K, int Kp, const int32_t* __restrict__ sorted_atoms,
                                                             const int32_t* __restrict__ type_start,
                                                             const double* __restrict__ gdf,
                                                             const double* __restrict__ C, const double* __restrict__ S,
                                                             double* __restrict__ Ct, double* __restrict__ St) {
    __shared__ double part[2][8][32];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, t = blockIdx.y;
    const int k = blockIdx.x * 32 + x;
    double sc = 0.0, ss = 0.0;
    if (k < K) {
        for (int q = type_start[t] + y; q < type_start[t + 1]; q += 8) {
            const size_t at = (size_t)sorted_atoms[q] * Kp + k;
            sc += C[at];
            ss += S[at];
        }
    }
    part[0][y][x] = sc;
    part[1][y][x] = ss;
    __syncthreads();
    if (y >= 2 || k >= Kp) return;
    double sum = 0.0;
    for (int q = 0; q < 8; q++) sum += part[y][q][x];
    (y == 0 ? Ct : St)[(size_t)t * Kp + k] = k < K ? gdf[k] * sum : 0.0;
}

struct LodeArgs {
    int Kp, S, L, N;            // Kp: k-vectors padded to LODE_KB
    LodeColumns cols;
    const int32_t* species;     // [n_atoms] species index of the system's atoms
    const double *C, *Sn;       // [n_atoms][Kp]
    const double *Ct, *St;      // [S][Kp] sums over the atoms of a type, times 4 pi / V f(k)
    const double* gdf;          // [Kp] 4 pi / V f(k), zero in the padding
    const double* T;            // [Kp][ld]
    const double* kvec;         // [Kp][3] |k| k^
    // values: rows are the atoms, for each type in `present`
    const int32_t* present;     // [n_present] types of the system
    const int32_t* row;         // [n_atoms][S] sample row of atom i in the blocks (type_i, t)
    const int64_t* off_values;  // [S][S][L + 1] offset of each block's values
    const int32_t* type_count;  // [S] atoms of each type in the system
    const double* center;       // [N] central-atom contribution
    const double* k0;           // [N] 4 pi / V times the k = 0 term
    double center_factor;       // 1 - center_atom_weight
    int add_k0;
    // gradients: rows are 3 task + x
    const int32_t* tasks;       // [n_tasks][4] (i, j, t, row)
    const int64_t* off_positions;
    double* out;
    // the product's tiling
    int64_t rows;               // rows of one type (values), or 3 tasks
    int tiles, tiles_even;      // column tiles, and those of the even l
    int splits, split_k;        // k-vectors [s split_k, (s + 1) split_k) in split s
    double* partial;            // [splits][types][rows][ld] when splits > 1
};

// one finished value into its block
template <bool GRAD>
__device__ __forceinline__ void lode_store(const LodeArgs& a, int64_t r, int type, int column, double sum) {
    const bool odd = column >= a.cols.odd0;
    const int pos = odd ? column - a.cols.odd0 : column;
    const int lm = pos / a.N, n = pos - lm * a.N;
    int l = odd ? 1 : 0;
    while (lode_lm_before(l + 2) <= lm) l += 2;
    const int mi = lm - lode_lm_before(l), M = 2 * l + 1;
    const double x = lode_phase(l) * sum;
    if (GRAD) {
        const int64_t task = r / 3;
        const int c = (int)(r - 3 * task);
        const int32_t* w = a.tasks + 4 * task;
        const int64_t off = a.off_positions[((size_t)a.species[w[0]] * a.S + w[2]) * (a.L + 1) + l];
        a.out[off + (((int64_t)w[3] * 3 + c) * M + mi) * a.N + n] = x;
        return;
    }
    const int t = a.present[type], ti = a.species[r];
    double v = 0.0;
    if (l == 0) {
        // central atom (:378-426), then the k = 0 term once per atom of type
        // t (:635-661)
        if (t == ti) v -= a.center_factor * a.center[n];
        if (a.add_k0)
            for (int j = 0; j < a.type_count[t]; j++) v += a.k0[n];
    }
    const int64_t off = a.off_values[((size_t)ti * a.S + t) * (a.L + 1) + l];
    a.out[off + ((int64_t)a.row[r * a.S + t] * M + mi) * a.N + n] = v + x;
}

__device__ __forceinline__ void lode_dmma(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

__device__ __forceinline__ void lode_cp16(void* dst, const void* src, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// Values (spherical_expansion.rs:616-723) and positions gradients (:725-873)
// as products with T.  A CTA of four warps owns 64 rows x 8 NB columns of one
// parity of l; a warp computes 16 rows of it.  Per LODE_KB k-vectors the 64
// rows of the left operand are built from cos and sin (loaded one step ahead
// into registers) and stored to shared memory, T's rows arrive by cp.async in
// two buffers.  Bound by the FP64 tensor pipe (2 x rows x k x columns flops;
// about 36 TFLOP/s; the longest stall is the pipe's throttle, 3.7 of 13 cycles an
// instruction); 64 rows keep the reads of T and of cos / sin, both from
// L2, below it, and 128 registers (four CTAs per SM) hide the two barriers of
// a step.  Values of 1000 atoms, 3 types, 4522 k-vectors and 392 coefficients
// (10.6 GFLOP): 0.51 ms = 20.7 TFLOP/s; 0.68 ms with three CTAs per SM and
// three splits; 2.33 ms as a sum over k on the CUDA cores, eight centres and
// four coefficients a thread.
template <int NB, bool GRAD>
__global__ void __launch_bounds__(LODE_THREADS, GRAD ? 3 : 4) lode_gemm_kernel(LodeArgs a) {
    constexpr int BN = 8 * NB;
    constexpr int LDB = ((BN + 11) / 16) * 16 + 4;  // >= BN, 4 (mod 16) doubles
    __shared__ __align__(16) double As[LODE_ROWS * LODE_LDA];
    __shared__ __align__(16) double Bs[2][LODE_KB * LDB];
    __shared__ __align__(16) double Ks[2][3][LODE_KB];  // values: Ct, St; gradients: gdf, k-vectors apart
    const int64_t row_tile = blockIdx.x / a.tiles;
    const int tile = (int)(blockIdx.x - row_tile * a.tiles);
    const int type = blockIdx.y, split = blockIdx.z;
    const bool odd = tile >= a.tiles_even;
    const int col0 = odd ? a.cols.odd0 + (tile - a.tiles_even) * BN : tile * BN;
    const int n_cols = min(BN, (odd ? a.cols.odd0 + a.cols.n_odd : a.cols.n_even) - col0);
    const int64_t row0 = row_tile * LODE_ROWS;
    const int kb = split * a.split_k, ke = min(a.Kp, kb + a.split_k);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // this thread's part of the left operand: one row, eight k-vectors
    const int ar = threadIdx.x >> 1, ak = (threadIdx.x & 1) * 8;
    const int64_t r = row0 + ar;
    const bool row_ok = r < a.rows;
    int i = 0, j = 0, t = 0, x = 0;
    bool same_type = false;
    if (GRAD) {
        const int64_t task = row_ok ? r / 3 : 0;
        x = row_ok ? (int)(r - 3 * task) : 0;
        i = a.tasks[4 * task];
        j = a.tasks[4 * task + 1];
        t = a.tasks[4 * task + 2];
        same_type = a.species[i] == t;
    } else {
        i = row_ok ? (int)r : 0;
        t = a.present[type];
    }
    const double* ci = a.C + (size_t)i * a.Kp + ak;
    const double* si = a.Sn + (size_t)i * a.Kp + ak;
    const double* cj = a.C + (size_t)j * a.Kp + ak;
    const double* sj = a.Sn + (size_t)j * a.Kp + ak;
    double c8[8], s8[8];
    auto load8 = [&](const double* src, double(&v)[8]) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double2 w = __ldg(reinterpret_cast<const double2*>(src) + q);
            v[2 * q] = w.x;
            v[2 * q + 1] = w.y;
        }
    };
    auto issue = [&](int k, int buf) {
        for (int q = threadIdx.x; q < LODE_KB * (BN / 2); q += LODE_THREADS) {
            const int kk = q / (BN / 2), c = 2 * (q - kk * (BN / 2));
            // columns past the parity's end: zeros, nothing read
            const bool ok = c < n_cols;
            lode_cp16(&Bs[buf][kk * LDB + c], a.T + (size_t)(k + kk) * a.cols.ld + (ok ? col0 + c : 0), ok);
        }
        if (!GRAD && threadIdx.x < LODE_KB) {
            const int half = threadIdx.x / (LODE_KB / 2), q = 2 * (threadIdx.x % (LODE_KB / 2));
            lode_cp16(&Ks[buf][half][q], (half ? a.St : a.Ct) + (size_t)t * a.Kp + k + q, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[2][NB][2];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < NB; n++) acc[m][n][0] = acc[m][n][1] = 0.0;

    if (kb < ke) {
        issue(kb, 0);
        load8(ci + kb, c8);
        load8(si + kb, s8);
    }
    int buf = 0;
    for (int k = kb; k < ke; k += LODE_KB, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // T's rows are there, and the last step's operands are done with
        double w[8];
        if (GRAD) {
            double cj8[8], sj8[8];
            load8(cj + k, cj8);
            load8(sj + k, sj8);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int kk = k + ak + q;
                // real / imaginary part of i e^{i k (r_i - r_j)}
                const double pair = a.gdf[kk] * (odd ? -2.0 * (c8[q] * cj8[q] + s8[q] * sj8[q])
                                                     : 2.0 * (s8[q] * cj8[q] - c8[q] * sj8[q]));
                double f = pair;
                if (i == j) {
                    // -sum_{j != i}: from the structure factor per centre
                    const double ct = a.Ct[(size_t)t * a.Kp + kk], st = a.St[(size_t)t * a.Kp + kk];
                    const double sum = odd ? 2.0 * (c8[q] * ct + s8[q] * st) : -2.0 * (s8[q] * ct - c8[q] * st);
                    f = same_type ? sum + pair : sum;
                }
                w[q] = row_ok ? f * a.kvec[3 * kk + x] : 0.0;
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++) {
                // structure factor per centre (:143-155), real or imaginary part
                const double ct = Ks[buf][0][ak + q], st = Ks[buf][1][ak + q];
                w[q] = row_ok ? 2.0 * (odd ? s8[q] * ct - c8[q] * st : c8[q] * ct + s8[q] * st) : 0.0;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            *reinterpret_cast<double2*>(&As[ar * LODE_LDA + ak + 2 * q]) = make_double2(w[2 * q], w[2 * q + 1]);
        if (k + LODE_KB < ke) {
            issue(k + LODE_KB, buf ^ 1);
            load8(ci + k + LODE_KB, c8);
            load8(si + k + LODE_KB, s8);
        }
        __syncthreads();
        const double* A0 = As + (16 * warp + (lane >> 2)) * LODE_LDA + (lane & 3);
        const double* B0 = Bs[buf] + (lane & 3) * LDB + (lane >> 2);
#pragma unroll
        for (int st = 0; st < LODE_KB / 4; st++) {
            const double a0 = A0[4 * st], a1 = A0[8 * LODE_LDA + 4 * st];
#pragma unroll
            for (int n = 0; n < NB; n++) {
                const double b = B0[4 * st * LDB + 8 * n];
                lode_dmma(acc[0][n], a0, b);
                lode_dmma(acc[1][n], a1, b);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 2; m++) {
        const int64_t ro = row0 + 16 * warp + 8 * m + (lane >> 2);
        if (ro >= a.rows) continue;
#pragma unroll
        for (int n = 0; n < NB; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int c = 8 * n + 2 * (lane & 3) + e;
                if (c >= n_cols) continue;
                if (a.splits > 1)
                    a.partial[(((int64_t)split * gridDim.y + type) * a.rows + ro) * a.cols.ld + col0 + c] = acc[m][n][e];
                else
                    lode_store<GRAD>(a, ro, type, col0 + c, acc[m][n][e]);
            }
    }
}

// the splits' sums added in order, thread per (row, column)
template <bool GRAD>
__global__ void __launch_bounds__(256) lode_splits_kernel(LodeArgs a, int n_types) {
    const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t per_split = (int64_t)n_types * a.rows * a.cols.ld;
    if (item >= per_split) return;
    const int64_t tr = item / a.cols.ld;
    const int column = (int)(item - tr * a.cols.ld);
    if (column >= a.cols.n_even && column < a.cols.odd0) return;
    if (column >= a.cols.odd0 + a.cols.n_odd) return;
    double sum = 0.0;
    for (int s = 0; s < a.splits; s++) sum += a.partial[s * per_split + item];
    const int type = (int)(tr / a.rows);
    lode_store<GRAD>(a, tr - type * a.rows, type, column, sum);
}

// Tiles and splits of one product.  The column tile is the one of 56 or 64
// that pads the two parities least (56 divides the 224 + 168 columns of lmax
// 6, nmax 8 exactly; 64 would do 14 % more).  The k-vectors are split, at
// least 128 to a split, so that the CTAs fill whole waves of the chip: 1000
// atoms have 336 CTAs for 592 places, and three splits of them, which fill
// two thirds of the third wave, took 0.56 ms where the rule's choice takes
// 0.51.  A split costs two steps (its prologue and its share of the sums) and
// the memory of the whole product, 512 MB of which are the most: more splits
// than that holds gain a few percent of many waves (by the rule's own time 2 %
// for 4500 k-vectors, up to 8 % for 19 200), and would take ten times the
// output for 160 000 k-vectors.
constexpr int64_t LODE_PARTIAL_BYTES = (int64_t)512 << 20;

template <int NB, bool GRAD>
int lode_resident() {
    int device = 0, sms = 0, per_sm = 0;
    CUDA_CHECK(cudaGetDevice(&device));
    CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lode_gemm_kernel<NB, GRAD>, LODE_THREADS, 0));
    return sms * std::max(1, per_sm);
}

template <bool GRAD>
void launch_lode_gemm(LodeArgs a, int64_t rows, int n_types, DeviceArena& arena, cudaStream_t stream) {
    if (rows == 0 || n_types == 0) return;
    auto tiles = [&](int bn, int n) { return (n + bn - 1) / bn; };
    const int t7 = tiles(56, a.cols.n_even) + tiles(56, a.cols.n_odd), t8 = tiles(64, a.cols.n_even) + tiles(64, a.cols.n_odd);
    const int nb = t7 * 7 < t8 * 8 ? 7 : 8;
    a.rows = rows;
    a.tiles_even = tiles(8 * nb, a.cols.n_even);
    a.tiles = a.tiles_even + tiles(8 * nb, a.cols.n_odd);
    const int64_t row_tiles = (rows + LODE_ROWS - 1) / LODE_ROWS;
    const int64_t ctas = row_tiles * a.tiles * n_types;
    const int steps = a.Kp / LODE_KB, resident = nb == 7 ? lode_resident<7, GRAD>() : lode_resident<8, GRAD>();
    const int64_t split_bytes = (int64_t)sizeof(double) * n_types * rows * a.cols.ld;
    int best = 1;
    double best_time = 1e300;
    for (int q = 1; q <= std::max(1, std::min(32, steps / 8)); q++) {
        if (q > 1 && q * split_bytes > LODE_PARTIAL_BYTES) break;
        const int64_t waves = (ctas * q + resident - 1) / resident;
        const double time = (double)waves * ((steps + q - 1) / q + 2);
        if (time < 0.98 * best_time) {
            best_time = time;
            best = q;
        }
    }
    a.split_k = (steps + best - 1) / best * LODE_KB;
    a.splits = (a.Kp + a.split_k - 1) / a.split_k;
    if (row_tiles * a.tiles > 0x7fffffffLL) throw invalid_parameter("the LODE product is too large for one launch");
    if (a.splits > 1) a.partial = (double*)arena.alloc_bytes("lode.partial", a.splits * split_bytes);
    const dim3 grid((unsigned)(row_tiles * a.tiles), (unsigned)n_types, (unsigned)a.splits);
    if (nb == 7) lode_gemm_kernel<7, GRAD><<<grid, LODE_THREADS, 0, stream>>>(a);
    else lode_gemm_kernel<8, GRAD><<<grid, LODE_THREADS, 0, stream>>>(a);
    CUDA_CHECK(cudaGetLastError());
    if (a.splits > 1) {
        const int64_t items = (int64_t)n_types * rows * a.cols.ld;
        lode_splits_kernel<GRAD><<<(unsigned)((items + 255) / 256), 256, 0, stream>>>(a, n_types);
        CUDA_CHECK(cudaGetLastError());
    }
}

}  // namespace

}  // namespace fb200

namespace fb200 {

LodeEngine::LodeEngine(const LodeHypers& h) : tables_(build_lode_tables(h)), ylm_(build_ylm_tables(h.max_angular)) {}

LodeEngine::~LodeEngine() {
    for (void* p : table_buffers_) cudaFree(p);
}

namespace {

// arrays of different types one after the other, for one copy to the device
struct HostPack {
    std::vector<unsigned char> bytes;
    template <typename T>
    size_t add(const std::vector<T>& v) {
        const size_t at = bytes.size();
        bytes.resize(at + (std::max<size_t>(1, v.size() * sizeof(T)) + 255) / 256 * 256);
        if (!v.empty()) std::memcpy(bytes.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
};

}  // namespace

void LodeEngine::upload_tables() {
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    if (tables_ready_ && dev == device_) return;
    if (tables_ready_) throw invalid_parameter("a calculator can only be used on the device it first ran on");
    device_ = dev;
    // every table in one allocation and one copy
    HostPack pack;
    const size_t at[] = {pack.add(ylm_.A),          pack.add(ylm_.B),          pack.add(ylm_.sq_plus),
                         pack.add(ylm_.sq_minus),   pack.add(ylm_.sq_2l1),     pack.add(ylm_.sq_half),
                         pack.add(ylm_.sq_ll1),     pack.add(ylm_.inv_ll),     pack.add(tables_.positions),
                         pack.add(tables_.values),  pack.add(tables_.derivs),  pack.add(tables_.knot_offset),
                         pack.add(tables_.knot_count)};
    unsigned char* d = nullptr;
    CUDA_CHECK(cudaMalloc(&d, pack.bytes.size()));
    table_buffers_.push_back(d);
    CUDA_CHECK(cudaMemcpy(d, pack.bytes.data(), pack.bytes.size(), cudaMemcpyHostToDevice));
    finish_copies();
    auto dbl = [&](int k) { return reinterpret_cast<const double*>(d + at[k]); };
    d_ylm_ = {ylm_.lmax, dbl(0), dbl(1), dbl(2), dbl(3), dbl(4), dbl(5), dbl(6), dbl(7)};
    d_spline_.lmax = tables_.h.max_angular;
    d_spline_.nmax = tables_.h.nmax();
    d_spline_.splined = tables_.positions.empty() ? 0 : 1;
    d_spline_.positions = dbl(8);
    d_spline_.values = dbl(9);
    d_spline_.derivs = dbl(10);
    d_spline_.knot_offset = reinterpret_cast<const int32_t*>(d + at[11]);
    d_spline_.knot_count = reinterpret_cast<const int32_t*>(d + at[12]);
    tables_ready_ = true;
}

namespace {

template <typename T>
T* put(DeviceArena& arena, const std::string& name, const std::vector<T>& v, cudaStream_t stream) {
    T* d = arena.alloc<T>(name, (int64_t)v.size());
    if (!v.empty()) CUDA_CHECK(cudaMemcpyAsync(d, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, stream));
    return d;
}

Labels labels_xyz() {
    Labels l;
    l.names = {"xyz"};
    l.values = {0, 1, 2};
    return l;
}

}  // namespace

// keys AllTypesPairsKeys x angular channels (spherical_expansion.rs:448-460,
// labels/keys.rs:36-57), samples and gradient samples LongRangeSamplesPerAtom
// (labels/samples/long_range.rs:21-74), then the kernels system by system
std::unique_ptr<TensorMap> LodeEngine::compute(const std::vector<HostSystem>& systems, const GradientOptions& g,
                                               bool device_output, const double* d_positions, cudaStream_t stream) {
    auto t_start = std::chrono::steady_clock::now();
    if (g.strain) throw invalid_parameter("the lode spherical expansion calculator does not support gradients with respect to strain");
    if (g.cell) throw invalid_parameter("the lode spherical expansion calculator does not support gradients with respect to cell");
    upload_tables();
    const LodeHypers& h = tables_.h;
    const int L = h.max_angular, N = h.nmax(), L2 = (L + 1) * (L + 1);

    // species and key pairs
    std::vector<int32_t> types;
    for (auto& s : systems) types.insert(types.end(), s.types.begin(), s.types.end());
    std::sort(types.begin(), types.end());
    types.erase(std::unique(types.begin(), types.end()), types.end());
    const int S = (int)types.size();
    auto species_of = [&](int32_t t) { return (int)(std::lower_bound(types.begin(), types.end(), t) - types.begin()); };
    std::vector<int32_t> pair_present((size_t)S * S, 0);
    std::vector<std::vector<int32_t>> sys_species(systems.size());
    for (size_t s = 0; s < systems.size(); s++) {
        std::vector<int32_t> present(S, 0);
        for (int32_t t : systems[s].types) present[species_of(t)] = 1;
        for (int a = 0; a < S; a++)
            for (int b = 0; b < S; b++)
                if (present[a] && present[b]) pair_present[(size_t)a * S + b] = 1;
        for (int32_t t : systems[s].types) sys_species[s].push_back(species_of(t));
        if (!systems[s].types.empty()) {
            const double* c = systems[s].cell;
            bool zero = true;
            for (int k = 0; k < 9; k++) zero &= c[k] == 0.0;
            if (zero) throw invalid_parameter("LODE can only be used with periodic systems");
        }
    }
    // blocks: pairs (a, b) in order, then l; per pair: samples and gradient rows
    struct PairPlan {
        Labels samples, grad_samples;
        int64_t n_samples = 0, n_grad = 0;
    };
    std::vector<PairPlan> pairs((size_t)S * S);
    std::vector<int32_t> keys_values;
    for (int a = 0; a < S; a++)
        for (int b = 0; b < S; b++) {
            if (!pair_present[(size_t)a * S + b]) continue;
            auto& pp = pairs[(size_t)a * S + b];
            pp.samples.names = {"system", "atom"};
            pp.grad_samples.names = {"sample", "system", "atom"};
            for (int l = 0; l <= L; l++) keys_values.insert(keys_values.end(), {l, 1, types[a], types[b]});
        }
    // per system: sample rows of every (atom, neighbour type) and gradient tasks
    std::vector<std::vector<int32_t>> rows(systems.size()), tasks(systems.size());
    for (size_t s = 0; s < systems.size(); s++) {
        const auto& sp = sys_species[s];
        const int n = (int)sp.size();
        std::vector<int32_t> count(S, 0);
        for (int32_t t : sp) count[t]++;
        rows[s].assign((size_t)n * S, -1);
        for (int i = 0; i < n; i++)
            for (int t = 0; t < S; t++) {
                if (!count[t]) continue;
                auto& pp = pairs[(size_t)sp[i] * S + t];
                const int32_t r = (int32_t)pp.n_samples++;
                rows[s][(size_t)i * S + t] = r;
                pp.samples.values.insert(pp.samples.values.end(), {(int32_t)s, i});
                if (!g.positions) continue;
                for (int j = 0; j < n; j++) {
                    if (sp[j] != t && j != i) continue;
                    tasks[s].insert(tasks[s].end(), {i, j, t, (int32_t)pp.n_grad});
                    pp.grad_samples.values.insert(pp.grad_samples.values.end(), {r, (int32_t)s, j});
                    pp.n_grad++;
                }
            }
    }
    // the samples of a block are ordered by system, then atom: rows above
    // were numbered per (atom, type) in that order within each system
    // offsets: per block values, then positions gradients
    std::vector<int64_t> off_values((size_t)S * S * (L + 1), -1), off_positions((size_t)S * S * (L + 1), -1);
    int64_t total = 0;
    for (int a = 0; a < S; a++)
        for (int b = 0; b < S; b++) {
            if (!pair_present[(size_t)a * S + b]) continue;
            const auto& pp = pairs[(size_t)a * S + b];
            for (int l = 0; l <= L; l++) {
                const size_t k = ((size_t)a * S + b) * (L + 1) + l;
                off_values[k] = total;
                total += pp.n_samples * (2 * l + 1) * N;
                if (g.positions) {
                    off_positions[k] = total;
                    total += pp.n_grad * 3 * (2 * l + 1) * N;
                }
            }
        }

    double* d_out = nullptr;
    std::shared_ptr<void> storage;
    {
        void* p = nullptr;
        CUDA_CHECK(cudaMallocAsync(&p, std::max<size_t>(8, sizeof(double) * (size_t)total), stream));
        CUDA_CHECK(cudaMemsetAsync(p, 0, std::max<size_t>(8, sizeof(double) * (size_t)total), stream));
        storage = std::shared_ptr<void>(p, [](void* q) { cudaFreeAsync(q, nullptr); });
        d_out = (double*)p;
    }
    cudaEvent_t ev0, ev1;
    CUDA_CHECK(cudaEventCreate(&ev0));
    CUDA_CHECK(cudaEventCreate(&ev1));
    CUDA_CHECK(cudaEventRecord(ev0, stream));

    int64_t atom_offset = 0;
    for (size_t s = 0; s < systems.size(); s++) {
        const HostSystem& sys = systems[s];
        const int n = (int)sys.n_atoms;
        if (n == 0) continue;
        KVectors kv = compute_k_vectors(sys.cell, h.k_cutoff);
        const int K = (int)kv.count();
        if (K == 0) throw invalid_parameter("No k-vectors for current combination of hyper parameters.");
        const double* c = sys.cell;
        const double volume = std::fabs(c[0] * (c[4] * c[8] - c[5] * c[7]) - c[1] * (c[3] * c[8] - c[5] * c[6]) +
                                        c[2] * (c[3] * c[7] - c[4] * c[6]));
        const double global = 4.0 * M_PI / volume;
        const int Kp = (K + LODE_KB - 1) / LODE_KB * LODE_KB;
        // the radial integral is evaluated on the device from its spline; the
        // analytic integral comes from here
        std::vector<double> kvec(3 * (size_t)Kp, 0.0), gdf(Kp, 0.0), radial(h.splined ? 0 : (size_t)K * (L + 1) * N);
#pragma omp parallel for schedule(static)
        for (int k = 0; k < K; k++) {
            for (int x = 0; x < 3; x++) kvec[3 * k + x] = kv.norm[k] * kv.direction[3 * k + x];
            gdf[k] = global * tables_.density_fourier(kv.norm[k]);
            if (h.splined) continue;
            for (int l = 0; l <= L; l++) tables_.radial(l, kv.norm[k], &radial[((size_t)k * (L + 1) + l) * N], nullptr);
        }
        std::vector<double> k0(N);
        for (int q = 0; q < N; q++) k0[q] = global * tables_.k0[q];
        std::vector<int32_t> count(S, 0);
        for (int32_t t : sys_species[s]) count[t]++;

        // the atoms by type, and the types of this system
        std::vector<int32_t> sorted_atoms, type_start(S + 1, 0), present;
        for (int t = 0; t < S; t++) {
            type_start[t + 1] = type_start[t] + count[t];
            if (count[t]) present.push_back(t);
        }
        sorted_atoms.resize(n);
        {
            std::vector<int32_t> next(type_start.begin(), type_start.end() - 1);
            for (int i = 0; i < n; i++) sorted_atoms[next[sys_species[s][i]]++] = i;
        }

        // everything the kernels read from here, in one copy
        HostPack pack;
        const size_t o_species = pack.add(sys_species[s]), o_kvec = pack.add(kvec), o_norm = pack.add(kv.norm),
                     o_dir = pack.add(kv.direction), o_gdf = pack.add(gdf), o_radial = pack.add(radial),
                     o_sorted = pack.add(sorted_atoms), o_start = pack.add(type_start), o_present = pack.add(present),
                     o_rows = pack.add(rows[s]), o_count = pack.add(count), o_center = pack.add(tables_.center),
                     o_k0 = pack.add(k0), o_offv = pack.add(off_values), o_offp = pack.add(off_positions),
                     o_positions = d_positions ? 0 : pack.add(sys.positions);
        const unsigned char* d_pack = put(arena_, "lode.pack", pack.bytes, stream);
        auto doubles = [&](size_t at) { return reinterpret_cast<const double*>(d_pack + at); };
        auto ints = [&](size_t at) { return reinterpret_cast<const int32_t*>(d_pack + at); };
        LodeArgs a{};
        a.Kp = Kp;
        a.S = S;
        a.cols = lode_columns(L, N);
        a.L = L;
        a.N = N;
        a.species = ints(o_species);
        a.kvec = doubles(o_kvec);
        a.gdf = doubles(o_gdf);
        // cos, sin, their sums by type and T in one allocation
        const int64_t phases = (int64_t)n * Kp, sums = (int64_t)S * Kp;
        double* C = arena_.alloc<double>("lode.work", 2 * phases + 2 * sums + (int64_t)Kp * a.cols.ld);
        double* Sn = C + phases;
        double* Ct = Sn + phases;
        double* St = Ct + sums;
        double* T = St + sums;
        a.T = T;
        a.C = C;
        a.Sn = Sn;
        a.Ct = Ct;
        a.St = St;
        a.present = ints(o_present);
        a.row = ints(o_rows);
        a.off_values = reinterpret_cast<const int64_t*>(d_pack + o_offv);
        a.off_positions = reinterpret_cast<const int64_t*>(d_pack + o_offp);
        a.type_count = ints(o_count);
        a.center = doubles(o_center);
        a.k0 = doubles(o_k0);
        a.center_factor = 1.0 - h.center_atom_weight;
        a.add_k0 = (h.exponent == 0 || h.exponent > 3) ? 1 : 0;
        a.out = d_out;
        const double* positions = d_positions ? d_positions + 3 * atom_offset : doubles(o_positions);
        // k-vectors per CTA of the projection: at most 8 and 48 KB of shared memory
        const size_t per_k = sizeof(double) * (size_t)((L + 1) * (L + 2) / 2 + L2 + (L + 1) * N);
        const int kc = (int)std::max<size_t>(1, std::min<size_t>(8, 48 * 1024 / per_k));
        allow_shared_memory(lode_projection_kernel, kc * per_k);
        lode_projection_kernel<<<(Kp + kc - 1) / kc, 128, kc * per_k, stream>>>(
            K, Kp, kc, N, a.cols, doubles(o_dir), doubles(o_norm), h.splined ? nullptr : doubles(o_radial), d_spline_, d_ylm_,
            T);
        CUDA_CHECK(cudaGetLastError());
        const int64_t nk = (int64_t)n * Kp;
        lode_phases_kernel<<<(unsigned)((nk + 255) / 256), 256, 0, stream>>>(n, K, Kp, positions, a.kvec, C, Sn);
        CUDA_CHECK(cudaGetLastError());
        lode_type_sums_kernel<<<dim3((Kp + 31) / 32, S), 256, 0, stream>>>(K, Kp, ints(o_sorted), ints(o_start), a.gdf, C,
                                                                          Sn, Ct, St);
        CUDA_CHECK(cudaGetLastError());
        launch_lode_gemm<false>(a, n, (int)present.size(), arena_, stream);
        if (g.positions && !tasks[s].empty()) {
            a.tasks = put(arena_, "lode.tasks", tasks[s], stream);
            launch_lode_gemm<true>(a, 3 * (int64_t)(tasks[s].size() / 4), 1, arena_, stream);
        }
        // the per-system buffers are reused by the next system
        CUDA_CHECK(cudaStreamSynchronize(stream));
        atom_offset += n;
    }
    CUDA_CHECK(cudaEventRecord(ev1, stream));

    auto tm = std::make_unique<TensorMap>();
    tm->on_device = device_output;
    tm->device = device_;
    tm->keys.names = {"o3_lambda", "o3_sigma", "center_type", "neighbor_type"};
    tm->keys.values = keys_values;
    double* base = d_out;
    if (device_output) {
        tm->storage = storage;
    } else {
        double* host = static_cast<double*>(std::malloc(std::max<size_t>(8, sizeof(double) * (size_t)total)));
        if (!host) throw std::bad_alloc();
        tm->storage = std::shared_ptr<void>(host, std::free);
        if (total) CUDA_CHECK(cudaMemcpyAsync(host, d_out, sizeof(double) * total, cudaMemcpyDeviceToHost, stream));
        base = host;
    }
    CUDA_CHECK(cudaStreamSynchronize(stream));
    Labels properties;
    properties.names = {"n"};
    for (int q = 0; q < N; q++) properties.values.push_back(q);
    for (int a = 0; a < S; a++)
        for (int b = 0; b < S; b++) {
            if (!pair_present[(size_t)a * S + b]) continue;
            const auto& pp = pairs[(size_t)a * S + b];
            for (int l = 0; l <= L; l++) {
                const size_t k = ((size_t)a * S + b) * (L + 1) + l;
                Labels mu;
                mu.names = {"o3_mu"};
                for (int m = -l; m <= l; m++) mu.values.push_back(m);
                auto blk = std::make_unique<Block>();
                blk->samples = pp.samples;
                blk->components = {mu};
                blk->properties = properties;
                blk->shape = {(size_t)pp.n_samples, (size_t)(2 * l + 1), (size_t)N};
                blk->data = base + off_values[k];
                if (g.positions) {
                    auto gb = std::make_unique<Block>();
                    gb->samples = pp.grad_samples;
                    gb->components = {labels_xyz(), mu};
                    gb->properties = properties;
                    gb->shape = {(size_t)pp.n_grad, 3, (size_t)(2 * l + 1), (size_t)N};
                    gb->data = base + off_positions[k];
                    blk->gradients.emplace_back("positions", std::move(gb));
                }
                tm->blocks.push_back(std::move(blk));
            }
        }
    float ms = 0.0f;
    CUDA_CHECK(cudaEventElapsedTime(&ms, ev0, ev1));
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    times_ = PhaseTimes{};
    times_.expansion = ms;
    times_.total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
    return tm;
}

}  // namespace fb200
