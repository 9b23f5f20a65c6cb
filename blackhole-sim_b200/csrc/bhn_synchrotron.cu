// bhn_synchrotron.cu -- coefficient-brick precompute on the GPU.
//
// The reference fills a brick cell by cell in Python
// (python/blackhole_sim/coefficient_bricks.py:119-152): per cell a local plasma
// frame (_fast_frame, :110-116: no line-of-sight pitch) and the Hybrid
// synchrotron model (bhn_synchrotron.cuh).  Here a warp owns a batch of cells.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>

#include "blackhole_native.h"
#include "bhn_internal.cuh"
#include "bhn_synchrotron.cuh"

namespace bhn {
namespace synch {

// Frames per warp: a batch amortises the per-frame scalars over its lanes, and
// below 32 frames a warp the GPU's resident warps come first.
static int frames_per_warp(int64_t n, int sms) {
    const int64_t resident = (int64_t)sms * 24;
    return (int)std::max<int64_t>(1, std::min<int64_t>(32, (n + resident - 1) / resident));
}

// Six 128-thread blocks per SM (80 registers): 30,011 Hybrid frames took 188
// us against 242 at five and 193 at seven and eight, before the power law's
// nodes were grouped.  Now 93 us and 27 us for the tables (728 us with one
// frame per warp and two exp() per node and pitch angle; 100 and 35 while the
// blocks copied their tables through the constant bank), 2.5 ns a frame at a
// million and more (22.6).  Leaving out the row lookups takes three quarters
// of it, cheap stand-ins for log or exp 9 % each; the issue slots are two
// thirds busy, fixed FP64 latencies and the shared-memory round trip of
// add_nodes fill the rest.  Two chunks of nodes per exchange, to overlap
// those, were slower (116 us; 125 at four blocks without spills).
struct PrecomputeParams {
    Model M;
    double nu;
    const double *rho, *theta_e, *b_con;
    void *out;
    int64_t cells;
    int out_bytes, per_warp;
};

__global__ void __launch_bounds__(128, 6) precompute_kernel(const __grid_constant__ PrecomputeParams P) {
    __shared__ TableSmem T;
    load_table(T, P.M);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t first = warp * P.per_warp; first < P.cells; first += warps * P.per_warp) {
        const int count = (int)min((int64_t)P.per_warp, P.cells - first);
        const int64_t cell = first + lane;
        Frame f = {0.0, 1.0, 0.0, 0.0, 0.0, P.nu};
        if (lane < count) {
            // coefficient_bricks.py:110-116 with calibration.py:113-119
            const double b1 = P.b_con[4 * cell + 1], b2 = P.b_con[4 * cell + 2], b3 = P.b_con[4 * cell + 3];
            const double b_code = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(b1, b1), __dmul_rn(b2, b2)), __dmul_rn(b3, b3)));
            f.b = fmax(b_code * P.M.b_unit, 0.0);
            f.n_e = P.rho[cell] * P.M.rho_unit / P.M.mu_e_mp;
            f.chi = b_code > 0.0 ? atan2(b3, b2) : 0.0;  // atan2(b_vec[2], b_vec[1]) of b_vec = b_con[1:]
            f.te = fmax(P.theta_e[cell], 1.0e-8);
        }
        double out[11];
        coefficients(T, P.M, f, count, out);
        if (lane >= count) continue;
        // the brick's dtype, then np.nan_to_num(nan=0, posinf=finfo.max, neginf=0) (coefficient_bricks.py:151)
#pragma unroll
        for (int k = 0; k < 11; ++k) {
            double v = out[k];
            if (P.out_bytes == 4) {
                float f32 = (float)v;
                f32 = isnan(f32) ? 0.0f : (isinf(f32) ? (f32 > 0.0f ? 3.402823466e38f : 0.0f) : f32);
                reinterpret_cast<float *>(P.out)[11 * cell + k] = f32;
            } else {
                v = isnan(v) ? 0.0 : (isinf(v) ? (v > 0.0 ? 1.7976931348623157e308 : 0.0) : v);
                reinterpret_cast<double *>(P.out)[11 * cell + k] = v;
            }
        }
    }
}

// The model's coefficients for given local plasma frames (synchrotron.py:248,
// :290, :318 -- ThermalSynchrotronCoefficients / NonthermalPowerLaw... /
// HybridSynchrotronCoefficients.coefficients(frame, nu_hz)):
// frames[5 i .. 5 i + 4] = (n_e [cm^-3], Theta_e, B [G], cos of the pitch
// to the line of sight, EVPA), out[11 i .. 11 i + 10] in PolarizedCoefficients
// field order (the brick's COEFF_NAMES order).  Theta_e is taken as given: the
// reference's models floor it only where they divide by it.
struct FrameParams {
    Model M;
    double nu;
    const double *frames;
    double *out;
    int64_t n;
    int per_warp;
};

__global__ void __launch_bounds__(128, 6) frame_coefficients_kernel(const __grid_constant__ FrameParams P) {
    __shared__ TableSmem T;
    load_table(T, P.M);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t first = warp * P.per_warp; first < P.n; first += warps * P.per_warp) {
        const int count = (int)min((int64_t)P.per_warp, P.n - first);
        Frame f = {0.0, 1.0, 0.0, 0.0, 0.0, P.nu};
        if (lane < count) {
            const double *p = P.frames + 5 * (first + lane);
            f = {p[0], p[1], p[2], p[3], p[4], P.nu};
        }
        double out[11];
        coefficients(T, P.M, f, count, out);
        if (lane < count) {
#pragma unroll
            for (int k = 0; k < 11; ++k) P.out[11 * (first + lane) + k] = out[k];
        }
    }
}

// ------------------------------------------------------------ tables
constexpr int kSeries = 12;  // Taylor terms before economisation

// Terms first, first + stride, ... of a row's Taylor series (F and G) about
// its centre, in units of the half width h, each times its degree's factorial.  A term sees the table segment at
// its x (numpy.interp: constant past either end of the knots).
__device__ inline void row_series(const KernelTable &K, const SumPlan &P, double centre, double h, int first, int stride,
                                  double aF[kSeries], double aG[kSeries]) {
    for (int d = 0; d < kSeries; ++d) aF[d] = aG[d] = 0.0;
    for (int t = first; t < P.n; t += stride) {
        const double x = centre - P.shift[t];
        int j = (int)((x - K.lx[0]) * P.inv_delta);
        j = j < 0 ? 0 : (j > kTable - 2 ? kTable - 2 : j);
        j -= j > 0 && x < K.lx[j] ? 1 : 0;  // the log-uniform knots' guess is within one segment
        j += j < kTable - 2 && x >= K.lx[j + 1] ? 1 : 0;
        double vF = K.sF[j] * (x - K.lx[j]) + K.lF[j], vG = K.sG[j] * (x - K.lx[j]) + K.lG[j];
        double sF = K.sF[j] * h, sG = K.sG[j] * h;
        if (x >= K.lx[kTable - 1] || x < K.lx[0]) {
            vF = x < K.lx[0] ? K.lF[0] : K.lF[kTable - 1];
            vG = x < K.lx[0] ? K.lG[0] : K.lG[kTable - 1];
            sF = sG = 0.0;
        }
        double uF = P.weight[t] * exp(vF), uG = P.weight[t] * exp(vG);
        for (int d = 0; d < kSeries; ++d) {  // moments; the factorials follow the sum
            aF[d] += uF;
            aG[d] += uG;
            uF *= sF;
            uG *= sG;
        }
    }
}

// The series of row_series economised to degree 7 (v^n -> v^n - T_n(v) / 2^(n-1), n = 11 .. 8,
// v = z / h) and scaled to powers of z.
__device__ inline void row_coefficients(double a[kSeries], double h, double co[8]) {
    // Chebyshev polynomials T_11 .. T_8 below their leading terms
    const double t11[5] = {-11.0, 220.0, -1232.0, 2816.0, -2816.0};  // v, v^3 .. v^9
    const double t10[5] = {-1.0, 50.0, -400.0, 1120.0, -1280.0};     // 1, v^2 .. v^8
    const double t9[4] = {9.0, -120.0, 432.0, -576.0};
    const double t8[4] = {1.0, -32.0, 160.0, -256.0};
    const double inverse[kSeries] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320,
                                     1.0 / 362880, 1.0 / 3628800, 1.0 / 39916800};  // factorials
#pragma unroll
    for (int d = 2; d < kSeries; ++d) a[d] *= inverse[d];
    for (int d = 0; d < 5; ++d) a[2 * d + 1] -= a[11] * t11[d] * (1.0 / 1024.0);
    for (int d = 0; d < 5; ++d) a[2 * d] -= a[10] * t10[d] * (1.0 / 512.0);
    for (int d = 0; d < 4; ++d) a[2 * d + 1] -= a[9] * t9[d] * (1.0 / 256.0);
    for (int d = 0; d < 4; ++d) a[2 * d] -= a[8] * t8[d] * (1.0 / 128.0);
    const double ih = h > 0.0 ? 1.0 / h : 0.0;
    double w = 1.0;
    for (int d = 0; d < 8; ++d, w *= ih) co[d] = a[d] * w;
}

// The row's cell, and its centre and half width in L.
__device__ inline void row_place(const SumPlan &P, int row, double &centre, double &h) {
    int c = 0, hi = P.cells;  // the cell whose first row is the last at or before `row`
    while (hi - c > 1) {
        const int mid = (c + hi) >> 1;
        if ((P.cell[mid] >> 4) <= row) c = mid;
        else hi = mid;
    }
    const int split = P.cell[c] & 15, in_cell = row - (P.cell[c] >> 4), k = in_cell >> split;
    const double width = P.edge[k + 1] - P.edge[k];
    centre = row_centre(P.y0, P.delta, (double)c, P.edge[k], width, split, in_cell & ((1 << split) - 1));
    h = 0.5 * width * P.delta / (double)(1 << split);
}

struct TableParams {
    KernelTable K;
    SumPlan plan[3];           // thermal pitch average, power-law group, power-law pitch average
    double2 *rows[3];          // NULL: off, or shared with an earlier one
    double2 *nt_nodes;         // NULL: no power law
    double *nt_norm;
    int nt_n, nt_group;
    double p, gamma_min, gamma_max;
};

// The tables of one call: two lanes per row, each half of the sum's terms and
// then one of the two kernels' coefficients; the last block makes the power
// law's nodes.  Tens of thousands of rows and no reuse: bound by the FP64 work
// of a term (two exponentials, 24 moments) and a row (economisation).  The
// default Hybrid model's 39,892 rows take 27 us (35 with the knots copied
// through the constant bank, then 43 with four lanes a row and two more rounds
// of 24 shuffles); 51 us with a product more per moment and with the rows past
// the far tail, a fifth of them, which no lookup reaches.
constexpr int kRowLanes = 2;
__global__ void __launch_bounds__(128) sum_table_kernel(const __grid_constant__ TableParams P) {
    __shared__ KernelTable K;
    if (blockIdx.x == gridDim.x - 1) {
        if (!P.nt_nodes) return;
        // Trapezoid weights c_i gamma_i^-p on gamma = geomspace(gamma_min, gamma_max, n): c_i = gamma_i (r - 1/r) / 2
        // inside, gamma_0 (r - 1) / 2 and gamma_{n-1} (1 - 1/r) / 2 at the ends.  Groups take every node at its inside
        // weight; the single nodes after them are the ends' differences and the nodes past the last whole group.
        const int n = P.nt_n, G = P.nt_group, groups = n / G;
        const double l0 = log(P.gamma_min), lr = (log(P.gamma_max) - l0) / (double)(n - 1);
        const double up = expm1(lr), down = -expm1(-lr);
        auto weight = [&](int i, double c) { return c * exp((1.0 - P.p) * fma((double)i, lr, l0)); };
        double norm = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const double c = i == 0 ? 0.5 * up : (i == n - 1 ? 0.5 * down : 0.5 * (up + down));
            norm += weight(i, c);
            if (i < groups) P.nt_nodes[i] = make_double2(weight(i * G, 0.5 * (up + down)), 2.0 * fma((double)(i * G), lr, l0));
            if (i >= groups * G && i < n - 1)
                P.nt_nodes[groups + 2 + i - groups * G] = make_double2(weight(i, 0.5 * (up + down)), 2.0 * fma((double)i, lr, l0));
        }
        if (threadIdx.x == 0) {
            const bool grouped = groups * G == n;  // the last node lies in a group
            P.nt_nodes[groups] = make_double2(weight(0, -0.5 * down), 2.0 * l0);
            P.nt_nodes[groups + 1] = make_double2(weight(n - 1, grouped ? -0.5 * up : 0.5 * down),
                                                  2.0 * fma((double)(n - 1), lr, l0));
        }
        __shared__ double part[4];
        norm = warp_sum(norm);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = norm;
        __syncthreads();
        if (threadIdx.x == 0) *P.nt_norm = (part[0] + part[1]) + (part[2] + part[3]);
        return;
    }
    const KernelTable &source = *lane_reads(&P.K);
    for (int i = threadIdx.x; i < kTable; i += blockDim.x) {
        K.lx[i] = source.lx[i];
        K.lF[i] = source.lF[i];
        K.lG[i] = source.lG[i];
        K.sF[i] = source.sF[i];
        K.sG[i] = source.sG[i];
    }
    __syncthreads();
    const int part = threadIdx.x % kRowLanes;
    int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kRowLanes), which = 0;
    for (; which < 3; ++which) {
        const int n = P.rows[which] ? P.plan[which].rows : 0;
        if (row < n) break;
        row -= n;
    }
    const bool live = which < 3;
    const SumPlan &L = P.plan[live ? which : 0];
    double aF[kSeries], aG[kSeries], centre = 0.0, h = 0.0;
    for (int d = 0; d < kSeries; ++d) aF[d] = aG[d] = 0.0;
    if (live) {
        row_place(L, row, centre, h);
        row_series(K, L, centre, h, part, kRowLanes, aF, aG);
    }
#pragma unroll
    for (int d = 0; d < kSeries; ++d)
#pragma unroll
        for (int o = 1; o < kRowLanes; o *= 2) {
            aF[d] += __shfl_xor_sync(0xffffffffu, aF[d], o);
            aG[d] += __shfl_xor_sync(0xffffffffu, aG[d], o);
        }
    if (!live || part > 1) return;
    double co[8];
#pragma unroll
    for (int d = 0; d < kSeries; ++d) aF[d] = part == 0 ? aF[d] : aG[d];
    row_coefficients(aF, h, co);
    double *out = reinterpret_cast<double *>(P.rows[which] + 8 * (int64_t)row) + part;
#pragma unroll
    for (int d = 0; d < 8; ++d) out[2 * d] = co[d];
}

namespace {

// ------------------------------------------------------------ host tables
// K_nu(x) = int_0^inf exp(-x cosh t) cosh(nu t) dt (DLMF 10.32.9), trapezoid
// rule with the step scaled to the integrand's width near t = 0 and the range
// cut where x (cosh t - 1) exceeds 750.
double bessel_k(double nu, double x) {
    const double h = std::min(0.02, 0.25 / std::sqrt(x));
    const double t_max = std::acosh(1.0 + 750.0 / x);
    double s = 0.5 * std::exp(-x);
    for (int k = 1;; ++k) {
        const double t = k * h;
        if (t > t_max + h) break;
        s += std::exp(-x * std::cosh(t)) * std::cosh(nu * t);
    }
    return h * s;
}

// synchrotron.py:120-172: x = geomspace(1e-8, 1e3, 256), F(x) = 1.25 x^(1/3)
// exp(-x) (648 + x^2)^(1/12), G(x) = x K_{2/3}(x), stored as log values
// floored at log(1e-300), with numpy.interp's segment slopes.
const KernelTable &host_table() {
    static KernelTable t;
    static std::once_flag once;
    std::call_once(once, [] {
        const double ls = std::log10(1.0e-8), le = std::log10(1.0e3), step = (le - ls) / (kTable - 1);
        for (int i = 0; i < kTable; ++i) {
            double x = i == 0 ? 1.0e-8 : (i == kTable - 1 ? 1.0e3 : std::pow(10.0, (double)i * step + ls));
            const double xc = std::min(std::max(x, 1.0e-12), 1.0e3);
            double F = 1.25 * std::pow(xc, 1.0 / 3.0) * std::exp(-xc) * std::pow(648.0 + xc * xc, 1.0 / 12.0);
            double G = xc * bessel_k(2.0 / 3.0, xc);
            if (!std::isfinite(F)) F = 0.0;
            if (!std::isfinite(G)) G = 0.0;
            t.lx[i] = std::log(x);
            t.lF[i] = std::log(std::max(F, 1.0e-300));
            t.lG[i] = std::log(std::max(G, 1.0e-300));
        }
        for (int i = 0; i < kTable; ++i) {
            const int j = std::min(i, kTable - 2);
            t.sF[i] = (t.lF[j + 1] - t.lF[j]) / (t.lx[j + 1] - t.lx[j]);
            t.sG[i] = (t.lG[j + 1] - t.lG[j]) / (t.lx[j + 1] - t.lx[j]);
        }
        // first knot from which both log F and log G stay below log(kTailValue):
        // the linear segments in between stay below it too
        const double tail = std::log(kTailValue);
        int j0 = kTable;
        while (j0 > 0 && t.lF[j0 - 1] < tail && t.lG[j0 - 1] < tail) --j0;
        t.lx_tail = j0 < kTable ? t.lx[j0] : INFINITY;
    });
    return t;
}

// Gauss-Legendre nodes (ascending, as numpy.polynomial.legendre.leggauss) by
// Newton's method on P_n from the three-term recurrence.
void gauss_legendre(int n, double *x, double *w) {
    for (int k = 0; k < (n + 1) / 2; ++k) {
        double z = std::cos(kPiD * (k + 0.75) / (n + 0.5)), dp = 0.0;
        for (int it = 0; it < 100; ++it) {
            double p0 = 1.0, p1 = z;
            for (int l = 2; l <= n; ++l) {
                const double p2 = ((2.0 * l - 1.0) * z * p1 - (l - 1.0) * p0) / l;
                p0 = p1;
                p1 = p2;
            }
            if (n == 1) p0 = 1.0, p1 = z;
            dp = n * (z * p1 - p0) / (z * z - 1.0);
            const double dz = p1 / dp;
            z -= dz;
            if (std::fabs(dz) < 1e-16) break;
        }
        double p0 = 1.0, p1 = z;
        for (int l = 2; l <= n; ++l) {
            const double p2 = ((2.0 * l - 1.0) * z * p1 - (l - 1.0) * p0) / l;
            p0 = p1;
            p1 = p2;
        }
        dp = n * (z * p1 - p0) / (z * z - 1.0);
        const double wk = 2.0 / ((1.0 - z * z) * dp * dp);
        x[k] = -z;
        x[n - 1 - k] = z;
        w[k] = w[n - 1 - k] = wk;
    }
    if (n % 2 == 1) x[n / 2] = 0.0;
}

// The pitch average's terms: shift log sin(alpha), weight the pitch weight times pref / B.
void pitch_terms(int n, SumPlan &ps) {
    double x[kMaxPitch], w[kMaxPitch];
    gauss_legendre(n, x, w);
    ps.n = 0;
    const double pref = std::sqrt(3.0) * kE * kE * kE / (kMe * kC * kC);  // synchrotron.py:185-186 per Gauss
    for (int m = 0; m < n; ++m) {
        const double sin_a = std::sqrt(std::max(0.0, 1.0 - x[m] * x[m]));
        if (!(sin_a > 0.0)) continue;  // Bp = B sin(alpha) <= 0 contributes nothing
        const double ls = std::log(sin_a), wt = 0.5 * w[m] * pref * sin_a;
        // the Gauss-Legendre nodes come in pairs +-mu with one sin(alpha) and one
        // weight: the pair's two lookups are the same numbers, so it is one node
        // of twice the weight
        int k = 0;
        while (k < ps.n && ps.shift[k] != ls) ++k;
        if (k < ps.n) {
            ps.weight[k] += wt;
            continue;
        }
        ps.shift[ps.n] = ls;
        ps.weight[ps.n] = wt;
        ++ps.n;
    }
}

// The pieces that the table knots seen through a sum's terms cut a cell into
// (wide gaps split: at most a quarter of a cell, or twice the mean) and every
// cell's split into rows.  The cells end with the far tail: no lookup passes it.
int cells_of(double y0, double shift_max) {
    const KernelTable &K = host_table();
    return (int)std::floor((K.lx_tail + shift_max - y0) * ((kTable - 1) / (K.lx[kTable - 1] - K.lx[0])) + 0.5) + 2;
}
void make_plan(SumPlan &P) {
    const KernelTable &K = host_table();
    P.delta = (K.lx[kTable - 1] - K.lx[0]) / (kTable - 1);
    P.inv_delta = 1.0 / P.delta;
    const double low = *std::min_element(P.shift, P.shift + P.n);
    P.shift_max = *std::max_element(P.shift, P.shift + P.n);
    P.y0 = K.lx[0] + low;
    double cut[kMaxTerms + 2];
    int cuts = 0;
    for (int t = 0; t < P.n; ++t) {
        const double u = (P.shift[t] - low) * P.inv_delta;
        cut[cuts++] = u - std::floor(u + 0.5);  // the knots' offset from the cells' centres, in [-1/2, 1/2)
    }
    cut[cuts++] = -0.5;
    cut[cuts++] = 0.5;
    std::sort(cut, cut + cuts);
    P.pieces = 0;
    const double gap = std::min(0.25, 2.0 / P.n);
    for (int i = 0; i + 1 < cuts; ++i) {
        if (!(cut[i + 1] > cut[i])) continue;
        const int parts = std::max(1, (int)std::ceil((cut[i + 1] - cut[i]) / gap - 1e-9));
        for (int q = 0; q < parts; ++q) P.edge[P.pieces++] = cut[i] + (cut[i + 1] - cut[i]) * q / parts;
    }
    P.edge[P.pieces] = 0.5;
    double widest = 0.0;
    for (int k = 0; k < P.pieces; ++k) widest = std::max(widest, P.edge[k + 1] - P.edge[k]);
    P.tries = 0;
    for (int b = 0; b < kBins; ++b) {
        const double left = (double)b / kBins - 0.5 - 1e-6, right = left + 1.0 / kBins + 2e-6;
        P.first[b] = 0;
        while (P.first[b] + 1 < P.pieces && P.edge[P.first[b] + 1] <= left) ++P.first[b];
        int in_bin = 0;
        while (P.first[b] + in_bin + 1 < P.pieces && P.edge[P.first[b] + in_bin + 1] <= right) ++in_bin;
        P.tries = std::max(P.tries, in_bin);
    }
    P.cells = cells_of(P.y0, P.shift_max);
    // Row half widths h with U = s h <= 0.07 x^(1/8) (x >= 1): the first term that economisation drops is then
    // U^8 / (8! 2^7) < 1.2e-16 x of the sum, below the rounding of an exponent of size x.  The terms' slopes are -x (1/3 - x near 0) with weights falling like exp(-x), x >= x_min: the eighth
    // root of their weighted eighth moment is at most s = 8 exp((x_min - 8) / 8) up to x_min = 8, x_min + 1 beyond.
    P.rows = 0;
    double x = std::exp(P.y0 + 0.5 * P.delta - P.shift_max);
    const double ratio = std::exp(P.delta);
    for (int c = 0; c < P.cells; ++c, x *= ratio) {
        const double s = x >= 8.0 ? x + 1.0 : (x < 0.5 ? 3.2 : 8.0 * std::exp((x - 8.0) / 8.0));
        const double most = 0.07 * std::sqrt(std::sqrt(std::sqrt(std::max(x, 1.0))));
        int split = 0;
        for (double h = 0.5 * widest * P.delta; s * h > most && split < 10; h *= 0.5) ++split;
        P.cell[c] = P.rows << 4 | split;
        P.rows += P.pieces << split;
    }
}

// The pitch average's plan, a function of the node count alone: made once per
// count and process (3.6 KB each), under T_lock.  The plans of a call bounded the
// small ones: one thermal frame 25.6 -> 22.8 us, a Hybrid of 64 pitch nodes
// 123 -> 37, the default Hybrid 34.9 -> 33.2 (its power-law group is planned anew).
const SumPlan &pitch_plan(int n) {
    static SumPlan plans[kMaxPitch + 1];
    SumPlan &P = plans[n];
    if (P.rows == 0) {
        pitch_terms(n, P);
        make_plan(P);
    }
    return P;
}

void set_table(SumTable &T, const SumPlan &P, const double2 *rows) {
    T.rows = rows;
    T.y0 = P.y0;
    T.delta = P.delta;
    T.inv_delta = P.inv_delta;
    T.y0_cells = -P.y0 * P.inv_delta;
    T.shift_max = P.shift_max;
    T.pieces = P.pieces;
    T.tries = P.tries;
    std::memcpy(T.edge, P.edge, sizeof P.edge);
    std::memcpy(T.cell, P.cell, sizeof P.cell);
    std::memcpy(T.first, P.first, sizeof P.first);
}

// Power-law nodes per row: 8 (28 rows of the default 224 nodes, one per lane)
// while the group's sum has at most 64 terms and its span fits the cells.  Bakes
// and images always take groups; frame batches from kGroupFrames on, where they
// repay the group's table (a call without and with groups: 5,000 Hybrid frames
// 53.6 and 59.6 us, 8,192 67.5 and 65.8; power law alone 4,000 38.6 and 41.2,
// 8,192 47.5 and 43.5, 12,000 60.6 and 47.3).
constexpr int64_t kGroupFrames = 8192;
int group_size(const SumPlan &A, int gamma_n, double lr, bool grouped) {
    int g = 1;
    while (grouped && 2 * g * A.n <= 64 && 2 * g <= 8 && 2 * g <= gamma_n &&
           cells_of(A.y0, A.shift_max + 2.0 * lr * (2 * g - 1)) <= kMaxCells)
        g *= 2;
    return g;
}

// The table plans of a model (T, under the lock), the model without its tables'
// addresses (M) and the tables' size.
TableParams T;  // ~25 KB: kept off the host stack; filled and launched under the lock
std::mutex T_lock;
int64_t T_rows[3];  // rows of each sum's own table (0: off, or another sum's)
int T_same[3];      // which table serves each sum
int plan_model(const bhn_synchrotron_model *m, bool grouped, Model &M, int64_t &bytes) {
    if (!m) return fail(BHN_ERR_VALUE, "synchrotron model must not be NULL");
    if (!std::isfinite(m->nu_hz)) return fail(BHN_ERR_VALUE, "nu_hz must be finite");
    auto check_comp = [](int on, int gn, int pn) {
        return !on || (gn >= 2 && gn <= kMaxGamma && pn >= 1 && pn <= kMaxPitch);
    };
    if (!check_comp(m->thermal, m->thermal_gamma_n, m->thermal_pitch_n) ||
        !check_comp(m->nonthermal, m->nonthermal_gamma_n, m->nonthermal_pitch_n))
        return fail(BHN_ERR_VALUE, "gamma grids need 2.." + std::to_string(kMaxGamma) + " nodes and pitch averages 1.." +
                                       std::to_string(kMaxPitch) + " nodes");
    if (m->nonthermal && !(m->nonthermal_gamma_min > 0.0 && m->nonthermal_gamma_max > m->nonthermal_gamma_min))
        return fail(BHN_ERR_VALUE, "the power law needs 0 < gamma_min < gamma_max");
    std::memset(&M, 0, sizeof M);
    M.lx_tail = host_table().lx_tail;
    M.rho_unit = m->rho_cgs_per_code;
    M.b_unit = m->b_gauss_per_code;
    M.mu_e_mp = std::max(m->mean_molecular_weight_per_electron * kMp, 1.0e-300);
    M.th.on = m->thermal != 0;
    if (M.th.on) {
        M.th.gamma_n = m->thermal_gamma_n;
        M.th.rotation_scale = m->thermal_rotation_scale;
        M.th.conversion_scale = m->thermal_conversion_scale;
    }
    M.nt.on = m->nonthermal != 0;
    if (M.nt.on) {
        M.nt.gamma_n = m->nonthermal_gamma_n;
        M.nt.p = m->nonthermal_p;
        M.nt.gamma_min = m->nonthermal_gamma_min;
        M.nt.gamma_max = m->nonthermal_gamma_max;
        M.nt.fraction = m->nonthermal_fraction;
        M.nt.absorption_scale = m->nonthermal_absorption_scale;
        M.nt.faraday_scale = m->nonthermal_faraday_scale;
    }
    bytes = 0;
    if (!M.th.on && !M.nt.on) return BHN_OK;
    std::memset(&T, 0, sizeof T);
    T.K = host_table();
    for (int k = 0; k < 3; ++k) {
        T_rows[k] = 0;
        T_same[k] = k;
    }
    if (M.th.on) {
        T.plan[0] = pitch_plan(m->thermal_pitch_n);
        T_rows[0] = T.plan[0].rows;
    }
    // A power law without an upper end has no grid of nodes (its log ratio is infinite, and so would the group's
    // shifts be): every integral over it is indefinite, which the coefficients report as no emission.
    if (M.nt.on && std::isfinite(M.nt.gamma_max)) {
        T.plan[2] = pitch_plan(m->nonthermal_pitch_n);
        const SumPlan &A = T.plan[2];
        SumPlan &B = T.plan[1];
        T.nt_n = M.nt.gamma_n;
        const double lr = (std::log(M.nt.gamma_max) - std::log(M.nt.gamma_min)) / (T.nt_n - 1);
        T.nt_group = group_size(A, T.nt_n, lr, grouped);
        T.p = M.nt.p;
        T.gamma_min = M.nt.gamma_min;
        T.gamma_max = M.nt.gamma_max;
        M.nt_groups = T.nt_n / T.nt_group;
        M.nt_single = 2 + std::max(0, T.nt_n - M.nt_groups * T.nt_group - 1);
        if (M.th.on && m->thermal_pitch_n == m->nonthermal_pitch_n) T_same[2] = 0;
        else T_rows[2] = A.rows;
        if (T.nt_group == 1) {
            T_same[1] = T_same[2];
            B = A;
        } else {
            for (int i = 0; i < T.nt_group; ++i)
                for (int t = 0; t < A.n; ++t) {
                    B.shift[B.n] = A.shift[t] + 2.0 * lr * i;
                    B.weight[B.n] = A.weight[t] * std::exp((1.0 - T.p) * lr * i);
                    ++B.n;
                }
            make_plan(B);
            T_rows[1] = B.rows;
        }
    }
    bytes = 128 * (T_rows[0] + T_rows[1] + T_rows[2]) + 16 * (int64_t)(M.nt_groups + M.nt_single + 1);
    return BHN_OK;
}

}  // namespace

int build_model(const bhn_synchrotron_model *m, bool grouped, Model &M, Scratch &tables, cudaStream_t stream) {
    std::lock_guard<std::mutex> g(T_lock);
    int64_t bytes = 0;
    int rc = plan_model(m, grouped, M, bytes);
    if (rc || bytes == 0) return rc;
    if (!tables.p) {
        rc = stream_alloc(&tables.p, bytes, stream);
        if (rc) return rc;
        tables.owned = true;
        tables.stream = stream;
    } else if (tables.bytes < bytes || reinterpret_cast<uintptr_t>(tables.p) % 256) {
        return fail(BHN_ERR_VALUE, "model scratch needs bhn_synchrotron_scratch_bytes() bytes, 256-byte aligned");
    }
    double2 *next = static_cast<double2 *>(tables.p);
    for (int k = 0; k < 3; ++k) {
        if (T_rows[k]) T.rows[k] = next;
        next += 8 * T_rows[k];
    }
    if (M.nt_single) {
        T.nt_nodes = next;
        T.nt_norm = reinterpret_cast<double *>(next + M.nt_groups + M.nt_single);
    }
    const unsigned blocks = (unsigned)((kRowLanes * (T_rows[0] + T_rows[1] + T_rows[2]) + 127) / 128 + 1);
    sum_table_kernel<<<blocks, 128, 0, stream>>>(T);
    BHN_LAUNCH_CHECK("sum_table_kernel");
    if (M.th.on) set_table(M.tth, T.plan[0], T.rows[0]);
    if (M.nt_single) {
        set_table(M.tnt, T.plan[1], T.rows[T_same[1]]);
        set_table(M.tnt1, T.plan[2], T.rows[T_same[2]]);
    }
    M.nt_nodes = T.nt_nodes;
    M.nt_norm = T.nt_norm;
    return BHN_OK;
}

// The launches behind the entry points: scratch as Scratch::p, or NULL.
static int precompute(const double *rho, const double *theta_e, const double *b_con, int64_t cells,
                      const bhn_synchrotron_model *m, void *coeffs, int32_t coeff_bytes, void *scratch,
                      int64_t scratch_bytes, cudaStream_t s) {
    if (cells < 1) return fail(BHN_ERR_VALUE, "the snapshot must contain at least one cell");
    if (!rho || !theta_e || !b_con || !coeffs) return fail(BHN_ERR_VALUE, "missing snapshot or output buffer");
    if (coeff_bytes != 4 && coeff_bytes != 8) return fail(BHN_ERR_VALUE, "brick values must be float32 or float64");
    PrecomputeParams P;
    Scratch tables{scratch, scratch_bytes};
    int rc = build_model(m, true, P.M, tables, s);  // always: a brick's values must not depend on its slabs
    if (rc) return rc;
    P.nu = m->nu_hz;
    P.rho = rho;
    P.theta_e = theta_e;
    P.b_con = b_con;
    P.out = coeffs;
    P.cells = cells;
    P.out_bytes = coeff_bytes;
    const int sms = std::max(1, sm_count_current_device());
    P.per_warp = frames_per_warp(cells, sms);
    const int64_t batches = (cells + P.per_warp - 1) / P.per_warp;
    const int64_t blocks = std::min<int64_t>((batches + 3) / 4, (int64_t)sms * 16);
    precompute_kernel<<<(unsigned)blocks, 128, 0, s>>>(P);
    BHN_LAUNCH_CHECK("precompute_kernel");
    return BHN_OK;
}

static int frame_coefficients(const double *frames, int64_t n, const bhn_synchrotron_model *m, double *out,
                              void *scratch, int64_t scratch_bytes, cudaStream_t s) {
    if (n < 1) return fail(BHN_ERR_VALUE, "at least one plasma frame is required");
    if (!frames || !out) return fail(BHN_ERR_VALUE, "missing frame or output buffer");
    FrameParams P;
    Scratch tables{scratch, scratch_bytes};
    int rc = build_model(m, n >= kGroupFrames, P.M, tables, s);
    if (rc) return rc;
    P.nu = m->nu_hz;
    P.frames = frames;
    P.out = out;
    P.n = n;
    const int sms = std::max(1, sm_count_current_device());
    P.per_warp = frames_per_warp(n, sms);
    const int64_t batches = (n + P.per_warp - 1) / P.per_warp;
    const int64_t blocks = std::min<int64_t>((batches + 3) / 4, (int64_t)sms * 16);
    frame_coefficients_kernel<<<(unsigned)blocks, 128, 0, s>>>(P);
    BHN_LAUNCH_CHECK("frame_coefficients_kernel");
    return BHN_OK;
}

}  // namespace synch
}  // namespace bhn

extern "C" {

int64_t bhn_synchrotron_scratch_bytes(const bhn_synchrotron_model *m) {
    std::lock_guard<std::mutex> g(bhn::synch::T_lock);
    bhn::synch::Model M;
    int64_t bytes = 0;
    if (bhn::synch::plan_model(m, true, M, bytes)) return -1;  // the grouped tables are the larger ones
    return (bytes + 255) & ~(int64_t)255;
}

int bhn_brick_precompute(const double *rho, const double *theta_e, const double *b_con, int64_t cells,
                         const bhn_synchrotron_model *m, void *coeffs, int32_t coeff_bytes, void *stream) {
    return bhn::synch::precompute(rho, theta_e, b_con, cells, m, coeffs, coeff_bytes, nullptr, 0, bhn::as_stream(stream));
}

int bhn_brick_precompute_scratch(const double *rho, const double *theta_e, const double *b_con, int64_t cells,
                                 const bhn_synchrotron_model *m, void *coeffs, int32_t coeff_bytes, void *scratch,
                                 int64_t scratch_bytes, void *stream) {
    if (!scratch) return bhn::fail(BHN_ERR_VALUE, "model scratch must not be NULL");
    return bhn::synch::precompute(rho, theta_e, b_con, cells, m, coeffs, coeff_bytes, scratch, scratch_bytes,
                                  bhn::as_stream(stream));
}

int bhn_synchrotron_coefficients(const double *frames, int64_t n, const bhn_synchrotron_model *m, double *out,
                                 void *stream) {
    return bhn::synch::frame_coefficients(frames, n, m, out, nullptr, 0, bhn::as_stream(stream));
}

int bhn_synchrotron_coefficients_scratch(const double *frames, int64_t n, const bhn_synchrotron_model *m, double *out,
                                         void *scratch, int64_t scratch_bytes, void *stream) {
    if (!scratch) return bhn::fail(BHN_ERR_VALUE, "model scratch must not be NULL");
    return bhn::synch::frame_coefficients(frames, n, m, out, scratch, scratch_bytes, bhn::as_stream(stream));
}

}  // extern "C"
