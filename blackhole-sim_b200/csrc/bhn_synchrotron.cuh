// bhn_synchrotron.cuh -- synchrotron transfer coefficients on the GPU (FP64).
//
// The Hybrid / thermal / power-law models of python/blackhole_sim/
// synchrotron.py:240-325: each component a pitch-angle-averaged
// (Gauss-Legendre) trapezoid integral over a Lorentz-factor grid of the
// F(x) / G(x) synchrotron kernels, looked up log-log in a 256-entry table
// (synchrotron.py:157-172).
//
// Sums of shifted kernels.  With log x = L - log sin(alpha), L = log nu -
// log(1.5 nu_B) - 2 log gamma, the pitch sum A(L) = sum_m W_m K(L - log sin_m)
// of a kernel K is a function of L alone: between two breakpoints (a table
// knot seen through one of the pitch angles) every term is one exponential of
// L, so A is a fixed sum of exponentials there.  Both sums (F and G) are
// therefore tabulated piecewise -- one row per interval between breakpoints,
// or a power-of-two fraction of it where the exponents are steep: a degree-7
// polynomial in L minus the row's centre -- and a Lorentz-factor node costs one
// row (128 B) and 16 multiply-adds instead of two exp() for each of the 8
// distinct pitch angles of the 16-node rule.  The polynomials are the Taylor
// series of the sums, economised from degree 11 (Lanczos, "Applied Analysis",
// 1956, ch. VII), with the rows narrow enough for a truncation below 1e-16 of
// the sum.
// The power law's nodes form a geometric grid with geometric weights, so G
// consecutive ones are a sum of shifted A's with fixed weights, the same for
// every such group: a second table of that kind, T(L) = sum_{i < G} rho^i
// A(L - i h), takes them in one row (8 nodes: 28 rows instead of 224).
// The tables depend on the model, and on whether the call takes groups (bakes and
// images always, frames from kGroupFrames on); a call builds them on its stream
// (sum_table_kernel) in the caller's scratch or a stream-ordered allocation.
//
// One warp then evaluates a batch of frames: the per-frame scalars are
// computed by one lane per frame, the frames' integrals one after the other
// by all lanes (a lane takes every 32nd Lorentz-factor node; warp reductions
// give the normalisation and the j_I, j_Q integrals), and the 11 coefficients
// by one lane per frame again.
//
// Rewrites that change rounding only:
//  * the trapezoid sum sum_i d_i (y_i + y_{i+1}) / 2 is evaluated as
//    sum_i c_i y_i with c_i = (d_{i-1} + d_i) / 2, which separates the
//    pitch sum from the Lorentz-factor sum; on the geometric grid x_i =
//    x_0 r^i, c_i = x_i (r - 1/r) / 2;
//  * the thermal f = gamma^2 beta exp(-gamma / theta_e) with gamma^2 beta =
//    gamma sqrt(x (x + 2)), x = gamma - 1.
// The thermal distribution's normalisation theta_e K_2(1/theta_e)
// (synchrotron.py:189-196) cancels against its own trapezoid normalisation and
// is left out.  The table's G(x) = x K_{2/3}(x) is computed on the host from
// the integral representation K_nu(x) = int_0^inf exp(-x cosh t) cosh(nu t) dt
// (DLMF 10.32.9) by the trapezoid rule.
#pragma once

#include "blackhole_native.h"
#include "bhn_internal.cuh"

namespace bhn {
namespace synch {


// python/blackhole_sim/calibration.py:18-25, synchrotron.py:177
constexpr double kC = 2.99792458e10;
constexpr double kMp = 1.67262192369e-24;
constexpr double kMe = 9.1093837015e-28;
constexpr double kKb = 1.380649e-16;
constexpr double kE = 4.80320471257e-10;
constexpr double kH = 6.62607015e-27;
constexpr double kPiD = 3.14159265358979323846;

constexpr int kTable = 256;      // synchrotron.py:158
constexpr double kTailValue = 1.0e-250;  // F, G below this are dropped with their node (add_nodes)
constexpr int kMaxPitch = 64;
constexpr int kMaxGamma = 4096;

constexpr int kMaxTerms = 72;    // terms of a tabulated sum: distinct pitch angles (<= 33) times group size, at most 66
constexpr int kMaxPieces = 104;  // intervals per table cell: one per term, and splits of wide gaps
constexpr int kMaxCells = 320;   // 255 table cells and the span of the shifts
constexpr int kBins = 64;        // first-guess bins of the interval search

// A sum of shifted kernels S(L) = sum_t weight_t K(L - shift_t) as rows: the
// intervals that its breakpoints cut the log-uniform table cells into.  Cell c
// is centred on y0 + c delta; its pieces' edges are offsets in cells, the same
// in every cell.  Each piece of cell c is split into 2^split equal rows.
struct SumPlan {
    int n;                       // terms
    int pieces, cells, rows;     // pieces per cell; cells; rows of all cells
    int tries;                   // the most edges in one bin
    double y0, delta, inv_delta; // L of cell 0's centre, cell width
    double shift_max;            // the largest shift (the term with the smallest x)
    double shift[kMaxTerms], weight[kMaxTerms];
    double edge[kMaxPieces + 1];
    int first[kBins];            // a piece at or left of every offset in the bin
    int cell[kMaxCells];         // cell c's first row << 4 | split
};

// The kernel table (log x knots, log F, log G, segment slopes).
struct KernelTable {
    double lx[kTable], lF[kTable], lG[kTable], sF[kTable], sG[kTable];
    double lx_tail;  // from this log x on, F and G are below kTailValue up to the table end (+inf: nowhere)
};

struct Component {
    int on, gamma_n;
    double p, gamma_min, gamma_max, fraction, absorption_scale, faraday_scale;  // power law
    double rotation_scale, conversion_scale;                                     // thermal
};

// A tabulated sum in the evaluation kernels: rows[8 r + d] = the degree-d
// coefficients of (F, G) of row r.
struct SumTable {
    const double2 *rows;
    double y0, y0_cells, delta, inv_delta, shift_max;  // y0_cells = -y0 / delta
    int pieces, tries;
    double edge[kMaxPieces + 1];
    int first[kBins], cell[kMaxCells];
};

// The model in device form: the two components with their sums' tables and the
// plasma scaling of calibration.py:113-119 (n_e = rho rho_unit / (mu_e m_p),
// B = |b| b_unit).
struct Model {
    double rho_unit, b_unit, mu_e_mp, lx_tail;
    Component th, nt;
    SumTable tth;             // thermal: the pitch average
    SumTable tnt, tnt1;       // power law: a group of nodes; the pitch average (its ungrouped nodes)
    int nt_groups, nt_single;
    const double2 *nt_nodes;  // power law: (weight, 2 log gamma) of every group, then of the ungrouped nodes
    const double *nt_norm;    // the sum of all nodes' weights (NULL: a power law without an upper end, no nodes)
};

// Shared-memory copy of a table's interval search.
struct PieceSmem {
    double edge[kMaxPieces + 1], width[kMaxPieces];
    float inv_width[kMaxPieces];
    int first[kBins], cell[kMaxCells];
};
// One warp's exchange between the nodes (a lane each) and the row loads (four
// lanes a row): per node its row and its weight times the powers of z.  Node n
// keeps powers 2 q and 2 q + 1 in pair 4 n + (q ^ (n / 2 & 3)), and its row
// at 4 (n % 8) + n / 8: the eight lanes of one 16-byte access, eight nodes
// writing or two being read, then lie on distinct banks.
struct __align__(16) NodeSmem {
    double2 pow[4 * 32];
    int row[32];
};
constexpr int kSynchWarps = 4;  // warps per block of the evaluation kernels
struct TableSmem {
    PieceSmem th, nt, nt1;
    NodeSmem node[kSynchWarps];
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// 2^n, -1022 <= n <= 1023
__device__ __forceinline__ double pow2(int n) { return __hiloint2double((n + 1023) << 20, 0); }

// L at the centre of row `sub` of 2^split in the piece [left, left + width) of cell c (table build and lookup alike).
__device__ __forceinline__ double row_centre(double y0, double delta, double c, double left, double width, int split,
                                             int sub) {
    double at = 0.5;
    if (split) at = ((double)sub + 0.5) * pow2(-split);  // exact
    return fma(c + fma(at, width, left), delta, y0);
}

// The row of L and L minus its centre.  The nearest cell comes from adding and
// subtracting 1.5 2^52 (round to nearest integer); the piece from the bin's
// first candidate and `tries` comparisons (the most edges a bin holds; the
// edge past the last piece is +inf).  A neighbouring piece taken for an L
// within rounding of an edge gives the same value to rounding: the sums are
// continuous (and smooth across a piece's rows, where single precision places L).
// L lies below the table's tail, so only its lower end needs the clamp
// (numpy.interp's constant value there).
__device__ __forceinline__ int sum_row(const SumTable &T, const PieceSmem &S, double L, double &z) {
    L = fmax(L, T.y0);
    constexpr double kRound = 6755399441055744.0;
    const double y = fma(L, T.inv_delta, T.y0_cells), t = y + kRound, whole = t - kRound;
    const int c = __double2loint(t);
    const double f = y - whole;
    int k = S.first[min((int)fmaf((float)f, (float)kBins, 0.5f * kBins), kBins - 1)];
    for (int q = 0; q < T.tries; ++q) k += f >= S.edge[k + 1] ? 1 : 0;
    const int cell = S.cell[c], split = cell & 15;
    const double left = S.edge[k];
    int sub = 0;
    if (split) sub = max(0, min((int)((float)(f - left) * S.inv_width[k] * (float)(1 << split)), (1 << split) - 1));
    z = L - row_centre(T.y0, T.delta, whole, left, S.width[k], split, sub);
    return (cell >> 4) + (k << split) + sub;
}

// Four doubles of read-only global memory in one load (32-byte aligned).
__device__ __forceinline__ void load_32_bytes(const void *p, double (&v)[4]) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

struct Integrals {
    double norm, I, Q;   // sum c_i f_i, sum c_i f_i sum_m W_m F, sum c_i f_i sum_m W_m G
};

// Adds w (F, G)(L) of one node per lane to the lanes' partial sums.  The rows
// lie anywhere in a table of a megabyte, so a lane reading its own row would
// touch 32 cache lines with every load (8 loads: 256 L1 wavefronts, which
// bound the kernel at 92 % of the L1 pipe, 24 ms for 2.46M cells); instead four
// lanes read a row together (one line, 32 bytes each), each multiplying the
// coefficients of its two degrees by the node's w z^degree from shared memory,
// and the sum over the degrees falls to the reduction that sums the nodes:
// 13.7 ms with eight lanes and 16 bytes.  The wide loads and paired powers
// halve the exchange's instructions: 30,011 Hybrid frames 106.6 -> 100.1 us (92.9
// with lane_reads).
// A node whose smallest x (the pitch with the largest sin) already lies in
// the table's far tail adds terms below kTailValue times the pitch weights
// (< 1e-270): nothing a cell that emits can resolve.  Skipping it leaves such
// cells unchanged to the last bit (one that does not emit at all gets 0
// instead of a sum of those terms).
__device__ __forceinline__ void add_nodes(const SumTable &T, const PieceSmem &S, NodeSmem &X, double lx_tail,
                                          double L, double w, Integrals &acc) {
    const int lane = threadIdx.x & 31;
    const bool live = w != 0.0 && __dsub_rn(L, T.shift_max) < lx_tail;
    if (!__any_sync(0xffffffffu, live)) return;
    double z = 0.0, p = 0.0;
    int row = 0;
    if (live) {
        row = sum_row(T, S, L, z);
        p = w;
    }
    X.row[4 * (lane & 7) + (lane >> 3)] = row;
    const double zz = z * z;
    double p1 = p * z;
#pragma unroll
    for (int q = 0; q < 4; ++q, p *= zz, p1 *= zz) X.pow[4 * lane + (q ^ ((lane >> 1) & 3))] = make_double2(p, p1);
    __syncwarp();
    const int q = lane & 3, g = lane >> 2;  // rows g, g + 8, g + 16, g + 24; degrees 2 q and 2 q + 1
    const int4 four = *reinterpret_cast<const int4 *>(X.row + 4 * g);
    const int rows[4] = {four.x, four.y, four.z, four.w};
    const double2 *power = X.pow + 4 * g + (q ^ ((g >> 1) & 3));
    const double2 *coefficient = T.rows + 2 * q;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double2 v = power[32 * j];
        double c[4];
        load_32_bytes(coefficient + 8 * rows[j], c);
        acc.I = fma(v.x, c[0], acc.I);
        acc.Q = fma(v.x, c[1], acc.Q);
        acc.I = fma(v.y, c[2], acc.I);
        acc.Q = fma(v.y, c[3], acc.Q);
    }
    __syncwarp();
}

// The thermal grid gamma = 1 + geomspace(1e-5, g1, n) of one frame.
struct ThermalGrid {
    double g1, inv_te, lr, r32, q, q0, q1;  // log ratio, ratio^-32, c_i / x_i inside and at the two ends
    double tail;                            // log x from which no node is looked up
};
// Besides the table's far tail, the nodes below gamma_r = 1 + 2 theta_e, next
// to the weights' maximum, end where x passes x_r + 64: each adds less than
// exp(-64) (1 + x)^(1/2) of node r's term, 4,096 of them below 1e-22 of the sum.
__device__ __forceinline__ ThermalGrid thermal_grid(double theta_e, int n, double base, double shift_max,
                                                    double lx_tail) {
    ThermalGrid g;
    g.g1 = fmax(10.0, 1.0 + 45.0 * theta_e) - 1.0;
    g.inv_te = 1.0 / fmax(theta_e, 1.0e-12);
    g.lr = (log(g.g1) - log(1.0e-5)) / (double)(n - 1);
    const double up = expm1(g.lr), down = -expm1(-g.lr);  // r - 1, 1 - 1/r
    g.r32 = exp(-32.0 * g.lr);
    g.q = 0.5 * (up + down);
    g.q0 = 0.5 * up;
    g.q1 = 0.5 * down;
    g.tail = lx_tail;
    if (theta_e >= 0.02) {  // colder: the weights themselves underflow towards r
        const double x_r = exp(base - shift_max - 2.0 * log(1.0 + 2.0 * theta_e));
        if (x_r + 64.0 < 600.0) g.tail = fmin(lx_tail, log(x_r + 64.0));
    }
    return g;
}

// The pitch-averaged trapezoid integrals of synchrotron.py:207-237 of the
// thermal distribution f = gamma^2 beta exp(-gamma / theta_e), split over the
// warp's lanes; every lane passes the same frame.  The nodes run from the top
// of the grid down, x by the grid's ratio, so the nodes that emit are a few
// multiplications from the exact end point; L rises on the way, and the chunk
// whose first node lies in the table's far tail ends the lookups.
__device__ __forceinline__ Integrals thermal_integrals(const Model &M, const PieceSmem &S, NodeSmem &X,
                                                       const ThermalGrid &g, double base, int lane) {
    const int n = M.th.gamma_n;
    Integrals acc = {0.0, 0.0, 0.0};
    double x = g.g1 * exp(-g.lr * (double)lane);
    bool tail = false;
    for (int top = n - 1; top >= 0; top -= 32, x *= g.r32) {
        const int i = top - lane;
        const double gamma = 1.0 + x;
        const double c = x * (i == n - 1 ? g.q1 : (i == 0 ? g.q0 : g.q));
        const double w = i >= 0 ? c * (gamma * sqrt(x * (x + 2.0)) * exp(-gamma * g.inv_te)) : 0.0;
        acc.norm += w;
        if (!tail) {
            const double L = fma(-2.0, log(gamma), base);
            add_nodes(M.tth, S, X, g.tail, L, w, acc);
            tail = __all_sync(0xffffffffu, !(__dsub_rn(L, M.tth.shift_max) < g.tail));
        }
    }
    acc.norm = warp_sum(acc.norm);
    acc.I = warp_sum(acc.I);
    acc.Q = warp_sum(acc.Q);
    return acc;
}

// The groups of the power law gamma^-p, whose nodes do not depend on the frame.
__device__ __forceinline__ Integrals powerlaw_integrals(const Model &M, const PieceSmem &S, NodeSmem &X,
                                                        double base, int lane) {
    Integrals acc = {0.0, 0.0, 0.0};
    for (int top = 0; top < M.nt_groups; top += 32) {
        const int i = top + lane;
        const double2 nd = i < M.nt_groups ? __ldg(M.nt_nodes + i) : make_double2(0.0, 0.0);
        add_nodes(M.tnt, S, X, M.lx_tail, base - nd.y, nd.x, acc);
    }
    acc.I = warp_sum(acc.I);
    acc.Q = warp_sum(acc.Q);
    return acc;
}

// Its ungrouped nodes (the two ends' trapezoid weights, a remainder), one
// frame per lane.
__device__ __forceinline__ void powerlaw_single(const Model &M, const PieceSmem &S, double base, Integrals &acc) {
    const SumTable &T = M.tnt1;
    for (int i = 0; i < M.nt_single; ++i) {
        const double2 nd = __ldg(M.nt_nodes + M.nt_groups + i);
        const double L = base - nd.y;
        if (!(nd.x != 0.0 && __dsub_rn(L, T.shift_max) < M.lx_tail)) continue;
        double z;
        const double2 *row = T.rows + 8 * sum_row(T, S, L, z);
        double2 v = __ldg(row + 7);
#pragma unroll
        for (int d = 6; d >= 0; --d) {
            const double2 c = __ldg(row + d);
            v = make_double2(fma(v.x, z, c.x), fma(v.y, z, c.y));
        }
        acc.I = fma(nd.x, v.x, acc.I);
        acc.Q = fma(nd.x, v.y, acc.Q);
    }
}

// synchrotron.py:175-182
__device__ __forceinline__ double planck_nu(double nu, double theta_e) {
    const double T = theta_e * kMe * kC * kC / kKb;
    const double x = kH * nu / fmax(kKb * T, 1.0e-300);
    if (x < 1.0e-3) return 2.0 * nu * nu * kKb * T / (kC * kC);
    return 2.0 * kH * nu * nu * nu / (kC * kC) / fmax(expm1(fmin(x, 700.0)), 1.0e-300);
}

// PolarizedCoefficients.rotated (synchrotron.py:67-77) of
// [jI, jQ, 0, 0, aI, aQ, 0, 0, rV, rQ, 0], added into out.
__device__ __forceinline__ void add_rotated(double *out, double jI, double jQ, double aI, double aQ, double rV,
                                            double rQ, double chi) {
    const double c = cos(2.0 * chi), s = sin(2.0 * chi);
    out[0] += jI;
    out[1] += jQ * c - 0.0 * s;
    out[2] += jQ * s + 0.0 * c;
    out[3] += 0.0;
    out[4] += aI;
    out[5] += aQ * c - 0.0 * s;
    out[6] += aQ * s + 0.0 * c;
    out[7] += 0.0;
    out[8] += rV;
    out[9] += rQ * c - 0.0 * s;
    out[10] += rQ * s + 0.0 * c;
}


// A pointer to a kernel parameter for reads that differ from lane to lane: plain
// loads through its generic address.  Left to the parameters' constant bank, a
// warp's read of 32 addresses is 32 reads: every block's copy of its tables took
// about 7 us (30,011 frames 99.5 -> 92.9 us, their tables 34.9 -> 26.7).
template <typename T>
__device__ __forceinline__ const T *lane_reads(const T *p) {
    asm volatile("" : "+l"(p));
    return p;
}

// Block-cooperative copy of the interval searches into shared memory.
__device__ __forceinline__ void load_pieces(PieceSmem &S, const SumTable &table) {
    const SumTable &T = *lane_reads(&table);
    for (int i = threadIdx.x; i < kMaxCells; i += blockDim.x) {
        S.cell[i] = T.cell[i];
        if (i <= kMaxPieces) S.edge[i] = i < T.pieces ? T.edge[i] : INFINITY;
        if (i < kMaxPieces) {
            S.width[i] = i < T.pieces ? T.edge[i + 1] - T.edge[i] : 0.0;
            S.inv_width[i] = i < T.pieces ? 1.0f / (float)(T.edge[i + 1] - T.edge[i]) : 0.0f;
        }
        if (i < kBins) S.first[i] = T.first[i];
    }
}
__device__ __forceinline__ void load_table(TableSmem &S, const Model &M) {
    load_pieces(S.th, M.tth);
    load_pieces(S.nt, M.tnt);
    load_pieces(S.nt1, M.tnt1);
}

// One local plasma frame (synchrotron.py:28-44): n_e [cm^-3], Theta_e (already
// floored), B [G], cos of the pitch to the line of sight, EVPA chi, at
// frequency nu.
struct Frame {
    double n_e, te, b, cos_los, chi, nu;
};

// The 11 coefficients of the model (synchrotron.py:248-325) for up to 32
// frames, one per lane (lane < count).  Warp-collective; each lane gets its
// frame's.  For one model and form of its tables, a frame's result does not depend
// on its lane or on the others.
__device__ __forceinline__ void coefficients(TableSmem &S, const Model &M, const Frame &f, int count,
                                             double out[11]) {
    constexpr unsigned kWarp = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    NodeSmem &X = S.node[threadIdx.x >> 5];
#pragma unroll
    for (int k = 0; k < 11; ++k) out[k] = 0.0;
    const bool emits = lane < count && f.n_e > 0.0 && f.b > 0.0 && f.nu > 0.0;
    const unsigned todo = __ballot_sync(kWarp, emits);
    if (todo == 0) return;
    const double nu_B = kE * f.b / (2.0 * kPiD * kMe * kC);
    const double base = emits ? log(f.nu) - log(1.5 * nu_B) : 0.0;
    Integrals th = {0.0, 0.0, 0.0}, nt = {0.0, 0.0, 0.0};
    if (M.th.on) {
        const ThermalGrid mine = thermal_grid(emits ? f.te : 1.0, M.th.gamma_n, base, M.tth.shift_max, M.lx_tail);
        for (unsigned left = todo; left; left &= left - 1) {
            const int src = __ffs(left) - 1;
            ThermalGrid g;
            g.g1 = __shfl_sync(kWarp, mine.g1, src);
            g.inv_te = __shfl_sync(kWarp, mine.inv_te, src);
            g.lr = __shfl_sync(kWarp, mine.lr, src);
            g.r32 = __shfl_sync(kWarp, mine.r32, src);
            g.q = __shfl_sync(kWarp, mine.q, src);
            g.q0 = __shfl_sync(kWarp, mine.q0, src);
            g.q1 = __shfl_sync(kWarp, mine.q1, src);
            g.tail = __shfl_sync(kWarp, mine.tail, src);
            const Integrals r = thermal_integrals(M, S.th, X, g, __shfl_sync(kWarp, base, src), lane);
            if (lane == src) th = r;
        }
    }
    if (M.nt.on && M.nt.fraction > 0.0) {
        for (unsigned left = todo; left; left &= left - 1) {
            const int src = __ffs(left) - 1;
            const Integrals r = powerlaw_integrals(M, S.nt, X, __shfl_sync(kWarp, base, src), lane);
            if (lane == src) nt = r;
        }
        if (emits) powerlaw_single(M, S.nt1, base, nt);
        nt.norm = M.nt_norm ? __ldg(M.nt_norm) : 0.0;
    }
    if (!emits) return;
    const double n_e = f.n_e, te = f.te, b = f.b, nu = f.nu;
    const double b_perp = fabs(b) * sqrt(fmax(0.0, 1.0 - f.cos_los * f.cos_los));  // synchrotron.py:37-39
    const double b_par = b * f.cos_los;                                            // synchrotron.py:41-43
    const double K3 = kE * kE * kE / (kPiD * kMe * kMe * kC * kC);
    const double K4 = kE * kE * kE * kE / (4.0 * kPiD * kPiD * kMe * kMe * kMe * kC * kC * kC);
    if (M.th.on) {  // synchrotron.py:248-275
        const double inv = th.norm > 0.0 ? 1.0 / th.norm : 1.0;
        const double jI = n_e * (b * th.I * inv) / (4.0 * kPiD);
        const double jQ = n_e * (b * th.Q * inv) / (4.0 * kPiD);
        const double Bnu = planck_nu(nu, te);
        const double aI = jI / fmax(Bnu, 1.0e-300), aQ = jQ / fmax(Bnu, 1.0e-300);
        const double rel_supp = fmax(1.0 / (te * te + 1.0), 1.0e-8);
        const double rV = M.th.rotation_scale * K3 * (n_e * b_par / fmax(nu * nu, 1.0e-300) * rel_supp);
        const double rQ = M.th.conversion_scale * K4 *
                          (n_e * b_perp * b_perp / fmax(nu * nu * nu, 1.0e-300) * fmax(te, 1.0e-8));
        add_rotated(out, fmax(jI, 0.0), fmax(jQ, 0.0), fmax(aI, 0.0), fmax(aQ, 0.0), rV, rQ, f.chi);
    }
    if (M.nt.on && M.nt.fraction > 0.0) {  // synchrotron.py:290-311
        const Component &C = M.nt;
        const double inv = 1.0 / fmax(nt.norm, 1.0e-300);
        const double n_s = n_e * C.fraction;
        const double jI = n_s * (b * nt.I * inv) / (4.0 * kPiD);
        double jQ = n_s * (b * nt.Q * inv) / (4.0 * kPiD);
        const double cg = fmax(C.gamma_min, sqrt(fmax(nu / fmax(4.2e6 * b_perp, 1.0e-300), 1.0)));
        const double energy = cg * kMe * kC * kC;
        const double aI = C.absorption_scale * jI / fmax(energy * nu * nu / (kC * kC), 1.0e-300);
        const double pol = fmin((C.p + 1.0) / (C.p + 7.0 / 3.0), 0.85);
        jQ = fmin(jQ, pol * jI);
        const double aQ = fmin(aI * pol, aI);
        const double rV = C.faraday_scale * K3 *
                          (n_s * b_par / fmax(nu * nu, 1.0e-300) / fmax(C.gamma_min * C.gamma_min, 1.0));
        const double rQ = C.faraday_scale * K4 *
                          (n_s * b_perp * b_perp / fmax(nu * nu * nu, 1.0e-300) *
                           log(fmax(C.gamma_max / C.gamma_min, 1.0)));
        add_rotated(out, fmax(jI, 0.0), fmax(jQ, 0.0), fmax(aI, 0.0), fmax(aQ, 0.0), rV, rQ, f.chi);
    }
}

// The tables' memory: the caller's (p, bytes), or with p NULL a stream-ordered
// allocation, freed on its stream after the owner's last kernel.
struct Scratch {
    void *p = nullptr;
    int64_t bytes = 0;
    bool owned = false;
    cudaStream_t stream = nullptr;
    Scratch(void *p_, int64_t bytes_) : p(p_), bytes(bytes_) {}
    Scratch(const Scratch &) = delete;
    ~Scratch() {
        if (owned) stream_free(p, stream);
    }
};

// Host: the device model for a C model, with its tables built on `stream` in
// `tables`, which outlives the caller's kernels.  grouped: the power law's
// nodes in groups where their sum fits (the same integrals to rounding, 2e-15
// over 8,191 frames; calls whose results should agree in every bit choose alike).
int build_model(const bhn_synchrotron_model *m, bool grouped, Model &out, Scratch &tables, cudaStream_t stream);

}  // namespace synch
}  // namespace bhn
