// bhn_sampler.cuh -- the plugin sampler (float64, bit-exact with the
// reference): sample_brick_trilinear and sample_and_step_stokes
// (native/core/src/lib.rs:171-208, 281-366 / native_kernels.py:137-186, 325-407).
// Included by bhn_api.cu.
//
// A warp takes 32 points in three phases:
//   1. a lane per point: the point's cell and weights (into shared memory);
//   2. a lane per (point, channel), 11 consecutive lanes a point: the eight
//      corners' channel and the reference's seven lerps.  A corner's 11
//      channels are 88 contiguous bytes, so a warp's load touches about three
//      points' cells, 4 cache lines or so; with a lane per point every one of
//      the 88 loads touched 32;
//   3. a lane per point again: the Stokes step on the 11 values from shared memory.
#pragma once

#include "bhn_exact.cuh"

namespace bhn {

constexpr int kSampleThreads = 1024, kSampleBlocks = 1, kCornerUnroll = 2;  // threads a block, blocks an SM
constexpr int kGridSmem = 4096;  // knots of the three axes kept in shared memory (32 KB at most); larger grids are read in place

struct SamplePoints {
    const double *coeffs, *rg, *tg, *pg, *pts, *initial;
    int nr, nt, np, broadcast, policy;
    int per_warp;                  // input order: points a warp takes at a time (32 in cell order)
    int64_t n;
    double ds;
    double *out;
    const uint32_t *keys, *order;  // cell order: sorted cell keys and point indices (NULL: input order)
    uint32_t invalid_key;
    uint32_t *bad_points;          // optional: += points with a non-finite coordinate
};

// The three axes' knots: shared memory (grid_smem bytes, dynamic) when they fit.
inline int grid_smem(int64_t nr, int64_t nt, int64_t np) {
    return nr + nt + np > kGridSmem ? 0 : (int)(8 * (nr + nt + np));
}
struct Axes {
    const double *r, *t, *p;
};
__device__ __forceinline__ Axes load_axes(double *buf, const double *rg, int nr, const double *tg, int nt,
                                          const double *pg, int np) {
    if (nr + nt + np > kGridSmem) return {rg, tg, pg};
    for (int i = threadIdx.x; i < nr; i += blockDim.x) buf[i] = rg[i];
    for (int i = threadIdx.x; i < nt; i += blockDim.x) buf[nr + i] = tg[i];
    for (int i = threadIdx.x; i < np; i += blockDim.x) buf[nr + nt + i] = pg[i];
    __syncthreads();
    return {buf, buf + nr, buf + nr + nt};
}

// The r or theta cell of x (lib.rs:75-87), false outside the axis.
__device__ __forceinline__ bool cell_linear(const double *g, int n, double x, int &i) {
    if (x < g[0] || x > g[n - 1]) return false;
    i = x == g[n - 1] ? n - 2 : max(0, min(search_right(g, 0, n, x) - 1, n - 2));
    return true;
}
// Its weight.
__device__ __forceinline__ double weight_linear(const double *g, int n, double x, int i) {
    if (x == g[n - 1]) return 1.0;
    double den = sub(g[i + 1], g[i]);
    if (den < 1.0e-300) den = 1.0e-300;
    return sub(x, g[i]) / den;
}
// The phi cell of the wrapped p (lib.rs:93-106).
__device__ __forceinline__ int cell_phi(const double *g, int n, double p) {
    const int i = search_right(g, 0, n, p) - 1;
    return i < 0 ? n - 1 : i;
}

// The axes' first-guess parameters for the key kernel: load_axis_hints' rule with
// a block per axis.  An axis of more than kHintKnots knots is searched instead:
// its classification, two passes with a logarithm per knot, would take longer
// than the searches of the smallest ordered set save.  A call of 300,000 points
// through a geometric axis of 2^12, 2^16 and 2^20 knots: 148, 191 and 372 us (one
// warp for all axes of any length: 181, 964 and 13,864).  (The warp's form as a
// call of a shared one cost the brick renderer 40 us an image.)
constexpr int kHintThreads = 1024, kHintKnots = 1 << 14;
__global__ void __launch_bounds__(kHintThreads) axis_hints_kernel(const double *rg, int nr, const double *tg, int nt,
                                                                  const double *pg, int np, AxisHints *out) {
    const int a = blockIdx.x, n = a == 0 ? nr : (a == 1 ? nt : np);
    const double *g = a == 0 ? rg : (a == 1 ? tg : pg);
    __shared__ double part[kHintThreads / 32];
    auto block_max = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();  // the previous call's reads
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
        __syncthreads();
        v = part[threadIdx.x & 31];
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    };
    int kind = kSearch;
    double off = 0.0, inv = 0.0;
    if (n <= kHintKnots) {
        const double d = (g[n - 1] - g[0]) / (n - 1);
        double dev = 0.0;
        for (int k = threadIdx.x; k < n; k += kHintThreads) dev = fmax(dev, fabs(g[k] - (g[0] + k * d)));
        if (block_max(dev) <= 0.25 * d) {
            kind = kUniform;
            inv = 1.0 / d;
            off = g[0] * inv;
        } else if (a < 2 && g[0] > 0.0) {
            const double dl = log(g[n - 1] / g[0]) / (n - 1);
            double devl = 0.0;
            for (int k = threadIdx.x; k < n; k += kHintThreads) devl = fmax(devl, fabs(log(g[k] / g[0]) - k * dl));
            if (block_max(devl) <= 0.25 * dl) {
                kind = kGeometric;
                inv = 1.0 / dl;
                off = log(g[0]) * inv;
            }
        }
    }
    if (threadIdx.x == 0) {
        out->kind[a] = isfinite(off) && isfinite(inv) ? kind : kSearch;
        out->off[a] = off;
        out->inv[a] = inv;
        out->g0[a] = g[0];
        out->gn[a] = g[n - 1];
    }
}

// The cell (r0, theta0, phi0) a point samples from, as one index; points the
// sampler rejects (outside the nonperiodic r/theta range) sort last.  The cells
// come from the axes' closed-form guess and its exact fix-up: a binary search
// makes 24 dependent reads whose lanes hit the shared-memory banks at random,
// which bound the kernel (12.6M points: 314 us with it, the same from global
// memory; 127 now).
__global__ void __launch_bounds__(256) cell_key_kernel(const double *__restrict__ rg, int nr,
                                                       const double *__restrict__ tg, int nt,
                                                       const double *__restrict__ pg, int np,
                                                       const double *__restrict__ pts, int64_t n,
                                                       uint32_t invalid_key, const AxisHints *hints,
                                                       uint32_t *__restrict__ keys, uint32_t *__restrict__ idx,
                                                       uint32_t *bad_points) {
    extern __shared__ double buf[];
    const Axes A = load_axes(buf, rg, nr, tg, nt, pg, np);
    const AxisHints h = *hints;
    uint32_t bad = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double r = pts[3 * i], th = pts[3 * i + 1], ph = pts[3 * i + 2];
        bad += !(isfinite(r) && isfinite(th) && isfinite(ph));
        uint32_t key = invalid_key;
        if (!(r < h.g0[0] || r > h.gn[0]) && !(th < h.g0[1] || th > h.gn[1])) {
            const int r0 = locate_linear(A.r, nr, r, h.kind[0], h.off[0], h.inv[0]);
            const int t0 = locate_linear(A.t, nt, th, h.kind[1], h.off[1], h.inv[1]);
            const int p0 = locate_phi(A.p, np, wrap_phi(ph, h.g0[2]), h.kind[2], h.off[2], h.inv[2]);
            key = (uint32_t)(((int64_t)r0 * nt + t0) * np + p0);
        }
        keys[i] = key;
        idx[i] = (uint32_t)i;
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && bad && bad_points) atomicAdd(bad_points, bad);
}

// STEP: sample and take one Stokes RK2 step per point; else write the samples.
// ORDERED: points in cell order, the cell decoded from the sorted key; a
// point's coordinates then lie anywhere, so the next batch's are loaded before
// this batch's corners.
// 12.6M points in cell order through a 738 MB brick: 917 us (1,590 with a lane
// per point), 100,003 through 11 MB in input order: 13 us (31).  Two thirds of
// it is the corners (L1 wavefronts 75 % busy, FP64 26 %: the reference's
// separately rounded lerps), the rest the scattered reads and writes of the
// cell order, where every lane's access is a wavefront of its own: a point's
// 24 bytes in two loads and its 32 in one store, where the arrays' alignment
// allows, instead of three and two (985 us; the loads alone give 992, the store
// alone 941).  One 1,024-thread block per SM on consecutive points keeps
// the theta rows that neighbouring points share in L1: 1,068 us at 128-thread
// blocks, 1,026 at 256, 1,008 at 512; a contiguous share of the points per
// block instead 1,211 (every SM then reads its own r slabs from memory); all
// eleven channel steps unrolled 1,407 (122 registers, half the warps).  Corners
// kept in registers from point to point of a cell or its phi neighbour save
// two thirds of the corner loads but wait for them in turn (22 lanes on runs of
// 16 points: 1,056; pairs of points: 961); the next batch's corners prefetched
// into L2: 1,003.
struct __align__(16) Place {  // a point's cells (r0, theta0, phi0) and (r0, theta0, phi1) and its weights
    double wr, wt, wp;
    uint32_t cell0, cell1;
};
struct WarpPoints {
    Place place[32];
    double value[32 * 11];
};
constexpr int kSampleSmem = (int)sizeof(WarpPoints) * (kSampleThreads / 32) + 8 * kGridSmem;  // the most a launch takes
// Four doubles in one 32-byte store (32-byte aligned).
__device__ __forceinline__ void store_32_bytes(double *p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]) : "memory");
}

template <bool STEP, bool ORDERED>
__global__ void __launch_bounds__(kSampleThreads, kSampleBlocks) sample_points_kernel(const SamplePoints P) {
    extern __shared__ __align__(16) unsigned char smem[];
    WarpPoints &W = reinterpret_cast<WarpPoints *>(smem)[threadIdx.x >> 5];
    const Axes A = load_axes(reinterpret_cast<double *>(smem + sizeof(WarpPoints) * (blockDim.x >> 5)), P.rg, P.nr, P.tg,
                             P.nt, P.pg, P.np);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ct = (uint32_t)P.np, cr = (uint32_t)(P.np * P.nt);  // cells to the next theta, r
    uint32_t bad = 0;
    const int group = ORDERED ? 32 : P.per_warp;
    const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * group;
    int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + warp) * group;
    uint32_t next_i = 0, next_key = P.invalid_key;
    double nr_ = 0.0, nt_ = 0.0, np_ = 0.0;
    const bool aligned16 = (reinterpret_cast<uintptr_t>(P.pts) & 15) == 0;  // else three 8-byte reads
    const bool aligned32 = (reinterpret_cast<uintptr_t>(P.out) & 31) == 0;  // else two 16-byte writes
    auto fetch = [&](int64_t k) {  // point k of the order (k < n) into next_*
        if (k >= P.n || (!ORDERED && lane >= group)) return;
        int64_t i = k;
        if (ORDERED) {
            next_i = __ldcs(P.order + k);
            next_key = __ldcs(P.keys + k);
            i = next_i;
        }
        if (ORDERED && aligned16) {  // an even point starts on 16 bytes, an odd one 8 before
            const bool odd = i & 1;
            const double *q = P.pts + 3 * i;
            const double2 two = *reinterpret_cast<const double2 *>(q + odd);
            const double one = q[odd ? 0 : 2];
            nr_ = odd ? one : two.x;
            nt_ = odd ? two.x : two.y;
            np_ = odd ? two.y : one;
        } else {
            nr_ = P.pts[3 * i];
            nt_ = P.pts[3 * i + 1];
            np_ = P.pts[3 * i + 2];
        }
    };
    fetch(base + lane);
    for (; base < P.n; base += step) {
        const int64_t k = base + lane, i = ORDERED ? (int64_t)next_i : k;
        const double r = nr_, th = nt_, ph = np_;
        bool inside = false;
        int r0 = 0, t0 = 0, p0 = 0;
        double wr = 0.0, wt = 0.0, wp = 0.0;
        const bool mine = k < P.n && (ORDERED || lane < group);
        if (mine) {
            const double p = wrap_phi(ph, A.p[0]);
            if (ORDERED) {
                inside = next_key != P.invalid_key;
                if (inside) {
                    const uint32_t row = next_key / ct;
                    p0 = (int)(next_key - row * ct);
                    r0 = (int)(row / (uint32_t)P.nt);
                    t0 = (int)(row - (uint32_t)r0 * (uint32_t)P.nt);
                }
            } else {
                bad += !(isfinite(r) && isfinite(th) && isfinite(ph));
                inside = cell_linear(A.r, P.nr, r, r0) && cell_linear(A.t, P.nt, th, t0);
                if (inside) p0 = cell_phi(A.p, P.np, p);
            }
            if (inside) {
                wr = weight_linear(A.r, P.nr, r, r0);
                wt = weight_linear(A.t, P.nt, th, t0);
                const double lo = A.p[p0], hi = p0 + 1 < P.np ? A.p[p0 + 1] : add(A.p[0], kTwoPi);
                const double pp = p >= lo ? p : add(p, kTwoPi);
                double den = sub(hi, lo);
                if (den < 1.0e-300) den = 1.0e-300;
                wp = sub(pp, lo) / den;
            }
        }
        const uint32_t cell = inside ? ((uint32_t)r0 * (uint32_t)P.nt + (uint32_t)t0) * ct + (uint32_t)p0 : 0u;
        W.place[lane] = {wr, wt, wp, cell, p0 + 1 < P.np ? cell + 1 : cell - (uint32_t)p0};
        const unsigned in_mask = __ballot_sync(0xffffffffu, inside);
        fetch(k + step);
        __syncwarp();
#pragma unroll kCornerUnroll
        for (int j = 0; j < (ORDERED ? 11 : (11 * group + 31) >> 5); ++j) {
            const int item = lane + 32 * j, pt = item / 11, ch = item - 11 * pt;
            if (in_mask >> pt & 1) {
                const Place w = W.place[pt];
                const double *q = P.coeffs + ch;
                auto at = [&](uint32_t c) { return __ldg(q + 11 * (int64_t)c); };
                const double v000 = at(w.cell0), v001 = at(w.cell1), v010 = at(w.cell0 + ct), v011 = at(w.cell1 + ct);
                const double v100 = at(w.cell0 + cr), v101 = at(w.cell1 + cr), v110 = at(w.cell0 + cr + ct),
                             v111 = at(w.cell1 + cr + ct);
                const double a = w.wr, b = w.wt, c = w.wp;
                const double oa = sub(1.0, a), ob = sub(1.0, b), oc = sub(1.0, c);
                // native_kernels.py:180-186: phi lerps, then theta, then r
                const double c00 = add(mul(oc, v000), mul(c, v001)), c01 = add(mul(oc, v010), mul(c, v011));
                const double c10 = add(mul(oc, v100), mul(c, v101)), c11 = add(mul(oc, v110), mul(c, v111));
                const double cc0 = add(mul(ob, c00), mul(b, c01)), cc1 = add(mul(ob, c10), mul(b, c11));
                W.value[item] = add(mul(oa, cc0), mul(a, cc1));
            } else {
                W.value[item] = __longlong_as_double(0x7ff8000000000000ULL);
            }
        }
        __syncwarp();
        if (STEP) {
            if (mine) {
                const double *s0 = P.initial + (P.broadcast ? 0 : 4 * i);
                double s[4] = {s0[0], s0[1], s0[2], s0[3]};
                if (inside) {
                    double c[11];
#pragma unroll
                    for (int ch = 0; ch < 11; ++ch) c[ch] = W.value[11 * lane + ch];
                    stokes_step_rk2_exact(s, c, P.ds);
                } else if (P.policy == BHN_POLICY_ZERO) {
                    s[0] = s[1] = s[2] = s[3] = 0.0;
                } else if (P.policy != BHN_POLICY_INITIAL) {
                    s[0] = s[1] = s[2] = s[3] = __longlong_as_double(0x7ff8000000000000ULL);
                }
                if (aligned32) {
                    store_32_bytes(P.out + 4 * i, s);
                } else {
                    reinterpret_cast<double2 *>(P.out + 4 * i)[0] = make_double2(s[0], s[1]);
                    reinterpret_cast<double2 *>(P.out + 4 * i)[1] = make_double2(s[2], s[3]);
                }
            }
        } else {
            if (ORDERED) W.place[lane].cell0 = (uint32_t)i;
            __syncwarp();
#pragma unroll 1
            for (int j = 0; j < (ORDERED ? 11 : (11 * group + 31) >> 5); ++j) {
                const int item = lane + 32 * j, pt = item / 11;
                const int64_t o = ORDERED ? (int64_t)W.place[pt].cell0 : base + pt;
                if (base + pt < P.n && (ORDERED || pt < group)) P.out[11 * o + item - 11 * pt] = W.value[item];
            }
        }
        __syncwarp();
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0 && bad && P.bad_points) atomicAdd(P.bad_points, bad);
}

// ------------------------------------------------------------------- checks
// Non-finite values, and for an axis non-increasing neighbours, of several
// arrays in one launch: a block takes one tile of one array.  Streams at the
// memory's rate on a large brick; on small calls one launch and one read-back
// replace one of each per array (~25 us apiece).
constexpr int kCheckArrays = 5, kCheckTile = 8192;
struct CheckArrays {
    const double *v[kCheckArrays];
    int64_t n[kCheckArrays], first[kCheckArrays + 1];  // elements; first block of the array
    int increasing[kCheckArrays];
    uint32_t *counts;  // [2 a] non-finite, [2 a + 1] non-increasing
};
__global__ void __launch_bounds__(256) check_arrays_kernel(const CheckArrays C) {
    int a = 0;
    while (a + 1 < kCheckArrays && (int64_t)blockIdx.x >= C.first[a + 1]) ++a;
    const double *v = C.v[a];
    const int64_t lo = ((int64_t)blockIdx.x - C.first[a]) * kCheckTile, hi = min(C.n[a], lo + kCheckTile);
    uint32_t bad = 0, nonmono = 0;
    if (!C.increasing[a] && (reinterpret_cast<uintptr_t>(v) & 15) == 0 && hi - lo == kCheckTile) {
        const double2 *w = reinterpret_cast<const double2 *>(v + lo);
#pragma unroll 8
        for (int i = threadIdx.x; i < kCheckTile / 2; i += 256) {
            const double2 x = w[i];
            bad += !isfinite(x.x) + !isfinite(x.y);
        }
    } else {
        for (int64_t i = lo + threadIdx.x; i < hi; i += 256) {
            const double x = v[i];
            bad += !isfinite(x);
            if (C.increasing[a] && i + 1 < C.n[a]) nonmono += !(v[i + 1] > x);
        }
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    nonmono = __reduce_add_sync(0xffffffffu, nonmono);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicAdd(C.counts + 2 * a, bad);
        if (nonmono) atomicAdd(C.counts + 2 * a + 1, nonmono);
    }
}

}  // namespace bhn
