// bhn_far.cuh -- RK2 steps outside the coefficient brick.
// Included by bhn_render.cu after Tracer32.
//
// A camera at 1000 M spends five of its six steps outside the brick (r > 40 M):
// nothing is sampled there and no stopping rule but the escape radius can
// apply.  far_steps takes those steps in a loop of their own, which drops the
// segment, the brick and termination tests and their constants, with the
// operations and roundings of Tracer32::step.  A step is only committed when
// the states before and after it are plainly outside; any other is left,
// untaken, to the general loop, so the results are the same bits.
// Bound by issue slots like the general loop (82 % busy): about 150 instructions
// a step instead of 240.  1024 x 1024 rays, 4096 steps: 14.43 -> 10.53 ms; 12
// uneven views 12.75 -> 9.54; a camera at 55 M, next to the brick, 1.91 ->
// 1.73.  Measured and not kept: two rays per thread on the paired FP32
// instructions (one issue slot for two operations, but the FP32 pipe takes them
// at the scalar rate; 14.2 ms, and half the warps of a small image); one loop
// per hemisphere (10.6 ms, and rays that cross the equator far out ran their
// warp through both); the loop unrolled twice (no change).

namespace bhn {

// The far steps of a ray.  Inside the loop the pole distance d (from the pole
// nearer at the step's start) is at least 1e-4 at the start and the midpoint, so
// sincos_pole's clamps do nothing; its far half (the midpoint past the equator)
// and a change of hemisphere are rare branches.  sg, oh and ol give d as
// (oh + sg theta_h) + (ol + sg theta_l): theta itself, or pi - theta in the
// south.  Escape radius and step bound are checked to be moderate, so a state
// that passes the tests has finite increments: an infinite dr or momentum
// fails them, and dphi cannot overflow before the momenta do.
__device__ __forceinline__ void far_steps(Tracer32 &t, const StepConst &C) {
    const float a = C.a, a2 = C.a2, dpm = C.dpm, hs = C.hs, hmin = C.hmin, hmax = C.hmax, rp_h = C.rp_h, rp_l = C.rp_l,
                esc = C.esc, far = C.r_far, pt = t.pt, pphi = t.pphi, H0 = t.H0;
    float rh = t.rh, rl = t.rl, th_h = t.th_h, th_l = t.th_l, ph_h = t.ph_h, ph_l = t.ph_l, pr = t.pr, pth = t.pth,
          drift = t.drift;
    const bool south = th_h > kHalfPiF;
    float sg = south ? -1.0f : 1.0f, oh = south ? kPiH : 0.0f, ol = south ? kPiL : 0.0f;
    float d0 = fmaf(sg, th_h, oh) + fmaf(sg, th_l, ol);
    auto plain = [&](float r, float d, float p, float q) {
        return r > far && d >= kPoleIsland && fabsf(p) < kMomentumIsland && fabsf(q) < kMomentumIsland;
    };
    if (!(plain(rh, d0, pr, pth) && d0 <= kHalfPiF && t.tau < C.max_tau && esc < 1.0e30f && hmax < 1.0e6f)) return;
    const int most = max(C.max_steps - t.steps - 1, 0);  // the last step is the general loop's
    int left = most;
    while (left > 0) {
        const float r0 = rh + rl;
        float s, c;
        sincos_quadrant(d0, s, c);
        const float x0 = (rh - rp_h) + (rl - rp_l);
        const float h = fminf(fmaxf(hs * r0, hmin), hmax);
        Deriv32 k1, k2;
        rhs32(r0, x0, s, c * sg, pr, pth, pt, pphi, a, a2, dpm, k1);
        const float hh = 0.5f * h, rm = fmaf(hh, k1.r, r0);
        float x = fmaf(hh * sg, k1.th, d0), cs = sg;
        if (x > kHalfPiF) {  // the midpoint lies past the equator
            x = (kPiH - x) + kPiL;
            cs = -sg;
        }
        sincos_quadrant(x, s, c);
        rhs32(rm, fmaf(hh, k1.r, x0), s, c * cs, fmaf(hh, k1.pr, pr), fmaf(hh, k1.pth, pth), pt, pphi, a, a2, dpm, k2);
        const float dr = __fmul_rn(h, k2.r), dth = __fmul_rn(h, k2.th), dph = __fmul_rn(h, k2.ph);
        const float prn = fmaf(h, k2.pr, pr), pthn = fmaf(h, k2.pth, pth);
        float nrh = rh, nrl = rl, nth_h = th_h, nth_l = th_l, nph_h = ph_h, nph_l = ph_l;
        kahan_add(nrh, nrl, dr);
        kahan_add(nth_h, nth_l, dth);
        kahan_add(nph_h, nph_l, dph);
        float dh = fmaf(sg, nth_h, oh), nd = dh + fmaf(sg, nth_l, ol);
        if (!(dh < kHalfPiF)) {  // the other hemisphere now (2 kHalfPiF = kPiH: dh = kHalfPiF is theta_h's own equator)
            if (dh == kHalfPiF) break;
            sg = -sg;
            oh = kPiH - oh;
            ol = kPiL - ol;
            dh = fmaf(sg, nth_h, oh);
            nd = dh + fmaf(sg, nth_l, ol);
        }
        if (!(plain(nrh, nd, prn, pthn) && rm > far && x >= kPoleIsland && !(nrh > esc && dr > 0.0f))) break;
        drift = fmaxf(drift, fabsf(fabsf(k1.H) - H0));
        if (__float_as_uint(nph_h) >= __float_as_uint(kTwoPiH)) {  // above 2 pi, or negative
            if (nph_h >= kTwoPiH) {
                two_sum_add(nph_h, nph_l, -kTwoPiH);
                nph_l -= kTwoPiL;
            } else if (nph_h < 0.0f) {
                two_sum_add(nph_h, nph_l, kTwoPiH);
                nph_l += kTwoPiL;
            }
        }
        rh = nrh, rl = nrl, th_h = nth_h, th_l = nth_l, ph_h = nph_h, ph_l = nph_l, pr = prn, pth = pthn;
        d0 = nd;
        --left;
    }
    t.rh = rh, t.rl = rl, t.th_h = th_h, t.th_l = th_l, t.ph_h = ph_h, t.ph_l = ph_l, t.pr = pr, t.pth = pth;
    t.drift = drift;
    t.steps += most - left;
}

}  // namespace bhn
