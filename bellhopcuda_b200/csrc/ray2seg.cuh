// 2-D ray step over the packed segment table (1-D profiles of types C, S and
// P with real sound speeds): ray2d.cuh's ray_update2d with the same operands
// and roundings, so that every trajectory, step and reflection decision is the
// same double, arranged for the latency of one ray.
//
// A trace is one dependent chain per ray and the chip waits for its longest
// ray, whatever the fan's size: latency is the bound. Through the general step
// a ray step takes 1,356 instructions, 424 of them FP64 and 194 branches, at
// 6.3 cycles each (one ray per warp), through this one about half. Trace times,
// general -> this step, with the same step and contribution counts: 201 rays
// of a Munk channel 4.9 -> 2.6 ms, 2001 rays 4.4 -> 2.1 ms, 20001 rays of the
// range-dependent workload 12.3 -> 6.8 ms, 24 uneven spline environments 153
// -> 72 ms. What it does:
//  * the profile segment's bounds and coefficients are one 64-byte record
//    (SspSeg), read by 16-byte loads when the ray changes segment;
//  * the profile at the start of a step is the one evaluated at the end of the
//    step before (same position, tangent and segment), or again after a
//    reflection;
//  * the tests for the beam box, both boundaries and the range segments of the
//    boundaries are one test of a rectangle known to be inside all of them
//    (SafeBox). Outside it the tests are made one by one; a step that only
//    crosses a range segment is cut there, one that meets the box or a
//    boundary takes the general routines;
//  * the horizontal gradient and the complex parts, which are zero, are not
//    computed (x - 0, p + 0 and 0 / c add nothing);
//  * divisions are branch-free and share reciprocals (device_math.cuh);
//  * a reflection rewrites the ray state in place after the segment has been
//    handed on, so the common step has one successor and few register copies.
// Calls in place of the inlined general routines were slower on every case
// (20001 rays 8.1 ms, the batch 99 ms), and so was a launch bound of 168 or 128
// registers (8.7 and 9.8 ms): the few hundred spilled bytes lie on the chain.
#pragma once
#include "ray2d.cuh"

namespace bhcb {

// Open rectangle in which no boundary, box or range-segment test of the step
// can hold: |x| and |y| inside the beam box, x inside the current boundary
// segments, y a millimetre below the surface segment's deeper node and above
// the bottom segment's shallower node. The signed distance to a boundary
// line there is below -1e-3 |n.y| <= -5e-5, past the step's INF_STEP (1e-6)
// tolerance and any rounding; steeper lines leave no such rectangle.
struct SafeBox {
    double xlo, xhi, ylo, yhi;
    __device__ __forceinline__ bool holds(double x, double y) const
    {
        return x > xlo && x < xhi && y > ylo && y < yhi;
    }
};

__device__ __forceinline__ BdState load_bdry(const BdryPtDev *bd, int i)
{
    BdState b;
    b.Iseg = i;
    b.lmin = bd[i].x[0];
    b.lmax = bd[i + 1].x[0];
    b.x = mk2(bd[i].x[0], bd[i].x[1]);
    b.n = mk2(bd[i].n[0], bd[i].n[1]);
    return b;
}

// the halfspace get_bdry_seg leaves: the boundary's, or the segment's (long format)
__device__ __forceinline__ HsDev load_hs(const HsDev &base, const BdryPtDev *bd, int i, bool islong)
{
    HsDev h = base;
    if(islong) {
        h.cPr = bd[i].cPr; h.cPi = bd[i].cPi;
        h.cSr = bd[i].cSr; h.cSi = bd[i].cSi;
        h.rho = bd[i].rho;
    }
    return h;
}

// The general routines for the steps that leave the rectangle.
__device__ __forceinline__ double reduce_rare(const EnvDev *e, int it, int ib, int iz, double x, double y, double ux,
                                           double uy, double h, RunCounters *ctr)
{
    StepGeo geo{e};
    int small = 0;
    reduce_step(geo, mk2(x, y), mk2(ux, uy), SegState{0, iz}, load_bdry(e->btop, it), load_bdry(e->bbot, ib), h, small,
                ctr);
    return h;
}
struct Landing {
    double x, y, h;
    int hit;              // 1: surface, 2: bottom
};
__device__ __forceinline__ Landing land_rare(const EnvDev *e, int it, int ib, int iz, double x, double y, double ux,
                                          double uy, double h)
{
    StepGeo geo{e};
    bool tr = false, br = false;
    V2<double> x2;
    step_to_bdry(geo, mk2(x, y), x2, mk2(ux, uy), h, tr, br, SegState{0, iz}, load_bdry(e->btop, it),
                 load_bdry(e->bbot, ib));
    return Landing{x2.x, x2.y, h, tr ? 1 : br ? 2 : 0};
}
// RayUpdate's boundary segments and signs of the distances at p1
struct BdryPos {
    int it, ib, end_top, end_bot;
};
__device__ __forceinline__ BdryPos bdry_rare(const EnvDev *e, int it, int ib, double x, double y, double tx,
                                          RunCounters *ctr)
{
    BdState top = load_bdry(e->btop, it), bot = load_bdry(e->bbot, ib);
    HsDev unused = e->top;
    get_bdry_seg(mk2(x, y), tx, top, e->btop, e->ntop, false, unused, true, false, ctr);
    get_bdry_seg(mk2(x, y), tx, bot, e->bbot, e->nbot, false, unused, false, false, ctr);
    double dt, db;
    distances(mk2(x, y), top, bot, dt, db);
    return BdryPos{top.Iseg, bot.Iseg, dt < 0.0, db < 0.0};
}
// the reflected point p2 of p1, where the profile is o
__device__ __forceinline__ BdryPos reflect_rare(const EnvDev *e, BdryPos b, bool istop, const SSPOut<double> &o,
                                                const RayPt<double> &p1, RayPt<double> &p2, RunCounters *ctr)
{
    const BdryPtDev *bd = istop ? e->btop + b.it : e->bbot + b.ib;
    V2<double> nI, tI;
    if(istop ? e->top_curv : e->bot_curv) {
        const double sss = dot2(sub2(p1.x, mk2(bd[0].x[0], bd[0].x[1])), mk2(bd[0].t[0], bd[0].t[1])) / bd[0].Len;
        nI = mk2((FLTD(1.0) - sss) * bd[0].Noden[0] + sss * bd[1].Noden[0],
                 (FLTD(1.0) - sss) * bd[0].Noden[1] + sss * bd[1].Noden[1]);
        tI = mk2((FLTD(1.0) - sss) * bd[0].Nodet[0] + sss * bd[1].Nodet[0],
                 (FLTD(1.0) - sss) * bd[0].Nodet[1] + sss * bd[1].Nodet[1]);
    } else {
        nI = mk2(bd[0].n[0], bd[0].n[1]);
        tI = mk2(bd[0].t[0], bd[0].t[1]);
    }
    const HsDev hs = istop ? load_hs(e->top, e->btop, b.it, e->top_long) : load_hs(e->bot, e->bbot, b.ib, e->bot_long);
    reflect2d_at(o, p1, p2, hs, istop, tI, nI, bd[0].kappa, *e, ctr);
    double dt, db;
    distances(p2.x, load_bdry(e->btop, b.it), load_bdry(e->bbot, b.ib), dt, db);
    b.end_top = dt < 0.0;
    b.end_bot = db < 0.0;
    return b;
}

// K: the profile type, or SSP_ANY for the one of the environment (kernels whose
// prologues differ by beam type, which would otherwise be compiled three times)
constexpr int SSP_ANY = -1;
template<int K> struct Ray2Seg {
    int kind;
    const EnvDev *e;
    const SspSeg *tab;
    RayPt<double> p0;
    double deltas, hmin;
    // current profile segment
    int iz, izmax;
    double z0, z1, k0, k1, k2, k3;
    // profile at p0 and the reciprocals of c and c^2
    double c, g, czz, csq, rc, rcsq;
    int it, ib;                       // boundary segments
    // the last step's start and end: beyond the surface / the bottom; the end
    // inside the rectangle; the amplitude below the stop threshold
    bool beg_top, beg_bot, end_top, end_bot, inside, low;
    BdryPos pos;
    SafeBox box;
    double lmin, lmax;                // range common to the two boundary segments

    __device__ __forceinline__ void load_seg(int i)
    {
        iz = i;
        const double2 *r = reinterpret_cast<const double2 *>(tab + i);
        const double2 a = r[0], b = r[1];
        z0 = a.x; z1 = a.y; k0 = b.x; k1 = b.y;
        if((K < 0 ? kind : K) != SSP_CLINEAR) {
            const double2 d = r[2];
            k2 = d.x; k3 = d.y;
        }
    }
    // update_seg (src/ssp.hpp:36-51) from the current segment
    __device__ __forceinline__ void find_seg(double y, bool tpos)
    {
        if(y > z0 && y < z1) return;
        for(;;) {
            const bool dn = iz > 0 && (tpos ? y < z0 : y <= z0);
            const bool up = iz < izmax && (tpos ? y >= z1 : y > z1);
            if(!(dn || up)) return;
            load_seg(iz + (up ? 1 : -1));
        }
    }
    // eval_ssp's arithmetic on the segment's coefficients
    __device__ __forceinline__ void eval(double y, double ty, double &c_, double &g_, double &czz_)
    {
        find_seg(y, ty >= 0.0);
        const double h = y - z0;
        const int k = K < 0 ? kind : K;
        if(k == SSP_CLINEAR) {
            c_ = k0 + h * k1;
            g_ = k1;
            czz_ = 0.0;
        } else if(k == SSP_CUBIC) {
            const double half = 0.5, sixth = (double)(1.0f / 6.0f);
            c_ = k0 + h * (k1 + h * (half * k2 + sixth * h * k3));
            g_ = k1 + h * (k2 + h * half * k3);
            czz_ = k2 + h * k3;
        } else {
            c_ = k0 + (k1 + (k2 + k3 * h) * h) * h;
            g_ = k1 + (2.0 * k2 + 3.0 * k3 * h) * h;
            czz_ = 2.0 * k2 + 6.0 * k3 * h;
        }
    }
    // the profile at p's position and tangent, kept for the step that starts there
    __device__ __forceinline__ void eval_here(const RayPt<double> &p)
    {
        eval(p.x.y, p.t.y, c, g, czz);
        csq = c * c;
        rc = rcp_rn(c);
        rcsq = rcp_square(csq, rc);
    }
    __device__ __forceinline__ void set_box()
    {
        const BdryPtDev *t = e->btop + it, *b = e->bbot + ib;
        const double ex = e->box_x, ey = e->box_y;
        lmin = max(t[0].x[0], b[0].x[0]);
        lmax = min(t[1].x[0], b[1].x[0]);
        box.xlo = max(lmin, -ex);
        box.xhi = min(lmax, ex);
        box.ylo = max(max(t[0].x[1], t[1].x[1]) + 1.0e-3, -ey);
        box.yhi = min(min(b[0].x[1], b[1].x[1]) - 1.0e-3, ey);
        if(!(t[0].n[1] < -0.05 && b[0].n[1] > 0.05)) box.ylo = 1.7976931348623157e308;
    }
    __device__ __forceinline__ void init(const RayState2<double> &st, const EnvDev &env)
    {
        e = &env;
        kind = env.ssp_type;
        tab = env.segtab;
        p0 = st.p0;
        deltas = env.deltas;
        hmin = INF_STEP * env.deltas;
        izmax = env.nssp - 2;
        k2 = k3 = 0.0;
        load_seg(st.iSeg.z);
        eval_here(p0);
        it = st.top.Iseg;
        ib = st.bot.Iseg;
        beg_top = st.dBegTop < 0.0;
        beg_bot = st.dBegBot < 0.0;
        low = p0.Amp < FLTD(0.005);
        set_box();
    }
    // Outside the rectangle: whether (x, y) meets the beam box or passes a
    // boundary line by more than -tol (box and topbot of StepGeo)
    __device__ __forceinline__ bool meets(double x, double y, double tol) const
    {
        const BdryPtDev *t = e->btop + it, *b = e->bbot + ib;
        const double wt = t->n[0] * (x - t->x[0]) + t->n[1] * (y - t->x[1]);
        const double wb = b->n[0] * (x - b->x[0]) + b->n[1] * (y - b->x[1]);
        return !(fabs(x) < e->box_x && fabs(y) < e->box_y && wt < tol && wb < tol);
    }
    // reduce_step: the step h along u shortened to the first crossing; za, zb:
    // the depth bounds of the segment at p0. The quotient for the profile node
    // is computed whether or not it is met: a branch costs a warp as much.
    __device__ __forceinline__ double reduce(V2<double> u, double h, double za, double zb, int s0, RunCounters *ctr)
    {
        const double xe = p0.x.x + h * u.x, ye = p0.x.y + h * u.y;
        const bool above = za > ye;
        const double hi = div_rn((above ? za : zb) - p0.x.y, u.y);
        double hn = (above || zb < ye) && fabs(u.y) > DBL_EPS && hi < h ? hi : h;
        if(!box.holds(xe, ye)) {
            if(meets(xe, ye, 0.0)) return reduce_rare(e, it, ib, s0, p0.x.x, p0.x.y, u.x, u.y, h, ctr);
            if(fabs(u.x) > DBL_EPS && (xe < lmin || xe > lmax)) {
                const double hr = div_rn(-(p0.x.x - (xe < lmin ? lmin : lmax)), u.x);
                hn = hr < hn ? hr : hn;
            }
        }
        if(hn < hmin) {
            if(hn < -1e-4) run_warn(ctr, WARN_STEP_NEGATIVE_H);
            hn = hmin;
        }
        return hn;
    }

    // Step (src/step.hpp:654-811) from p0 to p1 with RayUpdate's boundary
    // segments; returns the boundary to reflect at (0: none, 1: surface, 2:
    // bottom)
    __device__ __forceinline__ int step(RayPt<double> &p1, RunCounters *ctr)
    {
        const V2<double> x0 = p0.x, t0 = p0.t;
        const int s0 = iz;
        const double za = z0, zb = z1;
        const double c0 = c, g0 = g, csq0 = csq, rc0 = rc, rcsq0 = rcsq;
        // c-linear: czz is 0 and the paraxial p does not change within the step, but by
        // 0 q, which is not a number once q, here or at half the step, has grown past all
        // numbers (a test for that costs 2 % of the trace, the multiplications nothing)
        const double cnn0 = czz * t0.x * t0.x;
        const V2<double> pq0p = scl2(-cnn0, p0.q), pq0q = scl2(c0, p0.p);
        const V2<double> u0 = scl2(c0, t0);
        double h = reduce(u0, deltas, za, zb, s0, ctr);
        const double halfh = 0.5 * h, h2 = 2.0 * halfh;
        const V2<double> t1 = mk2(t0.x, t0.y - quot_rn(halfh * g0, csq0, rcsq0));
        const V2<double> pm = K == SSP_CLINEAR ? mk2(fma(0.0, p0.q.x, p0.p.x), fma(0.0, p0.q.y, p0.p.y))
                                               : add2(p0.p, scl2(halfh, pq0p));
        const V2<double> qm = add2(p0.q, scl2(halfh, pq0q));
        double c1, g1, czz1;
        eval(x0.y + halfh * u0.y, t1.y, c1, g1, czz1);
        const double csq1 = c1 * c1;
        const double rc1 = rcp_rn(c1), rcsq1 = rcp_square(csq1, rc1);
        const double cnn1 = czz1 * t1.x * t1.x;
        const V2<double> pq1p = scl2(-cnn1, qm), pq1q = scl2(c1, pm);
        const V2<double> u1 = scl2(c1, t1);
        h = reduce(u1, h, za, zb, s0, ctr);
        const double w1 = div_rn(h, h2);
        const double w0 = 1.0 - w1;
        const V2<double> u2 = add2(scl2(w0, u0), scl2(w1, u1));
        // step_to_bdry: the profile node, or whatever is met outside the box
        const double hs = h;
        V2<double> x2;
        {
            const double ye = x0.y + h * u2.y;
            const bool above = za > ye;
            const bool cross = (above || zb < ye) && fabs(u2.y) > DBL_EPS;
            const double zn = above ? za : zb;
            const double hz = div_rn(zn - x0.y, u2.y);
            h = cross ? hz : h;
            x2 = mk2(x0.x + h * u2.x, cross ? zn : ye);
        }
        int hit = 0;
        inside = box.holds(x2.x, x2.y);
        if(!inside || h < hmin) {
            bool rare = h < hmin || meets(x2.x, x2.y, -INF_STEP);
            if(!rare && fabs(u2.x) > DBL_EPS && (x2.x < lmin || x2.x > lmax)) {
                const double xn = x2.x < lmin ? lmin : lmax;
                h = div_rn(-(x0.x - xn), u2.x);
                x2 = mk2(xn, x0.y + h * u2.y);
                rare = h < hmin;
            }
            if(rare) {
                inside = false;
                const Landing l = land_rare(e, it, ib, s0, x0.x, x0.y, u2.x, u2.y, hs);
                x2 = mk2(l.x, l.y);
                h = l.h;
                hit = l.hit;
            }
        }
        const double hw0 = h * w0, hw1 = h * w1;
        p1.x = x2;
        p1.t = mk2(t0.x, (t0.y - quot_rn(hw0 * g0, csq0, rcsq0)) - quot_rn(hw1 * g1, csq1, rcsq1));
        p1.taur = p0.taur + quot_rn(hw0, c0, rc0) + quot_rn(hw1, c1, rc1);
        p1.taui = p0.taui;
        p1.p = K == SSP_CLINEAR ? mk2(fma(0.0, qm.x, pm.x), fma(0.0, qm.y, pm.y))
                                : add2(add2(p0.p, scl2(hw0, pq0p)), scl2(hw1, pq1p));
        p1.q = add2(add2(p0.q, scl2(hw0, pq0q)), scl2(hw1, pq1q));
        p1.Amp = p0.Amp;
        p1.Phase = p0.Phase;
        p1.ntop = p0.ntop;
        p1.nbot = p0.nbot;
        eval_here(p1);
        p1.c = c;
        {   // curvature jump across a profile node (src/step.hpp:589-649)
            const double gj = g - g0;
            const double cnj = gj * p1.t.x, csj = gj * p1.t.y;
            const double rm = div_rn(p1.t.x, p1.t.y);
            const double rn = quot_rn(rm * (2.0 * cnj - rm * csj), c, rc);
            if(iz != s0) p1.p = sub2(p1.p, scl2(rn, p1.q));
        }
        end_top = end_bot = false;
        if(!inside) {
            pos = bdry_rare(e, it, ib, p1.x.x, p1.x.y, p1.t.x, ctr);
            if(pos.it != it || pos.ib != ib) {
                it = pos.it;
                ib = pos.ib;
                set_box();
            }
            end_top = pos.end_top;
            end_bot = pos.end_bot;
        }
        return hit;
    }
    // Reflect (src/reflect.hpp:125-452) at p0, the end of the step
    __device__ __forceinline__ void reflect(int hit, RunCounters *ctr)
    {
        // the profile at p0 is at hand; only the density is read here
        SSPOut<double> o;
        const double w = (p0.x.y - z0) / (z1 - z0);
        o.rho = (1.0 - w) * e->rho[iz] + w * e->rho[iz + 1];
        o.c = c;
        o.gradc = mk2(0.0, g);
        RayPt<double> r;
        pos = reflect_rare(e, pos, hit == 1, o, p0, r, ctr);
        p0 = r;
        eval_here(p0);
        end_top = pos.end_top;
        end_bot = pos.end_bot;
        low = p0.Amp < FLTD(0.005);
    }

    // RayTerminate's stop conditions (src/trace.hpp:391-477) at p0; inside the
    // rectangle only a lost amplitude ends a ray
    __device__ __forceinline__ bool stops()
    {
        bool stop = low;
        if(!inside) {
            stop = stop || fabs(p0.x.x) >= e->box_x || fabs(p0.x.y) >= e->box_y || (beg_top && end_top)
                || (beg_bot && end_bot);
        }
        beg_top = end_top;
        beg_bot = end_bot;
        return stop;
    }
};

} // namespace bhcb
