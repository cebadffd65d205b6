// 3-D ray driver shared by the BELLHOP3D kernels: per-ray state, RayInit,
// RayUpdate and RayTerminate's stop conditions (src/trace.hpp:76-477).
#pragma once
#include "bhcb_internal.h"
#include "device_math.cuh"
#include "trace2d.cuh"
#include "influence2d.cuh"
#include "trace3d.cuh"
#include "walk3d.cuh"

namespace bhcb {

// Per-ray state of the 3-D ray loop.
struct RayState3 {
    Ray3 p0;
    Bd3 top, bot;
    Seg3 iSeg;
    V3 xs;
    double alpha, beta, c;
    double minx, miny, maxx, maxy;   // extent of the boundary grids (RayTerminate)
};

// RayInit (src/trace.hpp:76-266), 3-D: false when the source is on or outside
// the boundaries (the ray is not traced)
__device__ __forceinline__ bool ray_init3d(const Env3Dev &E, const Job3 &J, RayState3 &st, RunCounters *ctr)
{
    const double alpha = E.alpha[J.ialpha], beta = E.beta[J.ibeta];
    st.alpha = alpha;
    st.beta = beta;
    const double SrcDecl = (180.0 / BHCB_PI) * alpha;
    st.iSeg = Seg3{0, 0, 0};
    const V3 xs = v3(E.sx[J.isx], E.sy[J.isy], (double)E.sz[J.isz]);
    st.xs = xs;
    SSPOut3 o;
    eval_ssp3(xs, v3(0.0, 0.0, 1.0), o, E, st.iSeg, ctr);
    const double c = o.c;
    st.c = c;
    const int ibp = min(bsearch_leq2(E.sbp, E.nsbp, SrcDecl), E.nsbp - 2);
    const double s = (SrcDecl - E.sbp[2 * ibp]) / (E.sbp[2 * (ibp + 1)] - E.sbp[2 * ibp]);
    float amp0 = (float)((FLTD(1.0) - s) * E.sbp[2 * ibp + 1] + s * E.sbp[2 * (ibp + 1) + 1]);
    if(E.run0 == 'S') {
        const float om = (float)(FLTD(2.0) * BHCB_PI * E.freq0);
        amp0 = (float)(amp0 * ((double)sqrtf(2.0f) * fabs(sin(om / c * xs.z * sin(alpha)))));
    }
    Ray3 &p0 = st.p0;
    // launch direction from the host's cos / sin of the angles (the reference's RayInit computes them on the CPU)
    const double ca = E.acs[2 * J.ialpha], sa = E.acs[2 * J.ialpha + 1];
    const V3 tinit = v3(ca * E.bcs[2 * J.ibeta], ca * E.bcs[2 * J.ibeta + 1], sa);
    p0.x = xs;
    p0.c = c;
    p0.t = v3(tinit.x / c, tinit.y / c, tinit.z / c);
    p0.taur = p0.taui = 0.0;
    p0.Amp = (double)amp0;
    p0.Phase = 0.0;
    p0.ntop = p0.nbot = 0;
    p0.p = m2_diag(1.0);
    p0.q = m2_diag(0.0);
    p0.phi = 0.0;
    st.top.ix = st.top.iy = st.bot.ix = st.bot.iy = 0;
    st.top.justSteppedTo = st.bot.justSteppedTo = false;
    st.top.side = st.bot.side = false;
    st.top.outgoingSide = st.bot.outgoingSide = false;
    get_bdry_seg3(xs, p0.t, st.top, E.btop, E.top_nx, E.top_ny, true, true, ctr);
    get_bdry_seg3(xs, p0.t, st.bot, E.bbot, E.bot_nx, E.bot_ny, false, true, ctr);
    double dTop, dBot;
    distances3(xs, st.top, st.bot, dTop, dBot);
    if(dTop <= 0.0 || dBot <= 0.0) {
        run_warn(ctr, WARN_SOURCE_OUTSIDE_BOUNDARIES);
        return false;
    }
    const Bdry3PtDev *bb = E.bbot, *bt = E.btop;
    st.minx = max(bb[0].x[0], bt[0].x[0]);
    st.miny = max(bb[0].x[1], bt[0].x[1]);
    st.maxx = min(bb[(size_t)(E.bot_nx - 1) * E.bot_ny].x[0], bt[(size_t)(E.top_nx - 1) * E.top_ny].x[0]);
    st.maxy = min(bb[E.bot_ny - 1].x[1], bt[E.top_ny - 1].x[1]);
    return true;
}

// The reflection of p1 into p2 off boundary b (RayUpdate, src/trace.hpp:318-341)
__device__ __forceinline__ void reflect_at3d(const Ray3 &p1, Ray3 &p2, const Bd3 &b, bool tr, const Env3Dev &E,
                                             Seg3 &iSeg, RunCounters *ctr)
{
    V3 nI = b.n;
    double zxx = 0.0, zxy = 0.0, zyy = 0.0;
    if(tr ? E.top_curv : E.bot_curv) {
        // curvilinear grid: normal interpolated between the cell's node
        // normals, curvature of the cell (src/trace.hpp:318-341)
        const Bdry3PtDev *bd = tr ? E.btop : E.bbot;
        const int ny = tr ? E.top_ny : E.bot_ny;
        const double s1 = (p1.x.x - b.x.x) / (b.xmax - b.xmin), s2 = (p1.x.y - b.x.y) / (b.ymax - b.ymin);
        const double m1 = 1.0 - s1, m2 = 1.0 - s2;
        const Bdry3PtDev &d00 = bd[(size_t)b.ix * ny + b.iy], &d01 = bd[(size_t)b.ix * ny + b.iy + 1];
        const Bdry3PtDev &d10 = bd[(size_t)(b.ix + 1) * ny + b.iy], &d11 = bd[(size_t)(b.ix + 1) * ny + b.iy + 1];
        nI = v3(d00.noden[0] * m1 * m2 + d10.noden[0] * s1 * m2 + d11.noden[0] * s1 * s2 + d01.noden[0] * m1 * s2,
                d00.noden[1] * m1 * m2 + d10.noden[1] * s1 * m2 + d11.noden[1] * s1 * s2 + d01.noden[1] * m1 * s2,
                d00.noden[2] * m1 * m2 + d10.noden[2] * s1 * m2 + d11.noden[2] * s1 * s2 + d01.noden[2] * m1 * s2);
        zxx = d00.zxx;
        zxy = d00.zxy;
        zyy = d00.zyy;
    }
    reflect3d(p1, p2, tr ? E.top : E.bot, tr, nI, zxx, zxy, zyy, E, iSeg, ctr);
}

// RayUpdate (src/trace.hpp:274-381), 3-D: one step from st.p0 to p1 and, on a
// boundary hit, the reflected point p2; returns whether p2 was produced
__device__ __forceinline__ bool ray_update3d(RayState3 &st, Ray3 &p1, Ray3 &p2, int &small, const Env3Dev &E,
                                             RunCounters *ctr)
{
    bool tr = false, br = false;
    step3d(st.p0, p1, st.top, st.bot, st.xs, E, st.iSeg, small, tr, br, ctr);
    get_bdry_seg3(p1.x, p1.t, st.top, E.btop, E.top_nx, E.top_ny, true, false, ctr);
    get_bdry_seg3(p1.x, p1.t, st.bot, E.bbot, E.bot_nx, E.bot_ny, false, false, ctr);
    const bool two = tr || br;
    if(two) reflect_at3d(p1, p2, tr ? st.top : st.bot, tr, E, st.iSeg, ctr);
    return two;
}

// RayTerminate's stop conditions (src/trace.hpp:391-477), 3-D
__device__ __forceinline__ bool ray_stops3d(const RayState3 &st, int small, const Env3Dev &E)
{
    const V3 x = st.p0.x, t = st.p0.t;
    const bool leftbox = fabs(x.x - st.xs.x) >= E.box_x || fabs(x.y - st.xs.y) >= E.box_y || fabs(x.z) >= E.box_z;
    const bool esc0 = x.x < st.minx || x.y < st.miny || (x.x == st.minx && t.x < 0.0) || (x.y == st.miny && t.y < 0.0);
    const bool escN = x.x > st.maxx || x.y > st.maxy || (x.x == st.maxx && t.x > 0.0) || (x.y == st.maxy && t.y > 0.0);
    const bool lost = st.p0.Amp < FLTD(0.005);
    return leftbox || lost || esc0 || escN || small > 50;
}

// The step of a ray without a horizontal direction, and the reflection: called
// with copies of the state, for they are long and seldom taken.
struct Step3IO {
    Bd3 top, bot;
    V3 xs;
    Seg3 s;
    int small;
    bool tr, br;
};
static __device__ __noinline__ void step_cold(const Ray3 &r0, Ray3 &r2, Step3IO &io, const Env3Dev *E, RunCounters *ctr)
{
    step3d(r0, r2, io.top, io.bot, io.xs, *E, io.s, io.small, io.tr, io.br, ctr);
}
static __device__ __noinline__ void reflect_cold(const Ray3 &p1, Ray3 &p2, const Bd3 &b, bool tr, const Env3Dev *E,
                                                 Seg3 &iSeg, RunCounters *ctr)
{
    reflect_at3d(p1, p2, b, tr, *E, iSeg, ctr);
}

// The 3-D ray over Walk3: ray_update3d and ray_stops3d with what the ray
// carries at hand.
template<bool HEX> struct Ray3Walk {
    Walk3<HEX> w;
    Ray3 p0;
    Prof3 o0;                        // the profile at p0
    double minx, miny, maxx, maxy;   // extent of the boundary grids
    int small;
    bool bent;                       // the profile has a depth curvature (1-D, not c-linear)
    double cphi, sphi;               // cosine and sine of the last step's phi
    bool low, inside;                // amplitude below the stop threshold; p0 inside the box

    __device__ __forceinline__ void init(const Env3Dev &E, const RayState3 &st, RunCounters *ctr)
    {
        w.init(E, st.xs, st.top, st.bot, st.iSeg, ctr);
        p0 = st.p0;
        minx = st.minx; miny = st.miny; maxx = st.maxx; maxy = st.maxy;
        small = 0;
        bent = E.e1d.ssp_type != SSP_CLINEAR;
        cphi = 1.0;
        sphi = 0.0;
        low = p0.Amp < FLTD(0.005);
        inside = false;
        w.eval(p0.x, p0.t, o0, ctr);
    }
    static __device__ __forceinline__ bool past3(const Ray3 &r)
    {
        const double(&p)[2][2] = r.p.m, (&q)[2][2] = r.q.m;
        const int a = exponent_bits(p[0][0]), b = exponent_bits(p[0][1]), c = exponent_bits(p[1][0]);
        const int d = exponent_bits(p[1][1]);
        return past_numbers(max(max(a, b), max(c, d)), max(max(exponent_bits(q[0][0]), exponent_bits(q[0][1])),
                                                           max(exponent_bits(q[1][0]), exponent_bits(q[1][1]))))
            && min(min(a, b), min(c, d)) <= 0x7ff00000;
    }
    // delta_pq3: rate of the ray normals' angle (horizontal gradients only),
    // p' (with a depth curvature only); q' is c p
    __device__ __forceinline__ double phi_rate(V3 t, const Prof3 &o) const
    {
        if(!HEX) return 0.0;
        return div_rn(quot_rn(1.0, o.c, o.rc) * t.z * (t.y * o.g.x - t.x * o.g.y), t.x * t.x + t.y * t.y);
    }
    __device__ __forceinline__ M2 p_rate(const Ray3 &r, const Prof3 &o) const
    {
        SSPOut3 s;
        s.cxx = s.cyy = s.cxy = s.cxz = s.cyz = 0.0;
        s.czz = o.czz;
        s.c = o.c;
        s.gradc = o.g;
        return delta_pq3(r, s, c_partials3(r, s)).p;
    }
    // Step (src/step.hpp:654-811) and RayUpdate's boundary segments; returns
    // the boundary to reflect at (0: none, 1: surface, 2: bottom)
    __device__ __forceinline__ int step(Ray3 &r2, RunCounters *ctr)
    {
        const V3 t0 = p0.t;
        const Seg3 s0 = w.s;
        const double c0 = o0.c, csq0 = c0 * c0;
        bool tr = false, br = false;
        const Prof3 a = o0;
        w.begin();
        const bool steep = !(t0.x * t0.x + t0.y * t0.y > 1.0e-200);
        // without a curvature p changes by 0 q only (Ray2Seg::step), which matters while p
        // is a number and p or q is past all numbers
        const bool past = (HEX || !bent) && past3(p0);
        if(steep || past) {   // no horizontal direction, or such a p or q: the general step
            Step3IO io;
            io.top = w.general(w.top, w.E->btop, w.E->top_ny);
            io.bot = w.general(w.bot, w.E->bbot, w.E->bot_ny);
            io.xs = w.xs;
            io.s = s0;
            io.small = small;
            io.tr = io.br = false;
            Ray3 r0 = p0, q;
            step_cold(r0, q, io, w.E, ctr);
            r2 = q;
            tr = io.tr;
            br = io.br;
            small = io.small;
            // the step changes only the note of a landing on a diagonal
            w.top.justSteppedTo = io.top.justSteppedTo;
            w.top.outgoingSide = io.top.outgoingSide;
            w.bot.justSteppedTo = io.bot.justSteppedTo;
            w.bot.outgoingSide = io.bot.outgoingSide;
            w.set_cell(io.s);
            w.eval(r2.x, r2.t, o0, ctr);
            sincos(r2.phi, &sphi, &cphi);
            inside = false;
        } else {
            const double f0 = phi_rate(t0, a);
            const bool curved = !HEX && bent;
            M2 dp0, dp1;
            if(curved) dp0 = p_rate(p0, a);
            const V3 u0 = scl3(c0, t0);
            const M2 dq0 = m2_scl(c0, p0.p);
            // Three passes over one copy of the crossing tests and of the
            // evaluation: reduction along u0 and the half step, reduction along
            // u1, landing along u2. Unrolled, the loop outgrows the instruction
            // caches (12 cycles per instruction, 7.7 of them waiting for it).
            double h = w.deltas, halfh = 0.0, w0 = 0.0, w1 = 0.0, f1 = 0.0;
            V3 u = u0;
            Ray3 r1;
            Prof3 b;
#pragma unroll 1
            for(int pass = 0;; ++pass) {
                int snap;
                V3 x;
                inside = w.cross(pass == 2, p0.x, u, h, x, tr, br, s0, snap, small, ctr);
                if(pass == 1) {
                    w1 = div_rn(h, 2.0 * halfh);
                    w0 = 1.0 - w1;
                    u = add3(scl3(w0, u0), scl3(w1, u));
                    continue;
                }
                V3 t = t0;
                double k = h;
                if(pass == 0) {
                    halfh = k = 0.5 * h;
                    x = add3(p0.x, scl3(halfh, u0));
                } else {
                    k = h * w0;
                }
                if(HEX) {
                    t.x = t0.x - quot_rn(k * a.g.x, csq0, a.rcsq);
                    t.y = t0.y - quot_rn(k * a.g.y, csq0, a.rcsq);
                }
                t.z = t0.z - quot_rn(k * a.g.z, csq0, a.rcsq);
                if(pass == 2) {
                    const double hw1 = h * w1, csq1 = b.c * b.c;
                    if(HEX) {
                        t.x = t.x - quot_rn(hw1 * b.g.x, csq1, b.rcsq);
                        t.y = t.y - quot_rn(hw1 * b.g.y, csq1, b.rcsq);
                    }
                    t.z = t.z - quot_rn(hw1 * b.g.z, csq1, b.rcsq);
                    const Cx<double> d0 = a.ci == 0.0 ? cx<double>(quot_rn(k, c0, a.rc), 0.0)
                                                      : rdivc(k, cx<double>(c0, a.ci));
                    const Cx<double> d1 = b.ci == 0.0 ? cx<double>(quot_rn(hw1, b.c, b.rc), 0.0)
                                                      : rdivc(hw1, cx<double>(b.c, b.ci));
                    r2.taur = p0.taur + d0.r + d1.r;
                    r2.taui = p0.taui + d0.i + d1.i;
                    r2.phi = (p0.phi + k * f0) + hw1 * f1;
                    const M2 dq1 = m2_scl(b.c, r1.p);
                    r2.p = curved ? m2_add(m2_add(p0.p, m2_scl(k, dp0)), m2_scl(hw1, dp1)) : p0.p;
                    r2.q = m2_add(m2_add(p0.q, m2_scl(k, dq0)), m2_scl(hw1, dq1));
                    r2.x = x;
                    r2.t = t;
                }
                Prof3 o;
                w.eval(x, t, o, ctr);
                if(pass == 2) {
                    o0 = o;
                    break;
                }
                b = o;
                r1.x = x;
                r1.t = t;
                r1.phi = p0.phi + halfh * f0;
                r1.p = curved ? m2_add(p0.p, m2_scl(halfh, dp0)) : p0.p;
                if(curved) r1.q = m2_add(p0.q, m2_scl(halfh, dq0));
                f1 = phi_rate(t, o);
                if(curved) dp1 = p_rate(r1, o);
                u = scl3(o.c, t);
            }
            r2.Amp = p0.Amp;
            r2.Phase = p0.Phase;
            r2.ntop = p0.ntop;
            r2.nbot = p0.nbot;
            r2.c = o0.c;
            // once for the face correction and the influence's ray normals
            if(HEX || r2.phi != p0.phi) sincos(r2.phi, &sphi, &cphi);
            if(w.s.z != s0.z || w.s.x != s0.x || w.s.y != s0.y)
                face_corr3(r2, o0.rcsq, sub3(o0.g, a.g), w.s, s0, cphi, sphi);
        }
        w.boundaries(inside, r2.x, r2.t, ctr);
        return tr ? 1 : br ? 2 : 0;
    }
    __device__ __forceinline__ void reflect(int hit, RunCounters *ctr)
    {
        Ray3 old = p0, r;
        Seg3 s = w.s;
        Bd3 b = hit == 1 ? w.general(w.top, w.E->btop, w.E->top_ny) : w.general(w.bot, w.E->bbot, w.E->bot_ny);
        reflect_cold(old, r, b, hit == 1, w.E, s, ctr);
        w.set_cell(s);
        p0 = r;
        if(!HEX) sincos(p0.phi, &sphi, &cphi);
        w.eval(p0.x, p0.t, o0, ctr);
        low = p0.Amp < FLTD(0.005);
    }
    // ray_stops3d; inside the box only a lost amplitude or small steps end a ray
    __device__ __forceinline__ bool stops() const
    {
        bool stop = low || small > 50;
        if(!inside) {
            const V3 x = p0.x, t = p0.t;
            stop = stop || fabs(x.x - w.xs.x) >= w.E->box_x || fabs(x.y - w.xs.y) >= w.E->box_y
                || fabs(x.z) >= w.E->box_z || x.x < minx || x.y < miny || (x.x == minx && t.x < 0.0)
                || (x.y == miny && t.y < 0.0) || x.x > maxx || x.y > maxy || (x.x == maxx && t.x > 0.0)
                || (x.y == maxy && t.y > 0.0);
        }
        return stop;
    }
};

} // namespace bhcb
