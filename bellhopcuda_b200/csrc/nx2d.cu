// Nx2D field mode (BELLHOP3D's N x 2-D: O3D ocean, 2-D rays), TL runs, FP64.
//
// Each ray lives in the vertical plane of its bearing beta through its source:
// ray coordinates (r, z) map to ocean coordinates by x = xs + r (cos beta,
// sin beta), depth unchanged (RayToOceanX / RayToOceanT / OceanToRayX /
// OceanToRayT, src/common_run.hpp:221-317). The step is the 2-D one (scalar
// p-q) with the sound speed evaluated in the 3-D ocean and projected on the
// plane (src/ssp.hpp:446-463), the step-size reduction and boundary landing
// solved in ocean coordinates against the 3-D boundary grids
// (src/step.hpp:654-811, O3D branch), and reflection off the 3-D triangle
// normal projected on the plane with the 3-D halfspace coefficient
// (src/reflect.hpp:125-452). The influence is the 2-D Cartesian geometric one
// (src/influence.hpp:1201-1406) on the ray's own receiver bearing: beams are
// launched along the receiver bearings (src/module/rayangles.hpp:163-179).
//
//  trace_nx_kernel      one ray per thread: RayInit / RayUpdate / RayTerminate
//                       of the Nx2D path and the sequential part of the 2-D
//                       influence; one record per segment that brackets
//                       receiver ranges.
//  influence_nx_kernel  32 records per warp, their receivers flattened; contributions
//                       added into the [isz][isx][isy][itheta][iz][ir] field.
//  scale_nx_kernel      ScalePressure, 2-D form (src/influence.hpp:1556-1627).
//
// This file is compiled without multiply-add contraction (-fmad=false) and
// takes the plane's (cos beta, sin beta) and the launch (cos alpha, sin alpha)
// from host tables: the landing on an x or y grid line of the boundary
// (OceanToRayX's ulp nudges towards the forward side, at most four) decides
// whether the next step starts in the new cell or first takes a forced small
// step, and that decision follows the last bits of the ocean position. With
// separately rounded products and sums and the same direction doubles, those
// bits follow the reference's own arithmetic.
#include <cuda_runtime.h>

#include <algorithm>

#include "bhcb_internal.h"
#include "device_math.cuh"
#include "trace2d.cuh"
#include "influence2d.cuh"
#include "ray2d.cuh"
#include "trace3d.cuh"
#include "walk3d.cuh"

namespace bhcb {

namespace {

typedef RayPt<double> RayN;

struct OrgN {   // Origin<true, false>: source position and the radial direction
    V3 xs;
    double tx, ty;
};

__device__ __forceinline__ V3 to_ocean_x(V2<double> x, const OrgN &o)
{
    return v3(o.xs.x + x.x * o.tx, o.xs.y + x.x * o.ty, x.y);
}
__device__ __forceinline__ V3 to_ocean_t(V2<double> t, const OrgN &o) { return v3(t.x * o.tx, t.x * o.ty, t.y); }
__device__ __forceinline__ V2<double> to_ray_t(V3 t, const OrgN &o) { return mk2(t.x * o.tx + t.y * o.ty, t.z); }

// the floating-point value k representations away (RealBitsAddInt)
__device__ __forceinline__ double bits_add(double v, long long k)
{
    return __longlong_as_double(__double_as_longlong(v) + k);
}

// OceanToRayX (src/common_run.hpp:244-302): range from the larger radial
// component; when the landing coordinate snap was x or y, nudge the range by
// ulps (at most 4) until the point maps back on the forward side of it
__device__ V2<double> to_ray_x(V3 x, const OrgN &o, V2<double> t, int snap, RunCounters *ctr)
{
    V2<double> r;
    r.y = x.z;
    r.x = fabs(o.tx) >= fabs(o.ty) ? (x.x - o.xs.x) / o.tx : (x.y - o.xs.y) / o.ty;
    if(snap < -2 || snap == -1 || snap >= 2) return r;
    for(int i = 0; i < 4; ++i) {
        const V3 xb = to_ocean_x(r, o);
        const double wx = o.tx * t.x, wy = o.ty * t.x;
        const double ex = xb.x - x.x, ey = xb.y - x.y;
        const bool okx = wx * ex >= 0.0, oky = wy * ey >= 0.0;
        if((snap == 0 && okx) || (snap == 1 && oky) || (okx && oky)) return r;
        r.x = bits_add(r.x, t.x > 0.0 ? 1 : -1);
    }
    run_warn(ctr, WARN_OCEANTORAYX_GAVEUP);
    return r;
}

// EvaluateSSP<O3D = true, R3D = false> (src/ssp.hpp:376-463): the 3-D sound
// speed at the ocean point, its gradient and curvature projected on the plane
template<bool NEED_RHO = false> __device__ __forceinline__ void eval_ssp_nx(V2<double> x, V2<double> t,
                                                                           SSPOut<double> &o, const Env3Dev &E,
                                                                           const OrgN &org, Seg3 &s,
                                                                           RunCounters *ctr)
{
    SSPOut3 p;
    eval_ssp3<NEED_RHO>(to_ocean_x(x, org), to_ocean_t(t, org), p, E, s, ctr);
    o.gradc = mk2(org.tx * p.gradc.x + org.ty * p.gradc.y, p.gradc.z);
    o.crz = org.tx * p.cxz + org.ty * p.cyz;
    o.crr = p.cxx * org.tx * org.tx + FLTD(2.0) * p.cxy * org.tx * org.ty + p.cyy * org.ty * org.ty;
    o.c = p.c;
    o.ci = p.ci;
    o.rho = p.rho;
    o.czz = p.czz;
}

// Step, Nx2D (src/step.hpp:654-811 with R3D = false, O3D = true)
__device__ void step_nx(const RayN &ray0, RayN &ray2, Bd3 &top, Bd3 &bot, const OrgN &org, const Env3Dev &E,
                        Seg3 &iSeg, int &small, bool &tr, bool &br, RunCounters *ctr)
{
    SSPOut<double> o0, o1, o2;
    eval_ssp_nx(ray0.x, ray0.t, o0, E, org, iSeg, ctr);
    const double cnn0 = o0.crr * ray0.t.y * ray0.t.y - 2.0 * o0.crz * ray0.t.x * ray0.t.y
        + o0.czz * ray0.t.x * ray0.t.x;
    const V2<double> pq0p = scl2(-cnn0, ray0.q), pq0q = scl2(o0.c, ray0.p);
    const Seg3 s0 = iSeg;
    const double csq0 = o0.c * o0.c;
    const V2<double> u0 = scl2(o0.c, ray0.t);
    double h = E.deltas;
    const V3 x_o = to_ocean_x(ray0.x, org);
    reduce_step3(x_o, to_ocean_t(u0, org), s0, top, bot, org.xs, E, h, small, ctr);
    const double halfh = 0.5 * h;
    RayN ray1;
    ray1.x = add2(ray0.x, scl2(halfh, u0));
    ray1.t = sub2(ray0.t, div2(scl2(halfh, o0.gradc), csq0));
    ray1.p = add2(ray0.p, scl2(halfh, pq0p));
    ray1.q = add2(ray0.q, scl2(halfh, pq0q));

    eval_ssp_nx(ray1.x, ray1.t, o1, E, org, iSeg, ctr);
    const double cnn1 = o1.crr * ray1.t.y * ray1.t.y - 2.0 * o1.crz * ray1.t.x * ray1.t.y
        + o1.czz * ray1.t.x * ray1.t.x;
    const V2<double> pq1p = scl2(-cnn1, ray1.q), pq1q = scl2(o1.c, ray1.p);
    const double csq1 = o1.c * o1.c;
    const V2<double> u1 = scl2(o1.c, ray1.t);
    reduce_step3(x_o, to_ocean_t(u1, org), s0, top, bot, org.xs, E, h, small, ctr);
    const double w1 = h / (2.0 * halfh);
    const double w0 = 1.0 - w1;
    const V2<double> u2 = add2(scl2(w0, u0), scl2(w1, u1));
    V3 x2_o;
    int snap;
    step_to_bdry3(x_o, x2_o, to_ocean_t(u2, org), h, tr, br, s0, top, bot, org.xs, E, ctr, snap);
    ray2.x = to_ray_x(x2_o, org, u2, snap, ctr);
    const double hw0 = h * w0, hw1 = h * w1;
    ray2.t = sub2(sub2(ray0.t, div2(scl2(hw0, o0.gradc), csq0)), div2(scl2(hw1, o1.gradc), csq1));
    const Cx<double> d0 = o0.ci == 0.0 ? cx<double>(hw0 / o0.c, 0.0) : rdivc(hw0, cx<double>(o0.c, o0.ci));
    const Cx<double> d1 = o1.ci == 0.0 ? cx<double>(hw1 / o1.c, 0.0) : rdivc(hw1, cx<double>(o1.c, o1.ci));
    ray2.taur = ray0.taur + d0.r + d1.r;
    ray2.taui = ray0.taui + d0.i + d1.i;
    ray2.p = add2(add2(ray0.p, scl2(hw0, pq0p)), scl2(hw1, pq1p));
    ray2.q = add2(add2(ray0.q, scl2(hw0, pq0q)), scl2(hw1, pq1q));
    ray2.Amp = ray0.Amp;
    ray2.Phase = ray0.Phase;
    ray2.ntop = ray0.ntop;
    ray2.nbot = ray0.nbot;
    eval_ssp_nx(ray2.x, ray2.t, o2, E, org, iSeg, ctr);
    ray2.c = o2.c;
    if(iSeg.z != s0.z) {   // CurvatureCorrection, 2-D form, depth crossings only
        const V2<double> gj = sub2(o2.gradc, o0.gradc);
        const V2<double> n2 = mk2(-ray2.t.y, ray2.t.x);
        const double cnj = dot2(gj, n2), csj = dot2(gj, ray2.t);
        const double rm = ray2.t.x / ray2.t.y;
        const double rn = rm * (2.0 * cnj - rm * csj) / ray2.c;
        ray2.p = sub2(ray2.p, scl2(rn, ray2.q));
    }
}

// Reflect, Nx2D (src/reflect.hpp:125-452, O3D && !R3D): the 3-D boundary
// normal projected on the plane; kappa the boundary curvature along the plane
// (OceanToRayCurvature, src/reflect.hpp:94-121; 0 for flat triangles)
__device__ void reflect_nx(const RayN &old, RayN &np, const HsDev &hs, bool istop, V3 nB3, double kappa,
                           const Env3Dev &E, const OrgN &org, Seg3 &iSeg, RunCounters *ctr)
{
    V2<double> nB = to_ray_t(nB3, org);
    nB = scl2(1.0 / sqrt(dot2(nB, nB)), nB);
    const double Th = dot2(old.t, nB);
    V2<double> tB = sub2(old.t, scl2(Th, nB));
    tB = scl2(1.0 / sqrt(dot2(tB, tB)), tB);
    const double Tg = dot2(old.t, tB);
    np.ntop = old.ntop + (istop ? 1 : 0);
    np.nbot = old.nbot + (istop ? 0 : 1);
    np.x = old.x;
    np.t = sub2(old.t, scl2(2.0 * Th, nB));
    SSPOut<double> o;
    eval_ssp_nx<true>(old.x, np.t, o, E, org, iSeg, ctr);
    const double c = o.c;
    np.c = c;
    np.taur = old.taur;
    np.taui = old.taui;
    const V2<double> rayt = scl2(c, old.t), rayn = mk2(-rayt.y, rayt.x);
    const V2<double> rayt_t = scl2(c, np.t), rayn_t = mk2(rayt_t.y, -rayt_t.x);
    double rn = FLTD(2.0) * kappa / (c * c) / Th;
    double cnjump = -dot2(o.gradc, sub2(rayn_t, rayn));
    const double csjump = -dot2(o.gradc, sub2(rayt_t, rayt));
    if(istop) { cnjump = -cnjump; rn = -rn; }
    const double rm = Tg / Th;
    rn += rm * (2.0 * cnjump - rm * csjump) / (c * c);
    if(E.e1d.beam2 == 'D') rn *= 2.0;
    else if(E.e1d.beam2 == 'Z') rn = 0.0;
    np.p = add2(old.p, scl2(rn, old.q));
    np.q = old.q;
    if(hs.bc == 'R') {
        np.Amp = old.Amp;
        np.Phase = old.Phase;
    } else if(hs.bc == 'V') {
        np.Amp = old.Amp;
        np.Phase = old.Phase + BHCB_PI;
    } else if(hs.bc == 'F') {
        double theta = (180.0 / BHCB_PI) * fabs(atan2(Th, Tg));
        if(theta > 90.0) theta = 180.0 - theta;
        double rc, ph;
        refl_coef(istop ? E.e1d.trc : E.e1d.brc, istop ? E.e1d.ntrc : E.e1d.nbrc, theta, rc, ph, ctr);
        np.Amp = old.Amp * rc;
        np.Phase = old.Phase + ph;
    } else if(hs.bc == 'A' || hs.bc == 'G') {   // halfspace, gamma form of the 3-D ocean
        const double omega = FLTD(2.0) * BHCB_PI * E.freq0;
        const double gk = omega * Tg;
        const double wc = omega / c;
        const Cx<double> g1sq = cx<double>(wc * wc - gk * gk, -DBL_MIN_POS);
        const Cx<double> wP = rdivc(omega, cx<double>(hs.cPr, hs.cPi));
        Cx<double> g2sq = csub(cmul(wP, wP), cx<double>(gk * gk, 0.0));
        g2sq.i -= DBL_MIN_POS;
        const Cx<double> g1 = csqrt_(cx<double>(-g1sq.r, -g1sq.i));
        const Cx<double> g2 = csqrt_(cx<double>(-g2sq.r, -g2sq.i));
        const Cx<double> a = cscl(hs.rho, g1), b = cscl(o.rho, g2);
        const Cx<double> Refl = cdiv(csub(a, b), cadd(a, b));
        const double ar = cabs_(Refl);
        if(ar < FLTD(1.0e-5)) {
            np.Amp = 0.0;
            np.Phase = old.Phase;
        } else {
            np.Amp = ar * old.Amp;
            np.Phase = old.Phase + atan2(Refl.i, Refl.r);
        }
    } else {
        run_error(ctr, ERR_BOUNDARY_CONDITION_TYPE);
        np.Amp = NAN;
        np.Phase = NAN;
    }
}

struct RayStateN {
    RayN p0;
    Bd3 top, bot;
    Seg3 iSeg;
    OrgN org;
    double alpha, c;
    double minx, miny, maxx, maxy;
};

// RayInit, Nx2D (src/trace.hpp:76-266)
__device__ bool ray_init_nx(const Env3Dev &E, const Job3 &J, RayStateN &st, RunCounters *ctr)
{
    const double alpha = E.alpha[J.ialpha];
    st.alpha = alpha;
    const double SrcDecl = (180.0 / BHCB_PI) * alpha;
    st.iSeg = Seg3{0, 0, 0};
    const V3 xs = v3(E.sx[J.isx], E.sy[J.isy], (double)E.sz[J.isz]);
    SSPOut3 o;
    eval_ssp3(xs, v3(0.0, 0.0, 1.0), o, E, st.iSeg, ctr);
    const double c = o.c;
    st.c = c;
    st.org.xs = xs;
    st.org.tx = E.bcs[2 * J.ibeta];
    st.org.ty = E.bcs[2 * J.ibeta + 1];
    const int ibp = min(bsearch_leq2(E.sbp, E.nsbp, SrcDecl), E.nsbp - 2);
    const double s = (SrcDecl - E.sbp[2 * ibp]) / (E.sbp[2 * (ibp + 1)] - E.sbp[2 * ibp]);
    float amp0 = (float)((FLTD(1.0) - s) * E.sbp[2 * ibp + 1] + s * E.sbp[2 * (ibp + 1) + 1]);
    if(E.run0 == 'S') {
        const float om = (float)(FLTD(2.0) * BHCB_PI * E.freq0);
        amp0 = (float)(amp0 * ((double)sqrtf(2.0f) * fabs(sin(om / c * xs.z * sin(alpha)))));
    }
    RayN &p0 = st.p0;
    p0.x = mk2(0.0, xs.z);
    p0.c = c;
    p0.t = mk2(E.acs[2 * J.ialpha] / c, E.acs[2 * J.ialpha + 1] / c);
    p0.taur = p0.taui = 0.0;
    p0.Amp = (double)amp0;
    p0.Phase = 0.0;
    p0.ntop = p0.nbot = 0;
    p0.p = mk2(1.0, 0.0);
    p0.q = mk2(0.0, 1.0);
    st.top.ix = st.top.iy = st.bot.ix = st.bot.iy = 0;
    st.top.justSteppedTo = st.bot.justSteppedTo = false;
    st.top.side = st.bot.side = false;
    st.top.outgoingSide = st.bot.outgoingSide = false;
    const V3 t_o = to_ocean_t(p0.t, st.org);
    get_bdry_seg3(xs, t_o, st.top, E.btop, E.top_nx, E.top_ny, true, true, ctr);
    get_bdry_seg3(xs, t_o, st.bot, E.bbot, E.bot_nx, E.bot_ny, false, true, ctr);
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
__device__ void reflect_at_nx(const RayN &p1, RayN &p2, const Bd3 &b, bool tr, const Env3Dev &E, const OrgN &org,
                              Seg3 &iSeg, RunCounters *ctr)
{
    const V3 x_o = to_ocean_x(p1.x, org);
    V3 nI = b.n;
    double kappa = 0.0;
    if(tr ? E.top_curv : E.bot_curv) {   // curvilinear grid (src/trace.hpp:318-341)
        const Bdry3PtDev *bd = tr ? E.btop : E.bbot;
        const int ny = tr ? E.top_ny : E.bot_ny;
        const double s1 = (x_o.x - b.x.x) / (b.xmax - b.xmin), s2 = (x_o.y - b.x.y) / (b.ymax - b.ymin);
        const double m1 = 1.0 - s1, m2 = 1.0 - s2;
        const Bdry3PtDev &d00 = bd[(size_t)b.ix * ny + b.iy], &d01 = bd[(size_t)b.ix * ny + b.iy + 1];
        const Bdry3PtDev &d10 = bd[(size_t)(b.ix + 1) * ny + b.iy], &d11 = bd[(size_t)(b.ix + 1) * ny + b.iy + 1];
        nI = v3(d00.noden[0] * m1 * m2 + d10.noden[0] * s1 * m2 + d11.noden[0] * s1 * s2 + d01.noden[0] * m1 * s2,
                d00.noden[1] * m1 * m2 + d10.noden[1] * s1 * m2 + d11.noden[1] * s1 * s2 + d01.noden[1] * m1 * s2,
                d00.noden[2] * m1 * m2 + d10.noden[2] * s1 * m2 + d11.noden[2] * s1 * s2 + d01.noden[2] * m1 * s2);
        const double tx = org.tx, ty = org.ty;
        kappa = d00.kxx * tx * tx + FLTD(2.0) * d00.kxy * tx * ty + d00.kyy * ty * ty;
        if(tr) kappa = -kappa;
    }
    reflect_nx(p1, p2, tr ? E.top : E.bot, tr, nI, kappa, E, org, iSeg, ctr);
}

// RayUpdate, Nx2D (src/trace.hpp:274-381)
__device__ bool ray_update_nx(RayStateN &st, RayN &p1, RayN &p2, int &small, const Env3Dev &E, RunCounters *ctr)
{
    bool tr = false, br = false;
    step_nx(st.p0, p1, st.top, st.bot, st.org, E, st.iSeg, small, tr, br, ctr);
    const V3 x_o = to_ocean_x(p1.x, st.org), t_o = to_ocean_t(p1.t, st.org);
    get_bdry_seg3(x_o, t_o, st.top, E.btop, E.top_nx, E.top_ny, true, false, ctr);
    get_bdry_seg3(x_o, t_o, st.bot, E.bbot, E.bot_nx, E.bot_ny, false, false, ctr);
    const bool two = tr || br;
    if(two) {
        reflect_at_nx(p1, p2, tr ? st.top : st.bot, tr, E, st.org, st.iSeg, ctr);
    }
    return two;
}

// RayTerminate, Nx2D (src/trace.hpp:391-477, O3D branch)
__device__ __forceinline__ bool ray_stops_nx(const RayStateN &st, int small, const Env3Dev &E)
{
    const V3 x = to_ocean_x(st.p0.x, st.org), t = to_ocean_t(st.p0.t, st.org);
    const V3 xs = st.org.xs;
    const bool leftbox = fabs(x.x - xs.x) >= E.box_x || fabs(x.y - xs.y) >= E.box_y || fabs(x.z) >= E.box_z;
    const bool esc0 = x.x < st.minx || x.y < st.miny || (x.x == st.minx && t.x < 0.0) || (x.y == st.miny && t.y < 0.0);
    const bool escN = x.x > st.maxx || x.y > st.maxy || (x.x == st.maxx && t.x > 0.0) || (x.y == st.maxy && t.y > 0.0);
    const bool lost = st.p0.Amp < FLTD(0.005);
    return leftbox || lost || esc0 || escN || small > 50;
}

// called with copies of the state: long and seldom taken
static __device__ __noinline__ void reflect_cold_nx(const RayN &p1, RayN &p2, const Bd3 &b, bool tr, const Env3Dev *E,
                                                    const OrgN &org, Seg3 &iSeg, RunCounters *ctr)
{
    reflect_at_nx(p1, p2, b, tr, *E, org, iSeg, ctr);
}

// The Nx2D ray over Walk3: ray_update_nx and ray_stops_nx with what the ray
// carries at hand (walk3d.cuh has the reasons). 12,996 rays through the
// hexahedral ocean: trace 22 -> 16.5 ms, 793 rays 19.5 -> 7, the same step counts.
template<bool HEX> struct RayNWalk {
    Walk3<HEX> w;
    RayN p0;
    OrgN org;
    Prof3 o0;                        // the profile at p0
    double minx, miny, maxx, maxy;
    double rt;                       // reciprocal of the larger radial component
    int small;
    bool low, inside;

    __device__ __forceinline__ void init(const Env3Dev &E, const RayStateN &st, RunCounters *ctr)
    {
        w.init(E, st.org.xs, st.top, st.bot, st.iSeg, ctr);
        p0 = st.p0;
        org = st.org;
        minx = st.minx; miny = st.miny; maxx = st.maxx; maxy = st.maxy;
        rt = rcp_signed(fabs(org.tx) >= fabs(org.ty) ? org.tx : org.ty);
        small = 0;
        low = p0.Amp < FLTD(0.005);
        inside = false;
        w.eval(to_ocean_x(p0.x, org), to_ocean_t(p0.t, org), o0, ctr);
    }
    // the gradient projected on the plane (eval_ssp_nx)
    __device__ __forceinline__ V2<double> grad(const Prof3 &o) const
    {
        return mk2(org.tx * o.g.x + org.ty * o.g.y, o.g.z);
    }
    __device__ __forceinline__ V2<double> to_ray(V3 x, V2<double> t, int snap, RunCounters *ctr) const
    {
        if(snap < -2 || snap == -1 || snap >= 2) {
            V2<double> r;
            r.y = x.z;
            r.x = fabs(org.tx) >= fabs(org.ty) ? quot_rn(x.x - org.xs.x, org.tx, rt) : quot_rn(x.y - org.xs.y, org.ty, rt);
            return r;
        }
        return to_ray_x(x, org, t, snap, ctr);
    }
    // step_nx and the boundary segments; returns the boundary to reflect at
    __device__ __forceinline__ int step(RayN &r2, RunCounters *ctr)
    {
        const V2<double> t0 = p0.t, x0 = p0.x;
        const Seg3 s0 = w.s;
        const Prof3 a = o0;
        const double c0 = a.c, csq0 = c0 * c0;
        const V2<double> ga = grad(a);
        const double cnn0 = a.czz * t0.x * t0.x;
        const V2<double> pq0p = scl2(-cnn0, p0.q), pq0q = scl2(c0, p0.p);
        const V2<double> u0 = scl2(c0, t0);
        const V3 x_o = to_ocean_x(x0, org);
        bool tr = false, br = false;
        w.begin();
        double h = w.deltas, halfh = 0.0, w0 = 0.0, w1 = 0.0, cnn1 = 0.0;
        V2<double> u = u0, pm = p0.p, qm = p0.q, gb = ga;
        const bool past = HEX && past_numbers(max(exponent_bits(p0.p.x), exponent_bits(p0.p.y)),
                                              max(exponent_bits(p0.q.x), exponent_bits(p0.q.y)));
        Prof3 b = a;
        // one copy of the crossing tests and of the evaluation (Ray3Walk::step)
#pragma unroll 1
        for(int pass = 0;; ++pass) {
            int snap;
            V3 x2_o;
            w.cross(pass == 2, x_o, to_ocean_t(u, org), h, x2_o, tr, br, s0, snap, small, ctr);
            if(pass == 1) {
                w1 = div_rn(h, 2.0 * halfh);
                w0 = 1.0 - w1;
                u = add2(scl2(w0, u0), scl2(w1, u));
                continue;
            }
            double k;
            V2<double> x;
            if(pass == 0) {
                halfh = k = 0.5 * h;
                x = add2(x0, scl2(halfh, u0));
            } else {
                k = h * w0;
                x = to_ray(x2_o, u, snap, ctr);
            }
            V2<double> t = mk2(HEX ? t0.x - quot_rn(k * ga.x, csq0, a.rcsq) : t0.x, t0.y - quot_rn(k * ga.y, csq0, a.rcsq));
            if(pass == 2) {
                const double hw1 = h * w1, csq1 = b.c * b.c;
                if(HEX) t.x = t.x - quot_rn(hw1 * gb.x, csq1, b.rcsq);
                t.y = t.y - quot_rn(hw1 * gb.y, csq1, b.rcsq);
                const Cx<double> d0 = a.ci == 0.0 ? cx<double>(quot_rn(k, c0, a.rc), 0.0)
                                                  : rdivc(k, cx<double>(c0, a.ci));
                const Cx<double> d1 = b.ci == 0.0 ? cx<double>(quot_rn(hw1, b.c, b.rc), 0.0)
                                                  : rdivc(hw1, cx<double>(b.c, b.ci));
                r2.taur = p0.taur + d0.r + d1.r;
                r2.taui = p0.taui + d0.i + d1.i;
                const V2<double> pq1p = scl2(-cnn1, qm), pq1q = scl2(b.c, pm);
                if(HEX) r2.p = past ? add2(pm, scl2(0.0, qm)) : p0.p;
                else r2.p = add2(add2(p0.p, scl2(k, pq0p)), scl2(hw1, pq1p));
                r2.q = add2(add2(p0.q, scl2(k, pq0q)), scl2(hw1, pq1q));
                r2.x = x;
                r2.t = t;
            }
            Prof3 o;
            w.eval(to_ocean_x(x, org), to_ocean_t(t, org), o, ctr);
            if(pass == 2) {
                o0 = o;
                break;
            }
            b = o;
            gb = grad(o);
            cnn1 = o.czz * t.x * t.x;
            // HEX: czz is 0, and p changes by 0 q only (Ray2Seg::step)
            if(!HEX) pm = add2(p0.p, scl2(halfh, pq0p));
            else if(past) pm = add2(p0.p, scl2(0.0, p0.q));
            qm = add2(p0.q, scl2(halfh, pq0q));
            u = scl2(o.c, t);
        }
        r2.Amp = p0.Amp;
        r2.Phase = p0.Phase;
        r2.ntop = p0.ntop;
        r2.nbot = p0.nbot;
        r2.c = o0.c;
        if(w.s.z != s0.z) {   // CurvatureCorrection, 2-D form, depth crossings only
            const V2<double> gj = sub2(grad(o0), ga);
            const V2<double> n2 = mk2(-r2.t.y, r2.t.x);
            const double cnj = dot2(gj, n2), csj = dot2(gj, r2.t);
            const double rm = fabs(r2.t.y) > 1.0e-100 ? div_rn(r2.t.x, r2.t.y) : r2.t.x / r2.t.y;
            const double rn = quot_rn(rm * (2.0 * cnj - rm * csj), r2.c, o0.rc);
            r2.p = sub2(r2.p, scl2(rn, r2.q));
        }
        const V3 xe = to_ocean_x(r2.x, org);
        inside = w.holds(xe);
        w.boundaries(inside, xe, to_ocean_t(r2.t, org), ctr);
        return tr ? 1 : br ? 2 : 0;
    }
    __device__ __forceinline__ void reflect(int hit, RunCounters *ctr)
    {
        RayN old = p0, r;
        Seg3 s = w.s;
        Bd3 b = hit == 1 ? w.general(w.top, w.E->btop, w.E->top_ny) : w.general(w.bot, w.E->bbot, w.E->bot_ny);
        OrgN o = org;
        reflect_cold_nx(old, r, b, hit == 1, w.E, o, s, ctr);
        w.set_cell(s);
        p0 = r;
        w.eval(to_ocean_x(p0.x, org), to_ocean_t(p0.t, org), o0, ctr);
        low = p0.Amp < FLTD(0.005);
    }
    __device__ __forceinline__ bool stops() const
    {
        bool stop = low || small > 50;
        if(!inside) {
            const V3 x = to_ocean_x(p0.x, org), t = to_ocean_t(p0.t, org), xs = org.xs;
            stop = stop || fabs(x.x - xs.x) >= w.E->box_x || fabs(x.y - xs.y) >= w.E->box_y || fabs(x.z) >= w.E->box_z
                || x.x < minx || x.y < miny || (x.x == minx && t.x < 0.0) || (x.y == miny && t.y < 0.0)
                || x.x > maxx || x.y > maxy || (x.x == maxx && t.x > 0.0) || (x.y == maxy && t.y > 0.0);
        }
        return stop;
    }
};

struct CursorN {
    unsigned long long next = 0, end = 0;
};

__device__ __forceinline__ void emit_nx(const SegRec<double> &rec, SegRec<double> *segs, unsigned long long cap,
                                        RunCounters *ctr, CursorN &cur, bool &overflow)
{
    if(cur.next == cur.end) {
        const unsigned long long b = atomicAdd(&ctr->nseg, 32ull);
        if(b + 32 > cap) {
            overflow = true;
            return;
        }
        cur.next = b;
        cur.end = b + 32;
    }
    const uint4 *src = reinterpret_cast<const uint4 *>(&rec);
    uint4 *dst = reinterpret_cast<uint4 *>(segs + cur.next++);
#pragma unroll
    for(int k = 0; k < (int)(sizeof(SegRec<double>) / 16); ++k) dst[k] = src[k];
}

// M: 1 when every group of the launch has the hexahedral grid, 2 when every one
// has a 1-D profile (RayNWalk), 0 for a mixture (general step). Warps take
// `lanes` consecutive jobs at a time.
template<int M> __global__ void __launch_bounds__(64) trace_nx_kernel(const GroupDev *__restrict__ groups, int ngroups,
                                                                      long long job_end, SegRec<double> *segs,
                                                                      unsigned long long cap, RunCounters *ctr,
                                                                      unsigned long long *job_counter, int lanes)
{
    const int lane = (int)(threadIdx.x & 31);
    for(;;) {
        __syncwarp();
        unsigned long long base = 0;
        if(lane == 0) base = atomicAdd(job_counter, (unsigned long long)lanes);
        base = __shfl_sync(0xffffffffu, base, 0);
        if((long long)base >= job_end) break;
        const long long job = (long long)base + lane;
        if(lane >= lanes || job >= job_end) continue;
        const GroupDev &G = groups[find_group(groups, ngroups, job)];
        const Env3Dev &E = *G.env3;
        const Job3 J = job_indices3(E, (int)(job - G.job_base));
        if(J.isz >= E.nsz) { run_error(ctr, ERR_RAYINIT); continue; }
        RayStateN st;
        if(!ray_init_nx(E, J, st, ctr)) continue;
        RayN p1, p2;
        // Init_Influence, 2-D Cartesian geometric (src/influence.hpp:525-644)
        const EnvDev &e = E.e1d;   // the receiver ranges and beam flags of the plane
        double ratio1 = sqrt(fabs(cos(st.alpha)));
        if(e.gaussian) ratio1 /= sqrt(FLTD(2.0) * BHCB_PI);
        const double rcp_q0 = E.dalpha / st.c;
        const InflEnv ie(e);
        InflState inf;
        inf.phase = 0.0;
        inf.qOld = st.p0.q.x;
        inf.x = st.p0.x;
        inf.ir = bsearch_gt(e.rr, e.nrr, st.p0.x.x);
        if(st.p0.t.x < 0.0 && inf.ir > 0) --inf.ir;
        inf.r = e.rr[inf.ir];
        int small = 0, is = 0;
        bool overflow = false;
        unsigned int nsteps = 0;
        CursorN cur;
        auto influence = [&](const RayN &a, const RayN &b) {
            SegRec<double> rec;
            if(infl_prologue(a, b, inf, ie, rcp_q0, ratio1, (int)job, is, rec))
                emit_nx(rec, segs, cap, ctr, cur, overflow);
            ++is;
        };
        RayNWalk<M == 1> ray;
        if constexpr(M != 0) ray.init(E, st, ctr);
        for(;;) {
            if((nsteps & 31) == 0 && __ldcg(&ctr->err_bits) != 0u) break;
            ++nsteps;
            if constexpr(M != 0) {
                const int hit = ray.step(p1, ctr);
                influence(ray.p0, p1);
                ray.p0 = p1;
                if(hit) {
                    ray.reflect(hit, ctr);
                    // of no length but at range 0 (trace_kernel)
                    p2 = ray.p0;
                    if(p1.x.x == 0.0) influence(p1, p2);
                    else ++is;
                }
            } else {
                const bool two = ray_update_nx(st, p1, p2, small, E, ctr);
                influence(st.p0, p1);
                if(two) influence(p1, p2);
                st.p0 = two ? p2 : p1;
            }
            if(overflow) {
                atomicMin(&ctr->overflow_job, (unsigned int)job);
                run_error(ctr, ERR_SEG_OVERFLOW);
                break;
            }
            if constexpr(M != 0) {
                if(ray.stops()) break;
            } else {
                if(ray_stops_nx(st, small, E)) break;
            }
            if(is >= MAXN_STEPS - 3) {
                run_warn(ctr, WARN_ONERAY_OUTOFMEMORY);
                break;
            }
        }
        for(; cur.next < cur.end; ++cur.next) segs[cur.next].job = -1;
        atomicAdd(&ctr->nsteps, (unsigned long long)nsteps);
    }
}

// InfluenceGeoCore + ApplyContribution, 2-D Cartesian (src/influence.hpp:
// 423-473, 897-1024). A warp stages 32 records; their items inside the segments'
// depth windows (src/influence.hpp:1285-1292), RUN ranges at a depth each, are
// flattened, so that every lane evaluates receivers. Bound by the FP64 work of
// the items and the field's 8-byte atomics. With one thread per record and
// receiver depth, most of them outside the window, and the record read from
// global memory by each, 12,996 rays x 501 x 101 receivers took 22.9 ms; this 3.9.
//
// Blocks of 32 records are too few for the chip where rays are few, and uneven
// where receivers are dense, so a block's items are dealt to `parts` warps, for
// about four units of work a warp. One warp a block against this, and one thread
// per record and depth in brackets: 3 rays x 20000 x 2000 receivers 420 -> 1.8 ms
// (1.6), 361 x 10001 x 2001 113 -> 39 (42), 1001 x 10001 x 1001 83 -> 58 (67).
//
// RUN is 1 or 8 (launch_influence_nx): an item's search for its record, its
// division and the record's parts from shared memory are paid once a run, but a
// step that brackets two or three ranges has no runs. RUN 1 and 8: 361 rays x
// 10001 x 2001 receivers (50 ranges a step) 46 and 39 ms, 12,996 x 501 x 101
// (2.5 a step) 3.9 and 4.4.
constexpr int WARPSN = 4;
constexpr int NX_PASS = 1 << 25;   // items of one record in a pass
template<int RUN>
__global__ void __launch_bounds__(32 * WARPSN) influence_nx_kernel(const SegRec<double> *__restrict__ segs,
                                                                   unsigned long long cap,
                                                                   const GroupDev *__restrict__ groups, int ngroups,
                                                                   float2 *field, RunCounters *ctr)
{
    __shared__ SegRec<double> s_rec[WARPSN][32];
    __shared__ double s_rcp[WARPSN][32], s_fl[WARPSN][32];
    __shared__ const Env3Dev *s_env[WARPSN][32];
    __shared__ long long s_row[WARPSN][32];
    __shared__ int s_incl[WARPSN][32], s_iz0[WARPSN][32], s_niz[WARPSN][32];
    const unsigned long long nseg = min(__ldcg(&ctr->nseg), cap);
    const unsigned long long nchunks = (nseg + 31) / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned int nwarps = gridDim.x * WARPSN;
    const unsigned int parts = nchunks < 4 * nwarps ? 4 * nwarps / max((unsigned int)nchunks, 1u) : 1u;
    unsigned int evals = 0;
    for(unsigned long long u = blockIdx.x * (unsigned long long)WARPSN + w; u < nchunks * parts; u += nwarps) {
        const unsigned long long ch = u / parts;
        const unsigned int part = (unsigned int)(u - ch * parts);
        const int nvalid = (int)min(32ull, nseg - ch * 32);
        {
            const int words = sizeof(SegRec<double>) / 16;
            const uint4 *src = reinterpret_cast<const uint4 *>(segs + ch * 32);
            uint4 *dst = reinterpret_cast<uint4 *>(&s_rec[w][0]);
            for(int k = lane; k < nvalid * words; k += 32) dst[k] = __ldcs(src + k);
        }
        __syncwarp();
        long long items = 0;
        const SegRec<double> &M = s_rec[w][lane];
        if(lane < nvalid && M.job >= 0) {
            const GroupDev &G = groups[find_group(groups, ngroups, M.job)];
            const Env3Dev &E = *G.env3;
            const double freq = E.freq0;
            double sig = M.sigma_seg, fl = 0.0;
            if(E.gaussian) {   // AdjustSigma (src/influence.hpp:91-100)
                fl = min(FLTD(0.2) * freq * M.tau1r, BHCB_PI * (M.c0 / freq));
                sig = max(sig, fl);
            }
            int i0 = 0, i1 = E.nrz;
            // (a width that is not a number bounds nothing)
            if(fabs(M.tx) > FLTD(0.50001) && sig == sig) {
                const double rmax = (E.gaussian ? 4.0 : 1.0) * sig;
                i0 = lower_f(E.rz, E.nrz, M.zlo - rmax);
                i1 = upper_f(E.rz, E.nrz, M.zhi + rmax);
            }
            if(i1 > i0) {
                items = (long long)((M.ir_hi - M.ir_lo + RUN) / RUN) * (i1 - i0);
                const Job3 J = job_indices3(E, (int)((long long)M.job - G.job_base));
                s_row[w][lane] = G.field_base
                    + ((((long long)J.isz * E.nsx + J.isx) * E.nsy + J.isy) * E.ntheta + J.ibeta) * E.nrz * E.nrr;
                s_env[w][lane] = &E;
                s_iz0[w][lane] = i0;
                s_niz[w][lane] = i1 - i0;
                s_fl[w][lane] = fl;
                s_rcp[w][lane] = rcp_rn(M.rlen);
            }
        }
        // passes of at most NX_PASS items of every record, so that the sums of 32 fit an int
        const unsigned int passes = __reduce_max_sync(0xffffffffu, (unsigned int)((items + NX_PASS - 1) / NX_PASS));
        for(unsigned int pass = 0; pass < passes; ++pass) {
        const long long first = (long long)pass * NX_PASS;
        int incl = (int)min(max(items - first, 0LL), (long long)NX_PASS);
#pragma unroll
        for(int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if(lane >= o) incl += v;
        }
        s_incl[w][lane] = incl;
        __syncwarp();
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for(long long at = 32 * part + lane; at < total; at += 32 * parts) {
            const int it = (int)at;
            int lo = 0, hi = 31;   // first record j with incl[j] > it
            while(lo < hi) {
                const int mid = (lo + hi) >> 1;
                if(s_incl[w][mid] > it) hi = mid; else lo = mid + 1;
            }
            const int j = lo, local = it - (j ? s_incl[w][j - 1] : 0);
            const int niz = s_niz[w][j], run = pass ? (int)((first + local) / niz) : local / niz;
            const int iz = s_iz0[w][j] + (int)(first + local - (long long)run * niz);
            const SegRec<double> &S = s_rec[w][j];
            const Env3Dev &E = *s_env[w][j];
            const bool gauss = E.gaussian != 0, coherent = E.coherent != 0;
            const double dz = (double)E.rz[iz] - S.x0z, fl = s_fl[w][j], rcp = s_rcp[w][j];
            const double omega = FLTD(2.0) * BHCB_PI * E.freq0;
            float2 *row = field + s_row[w][j] + (long long)iz * E.nrr;
            int ir = S.ir_lo + run * RUN;
            const int ir1 = min(ir + RUN - 1, S.ir_hi);
#pragma unroll 1
            do {
                const double dr = E.rr[ir] - S.x0r;
                const double s = quot_rn(dr * S.tx + dz * S.tz, S.rlen, rcp);
                const double n1 = fabs(dz * S.tx - dr * S.tz);
                const double qF = S.q0 + s * S.dq;
                double sigma = fabs(qF * S.rcp_q0);
                const double sig0 = sigma;
                if(gauss) sigma = max(sigma, fl);
                if(n1 >= (gauss ? 4.0 : 1.0) * sigma) continue;
                const double cnst = S.cnst_num / sqrt(fabs(qF));
                const double wgt = gauss ? exp(FLTD(-0.5) * (n1 / sigma) * (n1 / sigma)) * (sig0 / sigma)
                                         : (sigma - n1) / sigma;
                const bool caustic = (qF <= 0.0 && S.q0 > 0.0) || (qF >= 0.0 && S.q0 < 0.0);
                const double ph = caustic ? S.phase_b : S.phase_a;
                const double di = S.tau0i + s * S.dtaui;
                float2 v;
                if(coherent) {
                    const double amp = cnst * wgt * exp(omega * di);
                    double sn, cs;
                    sincos(reduce_2pi(omega * (S.tau0r + s * S.dtaur) - ph), &sn, &cs);
                    v = make_float2((float)(amp * cs), (float)(-amp * sn));
                } else {
                    double vv = cnst * exp(omega * di);
                    vv = vv * vv * wgt;
                    if(gauss) vv *= sqrt(FLTD(2.0) * BHCB_PI);
                    v = make_float2((float)vv, 0.f);
                }
                atomicAdd(row + ir, v);
                ++evals;
            } while(RUN > 1 && ++ir <= ir1);
        }
        __syncwarp();
        }
        __syncwarp();
    }
    for(int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, o);
    if(lane == 0 && evals) atomicAdd(&ctr->nevals, (unsigned long long)evals);
}

// Arrivals, Nx2D: the contributions of influence_nx_kernel as arrival
// candidates (ApplyContribution with itheta = ibeta and AddArr,
// src/influence.hpp:434-451; ReceiverAngles 2-D form, src/influence.hpp:
// 123-136: receiver azimuth = the source azimuth) keyed (receiver cell, ray,
// step) for the shared radix sort and per-cell replay. With kb.eigen, the same
// contributions as eigen hits (RecordEigenHit with itheta = ibeta), keyed
// (trace group, ray, step, walk position of the receiver range, bearing,
// depth): the 2-D Cartesian walk visits the bracketed ranges towards point1,
// then the depths (src/influence.hpp:1295-1406). One thread per record.
// COUNT: counts into ctr->nevals; otherwise candidate i at atomicAdd(cursor).
template<bool COUNT>
__global__ void __launch_bounds__(128) arr_gather_nx_kernel(const SegRec<double> *__restrict__ segs,
                                                            unsigned long long cap,
                                                            const GroupDev *__restrict__ groups, int ngroups,
                                                            ArrCand *cands, uint64_t *keys, uint32_t *vals,
                                                            unsigned long long cand_cap, unsigned long long *cursor,
                                                            RunCounters *ctr, ArrKeyBits kb)
{
    const unsigned long long nseg = min(__ldcg(&ctr->nseg), cap);
    unsigned long long count = 0;
    for(unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < nseg;
        k += (unsigned long long)gridDim.x * blockDim.x) {
        const SegRec<double> &S = segs[k];
        if(S.job < 0) continue;
        const GroupDev &G = groups[find_group(groups, ngroups, S.job)];
        const Env3Dev &E = *G.env3;
        const bool gauss = E.gaussian != 0;
        const double freq = E.freq0;
        double sig = S.sigma_seg, fl = 0.0;
        if(gauss) {   // AdjustSigma (src/influence.hpp:91-100)
            fl = min(FLTD(0.2) * freq * S.tau1r, BHCB_PI * (S.c0 / freq));
            sig = max(sig, fl);
        }
        const double rmax = (gauss ? 4.0 : 1.0) * sig;
        const bool window = fabs(S.tx) > FLTD(0.50001);
        const int local = (int)((long long)S.job - G.job_base);
        const Job3 J = job_indices3(E, local);
        const long long plane = G.field_base
            + ((((long long)J.isz * E.nsx + J.isx) * E.nsy + J.isy) * E.ntheta + J.ibeta) * E.nrz * E.nrr;
        const float azim = (float)((180.0 / BHCB_PI) * E.beta[J.ibeta]);
        for(int iz = 0; iz < E.nrz; ++iz) {
            const double zr = (double)E.rz[iz];
            if(window && (zr < S.zlo - rmax || zr > S.zhi + rmax)) continue;
            const double dz = zr - S.x0z;
            for(int ir = S.ir_lo; ir <= S.ir_hi; ++ir) {
                const double dr = E.rr[ir] - S.x0r;
                const double s = (dr * S.tx + dz * S.tz) / S.rlen;
                const double n1 = fabs(dz * S.tx - dr * S.tz);
                const double qF = S.q0 + s * S.dq;
                double sigma = fabs(qF * S.rcp_q0);
                const double sig0 = sigma;
                if(gauss) sigma = max(sigma, fl);
                if(n1 >= (gauss ? 4.0 : 1.0) * sigma) continue;
                if(COUNT) {
                    ++count;
                    continue;
                }
                const unsigned long long i = atomicAdd(cursor, 1ull);
                if(i >= cand_cap) continue;
                if(kb.eigen) {
                    ArrCand c;
                    c.amp = c.phase = c.delay_re = c.delay_im = 0.0;
                    c.rcvr_decl = 0.f;
                    c.ntop = S.is;                   // step
                    c.nbot = ir;                     // receiver range
                    c.job = S.job;
                    c.aux = J.ibeta;                 // itheta = ibeta (src/influence.hpp:439)
                    c.rcvr_azim = __int_as_float(iz);
                    cands[i] = c;
                    const int walk = S.tx > 0.0 ? ir : E.nrr - 1 - ir;
                    const int gidx = (int)(&G - groups);
                    keys[i] = ((uint64_t)gidx << kb.sh_cell) | ((uint64_t)local << kb.sh_job)
                              | ((uint64_t)S.is << kb.sh_is) | ((uint64_t)walk << kb.sh_walk)
                              | ((uint64_t)J.ibeta << kb.sh_theta) | (uint64_t)iz;
                    vals[i] = (uint32_t)i;
                    continue;
                }
                const double w = gauss ? exp(FLTD(-0.5) * (n1 / sigma) * (n1 / sigma)) * (sig0 / sigma)
                                       : (sigma - n1) / sigma;
                const bool caustic = (qF <= 0.0 && S.q0 > 0.0) || (qF >= 0.0 && S.q0 < 0.0);
                const long long cell = plane + (long long)iz * E.nrr + ir;
                ArrCand c;
                c.amp = S.cnst_num / sqrt(fabs(qF)) * w;
                c.phase = caustic ? S.phase_b : S.phase_a;
                c.delay_re = S.tau0r + s * S.dtaur;
                c.delay_im = S.tau0i + s * S.dtaui;
                c.rcvr_decl = (float)S.rcvr_decl;
                c.rcvr_azim = azim;
                c.ntop = S.ntop;
                c.nbot = S.nbot;
                c.job = S.job;
                c.aux = J.ialpha;
                cands[i] = c;
                keys[i] = ((uint64_t)cell << kb.sh_cell) | ((uint64_t)local << kb.sh_job) | (uint64_t)S.is;
                vals[i] = (uint32_t)i;
            }
        }
    }
    if(COUNT && count) atomicAdd(&ctr->nevals, count);
}

// ScalePressure, 2-D form (src/influence.hpp:1556-1627): intensity to
// pressure for incoherent runs, then -1 / sqrt(r)
__global__ void scale_nx_kernel(float2 *field, const GroupDev *__restrict__ groups, int g)
{
    const GroupDev &G = groups[g];
    const Env3Dev &E = *G.env3;
    const long long n = (long long)E.nsz * E.nsx * E.nsy * E.ntheta * E.nrz * E.nrr;
    for(long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float2 u = field[G.field_base + i];
        if(!E.coherent) { u.x = sqrtf(u.x); u.y = 0.f; }
        const double r = E.rr[i % E.nrr];
        const double factor = fabs(r) < DBL_EPS ? 0.0 : FLTD(-1.0) / sqrt(fabs(r));
        const float ff = (float)factor;
        field[G.field_base + i] = make_float2(u.x * ff, u.y * ff);
    }
}

// Ray trajectories, Nx2D (MainRayMode, src/trace.hpp:485-519, with the
// points written in ocean coordinates as WriteRay does, src/mode/ray.hpp:
// 240-247): COUNT pass then fill pass as for the 2-D and 3-D rays.
template<bool COUNT>
__global__ void __launch_bounds__(64) ray_nx_kernel(const GroupDev *__restrict__ groups, int ngroups,
                                                    const long long *__restrict__ jobs, const int *__restrict__ limits,
                                                    int nitems, const long long *__restrict__ off, double *pts,
                                                    int *npts, int *bnc, RunCounters *ctr)
{
    for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < nitems; i += gridDim.x * blockDim.x) {
        const long long job = jobs[i];
        const GroupDev &G = groups[find_group(groups, ngroups, job)];
        const Env3Dev &E = *G.env3;
        const Job3 J = job_indices3(E, (int)(job - G.job_base));
        const int cap = COUNT ? 0x7fffffff : npts[i];
        const long long base = COUNT ? 0 : off[i];
        RayStateN st;
        auto put = [&](int idx, const RayN &p) {
            if(!COUNT && idx < cap) {
                const V3 x = to_ocean_x(p.x, st.org);
                double *q = pts + 3 * (base + idx);
                q[0] = x.x;
                q[1] = x.y;
                q[2] = x.z;
            }
        };
        if(J.isz >= E.nsz) {
            run_error(ctr, ERR_RAYINIT);
            if(COUNT) { npts[i] = 0; bnc[2 * i] = bnc[2 * i + 1] = 0; }
            continue;
        }
        int nsteps = -1, last_top = 0, last_bot = 0;
        if(!ray_init_nx(E, J, st, ctr)) {
            put(0, st.p0);
            nsteps = 1;
        } else {
            put(0, st.p0);
            const int limit = limits[i];
            int is = 0, small = 0, prev_top = 0, prev_bot = 0;
            RayN p1, p2;
            for(;;) {
                if((is & 31) == 0 && __ldcg(&ctr->err_bits) != 0u) {
                    nsteps = is + 1;
                    last_top = st.p0.ntop;
                    last_bot = st.p0.nbot;
                    break;
                }
                const bool two = ray_update_nx(st, p1, p2, small, E, ctr);
                put(is + 1, p1);
                if(two) put(is + 2, p2);
                if(limit >= 0 && is >= limit) {
                    nsteps = is + 2;
                    last_top = p1.ntop;
                    last_bot = p1.nbot;
                    break;
                }
                prev_top = two ? p1.ntop : st.p0.ntop;
                prev_bot = two ? p1.nbot : st.p0.nbot;
                is += two ? 2 : 1;
                st.p0 = two ? p2 : p1;
                if(ray_stops_nx(st, small, E)) {
                    nsteps = is + 1;
                    last_top = st.p0.ntop;
                    last_bot = st.p0.nbot;
                    break;
                }
                if(is >= MAXN_STEPS - 3) {
                    run_warn(ctr, WARN_ONERAY_OUTOFMEMORY);
                    nsteps = is;
                    last_top = prev_top;
                    last_bot = prev_bot;
                    break;
                }
            }
        }
        if(COUNT) {
            npts[i] = nsteps;
            bnc[2 * i] = last_top;
            bnc[2 * i + 1] = last_bot;
        }
    }
}

} // namespace

cudaError_t launch_rays_nx(const GroupDev *groups, int ngroups, const long long *jobs, const int *limits, int nitems,
                           const long long *off, double *pts, int *npts, int *bnc, RunCounters *ctr, bool count,
                           int sm_count, cudaStream_t st)
{
    if(nitems <= 0) return cudaSuccess;
    int grid = (nitems + 63) / 64;
    if(grid > sm_count * 16) grid = sm_count * 16;
    if(count)
        ray_nx_kernel<true><<<grid, 64, 0, st>>>(groups, ngroups, jobs, limits, nitems, off, pts, npts, bnc, ctr);
    else
        ray_nx_kernel<false><<<grid, 64, 0, st>>>(groups, ngroups, jobs, limits, nitems, off, pts, npts, bnc, ctr);
    return cudaGetLastError();
}

cudaError_t launch_trace_nx(const GroupDev *groups, int ngroups, long long njobs, long long job_end, void *segs,
                            unsigned long long cap, RunCounters *ctr, unsigned long long *job_counter, int sm_count,
                            int kind, cudaStream_t st)
{
    const int lanes = lanes3(njobs, sm_count, kind != 0);
    const long long warps = (njobs + lanes - 1) / lanes;
    const int grid = (int)std::max(1LL, std::min<long long>((warps + 1) / 2, (long long)sm_count * 16));
    auto k = kind == 1 ? trace_nx_kernel<1> : kind == 2 ? trace_nx_kernel<2> : trace_nx_kernel<0>;
    k<<<grid, 64, 0, st>>>(groups, ngroups, job_end, (SegRec<double> *)segs, cap, ctr, job_counter, lanes);
    return cudaGetLastError();
}

cudaError_t launch_arr_gather_nx(const void *segs, unsigned long long nseg, const GroupDev *groups, int ngroups,
                                 bool count, ArrCand *cands, uint64_t *keys, uint32_t *vals,
                                 unsigned long long cand_cap, unsigned long long *cursor, RunCounters *ctr,
                                 ArrKeyBits kb, int grid, cudaStream_t st)
{
    if(nseg == 0) return cudaSuccess;
    const SegRec<double> *S = (const SegRec<double> *)segs;
    if(count)
        arr_gather_nx_kernel<true><<<grid, 128, 0, st>>>(S, nseg, groups, ngroups, nullptr, nullptr, nullptr, 0,
                                                         nullptr, ctr, kb);
    else
        arr_gather_nx_kernel<false><<<grid, 128, 0, st>>>(S, nseg, groups, ngroups, cands, keys, vals, cand_cap,
                                                          cursor, ctr, kb);
    return cudaGetLastError();
}

// ranges_per_step: receiver ranges in a step of the densest environment
cudaError_t launch_influence_nx(const void *segs, unsigned long long cap, const GroupDev *groups, int ngroups,
                                float2 *field, RunCounters *ctr, int grid, double ranges_per_step, cudaStream_t st)
{
    auto k = ranges_per_step >= 16.0 ? influence_nx_kernel<8> : influence_nx_kernel<1>;
    k<<<grid, 32 * WARPSN, 0, st>>>((const SegRec<double> *)segs, cap, groups, ngroups, field, ctr);
    return cudaGetLastError();
}

cudaError_t launch_scale_nx(float2 *field, const GroupDev *groups, int g, int grid, cudaStream_t st)
{
    scale_nx_kernel<<<grid, 256, 0, st>>>(field, groups, g);
    return cudaGetLastError();
}

size_t nx_record_bytes() { return sizeof(SegRec<double>); }

} // namespace bhcb
