// 3-D (BELLHOP3D) field-mode kernels for sm_100a, FP64.
//
//  trace3d_kernel     one ray per thread (persistent, work-queue driven):
//                     RayInit / RayUpdate / RayTerminate of the 3-D path
//                     (src/trace.hpp:76-477) and the sequential part of
//                     Step_InfluenceGeoCart's 3-D branch (src/influence.hpp:
//                     1201-1292: duplicate-point skips, caustic phase, beam
//                     width bound, receiver-range walk); one compact record per
//                     segment that brackets at least one receiver range.
//  influence3d_kernel warp-cooperative evaluation of the (segment, range,
//                     bearing) work of 32 records at a time: a warp prefix sum
//                     flattens it so lanes stay busy; each lane applies the
//                     bearing rejections and walks the receiver depths in the
//                     segment's depth window (src/influence.hpp:1294-1406),
//                     evaluates InfluenceGeoCore (src/influence.hpp:897-1024)
//                     and adds the contribution into the field, laid out as
//                     the reference's [isz][isx][isy][itheta][iz][ir]
//                     (GetFieldAddr, src/common.hpp:393-405).
//  sqrt3d_kernel      ScalePressure's intensity-to-pressure conversion for
//                     incoherent and semi-coherent runs (src/influence.hpp:
//                     1596-1606); coherent 3-D fields are not scaled.
#include <cuda_runtime.h>

#include <algorithm>

#include "bhcb_internal.h"
#include "device_math.cuh"
#include "trace2d.cuh"
#include "influence2d.cuh"
#include "trace3d.cuh"
#include "ray3d.cuh"

namespace bhcb {

namespace {

constexpr int SEG_BLOCK3 = 32;

struct Cursor3 {
    unsigned long long next = 0, end = 0;
};

__device__ __forceinline__ void emit_seg3(const SegRec3 &rec, SegRec3 *segs, unsigned long long cap,
                                          RunCounters *ctr, Cursor3 &cur, bool &overflow)
{
    if(cur.next == cur.end) {
        unsigned long long b = atomicAdd(&ctr->nseg, (unsigned long long)SEG_BLOCK3);
        if(b + SEG_BLOCK3 > cap) {
            overflow = true;
            return;
        }
        cur.next = b;
        cur.end = b + SEG_BLOCK3;
    }
    static_assert(sizeof(SegRec3) % 16 == 0 && sizeof(SegRec3) == 288, "records are written in 16-byte words");
    const uint4 *src = reinterpret_cast<const uint4 *>(&rec);
    uint4 *dst = reinterpret_cast<uint4 *>(segs + cur.next++);
#pragma unroll
    for(int k = 0; k < (int)(sizeof(SegRec3) / 16); ++k) dst[k] = src[k];
}

// the carried part of InfluenceRayInfo for the 3-D Cartesian geometric beams
struct Infl3 {
    double phase, qOld;
    double ratio1, rcp_q0, rcp_qhat0;
    V3 xs;
    int ir;
    double r;            // horizontal distance of the last point from the source
    double rr;           // the receiver range E.rr[ir]
};

__device__ __forceinline__ double row_len(const M2 &q, int row, double s)
{
    const double a = q.m[0][row] * s, b = q.m[1][row] * s;
    return sqrt_any(a * a + b * b);
}

// Step_InfluenceGeoCart, 3-D, up to the receiver loop (src/influence.hpp:1201-1292).
// What only a segment that brackets a receiver range needs (ray normals, beam
// width bound) is computed after the range walk. cphi, sphi: of P1.phi.
__device__ __forceinline__ bool infl_prologue3(const Ray3 &P0, const Ray3 &P1, Infl3 &inf, const Env3Dev &E,
                                               double cphi, double sphi, int job, int is, SegRec3 &rec)
{
    const double bx = P1.x.x - inf.xs.x, by = P1.x.y - inf.xs.y;
    const double rA = inf.r, rB = sqrt_any(bx * bx + by * by);
    inf.r = rB;
    if(fabs(rA - rB) <= 1.0e3 * spacing_d(rA)) return false;   // IsDuplicatePoint(rB, rA)
    if(is == 0) {
        inf.ir = rB > rA ? 0 : E.nrr - 1;
        inf.rr = E.rr[inf.ir];
    }
    V3 rayt = sub3(P1.x, P0.x);
    const double dd = dot3(rayt, rayt);
    // |d| > 1e-12 |x| is above the threshold of 1000 spacings (2.3e-13 |x| at most)
    const bool long_seg = dd > 1.0e-24 * (P1.x.x * P1.x.x) && dd > 1.0e-200;
    const double rlen = long_seg ? sqrt_rn(dd) : sqrt(dd);
    if(!long_seg && rlen <= 1.0e3 * spacing_d(P1.x.x)) return false;
    const double phaseq = m2_det(P0.q);
    if((phaseq <= 0.0 && inf.qOld > 0.0) || (phaseq >= 0.0 && inf.qOld < 0.0)) inf.phase += BHCB_PI / FLTD(2.0);
    inf.qOld = phaseq;

    // receiver-range walk (src/influence.hpp:1294-1297, 1386-1399): the
    // bracketed ranges of one segment are contiguous
    const double *rr = E.rr;
    const int nrr = E.nrr;
    const double rmin = min(rA, rB), rmax = max(rA, rB);
    int lo = 0x7fffffff, hi = -1, ir = inf.ir;
    double r = inf.rr;
    for(;;) {
        if(r >= rmin && r < rmax) {
            lo = min(lo, ir);
            hi = max(hi, ir);
        }
        int irTT;
        double rTT;
        if(rB > r) {
            if(ir >= nrr - 1) break;
            irTT = ir + 1;
            rTT = rr[irTT];
            if(rTT >= rB) break;
        } else {
            if(ir <= 0) break;
            irTT = ir - 1;
            rTT = rr[irTT];
            if(rTT <= rB) break;
        }
        ir = irTT;
        r = rTT;
    }
    inf.ir = ir;
    inf.rr = r;
    if(hi < 0) return false;
    const double rl = rcp_rn(rlen);
    rayt = v3(quot_rn(rayt.x, rlen, rl), quot_rn(rayt.y, rlen, rl), quot_rn(rayt.z, rlen, rl));
    V3 e1, e2;
    ray_normal_unit(rayt, P1.phi, cphi, sphi, e1, e2);
    const double l1 = max(row_len(P0.q, 0, inf.rcp_q0), row_len(P1.q, 0, inf.rcp_q0));
    const double l2 = max(row_len(P0.q, 1, inf.rcp_qhat0), row_len(P1.q, 1, inf.rcp_qhat0));
    const double ldiag = sqrt_any(l1 * l1 + l2 * l2);
    rec.x0[0] = P0.x.x; rec.x0[1] = P0.x.y; rec.x0[2] = P0.x.z;
    rec.tau0r = P0.taur;
    rec.tau0i = P0.taui;
    rec.dtaur = P1.taur - P0.taur;
    rec.dtaui = P1.taui - P0.taui;
    rec.rayt[0] = rayt.x; rec.rayt[1] = rayt.y; rec.rayt[2] = rayt.z;
    rec.e1[0] = e1.x; rec.e1[1] = e1.y; rec.e1[2] = e1.z;
    rec.e2[0] = e2.x; rec.e2[1] = e2.y; rec.e2[2] = e2.z;
    rec.rlen = rlen;
    rec.q0[0] = P0.q.m[0][0]; rec.q0[1] = P0.q.m[0][1]; rec.q0[2] = P0.q.m[1][0]; rec.q0[3] = P0.q.m[1][1];
    rec.dq[0] = P1.q.m[0][0] - P0.q.m[0][0];
    rec.dq[1] = P1.q.m[0][1] - P0.q.m[0][1];
    rec.dq[2] = P1.q.m[1][0] - P0.q.m[1][0];
    rec.dq[3] = P1.q.m[1][1] - P0.q.m[1][1];
    rec.rcp_q0 = inf.rcp_q0;
    rec.rcp_qhat0 = inf.rcp_qhat0;
    rec.cnst_num = inf.ratio1 * P1.c * P1.Amp;
    rec.phase0 = P0.Phase + inf.phase;
    rec.qold = inf.qOld;
    rec.ldiag = ldiag;
    rec.zlo = min(P0.x.z, P1.x.z);
    rec.zhi = max(P0.x.z, P1.x.z);
    rec.ir_lo = lo;
    rec.ir_hi = hi;
    rec.job = job;
    rec.is = is;
    rec.ntop = P1.ntop;
    rec.nbot = P1.nbot;
    return true;
}

// M: 1 when every group of the launch has the hexahedral grid, 2 when every
// one has a 1-D profile (Ray3Walk), 0 for a mixture (general step). Warps take
// `lanes` consecutive jobs at a time.
template<int M> __global__ void __launch_bounds__(64) trace3d_kernel(const GroupDev *__restrict__ groups, int ngroups,
                                                                     long long job_end, SegRec3 *segs,
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
        RayState3 st;
        if(!ray_init3d(E, J, st, ctr)) continue;
        Ray3 p1, p2;
        const double alpha = st.alpha, c = st.c;
        // ---- Init_Influence (src/influence.hpp:525-644), 3-D Cartesian geometric
        Infl3 inf;
        inf.ratio1 = sqrt(fabs(cos(alpha)));
        inf.ratio1 *= sqrt(E.dalpha * E.dbeta) / c;
        if(E.gaussian) inf.ratio1 /= FLTD(2.0) * BHCB_PI;
        inf.rcp_q0 = E.dalpha / c;
        inf.rcp_qhat0 = fabs(cos(alpha)) * E.dbeta / c;
        inf.phase = 0.0;
        inf.qOld = m2_det(st.p0.q);
        inf.xs = st.p0.x;
        inf.ir = bsearch_gt(E.rr, E.nrr, 0.0);
        inf.r = 0.0;
        inf.rr = E.rr[inf.ir];

        int small = 0, is = 0;
        bool overflow = false;
        unsigned int nsteps = 0;
        Cursor3 cur;
        auto influence = [&](const Ray3 &a, const Ray3 &b, double cp, double sp) {
            SegRec3 rec;
            if(infl_prologue3(a, b, inf, E, cp, sp, (int)job, is, rec)) emit_seg3(rec, segs, cap, ctr, cur, overflow);
            ++is;
        };
        Ray3Walk<M == 1> ray;
        if constexpr(M != 0) ray.init(E, st, ctr);
        for(;;) {
            if((nsteps & 31) == 0 && __ldcg(&ctr->err_bits) != 0u) break;
            ++nsteps;
            if constexpr(M != 0) {
                const int hit = ray.step(p1, ctr);
                influence(ray.p0, p1, ray.cphi, ray.sphi);
                ray.p0 = p1;
                if(hit) {
                    ray.reflect(hit, ctr);
                    ++is;   // the reflected point is at the same place: a duplicate for the influence
                }
            } else {
                const bool two = ray_update3d(st, p1, p2, small, E, ctr);
                influence(st.p0, p1, cos(p1.phi), sin(p1.phi));
                if(two) influence(p1, p2, cos(p2.phi), sin(p2.phi));
                st.p0 = two ? p2 : p1;
            }
            if(overflow) {
                atomicMin(&ctr->overflow_job, (unsigned int)job);
                run_error(ctr, ERR_SEG_OVERFLOW);
                break;
            }
            // ---- RayTerminate (src/trace.hpp:391-477), 3-D
            if constexpr(M != 0) {
                if(ray.stops()) break;
            } else {
                if(ray_stops3d(st, small, E)) break;
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

// Ray trajectories, 3-D (MainRayMode, src/trace.hpp:485-519) of listed rays:
// every ray of a RunType 'R' run, or the rays of eigen hits re-traced up to the
// hit (EigenModePostWorker, src/mode/eigen.cpp:24-45). One ray per thread.
// limits[i] < 0: no limit; else the ray stops two points after step limits[i].
// COUNT: npts[i] = number of points, bounce counts of the last point in
// bnc[2i], bnc[2i + 1]; otherwise the points (x, y, z) go to pts + 3 off[i].
template<bool COUNT>
__global__ void __launch_bounds__(64) ray3d_kernel(const GroupDev *__restrict__ groups, int ngroups,
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
        auto put = [&](int idx, const Ray3 &p) {
            if(!COUNT && idx < cap) {
                double *q = pts + 3 * (base + idx);
                q[0] = p.x.x;
                q[1] = p.x.y;
                q[2] = p.x.z;
            }
        };
        if(J.isz >= E.nsz) {
            run_error(ctr, ERR_RAYINIT);
            if(COUNT) { npts[i] = 0; bnc[2 * i] = bnc[2 * i + 1] = 0; }
            continue;
        }
        RayState3 st;
        int nsteps = -1, last_top = 0, last_bot = 0;
        if(!ray_init3d(E, J, st, ctr)) {
            put(0, st.p0);
            nsteps = 1;
        } else {
            put(0, st.p0);
            const int limit = limits[i];
            int is = 0, small = 0, prev_top = 0, prev_bot = 0;
            Ray3 p1, p2;
            for(;;) {
                if((is & 31) == 0 && __ldcg(&ctr->err_bits) != 0u) {
                    nsteps = is + 1;
                    last_top = st.p0.ntop;
                    last_bot = st.p0.nbot;
                    break;
                }
                const bool two = ray_update3d(st, p1, p2, small, E, ctr);
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
                if(ray_stops3d(st, small, E)) {
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

constexpr int WARPS3 = 2;   // the records of 32 segments take 13 KB of shared memory per warp

// What the pair and receiver stages read of a record, in shared memory (the
// rest of the record only for accepted receivers).
struct Rec3S {
    double x0[3], rayt[3], e1[3], e2[3];
    double rlen, rcp_len;      // segment length, rcp_rn(rlen)
    double zlo, zhi, ldiag;
    double q0[4], dq[4], rcp_q0, rcp_qhat0;
    float q0f[4], dqf[4], rq0f, rq1f;   // the same in FP32 (mixed precision)
    // bearings_near: bearing of x0 from the source (in spacings from the first
    // receiver bearing), its range, the angle kappa between that bearing and the
    // ray's heading (|sin|, cos), and the bound E + F (distance to x0) on the
    // horizontal distance from the ray line that a beam reaches; F < 0: none
    float ib0, r0, sk, ck, E, F;
};

// Record fields of bearings_near (see there).
__device__ __forceinline__ void beam_reach(Rec3S &S, const Env3Dev &E, double xs, double ys, double margin)
{
    S.F = -1.f;
    const double th = sqrt(S.rayt[0] * S.rayt[0] + S.rayt[1] * S.rayt[1]);
    const double ax = S.x0[0] - xs, ay = S.x0[1] - ys, r0 = sqrt(ax * ax + ay * ay);
    if(!(E.dtheta > 0.f) || !(th > 1.0e-3) || !(r0 > 1.0)) return;
    const double q00 = fabs(S.q0[0] * S.rcp_q0), q10 = fabs(S.q0[2] * S.rcp_q0);
    const double q01 = fabs(S.q0[1] * S.rcp_qhat0), q11 = fabs(S.q0[3] * S.rcp_qhat0);
    const double d00 = fabs(S.dq[0] * S.rcp_q0), d10 = fabs(S.dq[2] * S.rcp_q0);
    const double d01 = fabs(S.dq[1] * S.rcp_qhat0), d11 = fabs(S.dq[3] * S.rcp_qhat0);
    const bool gauss = E.gaussian != 0;
    const double Q = gauss ? max(max(q00, q01), max(q10, q11)) : max(q00 + q01, q10 + q11);
    const double D = gauss ? max(max(d00, d01), max(d10, d11)) : max(d00 + d01, d10 + d11);
    const double zm = max(fabs((double)E.rz[0] - S.x0[2]), fabs((double)E.rz[E.nrz - 1] - S.x0[2]));
    const double w = (gauss ? 4.0 : 1.0) * 1.4142135623730951 * (1.0 + 2.0 * margin) + margin;
    const double sk = (ay * S.rayt[0] - ax * S.rayt[1]) / (r0 * th), ck = (ax * S.rayt[0] + ay * S.rayt[1]) / (r0 * th);
    if(!(ck > 0.5)) return;
    S.ib0 = (atan2f((float)ay, (float)ax) - E.theta0) / E.dtheta;
    S.r0 = (float)r0;
    S.sk = (float)fabs(sk);
    S.ck = (float)ck;
    S.E = (float)(w * (Q + D * zm * fabs(S.rayt[2]) / S.rlen) + margin);
    S.F = (float)(w * D / S.rlen);
}

// The receiver bearings [first, first + count) (modulo ntheta on a closed fan)
// at range rr that a segment's beam can reach; all of them where nothing
// smaller follows. For a receiver at angle d from x0's bearing (|d| <= 90
// degrees, the others are behind the source), its horizontal distance from the
// ray line is at least rr (sin(|d| + kappa) - sin kappa) - |rr - r0| sin kappa,
// its distance from x0 at most |rr - r0| + 2 rr sin(|d| / 2), and an accepted
// one's horizontal distance from the line is at most E + F (distance from x0):
// n1 and n2 are bounded as in depth_window, q by |q0| + |s| |dq|, and |s| by
// the distance over the segment length. So accepted receivers have
// f(d) = sin(d + kappa) - sin kappa - 2 F sin(d / 2) <= G. With kappa <= 60
// degrees and F <= 0.5 f is concave on [0, 90], so if f(90) > G, f stays above
// G once it is.
// Of the 51,984-ray workload's 36 bearings about 4 remain; the pair tests of the
// other 32 were 45 of the kernel's 55 ms.
__device__ __forceinline__ void bearings_near(const Rec3S &S, const Env3Dev &E, float rr, int &first, int &count)
{
    first = 0;
    count = E.ntheta;
    if(!(S.F >= 0.f && S.F <= 0.5f) || !(rr > 1.f)) return;
    const float G = (S.E + (S.F + S.sk) * fabsf(rr - S.r0)) / rr * 1.002f + 1.0e-5f;
    const float half = 0.70710678f;   // sin 45 degrees
    if(!(S.ck - S.sk - 2.f * S.F * half > G)) return;
    float d = max(E.dtheta, 1.1f * G);
    for(int it = 0; it < 40; ++it) {
        if(d >= 1.5707f) return;
        float sd, cd;
        __sincosf(d, &sd, &cd);
        if(sd * S.ck + cd * S.sk - S.sk - 2.f * S.F * __sinf(0.5f * d) > G) break;
        if(it == 39) return;
        d *= 1.3f;
    }
    const float k = d / E.dtheta + 0.01f;
    float b = S.ib0;
    if(!E.theta_full) {   // the turn of the circle nearest to the fan's middle
        const float turn = 6.28318531f / E.dtheta, mid = 0.5f * (float)(E.ntheta - 1);
        b -= turn * rintf((b - mid) / turn);
    }
    int lo = (int)ceilf(b - k), hi = (int)floorf(b + k);
    if(E.theta_full) {
        if(hi - lo + 1 >= E.ntheta) return;
        first = lo % E.ntheta;
        if(first < 0) first += E.ntheta;
        count = max(hi - lo + 1, 0);
    } else {
        lo = max(lo, 0);
        hi = min(hi, E.ntheta - 1);
        first = lo;
        count = max(hi - lo + 1, 0);
    }
}

// InfluenceGeoCore, 3-D Cartesian (src/influence.hpp:897-1024): beam-window
// test, then amplitude cnst, weight w, phase and complex delay of one receiver
struct Contrib3 {
    double cnst, w, ph, dr, di;
};
__device__ __forceinline__ bool geo_core3(const Rec3S &R, const SegRec3 &G, double s, double n1, double n2, bool gauss,
                                          Contrib3 &o)
{
    double q00 = R.q0[0] + s * R.dq[0], q01 = R.q0[1] + s * R.dq[1];
    double q10 = R.q0[2] + s * R.dq[2], q11 = R.q0[3] + s * R.dq[3];
    q00 *= R.rcp_q0;     // row 0 (m[0][0], m[1][0])
    q10 *= R.rcp_q0;
    q01 *= R.rcp_qhat0;  // row 1 (m[0][1], m[1][1])
    q11 *= R.rcp_qhat0;
    const double qF = q00 * q11 - q10 * q01;
    const double l1 = sqrt(q00 * q00 + q10 * q10);
    const double l2 = sqrt(q01 * q01 + q11 * q11);
    if(nearly_zero(l1) || nearly_zero(l2)) return false;
    if(nearly_zero(qF)) return false;
    const double n1p = fabs((-q01 * n2 + q11 * n1) / qF);
    const double n2p = fabs((q00 * n2 - q10 * n1) / qF);
    const double bw = gauss ? 4.0 : 1.0;
    const double dist = gauss ? n1p + n2p : max(n1p, n2p);
    if(dist > bw * 1.0) return false;
    o.dr = G.tau0r + s * G.dtaur;
    o.di = G.tau0i + s * G.dtaui;
    o.cnst = G.cnst_num / sqrt(fabs(qF));
    o.w = gauss ? exp(FLTD(-0.5) * (n1p * n1p + n2p * n2p)) : (FLTD(1.0) - n1p) * (FLTD(1.0) - n2p);
    o.ph = G.phase0;
    if((qF <= 0.0 && G.qold > 0.0) || (qF >= 0.0 && G.qold < 0.0)) o.ph += BHCB_PI / FLTD(2.0);
    return true;
}

// ApplyContribution's TL branch (src/influence.hpp:448-471)
__device__ __forceinline__ float2 tl_field3(const Contrib3 &o, bool gauss, bool coherent, double omega)
{
    if(coherent) {
        const double a = omega * o.dr - o.ph;
        const double m = exp(omega * o.di);
        double sa, ca;
        sincos(-a, &sa, &ca);
        const double cw = o.cnst * o.w;
        return make_float2((float)(cw * (m * ca)), (float)(cw * (m * sa)));
    }
    double v = o.cnst * exp(omega * o.di);
    v = v * v * o.w;
    if(gauss) v *= FLTD(2.0) * BHCB_PI;
    return make_float2((float)v, 0.0f);
}

// The TL contribution of one receiver in the mixed precision (FP32 q, beam
// window, amplitude and weight with the SFU's approximations; the delay's
// phase omega tau is formed and reduced mod 2 pi in FP64, the rest in FP32).
// Same tests and formulas as geo_core3 + tl_field3.
__device__ __forceinline__ bool geo_tl3_mixed(const Rec3S &R, const SegRec3 &G, double s, double n1, double n2,
                                              bool gauss, bool coherent, double omega, float2 &out)
{
    const float sf = (float)s;
    const float q00 = fmaf(sf, R.dqf[0], R.q0f[0]) * R.rq0f;
    const float q10 = fmaf(sf, R.dqf[2], R.q0f[2]) * R.rq0f;
    const float q01 = fmaf(sf, R.dqf[1], R.q0f[1]) * R.rq1f;
    const float q11 = fmaf(sf, R.dqf[3], R.q0f[3]) * R.rq1f;
    const float qF = q00 * q11 - q10 * q01;
    const float eps2 = (float)(DBL_EPS * DBL_EPS);
    if(q00 * q00 + q10 * q10 < eps2 || q01 * q01 + q11 * q11 < eps2) return false;
    if(fabsf(qF) < (float)DBL_EPS) return false;
    const float iq = 1.0f / qF;
    const float n1f = (float)n1, n2f = (float)n2;
    const float n1p = fabsf((q11 * n1f - q01 * n2f) * iq);
    const float n2p = fabsf((q00 * n2f - q10 * n1f) * iq);
    const float dist = gauss ? n1p + n2p : fmaxf(n1p, n2p);
    if(dist > (gauss ? 4.0f : 1.0f)) return false;
    const float cnst = (float)G.cnst_num * rsqrtf(fabsf(qF));
    const float w = gauss ? __expf(-0.5f * (n1p * n1p + n2p * n2p)) : (1.0f - n1p) * (1.0f - n2p);
    const float att = __expf((float)(omega * (G.tau0i + s * G.dtaui)));
    if(coherent) {
        float ph = (float)G.phase0;
        if((qF <= 0.0f && G.qold > 0.0) || (qF >= 0.0f && G.qold < 0.0)) ph += (float)(BHCB_PI / 2.0);
        const double a = omega * (G.tau0r + s * G.dtaur);
        const float ar = (float)(a - 6.28318530717958647692 * rint(a * 0.15915494309189533577));
        float sa, ca;
        __sincosf(ph - ar, &sa, &ca);
        const float cw = cnst * w * att;
        out = make_float2(cw * ca, cw * sa);
    } else {
        float v = cnst * att;
        v = v * v * w;
        if(gauss) v *= (float)(2.0 * BHCB_PI);
        out = make_float2(v, 0.0f);
    }
    return true;
}

// first index with (double)rz >= z (n if none); z rounded up to float selects the same
__device__ __forceinline__ int first_depth_at_or_above(const float *rz, int n, double z)
{
    const float zf = __double2float_ru(z);
    int lo = 0, hi = n;
    while(lo < hi) {
        const int m = (lo + hi) >> 1;
        if(__ldg(rz + m) < zf) lo = m + 1; else hi = m;
    }
    return lo;
}
// last index with (double)rz <= z (-1 if none)
__device__ __forceinline__ int last_depth_at_or_below(const float *rz, int n, double z)
{
    const float zf = __double2float_rd(z);
    int lo = 0, hi = n;
    while(lo < hi) {
        const int m = (lo + hi) >> 1;
        if(__ldg(rz + m) <= zf) lo = m + 1; else hi = m;
    }
    return lo - 1;
}

// The depths of a (range, bearing) pair's vertical line that InfluenceGeoCore's
// beam-window test can accept, as [zl, zh] shrunk from the window passed in
// (false: none). With A = [[q00, q01], [q10, q11]] the row-scaled q at s, the
// test's normalised offsets (a, b) give the normal offsets n1 = q00 a + q01 b
// and n2 = q10 a + q11 b. Gaussian beams accept |a| + |b| <= 4, so |n1| <= 4
// max(|q00|, |q01|); hat beams |a|, |b| <= 1, so |n1| <= |q00| + |q01|; n2
// likewise. Both bounds are convex in s, which is linear in depth, so over a
// window they are largest at its ends; n1 and n2 before the absolute value are
// linear in depth. Two passes: the second has the smaller window's bounds. The
// margin keeps rounding from dropping a receiver that the test accepts (FP32
// in the mixed precision).
// Why: the vertical extent of a beam is set by the spacing of the elevations,
// 15 times finer than that of the bearings in the 51,984-ray workload, while
// the window of L_diag is the wider of the two: nearly all 101 depths of every
// pair, 95 % of them rejected one by one.
__device__ __forceinline__ bool depth_window(const Rec3S &R, double h, double a1, double a2, bool gauss, double margin,
                                             double &zl, double &zh)
{
    const double w = (gauss ? 4.0 : 1.0) * (1.0 + margin);
    const double c1 = R.e1[2], c2 = R.e2[2];
#pragma unroll
    for(int pass = 0; pass < 2; ++pass) {
        double b1 = 0.0, b2 = 0.0, f1[2], f2[2];
#pragma unroll
        for(int e = 0; e < 2; ++e) {
            const double dz = (e ? zh : zl) - R.x0[2];
            const double s = (h + dz * R.rayt[2]) * R.rcp_len;
            const double q00 = fabs((R.q0[0] + s * R.dq[0]) * R.rcp_q0), q10 = fabs((R.q0[2] + s * R.dq[2]) * R.rcp_q0);
            const double q01 = fabs((R.q0[1] + s * R.dq[1]) * R.rcp_qhat0);
            const double q11 = fabs((R.q0[3] + s * R.dq[3]) * R.rcp_qhat0);
            b1 = max(b1, gauss ? max(q00, q01) : q00 + q01);
            b2 = max(b2, gauss ? max(q10, q11) : q10 + q11);
            f1[e] = a1 + dz * c1;
            f2[e] = a2 + dz * c2;
        }
        b1 = w * b1 + margin;
        b2 = w * b2 + margin;
        if((f2[0] > b2 && f2[1] > b2) || (f2[0] < -b2 && f2[1] < -b2)) return false;
        if((f1[0] > b1 && f1[1] > b1) || (f1[0] < -b1 && f1[1] < -b1)) return false;
        if(fabs(c1) > 1.0e-3) {
            const double r = 1.0 / c1, mid = R.x0[2] - a1 * r, half = b1 * fabs(r);
            zl = max(zl, mid - half);
            zh = min(zh, mid + half);
        }
        if(fabs(c2) > 1.0e-3) {
            const double r = 1.0 / c2, mid = R.x0[2] - a2 * r, half = b2 * fabs(r);
            zl = max(zl, mid - half);
            zh = min(zh, mid + half);
        }
        if(!(zl <= zh)) return false;
    }
    return true;
}

// Work is flattened three times per warp: (segment, range) units over the
// warp's 32 records, (unit, bearing) pairs over the bearings a beam can reach,
// then (pair, depth) items over the pairs' depth windows, so that every lane
// evaluates receivers. Bound by instruction issue. The 51,984-ray workload (287 M
// contributions, mixed) took 115 ms with every bearing tested and every depth
// within L_diag evaluated (one item in 18 applied), 55 with depth_window and
// the records in shared memory, 22.6 with bearings_near.
// MODE: INFL_TL adds the field; INFL_ARR_COUNT counts the arrival candidates;
// INFL_ARR_FILL writes them (AddArr's inputs, src/influence.hpp:444-447) with
// the key (receiver cell, ray, step) that restores the reference's order.
// INFL_EIG_COUNT / INFL_EIG_FILL: the same for eigenray hits (RecordEigenHit,
// src/eigenrays.hpp:24-40), keyed by (trace group, ray, step, position in the
// receiver-range walk, bearing, depth) — the reference's single-threaded order.
// INFL_TL_MIXED: INFL_TL with the receiver's contribution in mixed precision.
enum { INFL_TL = 0, INFL_ARR_COUNT = 1, INFL_ARR_FILL = 2, INFL_EIG_COUNT = 3, INFL_EIG_FILL = 4, INFL_TL_MIXED = 5 };
template<int MODE>
__global__ void __launch_bounds__(32 * WARPS3) influence3d_kernel(
    const SegRec3 *__restrict__ segs, unsigned long long nseg, const GroupDev *__restrict__ groups, int ngroups,
    float2 *field, RunCounters *ctr, ArrCand *cands, uint64_t *keys, uint32_t *vals, unsigned long long cand_cap,
    unsigned long long *cursor, ArrKeyBits kb)
{
    // per record of the warp's chunk
    __shared__ Rec3S s_rec[WARPS3][32];
    __shared__ int s_incl[WARPS3][32];
    __shared__ int s_grp[WARPS3][32], s_irlo[WARPS3][32];
    __shared__ const Env3Dev *s_env[WARPS3][32];
    __shared__ long long s_fbase[WARPS3][32];    // field offset of (isz, isx, isy)
    __shared__ double s_xs[WARPS3][32], s_ys[WARPS3][32];
    // per (record, range) unit of a 32-unit batch: candidate bearings
    __shared__ int s_uincl[WARPS3][32], s_urec[WARPS3][32], s_uir[WARPS3][32], s_uth[WARPS3][32];
    // per surviving pair of a 32-pair batch
    __shared__ int s_pincl[WARPS3][32];
    __shared__ int s_prec[WARPS3][32], s_piz0[WARPS3][32], s_pmeta[WARPS3][32];
    __shared__ double s_ph[WARPS3][32], s_pa1[WARPS3][32], s_pa2[WARPS3][32];
    __shared__ long long s_poff[WARPS3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double margin = MODE == INFL_TL_MIXED ? 1.0e-3 : 1.0e-6;
    const unsigned long long nchunk = (nseg + 31) / 32;
    unsigned long long nevals = 0;
    for(unsigned long long ch = (unsigned long long)blockIdx.x * WARPS3 + w; ch < nchunk;
        ch += (unsigned long long)gridDim.x * WARPS3) {
        const unsigned long long idx = ch * 32 + lane;
        int n = 0, g = 0;
        if(idx < nseg) {
            const SegRec3 &R = segs[idx];
            const int job = __ldg(&R.job);
            if(job >= 0) {
                g = find_group(groups, ngroups, job);
                const GroupDev &G = groups[g];
                const Env3Dev &E = *G.env3;
                const int lo = __ldg(&R.ir_lo), hi = __ldg(&R.ir_hi);
                n = hi - lo + 1;
                const Job3 J = job_indices3(E, (int)(job - G.job_base));
                s_fbase[w][lane] = G.field_base
                    + (long long)(((size_t)J.isz * E.nsx + J.isx) * E.nsy + J.isy) * E.ntheta * E.nrz * E.nrr;
                s_xs[w][lane] = E.sx[J.isx];
                s_ys[w][lane] = E.sy[J.isy];
                s_irlo[w][lane] = lo;
                s_env[w][lane] = &E;
                Rec3S &S = s_rec[w][lane];
#pragma unroll
                for(int i = 0; i < 3; ++i) {
                    S.x0[i] = R.x0[i];
                    S.rayt[i] = R.rayt[i];
                    S.e1[i] = R.e1[i];
                    S.e2[i] = R.e2[i];
                }
                S.rlen = R.rlen;
                S.rcp_len = rcp_rn(R.rlen);
                S.zlo = R.zlo;
                S.zhi = R.zhi;
                S.ldiag = R.ldiag;
#pragma unroll
                for(int i = 0; i < 4; ++i) {
                    S.q0[i] = R.q0[i];
                    S.dq[i] = R.dq[i];
                    S.q0f[i] = (float)R.q0[i];
                    S.dqf[i] = (float)R.dq[i];
                }
                S.rcp_q0 = R.rcp_q0;
                S.rcp_qhat0 = R.rcp_qhat0;
                S.rq0f = (float)R.rcp_q0;
                S.rq1f = (float)R.rcp_qhat0;
                beam_reach(S, E, s_xs[w][lane], s_ys[w][lane], margin);
            }
        }
        int incl = n;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if(lane >= o) incl += v;
        }
        s_incl[w][lane] = incl;
        s_grp[w][lane] = g;
        __syncwarp();
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for(int ub = 0; ub < total; ub += 32) {
        // ---- unit stage: one (record, range) per lane, the bearings its beam can reach
        int nb = 0;
        if(ub + lane < total) {
            const int k = ub + lane;
            int lo = 0, hi = 31;   // first record j with incl[j] > k
            while(lo < hi) {
                const int mid = (lo + hi) >> 1;
                if(s_incl[w][mid] > k) hi = mid; else lo = mid + 1;
            }
            const int j = lo, ir = s_irlo[w][j] + k - (j ? s_incl[w][j - 1] : 0);
            const Env3Dev &E = *s_env[w][j];
            bearings_near(s_rec[w][j], E, (float)E.rr[ir], s_uth[w][lane], nb);
            s_urec[w][lane] = j;
            s_uir[w][lane] = ir;
        }
        int uincl = nb;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, uincl, o);
            if(lane >= o) uincl += v;
        }
        s_uincl[w][lane] = uincl;
        __syncwarp();
        const int utotal = __shfl_sync(0xffffffffu, uincl, 31);
        for(int pb = 0; pb < utotal; pb += 32) {
            // ---- pair stage: bearing rejections and the depth window
            const int k = pb + lane;
            int m = 0;
            if(k < utotal) {
                int lo = 0, hi = 31;   // first unit u with uincl[u] > k
                while(lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if(s_uincl[w][mid] > k) hi = mid; else lo = mid + 1;
                }
                const int u = lo, j = s_urec[w][u], ir = s_uir[w][u];
                const Rec3S &R = s_rec[w][j];
                const Env3Dev &E = *s_env[w][j];
                int itheta = s_uth[w][u] + k - (u ? s_uincl[w][u - 1] : 0);
                if(itheta >= E.ntheta) itheta -= E.ntheta;
                const double xsx = s_xs[w][j], xsy = s_ys[w][j];
                const double tc = E.tcs[2 * itheta], ts = E.tcs[2 * itheta + 1];
                const double rr = E.rr[ir];
                const double xrx = xsx + rr * tc, xry = xsy + rr * ts;
                const double rtx = R.rayt[0], rty = R.rayt[1];
                const double dxr = xrx - R.x0[0], dyr = xry - R.x0[1];
                const bool gauss = E.gaussian != 0;
                const double mprime = fabs(dxr * (-rty) + dyr * rtx);
                bool keep = gauss || !(mprime > 1.0 * R.ldiag);
                keep = keep && !((xrx - xsx) * (R.x0[0] - xsx) + (xry - xsy) * (R.x0[1] - xsy) < 0.0);
                const double nrz = rtx * tc - rty * (-ts);
                keep = keep && !(fabs(nrz) < 1e-9);
                if(keep) {
                    const double Lz = (gauss ? 4.0 : 1.0) * R.ldiag / fabs(nrz);
                    // receiver depths are sorted: the window is an index range
                    const float *rz = E.rz;
                    const int nrz_ = E.nrz;
                    double zl = max(R.zlo - Lz, (double)rz[0]), zh = min(R.zhi + Lz, (double)rz[nrz_ - 1]);
                    const double h = dxr * rtx + dyr * rty;
                    const double a1 = dxr * R.e1[0] + dyr * R.e1[1], a2 = dxr * R.e2[0] + dyr * R.e2[1];
                    if(zl <= zh && depth_window(R, h, a1, a2, gauss, margin, zl, zh)) {
                        const int iz0 = first_depth_at_or_above(rz, nrz_, zl);
                        const int iz1 = last_depth_at_or_below(rz, nrz_, zh);
                        if(iz0 <= iz1) {
                            m = iz1 - iz0 + 1;
                            s_prec[w][lane] = j;
                            s_piz0[w][lane] = iz0;
                            s_ph[w][lane] = h;
                            s_pa1[w][lane] = a1;
                            s_pa2[w][lane] = a2;
                            s_poff[w][lane] = s_fbase[w][j] + (long long)itheta * nrz_ * E.nrr + ir;
                            s_pmeta[w][lane] = (itheta << 20) | ir;
                        }
                    }
                }
            }
            int pincl = m;
#pragma unroll
            for(int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, pincl, o);
                if(lane >= o) pincl += v;
            }
            s_pincl[w][lane] = pincl;
            __syncwarp();
            const int ptotal = __shfl_sync(0xffffffffu, pincl, 31);
            // ---- receiver stage: one (pair, depth) item per lane
            for(int q = lane; q < ptotal; q += 32) {
                int lo = 0, hi = 31;
                while(lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if(s_pincl[w][mid] > q) hi = mid; else lo = mid + 1;
                }
                const int pi = lo;
                const int iz = s_piz0[w][pi] + q - (pi ? s_pincl[w][pi - 1] : 0);
                const int j = s_prec[w][pi];
                const Rec3S &S = s_rec[w][j];
                const SegRec3 &R = segs[ch * 32 + j];
                const Env3Dev &E = *s_env[w][j];
                const double dz = (double)E.rz[iz] - S.x0[2];
                const double sv = quot_rn(s_ph[w][pi] + dz * S.rayt[2], S.rlen, S.rcp_len);
                const double n1 = fabs(s_pa1[w][pi] + dz * S.e1[2]);
                const double n2 = fabs(s_pa2[w][pi] + dz * S.e2[2]);
                if(MODE == INFL_TL_MIXED) {
                    float2 v;
                    if(!geo_tl3_mixed(S, R, sv, n1, n2, E.gaussian != 0, E.coherent != 0,
                                      FLTD(2.0) * BHCB_PI * E.freq0, v))
                        continue;
                    ++nevals;
                    atomicAdd(field + s_poff[w][pi] + (long long)iz * E.nrr, v);
                    continue;
                }
                Contrib3 o;
                if(!geo_core3(S, R, sv, n1, n2, E.gaussian != 0, o)) continue;
                ++nevals;
                const long long cell = s_poff[w][pi] + (long long)iz * E.nrr;
                if(MODE == INFL_TL) {
                    const double omega = FLTD(2.0) * BHCB_PI * E.freq0;
                    atomicAdd(field + cell, tl_field3(o, E.gaussian != 0, E.coherent != 0, omega));
                } else if(MODE == INFL_EIG_FILL) {
                    const unsigned long long i = atomicAdd(cursor, 1ull);
                    if(i >= cand_cap) continue;
                    const int itheta = s_pmeta[w][pi] >> 20, ir = s_pmeta[w][pi] & 0xfffff;
                    // the walk visits the bracketed ranges towards rB: ascending when rB > rA
                    const double xsx = s_xs[w][j], xsy = s_ys[w][j];
                    const double ax = R.x0[0] - xsx, ay = R.x0[1] - xsy;
                    const double bx = ax + R.rayt[0] * R.rlen, by = ay + R.rayt[1] * R.rlen;
                    const bool up = bx * bx + by * by > ax * ax + ay * ay;
                    const int walk = up ? ir - R.ir_lo : R.ir_hi - ir;
                    ArrCand c;
                    c.amp = c.phase = c.delay_re = c.delay_im = 0.0;
                    c.rcvr_decl = 0.0f;
                    c.ntop = R.is;
                    c.nbot = ir;
                    c.job = R.job;
                    c.aux = itheta;
                    c.rcvr_azim = __int_as_float(iz);
                    cands[i] = c;
                    keys[i] = ((uint64_t)s_grp[w][j] << kb.sh_cell) | ((uint64_t)R.job << kb.sh_job)
                        | ((uint64_t)R.is << kb.sh_is) | ((uint64_t)walk << kb.sh_walk)
                        | ((uint64_t)itheta << kb.sh_theta) | (uint64_t)iz;
                    vals[i] = (uint32_t)i;
                } else if(MODE == INFL_ARR_FILL) {
                    const unsigned long long i = atomicAdd(cursor, 1ull);
                    if(i >= cand_cap) continue;
                    ArrCand c;
                    c.amp = o.cnst * o.w;
                    c.phase = o.ph;
                    c.delay_re = o.dr;
                    c.delay_im = o.di;
                    // ReceiverAngles, 3-D (src/influence.hpp:123-138)
                    const double rtx = R.rayt[0], rty = R.rayt[1];
                    c.rcvr_decl = (float)((180.0 / BHCB_PI) * atan2(R.rayt[2], sqrt(rtx * rtx + rty * rty)));
                    c.rcvr_azim = (float)((180.0 / BHCB_PI) * atan2(rty, rtx));
                    c.ntop = R.ntop;
                    c.nbot = R.nbot;
                    c.job = R.job;
                    c.aux = 0;
                    cands[i] = c;
                    keys[i] = ((uint64_t)cell << kb.sh_cell) | ((uint64_t)R.job << kb.sh_job) | (uint64_t)R.is;
                    vals[i] = (uint32_t)i;
                }
            }
            __syncwarp();
        }
        }
        __syncwarp();
    }
    // one counter update per warp
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) nevals += __shfl_down_sync(0xffffffffu, nevals, o);
    if(MODE != INFL_ARR_FILL && MODE != INFL_EIG_FILL && lane == 0 && nevals) atomicAdd(&ctr->nevals, nevals);
}

// eigen hits in sorted order (RecordEigenHit layout, include/bhc/structs.hpp:353-361)
__global__ void eigen_emit3_kernel(const uint32_t *__restrict__ vals, const ArrCand *__restrict__ cands,
                                   unsigned long long n, const GroupDev *__restrict__ groups, int ngroups,
                                   EigenHitRec *hits, int32_t *group_of_hit)
{
    for(unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
        k += (unsigned long long)gridDim.x * blockDim.x) {
        const ArrCand &c = cands[vals[k]];
        const int g = find_group(groups, ngroups, c.job);
        const Job3 J = job_indices3(*groups[g].env3, (int)((long long)c.job - groups[g].job_base));
        EigenHitRec h;
        h.is = c.ntop;
        h.itheta = c.aux;
        h.ir = c.nbot;
        h.iz = __float_as_int(c.rcvr_azim);
        h.isx = J.isx;
        h.isy = J.isy;
        h.isz = J.isz;
        h.ialpha = J.ialpha;
        h.ibeta = J.ibeta;
        hits[k] = h;
        group_of_hit[k] = g;
    }
}

__global__ void sqrt3d_kernel(float2 *f, long long n)
{
    for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        f[i] = make_float2(sqrtf(f[i].x), 0.0f);
}

} // namespace

cudaError_t launch_rays3d(const GroupDev *groups, int ngroups, const long long *jobs, const int *limits, int nitems,
                          const long long *off, double *pts, int *npts, int *bnc, RunCounters *ctr, bool count,
                          int sm_count, cudaStream_t st)
{
    if(nitems <= 0) return cudaSuccess;
    int grid = (nitems + 63) / 64;
    if(grid > sm_count * 16) grid = sm_count * 16;
    if(count)
        ray3d_kernel<true><<<grid, 64, 0, st>>>(groups, ngroups, jobs, limits, nitems, off, pts, npts, bnc, ctr);
    else
        ray3d_kernel<false><<<grid, 64, 0, st>>>(groups, ngroups, jobs, limits, nitems, off, pts, npts, bnc, ctr);
    return cudaGetLastError();
}

// rays per warp for njobs rays (lanes3), the trace of jobs [*job_counter, job_end)
cudaError_t launch_trace3d(const GroupDev *groups, int ngroups, long long njobs, long long job_end, SegRec3 *segs,
                           unsigned long long cap, RunCounters *ctr, unsigned long long *job_counter, int sm_count,
                           int kind, cudaStream_t st)
{
    const int lanes = lanes3(njobs, sm_count, kind != 0);
    const long long warps = (njobs + lanes - 1) / lanes;
    const int grid = (int)std::max(1LL, std::min<long long>((warps + 1) / 2, (long long)sm_count * 16));
    auto k = kind == 1 ? trace3d_kernel<1> : kind == 2 ? trace3d_kernel<2> : trace3d_kernel<0>;
    k<<<grid, 64, 0, st>>>(groups, ngroups, job_end, segs, cap, ctr, job_counter, lanes);
    return cudaGetLastError();
}

// grid: CTAs of four warps
cudaError_t launch_influence3d(const SegRec3 *segs, unsigned long long nseg, const GroupDev *groups, int ngroups,
                               float2 *field, RunCounters *ctr, int grid, cudaStream_t st, bool mixed)
{
    if(nseg == 0) return cudaSuccess;
    grid = grid * 4 / WARPS3;
    if(mixed)
        influence3d_kernel<INFL_TL_MIXED><<<grid, 32 * WARPS3, 0, st>>>(segs, nseg, groups, ngroups, field, ctr,
                                                                         nullptr, nullptr, nullptr, 0, nullptr,
                                                                         ArrKeyBits{});
    else
        influence3d_kernel<INFL_TL><<<grid, 32 * WARPS3, 0, st>>>(segs, nseg, groups, ngroups, field, ctr, nullptr,
                                                                   nullptr, nullptr, 0, nullptr, ArrKeyBits{});
    return cudaGetLastError();
}

// arrival candidates of a 3-D run: count = true counts them into ctr->nevals;
// otherwise writes them at cursor (cand_cap slots)
cudaError_t launch_arr_gather3d(const SegRec3 *segs, unsigned long long nseg, const GroupDev *groups, int ngroups,
                                bool count, ArrCand *cands, uint64_t *keys, uint32_t *vals,
                                unsigned long long cand_cap, unsigned long long *cursor, RunCounters *ctr,
                                ArrKeyBits kb, int grid, cudaStream_t st)
{
    if(nseg == 0) return cudaSuccess;
    grid = grid * 4 / WARPS3;
    if(kb.eigen) {
        if(count)
            influence3d_kernel<INFL_EIG_COUNT><<<grid, 32 * WARPS3, 0, st>>>(segs, nseg, groups, ngroups, nullptr,
                                                                             ctr, nullptr, nullptr, nullptr, 0, nullptr,
                                                                             kb);
        else
            influence3d_kernel<INFL_EIG_FILL><<<grid, 32 * WARPS3, 0, st>>>(segs, nseg, groups, ngroups, nullptr,
                                                                            ctr, cands, keys, vals, cand_cap, cursor,
                                                                            kb);
    } else if(count)
        influence3d_kernel<INFL_ARR_COUNT><<<grid, 32 * WARPS3, 0, st>>>(segs, nseg, groups, ngroups, nullptr, ctr,
                                                                         nullptr, nullptr, nullptr, 0, nullptr, kb);
    else
        influence3d_kernel<INFL_ARR_FILL><<<grid, 32 * WARPS3, 0, st>>>(segs, nseg, groups, ngroups, nullptr, ctr,
                                                                        cands, keys, vals, cand_cap, cursor, kb);
    return cudaGetLastError();
}

cudaError_t launch_sqrt3d(float2 *f, long long n, int grid, cudaStream_t st)
{
    if(n <= 0) return cudaSuccess;
    sqrt3d_kernel<<<grid, 256, 0, st>>>(f, n);
    return cudaGetLastError();
}

cudaError_t launch_eigen_emit3(const uint32_t *vals, const ArrCand *cands, unsigned long long n,
                               const GroupDev *groups, int ngroups, EigenHitRec *hits, int32_t *group_of_hit,
                               int sm_count, cudaStream_t st)
{
    if(n == 0) return cudaSuccess;
    long long grid = (long long)((n + 255) / 256);
    if(grid > (long long)sm_count * 32) grid = (long long)sm_count * 32;
    eigen_emit3_kernel<<<(int)grid, 256, 0, st>>>(vals, cands, n, groups, ngroups, hits, group_of_hit);
    return cudaGetLastError();
}

} // namespace bhcb
