// What a 3-D or Nx2D ray carries from step to step beside its state, arranged
// for the latency of one ray (as ray2seg.cuh does for 2-D): the current cell of
// the sound-speed grid with its corner values, the boundary cells with the unit
// normals of their diagonals, and a box inside which no boundary, beam-box or
// cell-face test of the step can hold. Inside the box a step tests the profile
// interfaces and the two cell diagonals, outside it everything. Operands and
// roundings are those of the general routines of trace3d.cuh, so trajectories
// and step counts are the same.
//
// A trace is bound by the chain of its longest rays, and here by instruction
// fetch: of the general step's 14 cycles per instruction 9 wait for it. Per
// step the general routines evaluate the grid three times with index searches,
// test ten crossings for each of two reductions and the landing (six times with
// a square root and divisions for the diagonals' normals), search the boundary
// cells twice, and form the second derivatives of the sound speed along the ray
// normals, which are zero in a trilinear ocean. Trace times, general -> this:
// 51,984 rays through the hexahedral ocean 86 -> 42 ms, 13,032 rays 42 -> 25,
// 1,113 rays 31 -> 11. One ray's instructions fell from about 4,000 to 1,600 a
// step. Calls in place of the crossing tests were slower (144 ms: a call spills
// the ray's state), three copies of them as well (47 ms), and so were warps kept
// in step by a barrier (44 ms).
#pragma once
#include "trace3d.cuh"

namespace bhcb {

// Rays per warp of a 3-D or Nx2D trace: as few as keep the warps of all rays in
// flight at once, 6 per SM (plan_lanes has the reasons and the 2-D figures), or 1
// per SM where the launch takes the general step (walk false: a batch of hexahedral
// and 1-D oceans), whose code outgrows the instruction caches, so that warps delay
// one another. 6 and 1 per SM, and 32 rays a warp in brackets: 558 rays 5.5 and 5.1
// ms (6.3), 4514 rays 9.8 and 5.8 (5.9), 10010 rays 11.8 and 8.8 (8.7).
inline int lanes3(long long njobs, int sm_count, bool walk)
{
    const long long warps = (walk ? 6LL : 1LL) * sm_count;
    int l = 1;
    while(l < 32 && (njobs + l - 1) / l > warps) l *= 2;
    return l;
}

// Sound speed at a point: value, gradient, depth curvature, and the
// reciprocals of c and c^2 for quotients.
struct Prof3 {
    V3 g;
    double c, ci, czz, rc, rcsq;
};

// The deepest (sign > 0) or shallowest (sign < 0) depth of the planes of both
// triangles of the cell with corner node p over the rectangle d0..d1 from it;
// NaN when a plane is steep or faces the wrong way.
__device__ __forceinline__ double plane_extreme(const Bdry3PtDev *p, double z, double dx0, double dx1, double dy0,
                                             double dy1, double sign)
{
    double e = -1.7976931348623157e308;
    for(int k = 0; k < 2; ++k) {
        const V3 m = k ? ld3(p->n2) : ld3(p->n1);
        if(!(-sign * m.z > 0.05)) return NAN;
        const double r = 1.0 / m.z, ax = m.x * r, ay = m.y * r;
        e = max(e, max(max(sign * (z - (ax * dx0 + ay * dy0)), sign * (z - (ax * dx1 + ay * dy0))),
                       max(sign * (z - (ax * dx0 + ay * dy1)), sign * (z - (ax * dx1 + ay * dy1)))));
    }
    return sign * e;
}

// What a ray keeps of a boundary cell (Bd3): its index, its centre, the unit
// normals of its diagonal and the side the ray is on. Corner, limits and
// triangle normals are read from the grid when a test needs them.
struct Bd3w {
    int ix, iy;
    double xm, ym;           // cell centre
    double sx, sy;           // unit normal of the diagonal, divided (get_bdry_seg3)
    double tx, ty;           // the same, scaled by the reciprocal (tridiag3)
    bool onEdge, side, justSteppedTo, outgoingSide;

    __device__ __forceinline__ const Bdry3PtDev *corner(const Bdry3PtDev *bd, int ny) const
    {
        return bd + (size_t)ix * ny + iy;
    }
    __device__ __forceinline__ V3 normal(const Bdry3PtDev *bd, int ny) const
    {
        const Bdry3PtDev *p = corner(bd, ny);
        return side ? ld3(p->n2) : ld3(p->n1);
    }
    // the cell's centre and diagonal; a node that is not finite is an error
    __device__ __forceinline__ void load(const Bdry3PtDev *bd, int ny, RunCounters *ctr)
    {
        const Bdry3PtDev *p = corner(bd, ny), *q = p + ny + 1;
        const double x0 = p->x[0], y0 = p->x[1], x1 = bd[(size_t)(ix + 1) * ny].x[0], y1 = bd[iy + 1].x[1];
        xm = 0.5 * (x0 + q->x[0]);
        ym = 0.5 * (y0 + q->x[1]);
        const double a = -(y1 - bd[iy].x[1]), b = x1 - bd[(size_t)ix * ny].x[0];
        const double l = sqrt(a * a + b * b), r = 1.0 / l;
        sx = a / l;
        sy = b / l;
        tx = r * a;
        ty = r * b;
        if(!isfinite(p->x[2])) run_error(ctr, ERR_BOUNDARY_SEG_NAN);
    }
    __device__ __forceinline__ void check(const Bdry3PtDev *bd, int ny, RunCounters *ctr) const
    {
        const V3 n = normal(bd, ny);
        if(!isfinite(n.x) || !isfinite(n.y) || !isfinite(n.z)) run_error(ctr, ERR_BOUNDARY_SEG_NAN);
    }
    // the end of get_bdry_seg3: the active triangle at x
    __device__ __forceinline__ bool settle(V3 x, V3 t)
    {
        const double over = (x.x - xm) * sx + (x.y - ym) * sy;
        onEdge = fabs(over) < 3e-6;
        const bool was = side;
        if(justSteppedTo) side = outgoingSide;
        else if(onEdge) side = (t.x * sx + t.y * sy) >= 0.0;
        else side = over >= 0.0;
        justSteppedTo = false;
        return side != was;
    }
    // get_bdry_seg3 for an x outside the cell or on its limits: the search
    __device__ __forceinline__ bool search(V3 x, V3 t, const Bdry3PtDev *bd, int nx, int ny, bool istop, RunCounters *ctr)
    {
        int i = ix, j = iy;
        if(t.x >= 0.0) {
#pragma unroll 1
            while(i >= 0 && bd[(size_t)i * ny].x[0] > x.x) --i;
#pragma unroll 1
            while(i >= 0 && i < nx - 1 && bd[(size_t)(i + 1) * ny].x[0] <= x.x) ++i;
        } else {
#pragma unroll 1
            while(i < nx - 1 && bd[(size_t)(i + 1) * ny].x[0] < x.x) ++i;
#pragma unroll 1
            while(i >= 0 && i < nx - 1 && bd[(size_t)i * ny].x[0] >= x.x) --i;
        }
        if(t.y >= 0.0) {
#pragma unroll 1
            while(j >= 0 && bd[j].x[1] > x.y) --j;
#pragma unroll 1
            while(j >= 0 && j < ny - 1 && bd[j + 1].x[1] <= x.y) ++j;
        } else {
#pragma unroll 1
            while(j < ny - 1 && bd[j + 1].x[1] < x.y) ++j;
#pragma unroll 1
            while(j >= 0 && j < ny - 1 && bd[j].x[1] >= x.y) --j;
        }
        if(i == -1 && bd[0].x[0] == x.x) i = 0;
        if(i == nx - 1 && bd[(size_t)(nx - 1) * ny].x[0] == x.x) i = nx - 2;
        if(j == -1 && bd[0].x[1] == x.y) j = 0;
        if(j == ny - 1 && bd[ny - 1].x[1] == x.y) j = ny - 2;
        if(i < 0 || i >= nx - 1 || j < 0 || j >= ny - 1) {
            run_warn(ctr, istop ? WARN_OUTSIDE_ALTIMETRY : WARN_OUTSIDE_BATHYMETRY);
            i = min(max(i, 0), nx - 2);
            j = min(max(j, 0), ny - 2);
        }
        const bool moved = i != ix || j != iy;
        ix = i;
        iy = j;
        return moved;
    }
    // tridiag3: whether the way from p along u to x crosses the diagonal, and
    // the step to it
    __device__ __forceinline__ bool crosses(V3 x) const
    {
        const double over = (x.x - xm) * tx + (x.y - ym) * ty;
        return !onEdge && (over >= 0.0) != side && !(fabs(over) < 3e-6);
    }
    __device__ __forceinline__ double step_to(V3 p, V3 u) const
    {
        return div_rn(-((p.x - xm) * tx + (p.y - ym) * ty), u.x * tx + u.y * ty);
    }
};

// update_seg in few instructions (the loops run once or not at all)
__device__ __forceinline__ void walk_seg(double x, bool tpos, const double *a, int n, int &i)
{
#pragma unroll 1
    for(;;) {
        const double lo = a[i], hi = a[i + 1];
        const bool dn = i > 0 && (tpos ? x < lo : x <= lo), up = i < n - 2 && (tpos ? x >= hi : x > hi);
        if(!(dn || up)) return;
        i += up ? 1 : -1;
    }
}

// HEX: hexahedral grid; else a 1-D profile in depth.
template<bool HEX> struct Walk3 {
    const Env3Dev *E;
    V3 xs;
    double deltas, hmin;
    Bd3w top, bot;
    Seg3 s;                              // sound-speed cell
    double x0, x1, y0, y1, z0, z1;       // its limits (HEX)
    double dx, dy, rdx, rdy;
    double k11, k21, k12, k22, g11, g12, g21, g22;   // corner values and depth gradients
    SspSegCache sc;                      // 1-D
    double bx0, bx1, by0, by1, bz0, bz1; // the box
    bool dirty;                          // a cell has changed since the box was set
    double za, zb;                       // profile interfaces of the step's start

    __device__ __forceinline__ void load_cell()
    {
        const Env3Dev &e = *E;
        const int ny = e.hny, nz = e.hnz;
        const size_t a = (size_t)s.x * ny + s.y, b = (size_t)(s.x + 1) * ny + s.y;
        g11 = e.hcz[a * (nz - 1) + s.z];
        g12 = e.hcz[b * (nz - 1) + s.z];
        g21 = e.hcz[(a + 1) * (nz - 1) + s.z];
        g22 = e.hcz[(b + 1) * (nz - 1) + s.z];
        k11 = e.hc[a * nz + s.z];
        k21 = e.hc[b * nz + s.z];
        k12 = e.hc[(a + 1) * nz + s.z];
        k22 = e.hc[(b + 1) * nz + s.z];
        z0 = e.hz[s.z];
        z1 = e.hz[s.z + 1];
    }
    __device__ __forceinline__ void load_column()
    {
        const Env3Dev &e = *E;
        x0 = e.hx[s.x];
        x1 = e.hx[s.x + 1];
        y0 = e.hy[s.y];
        y1 = e.hy[s.y + 1];
        dx = x1 - x0;
        dy = y1 - y0;
        rdx = rcp_rn(dx);
        rdy = rcp_rn(dy);
        dirty = true;
    }
    // a new profile cell
    __device__ __forceinline__ void set_cell(const Seg3 &n)
    {
        const Seg3 o = s;
        s = n;
        if(!HEX) return;
        if(s.x != o.x || s.y != o.y) load_column();
        if(s.x != o.x || s.y != o.y || s.z != o.z) load_cell();
    }
    // eval_ssp3's arithmetic on the cell (the clamps of the weights act only
    // outside the grid, which is an error)
    __device__ __forceinline__ void eval(V3 x, V3 t, Prof3 &o, RunCounters *ctr)
    {
        if(HEX) {
            if(!(x.z > z0 && x.z < z1 && x.x > x0 && x.x < x1 && x.y > y0 && x.y < y1)) {
                const Env3Dev &e = *E;
                if(x.x < e.hx[0] || x.x > e.hx[e.hnx - 1] || x.y < e.hy[0] || x.y > e.hy[e.hny - 1])
                    run_error(ctr, ERR_OUTSIDE_SSP);
                Seg3 n = s;   // update_seg (src/ssp.hpp:36-51)
                walk_seg(x.x, t.x >= 0.0, e.hx, e.hnx, n.x);
                walk_seg(x.y, t.y >= 0.0, e.hy, e.hny, n.y);
                walk_seg(x.z, t.z >= 0.0, e.hz, e.hnz, n.z);
                set_cell(n);
            }
            const double s3 = x.z - z0;
            const double c11 = k11 + s3 * g11, c21 = k21 + s3 * g12, c12 = k12 + s3 * g21, c22 = k22 + s3 * g22;
            const double s1 = quot_rn(x.x - x0, dx, rdx), s2 = quot_rn(x.y - y0, dy, rdy);
            double c1 = c11 + s1 * (c21 - c11), c2 = c12 + s1 * (c22 - c12);
            o.g.y = quot_rn(c2 - c1, dy, rdy);
            c1 = c11 + s2 * (c12 - c11);
            c2 = c21 + s2 * (c22 - c21);
            o.c = c1 + s1 * (c2 - c1);
            o.g.x = quot_rn(c2 - c1, dx, rdx);
            const double e1 = g11 + s2 * (g21 - g11), e2 = g12 + s2 * (g22 - g12);
            o.g.z = e1 + s1 * (e2 - e1);
            o.ci = 0.0;
            o.czz = 0.0;
        } else {
            SSPOut<double> p;
            SegState s2{0, s.z};
            eval_ssp_cached(mk2(0.0, x.z), mk2(0.0, t.z), p, E->e1d, s2, sc, ctr);
            s.z = s2.z;
            o.g = v3(0.0, 0.0, p.gradc.y);
            o.c = p.c;
            o.ci = p.ci;
            o.czz = p.czz;
        }
        o.rc = rcp_rn(o.c);
        o.rcsq = rcp_square(o.c * o.c, o.rc);
    }
    // range of x (y) that the boundary cells and the profile cell of the step's
    // start share (cellseg3)
    __device__ __forceinline__ void faces(bool y, int sw, double &lo, double &hi) const
    {
        const Env3Dev &e = *E;
        const Bdry3PtDev *t = e.btop, *b = e.bbot;
        if(y) {
            lo = max(t[top.iy].x[1], b[bot.iy].x[1]);
            hi = min(t[top.iy + 1].x[1], b[bot.iy + 1].x[1]);
        } else {
            lo = max(t[(size_t)top.ix * e.top_ny].x[0], b[(size_t)bot.ix * e.bot_ny].x[0]);
            hi = min(t[(size_t)(top.ix + 1) * e.top_ny].x[0], b[(size_t)(bot.ix + 1) * e.bot_ny].x[0]);
        }
        if(HEX) {
            const double *w = y ? e.hy : e.hx;
            lo = max(lo, w[sw]);
            hi = min(hi, w[sw + 1]);
        }
    }
    __device__ __forceinline__ double extreme(const Bd3w &b, const Bdry3PtDev *bd, int ny, double sign) const
    {
        const Bdry3PtDev *p = b.corner(bd, ny);
        return plane_extreme(p, p->x[2], bd[(size_t)b.ix * ny].x[0] - p->x[0], bd[(size_t)(b.ix + 1) * ny].x[0] - p->x[0],
                             bd[b.iy].x[1] - p->x[1], bd[b.iy + 1].x[1] - p->x[1], sign);
    }
    __device__ __forceinline__ void set_box()
    {
        const Env3Dev &e = *E;
        double l, h;
        faces(false, s.x, l, h);
        bx0 = max(l, xs.x - e.box_x + 1.0e-3);
        bx1 = min(h, xs.x + e.box_x - 1.0e-3);
        faces(true, s.y, l, h);
        by0 = max(l, xs.y - e.box_y + 1.0e-3);
        by1 = min(h, xs.y + e.box_y - 1.0e-3);
        const double zt = extreme(top, e.btop, e.top_ny, 1.0), zl = extreme(bot, e.bbot, e.bot_ny, -1.0);
        bz0 = max(zt + 1.0e-3, -e.box_z + 1.0e-3);
        bz1 = min(zl - 1.0e-3, e.box_z - 1.0e-3);
        if(!(zt == zt && zl == zl)) bz0 = 1.7976931348623157e308;   // no box
        dirty = false;
    }
    __device__ __forceinline__ bool holds(V3 x) const
    {
        return x.x > bx0 && x.x < bx1 && x.y > by0 && x.y < by1 && x.z > bz0 && x.z < bz1;
    }
    __device__ __forceinline__ void from_general(Bd3w &w, const Bd3 &b, const Bdry3PtDev *bd, int ny, RunCounters *ctr)
    {
        w.ix = b.ix;
        w.iy = b.iy;
        w.onEdge = b.onEdge;
        w.side = b.side;
        w.justSteppedTo = b.justSteppedTo;
        w.outgoingSide = b.outgoingSide;
        w.load(bd, ny, ctr);
    }
    // start of the ray: boundary cells and profile cell as RayInit found them
    __device__ __forceinline__ void init(const Env3Dev &env, V3 src, const Bd3 &t, const Bd3 &b, const Seg3 &seg,
                                         RunCounters *ctr)
    {
        E = &env;
        xs = src;
        deltas = env.deltas;
        hmin = INF_STEP * env.deltas;
        from_general(top, t, env.btop, env.top_ny, ctr);
        from_general(bot, b, env.bbot, env.bot_ny, ctr);
        s = seg;
        if(HEX) {
            load_column();
            load_cell();
        } else {
            ssp_cache_init(sc, env.e1d);
        }
        dirty = true;
    }
    // start of a step: the interfaces above and below (none past the first /
    // last layer), and the box
    __device__ __forceinline__ void begin()
    {
        const double *z = E->e1d.z;
        za = s.z > 0 ? z[s.z] : -1.7976931348623157e308;
        zb = s.z + 1 < E->e1d.nssp - 1 ? z[s.z + 1] : 1.7976931348623157e308;
        if(dirty) set_box();
    }
    // signed distance of x beyond a boundary plane, and the step to the plane
    __device__ __forceinline__ double beyond(V3 x, const double *c, V3 n) const
    {
        return n.x * (x.x - c[0]) + n.y * (x.y - c[1]) + n.z * (x.z - c[2]);
    }
    // dot3(x - c, n) in topbot3's order
    __device__ __forceinline__ double beyond_dot(V3 x, const double *c, V3 n) const
    {
        return dot3(sub3(x, ld3(c)), n);
    }
    // The crossings on the way from p along u, in one copy of the code for
    // reduce_step3 (landing false: x2 stays p + h u, h becomes the shortest
    // step) and step_to_bdry3 (landing true: x2 is put onto what it meets, one
    // after the other); s0: the cell at the start of the step. Returns whether
    // the landing point is inside the box.
    __device__ __forceinline__ bool cross(bool landing, V3 p, V3 u, double &h, V3 &x2, bool &tr, bool &br,
                                          const Seg3 &s0, int &snap, int &small, RunCounters *ctr)
    {
        const Env3Dev &env = *E;
        double hn = h;   // reduction: the shortest step so far
        x2 = add3(p, scl3(h, u));
        snap = -1;
        tr = br = false;
        // a crossing at step c: taken over (true: x2 is there) or noted
        auto meet = [&](double c, int sn) {
            if(!landing) {
                hn = c < hn ? c : hn;
                return false;
            }
            h = c;
            x2 = add3(p, scl3(h, u));
            snap = sn;
            return true;
        };
        {
            const bool above = za > x2.z;
            if((above || zb < x2.z) && fabs(u.z) > DBL_EPS) {
                const double zn = above ? za : zb;
                if(meet(div_rn(zn - p.z, u.z), 2)) x2.z = zn;
            }
        }
        if(!holds(x2)) {
            if(fabs(x2.x - xs.x) >= env.box_x && meet(div_rn(env.box_x - fabs(p.x - xs.x), fabs(u.x)), 0))
                x2.x = xs.x + copysign(env.box_x, p.x - xs.x);
            if(fabs(x2.y - xs.y) >= env.box_y && meet(div_rn(env.box_y - fabs(p.y - xs.y), fabs(u.y)), 1))
                x2.y = xs.y + copysign(env.box_y, p.y - xs.y);
            if(fabs(x2.z) >= env.box_z && meet(div_rn(env.box_z - fabs(p.z), fabs(u.z)), 2))
                x2.z = copysign(env.box_z, p.z);
#pragma unroll 1
            for(int k = 0; k < 2; ++k) {
                const double *c = k ? bot.corner(env.bbot, env.bot_ny)->x : top.corner(env.btop, env.top_ny)->x;
                const V3 n = k ? bot.normal(env.bbot, env.bot_ny) : top.normal(env.btop, env.top_ny);
                const double w = beyond(x2, c, n);
                if(landing ? w > -INF_STEP : w >= 0.0) {
                    if(meet(div_rn(-beyond_dot(p, c, n), dot3(u, n)), 2)) {
                        if(fabs(n.x) < DBL_EPS && fabs(n.y) < DBL_EPS) x2.z = c[2];
                        tr = k == 0;
                        br = k == 1;
                    }
                }
            }
#pragma unroll 1
            for(int k = 0; k < 2; ++k) {
                double l, r;
                faces(k, k ? s0.y : s0.x, l, r);
                const double xw = k ? x2.y : x2.x, uw = k ? u.y : u.x;
                if((xw < l || xw > r) && fabs(uw) > DBL_EPS) {
                    const double f = xw < l ? l : r;
                    if(meet(div_rn(-((k ? p.y : p.x) - f), uw), k)) {
                        if(k) x2.y = f; else x2.x = f;
                        tr = br = false;
                    }
                }
            }
        }
#pragma unroll
        for(int k = 0; k < 2; ++k) {
            Bd3w &b = k ? bot : top;
            if(!b.crosses(x2)) continue;
            const double c = b.step_to(p, u);
            if(c < 0.0) run_warn(ctr, WARN_TRIDIAG_H_NEGATIVE);
            else if(landing && c >= h) run_warn(ctr, WARN_TRIDIAG_H_GROWING);
            const bool side = (x2.x - b.xm) * b.tx + (x2.y - b.ym) * b.ty >= 0.0;
            if(meet(c < 0.0 ? 0.0 : c, -2)) {
                b.justSteppedTo = true;
                b.outgoingSide = side;
                tr = br = false;
            }
        }
        if(!landing) {
            h = hn;
            if(h < hmin) {
                if(h < -1e-4) run_warn(ctr, WARN_STEP_NEGATIVE_H);
                h = hmin;
                ++small;
            } else {
                small = 0;
            }
            return false;
        }
        if(h < hmin) {
            h = hmin;
            x2 = add3(p, scl3(h, u));
            snap = -1;
            tr = br = false;
            const double *ct = top.corner(env.btop, env.top_ny)->x, *cb = bot.corner(env.bbot, env.bot_ny)->x;
            if(beyond(x2, ct, top.normal(env.btop, env.top_ny)) > DBL_EPS) {
                tr = true;
                top.justSteppedTo = bot.justSteppedTo = false;
                snap = 2;
            }
            if(beyond(x2, cb, bot.normal(env.bbot, env.bot_ny)) > DBL_EPS) {
                br = true;
                tr = false;
                top.justSteppedTo = bot.justSteppedTo = false;
                snap = 2;
            }
        }
        return holds(x2);
    }
    __device__ __forceinline__ void follow(Bd3w &b, bool inside, V3 x, V3 t, const Bdry3PtDev *bd, int nx, int ny,
                                           bool istop, RunCounters *ctr)
    {
        bool look = false;
        if(!inside && b.search(x, t, bd, nx, ny, istop, ctr)) {
            b.load(bd, ny, ctr);
            dirty = look = true;
        }
        if(b.settle(x, t) || look) b.check(bd, ny, ctr);
    }
    // RayUpdate's boundary segments at the end of the step
    __device__ __forceinline__ void boundaries(bool inside, V3 x, V3 t, RunCounters *ctr)
    {
        follow(top, inside, x, t, E->btop, E->top_nx, E->top_ny, true, ctr);
        follow(bot, inside, x, t, E->bbot, E->bot_nx, E->bot_ny, false, ctr);
    }
    // the general routines' form of a boundary cell
    __device__ __forceinline__ Bd3 general(const Bd3w &w, const Bdry3PtDev *bd, int ny) const
    {
        Bd3 b;
        const Bdry3PtDev *p = w.corner(bd, ny);
        b.ix = w.ix;
        b.iy = w.iy;
        b.xmin = bd[(size_t)w.ix * ny].x[0];
        b.xmax = bd[(size_t)(w.ix + 1) * ny].x[0];
        b.ymin = bd[w.iy].x[1];
        b.ymax = bd[w.iy + 1].x[1];
        b.x = ld3(p->x);
        b.xmid = scl3(0.5, add3(b.x, ld3(p[ny + 1].x)));
        b.n = w.normal(bd, ny);
        b.onEdge = w.onEdge;
        b.side = w.side;
        b.justSteppedTo = w.justSteppedTo;
        b.outgoingSide = w.outgoingSide;
        return b;
    }
};

// the general forms, for directions along the vertical or along a face
static __device__ __noinline__ void normal_cold(V3 t, double phi, V3 &e1, V3 &e2) { ray_normal(t, phi, true, 1.0, e1, e2); }
static __device__ __noinline__ void face_cold(Ray3 &r, V3 gj, Seg3 s, Seg3 s0) { interface_corr3(r, gj, s, s0); }

// ray_normal of a unit tangent (ignorephi0 = true, c = 1); cp, sp: cos and sin of phi
__device__ __forceinline__ void ray_normal_unit(V3 t, double phi, double cp, double sp, V3 &e1, V3 &e2)
{
    const double rl2 = t.x * t.x + t.y * t.y;
    if(!(rl2 > 1.0e-280)) {
        V3 a, b;
        normal_cold(t, phi, a, b);
        e1 = a;
        e2 = b;
        return;
    }
    const double rl = sqrt_rn(rl2), r = rcp_rn(rl);
    e1.x = quot_rn(t.x * t.z * cp + t.y * sp, rl, r);
    e1.y = quot_rn(t.y * t.z * cp - t.x * sp, rl, r);
    e1.z = -rl * cp;
    e2.x = quot_rn(t.x * t.z * sp - t.y * cp, rl, r);
    e2.y = quot_rn(t.y * t.z * sp + t.x * cp, rl, r);
    e2.z = -rl * sp;
}

// interface_corr3 at a face between cells (CurvatureCorrection3D with D = 0)
__device__ __forceinline__ void face_corr3(Ray3 &r, double rcsq, V3 gj, const Seg3 &s, const Seg3 &s0, double cp,
                                           double sp)
{
    V3 nB = v3(0.0, 0.0, 0.0);
    if(s.z != s0.z) nB.z = -copysign(1.0, r.t.z);
    else if(s.x != s0.x) nB.x = -copysign(1.0, r.t.x);
    else nB.y = -copysign(1.0, r.t.y);
    const double Th = dot3(r.t, nB);
    V3 tB = sub3(r.t, scl3(Th, nB));
    const double l2 = dot3(tB, tB);
    const V3 rayt = scl3(r.c, r.t);
    if(!(l2 > 1.0e-280 && fabs(Th) > 1.0e-100 && rayt.x * rayt.x + rayt.y * rayt.y > 1.0e-280)) {
        Ray3 c = r;
        face_cold(c, gj, s, s0);
        r.p = c.p;
        return;
    }
    tB = scl3(div_rn(1.0, sqrt_rn(l2)), tB);
    const double Tg = dot3(r.t, tB);
    V3 rayn2 = cross3(rayt, nB);
    rayn2 = scl3(div_rn(1.0, sqrt_rn(dot3(rayn2, rayn2))), rayn2);
    const V3 rayn1 = scl3(-1.0, cross3(rayt, rayn2));
    V3 e1, e2;
    ray_normal_unit(rayt, r.phi, cp, sp, e1, e2);
    const double cn1j = dot3(gj, rayn1), cn2j = dot3(gj, rayn2), csj = dot3(gj, rayt);
    const double rm = div_rn(Tg, Th), csq = r.c * r.c;
    M2 R;
    R.m[0][0] = -quot_rn(rm * (2.0 * cn1j - rm * csj), csq, rcsq);
    R.m[0][1] = R.m[1][0] = -quot_rn(rm * cn2j, csq, rcsq);
    R.m[1][1] = 0.0;
    M2 Rot;
    Rot.m[0][0] = dot3(rayn1, e1);
    Rot.m[1][0] = dot3(rayn1, e2);
    Rot.m[0][1] = -Rot.m[1][0];
    Rot.m[1][1] = dot3(rayn2, e2);
    const M2 pin = m2_mul(Rot, r.p);
    const M2 qin = m2_mul(Rot, r.q);
    r.p = m2_mul(m2_T(Rot), m2_add(pin, m2_mul(R, qin)));
}

} // namespace bhcb
