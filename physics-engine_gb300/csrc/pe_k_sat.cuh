// Kernels of the rigid-body step, part 4: the convex SAT and face clipping (staged, pruned, and
// the contact step).
#pragma once
#include "pe_k_narrowphase.cuh"

namespace pe {

// ---------------------------------------------------------------- warp-cooperative SAT
// (convex_convex_collision_algorithm.cpp:251-432) for cylinder-cylinder, box-hull and hull-hull:
// one warp per pair, lanes over candidate axes.  The reference scans axes in order and keeps
// the first strictly smaller depth; that is the lexicographic minimum of (depth, axis index),
// which the warp reduces.  Any separating axis ends the test (the reference returns at the
// first one it meets; what it computed before that is discarded except the corner point).
template <class R> __device__ __forceinline__ void warp_argmin(R& d, int& idx) {
    for (int o = 16; o > 0; o >>= 1) {
        const R od = __shfl_xor_sync(0xffffffffu, d, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (od < d || (od == d && oi < idx)) { d = od; idx = oi; }
    }
}
template <class R> __device__ __forceinline__ void warp_min(R& d) {
    for (int o = 16; o > 0; o >>= 1) {
        const R od = __shfl_xor_sync(0xffffffffu, d, o);
        if (od < d) d = od;
    }
}
template <class R> __device__ __forceinline__ void warp_argmax(R& d, int& idx) {
    for (int o = 16; o > 0; o >>= 1) {
        const R od = __shfl_xor_sync(0xffffffffu, d, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (od > d || (od == d && oi < idx)) { d = od; idx = oi; }
    }
}
template <class R> __device__ __forceinline__ V3<R> shfl3(const V3<R>& v, int src) {
    return V3<R>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src), __shfl_sync(0xffffffffu, v.z, src));
}

__device__ __forceinline__ V3<float> ldv(const float* p, int i) {
    const float4 f = reinterpret_cast<const float4*>(p)[i];
    return V3<float>(f.x, f.y, f.z);
}
__device__ __forceinline__ V3<double> ldv(const double* p, int i) {
    const double2* q = reinterpret_cast<const double2*>(p) + 2 * i;
    const double2 a = q[0], b = q[1];
    return V3<double>(a.x, a.y, b.x);
}
template <class R> __device__ __forceinline__ void stv(R* p, int i, const V3<R>& v) {
    p[4 * i] = v.x; p[4 * i + 1] = v.y; p[4 * i + 2] = v.z; p[4 * i + 3] = R(0);
}


// support interval of a shape along a world axis (Shape::project without the witness points);
// for hulls the indices of the witness vertices are returned (the first vertex never becomes
// the maximum, like convex_mesh_shape.cpp:171-175)
template <class R>
__device__ __forceinline__ void shape_interval(const ShapeView<R>& s, const Xf<R>& t, const V3<R>& axis, const R* lv, R& mnp, R& mxp,
                                               int& imn, int& imx) {
    if (s.type == ST_SPHERE) {
        const R off = dot(t.o, axis);
        mnp = off - s.radius; mxp = off + s.radius;
        return;
    }
    const V3<R> la = mtv(t.b, axis);
    const R off = dot(t.o, axis);
    if (s.type == ST_BOX) {
        const V3<R> ext(la.x > 0 ? s.half.x : -s.half.x, la.y > 0 ? s.half.y : -s.half.y, la.z > 0 ? s.half.z : -s.half.z);
        const R he = dot(ext, la);
        mnp = off - he; mxp = off + he;
        return;
    }
    if (s.type == ST_CYLINDER) {
        const R hh = s.height * R(0.5);
        if (rabs(la.x - 0) < eps<R>() && rabs(la.z - 0) < eps<R>()) { mnp = off - hh; mxp = off + hh; }
        else if (rabs(la.y - 0) < eps<R>()) { mnp = off - s.radius; mxp = off + s.radius; }
        else {
            const R r = real_sqrt(la.x * la.x + la.z * la.z);
            const R x = s.radius * la.x / r, z = s.radius * la.z / r;
            const R y = hh * (la.y > 0 ? 1 : -1);
            const R el = dot(V3<R>(x, y, z), la);
            mnp = off - el; mxp = off + el;
        }
        return;
    }
    mnp = Lim<R>::max();
    mxp = Lim<R>::min();
    imn = -1; imx = -1;
    for (int i = 0; i < s.nv; i++) {
        const R v = dot(ldv(lv, i), la);
        if (v < mnp) { mnp = v; imn = i; }
        else if (v > mxp) { mxp = v; imx = i; }
    }
    mnp += off;
    mxp += off;
}

// witness point of Shape::project on the min (want_max = false) or max side
template <class R>
__device__ V3<R> shape_witness(const ShapeView<R>& s, const Xf<R>& t, const V3<R>& axis, bool want_max, int idx, const R* lv) {
    R a, b;
    V3<R> pmin, pmax;
    if (s.type == ST_HULL) {
        // an index never set leaves the reference's witness undefined; that only happens on a
        // separating axis, whose witness is never used
        const V3<R> p = idx >= 0 ? ldv(lv, idx) : V3<R>(0, 0, 0);
        return t.apply(p);
    }
    shape_project(s, t, axis, a, b, pmin, pmax);
    return want_max ? pmax : pmin;
}

// ---- staged SAT: bounds first, exact projections for what the bounds leave.
//
// The pair's minimum depth decides everything, and few axes come near it.  For every candidate axis a
// cheap lower bound of its overlap depth is taken (fused multiply-adds, unnormalised axes, a few
// supporting points per hull), and only axes whose bound does not exceed a depth the pair is known to
// reach are queued and projected with the reference's formulas (Shape::project, the same bits).  A
// skipped axis is certainly above that depth, so it can neither separate the pair nor be its first
// minimum, and candidates compare by (depth, reference axis index), the reference's first strict
// minimum in any visiting order.
//
// What bounds it is instruction fetch and issue: 32 axes cost about 60 instructions for the bound (two
// hulls' edge pairs mostly some 25, see `hulls`), and most pairs one round of exact projections for the
// faces and one for the edges.  Per step of the 4,096 piles, before (every axis past a ball test projected
// exactly, two per lane) and now: hull-hull 1,750 / 521 us, its heavy pairs 778 / 297, box-hull
// 2,311 / 1,286, hull-box 699 / 411, cylinder-cylinder 935 / 245.

// One side's bound data.  rel: the support points are taken relative to the shape's own origin.
constexpr int kSub = 8;          // supporting points per hull
template <class R> struct SatSide {
    V3<R> e0, e1, e2;            // box: half axes; cylinder: e0 the unit axis
    R r, hh;                     // cylinder
    R inner;                     // a ball about the origin inside the shape (<= 0: none)
    R mag;                       // bound of the distances entering the projections' rounding
};
constexpr int kSatBase = 4 * (kSub + 2);   // reals of one hull's supporting points: kSub of them, then vertices 0 and 1
template <class R> __device__ __forceinline__ R fma3(const V3<R>& a, const V3<R>& b) { return fma(a.z, b.z, fma(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ float fast_sqrt(float x) { float r; asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ double fast_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float fast_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double fast_max(double a, double b) { return fmax(a, b); }
template <class R> constexpr R sat_slack() { return sizeof(R) == 4 ? R(96 * 1.1920929e-7) : R(96 * 2.220446049250313e-16); }

// Lower bound of the support of a shape along y (of length ny): box and cylinder in closed form (a
// cylinder lowered by what the reference's branches for nearly axial and nearly radial axes drop: they
// take the half height or the radius whatever the axis's length, and one normal of the cylinder mesh is
// 1.0188 long), a hull by its supporting points.  For the second shape (QUIRK) a hull's bound counts only when vertex 0
// or 1, which come before every supporting point, lies below it: the reference never lets a new
// minimum become the maximum (convex_mesh_shape.cpp:171-175), and a point above an earlier vertex is no
// new minimum.
template <class R, int T, bool QUIRK>
__device__ __forceinline__ R sat_support(int type, const SatSide<R>& s, const V3<R>& y, R ny, const R* sub, R slack) {
    const int t = T >= 0 ? T : type;
    if (t == ST_BOX) return rabs(fma3(y, s.e0)) + rabs(fma3(y, s.e1)) + rabs(fma3(y, s.e2));
    if (t == ST_CYLINDER) {
        const R c = fma3(y, s.e0);
        const R n2 = ny * ny;   // the axis's part across the cylinder's, its square lowered by its own roundoff
        return fma(s.hh, rabs(c), s.r * fast_sqrt(fast_max(fma(-c, c, n2) - R(0.125) * sat_slack<R>() * n2, R(0)))) -
               (s.r + s.hh) * fma(R(3e-5), ny, fast_max(ny - R(1), R(0)));
    }
    R m = fma3(y, ldv(sub, 0));
#pragma unroll
    for (int k = 1; k < kSub; k++) m = fast_max(m, fma3(y, ldv(sub, k)));
    if (QUIRK) {
        const R u0 = fma3(y, ldv(sub, kSub)), u1 = fma3(y, ldv(sub, kSub + 1));
        if (!(m > (u0 < u1 ? u0 : u1) + slack * ny)) m = Lim<R>::min();
    }
    return m;
}

// Picks the kSub vertices of a hull furthest along dir (its local frame) among those from `first` on,
// and stores them turned into the world and multiplied by sgn.  One warp.
template <class R>
__device__ __forceinline__ void sat_pick(const ShapeView<R>& s, const M3<R>& b, const R* lv, const V3<R>& dir, int first, R sgn, R* sub, int lane) {
    auto key = [&](int i) -> unsigned {   // order bits of the projection, the index in the low bits
        if (i < first || i >= s.nv) return 0u;
        const V3<R> p = ldv(lv, i);
        const unsigned u = __float_as_uint((float)fma3(p, dir));
        return (((u & 0x80000000u) ? ~u : (u | 0x80000000u)) & ~(unsigned)(kSatV - 1)) | (unsigned)i | kSatV;
    };
    unsigned k0 = key(lane), k1 = key(lane + 32), mine = 0, top = 0;
#pragma unroll
    for (int n = 0; n < kSub; n++) {
        const unsigned m = __reduce_max_sync(0xffffffffu, k0 > k1 ? k0 : k1);
        if (n == 0) top = m;
        if (k0 == m) k0 = 0;
        if (k1 == m) k1 = 0;
        if (lane == n) mine = m ? m : top;   // fewer vertices than points: the first again
    }
    if (lane < kSub + 2) {
        const int i = lane < kSub ? (int)(mine & (unsigned)(kSatV - 1)) : lane - kSub;
        stv(sub, lane, mv(b, ldv(lv, i)) * sgn);
    }
}

// Group primitives of the staged SAT: a group is one warp (G = 1) or a whole block of G warps.
// Reductions are lexicographic (value, axis index) minima/maxima, so their result does not depend
// on the order lanes and warps are combined in.
template <int G> __device__ __forceinline__ bool group_any(bool p) {
    if (G == 1) return __any_sync(0xffffffffu, p);
    return __syncthreads_or(p) != 0;
}
template <int G> __device__ __forceinline__ void group_sync() {
    if (G == 1) __syncwarp(); else __syncthreads();
}
template <class R, int G> __device__ __forceinline__ void group_argmin(R& d, int& idx, int tid, R* rd, int* ri) {
    warp_argmin(d, idx);
    if (G == 1) return;
    if ((tid & 31) == 0) { rd[tid >> 5] = d; ri[tid >> 5] = idx; }
    __syncthreads();
    d = rd[0]; idx = ri[0];
    for (int k = 1; k < G; k++)
        if (rd[k] < d || (rd[k] == d && ri[k] < idx)) { d = rd[k]; idx = ri[k]; }
    __syncthreads();
}
template <class R, int G> __device__ __forceinline__ void group_argmax(R& d, int& idx, int tid, R* rd, int* ri) {
    warp_argmax(d, idx);
    if (G == 1) return;
    if ((tid & 31) == 0) { rd[tid >> 5] = d; ri[tid >> 5] = idx; }
    __syncthreads();
    d = rd[0]; idx = ri[0];
    for (int k = 1; k < G; k++)
        if (rd[k] > d || (rd[k] == d && ri[k] < idx)) { d = rd[k]; idx = ri[k]; }
    __syncthreads();
}
// value of the one thread of the group with `mine` set (the thread that evaluated the winning axis)
template <class R, int G> __device__ __forceinline__ V3<R> group_bcast3(const V3<R>& v, bool mine, R* buf) {
    if (G == 1) return shfl3(v, __ffs(__ballot_sync(0xffffffffu, mine)) - 1);
    if (mine) { buf[0] = v.x; buf[1] = v.y; buf[2] = v.z; }
    __syncthreads();
    const V3<R> r(buf[0], buf[1], buf[2]);
    __syncthreads();
    return r;
}
// The inner balls' bound of an axis x of length nx, held against the depth `best`: lo <= the computed
// maximum of a shape's projection (a hull: its inner ball about the local origin; another shape: its
// closed-form interval), hi >= the computed minimum, mag the magnitudes entering their rounding, and 64
// units of roundoff of those on top of `best`.
template <class R>
__device__ __forceinline__ void ball_side(const ShapeView<R>& s, const Xf<R>& t, const V3<R>& x, R nx, R& lo, R& hi, R& mag) {
    if (s.type == ST_HULL) {
        const R o = dot(t.o, x);
        lo = o + s.inner * nx;
        hi = o - s.inner * nx;
        mag = rabs(o) + s.outer * nx;
        return;
    }
    int i0, i1;
    shape_interval(s, t, x, (const R*)nullptr, hi, lo, i0, i1);
    mag = rabs(hi) + rabs(lo);
}
template <class R>
__device__ __forceinline__ bool balls_above(const Pair<R>& c, const V3<R>& x, R nx, R best) {
    R loA, hiA, mA, loB, hiB, mB;
    ball_side(c.sa, c.ta(), x, nx, loA, hiA, mA);
    ball_side(c.sb, c.tb(), x, nx, loB, hiB, mB);
    const R d0 = loA - hiB, d1 = loB - hiA;
    const R lb = d0 < d1 ? d0 : d1;
    constexpr R u = sizeof(R) == 4 ? R(1.1920929e-7) : R(2.220446049250313e-16);
    return lb > nx * best + R(64) * u * (mA + mB + nx * rabs(best));
}
// reals of per-group scratch: G reduction values, G indices, 3 broadcast, the group's bound
template <class R> constexpr int sat_scratch_reals(int G) { return G == 1 ? 0 : 2 * G + 4; }
// What the staged SAT leaves for the contact step (one record of kSatOut reals per pair, written by
// thread 0): the face-stage point, the edge-stage point, the final axis and the clipping faces,
// in the order the reference adds them (convex_convex_collision_algorithm.cpp:300-308, :363-395,
// :420-430).  flags: 1 face point, 2 edge point, 4 clip.
enum SatOutField { SO_FLAGS = 0, SO_FN = 1, SO_FP = 4, SO_FD = 7, SO_EN = 8, SO_EP = 11, SO_ED = 14, SO_SEP = 15, SO_FB = 18,
                   SO_FA = 19, kSatOut = 20 };
template <class R> __device__ __forceinline__ void so_put3(R* o, int k, const V3<R>& v) { o[k] = v.x; o[k + 1] = v.y; o[k + 2] = v.z; }
template <class R> __device__ __forceinline__ V3<R> so_get3(const R* o, int k) { return V3<R>(o[k], o[k + 1], o[k + 2]); }

// group layout in shared memory: both edge lists (the face axes before them), both shapes' vertices, the supporting points, the
// queues (one per warp), the scratch
constexpr int kSatFree = 64, kSatBlock = 512;   // see sat_staged's balls
constexpr int kCertain = 5;      // the first shape's first vertices, turned into the world (see sat_staged's certain)
constexpr int kSatQueue = 64;    // queued axes per warp: a round's 32 and what the next 32 candidates can add
template <class R> constexpr int sat_group_reals(int G) {
    const int q = (kSatQueue * G * (int)sizeof(int) + (int)sizeof(R) - 1) / (int)sizeof(R);
    return (4 * 2 * kSatE + 4 * 2 * kSatV + 2 * kSatBase + 4 * kCertain + q + sat_scratch_reals<R>(G) + 3) & ~3;
}

// Staged SAT of one pair by a group of G warps (tid in [0, 32 G)).
template <class R, int G, int TA, int TB>
__device__ void sat_staged(Pair<R>& c, int tid, R* smem, R* out) {
    constexpr int T = 32 * G;
    const unsigned full = 0xffffffffu;
    const int lane = tid & 31, warp = tid >> 5;
    if (tid == 0) out[SO_FLAGS] = R(0);
    if (TA >= 0) c.sa.type = TA;   // shape types known at compile time: the other branches fold away
    if (TB >= 0) c.sb.type = TB;
    const R margin = c.margin;
    R* ea = smem;
    R* eb = ea + 4 * kSatE;
    R* vA = eb + 4 * kSatE;
    R* vB = vA + 4 * kSatV;
    R* subA = vB + 4 * kSatV;
    R* subB = subA + kSatBase;
    R* cerA = subB + kSatBase;
    int* queue = reinterpret_cast<int*>(cerA + 4 * kCertain) + warp * kSatQueue;
    R* rd = smem + sat_group_reals<R>(G) - ((sat_scratch_reals<R>(G) + 3) & ~3);
    int* ri = reinterpret_cast<int*>(rd + G);
    R* bc = rd + 2 * G;
    const int fa = c.sa.face_count(), fb = c.sb.face_count();
    const int na = c.sa.edge_count(), nb = c.sb.edge_count();
    const bool boxA = c.sa.type == ST_BOX, boxB = c.sb.type == ST_BOX;
    if (c.sa.type == ST_HULL) for (int i = tid; i < c.sa.nv; i += T) stv(vA, i, c.sa.vert(i));
    if (c.sb.type == ST_HULL) for (int i = tid; i < c.sb.nv; i += T) stv(vB, i, c.sb.vert(i));
    group_sync<G>();
    const V3<R> dc = c.ta().o - c.tb().o;

    // ---- bound data
    auto side = [](const ShapeView<R>& s, const Xf<R>& t) {
        SatSide<R> q;
        if (s.type == ST_BOX) {
            q.e0 = t.b.col(0) * s.half.x; q.e1 = t.b.col(1) * s.half.y; q.e2 = t.b.col(2) * s.half.z;
            q.inner = rmin(s.half.x, rmin(s.half.y, s.half.z));
            q.mag = s.half.x + s.half.y + s.half.z;
        } else if (s.type == ST_CYLINDER) {
            q.e0 = t.b.col(1); q.r = s.radius; q.hh = s.height * R(0.5);
            q.inner = rmin(q.r, q.hh) * R(0.99);
            q.mag = q.r + q.hh;
        } else {
            q.inner = s.inner;
            q.mag = s.outer;
        }
        return q;
    };
    const SatSide<R> qa = side(c.sa, c.ta()), qb = side(c.sb, c.tb());
    // A hull's supporting points: its vertices furthest towards the other shape, from the nearest point
    // of a box (a floor's centre says nothing about where a hull touches it), else the other's centre
    {
        V3<R> dir = dc;   // from B towards A
        auto from_box = [](const ShapeView<R>& s, const Xf<R>& t, const V3<R>& o) {   // from the box's nearest point to o
            const V3<R> p = t.inv_apply(o), h = s.half;
            V3<R> d = p - V3<R>(rclamp(p.x, -h.x, h.x), rclamp(p.y, -h.y, h.y), rclamp(p.z, -h.z, h.z));
            if (!(sqnorm(d) > 0)) {   // inside: out of the nearest face
                const V3<R> g(h.x - rabs(p.x), h.y - rabs(p.y), h.z - rabs(p.z));
                const int k = g.x <= g.y && g.x <= g.z ? 0 : g.y <= g.z ? 1 : 2;
                d[k] = p[k] < 0 ? R(-1) : R(1);
            }
            return mv(t.b, d);
        };
        if (boxB && !boxA) dir = from_box(c.sb, c.tb(), c.ta().o);
        else if (boxA && !boxB) dir = -from_box(c.sa, c.ta(), c.tb().o);
        if (G == 1 || warp == 0) if (c.sa.type == ST_HULL) sat_pick(c.sa, c.ta().b, vA, mtv(c.ta().b, -dir), 0, R(-1), subA, lane);
        if (G == 1 || warp == 0) if (c.sb.type == ST_HULL) sat_pick(c.sb, c.tb().b, vB, mtv(c.tb().b, dir), c.sb.nv > 2 ? 2 : 0, R(1), subB, lane);
        if (c.sa.type == ST_HULL && tid < kCertain) stv(cerA, tid, mv(c.ta().b, ldv(vA, min(tid, c.sa.nv - 1))));
    }
    // everything that enters a projection, in units of roundoff: the bounds' and the projections' errors
    const R slack = sat_slack<R>() * (norm(c.ta().o) + norm(c.tb().o) + qa.mag + qb.mag);
    const R deep = qa.inner + qb.inner - slack;   // the inner balls keep every axis's other depth (the first shape past the second) above this
    const bool able = qa.inner > 0 && qb.inner > 0 && (c.sb.type != ST_HULL || c.sb.nv > 2);
    group_sync<G>();
    // lower bound of the depth along y, of length ny and oriented from B towards A (the reference takes the
    // edge axes normalised and the face axes as they are: the cylinder mesh's normals are not all unit)
    auto bound = [&](const V3<R>& y, R ny) {
        return sat_support<R, TA, false>(c.sa.type, qa, y, ny, subA, slack) + sat_support<R, TB, true>(c.sb.type, qb, y, ny, subB, slack) - fma3(y, dc);
    };
    // The other depth, the first shape past the second, has its own quirk: the reference's projection of
    // the first shape passes over the vertices of its first falling run, so its maximum may lie below
    // the inner ball's.  Among the first kCertain vertices, one that certainly lies above an earlier
    // one is never passed over; an axis is skipped only if such a vertex keeps the other depth above pb,
    // or if the run ends with vertex 0, which the inner ball leaves out.  (One axis in a hundred has a
    // longer run and is projected; a loop over eight vertices cost the longest pair of a 501-body pile 50 us.)
    auto certain = [&](const V3<R>& y, R ny, R pb) {
        if (c.sa.type != ST_HULL) return true;
        const R tol = R(2) * slack * ny, need = ny * (pb - qb.inner) - fma3(y, dc) + tol;
        R u[kCertain];
#pragma unroll
        for (int i = 0; i < kCertain; i++) u[i] = fma3(y, ldv(cerA, i));
        bool ok = u[1] > u[0] + tol;
        R low = u[0] < u[1] ? u[0] : u[1];
#pragma unroll
        for (int i = 2; i < kCertain; i++) {
            ok = ok || (u[i] > low + tol && u[i] > need);
            low = low < u[i] ? low : u[i];
        }
        return ok;
    };
    auto pruned = [&](const V3<R>& y, R ny, R pb) { return able && pb < deep && bound(y, ny) > ny * (pb + slack) && certain(y, ny, pb); };
    // The inner balls' bound of the same depth.  It alone also decides which axes of a hull count: the
    // balls are certified for a projection that never takes vertex 0 as the maximum, but the reference
    // passes over the vertices after it too while the projections keep falling, so along a few axes its
    // depth is below the balls' bound, and those that the balls rule out stay out.  Face axes from
    // kSatFree on are held against the least depth of the axes before them, edge axes against the least
    // depth known when their block of kSatBlock axes begins.
    constexpr bool has_hull = TA < 0 || TA == ST_HULL || TB == ST_HULL;
    auto ball = [&](const V3<R>& y, R ny) {
        auto one = [&](int type, const SatSide<R>& q) {
            return type == ST_HULL ? q.inner * ny : rabs(fma3(y, q.e0)) + rabs(fma3(y, q.e1)) + rabs(fma3(y, q.e2));
        };
        return one(c.sa.type, qa) + one(c.sb.type, qb) - rabs(fma3(y, dc));
    };
    const bool balls = has_hull && able && (c.sa.type == ST_HULL || c.sb.type == ST_HULL);

    // ---- exact projections along one axis per lane
    R min0, max0, min1, max1;
    int a0, a1, b0, b1;
    auto project = [&](const V3<R>& n) {
        shape_interval(c.sa, c.ta(), n, vA, min0, max0, a0, a1);
        shape_interval(c.sb, c.tb(), n, vB, min1, max1, b0, b1);
    };
    int cnt = 0;   // queued axes, in order; a round takes the first 32
    const unsigned lt = (1u << lane) - 1u;
    auto push = [&](bool keep, int v) {   // at most 32 more
        const unsigned m = __ballot_sync(full, keep);
        if (keep) queue[cnt + __popc(m & lt)] = v;
        cnt += __popc(m);
    };
    auto pop = [&](int& v) {   // this lane's axis of the round
        __syncwarp();
        const bool ok = lane < cnt;
        v = ok ? queue[lane] : 0;
        const int rest = cnt - 32, next = lane < rest ? queue[32 + lane] : 0;
        __syncwarp();
        if (lane < rest) queue[lane] = next;
        cnt = rest > 0 ? rest : 0;
        return ok;
    };

    // ---- face axes of A, then of B (findSeparatingAxis :265-308)
    R* axes = ea;   // the face axes, until the edge lists take their place
    for (int f = tid; f < fa + fb; f += T) {
        V3<R> n = f < fa ? mv(c.ta().b, c.sa.face_normal(f)) : mv(c.tb().b, c.sb.face_normal(f - fa));
        if (dot(dc, n) < 0) n = n * R(-1.0);
        stv(axes, f, n);
    }
    group_sync<G>();
    auto face_axis = [&](int f) { return ldv(axes, f); };
    R pb = Lim<R>::max();   // a depth above which an axis is skipped
    const int nfree = G == 1 && has_hull ? min(fa + fb, kSatFree) : fa + fb;
    if (able) {   // the axis of the least bound, projected (upper bound of its depth): the first depth to beat
        R least = Lim<R>::max();
        int at = 0x7fffffff;
        for (int f = tid; f < nfree; f += T) {
            const V3<R> n = face_axis(f);
            const R lb = bound(n, TA == ST_CYLINDER || TA < 0 ? fast_sqrt(fma3(n, n)) : R(1));
            if (lb < least) { least = lb; at = f; }
        }
        group_argmin<R, G>(least, at, tid, rd, ri);
        if (at < 0x7fffffff) {
            const V3<R> y = face_axis(at);
            auto whole = [&](const ShapeView<R>& s, const SatSide<R>& q, const Xf<R>& t, const R* lv, R sgn) {
                if (s.type == ST_BOX) return rabs(fma3(y, q.e0)) + rabs(fma3(y, q.e1)) + rabs(fma3(y, q.e2));
                if (s.type == ST_CYLINDER) {
                    const R k = fma3(y, q.e0);
                    const R n2 = fma3(y, y);
                    return fma(q.hh, rabs(k), q.r * fast_sqrt(fast_max(fma(-k, k, n2) + R(0.125) * sat_slack<R>() * n2, R(0))));
                }
                const V3<R> yl = mtv(t.b, y) * sgn;
                R m = Lim<R>::min();
                for (int i = lane; i < s.nv; i += 32) m = fast_max(m, fma3(yl, ldv(lv, i)));
                for (int o = 16; o > 0; o >>= 1) m = fast_max(m, __shfl_xor_sync(full, m, o));
                return m;
            };
            pb = whole(c.sa, qa, c.ta(), vA, R(-1)) + whole(c.sb, qb, c.tb(), vB, R(1)) - fma3(y, dc) + slack;
        }
    }
    R bd = Lim<R>::max();
    int bf = 0x7fffffff, bside = 0, bia = -1, bib = -1;
    bool sepd = false;
    R hold_f = 0;   // the least depth of the first kSatFree axes
    // (one loop holds one copy of the bound and one of the round: the warps of an SM are at different
    // places of this kernel, and fetching instructions was what they waited for most)
    for (int f0 = warp * 32, end = nfree, held = 0;;) {
        while (f0 < end && cnt <= 32) {
            const int f = f0 + lane;
            const V3<R> n = face_axis(f < end ? f : 0);
            const R ny = TA == ST_CYLINDER || TA < 0 ? fast_sqrt(fma3(n, n)) : R(1);
            bool keep = f < end && !pruned(n, ny, pb);
            if (G == 1 && has_hull && held && __any_sync(full, keep)) keep = keep && !balls_above(c, n, R(1), hold_f);
            push(keep, f);
            f0 += T;
        }
        if (cnt == 0) {
            if (end == fa + fb) break;
            if (__any_sync(full, sepd)) return;   // G == 1
            hold_f = bd;
            warp_min(hold_f);
            held = balls;
            f0 = nfree;
            end = fa + fb;
            continue;
        }
        int f;
        if (pop(f)) {
            project(face_axis(f));
            const R d0 = max0 - min1, d1 = max1 - min0;
            const R d = d0 < d1 ? d0 : d1;
            if (max0 < min1 || max1 < min0) sepd = true;
            else if (d < bd || (d == bd && f < bf)) {
                bd = d; bf = f; bside = d0 < d1;
                bia = d0 < d1 ? a1 : a0; bib = d0 < d1 ? b0 : b1;
            }
        }
        R m = bd;
        warp_min(m);
        pb = pb < m ? pb : m;
    }
    if (group_any<G>(sepd)) return;
    R dmin = bd;
    int wf = bf;
    group_argmin<R, G>(dmin, wf, tid, rd, ri);
    V3<R> sep, dpt;
    const bool on_a = wf >= fa;
    if (wf < 0x7fffffff) {
        const bool mine = bf == wf;
        if (mine) {
            const V3<R> n = face_axis(wf);
            sep = n;
            // testSepAxis witnesses: d0 < d1 -> (max of A, min of B), else (min of A, max of B)
            if (!on_a) dpt = shape_witness(c.sb, c.tb(), n, !bside, bib, vB);
            else dpt = shape_witness(c.sa, c.ta(), n, bside, bia, vA) + n * bd;
        }
        sep = group_bcast3<R, G>(sep, mine, bc);
        dpt = group_bcast3<R, G>(dpt, mine, bc);
        if (tid == 0 &&
            ((on_a && shape_inside(c.sb, c.tb().inv_apply(dpt))) || (!on_a && shape_inside(c.sa, c.ta().inv_apply(dpt))))) {
            out[SO_FLAGS] = R(1);
            so_put3(out, SO_FN, sep);
            so_put3(out, SO_FP, dpt - sep * margin);
            out[SO_FD] = -dmin + margin * 2;
        }
    }

    // ---- edge-pair axes (:323-361).  A box's 12 edges come in 3 classes of 4 whose direction
    // vectors are bit-identical (scaled unit-mesh differences), so they give identical axes,
    // projections and witnesses: each class is projected once, and a candidate takes the first
    // edge pair of the class (in the reference's e0-major order) whose lines hold the witnesses.
    const int ua = boxA ? 3 : na, ub = boxB ? 3 : nb;
    // unit edge directions: a hull's come precomputed (k_hull_edge_dirs, the same arithmetic)
    auto edge_dir = [](const ShapeView<R>& sh, const Xf<R>& t, int u) {
        V3<R> d;
        if (sh.type == ST_HULL) d = sh.edge_dir(u);
        else {
            V3<R> p0, p1;
            sh.edge(sh.type == ST_BOX ? 4 * u : u, p0, p1);
            d = normalized(p0 - p1);
        }
        return mv(t.b, d);
    };
    pb = pb < dmin ? pb : dmin;
    group_sync<G>();   // the last reads of the face axes
    // Both edge lists, without the edges whose every axis is skipped: an axis is perpendicular to its
    // edges, so its component along the centres' line is at most that of the line's part across the
    // edge, and the inner balls give the rest of the bound.  (The cross product of nearly parallel edges
    // is perpendicular to them only up to a few roundoffs over its length, at least 1e-5: `lean`.)
    const R lean = sizeof(R) == 4 ? R(0.03) : R(1e-9);
    const R gap = able && pb < deep ? qa.inner + qb.inner - pb - slack * R(2) : R(-1);
    auto list_edges = [&](const ShapeView<R>& s, const Xf<R>& t, int u, R* list) {   // one warp; returns the length
        int n = 0;
        for (int e0 = 0; e0 < u; e0 += 32) {
            const int e = e0 + lane;
            const V3<R> d = edge_dir(s, t, e < u ? e : 0);
            const R k = fma3(d, dc);
            const V3<R> w(fma(-k, d.x, dc.x), fma(-k, d.y, dc.y), fma(-k, d.z, dc.z));
            const R g = gap - lean * rabs(k);
            const bool keep = e < u && !(g > 0 && fma3(w, w) < g * g);
            const unsigned m = __ballot_sync(full, keep);
            if (keep) {
                R* p = list + 4 * (n + __popc(m & lt));
                p[0] = d.x; p[1] = d.y; p[2] = d.z;
                reinterpret_cast<int*>(p + 3)[0] = e;
            }
            n += __popc(m);
        }
        return n;
    };
    int la = 0, lb = 0;
    if (G == 1) {
        la = list_edges(c.sa, c.ta(), ua, ea);
        lb = list_edges(c.sb, c.tb(), ub, eb);
        __syncwarp();
    } else {
        if (warp == 0) la = list_edges(c.sa, c.ta(), ua, ea);
        if (warp == 1) lb = list_edges(c.sb, c.tb(), ub, eb);
        __syncthreads();
        if (tid == 0) ri[0] = la;
        if (tid == 32) ri[1] = lb;
        __syncthreads();
        la = ri[0]; lb = ri[1];
        if (tid == 0) bc[3] = pb;
        __syncthreads();
    }
    // a queued candidate: its places in the lists; the axis index: edge of A major
    auto list_edge = [](const R* list, int k) { return reinterpret_cast<const int*>(list + 4 * k + 3)[0]; };
    auto edge_axis = [&](int v, V3<R>& x, R& nx, V3<R>& a) {   // false for parallel edges
        x = cross(ldv(ea, v & 0xffff), ldv(eb, v >> 16));
        nx = norm(x);
        if (rabs(nx - 0) < eps<R>()) return false;
        a = normalized(x);
        if (dot(dc, a) < 0) a = a * R(-1.0);
        return true;
    };
    R ed = dmin;
    int ep = 0x7fffffff;
    V3<R> ewa, ewb, en;
    R seen = dmin;           // this warp's least depth so far
    R hold = dmin;           // the balls' measure of the block being resolved,
    int block = 0;           // and which one that is
    R measure = dmin;        // the balls' measure for the candidates: `hold` or a larger one of an earlier block
    // candidates in the order of their index: B's list inside A's
    const int nc = la * lb, di = lb > 0 ? T / lb : 0, dj = T - di * lb;
    int i = lb > 0 ? tid / lb : 0, j = tid - i * lb;
    for (int k0 = warp * 32;;) {
        while (k0 < nc && cnt <= 32) {
            const bool in = k0 + lane < nc;
            const int ci = in ? i : la - 1, cj = in ? j : lb - 1;
            const V3<R> d0 = ldv(ea, ci), d1 = ldv(eb, cj);
            V3<R> x = cross(d0, d1);
            const R n2 = fma3(x, x), g = fma3(x, dc);
            bool keep = in;
            if (able) {
                if (G == 1 && has_hull && (list_edge(ea, __shfl_sync(full, ci, 0)) * ub + list_edge(eb, __shfl_sync(full, cj, 0))) / kSatBlock > block)
                    measure = seen;
                constexpr bool hulls = TA == ST_HULL && TB == ST_HULL;
                if (hulls) {   // the balls without a square root
                    const R t = qa.inner + qb.inner - measure - slack;
                    keep = keep && !(t > 0 && n2 * t * t > g * g);
                }
                if (!hulls || __any_sync(full, keep)) {
                    const R ny = fast_sqrt(n2);
                    if (!hulls && has_hull && balls) keep = keep && !(ball(x, ny) > ny * (measure + slack));
                    x = x * (g < 0 ? R(-1) : R(1));
                    keep = keep && !pruned(x, ny, pb);
                }
            }
            push(keep, ci | cj << 16);
            k0 += T;
            i += di;
            j += dj;
            if (j >= lb) { j -= lb; i++; }
        }
        if (cnt == 0) break;
        // a round: the exact projections of up to 32 queued axes
        int v;
        bool ok = pop(v);
        const int iu = list_edge(ea, v & 0xffff), ju = list_edge(eb, v >> 16), q = iu * ub + ju;
        V3<R> cr(0, 0, 0), x, wa, wb;
        R dist = 0, nx = 0;
        bool split = false;
        int qref = 0x7fffffff;
        if (ok) ok = edge_axis(v, x, nx, cr);
        if (ok) {
            project(cr);
            split = max0 < min1 || max1 < min0;
            const R d0 = max0 - min1, d1 = max1 - min0;
            dist = d0 < d1 ? d0 : d1;
            if (!split && (dist < ed || (dist == ed && ep != 0x7fffffff))) {
                const bool s = d0 < d1;
                wa = shape_witness(c.sa, c.ta(), cr, s, s ? a1 : a0, vA);
                wb = shape_witness(c.sb, c.tb(), cr, !s, s ? b0 : b1, vB);
                const V3<R> la = c.ta().inv_apply(wa), lb = c.tb().inv_apply(wb);
#pragma unroll 1
                for (int m0 = 0; m0 < (boxA ? 4 : 1) && qref == 0x7fffffff; m0++) {
                    const int e0 = boxA ? 4 * iu + m0 : iu;
                    V3<R> p0, p1;
                    c.sa.edge(e0, p0, p1);
                    if (!on_line(p0, p1, la)) continue;
#pragma unroll 1
                    for (int m1 = 0; m1 < (boxB ? 4 : 1); m1++) {
                        const int e1 = boxB ? 4 * ju + m1 : ju;
                        V3<R> q0, q1;
                        c.sb.edge(e1, q0, q1);
                        if (on_line(q0, q1, lb)) { qref = e0 * nb + e1; break; }
                    }
                }
            }
        }
        // block by block (queued axes are in order), each against the depth known when it began
        const int mine = q / kSatBlock;
        for (unsigned todo = __ballot_sync(full, ok); todo;) {
            const int b = __shfl_sync(full, mine, __ffs(todo) - 1);
            if (G == 1 && has_hull && b != block) { block = b; hold = seen; }
            const unsigned now = todo & __ballot_sync(full, mine == b);
            todo &= ~now;
            if (ok && mine == b && !(has_hull && balls && balls_above(c, x, nx, hold))) {
                if (split) sepd = true;
                else if (qref != 0x7fffffff && (dist < ed || qref < ep)) { ed = dist; ep = qref; ewa = wa; ewb = wb; en = cr; }
            }
            seen = ed;
            warp_min(seen);
        }
        pb = pb < seen ? pb : seen;
        if (G > 1) {   // the warps' bounds together
            volatile R* shared = bc + 3;
            const R o = *shared;
            if (o < pb) pb = o;
            else if (lane == 0 && pb < o) *shared = pb;   // any warp's bound will do
        }
        if (G == 1 && __any_sync(full, sepd)) return;
    }
    if (group_any<G>(sepd)) return;
    R emin = ed;
    int wq = ep;
    group_argmin<R, G>(emin, wq, tid, rd, ri);
    if (wq < 0x7fffffff) {
        const bool mine = ep == wq;
        const V3<R> wpa = group_bcast3<R, G>(ewa, mine, bc), wpb = group_bcast3<R, G>(ewb, mine, bc);
        sep = group_bcast3<R, G>(en, mine, bc);
        if (tid == 0) {   // segmentsClosestPoints with unbounded half-lengths (:172-214, :363-395)
            const int e0 = wq / nb, e1 = wq - e0 * nb;
            const V3<R> wea = edge_dir(c.sa, c.ta(), boxA ? e0 / 4 : e0), web = edge_dir(c.sb, c.tb(), boxB ? e1 / 4 : e1);
            const V3<R> tr = wpb - wpa;
            const R ab = dot(wea, web), at = dot(wea, tr), bt = dot(web, tr);
            const R d = R(1.0) - ab * ab;
            const R ha = Lim<R>::max(), hb = Lim<R>::max();
            R ta, tb;
            if (d == 0) ta = 0;
            else { ta = (at - bt * ab) / d; if (ta < -ha) ta = -ha; else if (ta > ha) ta = ha; }
            tb = ta * ab - bt;
            if (tb < -hb) { tb = -hb; ta = tb * ab + at; if (ta < -ha) ta = -ha; else if (ta > ha) ta = ha; }
            else if (tb > hb) { tb = hb; ta = tb * ab + at; if (ta < -ha) ta = -ha; else if (ta > ha) ta = ha; }
            const V3<R> oa = wea * ta, ob = web * tb;
            V3<R> pts = tr - oa + ob;
            const R nl2 = sqnorm(pts);
            if (nl2 > eps<R>()) {
                const R nl = real_sqrt(nl2);
                pts = pts * (R(1.0) / nl);
                if (dot(pts, dc) < 0) pts = pts * R(-1.0);
                out[SO_FLAGS] += R(2);
                so_put3(out, SO_EN, pts);
                so_put3(out, SO_EP, wpb + ob - pts * margin);
                out[SO_ED] = -nl + margin * 2;
            }
        }
    }
    if (dot(dc, sep) < 0) sep = -sep;
    // ---- clipping (:63-170): incident face of B (first maximum), reference face of A (first minimum)
    R dmax = Lim<R>::min();
    int fbest = 0x7fffffff;
    for (int f = tid; f < fb; f += T) {
        const R d = dot(mv(c.tb().b, c.sb.face_normal(f)), sep);
        if (d > dmax) { dmax = d; fbest = f; }
    }
    group_argmax<R, G>(dmax, fbest, tid, rd, ri);
    R dmn = Lim<R>::max();
    int fabest = 0x7fffffff;
    for (int f = tid; f < fa; f += T) {
        const R d = dot(mv(c.ta().b, c.sa.face_normal(f)), sep);
        if (d < dmn) { dmn = d; fabest = f; }
    }
    group_argmin<R, G>(dmn, fabest, tid, rd, ri);
    if (tid == 0 && fbest < 0x7fffffff && fabest < 0x7fffffff) {
        out[SO_FLAGS] += R(4);
        so_put3(out, SO_SEP, sep);
        out[SO_FB] = R(fbest);
        out[SO_FA] = R(fabest);
    }
}

template <class R>
__device__ bool sat_warp(Pair<R>& c, int lane) {
    const R margin = c.margin;
    const V3<R> dc = c.ta().o - c.tb().o;
    const int fa = c.sa.face_count(), fb = c.sb.face_count();
    // face axes of A, then of B
    R bd = Lim<R>::max();
    int bf = 0x7fffffff;
    V3<R> bn, bpt;
    bool sep_found = false;
    for (int f = lane; f < fa + fb; f += 32) {
        const bool is_a = f < fa;
        V3<R> n = is_a ? mv(c.ta().b, c.sa.face_normal(f)) : mv(c.tb().b, c.sb.face_normal(f - fa));
        if (dot(dc, n) < 0) n = n * R(-1.0);
        R d;
        V3<R> wa, wb;
        if (!sep_test(c, n, d, wa, wb)) { sep_found = true; break; }
        if (d < bd) { bd = d; bf = f; bn = n; bpt = is_a ? wb : wa + n * d; }
    }
    if (__any_sync(0xffffffffu, sep_found)) return false;
    R dmin = bd;
    int wf = bf;
    warp_argmin(dmin, wf);
    const int src_lane = wf < 0x7fffffff ? wf % 32 : 0;
    V3<R> sep = shfl3(bn, src_lane);
    const V3<R> dpt = shfl3(bpt, src_lane);
    const bool on_a = wf >= fa;
    if (wf < 0x7fffffff && lane == 0) {
        if ((on_a && shape_inside(c.sb, c.tb().inv_apply(dpt))) || (!on_a && shape_inside(c.sa, c.ta().inv_apply(dpt))))
            c.add(sep, dpt - sep * margin, -dmin + margin * 2);
    }
    // edge-pair axes
    const int na = c.sa.edge_count(), nb = c.sb.edge_count();
    const int ne = na * nb;
    R ed = dmin;
    int ep = 0x7fffffff;
    V3<R> ewa, ewb, ew0, ew1, en;
    sep_found = false;
    for (int q = lane; q < ne; q += 32) {
        const int e0 = q / nb, e1 = q - e0 * nb;
        V3<R> a0, a1, b0, b1;
        c.sa.edge(e0, a0, a1);
        c.sb.edge(e1, b0, b1);
        const V3<R> w0 = mv(c.ta().b, normalized(a0 - a1));
        const V3<R> w1 = mv(c.tb().b, normalized(b0 - b1));
        V3<R> cr = cross(w0, w1);
        if (rabs(norm(cr) - 0) < eps<R>()) continue;
        cr = normalized(cr);
        if (dot(dc, cr) < 0) cr = cr * R(-1.0);
        R dist;
        V3<R> wa, wb;
        if (!sep_test(c, cr, dist, wa, wb)) { sep_found = true; break; }
        if (dist < ed) {
            if (!on_line(a0, a1, c.ta().inv_apply(wa)) || !on_line(b0, b1, c.tb().inv_apply(wb))) continue;
            ed = dist; ep = q; ewa = wa; ewb = wb; ew0 = w0; ew1 = w1; en = cr;
        }
    }
    if (__any_sync(0xffffffffu, sep_found)) return false;
    R emin = ed;
    int wq = ep;
    warp_argmin(emin, wq);
    if (wq < 0x7fffffff) {
        const int sl = wq % 32;
        const V3<R> wpa = shfl3(ewa, sl), wpb = shfl3(ewb, sl), wea = shfl3(ew0, sl), web = shfl3(ew1, sl);
        sep = shfl3(en, sl);
        if (lane == 0) {   // segmentsClosestPoints with unbounded half-lengths (:172-214, :363-395)
            const V3<R> tr = wpb - wpa;
            const R ab = dot(wea, web), at = dot(wea, tr), bt = dot(web, tr);
            const R d = R(1.0) - ab * ab;
            const R ha = Lim<R>::max(), hb = Lim<R>::max();
            R ta, tb;
            if (d == 0) ta = 0;
            else { ta = (at - bt * ab) / d; if (ta < -ha) ta = -ha; else if (ta > ha) ta = ha; }
            tb = ta * ab - bt;
            if (tb < -hb) { tb = -hb; ta = tb * ab + at; if (ta < -ha) ta = -ha; else if (ta > ha) ta = ha; }
            else if (tb > hb) { tb = hb; ta = tb * ab + at; if (ta < -ha) ta = -ha; else if (ta > ha) ta = ha; }
            const V3<R> oa = wea * ta, ob = web * tb;
            V3<R> pts = tr - oa + ob;
            const R nl2 = sqnorm(pts);
            if (nl2 > eps<R>()) {
                const R nl = real_sqrt(nl2);
                pts = pts * (R(1.0) / nl);
                if (dot(pts, dc) < 0) pts = pts * R(-1.0);
                c.add(pts, wpb + ob - pts * margin, -nl + margin * 2);
            }
        }
    }
    if (dot(dc, sep) < 0) sep = -sep;
    // clipping (:63-170): incident face of B (first maximum), reference face of A (first minimum)
    R dmax = Lim<R>::min();
    int fbest = 0x7fffffff;
    for (int f = lane; f < fb; f += 32) {
        const R d = dot(mv(c.tb().b, c.sb.face_normal(f)), sep);
        if (d > dmax) { dmax = d; fbest = f; }
    }
    warp_argmax(dmax, fbest);
    R dmn = Lim<R>::max();
    int fabest = 0x7fffffff;
    for (int f = lane; f < fa; f += 32) {
        const R d = dot(mv(c.ta().b, c.sa.face_normal(f)), sep);
        if (d < dmn) { dmn = d; fabest = f; }
    }
    warp_argmin(dmn, fabest);
    if (lane == 0 && fbest < 0x7fffffff && fabest < 0x7fffffff) clip_faces(c, sep, -c.ref_scale, c.margin, fbest, fabest);
    return true;
}

// SAT pairs: G = 1 runs kSatWarps pairs per block, one warp each, instantiated per shape pairing
// (TA, TB; one launch per pairing); G = kSatGroup runs one heavy pair per block, any pairing (-1).
// Only thread 0 holds the pair's contact cache.
static_assert(2 * kSatF <= 2 * kSatE, "the face axes fit the edge lists' room");
static_assert(sat_group_reals<float>(1) % 4 == 0 && kSatBase % 4 == 0, "SAT staging alignment");
template <class R, int G, int TA, int TB>
__global__ void __launch_bounds__(G == 1 ? 32 * kSatWarps : 32 * G, G == 1 ? kSatBlocksPerSm : 2)
k_np_sat(const int2* rng, int* cursor, const int* order, const int2* pairs, Bodies<R> B, ShapeTable<R> S, R* sat_out) {
    extern __shared__ __align__(16) unsigned char sat_smem[];
    const int grp = G == 1 ? (int)(threadIdx.x >> 5) : 0;
    const int tid = G == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
    R* smem = reinterpret_cast<R*>(sat_smem) + (size_t)grp * sat_group_reals<R>(G);
    auto one = [&](int t) {
        const int2 q = pairs[order[t]];
        Pair<R> pr;
        pr.xa = B.xf(q.x);
        pr.xb = B.xf(q.y);
        pr.sa = S.view(B.shape[q.x]);
        pr.sb = S.view(B.shape[q.y]);
        pr.margin = S.margin;
        pr.c = nullptr;
        sat_staged<R, G, TA, TB>(pr, tid, smem, sat_out + (size_t)t * kSatOut);
    };
    if (G == 1) {
        warp_items(*rng, cursor, one);
    } else {
        __shared__ int slot;
        block_items(*rng, cursor, &slot, one);
    }
}

// contact step of the staged SAT pairs, one thread per pair: the pooled result is set up, the
// recorded face-stage and edge-stage points are added and the faces clipped, in the reference's
// order, and the result is sorted and written out
template <class R>
__global__ void k_np_sat_finish(const int2* rng, const int* order, const int2* pairs, Bodies<R> B, ShapeTable<R> S, Results<R> res,
                                const int* pair_scene_off, const int* prev_off, const R* sat_out) {
    thread_items(*rng, [&](int t) {
        const int p = order[t];
        Cache<R> cache;
        Pair<R> pr;
        np_setup(p, pairs, B, S, res, pair_scene_off, prev_off, cache, pr);
        const R* o = sat_out + (size_t)t * kSatOut;
        const int fl = (int)o[SO_FLAGS];
        if (fl & 1) pr.add(so_get3(o, SO_FN), so_get3(o, SO_FP), o[SO_FD]);
        if (fl & 2) pr.add(so_get3(o, SO_EN), so_get3(o, SO_EP), o[SO_ED]);
        if (fl & 4) clip_faces(pr, so_get3(o, SO_SEP), -pr.ref_scale, pr.margin, (int)o[SO_FB], (int)o[SO_FA]);
        np_finish(p, pairs, B, res, cache);
    });
}

// ---------------------------------------------------------------- cylinder or sphere against a hull
// One warp per pair.  The reference walks the faces that the other shape's box reaches in descending
// index (the face tree's order for a hull) and adds the points a face gives one after the other: the
// cache's merging depends on that order, the candidate points do not.  The hit faces are queued in
// order, up to 32 at a time, and their pieces of work (a face and a cylinder segment, a hull edge, or a
// fan triangle) go to the lanes one each; lane 0 then adds the points the pieces gave, in order.  (With a
// whole face per lane, its four to six segments or its edges one after the other, a lone pair took 97 us,
// and the room for all points of 32 faces kept two blocks on an SM.)
template <class R> struct HullFaces {
    int nf, lane;
    int* queue;   // [64]
    // hit(f): is face f reached; work(n): the first n <= 32 queued faces
    template <class H, class F> __device__ __forceinline__ void each(H&& hit, F&& work) const {
        const unsigned full = 0xffffffffu;
        int cnt = 0;
        for (int base = 0; base < nf || cnt > 0;) {
            while (base < nf && cnt < 32) {
                const int f = nf - 1 - base - lane;
                const bool h = f >= 0 && hit(f);
                const unsigned m = __ballot_sync(full, h);
                if (h) queue[cnt + __popc(m & ((1u << lane) - 1u))] = f;
                cnt += __popc(m);
                base += 32;
            }
            __syncwarp();
            const int n = cnt < 32 ? cnt : 32;
            if (n) work(n);
            __syncwarp();
            const int rest = cnt - n, v = lane < rest ? queue[32 + lane] : 0;
            __syncwarp();
            if (lane < rest) queue[lane] = v;
            cnt = rest;
        }
    }
    // the pieces of n queued faces, size(f) of face f: piece(f, k) for each, 32 at a time, then done()
    template <class S, class F, class D> __device__ __forceinline__ void pieces(int n, S&& size, F&& piece, D&& done) const {
        const int mine = lane < n ? size(queue[lane]) : 0, end = warp_incl_scan(mine);
        const int total = __shfl_sync(0xffffffffu, end, 31);
        for (int t0 = 0; t0 < total; t0 += 32) {
            const int t = t0 + lane;
            int lo = 0;   // the first face whose pieces end after t
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (__shfl_sync(0xffffffffu, end, lo + o - 1) <= t) lo += o;
            const int first = __shfl_sync(0xffffffffu, end - mine, lo < 32 ? lo : 31);
            if (t < total) piece(queue[lo], t - first);
            done();
        }
    }
};
// a piece's points, for lane 0 to add (P points of 7 reals per lane)
template <class R, int P> struct PieceOut {
    R* buf;   // this lane's
    int n;
    __device__ __forceinline__ void push(const V3<R>& nrm, const V3<R>& pt, R d) {
        R* e = buf + 7 * n++;
        e[0] = nrm.x; e[1] = nrm.y; e[2] = nrm.z; e[3] = pt.x; e[4] = pt.y; e[5] = pt.z; e[6] = d;
    }
    __device__ __forceinline__ void drain(Pair<R>& c, int lane) {   // the warp's points in order, into lane 0's cache
        __syncwarp();
        const unsigned one = __ballot_sync(0xffffffffu, n > 0), two = __ballot_sync(0xffffffffu, n > 1);
        if (lane == 0)
            for (unsigned m = one; m; m &= m - 1) {
                const int l = __ffs(m) - 1;
                for (int k = 0; k < 1 + (int)((two >> l) & 1u); k++) {
                    const R* e = buf + l * (7 * P) + 7 * k;
                    c.add(V3<R>(e[0], e[1], e[2]), V3<R>(e[3], e[4], e[5]), e[6]);
                }
            }
        __syncwarp();
        n = 0;
    }
};

// CylinderConvexCollisionAlgorithm (cylinder_convex_collision_algorithm.cpp:109-203)
template <class R> constexpr int cyl_hull_warps() { return sizeof(R) == 4 ? 4 : 2; }
template <class R>
__global__ void __launch_bounds__(32 * cyl_hull_warps<R>())
k_np_cyl_hull(const int2* rng, int* cursor, const int* order, const int2* pairs, Bodies<R> B, ShapeTable<R> S, Results<R> res,
              const int* pair_scene_off, const int* prev_off) {
    constexpr int W = cyl_hull_warps<R>();
    __shared__ R cand[W][32 * 14];
    __shared__ int queue[W][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    warp_items(*rng, cursor, [&](int t) {
    const int p = order[t];
    Cache<R> cache;
    Pair<R> c;
    np_setup(p, pairs, B, S, res, pair_scene_off, prev_off, cache, c, lane == 0);
    const bool a_hull = c.sa.type == ST_HULL;
    const ShapeView<R>& m = a_hull ? c.sa : c.sb;
    const ShapeView<R>& cy = a_hull ? c.sb : c.sa;
    const Xf<R>& to = a_hull ? c.ta() : c.tb();
    const Xf<R>& tc = a_hull ? c.tb() : c.ta();
    const R margin = c.margin;
    if (lane == 0) cache.swap = a_hull;
    const R cr = cy.radius, ch = cy.height / R(2.0);
    const Xf<R> rel = to.inverse() * tc;
    const V3<R> axis = rel.b.col(1), pos = rel.o;
    V3<R> aa, bb;
    shape_aabb(cy, rel, aa, bb);
    HullFaces<R> faces;
    faces.nf = m.nf; faces.lane = lane; faces.queue = queue[warp];
    PieceOut<R, 2> out;
    out.buf = cand[warp] + lane * 14; out.n = 0;
    auto hit = [&](int f) { return face_hit(m, f, aa, bb); };
    auto done = [&]() { out.drain(c, lane); };
    // cylinder side segments against the faces the cylinder's box reaches: four of a face, and two more
    // when its normal is the axis
    faces.each(hit, [&](int n) {
        faces.pieces(n, [](int) { return 6; }, [&](int f, int k) {
            const V3<R> fn = m.face_normal(f);
            const R adc = dot(axis, fn);
            const V3<R> ddy = axis;
            const bool vertical = rabs(rabs(adc) - 1) < eps<R>();
            if (k >= 4 && !vertical) return;
            V3<R> ddx, ddz;
            if (vertical) {
                ddz = normalized(cross(axis, V3<R>(1, 0, 0)));
                ddx = normalized(cross(axis, ddz));
            } else {
                ddx = normalized(cross(cross(fn, axis), axis));
            }
            const int i = k < 4 ? k : 2 * (k - 4);
            const int dx = i == 0 || i == 3 ? 1 : -1, dy = i < 2 ? 1 : -1;   // (1,1) (-1,1) (-1,-1) (1,-1)
            const V3<R> ps = pos + (k < 4 ? ddx : ddz) * R(dx) * cr + ddy * R(dy) * ch;
            const V3<R> ds = (k >= 4 || dx == dy ? ddy : ddx) * R(-dx);
            const R ls = (k >= 4 || dx == dy ? ch : cr) * 2;
            R t1, t2, d1, d2;
            if (segment_face(m, f, ps, ds, ls, margin, t1, t2, d1, d2)) {
                const V3<R> p1 = to.apply(ps + ds * t1 - fn * d1);
                const V3<R> p2 = to.apply(ps + ds * t2 - fn * d2);
                const V3<R> nw = mv(to.b, fn);
                out.push(nw, p1 - nw * margin, d1 + margin * 2);
                out.push(nw, p2 - nw * margin, d2 + margin * 2);
            }
        }, done);
    });
    // hull edges of those faces against the cylinder
    faces.each(hit, [&](int n) {
        faces.pieces(n, [&](int f) { return m.face_size(f); }, [&](int f, int i) {
            const V3<R> v1 = m.vert(m.face_vert(f, i));
            const V3<R> v2 = m.vert(m.face_vert(f, (i + 1) % m.face_size(f)));
            R t1, t2;
            const V3<R> start = (v1 + v2) / R(2);
            const R ls = norm(v2 - v1) / 2;
            const V3<R> dir = (v2 - v1) / (ls * 2);
            if (segment_cylinder(start, dir, ls, pos, axis, ch, cr, margin, t1, t2)) {
                const V3<R> p1 = start + dir * t1, p2 = start + dir * t2;
                V3<R> wn, wp;
                R wd;
                cyl_contact((p1 + p2) / R(2), pos, axis, cr, ch, to, margin, wn, wp, wd);
                out.push(wn, wp, wd);
            }
        }, done);
    });
    if (lane == 0) {
        cache.swap = false;
        np_finish(p, pairs, B, res, cache);
    }
    });
}

// SphereConvexCollisionAlgorithm (sphere_convex_collision_algorithm.cpp:185-210) for a convex hull: the
// sphere against the fan triangles of the faces its box reaches
template <class R> constexpr int sphere_hull_warps() { return sizeof(R) == 4 ? 4 : 2; }
template <class R>
__global__ void __launch_bounds__(32 * sphere_hull_warps<R>())
k_np_sphere_hull(const int2* rng, int* cursor, const int* order, const int2* pairs, Bodies<R> B, ShapeTable<R> S, Results<R> res,
                 const int* pair_scene_off, const int* prev_off) {
    constexpr int W = sphere_hull_warps<R>();
    __shared__ R cand[W][32 * 7];
    __shared__ int queue[W][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    warp_items(*rng, cursor, [&](int t) {
    const int p = order[t];
    Cache<R> cache;
    Pair<R> c;
    np_setup(p, pairs, B, S, res, pair_scene_off, prev_off, cache, c, lane == 0);
    const bool a_hull = c.sa.type == ST_HULL;
    const ShapeView<R>& m = a_hull ? c.sa : c.sb;
    const ShapeView<R>& sp = a_hull ? c.sb : c.sa;
    const Xf<R>& tm = a_hull ? c.ta() : c.tb();
    const Xf<R>& ts = a_hull ? c.tb() : c.ta();
    const R margin = c.margin;
    if (lane == 0) cache.swap = a_hull;
    const V3<R> rel = tm.inv_apply(ts.o);
    const R r = sp.radius;
    const V3<R> aa = rel - V3<R>(r, r, r), bb = rel + V3<R>(r, r, r);
    HullFaces<R> faces;
    faces.nf = m.nf; faces.lane = lane; faces.queue = queue[warp];
    PieceOut<R, 1> out;
    out.buf = cand[warp] + lane * 7; out.n = 0;
    faces.each([&](int f) { return face_hit(m, f, aa, bb); }, [&](int n) {
        faces.pieces(n, [&](int f) { const int k = m.face_size(f) - 2; return k > 0 ? k : 0; }, [&](int f, int i) {
            const V3<R> vs[3] = {m.vert(m.face_vert(f, 0)), m.vert(m.face_vert(f, i + 1)), m.vert(m.face_vert(f, i + 2))};
            V3<R> point, normal;
            R depth = 0;
            if (sphere_triangle(rel, r, vs, point, normal, depth)) {
                normal = mv(tm.b, normal);
                point = tm.apply(point);
                out.push(normal, point - normal * margin, depth + 2 * margin);
            }
        }, [&]() { out.drain(c, lane); });
    });
    if (lane == 0) {
        cache.swap = false;
        np_finish(p, pairs, B, res, cache);
    }
    });
}

// SAT pairs with a shape beyond the staging limits (PC_CONVEX_BIG): one warp each, unstaged
template <class R>
__global__ void k_np_sat_big(const int2* rng, int* cursor, const int* order, const int2* pairs, Bodies<R> B, ShapeTable<R> S,
                             Results<R> res, const int* pair_scene_off, const int* prev_off) {
    const int lane = threadIdx.x & 31;
    warp_items(*rng, cursor, [&](int t) {
        const int p = order[t];
        Cache<R> cache;
        Pair<R> pr;
        np_setup(p, pairs, B, S, res, pair_scene_off, prev_off, cache, pr);
        sat_warp(pr, lane);
        if (lane == 0) np_finish(p, pairs, B, res, cache);
    });
}

} // namespace pe
