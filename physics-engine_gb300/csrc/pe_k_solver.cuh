// Kernels of the rigid-body step, part 6: sequential-impulse rows, joints and contact islands.
#pragma once
#include "pe_k_mesh.cuh"

namespace pe {

// ===================================================================== solver
// One solver row in registers, and its moves to and from memory: a row is 24 consecutive reals (six
// 16-byte words in FP32, twelve in FP64), so a lane's row is three full sectors wherever it lies
// (field-major rows took one sector per field once the lanes of a warp work on scattered islands).
template <class R> struct RowReg {
    V3<R> ra, rb, n, t0, t1;
    R njmj, rhs, t0jmj, t1jmj, mu, nacc, t0acc, t1acc;
};
__device__ __forceinline__ void row_load(const Rows<float>& rows, int r, RowReg<float>& q) {
    const float4* p = reinterpret_cast<const float4*>(rows.f + (size_t)r * NRF);
    const float4 a = p[0], b = p[1], c = p[2], d = p[3], e = p[4], f = p[5];
    q.ra = V3<float>(a.x, a.y, a.z); q.njmj = a.w;
    q.rb = V3<float>(b.x, b.y, b.z); q.rhs = b.w;
    q.n = V3<float>(c.x, c.y, c.z); q.t0jmj = c.w;
    q.t0 = V3<float>(d.x, d.y, d.z); q.t1jmj = d.w;
    q.t1 = V3<float>(e.x, e.y, e.z);
    q.mu = f.x; q.nacc = f.y; q.t0acc = f.z; q.t1acc = f.w;
}
__device__ __forceinline__ void row_load(const Rows<double>& rows, int r, RowReg<double>& q) {
    const double2* p = reinterpret_cast<const double2*>(rows.f + (size_t)r * NRF);
    double2 a[12];
#pragma unroll
    for (int k = 0; k < 12; k++) a[k] = p[k];
    q.ra = V3<double>(a[0].x, a[0].y, a[1].x); q.njmj = a[1].y;
    q.rb = V3<double>(a[2].x, a[2].y, a[3].x); q.rhs = a[3].y;
    q.n = V3<double>(a[4].x, a[4].y, a[5].x); q.t0jmj = a[5].y;
    q.t0 = V3<double>(a[6].x, a[6].y, a[7].x); q.t1jmj = a[7].y;
    q.t1 = V3<double>(a[8].x, a[8].y, a[9].x);
    q.mu = a[10].x; q.nacc = a[10].y; q.t0acc = a[11].x; q.t1acc = a[11].y;
}
__device__ __forceinline__ void row_store_acc(const Rows<float>& rows, int r, const RowReg<float>& q) {
    reinterpret_cast<float4*>(rows.f + (size_t)r * NRF)[5] = make_float4(q.mu, q.nacc, q.t0acc, q.t1acc);
}
__device__ __forceinline__ void row_store_acc(const Rows<double>& rows, int r, const RowReg<double>& q) {
    double2* p = reinterpret_cast<double2*>(rows.f + (size_t)r * NRF);
    p[10] = make_double2(q.mu, q.nacc);
    p[11] = make_double2(q.t0acc, q.t1acc);
}
__device__ __forceinline__ void row_store(const Rows<float>& rows, int r, const RowReg<float>& q) {
    float4* p = reinterpret_cast<float4*>(rows.f + (size_t)r * NRF);
    p[0] = make_float4(q.ra.x, q.ra.y, q.ra.z, q.njmj);
    p[1] = make_float4(q.rb.x, q.rb.y, q.rb.z, q.rhs);
    p[2] = make_float4(q.n.x, q.n.y, q.n.z, q.t0jmj);
    p[3] = make_float4(q.t0.x, q.t0.y, q.t0.z, q.t1jmj);
    p[4] = make_float4(q.t1.x, q.t1.y, q.t1.z, 0.0f);
    row_store_acc(rows, r, q);
}
__device__ __forceinline__ void row_store(const Rows<double>& rows, int r, const RowReg<double>& q) {
    double2* p = reinterpret_cast<double2*>(rows.f + (size_t)r * NRF);
    const V3<double> v[5] = {q.ra, q.rb, q.n, q.t0, q.t1};
    const double s[5] = {q.njmj, q.rhs, q.t0jmj, q.t1jmj, 0.0};
#pragma unroll
    for (int k = 0; k < 5; k++) { p[2 * k] = make_double2(v[k].x, v[k].y); p[2 * k + 1] = make_double2(v[k].z, s[k]); }
    row_store_acc(rows, r, q);
}

// FrictionContactConstraint::initSequentialImpulse (friction_contact_constraint.cpp:9-73), one thread per result
template <class R>
__device__ __forceinline__ void si_setup_result(int p, const Results<R>& res, const Bodies<R>& B, const Rows<R>& rows,
                                                const StepParams& prm) {
    const int np = res.npts[p];
    if (np == 0) return;
    const int ia = res.a[p], ib = res.b[p];
    const bool ka = (B.flags[ia] & BF_KINEMATIC) != 0, kb = (B.flags[ib] & BF_KINEMATIC) != 0;
    const R ims = (ka ? R(0) : B.at(INVM, ia)) + (kb ? R(0) : B.at(INVM, ib));
    const M3<R> Ia = ka ? M3<R>() : B.mat(I00, ia);
    const M3<R> Ib = kb ? M3<R>() : B.mat(I00, ib);
    const M3<R> Ra = B.mat(B00, ia), Rb = B.mat(B00, ib);
    const V3<R> va0 = B.vec(VX, ia), wa0 = B.vec(WX, ia), vb0 = B.vec(VX, ib), wb0 = B.vec(WX, ib);
    const R dt = R(prm.dt), kerp = R(0.2), pen_th = R(0.3), rest_th = R(0.1);
    const R mu = res.fr[p], e = res.re[p];
    const int r0 = p * kSlots;
    for (int k = 0; k < np; k++) {
        const int o = p * kSlots + k;
        const V3<R> la(res.pt(LAX, o), res.pt(LAY, o), res.pt(LAZ, o));
        const V3<R> lb(res.pt(LBX, o), res.pt(LBY, o), res.pt(LBZ, o));
        const V3<R> n(res.pt(NX, o), res.pt(NY, o), res.pt(NZ, o));
        const V3<R> t0(res.pt(T0X, o), res.pt(T0Y, o), res.pt(T0Z, o));
        const V3<R> t1(res.pt(T1X, o), res.pt(T1Y, o), res.pt(T1Z, o));
        const V3<R> ra = mv(Ra, la), rb = mv(Rb, lb);
        auto jmj = [&](const V3<R>& d) {
            const V3<R> xa = cross(ra, d), xb = cross(rb, d);
            return R(1.0) / (ims + dot(mv(Ia, xa), xa) + dot(mv(Ib, xb), xb));
        };
        const R nj = jmj(n), j0 = jmj(t0), j1 = jmj(t1);
        const V3<R> va = va0 + cross(wa0, ra), vb = vb0 + cross(wb0, rb);
        R rev = -dot(n, va - vb);
        if (rabs(rev) < rest_th) rev = 0;
        rev *= e;
        R pen = res.dist[p * kSlots + k];
        pen = pen > -pen_th ? pen : -pen_th;
        RowReg<R> q;
        q.ra = ra; q.rb = rb; q.n = n; q.t0 = t0; q.t1 = t1;
        q.njmj = nj; q.rhs = (rev - kerp * pen / dt) * nj; q.t0jmj = j0; q.t1jmj = j1;
        q.mu = mu; q.nacc = 0; q.t0acc = 0; q.t1acc = 0;
        row_store(rows, r0 + k, q);
    }
}
template <class R>
__global__ void k_si_setup(const int* Rd, Results<R> res, Bodies<R> B, Rows<R> rows, StepParams prm) {
    const int P = *Rd;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) si_setup_result(p, res, B, rows, prm);
}

// One body of an item while the solver works on it: temporary velocities and the constants its
// impulses need.  A kinematic body's temporary velocity is zero and takes no impulse.
template <class R> struct Side {
    V3<R> v, w;
    M3<R> I;
    R im;
    bool kin;
    __device__ void load(const Bodies<R>& B, int i) {   // all but the velocities
        kin = (B.flags[i] & BF_KINEMATIC) != 0;
        im = B.at(INVM, i);
        I = B.mat(I00, i);
        v = V3<R>(0, 0, 0);
        w = V3<R>(0, 0, 0);
    }
};
// FrictionContactConstraint::iterateSequentialImpulse (friction_contact_constraint.cpp:75-108) for
// one point: the row applied to the two bodies' temporary velocities and its accumulators updated
template <class R> __device__ __forceinline__ void si_row(RowReg<R>& q, Side<R>& a, Side<R>& b) {
    const V3<R> vr = a.v + cross(a.w, q.ra) - b.v - cross(b.w, q.rb);
    R ni = q.rhs - dot(q.n, vr) * q.njmj;
    ni = ni > -q.nacc ? ni : -q.nacc;
    q.nacc += ni;
    R tt0 = q.t0acc - dot(q.t0, vr) * q.t0jmj;
    R tt1 = q.t1acc - dot(q.t1, vr) * q.t1jmj;
    const R scale = friction_scale(q.mu * q.nacc, tt0 * tt0 + tt1 * tt1);
    if (scale < 1) { tt0 *= scale; tt1 *= scale; }
    const V3<R> imp = ni * q.n + (tt0 - q.t0acc) * q.t0 + (tt1 - q.t1acc) * q.t1;
    q.t0acc = tt0;
    q.t1acc = tt1;
    if (!a.kin) { a.v = a.v + imp * a.im; a.w = a.w + mv(a.I, cross(q.ra, imp)); }
    const V3<R> nimp = -imp;
    if (!b.kin) { b.v = b.v + nimp * b.im; b.w = b.w + mv(b.I, cross(q.rb, nimp)); }
}
// All points of one result, in order; q holds the first row, before and after.  The next row is loaded
// while one is worked on: its loads would otherwise wait behind the stores of the accumulators, and
// the first row's until the bodies' velocities arrive.
template <class R> __device__ __forceinline__ void si_rows(const Rows<R>& rows, int r0, int np, RowReg<R>& q, Side<R>& a, Side<R>& b) {
    for (int k = 0; k < np; k++) {
        RowReg<R> next;
        if (np > 1) row_load(rows, r0 + (k + 1 < np ? k + 1 : 0), next);
        si_row(q, a, b);
        row_store_acc(rows, r0 + k, q);
        if (np > 1) q = next;
    }
}

// ---------------------------------------------------------------- joints
// Ball/Hinge/SliderJointConstraint::initSequentialImpulse and iterateSequentialImpulse
// (ball_joint_constraint.cpp:6-27, hinge_joint_constraint.cpp:6-97, slider_joint_constraint.cpp:7-65)
// in the reference's operation order.  A kinematic body contributes no inverse mass or inertia
// (RigidBody::getKinematicInvMass / getKinematicWorldInvInertia) and takes no impulse.
template <class R> __device__ __forceinline__ M3<R> skew3(const V3<R>& v) {   // Constraint::getSkewSymmetricMatrix
    M3<R> m;
    m.m[0][0] = 0; m.m[0][1] = -v.z; m.m[0][2] = v.y;
    m.m[1][0] = v.z; m.m[1][1] = 0; m.m[1][2] = -v.x;
    m.m[2][0] = -v.y; m.m[2][1] = v.x; m.m[2][2] = 0;
    return m;
}
template <class R> __device__ __forceinline__ M3<R> madd3(const M3<R>& a, const M3<R>& b) {
    M3<R> o;
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) o.m[i][j] = a.m[i][j] + b.m[i][j];
    return o;
}
template <class R> __device__ __forceinline__ V3<R> jp3(const R* p, int k) { return V3<R>(p[k], p[k + 1], p[k + 2]); }
template <class R> __device__ __forceinline__ void jw3(R* p, int k, const V3<R>& v) { p[k] = v.x; p[k + 1] = v.y; p[k + 2] = v.z; }
template <class R> __device__ __forceinline__ M3<R> jp9(const R* p, int k) {
    M3<R> m;
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) m.m[i][j] = p[k + i * 3 + j];
    return m;
}
template <class R> __device__ __forceinline__ void jw9(R* p, int k, const M3<R>& m) {
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) p[k + i * 3 + j] = m.m[i][j];
}

template <class R>
__global__ void k_joint_init(Joints<R> J, Bodies<R> B, StepParams P) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= J.n) return;
    const int ia = J.body[j].x, ib = J.body[j].y, type = J.type[j], fl = J.flag[j];
    const bool ka = (B.flags[ia] & BF_KINEMATIC) != 0, kb = (B.flags[ib] & BF_KINEMATIC) != 0;
    const R* q = J.param + (size_t)j * NJP;
    R* w = J.row + (size_t)j * NJR;
    const R dt = R(P.dt), kerp = R(0.2);
    const Xf<R> ta = B.xf(ia), tb = B.xf(ib);
    const V3<R> anc_a = jp3(q, JP_ANCHOR_A), anc_b = jp3(q, JP_ANCHOR_B);
    const V3<R> ra = mv(ta.b, anc_a), rb = mv(tb.b, anc_b);
    jw3(w, JR_RA, ra);
    jw3(w, JR_RB, rb);
    const R ims = (ka ? R(0) : B.at(INVM, ia)) + (kb ? R(0) : B.at(INVM, ib));
    const M3<R> Ia = ka ? M3<R>() : B.mat(I00, ia), Ib = kb ? M3<R>() : B.mat(I00, ib);
    const V3<R> rel = ta.apply(anc_a) - tb.apply(anc_b);
    auto ball = [&]() {
        M3<R> d;
        for (int k = 0; k < 3; k++) d.m[k][k] = ims;
        const M3<R> jmj = inverse3(madd3(madd3(d, world_inertia(skew3(ra), Ia)), world_inertia(skew3(rb), Ib)));
        jw9(w, JR_JMJ_BALL, jmj);
        jw3(w, JR_RHS_BALL, mv(jmj, rel) * (-kerp / dt));
    };
    if (type == JT_BALL) { ball(); return; }
    const V3<R> wax = mv(ta.b, jp3(q, JP_AXIS_A)), wbx = mv(tb.b, jp3(q, JP_AXIS_B));
    V3<R> t0, t1, u0, u1;
    ortho_units(jp3(q, JP_AXIS_A), t0, t1);
    t0 = mv(ta.b, t0);
    t1 = mv(ta.b, t1);
    jw3(w, JR_WAX, wax);
    jw3(w, JR_T0, t0);
    jw3(w, JR_T1, t1);
    if (type == JT_HINGE) {
        const bool lim = (fl & 1) != 0, mot = (fl & 2) != 0;
        if (lim) {
            ortho_units(jp3(q, JP_AXIS_B), u0, u1);
            u0 = mv(tb.b, u0);
        }
        ball();
        const M3<R> Is = madd3(Ia, Ib);
        const R j0 = R(1.0) / dot(t0, mv(Is, t0)), j1 = R(1.0) / dot(t1, mv(Is, t1));
        const V3<R> u = cross(wax, wbx);
        w[JR_JMJ2] = j0;
        w[JR_JMJ2 + 1] = j1;
        w[JR_RHS2] = j0 * (dot(u, t0) * kerp / dt);
        w[JR_RHS2 + 1] = j1 * (dot(u, t1) * kerp / dt);
        R jml = 0;
        if (mot || lim) jml = R(1.0) / dot(wax, mv(Is, wax));
        w[JR_JMJ_ML] = jml;
        if (mot) w[JR_RHS_MOTOR] = jml * -q[JP_SPEED];
        w[JR_LIMIT] = 0;
        if (lim) {
            const R c = dot(t0, u0), sn = dot(cross(t0, u0), wax);
            const R angle = atan2(sn, c);
            if (angle < q[JP_MIN]) {
                w[JR_LIMIT] = 1;
                w[JR_RHS_LIMIT] = -jml * (q[JP_MIN] - angle) * kerp / dt;
            } else if (angle > q[JP_MAX]) {
                w[JR_LIMIT] = 1;
                w[JR_RHS_LIMIT] = -jml * (q[JP_MAX] - angle) * kerp / dt;
            }
        }
        return;
    }
    // slider
    ortho_units(jp3(q, JP_AXIS_B), u0, u1);
    const V3<R> ts[2] = {t0, t1};
    R jp[2];
    for (int k = 0; k < 2; k++) {
        const V3<R> xa = cross(ra, ts[k]), xb = cross(rb, ts[k]);
        jp[k] = R(1.0) / (ims + dot(mv(Ia, xa), xa) + dot(mv(Ib, xb), xb));
    }
    w[JR_JMJ2] = jp[0];
    w[JR_JMJ2 + 1] = jp[1];
    w[JR_RHS2] = jp[0] * (dot(rel, t0) * (-kerp / dt));
    w[JR_RHS2 + 1] = jp[0] * (dot(rel, t1) * (-kerp / dt));   // the first row's jmj, as slider_joint_constraint.cpp:40
    jw9(w, JR_JMJ_ROT, inverse3(madd3(Ia, Ib)));
}

// RigidBody::applyTempImpulse / applyTempAngularImpulse (rigidbody.cpp:166-181)
template <class R> __device__ __forceinline__ void jt_impulse(Side<R>& s, const V3<R>& r, const V3<R>& imp) {
    if (s.kin) return;
    s.v = s.v + imp * s.im;
    s.w = s.w + mv(s.I, cross(r, imp));
}
template <class R> __device__ __forceinline__ void jt_ang_impulse(Side<R>& s, const V3<R>& imp) {
    if (s.kin) return;
    s.w = s.w + mv(s.I, imp);
}

template <class R> __device__ void joint_iterate(const Joints<R>& J, int j, Side<R>& a, Side<R>& b) {
    const int type = J.type[j], fl = J.flag[j];
    const R* w = J.row + (size_t)j * NJR;
    const V3<R> ra = jp3(w, JR_RA), rb = jp3(w, JR_RB);
    const V3<R> va = a.v + cross(a.w, ra), vb = b.v + cross(b.w, rb);
    if (type == JT_SLIDER) {
        const V3<R> t0 = jp3(w, JR_T0), t1 = jp3(w, JR_T1);
        const R p0 = w[JR_RHS2] - w[JR_JMJ2] * dot(t0, va - vb);
        const R p1 = w[JR_RHS2 + 1] - w[JR_JMJ2 + 1] * dot(t1, va - vb);
        const V3<R> pv = t0 * p0 + t1 * p1;
        jt_impulse(a, ra, pv);
        jt_impulse(b, rb, -pv);
        const V3<R> rot = mv(jp9(w, JR_JMJ_ROT), a.w - b.w);
        const V3<R> ri = -rot;
        jt_ang_impulse(a, ri);
        jt_ang_impulse(b, -ri);
        return;
    }
    const V3<R> bi = jp3(w, JR_RHS_BALL) - mv(jp9(w, JR_JMJ_BALL), va - vb);
    jt_impulse(a, ra, bi);
    jt_impulse(b, rb, -bi);
    if (type == JT_BALL) return;
    // hinge rows; motor and limit read the angular velocities left by the impulses before them
    const V3<R> t0 = jp3(w, JR_T0), t1 = jp3(w, JR_T1), wax = jp3(w, JR_WAX);
    const V3<R> dw = a.w - b.w;
    const R h0 = w[JR_RHS2] - w[JR_JMJ2] * dot(t0, dw);
    const R h1 = w[JR_RHS2 + 1] - w[JR_JMJ2 + 1] * dot(t1, dw);
    const V3<R> iv = t0 * h0 + t1 * h1;
    jt_ang_impulse(a, iv);
    jt_ang_impulse(b, -iv);
    if (fl & 2) {
        const R mi = w[JR_RHS_MOTOR] - w[JR_JMJ_ML] * dot(wax, a.w - b.w);
        jt_ang_impulse(a, wax * mi);
        jt_ang_impulse(b, -wax * mi);
    }
    if ((fl & 1) && w[JR_LIMIT] != 0) {
        const R delta = dot(wax, a.w - b.w);
        const R nd = delta * w[JR_RHS_LIMIT] > 0 ? R(0) : delta;
        const R li = w[JR_RHS_LIMIT] - w[JR_JMJ_ML] * nd;
        jt_ang_impulse(a, wax * li);
        jt_ang_impulse(b, -wax * li);
    }
}

// Island items: a contact result index, or a joint index with kJointItem set.  Within an island
// the contacts come first in result order, then the joints in order, so one pass over an island's
// items is the reference's iteration (every contact, then every other constraint) restricted to
// the island.
constexpr uint32_t kJointItem = 0x80000000u;
template <class R> __device__ __forceinline__ int2 item_bodies(uint32_t item, const Results<R>& res, const Joints<R>& J) {
    if (item & kJointItem) return J.body[item & ~kJointItem];
    return make_int2(res.a[item], res.b[item]);
}
// ---------------------------------------------------------------- contact islands
// Islands: connected components of dynamic bodies linked by contact results (a kinematic body
// links nothing: its temporary velocity never changes).  Results of different islands touch
// disjoint dynamic bodies, so running each island's results in the reference's global order
// (SequentialImpulseSolver::solve, sequential_impulse_solver.cpp:60-69) yields exactly the
// reference's velocities while islands proceed in parallel.
__device__ __forceinline__ int uf_find(const int* parent, int x) {
    int p = parent[x];
    while (p != x) { x = p; p = parent[x]; }   // parents always point to smaller indices
    return x;
}
__device__ __forceinline__ void uf_union(int* parent, int a, int b) {
    for (;;) {
        a = uf_find(parent, a);
        b = uf_find(parent, b);
        if (a == b) return;
        if (a < b) { const int t = a; a = b; b = t; }
        // hook the larger root below the smaller one; retry if another thread moved it first
        if (atomicCAS(&parent[a], a, b) == a) return;
    }
}

__global__ void k_step_counters(const int* status, const int* rows, const int* active, const int* islands, const int* n_big, const int* big,
                                const int* isl_levels, const int* colors, const int* cls, int* out);

} // namespace pe
