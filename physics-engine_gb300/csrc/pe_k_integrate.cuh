// Kernels of the rigid-body step, part 1: integration (RigidBody::step and the world AABB).
#pragma once
#include <cstdint>
#include <cooperative_groups.h>
#include "pe_state.cuh"

namespace pe {

constexpr int kBlock = 256;

constexpr int kWideHull = 96;   // vertices above which a mesh's box is taken by a warp
// ===================================================================== integration
// World::updateObjectStatus (world.cpp:35-119) + applyExternalForce (:121-127), fused per body.
template <class R>
__global__ void k_integrate(Bodies<R> B, ShapeTable<R> S, StepParams P, int do_move) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned in = __ballot_sync(0xffffffffu, i < B.n);
    if (i >= B.n) return;
    const ShapeView<R> sh = S.view(B.shape[i]);
    const bool kin = (B.flags[i] & BF_KINEMATIC) != 0;
    Xf<R> t = B.xf(i);
    const R dt = R(P.dt);
    if (!kin && do_move) {
        // RigidBody::step (rigidbody.cpp:207-243)
        const V3<R> v = B.vec(VX, i), w = B.vec(WX, i);
        t.o = t.o + v * dt;
        const Quat<R> q = quat_from_basis(t.b);
        const V3<R> dr = w * dt * R(0.5);
        Quat<R> d0;
        d0.x = dr.x; d0.y = dr.y; d0.z = dr.z; d0.w = 0;
        const Quat<R> dq = quat_mul(d0, q);
        Quat<R> qn;
        qn.x = q.x + dq.x; qn.y = q.y + dq.y; qn.z = q.z + dq.z; qn.w = q.w + dq.w;
        quat_normalize(qn);
        t.b = quat_to_basis(qn);
        const M3<R> iw = world_inertia(t.b, B.mat(L00, i));
        B.set_mat(I00, i, iw);
        B.set_vec(OX, i, t.o);
        B.set_mat(B00, i, t.b);
        // applyDamping (rigidbody.cpp:201-204)
        const R ld = pow(R(1.0) - B.at(LDAMP, i), dt), ad = pow(R(1.0) - B.at(ADAMP, i), dt);
        V3<R> nv = v * ld, nw = w * ad;
        // applyExternalForce: force = 0 + g*m, v += force * inv_mass * dt, w += Iw * (torque * dt)
        const R m = B.at(MASS, i), im = B.at(INVM, i);
        const V3<R> force = V3<R>(0, 0, 0) + V3<R>(R(P.g[0]), R(P.g[1]), R(P.g[2])) * m;
        nv = nv + force * im * dt;
        nw = nw + mv(iw, V3<R>(0, 0, 0) * dt);
        B.set_vec(VX, i, nv);
        B.set_vec(WX, i, nw);
    }
    V3<R> mn, mx;
    const bool wide = (sh.type == ST_HULL || sh.type == ST_CONCAVE) && sh.nv > kWideHull;
    if (sh.type == ST_COMPOUND) compound_aabb(S, B.shape[i], t, mn, mx);
    else if (!wide) shape_aabb(sh, t, mn, mx);
    // a mesh of many vertices takes the whole warp (one thread walked a terrain of 2,401 vertices in 151 us)
    const int lane = threadIdx.x & 31;
    for (unsigned todo = __ballot_sync(in, wide); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        Xf<R> x;
        x.o = V3<R>(__shfl_sync(in, t.o.x, src), __shfl_sync(in, t.o.y, src), __shfl_sync(in, t.o.z, src));
        for (int r = 0; r < 3; r++) for (int c = 0; c < 3; c++) x.b.m[r][c] = __shfl_sync(in, t.b.m[r][c], src);
        ShapeView<R> part = S.view(B.shape[__shfl_sync(in, i, src)]);
        const int per = (part.nv + __popc(in) - 1) / __popc(in), v0 = min(lane * per, part.nv);   // lanes in `in` are the first ones
        part.hv += v0 * 3;
        part.nv = min(per, part.nv - v0);
        V3<R> a, b;
        Xf<R> turn = x;
        turn.o = V3<R>(0, 0, 0);
        shape_aabb(part, turn, a, b);
        for (int o = 16; o > 0; o >>= 1)
            for (int d = 0; d < 3; d++) {
                const R u = __shfl_xor_sync(in, a[d], o), w = __shfl_xor_sync(in, b[d], o);
                if ((in >> (lane ^ o)) & 1u) { a[d] = a[d] < u ? a[d] : u; b[d] = b[d] > w ? b[d] : w; }
            }
        // (lanes past the world's last body are missing, so only lane 0 is sure to have met every part)
        for (int d = 0; d < 3; d++) { a[d] = __shfl_sync(in, a[d], 0); b[d] = __shfl_sync(in, b[d], 0); }
        if (lane == src) { mn = a + x.o; mx = b + x.o; }
    }
    B.set_vec(MNX, i, mn);
    B.set_vec(MXX, i, mx);
    // RigidBody::getAABBScale (rigidbody.cpp:119-123)
    const R sc = norm(mx - mn), df = norm(mx + mn - t.o * R(2));
    B.at(SCALE, i) = (sc + df) * R(0.5);
}

// unit direction of every hull edge, normalized(a - b) in the world's real type: the staged SAT
// reads these instead of normalising each edge of both shapes for every pair
template <class R>
__global__ void k_hull_edge_dirs(int n, const R* ea, const R* eb, R* ed) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const V3<R> a(ea[3 * e], ea[3 * e + 1], ea[3 * e + 2]), b(eb[3 * e], eb[3 * e + 1], eb[3 * e + 2]);
    const V3<R> d = normalized(a - b);
    ed[3 * e] = d.x; ed[3 * e + 1] = d.y; ed[3 * e + 2] = d.z;
}

} // namespace pe
