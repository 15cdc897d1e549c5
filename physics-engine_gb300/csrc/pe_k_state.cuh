// Kernels of the rigid-body step, part 8: body-state transfer in the C ABI's layout.
#pragma once
#include "pe_k_flow.cuh"

namespace pe {

// Body-state transfer in the C ABI's layout: per group g, fields k0[g] .. k0[g] + nk[g] - 1 of every body,
// body-major at ptr[g], in the caller's type T (double, or float, pe::Real of the reference's default
// build).  ptr is a device staging buffer, or the caller's own page-locked memory (World::direct).  One
// thread per value, groups along y, so that the caller's side is read and written in whole lines (a
// thread per body wrote its 18 values one after the other: 11 us for 1,000 bodies).
template <class T> struct XferGroups {
    int k0[8], nk[8];
    T* ptr[8];
    int n;
};
template <class R, class T>
__global__ void k_state_pack(Bodies<R> B, XferGroups<T> G) {
    const int g = blockIdx.y, nk = G.nk[g];
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(e / nk);
    if (i < B.n) G.ptr[g][e] = (T)B.at(G.k0[g] + (int)(e - (long long)i * nk), i);
}
// the inverse; with so, smn, smx >= 0 (the groups of origin, AABB min and max) it also sets the
// body's AABB scale from them, as RigidBody::getAABBScale does (rigidbody.cpp:119-123)
template <class R, class T>
__global__ void k_state_unpack(Bodies<R> B, XferGroups<T> G, int so, int smn, int smx) {
    const int g = blockIdx.y, nk = G.nk[g];
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(e / nk);
    if (i < B.n) B.at(G.k0[g] + (int)(e - (long long)i * nk), i) = R(G.ptr[g][e]);
    if (g == so && e < B.n) {
        auto v3 = [&](int q) {
            const T* v = G.ptr[q] + (size_t)e * 3;
            return V3<R>(R(v[0]), R(v[1]), R(v[2]));
        };
        const V3<R> a = v3(smn), d = v3(smx), org = v3(so);
        const R sc = norm(d - a), df = norm(d + a - org * R(2));
        B.at(SCALE, (int)e) = (sc + df) * R(0.5);
    }
}

} // namespace pe
