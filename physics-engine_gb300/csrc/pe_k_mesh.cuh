// Kernels of the rigid-body step, part 5: pairs with a concave mesh or a compound shape.
#pragma once
#include "pe_k_sat.cuh"

namespace pe {

// CompoundCompoundCollisionAlgorithm::processCollision (compound_compound_collision_algorithm.cpp:8-46)
// and the Concave*CollisionAlgorithm family, one warp per pair.  A compound second swaps the pair
// (shapes, transforms and the result's objects: ContactResult::setObjects(B, A), so the result names
// the compound as object A); then every child of the compound, against every child of a second
// compound or against the other shape, runs its shape pair's algorithm into the same contact cache
// at the child's world transform (body transform * local transform).  Local contact positions stay
// relative to the bodies.
//
// A pair is cut into pieces that do not depend on each other: one child against one child or shape,
// and against a concave mesh one face (for a cylinder, one face's sides or one face's edges: the
// reference makes two passes over the faces).  Lanes run a piece each into a recorder, and lane 0 adds
// the recorded points to the pair's cache in the reference's order; a piece with more points than a
// recorder holds runs again on lane 0.  The leaves of a concave mesh's face tree are tested 32 at a
// time.  (What bounds a pair is the serial code of one piece; with one thread per pair, walking some
// 2,000 leaves and then face after face, a step of 300 bodies on a terrain of 4,608 triangles spent 13.9 ms
// on its compound pairs and 4.5 ms on the others beside them, and took 18.9 ms; it takes 0.7 ms so.)
constexpr int kMeshPoints = 12, kMeshQueue = 64;
struct MeshPiece {
    int i, j;      // child of A, of B; -1: the shape itself
    int face;      // kPieceWhole: the whole pair of shapes; kPieceEnd: a mesh's faces are done
    int pass;      // cylinder against a face: 0 sides, 1 edges; kPassHull: a hull against a face
};
constexpr int kPassHull = 2;
constexpr int kPieceWhole = -1, kPieceEnd = -2;

// the mesh's face f against the convex shape on the other side; `c` names the pair's shapes in order
template <class R, class C> __device__ void mesh_face(Pair<R, C>& c, int f, int pass) {
    const bool a_mesh = c.sa.type == ST_CONCAVE;
    const ShapeView<R>& m = a_mesh ? c.sa : c.sb;
    const ShapeView<R>& o = a_mesh ? c.sb : c.sa;
    const Xf<R>& tm = a_mesh ? c.xa : c.xb;
    const Xf<R>& to = a_mesh ? c.xb : c.xa;
    c.c->swap = a_mesh;
    if (o.type == ST_SPHERE) {
        sphere_face(c, m, tm, tm.inv_apply(to.o), o.radius, f);
    } else if (o.type == ST_CYLINDER) {
        const Xf<R> rel = tm.inverse() * to;
        const CylinderFrame<R> q{rel.b.col(1), rel.o, o.radius, o.height / R(2.0), tm};
        if (pass == 0) cylinder_face_sides(c, m, q, f);
        else cylinder_face_edges(c, m, q, f);
    } else {
        concave_face(c, m, o, tm, to, f);
    }
}

// the shapes and transforms of children (or of the pair's shapes themselves) i and j
template <class R, class C>
__device__ __forceinline__ void mesh_place(const Pair<R>& pr, const ShapeTable<R>& S, int i, int j, C* sink, Pair<R, C>& c) {
    c.ref_scale = pr.ref_scale;
    c.margin = pr.margin;
    c.c = sink;
    c.sa = i < 0 ? pr.sa : S.view(S.c_shape[i]);
    c.xa = i < 0 ? pr.xa : pr.xa * S.child_xf(i);
    c.sb = j < 0 ? pr.sb : S.view(S.c_shape[j]);
    c.xb = j < 0 ? pr.xb : pr.xb * S.child_xf(j);
}
// out of line: one copy per sink, with its clipping buffers on the stack only while it runs
template <class R, class C> __device__ __noinline__ void mesh_piece(const MeshPiece& q, const Pair<R>& pr, const ShapeTable<R>& S, C* sink) {
    if (q.face == kPieceEnd) { sink->swap = false; return; }
    Pair<R, C> c;
    mesh_place(pr, S, q.i, q.j, sink, c);
    if (q.face == kPieceWhole) collide(c, pair_class(c.sa.type, c.sb.type));
    else mesh_face(c, q.face, q.pass);
}
// A mesh's face against a hull is the work of up to 128 axes, each projecting every vertex: by one lane,
// hundreds of microseconds.  The lanes first hold a face each against its own normal, which most faces
// near a hull are apart along (an axis that separates ends the reference's test, and nothing has been
// added before the edge axes, which a face has none of); the faces left meet the hull by the whole warp,
// one after the other in their turn.
template <class R, class F> __device__ __forceinline__ void mesh_hull_pair(const MeshPiece& q, const Pair<R>& pr, const ShapeTable<R>& S, Cache<R>* cache, F&& f) {
    Pair<R> c;
    mesh_place(pr, S, q.i, q.j, cache, c);
    const bool a_mesh = c.sa.type == ST_CONCAVE;
    FaceBuf<R> b;
    Pair<R> s = face_pair(c, a_mesh ? c.sa : c.sb, a_mesh ? c.sb : c.sa, a_mesh ? c.xa : c.xb, a_mesh ? c.xb : c.xa, q.face, b);
    f(s, a_mesh);
}
template <class R> __device__ __noinline__ bool mesh_hull_near(const MeshPiece& q, const Pair<R>& pr, const ShapeTable<R>& S, Cache<R>* cache) {
    bool near = true;
    mesh_hull_pair(q, pr, S, cache, [&](Pair<R>& s, bool) {
        V3<R> n = mv(s.tb().b, s.sb.face_normal(0)), wa, wb;
        if (dot(s.ta().o - s.tb().o, n) < 0) n = n * R(-1.0);
        R d;
        near = sep_test(s, n, d, wa, wb);
    });
    return near;
}
template <class R> __device__ __noinline__ void mesh_hull_face(const MeshPiece& q, const Pair<R>& pr, const ShapeTable<R>& S, Cache<R>* cache, int lane) {
    mesh_hull_pair(q, pr, S, cache, [&](Pair<R>& s, bool a_mesh) {
        if (lane == 0) cache->swap = a_mesh;
        sat_warp(s, lane);
    });
}
template <class R> __device__ __noinline__ void mesh_sat(const Pair<R>& pr, const ShapeTable<R>& S, int i, int j, Cache<R>* cache, int lane) {
    Pair<R> c;
    mesh_place(pr, S, i, j, cache, c);
    sat_warp(c, lane);
}

template <class R>
__global__ void __launch_bounds__(32)
k_np_mesh(const int2* rng, int* cursor, const int* order, const int2* pairs, Bodies<R> B, ShapeTable<R> S, Results<R> res,
          const int* pair_scene_off, const int* prev_off) {
    __shared__ R rec[32][kMeshPoints * kRecReals];
    __shared__ int rec_n[32], rec_swap[32];
    __shared__ MeshPiece queue[kMeshQueue];
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    warp_items(*rng, cursor, [&](int t) {
        const int p = order[t];
        Cache<R> cache;
        Pair<R> pr;
        np_setup(p, pairs, B, S, res, pair_scene_off, prev_off, cache, pr, lane == 0);
        int sa = B.shape[pairs[p].x], sb = B.shape[pairs[p].y];
        bool swapped = false;
        if (pr.sb.type == ST_COMPOUND) {
            const ShapeView<R> v = pr.sa; pr.sa = pr.sb; pr.sb = v;
            const Xf<R> x = pr.xa; pr.xa = pr.xb; pr.xb = x;
            if (lane == 0) {
                const Xf<R> y = cache.ta; cache.ta = cache.tb; cache.tb = y;
                const R z = cache.scale_a; cache.scale_a = cache.scale_b; cache.scale_b = z;
            }
            const int w = sa; sa = sb; sb = w;
            swapped = true;
        }
        int qn = 0;   // queued pieces
        auto flush = [&](int n) {   // runs the first n (at most 32) queued pieces
            __syncwarp();
            bool by_warp = false;
            if (lane < n) {
                if (queue[lane].pass == kPassHull) {
                    by_warp = mesh_hull_near(queue[lane], pr, S, &cache);
                    rec_n[lane] = 0;
                    rec_swap[lane] = Recorder<R>::kSwapInherit;
                } else {
                    Recorder<R> r{rec[lane], 0, kMeshPoints, Recorder<R>::kSwapInherit};
                    mesh_piece(queue[lane], pr, S, &r);
                    rec_n[lane] = r.n;
                    rec_swap[lane] = r.swap;
                }
            }
            unsigned whole = __ballot_sync(full, by_warp);
            for (int l = 0; l < n;) {
                const int stop = whole ? __ffs(whole) - 1 : n;
                if (lane == 0)
                    for (; l < stop; l++) {
                        if (rec_n[l] > kMeshPoints) mesh_piece(queue[l], pr, S, &cache);
                        else Recorder<R>{rec[l], rec_n[l], kMeshPoints, rec_swap[l]}.replay(cache);
                    }
                __syncwarp();
                if (stop < n) mesh_hull_face(queue[stop], pr, S, &cache, lane);
                whole &= whole - 1;
                l = stop + 1;
            }
            __syncwarp();
            if (lane < qn - n) queue[lane] = queue[n + lane];   // at most 31 stay
            qn -= n;
            __syncwarp();
        };
        auto push = [&](bool mine, int at, int count, const MeshPiece& q) {   // `count` pieces, this lane's at `at`
            if (mine) queue[qn + at] = q;
            qn += count;
            if (qn >= 32) flush(32);
        };
        auto meet = [&](int i, int j) {
            Pair<R> c;
            mesh_place(pr, S, i, j, &cache, c);
            const ShapeView<R>&va = c.sa, &vb = c.sb;
            const Xf<R>&xa = c.xa, &xb = c.xb;
            const int cls = pair_class(va.type, vb.type);
            if (cls == PC_CONVEX) {   // the whole warp on one pair of convex shapes, points added as they come
                flush(qn);
                mesh_sat(pr, S, i, j, &cache, lane);
                __syncwarp();
                return;
            }
            if (cls != PC_CONCAVE) {
                push(lane == 0, 0, 1, MeshPiece{i, j, kPieceWhole, 0});
                return;
            }
            const bool a_mesh = va.type == ST_CONCAVE;
            if (a_mesh && vb.type == ST_CONCAVE) return;   // concave-concave has no algorithm
            const ShapeView<R>& m = a_mesh ? va : vb;
            const ShapeView<R>& o = a_mesh ? vb : va;
            const Xf<R>& tm = a_mesh ? xa : xb;
            const Xf<R>& to = a_mesh ? xb : xa;
            V3<R> aa, bb;   // the convex shape's box in the mesh's frame
            if (o.type == ST_SPHERE) {
                const V3<R> rel = tm.inv_apply(to.o), r(o.radius, o.radius, o.radius);
                aa = rel - r; bb = rel + r;
            } else {
                shape_aabb(o, tm.inverse() * to, aa, bb);
            }
            const int passes = o.type == ST_CYLINDER ? 2 : 1, hull = o.type == ST_HULL ? kPassHull : 0;
            // mesh_query: leaves in descending order, the faces of an overlapping leaf ascending
            // (four rounds of 32 leaves at a time, their boxes loaded first: 16 rounds of the 512 leaves of a
            // 4,608-triangle terrain, once per child and pass, each waited for memory otherwise)
            constexpr int U = 4;
            for (int pass = 0; pass < passes; pass++)
                for (int l0 = m.nl - 1; l0 >= 0; l0 -= 32 * U) {
                    unsigned hit = 0;
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int l = l0 - 32 * u - lane, k = l >= 0 ? l : 0;
                        const R* mn = m.l_min + k * 3;
                        const R* mx = m.l_max + k * 3;
                        const V3<R> lo(mn[0], mn[1], mn[2]), hi(mx[0], mx[1], mx[2]);
                        if (l >= 0 && !(lo.x > bb.x || lo.y > bb.y || lo.z > bb.z) && !(hi.x < aa.x || hi.y < aa.y || hi.z < aa.z)) hit |= 1u << u;
                    }
                    if (!__any_sync(full, hit)) continue;
#pragma unroll 1
                    for (int u = 0; u < U; u++)
                        for (unsigned hits = __ballot_sync(full, hit >> u & 1u); hits; hits &= hits - 1) {
                            const int leaf = l0 - 32 * u - (__ffs(hits) - 1), first = m.l_beg[leaf], cnt = m.l_cnt[leaf];
                            for (int f0 = 0; f0 < cnt; f0 += 32)
                                push(f0 + lane < cnt, lane, min(32, cnt - f0), MeshPiece{i, j, first + f0 + lane, pass + hull});
                        }
                }
            push(lane == 0, 0, 1, MeshPiece{i, j, kPieceEnd, 0});
        };
        const int ib = pr.sa.type == ST_COMPOUND ? S.c_beg[sa] : -1, ie = pr.sa.type == ST_COMPOUND ? ib + S.c_cnt[sa] : 0;
        const int jb = pr.sb.type == ST_COMPOUND ? S.c_beg[sb] : -1, je = pr.sb.type == ST_COMPOUND ? jb + S.c_cnt[sb] : 0;
        for (int i = ib; i < ie; i++)
            for (int j = jb; j < je; j++) meet(i, j);
        flush(qn);
        if (lane == 0) np_finish(p, pairs, B, res, cache, swapped);
    });
}

} // namespace pe
