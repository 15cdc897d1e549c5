// Kernels of the rigid-body step, part 7: the solver's iterations, run as a flow of body velocities
// between island items.
//
// An island's items (contact results, then joints) act on their two bodies' temporary velocities in
// a fixed order.  Instead of running that order level by level with a barrier after every level, each
// body's velocity is a token that its items hand on: an item runs once it holds the tokens of its
// dynamic bodies, then passes each to the body's next item, the last one back to the first for the
// next iteration.  Every body takes its updates in the same order as before, so the results are the
// same bits, while different parts of an island, and its successive iterations, overlap: the steps
// in a row are the longest chain of the unrolled order (472 for a 55,690-contact island of 304
// levels and 10 iterations) instead of levels x iterations (3,040), and none waits for a barrier.
//
// Islands of up to kWarpIsland items run inside one warp with the tokens in shared memory
// (k_isl_warp); larger ones over the whole grid with the tokens in global memory (k_isl_flow).
//
// A caller's result may name one body on both sides (SELF; no sweep gives such a pair).  Its item holds
// the body's token once, on side b; side a starts every iteration from the same velocities and is dropped
// after it.
#pragma once
#include "pe_k_solver.cuh"

namespace pe {

constexpr int kMaxColors = 512;      // colours reported for an island of up to big_island_items items
constexpr int kMaxColorsBig = 1024;  // first-fit colours of a bigger island, the last one for leftovers

// an item's dynamic bodies, loaded with everything but the velocities
template <class R, bool JOINTS> struct Item {
    uint32_t id;
    int ia, ib, r0, np;
    Side<R> a, b;
    RowReg<R> q;   // a result's first row
    __device__ __forceinline__ void load(uint32_t item, const Results<R>& res, const Joints<R>& J, const Bodies<R>& B, const Rows<R>& rows) {
        id = item;
        if (JOINTS && (item & kJointItem)) {
            const int2 q = J.body[item & ~kJointItem];
            ia = q.x; ib = q.y; r0 = 0; np = 0;
        } else {
            ia = res.a[item]; ib = res.b[item]; r0 = (int)item * kSlots; np = res.npts[item];
            row_load(rows, r0, q);
        }
        a.load(B, ia);
        b.load(B, ib);
    }
    __device__ __forceinline__ void iterate(const Joints<R>& J, const Rows<R>& rows) {
        if (JOINTS && (id & kJointItem)) joint_iterate(J, (int)(id & ~kJointItem), a, b);
        else si_rows(rows, r0, np, q, a, b);
    }
};

// ---------------------------------------------------------------- one result by a whole warp (FP64)
// A double-precision instruction holds a warp for 64 cycles on this chip, with one lane in it or 32,
// and the next one waits even if it does not depend on it (measured: dependent and independent chains
// alike), so a row costs its instruction count: some 170, 5 us, when one lane runs it.  Here lanes 0 to 8
// share a row: lane 3 s + k holds component k of body s's velocities, lane 3 q + k component k of
// direction q (normal, tangents), some 40 instructions with shuffles between them.  Operations and
// their order are si_row's.  The step of a 1,000-box tower: 7,079 / 3,181 us.  (Not in FP32: there the
// shuffles take longer than the instructions they save, 855 / 1,180 us.)
struct WarpRow {   // what a lane holds of one row
    double r1, r2, d, jmj, base, mu, nacc;
    __device__ __forceinline__ void load(const Rows<double>& rows, int row, int s, int q, int k) {
        const double* p = rows.f + (size_t)row * NRF;
        const int k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
        r1 = p[4 * s + k1]; r2 = p[4 * s + k2];
        d = p[8 + 4 * q + k];
        jmj = p[q == 0 ? 3 : q == 1 ? 11 : 15];
        base = p[q == 0 ? 7 : 21 + q];
        mu = p[20]; nacc = p[21];
    }
};
constexpr int kWarpItem = 32;   // doubles of an item in shared memory: velocities of a and b (6 each), inverse inertias (9 each), inverse masses
__device__ __forceinline__ double shfl_d(double x, int src) { return __shfl_sync(0xffffffffu, x, src); }
// item's rows r0 .. r0 + np - 1 (every lane's arguments the same); its velocities are updated in `item`
__device__ __forceinline__ void si_rows_warp(const Rows<double>& rows, int r0, int np, bool kin_a, bool kin_b, double* item, int lane) {
    const int l = lane < 9 ? lane : 8, q = l / 3, k = l - 3 * q, s = q < 2 ? q : 1;   // lanes past the last role repeat one
    const int k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1, at = 3 * s;
    double v = item[6 * s + k], w = item[6 * s + 3 + k];
    const double i0 = item[12 + 9 * s + 3 * k], i1 = item[13 + 9 * s + 3 * k], i2 = item[14 + 9 * s + 3 * k], im = item[30 + s];
    const bool kin = s == 0 ? kin_a : kin_b;
    WarpRow row;
    row.load(rows, r0, s, q, k);
    for (int n = 0; n < np; n++) {
        WarpRow next;
        if (n + 1 < np) next.load(rows, r0 + n + 1, s, q, k);
        const double w1 = shfl_d(w, at + k1), w2 = shfl_d(w, at + k2);
        const double turn = w1 * row.r2 - w2 * row.r1;
        const double vr = ((shfl_d(v, k) + shfl_d(turn, k)) - shfl_d(v, 3 + k)) - shfl_d(turn, 3 + k);
        const double part = row.d * vr;
        const double dotq = (shfl_d(part, 3 * q) + shfl_d(part, 3 * q + 1)) + shfl_d(part, 3 * q + 2);
        double val = row.base - dotq * row.jmj;
        double ni = shfl_d(val, 0);
        ni = ni > -row.nacc ? ni : -row.nacc;
        const double nacc = row.nacc + ni;
        const double sq = val * val;
        const double scale = friction_scale(row.mu * nacc, shfl_d(sq, 3) + shfl_d(sq, 6));
        if (scale < 1) val = val * scale;
        const double push = (q == 0 ? ni : val - row.base) * row.d;
        double imp = (shfl_d(push, k) + shfl_d(push, 3 + k)) + shfl_d(push, 6 + k);
        if (s == 1) imp = -imp;
        const double p1 = shfl_d(imp, at + k1), p2 = shfl_d(imp, at + k2);
        const double x = row.r1 * p2 - row.r2 * p1;
        const double m0 = i0 * shfl_d(x, at), m1 = i1 * shfl_d(x, at + 1), m2 = i2 * shfl_d(x, at + 2);
        const double turned = ((k < 2 ? m0 : m1) + (k < 2 ? m1 : m2)) + (k < 2 ? m2 : m0);   // mv: the last row right to left
        if (!kin) { v = v + imp * im; w = w + turned; }
        double* p = rows.f + (size_t)(r0 + n) * NRF;
        if (lane == 0) p[21] = nacc;
        else if (lane == 3 || lane == 6) p[21 + q] = val;
        row = next;
    }
    __syncwarp();
    if (lane < 6) { item[6 * s + k] = v; item[6 * s + 3 + k] = w; }
    __syncwarp();
}

// ---------------------------------------------------------------- islands inside a warp
// Islands of up to kWarpIsland items, listed by size class: 1, 2, 3-4, 5-8, 9-16 and 17-32 items, so
// that a warp works on islands of about one length (32, 16, 8, 4, 2 or 1 of them), one lane per item.
constexpr int kWarpIsland = 32, kWarpClasses = 6, kWarpBlock = 128;
__host__ __device__ inline int warp_class(int m) { return m <= 1 ? 0 : m <= 2 ? 1 : m <= 4 ? 2 : m <= 8 ? 3 : m <= 16 ? 4 : 5; }
// first slot of class c in the island list: a class holds at most bound / (its smallest size) islands
__host__ __device__ inline long long class_base(int c, long long bound) {
    const int least[kWarpClasses] = {1, 2, 3, 5, 9, 17};
    long long at = 0;
    for (int k = 0; k < c; k++) at += bound / least[k] + 1;
    return at;
}
// An island that a warp does not take (more than kWarpIsland items, or above big_items, which
// k_isl_flow may have to colour) gets a range of flow items at base[island]; those above big_items
// are also listed in big (k_isl_classes).

// One lane per item, tokens in shared memory.  A round runs every item whose tokens are there; what
// bounds it is the chain of dependent rows of the longest island of the warp, which the rounds follow
// item by item.  The lanes find their bodies' next items by comparing bodies across their island.
// (One thread per island of up to 16 items, the larger ones a block each with a barrier per level:
// 266 + 150 us of the 501-body pile's step, 1,448 + 718 us of the 4,096 piles'; together with the
// item-sized islands in one kernel here the steps are 309 us and 1.24 ms shorter.)
template <class R, bool JOINTS, bool SELF>
__global__ void __launch_bounds__(kWarpBlock, sizeof(R) == 4 ? 4 : 2)
k_isl_warp(const int* list, const int* n_list, int bound, const int* isl_off, const uint32_t* order, Results<R> res, Joints<R> J, Bodies<R> B,
           Rows<R> rows, int iterations, int color_min, int* n_colors, int* status) {
    constexpr int W = kWarpBlock / 32;
    __shared__ R tok_v[W][2][6][32];     // per side and lane: the token's linear and angular velocity
    __shared__ int tok_it[W][2][32];     // the iteration the token is for
    __shared__ int tok_lev[W][2][32];    // its level (the first iteration's)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    // Islands per warp: as many as its lanes hold, and fewer while there are warps to spare.  A warp takes
    // as long as its slowest lanes in every round, and its lanes' joints and rows of different length run
    // one after the other (200 FP64 chains, four islands a warp before and one now, in turn on one GPU:
    // 921 / 857 us; 835 to 1,050 us from one GPU to another).
    int units[kWarpClasses], total = 0, spread = 0;
    for (int sp = 0; sp <= 5; sp++) {
        int sum = 0;
#pragma unroll
        for (int c = 0; c < kWarpClasses; c++) {
            const int per = max(1, 32 >> (c + sp));
            sum += (n_list[c] + per - 1) / per;
        }
        if (sp > 0 && sum > (int)gridDim.x) break;   // the grid is up to four times the resident blocks, four warps each
        spread = sp;
    }
#pragma unroll
    for (int c = kWarpClasses - 1; c >= 0; c--) {   // the longest islands first
        const int per = max(1, 32 >> (c + spread));
        units[c] = (n_list[c] + per - 1) / per;
        total += units[c];
    }
    const int its = iterations > 0 ? iterations : 1;   // without iterations the levels are still counted
    int deepest = 0;
    // neighbours in a block, or over the SMs first while there are warps to spare
    for (int u = spread ? warp * gridDim.x + blockIdx.x : blockIdx.x * W + warp; u < total; u += gridDim.x * W) {
        int c = kWarpClasses - 1, k = u;
        while (k >= units[c]) { k -= units[c]; c--; }
        const int s = 1 << c, per = max(1, 32 >> (c + spread));
        const int li = k * per + (lane >> c), idx = lane & (s - 1), g0 = lane - idx;
        int lo = 0, m = 0;
        if ((lane >> c) < per && li < n_list[c]) {
            const int isl = list[class_base(c, bound) + li];
            lo = isl_off[isl];
            m = isl_off[isl + 1] - lo;
        }
        const bool active = idx < m;
        Item<R, JOINTS> t;
        t.ia = -1; t.ib = -1;
        if (active) t.load(order[lo + idx], res, J, B, rows);
        // the island's items on this item's bodies (bit per item), and on which side they hold them
        const bool own_a = active && !t.a.kin && !(SELF && t.ia == t.ib);   // side a has a token of its own
        const int da = own_a ? t.ia : -2, db = active && !t.b.kin ? t.ib : -2;
        unsigned ma = 0, mab = 0, mb = 0, mbb = 0;
        for (int j = 0; j < s; j++) {
            const int oa = __shfl_sync(full, t.ia, g0 + j), ob = __shfl_sync(full, t.ib, g0 + j);
            const unsigned bit = 1u << j;
            if (oa == da) ma |= bit;
            if (ob == da) { ma |= bit; mab |= bit; }
            if (oa == db) mb |= bit;
            if (ob == db) { mb |= bit; mbb |= bit; }
        }
        const unsigned before = (1u << idx) - 1u, after = ~(before | (1u << idx));
        const bool wrap_a = (ma & after) == 0, wrap_b = (mb & after) == 0;
        const int na = own_a ? __ffs(wrap_a ? ma : ma & after) - 1 : 0, nb = active && !t.b.kin ? __ffs(wrap_b ? mb : mb & after) - 1 : 0;
        const int sa = (mab >> na) & 1, sb = (mbb >> nb) & 1;
        const bool keep_a = na == idx, keep_b = nb == idx;   // the body's only item: its token stays in registers
        tok_it[warp][0][lane] = tok_it[warp][1][lane] = -1;
        int lev_a = 0, lev_b = 0;
        bool have_a = !own_a, have_b = !active || t.b.kin;
        if (own_a && (ma & before) == 0) { t.a.v = B.vec(VX, t.ia); t.a.w = B.vec(WX, t.ia); have_a = true; }
        if (active && !t.b.kin && (mb & before) == 0) { t.b.v = B.vec(VX, t.ib); t.b.w = B.vec(WX, t.ib); have_b = true; }
        int it = active ? 0 : its;
        __syncwarp();
        while (__any_sync(full, it < its)) {
            if (it < its) {
                auto take = [&](int side, Side<R>& x, int& lev) {
                    if (tok_it[warp][side][lane] != it) return false;
                    const R* v = &tok_v[warp][side][0][lane];
                    x.v = V3<R>(v[0], v[32], v[64]);
                    x.w = V3<R>(v[96], v[128], v[160]);
                    lev = tok_lev[warp][side][lane];
                    return true;
                };
                if (!have_a) have_a = take(0, t.a, lev_a);
                if (!have_b) have_b = take(1, t.b, lev_b);
            }
            const bool run = it < its && have_a && have_b;
            if (!__any_sync(full, run)) {   // some item always holds its tokens
                if (lane == 0) atomicOr(status, ST_FLOW_STALL);
                break;
            }
            // (the vote also puts every read of this round's tokens before its writes)
            if (run) {
                if (SELF && t.ia == t.ib) { t.a.v = t.b.v; t.a.w = t.b.w; }
                if (iterations > 0) t.iterate(J, rows);
                const int lev = (lev_a > lev_b ? lev_a : lev_b) + 1;
                if (it == 0 && m > color_min) deepest = deepest > lev ? deepest : lev;
                auto give = [&](Side<R>& x, int i, bool wrap, int nl, int side, bool keep, bool& have) {
                    if (x.kin) return;
                    if (wrap && it == its - 1) {
                        B.set_vec(VX, i, x.v);
                        B.set_vec(WX, i, x.w);
                        return;
                    }
                    if (keep) return;
                    R* v = &tok_v[warp][side][0][g0 + nl];
                    v[0] = x.v.x; v[32] = x.v.y; v[64] = x.v.z;
                    v[96] = x.w.x; v[128] = x.w.y; v[160] = x.w.z;
                    tok_lev[warp][side][g0 + nl] = lev;
                    tok_it[warp][side][g0 + nl] = it + (wrap ? 1 : 0);
                    have = false;
                };
                if (!SELF || own_a) give(t.a, t.ia, wrap_a, na, sa, keep_a, have_a);
                give(t.b, t.ib, wrap_b, nb, sb, keep_b, have_b);
                it++;
            }
            __syncwarp();
        }
    }
    if (n_colors) {
        deepest = __reduce_max_sync(full, deepest < kMaxColors ? deepest : kMaxColors);
        if (lane == 0 && deepest > 0) atomicMax(n_colors, deepest);
    }
}

// ---------------------------------------------------------------- islands over the grid
// A token in global memory: 16-byte words of three payload words and a tag, each word stored and
// loaded whole (128-bit accesses), so that a reader that finds the tag it waits for in every word
// has the token, without a fence between payload and flag.  The tag is the iteration + 1; during the
// first iteration the last word's tag carries the level instead, with the top bit set.
template <class R> constexpr int token_words() { return 6 * (int)sizeof(R) / 12; }
__device__ __forceinline__ void st_word(uint4* p, uint4 w) {
    const unsigned long long lo = (unsigned long long)w.x | (unsigned long long)w.y << 32, hi = (unsigned long long)w.z | (unsigned long long)w.w << 32;
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ uint4 ld_word(const uint4* p) {
    unsigned long long lo, hi;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}
constexpr unsigned kLevelTag = 0x80000000u;
template <class R> __device__ __forceinline__ void token_put(uint4* box, const Side<R>& x, int it, int lev) {
    constexpr int NW = token_words<R>();
    union { R r[6]; unsigned u[3 * NW]; } q;
    q.r[0] = x.v.x; q.r[1] = x.v.y; q.r[2] = x.v.z; q.r[3] = x.w.x; q.r[4] = x.w.y; q.r[5] = x.w.z;
    const unsigned tag = (unsigned)it + 1u;
#pragma unroll
    for (int k = 0; k < NW; k++)
        st_word(box + k, make_uint4(q.u[3 * k], q.u[3 * k + 1], q.u[3 * k + 2], k == NW - 1 && it == 0 ? kLevelTag | (unsigned)lev : tag));
}
template <class R> __device__ __forceinline__ bool token_get(const uint4* box, Side<R>& x, int it, int& lev) {
    constexpr int NW = token_words<R>();
    union { R r[6]; unsigned u[3 * NW]; } q;
    const unsigned tag = (unsigned)it + 1u;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NW; k++) {
        const uint4 w = ld_word(box + k);
        q.u[3 * k] = w.x; q.u[3 * k + 1] = w.y; q.u[3 * k + 2] = w.z;
        if (k == NW - 1 && it == 0) {
            ok = ok && (w.w & kLevelTag);
            lev = (int)(w.w & ~kLevelTag);
        } else {
            ok = ok && w.w == tag;
        }
    }
    if (!ok) return false;
    x.v = V3<R>(q.r[0], q.r[1], q.r[2]);
    x.w = V3<R>(q.r[3], q.r[4], q.r[5]);
    return true;
}

template <class R> struct FlowArgs {
    const int* n_items;        // island items (contacts and joints) in the sorted order
    const int* isl_scan;       // island starts before each sorted item
    const int* isl_off;
    const uint32_t* order;
    const int* base;           // first flow item of each island that a warp does not take
    const int* n_flow;         // flow items
    const int* big;            // islands above big_items
    const int* n_big;
    int big_items, color_min, exact_levels, mode, iterations;
    uint32_t* item;            // per flow item: the item,
    int* isl;                  // its island,
    int* color;                // and its first-fit colour, where its island runs in colour order
    int* head;                 // per body: its entries (2 x flow item + side) as a list
    int* next;                 // per entry: the list's next entry
    int* succ;                 // per entry: 2 x (the entry its token goes to) + 1 when that is the next iteration's
    uint4* box;                // per entry: its token
    int* isl_levels;           // per island: levels,
    int* isl_colors;           // first-fit colours in use,
    int* isl_state;            // kFlowFirstFit, kFlowLeft
    int* any_first_fit;
    int* n_colors;
    int* status;
};
constexpr int kFlowBlock = 128, kFlowFirstFit = 1, kFlowLeft = 2;
constexpr int kByWarpMost = 4;   // ready results of a warp up to which each takes the whole warp: 4 x 40 instructions against 170 for all at once, so that
                               // five would take longer
// Polls in a row without progress after which a warp gives up (some ten seconds).  A warp holds an item of
// every stride (38,912 in FP64, 77,824 in FP32), so it waits for a chain of about that many others at most,
// however long the island: 0.4 s at the 10 us an item that 1,000,000 hinges in a row take in FP64 and, at
// eight points an item beside a busy FP64 pipe, a second, where 1 << 21 polls would end.
constexpr int kFlowStall = 1 << 24;

// Islands that one warp does not take, all of them in one cooperative launch (a waiting item needs
// the items it waits for to be resident).  Flow item j belongs to lane j mod `per` of warp j / per, with
// as few lanes per warp as the item count allows: lanes of a warp run one after the other, and the
// time is the latency of the longest chain, a hand-over through L2 plus one item's rows.  (A block
// per island with a barrier per level, and one barrier over the whole grid per level for large
// islands, took 3.4 and 11 us per level and iteration.)
template <class R, bool JOINTS, bool SELF>
__global__ void __launch_bounds__(kFlowBlock, sizeof(R) == 4 ? 4 : 2)
k_isl_flow(FlowArgs<R> f, Results<R> res, Joints<R> J, Bodies<R> B, Rows<R> rows) {
    constexpr int NW = token_words<R>();
    const int M = *f.n_flow;
    if (M == 0) return;   // the same for every thread
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31, gw = t >> 5, GW = T >> 5;
    const unsigned full = 0xffffffffu;
    const int its = f.iterations > 0 ? f.iterations : 1;
    const bool coloring = f.mode != 0 && *f.n_big > 0;
    auto dynamic = [&](int i) { return (B.flags[i] & BF_KINEMATIC) == 0; };
    auto own_a = [&](int2 q) { return !(SELF && q.x == q.y) && dynamic(q.x); };   // side a has a token of its own
    auto island_size = [&](int s) { return f.isl_off[s + 1] - f.isl_off[s]; };

    // the flow items, in island order
    for (int k = t, n = *f.n_items; k < n; k += T) {
        const int s = f.isl_scan[k + 1] - 1, lo = f.isl_off[s], b = f.base[s];
        if (b < 0) continue;
        const int j = b + k - lo;
        const uint32_t id = f.order[k];
        const int2 q = item_bodies(id, res, J);
        f.item[j] = id;
        f.isl[j] = s;
        f.color[j] = 0;
        f.head[q.x] = -1;
        f.head[q.y] = -1;
        if (k == lo) { f.isl_levels[s] = 0; f.isl_colors[s] = 0; f.isl_state[s] = 0; }
    }
    if (t == 0) *f.any_first_fit = 0;
    grid.sync();
    // every body's entries
    for (int j = t; j < M; j += T) {
        const int2 q = item_bodies(f.item[j], res, J);
        if (own_a(q)) f.next[2 * j] = atomicExch(&f.head[q.x], 2 * j);
        if (dynamic(q.y)) f.next[2 * j + 1] = atomicExch(&f.head[q.y], 2 * j + 1);
    }
    grid.sync();
    // Where each entry's token goes: the body's next entry by (colour, position), the first one after
    // the last.  A body's first entry starts with its token: the velocity, or, where the island is to be
    // coloured first, an empty colour mask.
    auto link = [&](int e, int body, bool colors) {
        auto key = [&](int en) { return (unsigned long long)(unsigned)f.color[en >> 1] << 32 | (unsigned)(en >> 1); };
        const unsigned long long mine = key(e);
        unsigned long long up = ~0ull, least = mine;
        int eu = -1, el = e;
        for (int en = f.head[body]; en >= 0; en = f.next[en]) {
            const unsigned long long q = key(en);
            if (q > mine && q < up) { up = q; eu = en; }
            if (q < least) { least = q; el = en; }
        }
        f.succ[e] = eu >= 0 ? 2 * eu : 2 * el + 1;
        uint4* box = f.box + (size_t)e * NW;
        if (least != mine || colors)
            for (int k = 0; k < NW; k++) box[k] = make_uint4(0, 0, 0, least == mine && k == 0 ? 1u : 0u);
        else {
            Side<R> x;
            x.v = B.vec(VX, body);
            x.w = B.vec(WX, body);
            token_put(box, x, 0, 0);
        }
    };
    for (int j = t; j < M; j += T) {
        const int2 q = item_bodies(f.item[j], res, J);
        const bool colors = coloring && island_size(f.isl[j]) > f.big_items;
        if (own_a(q)) link(2 * j, q.x, colors);
        if (dynamic(q.y)) link(2 * j + 1, q.y, colors);
    }
    grid.sync();

    const int per = min(32, max(1, (M + GW - 1) / GW)), stride = GW * per;
    const int j0 = lane < per && gw * per + lane < M ? gw * per + lane : M;   // this lane's items: j0, j0 + stride, ..
    int stall = 0;
    // no progress in this round: give up after kFlowStall rounds (a lost token), else wait a little
    // where many lanes poll
    auto stalled = [&]() {
        if (++stall > kFlowStall) {
            if (lane == 0) atomicOr(f.status, ST_FLOW_STALL);
            return true;
        }
        if (per > 4) __nanosleep(40);
        return false;
    };

    if (coloring) {
        // Levels and first-fit colours of the islands above big_items, passed on like velocities: an
        // item's level is one above its bodies' (the round in which a colouring by rounds takes it), its
        // colour the smallest that no earlier item of its bodies holds.  Islands within exact_levels
        // levels keep the order of their items, the others run by colour.
        int j = j0;
        while (j < M && island_size(f.isl[j]) <= f.big_items) j += stride;
        while (__any_sync(full, j < M)) {
            bool moved = false;
            if (j < M) {
                const int2 q = item_bodies(f.item[j], res, J);
                const bool da = own_a(q), db = dynamic(q.y);
                uint4 wa = make_uint4(0, 0, 0, 1), wb = wa;
                if (da) wa = ld_word(f.box + (size_t)(2 * j) * NW);
                if (db) wb = ld_word(f.box + (size_t)(2 * j + 1) * NW);
                if (wa.w == 1u && wb.w == 1u) {
                    const int s = f.isl[j], lev = (int)max(wa.x, wb.x);
                    unsigned long long ka = (unsigned long long)wa.y | (unsigned long long)wa.z << 32;
                    unsigned long long kb = (unsigned long long)wb.y | (unsigned long long)wb.z << 32;
                    int c = kMaxColorsBig - 1;
                    if (lev < kMaxColorsBig - 1) {
                        const unsigned long long used = ka | kb;
                        if (used != ~0ull) {
                            c = __ffsll((long long)~used) - 1;
                            ka |= 1ull << c;
                            kb |= 1ull << c;
                        }
                        atomicMax(&f.isl_levels[s], lev + 1);
                    } else {
                        atomicOr(&f.isl_state[s], kFlowFirstFit);
                    }
                    if (c == kMaxColorsBig - 1) atomicOr(&f.isl_state[s], kFlowLeft);
                    else atomicMax(&f.isl_colors[s], c + 1);
                    f.color[j] = c;
                    auto pass = [&](int e, unsigned long long k) {
                        const int to = f.succ[e];
                        if (!(to & 1)) st_word(f.box + (size_t)(to >> 1) * NW, make_uint4((unsigned)lev + 1u, (unsigned)k, (unsigned)(k >> 32), 1u));
                    };
                    if (da) pass(2 * j, ka);
                    if (db) pass(2 * j + 1, kb);
                    do j += stride; while (j < M && island_size(f.isl[j]) <= f.big_items);
                    moved = true;
                }
            }
            if (__any_sync(full, moved)) stall = 0;
            else if (stalled()) break;
        }
        grid.sync();
        for (int k = t; k < *f.n_big; k += T) {
            const int s = f.big[k], lev = f.isl_levels[s];
            const bool left = (f.isl_state[s] & kFlowLeft) != 0;
            int used = lev;
            if (lev > f.exact_levels || (f.isl_state[s] & kFlowFirstFit)) {
                f.isl_state[s] |= kFlowFirstFit;
                atomicOr(f.any_first_fit, 1);
                used = (left ? lev : min(f.isl_colors[s], lev)) + (left ? 1 : 0);
            }
            atomicMax(f.n_colors, used);
        }
        grid.sync();
        for (int j = t; j < M; j += T)
            if (!(f.isl_state[f.isl[j]] & kFlowFirstFit)) f.color[j] = 0;   // item order
        grid.sync();
        for (int j = t; j < M; j += T) {
            if (island_size(f.isl[j]) <= f.big_items) continue;
            const int2 q = item_bodies(f.item[j], res, J);
            if (own_a(q)) link(2 * j, q.x, false);
            if (dynamic(q.y)) link(2 * j + 1, q.y, false);
        }
        grid.sync();
    }

    // FP64: a warp with few ready results runs them one by one, all lanes on each (si_rows_warp)
    constexpr bool kByWarp = sizeof(R) == 8;
    __shared__ R shared_item[kByWarp ? kFlowBlock : 1][kByWarp ? kWarpItem : 1];
    const bool reorder = coloring && *(volatile int*)f.any_first_fit != 0;
    const bool single = M <= stride;   // one item per lane: its constants stay in registers
    Item<R, JOINTS> x;
    int succ_a = 0, succ_b = 0, lev_a = 0, lev_b = 0, m = 0, deepest = 0;
    bool have_a = false, have_b = false;
    auto take_item = [&](int j) {
        x.load(f.item[j], res, J, B, rows);
        have_a = x.a.kin || (SELF && x.ia == x.ib);
        have_b = x.b.kin;
        if (!have_a) succ_a = f.succ[2 * j];
        if (!x.b.kin) succ_b = f.succ[2 * j + 1];
        lev_a = 0;
        lev_b = 0;
        m = island_size(f.isl[j]);
        if constexpr (kByWarp) {
            R* it = shared_item[threadIdx.x];
            for (int a = 0; a < 3; a++)
                for (int b = 0; b < 3; b++) { it[12 + 3 * a + b] = x.a.I.m[a][b]; it[21 + 3 * a + b] = x.b.I.m[a][b]; }
            it[30] = x.a.im; it[31] = x.b.im;
        }
    };
    // the lane's next item of the iteration, by position or by (colour, position); M after the last
    auto next_item = [&](int j) {
        if (!reorder) return j + stride < M ? j + stride : M;
        auto key = [&](int i) { return (unsigned long long)(unsigned)f.color[i] << 32 | (unsigned)i; };
        unsigned long long mine = j < M ? key(j) + 1 : 0ull, best = ~0ull;
        int at = M;
        for (int i = j0; i < M; i += stride) {
            const unsigned long long k = key(i);
            if (k >= mine && k < best) { best = k; at = i; }
        }
        return at;
    };
    int it = 0, j = single || !reorder ? j0 : next_item(M);
    stall = 0;
    if (j < M) take_item(j);
    while (__any_sync(full, j < M)) {
        bool moved = false, done = false;
        if (j < M) {
            if (!have_a) have_a = token_get(f.box + (size_t)(2 * j) * NW, x.a, it, lev_a);
            if (!have_b) have_b = token_get(f.box + (size_t)(2 * j + 1) * NW, x.b, it, lev_b);
            if (SELF && have_b && x.ia == x.ib) { x.a.v = x.b.v; x.a.w = x.b.w; }
        }
        if constexpr (kByWarp) {
            const bool ready = j < M && have_a && have_b && f.iterations > 0 && !(JOINTS && (x.id & kJointItem));
            unsigned todo = __ballot_sync(full, ready);
            if (__popc(todo) <= kByWarpMost) {
                done = ready;
                if (ready) {
                    R* p = shared_item[threadIdx.x];
                    p[0] = x.a.v.x; p[1] = x.a.v.y; p[2] = x.a.v.z; p[3] = x.a.w.x; p[4] = x.a.w.y; p[5] = x.a.w.z;
                    p[6] = x.b.v.x; p[7] = x.b.v.y; p[8] = x.b.v.z; p[9] = x.b.w.x; p[10] = x.b.w.y; p[11] = x.b.w.z;
                }
                __syncwarp();
                for (; todo; todo &= todo - 1) {
                    const int o = __ffs(todo) - 1;
                    const int r0 = __shfl_sync(full, x.r0, o), np = __shfl_sync(full, x.np, o);
                    const int kins = __shfl_sync(full, (x.a.kin ? 1 : 0) | (x.b.kin ? 2 : 0), o);
                    si_rows_warp(rows, r0, np, kins & 1, kins & 2, shared_item[(threadIdx.x & ~31) + o], lane);
                }
                if (ready) {
                    const R* p = shared_item[threadIdx.x];
                    x.a.v = V3<R>(p[0], p[1], p[2]); x.a.w = V3<R>(p[3], p[4], p[5]);
                    x.b.v = V3<R>(p[6], p[7], p[8]); x.b.w = V3<R>(p[9], p[10], p[11]);
                }
            }
        }
        if (j < M) {
            if (have_a && have_b) {
                moved = true;
                if (f.iterations > 0 && !done) {
                    if (kByWarp && !(JOINTS && (x.id & kJointItem))) row_load(rows, x.r0, x.q);   // the warp keeps no row in registers
                    x.iterate(J, rows);
                }
                const int lev = max(lev_a, lev_b) + 1;
                auto give = [&](Side<R>& s, int i, int entry, int to, bool& have) {
                    if (s.kin) return;
                    if ((to & 1) && it == its - 1) {
                        B.set_vec(VX, i, s.v);
                        B.set_vec(WX, i, s.w);
                    } else if (single && (to >> 1) == entry) {
                        return;   // the body's only item: its token stays
                    } else {
                        token_put(f.box + (size_t)(to >> 1) * NW, s, it + (to & 1), lev);
                    }
                    have = false;
                };
                if (!SELF || x.ia != x.ib) give(x.a, x.ia, 2 * j, succ_a, have_a);
                give(x.b, x.ib, 2 * j + 1, succ_b, have_b);
                if (it == 0) {
                    if (m > f.big_items) { if (f.mode == 0) atomicMax(&f.isl_levels[f.isl[j]], lev); }
                    else if (m > f.color_min) deepest = max(deepest, lev);
                }
                if (single) {
                    if (++it == its) j = M;
                } else {
                    j = next_item(j);
                    if (j >= M && ++it < its) j = reorder ? next_item(M) : j0;
                    if (j < M) take_item(j);
                }
            }
        }
        if (__any_sync(full, moved)) stall = 0;
        else if (stalled()) break;
    }
    if (f.mode != 0) {
        deepest = __reduce_max_sync(full, deepest < kMaxColors ? deepest : kMaxColors);
        if (lane == 0 && deepest > 0) atomicMax(f.n_colors, deepest);
    }
}

} // namespace pe
