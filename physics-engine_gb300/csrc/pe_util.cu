// Precision-independent device utilities: exclusive scan, stable LSD radix sort passes, pair bucketing,
// and contact islands.
#include "pe_kernels.cuh"

namespace pe {

// ---------------------------------------------------------------- scan
__global__ void __launch_bounds__(kScanOneBlock) k_scan_one(int* data, int n, int* total, int* host_total) {
    int carry = 0;
    for (int r = 0; r < n; r += kScanOneBlock * kScanOneItems) {
        const int base = r + threadIdx.x * kScanOneItems;
        int v[kScanOneItems], s = 0, t;
#pragma unroll
        for (int k = 0; k < kScanOneItems; k++) { v[k] = base + k < n ? data[base + k] : 0; s += v[k]; }
        int run = carry + block_excl_scan<kScanOneBlock>(s, &t);
#pragma unroll
        for (int k = 0; k < kScanOneItems; k++) { if (base + k < n) data[base + k] = run; run += v[k]; }
        carry += t;
    }
    if (threadIdx.x == 0) { *total = carry; if (host_total) *host_total = carry; }
}

__global__ void k_scan_sums(const int* data, int n, int* aux) {
    int s = 0, t;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const int i = blockIdx.x * kScanTile + k * kBlock + threadIdx.x;
        s += i < n ? data[i] : 0;
    }
    block_excl_scan<kBlock>(s, &t);
    if (threadIdx.x == 0) aux[blockIdx.x] = t;
}

__global__ void k_scan_apply(int* data, int n, const int* aux, int* total, int* host_total) {
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems], s = 0, t;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) { v[k] = base + k < n ? data[base + k] : 0; s += v[k]; }
    const int before = tiles_before<kBlock>(aux, blockIdx.x);
    int run = before + block_excl_scan<kBlock>(s, &t);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) { if (base + k < n) data[base + k] = run; run += v[k]; }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) { *total = before + t; if (host_total) *host_total = before + t; }
}

// ---------------------------------------------------------------- radix sort
// one block per digit: its counts in the tiles become the counts of the tiles before, its total goes to the last row
__global__ void __launch_bounds__(kBlock) k_radix_offsets(int* hist, int tiles, int tile_items, int n0, const int* nd) {
    const int n = nd ? *nd : n0, d = blockIdx.x;
    const int live = (n + tile_items - 1) / tile_items;
    int carry = 0;
    for (int t0 = 0; t0 < live; t0 += kBlock) {
        const int t = t0 + threadIdx.x, v = t < live ? hist[t * 256 + d] : 0;
        int all;
        const int ex = block_excl_scan<kBlock>(v, &all);
        if (t < live) hist[t * 256 + d] = carry + ex;
        carry += all;
    }
    if (threadIdx.x == 0) hist[tiles * 256 + d] = carry;
}

// ---------------------------------------------------------------- narrowphase bucketing
// pairs grouped by class (order inside a class is free: every pair's result has its own slot);
// one atomic per class present in a warp.  The pair count is on the device; whole warps stride
// over it (the loop bound is block-uniform, so every lane takes part in the warp votes).
__global__ void k_np_bucket(NpPlan a, const int* cls) {
    const int P = *a.P;
    int *cursor = a.cursor, *order = a.order;
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x; base < P; base += gridDim.x * blockDim.x) {
        const int p = base + threadIdx.x;
        const int c = p < P ? cls[p] : -1 - lane;
        const unsigned peers = __match_any_sync(0xffffffffu, c);
        const int leader = __ffs(peers) - 1;
        int b = 0;
        if (c >= 0 && lane == leader) b = atomicAdd(&cursor[c], __popc(peers));
        b = __shfl_sync(0xffffffffu, b, leader);
        if (c >= 0) order[b + __popc(peers & ((1u << lane) - 1u))] = p;
    }
}

// class ranges from the class counts, by one warp: range[c] = [first, end) of class c in the bucketed
// order, the bucketing cursors at each class's first slot, and the work cursors of the kernels that
// hand pairs out one at a time (they start at the class's first slot).  The counts are kept for the
// step's counters and cleared for the next step.
__device__ void np_ranges(const NpPlan& a, int count) {   // lane c: class c's count
    const int c = threadIdx.x & 31, v = c < PC_COUNT ? count : 0, end = warp_incl_scan(v);
    if (c >= PC_COUNT) return;
    a.range[c] = make_int2(end - v, end);
    a.cursor[c] = end - v;
    a.work[c] = end - v;
    a.last[c] = v;
    a.count[c] = 0;
}
__global__ void k_np_ranges(NpPlan a) { np_ranges(a, threadIdx.x < PC_COUNT ? a.count[threadIdx.x] : 0); }

} // namespace pe

namespace pe {

// ---------------------------------------------------------------- islands
// a result's or joint's part in the union-find: its bodies are of one island when both are dynamic
__device__ __forceinline__ void isl_union(const IslandArgs& a, int* parent, int ia, int ib) {
    if ((a.flags[ia] & BF_KINEMATIC) || (a.flags[ib] & BF_KINEMATIC)) return;
    uf_union(parent, ia, ib);
}
// an item's island label: the smallest body of its island (N for a joint that moves nothing)
__device__ __forceinline__ uint32_t isl_label(const IslandArgs& a, const int* parent, uint32_t item) {
    if (item & kJointItem) {
        const int2 q = a.jbody[item & ~kJointItem];
        const bool ka = (a.flags[q.x] & BF_KINEMATIC) != 0, kb = (a.flags[q.y] & BF_KINEMATIC) != 0;
        return ka && kb ? (uint32_t)a.N : (uint32_t)uf_find(parent, ka ? q.y : q.x);
    }
    const int ia = a.res_a[item];
    return (uint32_t)uf_find(parent, (a.flags[ia] & BF_KINEMATIC) ? a.res_b[item] : ia);
}
// an active result counts one item (high half) and its points (low half)
__device__ __forceinline__ unsigned long long act_value(int np) { return np > 0 ? 1ull << 32 | (unsigned)np : 0ull; }

__global__ void __launch_bounds__(kIslandBlock) k_islands_one(IslandArgs a, int label_passes) {
    constexpr int W = kIslandBlock / 32;
    extern __shared__ int s_dyn[];
    uint32_t* key = (uint32_t*)s_dyn;                 // [kIslandOne]
    uint32_t* val = key + kIslandOne;                 // [kIslandOne]
    int* off = (int*)(val + kIslandOne);              // [kIslandOne + 1]
    unsigned short* cnt = (unsigned short*)(off + kIslandOne + 2);   // [W][256]
    int* parent = (int*)(cnt + W * 256);              // [N]
    __shared__ int digit_base[256], n_cls[kWarpClasses + 2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int P = *a.P;
    for (int k = tid; k < a.N; k += kIslandBlock) parent[k] = k;
    if (tid < kWarpClasses + 2) n_cls[tid] = 0;
    // active results in order, then the joints; their unions
    unsigned long long v[2], all;
#pragma unroll
    for (int k = 0; k < 2; k++) v[k] = 2 * tid + k < P ? act_value(a.npts[2 * tid + k]) : 0ull;
    unsigned long long run = block_excl_scan<kIslandBlock>(v[0] + v[1], &all);
    const int A = (int)(all >> 32), M = A + a.NJ;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        if (v[k]) {
            const int p = 2 * tid + k;
            val[run >> 32] = (uint32_t)p;
            isl_union(a, parent, a.res_a[p], a.res_b[p]);
        }
        run += v[k];
    }
    for (int j = tid; j < a.NJ; j += kIslandBlock) {
        val[A + j] = kJointItem | (uint32_t)j;
        const int2 q = a.jbody[j];
        isl_union(a, parent, q.x, q.y);
    }
    __syncthreads();
    // items warp * 64 + r * 32 + lane, sorted by label
    uint32_t kr[2], vr[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int i = warp * 64 + r * 32 + lane;
        vr[r] = i < M ? val[i] : 0u;
        kr[r] = i < M ? isl_label(a, parent, vr[r]) : 0u;
    }
    for (int pass = 0; pass < label_passes; pass++) {
        for (int k = tid; k < W * 128; k += kIslandBlock) ((unsigned*)cnt)[k] = 0u;
        __syncthreads();
        int digit[2], rank[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const bool live = warp * 64 + r * 32 + lane < M;
            digit[r] = live ? (int)(kr[r] >> (8 * pass)) & 0xff : 256 + lane;
            const unsigned peers = __match_any_sync(0xffffffffu, digit[r]);
            rank[r] = live ? cnt[warp * 256 + digit[r]] + __popc(peers & ((1u << lane) - 1u)) : 0;
            __syncwarp();
            if (live && lane == __ffs(peers) - 1) cnt[warp * 256 + digit[r]] += (unsigned short)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        int total = 0, sum;
        if (tid < 256)
            for (int w = 0; w < W; w++) { const int c = cnt[w * 256 + tid]; cnt[w * 256 + tid] = (unsigned short)total; total += c; }
        const int before = block_excl_scan<kIslandBlock>(total, &sum);
        if (tid < 256) digit_base[tid] = before;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (warp * 64 + r * 32 + lane < M) {
                const int pos = digit_base[digit[r]] + cnt[warp * 256 + digit[r]] + rank[r];
                key[pos] = kr[r];
                val[pos] = vr[r];
            }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int i = warp * 64 + r * 32 + lane;
            if (i < M) { kr[r] = key[i]; vr[r] = val[i]; }
        }
    }
    // islands of the sorted items
    int head[2], n_isl;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = 2 * tid + k;
        head[k] = i < M && (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
    }
    int at = block_excl_scan<kIslandBlock>(head[0] + head[1], &n_isl);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = 2 * tid + k;
        if (i < M) {
            a.val[0][i] = val[i];
            a.isl_scan[i] = at;
            if (head[k]) off[at] = a.isl_off[at] = i;
        }
        at += head[k];
    }
    if (tid == 0) {
        off[n_isl] = a.isl_off[n_isl] = M;
        a.isl_scan[M] = n_isl;
        *a.n_active = A;
        *a.n_items = M;
        *a.n_rows = (int)(all & 0xffffffffull);
        *a.n_isl = n_isl;
        if (a.n_colors) *a.n_colors = 0;
    }
    __syncthreads();
    for (int s = tid; s < n_isl; s += kIslandBlock) {
        const int m = off[s + 1] - off[s];
        if (m <= kWarpIsland && m <= a.big_items) {
            const int c = warp_class(m);
            a.list[class_base(c, a.bound) + atomicAdd(&n_cls[c], 1)] = s;
            a.base[s] = -1;
        } else {
            a.base[s] = atomicAdd(&n_cls[kWarpClasses], m);
            if (m > a.big_items) a.big[atomicAdd(&n_cls[kWarpClasses + 1], 1)] = s;
        }
    }
    __syncthreads();
    if (tid < kWarpClasses + 2) a.n_list[tid] = n_cls[tid];
}

__global__ void __launch_bounds__(kBlock) k_act_sums(IslandArgs a) {
    const int P = *a.P;
    const int t = blockIdx.x * kBlock + threadIdx.x;
    for (int k = t; k < a.N; k += gridDim.x * kBlock) a.parent[k] = k;
    if (t < kWarpClasses + 2) a.n_list[t] = 0;
    if (t == 0 && a.n_colors) *a.n_colors = 0;
    for (int tile = blockIdx.x; tile * kActTile < P; tile += gridDim.x) {   // a block's tiles one after the other
        unsigned long long s = 0, all;
#pragma unroll
        for (int k = 0; k < kActItems; k++) {
            const int p = tile * kActTile + k * kBlock + threadIdx.x;
            s += p < P ? act_value(a.npts[p]) : 0ull;
        }
        block_excl_scan<kBlock>(s, &all);
        if (threadIdx.x == 0) a.aux[tile] = all;
    }
}

__global__ void __launch_bounds__(kBlock) k_act_apply(IslandArgs a) {
    const int P = *a.P, tiles = max((P + kActTile - 1) / kActTile, 1), tile = blockIdx.x;
    for (int j = blockIdx.x * kBlock + threadIdx.x; j < a.NJ; j += gridDim.x * kBlock) {
        const int2 q = a.jbody[j];
        isl_union(a, a.parent, q.x, q.y);
    }
    if (tile >= tiles) return;
    const int base = tile * kActTile + threadIdx.x * kActItems;
    unsigned long long v[kActItems], s = 0, all;
#pragma unroll
    for (int k = 0; k < kActItems; k++) { v[k] = base + k < P ? act_value(a.npts[base + k]) : 0ull; s += v[k]; }
    const unsigned long long before = tiles_before<kBlock>(a.aux, tile);
    unsigned long long run = before + block_excl_scan<kBlock>(s, &all);
#pragma unroll
    for (int k = 0; k < kActItems; k++) {
        if (v[k]) {
            const int p = base + k;
            a.active[run >> 32] = p;
            isl_union(a, a.parent, a.res_a[p], a.res_b[p]);
        }
        run += v[k];
    }
    if (tile == tiles - 1 && threadIdx.x == 0) {
        const int A = (int)((before + all) >> 32);
        *a.n_active = A;
        *a.n_items = A + a.NJ;
        *a.n_rows = (int)((before + all) & 0xffffffffull);
    }
}

__global__ void k_isl_keys(IslandArgs a) {
    const int A = *a.n_active, M = A + a.NJ;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
        const uint32_t item = t < A ? (uint32_t)a.active[t] : kJointItem | (uint32_t)(t - A);
        a.key[0][t] = isl_label(a, a.parent, item);
        a.val[0][t] = item;
    }
}

__device__ __forceinline__ int isl_head(const uint32_t* key, int k, int M) { return k < M && (k == 0 || key[k] != key[k - 1]) ? 1 : 0; }
__global__ void __launch_bounds__(kBlock) k_head_sums(IslandArgs a, const uint32_t* key) {
    const int M = *a.n_items;
    if ((int)blockIdx.x * kScanTile >= M) return;
    unsigned long long s = 0, all;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) s += (unsigned)isl_head(key, blockIdx.x * kScanTile + k * kBlock + threadIdx.x, M);
    block_excl_scan<kBlock>(s, &all);
    if (threadIdx.x == 0) a.aux[blockIdx.x] = all;
}
__global__ void __launch_bounds__(kBlock) k_head_apply(IslandArgs a, const uint32_t* key) {
    const int M = *a.n_items, tiles = max((M + kScanTile - 1) / kScanTile, 1), tile = blockIdx.x;
    if (tile >= tiles) return;
    const int base = tile * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    unsigned long long s = 0, all;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) { v[k] = isl_head(key, base + k, M); s += (unsigned)v[k]; }
    const unsigned long long before = tiles_before<kBlock>(a.aux, tile);
    int run = (int)(before + block_excl_scan<kBlock>(s, &all));
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < M) a.isl_scan[base + k] = run;
        if (v[k]) a.isl_off[run] = base + k;
        run += v[k];
    }
    if (tile == tiles - 1 && threadIdx.x == 0) {
        const int n = (int)(before + all);
        a.isl_scan[M] = n;
        a.isl_off[n] = M;
        *a.n_isl = n;
    }
}

// size classes of the islands (see k_isl_warp and k_isl_flow), one atomic per class present in a warp
__global__ void k_isl_classes(IslandArgs a) {
    const int NI = *a.n_isl, lane = threadIdx.x & 31;
    int *n_flow = a.n_list + kWarpClasses, *n_big = n_flow + 1;
    for (int s0 = blockIdx.x * blockDim.x; s0 < NI; s0 += gridDim.x * blockDim.x) {
        const int s = s0 + threadIdx.x;
        int c = -1 - lane, m = 0;   // lanes without a warp-sized island match no other
        if (s < NI) {
            m = a.isl_off[s + 1] - a.isl_off[s];
            if (m <= kWarpIsland && m <= a.big_items) c = warp_class(m);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, c);
        const int leader = __ffs(peers) - 1;
        int at = 0;
        if (c >= 0 && lane == leader) at = atomicAdd(&a.n_list[c], __popc(peers));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (s >= NI) continue;
        if (c >= 0) {
            a.list[class_base(c, a.bound) + at + __popc(peers & ((1u << lane) - 1u))] = s;
            a.base[s] = -1;
        } else {
            a.base[s] = atomicAdd(n_flow, m);
            if (m > a.big_items) a.big[atomicAdd(n_big, 1)] = s;
        }
    }
}

// the step's counters, by one warp into page-locked host memory (World::HostStat order).  Colours: those the
// coloured mode counted; in serial order the levels of the islands above big_island_items, where they
// are within the first-fit colours' number.
__global__ void k_step_counters(const int* status, const int* rows, const int* active, const int* islands, const int* n_big, const int* big,
                                const int* isl_levels, const int* colors, const int* cls, int* out) {
    const int lane = threadIdx.x & 31;
    int used = 0;
    if (colors) used = *colors;
    else
        for (int k = lane; k < *n_big; k += 32)
            if (isl_levels[big[k]] < kMaxColorsBig) used = max(used, isl_levels[big[k]]);
    used = __reduce_max_sync(0xffffffffu, used);
    const int* head[5] = {status, rows, active, islands, n_big};
    if (lane < 5) out[lane] = *head[lane];
    if (lane == 5) out[5] = used;
    if (lane < PC_COUNT) out[7 + lane] = cls[lane];
}

// exclusive offsets of the crowded positions' chunks (one warp)
__global__ void k_bp_chunk_offsets(const int* n_big, const int* nchunk, int* choff, int* total) {
    const int lane = threadIdx.x & 31, nb = *n_big;
    int run = 0;
    for (int b0 = 0; b0 < nb; b0 += 32) {
        const int b = b0 + lane, v = b < nb ? nchunk[b] : 0, incl = warp_incl_scan(v);
        if (b < nb) choff[b] = run + incl - v;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) *total = run;
}
__global__ void k_bp_chunk_sums(const int* big, const int* n_big, const int* choff, const int* nchunk, const int* ccount, int* cpref,
                                int* count) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < *n_big; b += gridDim.x * blockDim.x) {
        int run = 0;
        for (int k = choff[b]; k < choff[b] + nchunk[b]; k++) { cpref[k] = run; run += ccount[k]; }
        count[big[b]] = run;
    }
}


} // namespace pe
