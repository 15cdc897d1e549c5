// Kernels of the rigid-body step, part 3: the sweep-and-prune broadphase.
#pragma once
#include "pe_k_sort.cuh"

namespace pe {

template <class R> struct KeyOf { using type = uint32_t; };
template <> struct KeyOf<double> { using type = uint64_t; };
__device__ inline uint32_t order_bits(float x) {
    if (x == 0.0f) x = 0.0f;   // -0 and +0 compare equal: give them one key
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ inline uint64_t order_bits(double x) {
    if (x == 0.0) x = 0.0;
    const uint64_t u = (uint64_t)__double_as_longlong(x);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}

// sort key of each body: its AABB minimum along its scene's sweep axis
template <class R>
__global__ void k_bp_keys(Bodies<R> B, const int* scene_axis, typename KeyOf<R>::type* key, uint32_t* val) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.n) return;
    const int ax = scene_axis[B.scene[i]];
    key[i] = order_bits(B.at(MNX + ax, i));
    val[i] = (uint32_t)i;
}

// sorted copy of the sweep inputs (coalesced reads in the sweep)
template <class R> struct SweepBoxes {
    R *mn, *mx;
    int *flag, *scene;
    int* lost;   // set where a box's minimum is not a number (cleared by k_bp_axis)
    __device__ __forceinline__ void copy(const Bodies<R>& B, int k, int i) const {
        for (int d = 0; d < 3; d++) {
            const R m = B.at(MNX + d, i);
            mn[(size_t)d * B.n + k] = m;
            mx[(size_t)d * B.n + k] = B.at(MXX + d, i);
            if (m != m) *lost = 1;
        }
        flag[k] = B.flags[i];
        scene[k] = B.scene[i];
    }
};

// Sort of every scene's bodies by the AABB minimum along the scene's axis, one block per scene of
// at most kSceneSortMax bodies: a bitonic sort in shared memory of (key, body index) pairs, whose
// order, ties by body index, is the stable LSD radix sort's.  Replaces the radix passes (four
// per key byte plus one per scene-id byte, five launches each) when every scene fits a block.
constexpr int kSceneSortMax = 2048;
constexpr int kSceneSortBlock = 512;
// The block then copies the sweep's inputs in that order (k_bp_gather's work).
template <class R>
__global__ void __launch_bounds__(kSceneSortBlock) k_bp_sort_scenes(Bodies<R> B, const int* scene_axis, const int* scene_off,
                                                                   uint32_t* order, SweepBoxes<R> out, int* n_big) {
    __shared__ uint64_t key[kSceneSortMax];
    __shared__ uint32_t idx[kSceneSortMax];
    const int s = blockIdx.x;
    if (s == 0 && threadIdx.x == 0) *n_big = 0;
    const int lo = scene_off[s], cnt = scene_off[s + 1] - lo;
    if (cnt <= 0) return;   // whole block
    int P = 1;
    while (P < cnt) P <<= 1;
    const int ax = scene_axis[s];
    for (int k = threadIdx.x; k < P; k += blockDim.x) {
        if (k < cnt) { key[k] = order_bits(B.at(MNX + ax, lo + k)); idx[k] = (uint32_t)k; }
        else { key[k] = ~0ull; idx[k] = 0xffffffffu; }   // padding sorts last
    }
    __syncthreads();
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < P / 2; t += blockDim.x) {
                const int i = 2 * t - (t & (stride - 1)), j = i + stride;   // the t-th pair of this stage
                const bool up = (i & size) == 0;
                const uint64_t ki = key[i], kj = key[j];
                const uint32_t ii = idx[i], ij = idx[j];
                const bool gt = ki > kj || (ki == kj && ii > ij);
                if (gt == up) { key[i] = kj; key[j] = ki; idx[i] = ij; idx[j] = ii; }
            }
            __syncthreads();
        }
    }
    for (int k = threadIdx.x; k < cnt; k += blockDim.x) {
        const int i = lo + (int)idx[k];
        order[lo + k] = (uint32_t)i;
        out.copy(B, lo + k, i);
    }
}
template <class R>
__global__ void k_bp_gather(Bodies<R> B, const uint32_t* order, SweepBoxes<R> out, int* n_big) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *n_big = 0;
    if (k < B.n) out.copy(B, k, (int)order[k]);
}

// BroadPhaseSweepAndPrune::calcCollisionPairs sweep (broad_phase_sweep_and_prune.cpp:24-35)
// with BroadPhaseBase::validateCollisionPair (broad_phase_base.cpp:5-19).
//
// One warp per sorted position i; the lanes test candidates j = i+1+lane, i+33+lane, ... with
// coalesced loads of the sorted AABBs.  The reference stops at the first j whose minimum along
// the axis exceeds i's maximum; minima are sorted, so the lanes still in range form a prefix and
// the warp stops after the first chunk that is not full.  Overlapping partners are compacted in
// ascending j with a ballot and a prefix popcount, which is the reference's pair order.
// Pass 0 counts the pairs of each position and keeps its first kStage partners; pass 1 writes the
// pairs at the scanned offsets, copying staged partners and re-sweeping only crowded positions.
constexpr int kStage = 8;   // a position with more pairs is swept again to write them
// U chunks of 32 candidates from j0 on, tested in order after all their loads are under way; false
// once a chunk is not full.  (c is the position's pairs so far.)
template <class R, bool WRITE, int U>
__device__ __forceinline__ bool sweep_chunks(int i, int j0, int n, int lane, int sc, const R* amin, R maxi_ax, const V3<R>& mn, const V3<R>& mx,
                                             int fi, const R* smn, const R* smx, const int* sflag, const int* sscene, int* stage, int2* out,
                                             int a, const uint32_t* order, const IgnoreLists& ign, int& c) {
    R am[U];
    V3<R> lo[U], hi[U];
    int fl[U], scn[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int j = min(j0 + 32 * u + lane, n - 1);   // past the end: the last one, not `in` below
        am[u] = amin[j];
        scn[u] = sscene[j];
        fl[u] = sflag[j];
        lo[u] = V3<R>(smn[j], smn[n + j], smn[2 * (size_t)n + j]);
        hi[u] = V3<R>(smx[j], smx[n + j], smx[2 * (size_t)n + j]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int j = j0 + 32 * u + lane;
        const bool in = j < n && !(am[u] > maxi_ax) && scn[u] == sc;
        const unsigned live = __ballot_sync(0xffffffffu, in);
        bool hit = in && !(fl[u] & BF_IGNORE) && !((fi & BF_KINEMATIC) && (fl[u] & BF_KINEMATIC)) &&
                   !(mn.x > hi[u].x || lo[u].x > mx.x) && !(mn.y > hi[u].y || lo[u].y > mx.y) && !(mn.z > hi[u].z || lo[u].z > mx.z);
        if (hit && ign.off && ((fi | fl[u]) & BF_IGN_LIST)) hit = !ign.ignored(i, j);
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int k = c + __popc(m & ((1u << lane) - 1u));
            if (WRITE) out[k] = make_int2(a, (int)order[j]);
            else if (k < kStage) stage[(size_t)i * kStage + k] = j;
        }
        c += __popc(m);
        if (live != 0xffffffffu) return false;
    }
    return true;
}
// The sweep of one position by a warp.  A window is a chain of chunks, each some 3 us of dependent
// loads and votes when taken alone: the floor of a 1,600-body scene, 50 chunks, held the count for
// 81 us and the write for 169 us (now 31 and 46).  Most windows end in the first two chunks; longer
// ones go four chunks at a time, loads first.
template <class R, bool WRITE>
__device__ __forceinline__ int sweep_warp(int i, int n, int lane, const int* scene_axis, const R* smn, const R* smx,
                                          const int* sflag, const int* sscene, int* stage, int2* out, const uint32_t* order,
                                          const IgnoreLists& ign) {
    const int sc = sscene[i];
    const int ax = scene_axis[sc];
    const R* amin = smn + (size_t)ax * n;
    const R maxi_ax = smx[(size_t)ax * n + i];
    const V3<R> mn(smn[i], smn[n + i], smn[2 * (size_t)n + i]), mx(smx[i], smx[n + i], smx[2 * (size_t)n + i]);
    const int fi = sflag[i];
    if (fi & BF_IGNORE) return 0;
    const int a = WRITE ? (int)order[i] : 0;
    int c = 0, j0 = i + 1;
    for (int k = 0; k < 2; k++, j0 += 32)
        if (j0 >= n || !sweep_chunks<R, WRITE, 1>(i, j0, n, lane, sc, amin, maxi_ax, mn, mx, fi, smn, smx, sflag, sscene, stage, out, a, order, ign, c))
            return c;
    for (; j0 < n; j0 += 128)
        if (!sweep_chunks<R, WRITE, 4>(i, j0, n, lane, sc, amin, maxi_ax, mn, mx, fi, smn, smx, sflag, sscene, stage, out, a, order, ign, c)) break;
    return c;
}

// A position whose window along the axis holds more than big_window_limit candidates (a floor or a wall
// spanning the scene) is swept by blocks instead of a warp, in chunks (below): 256 candidates at a
// time, warp ballots plus a block prefix of the warp counts keep the pairs in ascending j.
// The limit: what a warp sweeps in some 32 steps of four chunks, and at least an eighth of the largest
// scene, so that only bodies that span the scene exceed it.  Where bodies lie so close that ordinary
// windows hold thousands, nearly every position would go to the blocks, two searches and a chunk each
// (POUR_FIGURES).
constexpr int kBigWindow = 4096;
inline int big_window_limit(int largest_scene) { return kBigWindow > largest_scene / 8 ? kBigWindow : largest_scene / 8; }
constexpr int kNoBigWindow = 1 << 30;   // limit of a caller without the chunk kernels
// A box that is not a number compares as overlapping everything and lies anywhere in the order.  What a
// position meets of it past its window's end depends on where the window's chunks of 32 begin and on
// which kernel sweeps it; so in a world with one every window up to kLostWindow is swept by a warp of
// its own, in chunks from the position on, by the count and the write alike.
constexpr int kLostWindow = 32768;
__device__ __forceinline__ int window_limit(int limit, const int* lost) { return lost && *lost ? max(limit, kLostWindow) : limit; }
template <class R>
__device__ __forceinline__ bool big_window(int i, int n, int limit, const int* scene_axis, const R* smn, const R* smx, const int* sscene) {
    if (limit >= n - i) return false;
    const int j = i + limit;
    const int sc = sscene[i], ax = scene_axis[sc];
    return sscene[j] == sc && !(smn[(size_t)ax * n + j] > smx[(size_t)ax * n + i]);
}
// A crowded position's window (the candidates j > i of its scene whose minimum along the axis does
// not exceed i's maximum: a prefix of the scene's sorted positions, found by binary search) swept in
// up to kMaxChunks chunks of at least kChunk candidates, one block per chunk: chunk counts are summed
// per position, and each chunk writes its pairs after those of the chunks before it, so the pairs
// keep ascending j.
constexpr int kChunk = 1024;
constexpr int kMaxChunks = 32;
template <class R, bool WRITE>
__device__ int sweep_range_block(int i, int jb, int je, int n, const R* smn, const R* smx, const int* sflag, int2* out,
                                 const uint32_t* order, int* wcnt, const IgnoreLists& ign) {
    const R mnx = smn[i], mny = smn[n + i], mnz = smn[2 * (size_t)n + i];
    const R mxx = smx[i], mxy = smx[n + i], mxz = smx[2 * (size_t)n + i];
    const int fi = sflag[i];
    if (fi & BF_IGNORE) return 0;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const int a = WRITE ? (int)order[i] : 0;
    const unsigned lt = (1u << lane) - 1u;
    int c = 0;
    for (int j0 = jb; j0 < je; j0 += blockDim.x) {
        const int j = j0 + tid;
        bool hit = false;
        if (j < je) {
            const int fj = sflag[j];
            hit = !(fj & BF_IGNORE) && !((fi & BF_KINEMATIC) && (fj & BF_KINEMATIC)) &&
                  !(mnx > smx[j] || smn[j] > mxx) && !(mny > smx[n + j] || smn[n + j] > mxy) &&
                  !(mnz > smx[2 * (size_t)n + j] || smn[2 * (size_t)n + j] > mxz);
            if (hit && ign.off && ((fi | fj) & BF_IGN_LIST)) hit = !ign.ignored(i, j);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) wcnt[w] = __popc(m);
        __syncthreads();
        int before = 0, total = 0;
        for (int k = 0; k < nw; k++) { if (k < w) before += wcnt[k]; total += wcnt[k]; }
        if (WRITE && hit) out[c + before + __popc(m & lt)] = make_int2(a, (int)order[j]);
        c += total;
        __syncthreads();   // wcnt is rewritten next iteration
    }
    return c;
}
// per crowded position: window end, chunk size and chunk count
template <class R>
__global__ void k_bp_big_windows(int n, const int* scene_axis, const int* scene_off, const R* smn, const R* smx, const int* sscene,
                                 const int* big, const int* n_big, int* wend, int* csize, int* nchunk) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < *n_big; b += gridDim.x * blockDim.x) {
        const int i = big[b], sc = sscene[i];
        const R* amin = smn + (size_t)scene_axis[sc] * n;
        const R mx = smx[(size_t)scene_axis[sc] * n + i];
        int lo = i + 1, hi = scene_off[sc + 1];   // first j with amin[j] > mx, else the scene's end
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (amin[mid] > mx) hi = mid;
            else lo = mid + 1;
        }
        const int len = lo - (i + 1);
        int cs = (len + kMaxChunks - 1) / kMaxChunks;
        cs = cs < kChunk ? kChunk : cs;
        wend[b] = lo;
        csize[b] = cs;
        nchunk[b] = (len + cs - 1) / cs;
    }
}
__global__ void k_bp_chunk_offsets(const int* n_big, const int* nchunk, int* choff, int* total);
__device__ __forceinline__ int chunk_owner(int c, const int* choff, int nb) {   // last b with choff[b] <= c
    int lo = 0, hi = nb - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (choff[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
template <class R>
__global__ void k_bp_count_chunks(int n, const R* smn, const R* smx, const int* sflag, const int* big, const int* n_big, const int* wend,
                                  const int* csize, const int* choff, const int* total, int* ccount, IgnoreLists ign) {
    __shared__ int wcnt[32];
    for (int c = blockIdx.x; c < *total; c += gridDim.x) {
        const int b = chunk_owner(c, choff, *n_big), i = big[b];
        const int jb = i + 1 + (c - choff[b]) * csize[b], je = jb + csize[b] < wend[b] ? jb + csize[b] : wend[b];
        const int k = sweep_range_block<R, false>(i, jb, je, n, smn, smx, sflag, nullptr, nullptr, wcnt, ign);
        if (threadIdx.x == 0) ccount[c] = k;
    }
}
// per crowded position: its pair count and the offsets of its chunks' pairs
__global__ void k_bp_chunk_sums(const int* big, const int* n_big, const int* choff, const int* nchunk, const int* ccount, int* cpref,
                                int* count);
template <class R>
__global__ void k_bp_write_chunks(int n, const R* smn, const R* smx, const int* sflag, const uint32_t* order, const int* offset,
                                  const int* big, const int* n_big, const int* wend, const int* csize, const int* choff, const int* total,
                                  const int* cpref, int2* pairs, int pair_cap, int* status, IgnoreLists ign) {
    __shared__ int wcnt[32];
    for (int c = blockIdx.x; c < *total; c += gridDim.x) {
        const int b = chunk_owner(c, choff, *n_big), i = big[b];
        if (offset[i + 1] > pair_cap) {
            if (threadIdx.x == 0) atomicOr(status, ST_PAIR_OVERFLOW);
            continue;
        }
        const int jb = i + 1 + (c - choff[b]) * csize[b], je = jb + csize[b] < wend[b] ? jb + csize[b] : wend[b];
        sweep_range_block<R, true>(i, jb, je, n, smn, smx, sflag, pairs + offset[i] + cpref[c], order, wcnt, ign);
    }
}

template <class R>
__global__ void k_bp_count(int n, int limit0, const int* lost, const int* scene_axis, const R* smn, const R* smx, const int* sflag, const int* sscene,
                           int* count, int* stage, int* big, int* n_big, IgnoreLists ign) {
    const int limit = window_limit(limit0, lost);
    const int i = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    if (i == 0 && lane == 0) count[n] = 0;   // the scan's last place
    if (big_window(i, n, limit, scene_axis, smn, smx, sscene)) {   // left to k_bp_count_chunks
        if (lane == 0) big[atomicAdd(n_big, 1)] = i;
        return;
    }
    const int c = sweep_warp<R, false>(i, n, lane, scene_axis, smn, smx, sflag, sscene, stage, nullptr, nullptr, ign);
    if (lane == 0) count[i] = c;
}
// The count of kSweepShare consecutive positions by one warp: their windows nearly coincide, so each
// chunk of candidates is loaded once for all of them.  With a warp per position, 65,536 scattered
// bodies read 23 chunks each, some 1.5 GB out of the L2 cache (their step 1,469 / 1,454 us, that of
// 40,000 poured ones and 4,096 piles each some 2 % shorter).  From kSweepSharedFrom bodies on: below
// that a warp per position fills the GPU, and the longest window decides.
constexpr int kSweepShare = 4, kSweepSharedFrom = 16384;
template <class R>
__global__ void k_bp_count_shared(int n, int limit0, const int* lost, const int* scene_axis, const R* smn, const R* smx, const int* sflag,
                                  const int* sscene, int* count, int* stage, int* big, int* n_big, IgnoreLists ign) {
    const int limit = window_limit(limit0, lost);
    constexpr int U = kSweepShare;
    const int i0 = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5) * U;
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    if (i0 >= n) return;
    if (i0 == 0 && lane == 0) count[n] = 0;   // the scan's last place
    V3<R> mn[U], mx[U];
    R top[U];
    int sc[U], ax[U], fi[U], c[U];
    unsigned alive = 0;   // bit u: position i0 + u's window goes on
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int i = min(i0 + u, n - 1);
        mn[u] = V3<R>(smn[i], smn[n + i], smn[2 * (size_t)n + i]);
        mx[u] = V3<R>(smx[i], smx[n + i], smx[2 * (size_t)n + i]);
        sc[u] = sscene[i];
        ax[u] = scene_axis[sc[u]];
        fi[u] = sflag[i];
        top[u] = ax[u] == 0 ? mx[u].x : ax[u] == 1 ? mx[u].y : mx[u].z;
        c[u] = 0;
        if (i0 + u >= n) continue;
        if (big_window(i, n, limit, scene_axis, smn, smx, sscene)) {   // left to k_bp_count_chunks
            if (lane == 0) big[atomicAdd(n_big, 1)] = i;
            c[u] = -1;
        } else if (!(fi[u] & BF_IGNORE)) {
            alive |= 1u << u;
        }
    }
    const bool alone = *lost != 0;   // one position after the other then (see window_limit)
    for (unsigned left = alive; left;) {
        alive = alone ? left & (0u - left) : left;
        left &= ~alive;
        for (int j0 = i0 + __ffs(alive); alive && j0 < n; j0 += 32) {
            const int j = j0 + lane, k = min(j, n - 1);
            const V3<R> lo(smn[k], smn[n + k], smn[2 * (size_t)n + k]), hi(smx[k], smx[n + k], smx[2 * (size_t)n + k]);
            const int fj = sflag[k], sj = sscene[k];
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (!(alive >> u & 1u)) continue;   // the same for the whole warp
                const R low = ax[u] == 0 ? lo.x : ax[u] == 1 ? lo.y : lo.z;
                const bool past = j <= i0 + u, in = j < n && !(low > top[u]) && sj == sc[u];
                const unsigned live = __ballot_sync(full, past || in);
                bool hit = in && !past && !(fj & BF_IGNORE) && !((fi[u] & BF_KINEMATIC) && (fj & BF_KINEMATIC)) &&
                           !(mn[u].x > hi.x || lo.x > mx[u].x) && !(mn[u].y > hi.y || lo.y > mx[u].y) && !(mn[u].z > hi.z || lo.z > mx[u].z);
                if (hit && ign.off && ((fi[u] | fj) & BF_IGN_LIST)) hit = !ign.ignored(i0 + u, j);
                const unsigned m = __ballot_sync(full, hit);
                if (hit) {
                    const int at = c[u] + __popc(m & ((1u << lane) - 1u));
                    if (at < kStage) stage[(size_t)(i0 + u) * kStage + at] = j;
                }
                c[u] += __popc(m);
                if (live != full) alive &= ~(1u << u);
            }
        }
    }
    if (lane == 0)
        for (int u = 0; u < U; u++)
            if (i0 + u < n && c[u] >= 0) count[i0 + u] = c[u];
}

template <class R>
__global__ void k_bp_write(int n, int limit0, const int* lost, const int* scene_axis, const R* smn, const R* smx, const int* sflag, const int* sscene,
                           const uint32_t* order, const int* offset, const int* stage, int2* pairs, int pair_cap, int* status,
                           IgnoreLists ign, int n_scenes, const int* scene_off, int* pair_scene_off) {
    const int i = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    // each scene's first pair: that of its first sorted position
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s <= n_scenes; s += gridDim.x * blockDim.x) pair_scene_off[s] = offset[scene_off[s]];
    if (i >= n) return;
    const int limit = window_limit(limit0, lost);
    const int base = offset[i], c = offset[i + 1] - base;
    if (c == 0 || big_window(i, n, limit, scene_axis, smn, smx, sscene)) return;   // big windows: k_bp_write_chunks
    if (base + c > pair_cap) {
        if (lane == 0) atomicOr(status, ST_PAIR_OVERFLOW);
        return;
    }
    if (c <= kStage) {
        if (lane < c) pairs[base + lane] = make_int2((int)order[i], (int)order[stage[(size_t)i * kStage + lane]]);
    } else {
        sweep_warp<R, true>(i, n, lane, scene_axis, smn, smx, sflag, sscene, nullptr, pairs + base, order, ign);
    }
}

// Next sweep axis of each scene (BroadPhaseSweepAndPrune::calcCollisionPairs,
// broad_phase_sweep_and_prune.cpp:18-22, 37-40): the AABB centres (min + max) * 0.5 summed in the
// scene's sorted order, in the world's real type, one running sum per component for the centres and
// one for their squares, exactly as the reference accumulates them; then the variances
// s2 - s * s / n and the reference's strict comparisons.  A float sum is not associative, so the
// six sums run sequentially: one block of two warps per scene, warp 1 stages the next chunk of
// centres in shared memory while six lanes of warp 0 add up the current one.  A scene below two
// bodies keeps its axis (the reference returns before updating it).
template <class R> constexpr int axis_chunk() { return sizeof(R) == 4 ? 1024 : 512; }   // centres per staged chunk
template <class R>
__global__ void __launch_bounds__(64) k_bp_axis(const R* smn, const R* smx, int n, const int* scene_off, int* scene_axis, int* lost) {
    constexpr int CH = axis_chunk<R>(), PAD = CH + 1;   // the padding puts the three rows in different banks
    __shared__ R cbuf[2][3 * PAD];
    __shared__ R sums[6];
    const int s = blockIdx.x, tid = threadIdx.x;
    const int lo = scene_off[s], hi = scene_off[s + 1], cnt = hi - lo;
    if (s == 0 && tid == 0) *lost = 0;   // (the last kernel of a broadphase)
    if (cnt < 2) return;   // whole block
    auto stage = [&](int buf, int base, int t) {   // t in [0, 32): the staging warp's lane
        const int e = min(CH, hi - base);
        for (int k = t; k < e; k += 32)
            for (int d = 0; d < 3; d++)
                cbuf[buf][d * PAD + k] = (smn[(size_t)d * n + base + k] + smx[(size_t)d * n + base + k]) * R(0.5);
    };
    if (tid >= 32) stage(0, lo, tid - 32);
    __syncthreads();
    R acc = 0;   // tid d < 3: running sum of centre component d; tid 3 + d: of its square
    int buf = 0;
    for (int base = lo; base < hi; base += CH) {
        if (tid >= 32) {
            if (base + CH < hi) stage(buf ^ 1, base + CH, tid - 32);
        } else if (tid < 6) {
            const int e = min(CH, hi - base);
            const R* c = cbuf[buf] + (tid < 3 ? tid : tid - 3) * PAD;
            const bool sq = tid >= 3;
            int k = 0;
            for (; k + 8 <= e; k += 8) {   // loads ahead of the dependent adds, which stay in order
                R v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    v[u] = c[k + u];
                    if (sq) v[u] = v[u] * v[u];
                }
#pragma unroll
                for (int u = 0; u < 8; u++) acc = acc + v[u];
            }
            for (; k < e; k++) {
                R v = c[k];
                if (sq) v = v * v;
                acc = acc + v;
            }
        }
        __syncthreads();
        buf ^= 1;
    }
    if (tid < 6) sums[tid] = acc;
    __syncthreads();
    if (tid == 0) {
        R v[3];
        for (int d = 0; d < 3; d++) {
            const R ss = sums[d] * sums[d];
            v[d] = sums[3 + d] - ss / R(cnt);
        }
        int ax = 0;
        if (v[1] > v[0]) ax = 1;
        if (v[2] > v[ax]) ax = 2;
        scene_axis[s] = ax;
    }
}

} // namespace pe
