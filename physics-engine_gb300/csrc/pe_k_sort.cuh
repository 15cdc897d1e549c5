// Kernels of the rigid-body step, part 2: exclusive scans and the stable LSD radix sort.
#pragma once
#include "pe_k_integrate.cuh"

namespace pe {

// ===================================================================== scan
// Exclusive scan of n ints in place, the total to *total (and to page-locked *host_total, if set): up to kScanOne in one block, else tile sums
// and a second launch whose blocks add up the tile sums before their own (no third launch for the
// sums' scan: a block's share is some hundred loads).  16 tiles of 1,024 took 29 us as rounds of one
// 256-thread block; 16,384 now take four rounds of 1,024 threads.
constexpr int kScanItems = 8, kScanTile = kBlock * kScanItems;
constexpr int kScanOne = 16384, kScanOneBlock = 1024, kScanOneItems = 4;
__global__ void k_scan_one(int* data, int n, int* total, int* host_total);
__global__ void k_scan_sums(const int* data, int n, int* aux);
__global__ void k_scan_apply(int* data, int n, const int* aux, int* total, int* host_total);
inline int scan_tiles(long long n) { return (int)((n + kScanTile - 1) / kScanTile); }

#ifdef __CUDACC__
template <class T> __device__ __forceinline__ T warp_incl_scan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}
// block-wide exclusive scan of one value per thread (every thread of a block of BLOCK); the block's total in *total
template <int BLOCK, class T> __device__ __forceinline__ T block_excl_scan(T v, T* total) {
    __shared__ T warp_sums[BLOCK / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T incl = warp_incl_scan(v);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        T w = lane < BLOCK / 32 ? warp_sums[lane] : T(0);
        w = warp_incl_scan(w);
        if (lane < BLOCK / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    const T before = warp == 0 ? T(0) : warp_sums[warp - 1];
    *total = warp_sums[BLOCK / 32 - 1];
    __syncthreads();
    return before + incl - v;
}
// the sum of aux[0 .. tile), the same in every thread of the block
template <int BLOCK, class T> __device__ __forceinline__ T tiles_before(const T* aux, int tile) {
    T s = 0, all;
    for (int k = threadIdx.x; k < tile; k += BLOCK) s += aux[k];
    block_excl_scan<BLOCK>(s, &all);
    return all;
}
#endif

// ===================================================================== radix sort
// Stable sort of (key, value) pairs, least-significant digit first, 8-bit digits.  A pass is a
// histogram per tile and a scatter; with more than kRadixFused tiles a third launch turns the tiles'
// histograms into offsets, else the scatter's blocks add up the tiles before theirs themselves.  The
// digit is the key's, or, with `scene` set, that of scene[value] (the more significant key of
// bodies of several scenes).  The item count is n, or *nd when nd is set (a count the device computed:
// the grid covers the upper bound n, and the tiles past the count do nothing).
//
// A tile's items are ranked warp by warp: each warp counts its own 32 x ITEMS items in order, and the
// block meets three times per tile (4,096 items in 16 rounds of six barriers took 35 us alone on an SM).
// Small sorts take small tiles, so that they cover the SMs: 1,024 items up to kRadixSmallTiles tiles.
constexpr int kRadixFused = 64, kRadixSmallTiles = 256;
constexpr int kRadixItems = 4, kRadixItemsBig = 16;
inline bool radix_big(int n) { return n > kRadixSmallTiles * kBlock * kRadixItems; }
inline int radix_tile(int n) { return kBlock * (radix_big(n) ? kRadixItemsBig : kRadixItems); }
inline int radix_tiles(int n) { return (n + radix_tile(n) - 1) / radix_tile(n); }
inline size_t radix_hist_ints(int n) { return (size_t)256 * (radix_tiles(n) + 1); }   // tile-major, then the digits' totals
template <class K> struct RadixArgs {
    const K* key;
    const uint32_t* val;
    K* key_out;
    uint32_t* val_out;
    const int* scene;
    int n;
    const int* nd;
    int shift;
    int* hist;
    int tiles;
};
__global__ void k_radix_offsets(int* hist, int tiles, int tile_items, int n, const int* nd);

template <class K> __device__ __forceinline__ int digit_of(const RadixArgs<K>& a, K key, uint32_t val) {
    return a.scene ? (a.scene[val] >> a.shift) & 0xff : (int)(key >> a.shift) & 0xff;
}

template <class K, int ITEMS> __global__ void __launch_bounds__(kBlock) k_radix_hist(RadixArgs<K> a) {
    __shared__ int cnt[256];
    const int n = a.nd ? *a.nd : a.n;
    const int base = blockIdx.x * (kBlock * ITEMS);
    if (base >= n) return;
    cnt[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int i = base + r * kBlock + threadIdx.x;
        if (i < n) atomicAdd(&cnt[digit_of(a, a.scene ? K(0) : a.key[i], a.scene ? a.val[i] : 0u)], 1);
    }
    __syncthreads();
    a.hist[blockIdx.x * 256 + threadIdx.x] = cnt[threadIdx.x];
}

template <class K, int ITEMS> __global__ void __launch_bounds__(kBlock) k_radix_scatter(RadixArgs<K> a) {
    constexpr int W = kBlock / 32, TILE = kBlock * ITEMS;
    __shared__ int cnt[W][256];   // per warp and digit: items so far, then the first one's place
    const int n = a.nd ? *a.nd : a.n;
    if ((int)blockIdx.x * TILE >= n) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d0 = threadIdx.x;
    const int first = blockIdx.x * TILE + warp * 32 * ITEMS + lane;
    K key[ITEMS];
    uint32_t val[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int i = first + r * 32;
        key[r] = i < n ? a.key[i] : K(0);
        val[r] = i < n ? a.val[i] : 0u;
    }
    for (int w = 0; w < W; w++) cnt[w][d0] = 0;
    // the digit's items in the tiles before, and in all of them
    int before = 0, total = 0;
    if (a.tiles <= kRadixFused) {
        const int live = (n + TILE - 1) / TILE;
#pragma unroll 8
        for (int t = 0; t < live; t++) {
            const int v = a.hist[t * 256 + d0];
            before += t < (int)blockIdx.x ? v : 0;
            total += v;
        }
    } else {
        before = a.hist[blockIdx.x * 256 + d0];
        total = a.hist[a.tiles * 256 + d0];
    }
    int all;
    before += block_excl_scan<kBlock>(total, &all);   // (also the barrier after the counters' clearing)
    int digit[ITEMS], rank[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const bool live = first + r * 32 < n;
        digit[r] = live ? digit_of(a, key[r], val[r]) : 256 + lane;   // dead lanes match no live one
        const unsigned peers = __match_any_sync(0xffffffffu, digit[r]);
        rank[r] = live ? cnt[warp][digit[r]] + __popc(peers & ((1u << lane) - 1u)) : 0;
        __syncwarp();
        if (live && (int)lane == __ffs(peers) - 1) cnt[warp][digit[r]] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (int w = 0; w < W; w++) { const int c = cnt[w][d0]; cnt[w][d0] = before; before += c; }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        if (first + r * 32 >= n) continue;
        const int pos = cnt[warp][digit[r]] + rank[r];
        a.key_out[pos] = key[r];
        a.val_out[pos] = val[r];
    }
}

} // namespace pe
