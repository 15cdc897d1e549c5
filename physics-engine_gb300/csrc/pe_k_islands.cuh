// Kernels of the rigid-body step, part 8: what the solver's iterations need to know of the contact
// graph (active results, islands in item order, and the islands' size classes).
#pragma once
#include "pe_k_flow.cuh"

namespace pe {

// Inputs and outputs of the island kernels.  P results (*P), NJ joints, N bodies; `bound` is the most items
// there can be.  Items are the A active results (those with points), in result order, then the joints.
struct IslandArgs {
    const int* P;
    int NJ, N, bound;
    const int *res_a, *res_b, *npts, *flags;
    const int2* jbody;
    int* parent;           // union-find over the bodies
    int* active;           // active results
    int* n_active;         // A
    int* n_items;          // M = A + NJ
    int* n_rows;           // contact points of all results
    uint32_t* key[2];      // the items' island labels and ids, sorted by label
    uint32_t* val[2];
    unsigned long long* aux;   // tile sums
    int* isl_scan;         // island starts before each sorted item, [M + 1]
    int* isl_off;          // the islands' first items, [islands + 1]
    int* n_isl;
    int big_items;         // and their size classes (k_isl_warp, k_isl_flow)
    int* list;
    int* n_list;           // [kWarpClasses], then n_flow, n_big
    int* base;
    int* big;
    int* n_colors;         // cleared
};

// Up to kIslandOne bodies, results and joints: everything in one block (17 launches before, 8 of them
// with one block of work).  Elsewhere:
//   k_act_sums, k_act_apply    active results, their count and the rows' total; union-find
//   k_isl_keys                 labels; then the radix sort
//   k_head_sums, k_head_apply  islands of the sorted items
//   k_isl_classes              their size classes
constexpr int kActItems = 2, kActTile = kBlock * kActItems;   // small tiles: a thread's unions are a chain (8 of them took 34 us for 6,500 results)
inline int act_tiles(long long n) { return (int)((n + kActTile - 1) / kActTile); }
constexpr int kIslandOne = 2048, kIslandBlock = 1024, kIslandOneBodies = 8192;
inline size_t island_one_smem(int n_bodies) {   // sorted keys and values, island offsets, digit counters, union-find
    return (size_t)(3 * kIslandOne + 2) * 4 + (size_t)(kIslandBlock / 32) * 256 * 2 + (size_t)n_bodies * 4;
}
__global__ void k_islands_one(IslandArgs a, int label_passes);
__global__ void k_act_sums(IslandArgs a);
__global__ void k_act_apply(IslandArgs a);
__global__ void k_isl_keys(IslandArgs a);
__global__ void k_head_sums(IslandArgs a, const uint32_t* key);
__global__ void k_head_apply(IslandArgs a, const uint32_t* key);
__global__ void k_isl_classes(IslandArgs a);

} // namespace pe
