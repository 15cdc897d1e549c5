// World<R> member definitions, part 2: the step, phase by phase (sort and scan utilities,
// integrate, broadphase, narrowphase, solve, big islands), and its captured CUDA graph.
#pragma once
#include "pe_world_setup.cuh"

namespace pe {

// ------------------------------------------------------------------ utilities
template <class R> void World<R>::scan_async(int* data, int n, int* total, int* host_total) {
    if (n <= kScanOne) {
        launch_block(K_SCAN, 1, kScanOneBlock, k_scan_one, data, n, total, host_total);
    } else {
        const int tiles = scan_tiles(n);
        aux_.ensure(tiles);
        launch(K_SCAN, tiles, k_scan_sums, (const int*)data, n, aux_.p);
        launch(K_SCAN, tiles, k_scan_apply, data, n, (const int*)aux_.p, total, host_total);
    }
}

// one pass of the radix sort over up to n items; the buffers a holds are swapped
template <class R> template <class K> void World<R>::radix_pass(RadixArgs<K>& a) {
    a.tiles = radix_tiles(a.n);
    a.hist = hist_.p;
    const bool big = radix_big(a.n);
    launch(K_RADIX, a.tiles, big ? k_radix_hist<K, kRadixItemsBig> : k_radix_hist<K, kRadixItems>, a);
    if (a.tiles > kRadixFused) launch(K_RADIX, 256, k_radix_offsets, a.hist, a.tiles, radix_tile(a.n), a.n, a.nd);
    launch(K_RADIX, a.tiles, big ? k_radix_scatter<K, kRadixItemsBig> : k_radix_scatter<K, kRadixItems>, a);
    K* key = a.key_out;
    uint32_t* val = a.val_out;
    a.key_out = const_cast<K*>(a.key);
    a.val_out = const_cast<uint32_t*>(a.val);
    a.key = key;
    a.val = val;
}

template <class R> void World<R>::ensure_pair_capacity(int P) {
    if (P <= pair_cap_) return;
    const int cap = std::max(P + P / 2, 1024);
    pairs_.ensure(cap);
    cls_.ensure(cap); order_np_.ensure(cap);
    res_a_.ensure(cap); res_b_.ensure(cap); res_np_.ensure(cap + 1);
    res_fr_.ensure(cap); res_re_.ensure(cap);
    res_pts_.ensure((size_t)NPF * cap * kSlots);
    // result slot distances survive between steps: grow both generations keeping contents
    res_dist_[0].ensure((size_t)cap * kSlots, true);
    res_dist_[1].ensure((size_t)cap * kSlots, true);
    active_.ensure(cap + 1);
    sat_out_.ensure((size_t)cap * kSatOut);
    // point buffer: field-major over the capacity; its contents live for one step only
    pair_cap_ = cap;
}

// ------------------------------------------------------------------ phases
template <class R> void World<R>::integrate() {
    if (N_ == 0) return;
    launch(K_INTEGRATE, grid(N_), k_integrate<R>, bodies(), shapes(), prm_, 1);
    PE_CK(cudaGetLastError());
}

// Broadphase up to the pair count: sort, sweep counts, scan; the host waits for the count (the
// pair capacity follows it).  The count also stays on the device for the kernels after it.
template <class R> int World<R>::bp_count() {
    if (N_ < 2) return P_;   // the reference leaves the pair list untouched below two bodies
    bp_count_enqueue();
    PE_CK(cudaStreamSynchronize(st_));
    return hstat_[HS_P];
}

// the launches of bp_count, the last of which writes the count to page-locked memory (no wait)
template <class R> void World<R>::bp_count_enqueue() {
    const int n = N_;
    if (n < 2) return;
    for (int k = 0; k < 2; k++) { key_[k].ensure(n); val_[k].ensure(n); }
    smn_.ensure((size_t)3 * n); smx_.ensure((size_t)3 * n); sflag_.ensure(n); ssc_.ensure(n);
    count_.ensure(n + 1);
    bp_stage_.ensure((size_t)n * kStage);
    bp_big_.ensure(n + 1);
    SweepBoxes<R> boxes;
    boxes.mn = smn_.p; boxes.mx = smx_.p; boxes.flag = sflag_.p; boxes.scene = ssc_.p; boxes.lost = bp_nbig_.p + 1;
    if (max_scene_ <= std::min(tun_.scene_sort_max, kSceneSortMax)) {   // every scene sorted inside one block
        launch_block(K_RADIX, NS_, kSceneSortBlock, k_bp_sort_scenes<R>, bodies(), (const int*)scene_axis_.p, (const int*)scene_off_.p,
                     val_[0].p, boxes, bp_nbig_.p);
        order_ = val_[0].p;
    } else {
        using K = typename KeyOf<R>::type;
        K* key[2] = {reinterpret_cast<K*>(key_[0].p), reinterpret_cast<K*>(key_[1].p)};
        launch(K_BP_KEYS, grid(n), k_bp_keys<R>, bodies(), scene_axis_.p, key[0], val_[0].p);
        RadixArgs<K> a{key[0], val_[0].p, key[1], val_[1].p, nullptr, n, nullptr, 0, nullptr, 0};
        hist_.ensure(radix_hist_ints(n));
        for (a.shift = 0; a.shift < (int)sizeof(K) * 8; a.shift += 8) radix_pass(a);
        a.scene = bscene_.p;
        a.shift = 0;
        for (int m = NS_ - 1; m > 0; m >>= 8, a.shift += 8) radix_pass(a);
        order_ = const_cast<uint32_t*>(a.val);
        launch(K_BP_GATHER, grid(n), k_bp_gather<R>, bodies(), (const uint32_t*)order_, boxes, bp_nbig_.p);
    }
    IgnoreLists ign;
    if (n_ign_ > 0) { ign.off = ign_off_.p; ign.ids = ign_ids_.p; ign.order = order_; }
    const bool share = n >= kSweepSharedFrom;
    const int limit = big_window_limit(max_scene_);
    launch(K_BP_SWEEP, grid_warps(share ? (n + kSweepShare - 1) / kSweepShare : n), share ? k_bp_count_shared<R> : k_bp_count<R>, n, limit,
           (const int*)boxes.lost, scene_axis_.p, smn_.p, smx_.p, sflag_.p, ssc_.p, count_.p, bp_stage_.p,
           bp_big_.p, bp_nbig_.p, ign);
    // crowded positions: windows in chunks of one block each (at most kMaxChunks per position); a
    // window holds at most the scene's other bodies, so scenes of at most `limit` bodies have none
    const bool crowded = max_scene_ > limit;
    bp_wend_.ensure(n + 1); bp_csize_.ensure(n + 1); bp_nch_.ensure(n + 1); bp_choff_.ensure(n + 1); bp_ctot_.ensure(1);
    bp_ccount_.ensure((size_t)kMaxChunks * n + 1); bp_cpref_.ensure((size_t)kMaxChunks * n + 1);
    if (crowded) launch(K_BP_SWEEP, kBigSweepBlocks, k_bp_big_windows<R>, n, (const int*)scene_axis_.p, (const int*)scene_off_.p, (const R*)smn_.p,
           (const R*)smx_.p, (const int*)ssc_.p, (const int*)bp_big_.p, (const int*)bp_nbig_.p, bp_wend_.p, bp_csize_.p, bp_nch_.p);
    if (crowded) launch_block(K_BP_SWEEP, 1, 32, k_bp_chunk_offsets, (const int*)bp_nbig_.p, (const int*)bp_nch_.p, bp_choff_.p, bp_ctot_.p);
    if (crowded) launch(K_BP_SWEEP, 2 * kBigSweepBlocks, k_bp_count_chunks<R>, n, (const R*)smn_.p, (const R*)smx_.p, (const int*)sflag_.p,
           (const int*)bp_big_.p, (const int*)bp_nbig_.p, (const int*)bp_wend_.p, (const int*)bp_csize_.p, (const int*)bp_choff_.p,
           (const int*)bp_ctot_.p, bp_ccount_.p, ign);
    if (crowded) launch(K_BP_SWEEP, kBigSweepBlocks, k_bp_chunk_sums, (const int*)bp_big_.p, (const int*)bp_nbig_.p, (const int*)bp_choff_.p,
           (const int*)bp_nch_.p, (const int*)bp_ccount_.p, bp_cpref_.p, count_.p);
    scan_async(count_.p, n + 1, dcnt_.p + DC_P, hstat_ + HS_P);
}

// Every buffer the rest of the step writes, sized for P pairs before any of its launches, so that
// nothing is allocated while a step graph is captured.  Island items (active results and joints)
// are bounded by the pair capacity plus the joints.
template <class R> void World<R>::prepare_tail(int P) {
    ensure_pair_capacity(std::max(P, 1));
    // a result has at most kSlots points: its rows start at kSlots times its index
    rows_.ensure((size_t)NRF * kSlots * pair_cap_);
    const int bound = pair_cap_ + n_joints_;
    const int keys = std::max(N_, bound);
    // the sort buffers also hold the broadphase's body order until the pair list is written: a
    // growth keeps their contents and order_ follows its buffer
    const int oi = order_ == val_[1].p ? 1 : 0;
    const bool ordered = order_ != nullptr;
    for (int k = 0; k < 2; k++) { key_[k].ensure(keys); val_[k].ensure(keys, true); }
    if (ordered) order_ = val_[oi].p;
    hist_.ensure(radix_hist_ints(bound));
    isl_aux_.ensure(std::max(scan_tiles(bound), act_tiles(pair_cap_)) + 1);
    isl_flag_.ensure(bound + 1); isl_off_.ensure(bound + 1);
    isl_n_.ensure(1); ncol_.ensure(1);
    isl_list_.ensure(class_base(kWarpClasses, bound)); isl_base_.ensure(bound + 1); isl_big_.ensure(bound + 1);
    isl_levels_.ensure(bound + 1); isl_colors_.ensure(bound + 1); isl_state_.ensure(bound + 1);
    flow_item_.ensure(bound); flow_isl_.ensure(bound); flow_color_.ensure(bound);
    flow_next_.ensure((size_t)2 * bound); flow_succ_.ensure((size_t)2 * bound);
    flow_box_.ensure((size_t)2 * bound * token_words<R>());
    flow_head_.ensure(N_ + 1); flow_ff_.ensure(1);
    parent_.ensure(N_ + 1);
    cls_rng_.ensure(PC_COUNT); cls_work_.ensure(PC_COUNT);
    if (!sat_attr_) {   // dynamic shared memory of the staged SAT kernels (above the 48 KB default for FP64)
        const int light = (int)(kSatWarps * sat_group_reals<R>(1) * sizeof(R));
        PE_CK(cudaFuncSetAttribute(k_np_sat<R, 1, ST_BOX, ST_HULL>, cudaFuncAttributeMaxDynamicSharedMemorySize, light));
        PE_CK(cudaFuncSetAttribute(k_np_sat<R, 1, ST_HULL, ST_BOX>, cudaFuncAttributeMaxDynamicSharedMemorySize, light));
        PE_CK(cudaFuncSetAttribute(k_np_sat<R, 1, ST_HULL, ST_HULL>, cudaFuncAttributeMaxDynamicSharedMemorySize, light));
        PE_CK(cudaFuncSetAttribute(k_np_sat<R, 1, ST_CYLINDER, ST_CYLINDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, light));
        PE_CK(cudaFuncSetAttribute(k_np_sat<R, kSatGroup, -1, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(sat_group_reals<R>(kSatGroup) * sizeof(R))));
        PE_CK(cudaFuncSetAttribute(k_islands_one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)island_one_smem(kIslandOneBodies)));
        sat_attr_ = true;
    }
}

// the pair list from the counted sweep, and each scene's first pair
template <class R> void World<R>::bp_tail() {
    const int n = N_, limit = big_window_limit(max_scene_);
    if (n < 2) return;
    IgnoreLists ign;
    if (n_ign_ > 0) { ign.off = ign_off_.p; ign.ids = ign_ids_.p; ign.order = order_; }
    launch(K_BP_SWEEP, grid_warps(n), k_bp_write<R>, n, limit, (const int*)bp_nbig_.p + 1, scene_axis_.p, smn_.p, smx_.p, sflag_.p, ssc_.p, order_, count_.p, bp_stage_.p,
           pairs_.p, pair_cap_, status_.p, ign, NS_, (const int*)scene_off_.p, pair_scene_off_.p);
    if (max_scene_ > limit)
        launch(K_BP_SWEEP, 2 * kBigSweepBlocks, k_bp_write_chunks<R>, n, (const R*)smn_.p, (const R*)smx_.p, (const int*)sflag_.p,
               (const uint32_t*)order_, (const int*)count_.p, (const int*)bp_big_.p, (const int*)bp_nbig_.p, (const int*)bp_wend_.p,
               (const int*)bp_csize_.p, (const int*)bp_choff_.p, (const int*)bp_ctot_.p, (const int*)bp_cpref_.p, pairs_.p, pair_cap_,
               status_.p, ign);
}

// The scenes' next sweep axes, from the sorted boxes.  A sum of all bodies in order is a chain (378 us
// for 65,536 bodies in FP32, 157 us for 1,601 in FP64) that nothing reads before the next step: a
// step runs it beside its narrowphase and solver, on a stream of its own.
template <class R> void World<R>::bp_axis() {
    if (N_ < 2) return;
    launch_block(K_BP_AXIS, NS_, 64, k_bp_axis<R>, (const R*)smn_.p, (const R*)smx_.p, N_, (const int*)scene_off_.p, scene_axis_.p, bp_nbig_.p + 1);
}
template <class R> void World<R>::bp_axis_begin() {
    PE_CK(cudaEventRecord(axis_ev_[0], st_));   // the pair list has been written: its sweep reads the axes
    PE_CK(cudaStreamWaitEvent(axis_st_, axis_ev_[0], 0));
    cur_ = axis_st_;
    bp_axis();
    cur_ = nullptr;
}
template <class R> void World<R>::bp_axis_end() {
    PE_CK(cudaEventRecord(axis_ev_[1], axis_st_));
    PE_CK(cudaStreamWaitEvent(st_, axis_ev_[1], 0));
}

template <class R> int World<R>::broadphase() {
    const int P = bp_count();
    prepare_tail(P);
    bp_tail();
    bp_axis();
    PE_CK(cudaGetLastError());
    P_ = P;
    if (N_ >= 2) self_pairs_ = false;   // (below two bodies the pair list stays)
    return P;
}

// Side streams for the pair classes, largest estimated work first (the last counts x a rough
// per-pair cost), each to the least loaded stream.
template <class R> void World<R>::plan_streams(int* plan) const {
    static_assert(PC_COUNT == 15, "one cost per pair class");
    static constexpr double kClassCost[PC_COUNT] = {2, 1, 1, 1, 4, 20, 6, 12, 400, 40, 40, 60, 20, 30, 30};
    int order_c[PC_COUNT];
    double load[kSideStreams] = {};
    for (int c = 0; c < PC_COUNT; c++) order_c[c] = c;
    std::stable_sort(order_c, order_c + PC_COUNT, [&](int a, int b) { return h_cls_[a] * kClassCost[a] > h_cls_[b] * kClassCost[b]; });
    for (int k = 0; k < PC_COUNT; k++) {
        const int c = order_c[k];
        const int best = (int)(std::min_element(load, load + kSideStreams) - load);
        plan[c] = best;
        load[best] += h_cls_[c] * kClassCost[c];
    }
}

// The pair classes (bit per class) that pairs of the tables' shapes can have (k_np_classify).  The others'
// kernels, up to 17 of 20, are not launched: each is a node of some 2 us in one of four chains.
template <class R> unsigned World<R>::possible_classes() const {
    static_assert(kCylF <= kSatF && kCylE <= kSatE && kBoxE <= kSatE, "boxes and cylinders fit the staged SAT");
    auto has = [&](int t) { return (kinds_ >> t & 1u) != 0; };
    unsigned m = 0;
    for (int a = 0; a < 32; a++)
        for (int b = 0; b <= a; b++)
            if (has(a) && has(b)) m |= 1u << pair_class(a, b);
    if (!(m >> PC_CONVEX & 1u)) return m;
    const bool hull = has(ST_HULL);
    if (!(hull && has(ST_BOX))) m &= ~(1u << PC_CONVEX);
    else m |= 1u << PC_CONVEX_HULL_BOX;
    if (hull) m |= 1u << PC_CONVEX_HULL_HULL;
    if (has(ST_CYLINDER)) m |= 1u << PC_CONVEX_CYL_CYL;
    if (most_faces_ > kSatF || most_edges_ > kSatE || most_verts_ > kSatV) m |= 1u << PC_CONVEX_BIG;
    const long long f = std::max(most_faces_, kCylF), e = std::max(most_edges_, kCylE), v = std::max(most_verts_, 12);
    if ((2 * f + e * e) * (2 * v) >= tun_.sat_heavy_cost) m |= 1u << PC_CONVEX_HEAVY;
    return m;
}

// Narrowphase without host waits: pairs classified and bucketed by class on the device, the class
// ranges computed there, and every class's kernel launched over its range (grids from the pair
// capacity, persistent up to the resident blocks), side by side on the side streams.
template <class R> void World<R>::np_enqueue() {
    const int cap = pair_cap_;
    const int* Pd = dcnt_.p + DC_P;
    const Results<R> rs = results();
    const Bodies<R> bd = bodies();
    const ShapeTable<R> sh = shapes();
    NpPlan plan;
    plan.P = Pd; plan.n_scenes = NS_;
    plan.pair_off = pair_scene_off_.p; plan.res_off = res_scene_off_.p; plan.prev_off = prev_res_off_.p; plan.n_res = dcnt_.p + DC_R;
    plan.count = cls_count_.p; plan.cursor = cls_count_.p + PC_COUNT; plan.last = cls_count_.p + 2 * PC_COUNT; plan.work = cls_work_.p;
    plan.range = cls_rng_.p; plan.order = order_np_.p;
    const long long heavy = tun_.sat_heavy_cost;
    if (cap <= kPlanOne) {
        launch_block(K_NP_BUCKET, 1, kPlanBlock, k_np_plan_one<R>, plan, (const int2*)pairs_.p, bd, sh, heavy);
    } else {
        launch(K_NP_BUCKET, pgrid(cap, kBlock, k_np_classify<R>), k_np_classify<R>, plan, (const int2*)pairs_.p, bd, sh, cls_.p, heavy);
        launch_block(K_NP_BUCKET, 1, 32, k_np_ranges, plan);
        launch(K_NP_BUCKET, pgrid(cap, kBlock, k_np_bucket), k_np_bucket, plan, (const int*)cls_.p);
    }
    // The classes' kernels touch disjoint pairs and results: they run side by side on the side
    // streams, so the long tails of the per-pair kernels overlap the other classes.
    fork_streams();
    const unsigned possible = possible_classes();
    for (int c = 0; c < PC_COUNT; c++) {
        if (!(possible >> c & 1u)) continue;
        use_stream(stream_of_[c] % tun_.side_streams);
        const int2* rg = cls_rng_.p + c;
        int* wk = cls_work_.p + c;
        const int* on = order_np_.p;
        const int2* pp = pairs_.p;
        const int* pso = pair_scene_off_.p;
        const int* pro = prev_res_off_.p;
        switch (c) {
            case PC_BOX_BOX: launch(K_NP, pgrid(cap, kBlock, k_np_class<R, PC_BOX_BOX>), k_np_class<R, PC_BOX_BOX>, rg, on, pp, bd, sh, rs, pso, pro); break;
            case PC_BOX_SPHERE: launch(K_NP, pgrid(cap, kBlock, k_np_class<R, PC_BOX_SPHERE>), k_np_class<R, PC_BOX_SPHERE>, rg, on, pp, bd, sh, rs, pso, pro); break;
            case PC_SPHERE_SPHERE: launch(K_NP, pgrid(cap, kBlock, k_np_class<R, PC_SPHERE_SPHERE>), k_np_class<R, PC_SPHERE_SPHERE>, rg, on, pp, bd, sh, rs, pso, pro); break;
            case PC_SPHERE_CYL: launch(K_NP, pgrid(cap, kBlock, k_np_class<R, PC_SPHERE_CYL>), k_np_class<R, PC_SPHERE_CYL>, rg, on, pp, bd, sh, rs, pso, pro); break;
            case PC_BOX_CYL: launch(K_NP, pgrid(cap, kBlock, k_np_class<R, PC_BOX_CYL>), k_np_class<R, PC_BOX_CYL>, rg, on, pp, bd, sh, rs, pso, pro); break;
            case PC_CONCAVE:
            case PC_COMPOUND:
                launch_block(K_NP, pgrid(cap, 1, k_np_mesh<R>, 32), 32, k_np_mesh<R>, rg, wk, on, pp, bd, sh, rs, pso, pro);
                break;
            case PC_SPHERE_HULL: {
                const int w = sphere_hull_warps<R>();
                launch_block(K_NP, pgrid(cap, w, k_np_sphere_hull<R>, 32 * w), 32 * w, k_np_sphere_hull<R>, rg, wk, on, pp, bd, sh, rs, pso, pro);
                break;
            }
            case PC_CYL_HULL: {
                const int w = cyl_hull_warps<R>();
                launch_block(K_NP, pgrid(cap, w, k_np_cyl_hull<R>, 32 * w), 32 * w, k_np_cyl_hull<R>, rg, wk, on, pp, bd, sh, rs, pso, pro);
                break;
            }
            case PC_CONVEX:
            case PC_CONVEX_HULL_BOX:
            case PC_CONVEX_HULL_HULL:
            case PC_CONVEX_CYL_CYL: {
                const size_t smem = (size_t)kSatWarps * sat_group_reals<R>(1) * sizeof(R);
                const int bs = 32 * kSatWarps;
                auto kern = c == PC_CONVEX ? k_np_sat<R, 1, ST_BOX, ST_HULL>
                          : c == PC_CONVEX_HULL_BOX ? k_np_sat<R, 1, ST_HULL, ST_BOX>
                          : c == PC_CONVEX_HULL_HULL ? k_np_sat<R, 1, ST_HULL, ST_HULL>
                          : k_np_sat<R, 1, ST_CYLINDER, ST_CYLINDER>;
                launch_smem(K_NP_SAT, pgrid(cap, kSatWarps, kern, bs, smem), bs, smem, kern, rg, wk, on, pp, bd, sh, sat_out_.p);
                launch(K_NP_SAT, pgrid(cap, kBlock, k_np_sat_finish<R>), k_np_sat_finish<R>, rg, on, pp, bd, sh, rs, pso, pro,
                       (const R*)sat_out_.p);
                break;
            }
            case PC_CONVEX_HEAVY: {
                const size_t smem = (size_t)sat_group_reals<R>(kSatGroup) * sizeof(R);
                auto kern = k_np_sat<R, kSatGroup, -1, -1>;
                launch_smem(K_NP_SAT, pgrid(cap, 1, kern, 32 * kSatGroup, smem), 32 * kSatGroup, smem, kern, rg, wk, on, pp, bd, sh, sat_out_.p);
                launch(K_NP_SAT, pgrid(cap, kBlock, k_np_sat_finish<R>), k_np_sat_finish<R>, rg, on, pp, bd, sh, rs, pso, pro,
                       (const R*)sat_out_.p);
                break;
            }
            default:   // PC_CONVEX_BIG
                launch(K_NP_SAT, pgrid(cap, kBlock / 32, k_np_sat_big<R>), k_np_sat_big<R>, rg, wk, on, pp, bd, sh, rs, pso, pro);
                break;
        }
    }
    join_streams();
}

template <class R> void World<R>::narrowphase() {
    prepare_tail(P_);
    plan_streams(stream_of_);
    cur_dist_ ^= 1;
    np_enqueue();
    PE_CK(cudaGetLastError());
    R_ = P_;
    self_ = self_pairs_;
}

// Solver without host waits: rows (on a side stream), islands (pe_k_islands.cuh), the iterations
// (pe_k_flow.cuh); then the step's counters, written to host memory by the last kernel.
template <class R> void World<R>::solve_enqueue(int mode) {
    if (N_ == 0) return;
    const int cap = pair_cap_, NJ = n_joints_, bound = cap + NJ;
    const int* Rd = dcnt_.p + DC_R;
    int *Ad = dcnt_.p + DC_A, *Md = dcnt_.p + DC_M;
    const Joints<R> jt = joints();
    PE_CK(cudaEventRecord(fork_ev_, st_));
    PE_CK(cudaStreamWaitEvent(side_[0], fork_ev_, 0));
    use_stream(0);
    launch(K_SI_SETUP, pgrid(cap, kBlock, k_si_setup<R>), k_si_setup<R>, Rd, results(), bodies(), rows(), prm_);
    if (NJ > 0) launch(K_SI_SETUP, grid(NJ), k_joint_init<R>, jt, bodies(), prm_);
    cur_ = nullptr;
    IslandArgs a;
    a.P = Rd; a.NJ = NJ; a.N = N_; a.bound = bound;
    a.res_a = res_a_.p; a.res_b = res_b_.p; a.npts = res_np_.p; a.flags = bflags_.p; a.jbody = jbody_.p;
    a.parent = parent_.p; a.active = active_.p; a.n_active = Ad; a.n_items = Md; a.n_rows = rows_total_.p;
    for (int k = 0; k < 2; k++) { a.key[k] = reinterpret_cast<uint32_t*>(key_[k].p); a.val[k] = val_[k].p; }
    a.aux = isl_aux_.p; a.isl_scan = isl_flag_.p; a.isl_off = isl_off_.p; a.n_isl = isl_n_.p;
    a.big_items = tun_.big_island_items;
    a.list = isl_list_.p; a.n_list = dcnt_.p + DC_NLIST; a.base = isl_base_.p; a.big = isl_big_.p;
    a.n_colors = mode == 0 ? nullptr : ncol_.p;
    const uint32_t* order = val_[0].p;
    int label_passes = 0;
    for (int m = std::max(NJ > 0 ? N_ : N_ - 1, 1); m > 0; m >>= 8) label_passes++;   // joint labels reach n_bodies; one at least places the keys
    if (bound <= kIslandOne && N_ <= kIslandOneBodies) {
        const size_t smem = island_one_smem(N_);
        launch_smem(K_ISLAND, 1, kIslandBlock, smem, k_islands_one, a, label_passes);
    } else {
        launch(K_ISLAND, pgrid(std::max(cap, N_), kActTile, k_act_sums), k_act_sums, a);
        launch(K_ISLAND, act_tiles(cap), k_act_apply, a);
        launch(K_ISLAND, pgrid(bound, kBlock, k_isl_keys), k_isl_keys, a);
        RadixArgs<uint32_t> r{a.key[0], a.val[0], a.key[1], a.val[1], nullptr, bound, Md, 0, nullptr, 0};
        for (int k = 0; k < label_passes; k++, r.shift += 8) radix_pass(r);
        order = r.val;
        launch(K_ISLAND, scan_tiles(bound), k_head_sums, a, r.key);
        launch(K_ISLAND, scan_tiles(bound), k_head_apply, a, r.key);
        launch(K_ISLAND, pgrid(bound, kBlock, k_isl_classes), k_isl_classes, a);
    }
    PE_CK(cudaEventRecord(join_ev_[0], side_[0]));
    PE_CK(cudaStreamWaitEvent(st_, join_ev_[0], 0));
    if (self_) solve_islands<true, true>(mode, order);
    else if (NJ > 0) solve_islands<true, false>(mode, order);
    else solve_islands<false, false>(mode, order);
    launch_block(K_MISC, 1, 32, k_step_counters, (const int*)status_.p, (const int*)rows_total_.p, Ad, (const int*)isl_n_.p,
                 (const int*)(dcnt_.p + DC_NBIG), (const int*)isl_big_.p, (const int*)isl_levels_.p,
                 mode == 0 ? (const int*)nullptr : (const int*)ncol_.p, (const int*)cls_count_.p + 2 * PC_COUNT, hstat_);
}

// The solver's iterations: the islands that fit a warp, then those that do not.
template <class R> template <bool JOINTS, bool SELF> void World<R>::solve_islands(int mode, const uint32_t* order) {
    const int bound = pair_cap_ + n_joints_, small = tun_.small_island_items, big = tun_.big_island_items;
    int* n_list = dcnt_.p + DC_NLIST;
    int* colors = mode == 0 ? nullptr : ncol_.p;
    // (a warp for every island, up to the resident ones: see the islands per warp)
    launch_block(K_SI_SERIAL, pgrid(bound, kWarpBlock / 32, k_isl_warp<R, JOINTS, SELF>, kWarpBlock), kWarpBlock, k_isl_warp<R, JOINTS, SELF>,
                 (const int*)isl_list_.p, (const int*)n_list, bound, (const int*)isl_off_.p, order, results(), joints(), bodies(), rows(),
                 prm_.iterations, small, colors, status_.p);
    FlowArgs<R> f;
    f.n_items = dcnt_.p + DC_M; f.isl_scan = isl_flag_.p; f.isl_off = isl_off_.p; f.order = order;
    f.base = isl_base_.p; f.n_flow = dcnt_.p + DC_NFLOW; f.big = isl_big_.p; f.n_big = dcnt_.p + DC_NBIG;
    f.big_items = big; f.color_min = small; f.exact_levels = tun_.exact_levels_colored; f.mode = mode; f.iterations = prm_.iterations;
    f.item = flow_item_.p; f.isl = flow_isl_.p; f.color = flow_color_.p; f.head = flow_head_.p; f.next = flow_next_.p; f.succ = flow_succ_.p;
    f.box = flow_box_.p; f.isl_levels = isl_levels_.p; f.isl_colors = isl_colors_.p; f.isl_state = isl_state_.p;
    f.any_first_fit = flow_ff_.p; f.n_colors = ncol_.p; f.status = status_.p;
    launch_coop(K_SI_COLOR, resident(k_isl_flow<R, JOINTS, SELF>, kFlowBlock, 0), kFlowBlock, k_isl_flow<R, JOINTS, SELF>, f, results(),
                joints(), bodies(), rows());
}

// The step's second host wait: its counters and status.
template <class R> void World<R>::finish() {
    PE_CK(cudaStreamSynchronize(st_));
    if (N_ == 0) return;
    n_rows_ = hstat_[HS_ROWS];
    n_active_ = hstat_[HS_ACTIVE];
    n_islands_ = hstat_[HS_ISLANDS];
    n_colors_ = hstat_[HS_COLORS];
    for (int c = 0; c < PC_COUNT; c++) h_cls_[c] = hstat_[HS_CLS + c];
    const int status = hstat_[HS_STATUS];
    if (status) {
        PE_CK(cudaMemsetAsync(status_.p, 0, sizeof(int), st_));
        PE_CK(cudaStreamSynchronize(st_));
        throw std::runtime_error((status & ST_FLOW_STALL ? "solver stalled (status " : "device capacity overflow (status ") +
                                 std::to_string(status) + ")");
    }
}

template <class R> void World<R>::solve(int mode) {
    prepare_tail(R_);
    solve_enqueue(mode);
    PE_CK(cudaGetLastError());
    finish();
}

// What a captured step graph holds fixed: buffer addresses (any reallocation changes the
// generation), sizes and capacities, the side-stream plan, the parameters and the settings.
// (Filled in place and compared bytewise: padding is zeroed here and copied with memcpy.)
template <class R> void World<R>::graph_sig(GraphSig& g) const {
    std::memset(&g, 0, sizeof g);
    g.gen = dbuf_generation().load();
    g.order = order_;
    g.n = N_; g.ns = NS_; g.pair_cap = pair_cap_; g.nj = n_joints_; g.n_ign = n_ign_; g.s = S_;
    g.classes = possible_classes();
    g.self = self_;
    g.bcap = bcap_;
    g.max_scene = max_scene_;   // which sort the scenes take, and whether windows are swept in chunks
    std::memcpy(g.plan, stream_of_, sizeof g.plan);
    std::memcpy(&g.prm, &prm_, sizeof prm_);
    std::memcpy(&g.margin, &margin_, sizeof margin_);
    std::memcpy(&g.tun, &tun_, sizeof tun_);
    g.tun.color_block = g.tun.level_block = 0;   // no kernel reads them
}

// Replays `ex` if its signature `held` matches `sig`, else captures `enqueue` into it (updating the
// executable graph in place when the topology allows) once a step repeats its predecessor's
// signature `last`; until then `enqueue` launches directly.  Keeps the step's launch count.
template <class R>
template <class F>
void World<R>::graph_run(cudaGraphExec_t& ex, GraphSig& held, long long& held_launches, GraphSig& last, const GraphSig& sig, F&& enqueue) {
    const bool same_as_last = std::memcmp(&sig, &last, sizeof sig) == 0;
    std::memcpy(&last, &sig, sizeof sig);
    if (!ex || std::memcmp(&sig, &held, sizeof sig) != 0) {
        // a world that changes every step (a serving loop admitting and retiring scenes) would pay
        // a capture per step: capture only once the step has repeated its predecessor's settings
        if (!same_as_last) { enqueue(); return; }
        const long long before = step_launches_;
        cudaGraph_t g = nullptr;
        PE_CK(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
        capturing_ = true;
        try {
            enqueue();
        } catch (...) {
            capturing_ = false;
            cur_ = nullptr;
            cudaStreamEndCapture(st_, &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        capturing_ = false;
        PE_CK(cudaStreamEndCapture(st_, &g));
        cudaError_t e = cudaErrorUnknown;
        if (ex) {   // same topology (the usual case after a reallocation): update the executable graph in place
            cudaGraphExecUpdateResultInfo info;
            e = cudaGraphExecUpdate(ex, g, &info);
            if (e != cudaSuccess) {
                (void)cudaGetLastError();
                cudaGraphExecDestroy(ex);
                ex = nullptr;
            }
        }
        if (!ex) e = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) { ex = nullptr; PE_CK(e); }
        std::memcpy(&held, &sig, sizeof sig);
        held_launches = step_launches_ - before;
        step_launches_ = before;
    }
    PE_CK(cudaGraphLaunch(ex, st_));
    step_launches_ += held_launches;
}

// The step's head (integration and the broadphase up to the pair count's copy to the host) as one
// CUDA graph; the host then waits for the count.
template <class R> void World<R>::run_head() {
    auto enqueue = [&]() {
        ev_begin(4);
        ev_begin(0); integrate(); ev_end(0);
        ev_begin(1);
        bp_count_enqueue();
    };
    if (!graphs_ || prof_) { enqueue(); return; }
    GraphSig sig;
    graph_sig(sig);
    graph_run(ghead_, gsig_head_, glaunch_head_, last_sig_head_, sig, enqueue);
}

// The step's device part after the pair count (pair list, narrowphase, solver): launched directly,
// or captured once as a CUDA graph per solver mode and contact-distance generation and replayed
// while nothing it holds fixed has changed.  The side-stream plan follows the last step's class
// counts; it is revised every 64 steps (a changed plan is a new capture).
template <class R> void World<R>::run_tail(int mode) {
    auto enqueue = [&]() {
        bp_tail();
        bp_axis_begin();
        ev_end(1);
        ev_begin(2); np_enqueue(); ev_end(2);
        ev_begin(3); solve_enqueue(mode); ev_end(3);
        bp_axis_end();
        ev_end(4);
    };
    bool counted = false;
    for (int c = 0; c < PC_COUNT; c++) counted |= h_cls_[c] > 0;
    if (!graphs_ || prof_ || !counted) {   // no graph (or no class counts yet for the plan)
        plan_streams(stream_of_);
        enqueue();
        return;
    }
    const int m = mode ? 1 : 0, d = cur_dist_;
    if (!gexec_[m][d] || ++steps_since_plan_ >= 64) {
        steps_since_plan_ = 0;
        plan_streams(stream_of_);
    }
    GraphSig sig;
    graph_sig(sig);
    graph_run(gexec_[m][d], gsig_[m][d], glaunch_[m][d], last_sig_, sig, enqueue);
}

template <class R> void World<R>::step(int n, int mode) {
    for (int s = 0; s < n; s++) {
        step_launches_ = 0;
        run_head();
        PE_CK(cudaStreamSynchronize(st_));   // the first host wait: the pair count
        const int P = N_ < 2 ? P_ : hstat_[HS_P];
        prepare_tail(P);
        P_ = P;
        if (N_ >= 2) self_pairs_ = false;
        self_ = self_pairs_;
        cur_dist_ ^= 1;
        run_tail(mode);
        R_ = P;
        finish();                   // the second
        ev_collect();
        last_step_launches_ = step_launches_;
    }
    resolve_prof();
}

} // namespace pe
