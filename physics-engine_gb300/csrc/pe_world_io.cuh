// World<R> member definitions, part 3: transfers between the caller's arrays and the device
// (body state, sweep axes, pairs, contact results).
#pragma once
#include <cuda.h>
#include "pe_world_step.cuh"

namespace pe {

// ------------------------------------------------------------------ transfers
// The body state is converted on the device (k_state_pack / k_state_unpack), in place in page-locked arrays
// of up to kDirectBytes and through a device staging buffer otherwise: in place one launch does what
// took a copy per array too; pairs copy straight into the caller's
// array, contact results through host vectors (their layout changes on the host), and the serving
// reads of finished scenes through pinned host memory (staging).  These are the host<->device copies
// a drop-in caller pays.
template <class R> R* World<R>::staging(size_t n) {
    if (n > stage_n_) {
        if (stage_) cudaFreeHost(stage_);
        stage_ = nullptr;
        PE_CK(cudaMallocHost(&stage_, n * sizeof(R)));
        stage_n_ = n;
    }
    return stage_;
}

// The allocation or registration that a device address lies in; false where there is none.
static bool pinned_range(const void* p, unsigned long long& start, size_t& size) {
    using Query = CUresult(CUDAAPI*)(void*, CUpointer_attribute, CUdeviceptr);
    static const Query query = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Query>(f);
    }();
    const CUdeviceptr d = reinterpret_cast<CUdeviceptr>(p);
    return query && query(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, d) == CUDA_SUCCESS &&
           query(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, d) == CUDA_SUCCESS;
}

// The device's address of a caller's array of `bytes` bytes that kernels may use in place: page-locked
// memory from end to end (one allocation or registration holds it all: between two lies memory that no
// kernel may touch), aligned for its values.  nullptr: it goes through the staging buffer.
static void* direct_address(const void* p, size_t bytes, size_t align) {
    if (bytes == 0 || bytes > kDirectBytes || reinterpret_cast<uintptr_t>(p) % align != 0) return nullptr;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    unsigned long long start = 0;
    size_t size = 0;
    if (at.type != cudaMemoryTypeHost || !at.devicePointer || !pinned_range(at.devicePointer, start, size) ||
        !range_holds(start, size, reinterpret_cast<unsigned long long>(at.devicePointer), bytes))
        return nullptr;
    return at.devicePointer;
}

// The groups of the arrays given (null: left out), each in place or in the staging buffer: src[g] is the
// caller's array of a staged group, its bytes size[g].
template <class R> template <class T>
typename World<R>::template Xfer<T> World<R>::xfer_groups(T* const* arrays) {
    static const int k0[7] = {OX, B00, VX, WX, MNX, MXX, I00}, nk[7] = {3, 9, 3, 3, 3, 3, 9};
    Xfer<T> x;
    size_t tot = 0, off[7];
    for (int g = 0; g < 7; g++) {
        if (!arrays[g]) continue;
        const int n = x.G.n++;
        x.at[g] = n;
        x.G.k0[n] = k0[g]; x.G.nk[n] = nk[g];
        x.size[n] = (size_t)nk[g] * N_ * sizeof(T);
        x.G.ptr[n] = static_cast<T*>(direct_address(arrays[g], x.size[n], sizeof(T)));
        x.staged[n] = x.G.ptr[n] ? nullptr : arrays[g];
        off[n] = tot;
        if (x.staged[n]) tot += (size_t)nk[g] * N_;
        x.widest = std::max(x.widest, nk[g]);
    }
    if (tot) xfer_.ensure((tot * sizeof(T) + sizeof(double) - 1) / sizeof(double));
    for (int n = 0; n < x.G.n; n++)
        if (x.staged[n]) x.G.ptr[n] = reinterpret_cast<T*>(xfer_.p) + off[n];
    return x;
}

template <class R> template <class T>
void World<R>::get_state_t(T* o, T* b, T* v, T* w, T* mn, T* mx, T* iw) {
    T* const dst[7] = {o, b, v, w, mn, mx, iw};
    if (!N_) return;
    const Xfer<T> x = xfer_groups(dst);
    if (!x.G.n) return;
    launch(K_MISC, dim3(grid(N_ * (long long)x.widest), x.G.n), k_state_pack<R, T>, bodies(), x.G);
    for (int n = 0; n < x.G.n; n++)
        if (x.staged[n]) PE_CK(cudaMemcpyAsync(x.staged[n], x.G.ptr[n], x.size[n], cudaMemcpyDeviceToHost, st_));
    PE_CK(cudaStreamSynchronize(st_));
}

template <class R> template <class T>
void World<R>::set_state_t(const T* o, const T* b, const T* v, const T* w, const T* mn, const T* mx, const T* iw) {
    T* const src[7] = {const_cast<T*>(o), const_cast<T*>(b), const_cast<T*>(v), const_cast<T*>(w), const_cast<T*>(mn),
                       const_cast<T*>(mx), const_cast<T*>(iw)};   // only read
    if (!N_) return;
    const Xfer<T> x = xfer_groups(src);
    if (!x.G.n) return;
    for (int n = 0; n < x.G.n; n++)
        if (x.staged[n]) PE_CK(cudaMemcpyAsync(x.G.ptr[n], x.staged[n], x.size[n], cudaMemcpyHostToDevice, st_));
    const bool scale = mn && mx && o;   // the injected box's AABB scale
    launch(K_MISC, dim3(grid(N_ * (long long)x.widest), x.G.n), k_state_unpack<R, T>, bodies(), x.G, scale ? x.at[0] : -1,
           scale ? x.at[4] : -1, scale ? x.at[5] : -1);
    PE_CK(cudaStreamSynchronize(st_));
}

template <class R> void World<R>::get_axes(int* a) {
    PE_CK(cudaMemcpyAsync(a, scene_axis_.p, NS_ * sizeof(int), cudaMemcpyDeviceToHost, st_));
    PE_CK(cudaStreamSynchronize(st_));
}
template <class R> void World<R>::set_axes(const int* a) {
    PE_CK(cudaMemcpyAsync(scene_axis_.p, a, NS_ * sizeof(int), cudaMemcpyHostToDevice, st_));
    PE_CK(cudaStreamSynchronize(st_));
}

template <class R> void World<R>::get_pairs(int* p) {
    if (P_) PE_CK(cudaMemcpyAsync(p, pairs_.p, (size_t)P_ * sizeof(int2), cudaMemcpyDeviceToHost, st_));
    PE_CK(cudaStreamSynchronize(st_));
}

// per-scene offsets of a list grouped by scene (scene of its first body)
static std::vector<int> scene_offsets(int n, const int* a, const std::vector<int>& scene_off) {
    const int ns = (int)scene_off.size() - 1;
    std::vector<int> off(ns + 1, 0);
    int s = 0;
    for (int i = 0; i < n; i++) {
        const int b = a[i * 2];
        const int sb = (int)(std::upper_bound(scene_off.begin(), scene_off.end(), b) - scene_off.begin()) - 1;
        if (sb < s) throw std::runtime_error("list must be grouped by scene in scene order");
        while (s < sb) off[++s] = i;
    }
    while (s < ns) off[++s] = n;
    return off;
}

template <class R> void World<R>::set_pairs(int n, const int* p) {
    for (int i = 0; i < 2 * n; i++) if (p[i] < 0 || p[i] >= N_) throw std::runtime_error("pair body index out of range");
    ensure_pair_capacity(std::max(n, 1));
    self_pairs_ = false;
    for (int i = 0; i < n; i++) self_pairs_ = self_pairs_ || p[2 * i] == p[2 * i + 1];
    if (n) PE_CK(cudaMemcpyAsync(pairs_.p, p, (size_t)n * sizeof(int2), cudaMemcpyHostToDevice, st_));
    h_pair_scene_off_ = scene_offsets(n, p, h_scene_off_);
    PE_CK(cudaMemcpyAsync(pair_scene_off_.p, h_pair_scene_off_.data(), (NS_ + 1) * sizeof(int), cudaMemcpyHostToDevice, st_));
    PE_CK(cudaMemcpyAsync(dcnt_.p + DC_P, &n, sizeof(int), cudaMemcpyHostToDevice, st_));
    PE_CK(cudaStreamSynchronize(st_));
    P_ = n;
}

template <class R> void World<R>::get_results(int* a, int* b, int* ps, double* fr, double* re, double* slots) {
    const int P = R_;
    std::vector<int> ha(P), hb(P), hn(P);
    std::vector<R> hfr(P), hre(P), hd((size_t)P * kSlots), pts((size_t)NPF * pair_cap_ * kSlots);
    if (P) {
        PE_CK(cudaMemcpyAsync(ha.data(), res_a_.p, P * sizeof(int), cudaMemcpyDeviceToHost, st_));
        PE_CK(cudaMemcpyAsync(hb.data(), res_b_.p, P * sizeof(int), cudaMemcpyDeviceToHost, st_));
        PE_CK(cudaMemcpyAsync(hn.data(), res_np_.p, P * sizeof(int), cudaMemcpyDeviceToHost, st_));
        PE_CK(cudaMemcpyAsync(hfr.data(), res_fr_.p, P * sizeof(R), cudaMemcpyDeviceToHost, st_));
        PE_CK(cudaMemcpyAsync(hre.data(), res_re_.p, P * sizeof(R), cudaMemcpyDeviceToHost, st_));
        PE_CK(cudaMemcpyAsync(hd.data(), res_dist_[cur_dist_].p, hd.size() * sizeof(R), cudaMemcpyDeviceToHost, st_));
        PE_CK(cudaMemcpyAsync(pts.data(), res_pts_.p, pts.size() * sizeof(R), cudaMemcpyDeviceToHost, st_));
    }
    PE_CK(cudaStreamSynchronize(st_));
    const size_t stride = (size_t)pair_cap_ * kSlots;
    for (int p = 0; p < P; p++) {
        if (a) a[p] = ha[p];
        if (b) b[p] = hb[p];
        if (ps) ps[p] = hn[p];
        if (fr) fr[p] = hfr[p];
        if (re) re[p] = hre[p];
        if (!slots) continue;
        for (int k = 0; k < kSlots; k++) {
            double* o = slots + ((size_t)p * kSlots + k) * 19;
            for (int q = 0; q < 19; q++) o[q] = 0;
            o[12] = hd[(size_t)p * kSlots + k];
            if (k >= hn[p]) continue;
            const size_t s = (size_t)p * kSlots + k;
            for (int g = 0; g < 4; g++) for (int d = 0; d < 3; d++) o[g * 3 + d] = pts[(size_t)(g * 3 + d) * stride + s];
            for (int g = 4; g < 6; g++) for (int d = 0; d < 3; d++) o[13 + (g - 4) * 3 + d] = pts[(size_t)(g * 3 + d) * stride + s];
        }
    }
}

template <class R>
void World<R>::set_results(int n, const int* a, const int* b, const int* ps, const double* fr, const double* re,
                           const double* slots) {
    ensure_pair_capacity(std::max(n, 1));
    std::vector<int> ab(2 * n);
    for (int i = 0; i < n; i++) {
        if (a[i] < 0 || a[i] >= N_ || b[i] < 0 || b[i] >= N_ || ps[i] < 0 || ps[i] > kSlots)
            throw std::runtime_error("result " + std::to_string(i) + " out of range");
        ab[2 * i] = a[i];
        ab[2 * i + 1] = b[i];
    }
    std::vector<int> off = scene_offsets(n, ab.data(), h_scene_off_);
    std::vector<R> hfr(n), hre(n), hd((size_t)n * kSlots), pts((size_t)NPF * pair_cap_ * kSlots, R(0));
    const size_t stride = (size_t)pair_cap_ * kSlots;
    for (int p = 0; p < n; p++) {
        hfr[p] = R(fr[p]);
        hre[p] = R(re[p]);
        for (int k = 0; k < kSlots; k++) {
            const double* o = slots + ((size_t)p * kSlots + k) * 19;
            const size_t s = (size_t)p * kSlots + k;
            hd[s] = R(o[12]);
            for (int g = 0; g < 4; g++) for (int d = 0; d < 3; d++) pts[(size_t)(g * 3 + d) * stride + s] = R(o[g * 3 + d]);
            for (int g = 4; g < 6; g++) for (int d = 0; d < 3; d++) pts[(size_t)(g * 3 + d) * stride + s] = R(o[13 + (g - 4) * 3 + d]);
        }
    }
    if (n) {
        PE_CK(cudaMemcpyAsync(res_a_.p, a, n * sizeof(int), cudaMemcpyHostToDevice, st_));
        PE_CK(cudaMemcpyAsync(res_b_.p, b, n * sizeof(int), cudaMemcpyHostToDevice, st_));
        PE_CK(cudaMemcpyAsync(res_np_.p, ps, n * sizeof(int), cudaMemcpyHostToDevice, st_));
        PE_CK(cudaMemcpyAsync(res_fr_.p, hfr.data(), n * sizeof(R), cudaMemcpyHostToDevice, st_));
        PE_CK(cudaMemcpyAsync(res_re_.p, hre.data(), n * sizeof(R), cudaMemcpyHostToDevice, st_));
        PE_CK(cudaMemcpyAsync(res_dist_[cur_dist_].p, hd.data(), hd.size() * sizeof(R), cudaMemcpyHostToDevice, st_));
        PE_CK(cudaMemcpyAsync(res_pts_.p, pts.data(), pts.size() * sizeof(R), cudaMemcpyHostToDevice, st_));
    }
    PE_CK(cudaMemcpyAsync(res_scene_off_.p, off.data(), (NS_ + 1) * sizeof(int), cudaMemcpyHostToDevice, st_));
    PE_CK(cudaMemcpyAsync(dcnt_.p + DC_R, &n, sizeof(int), cudaMemcpyHostToDevice, st_));
    PE_CK(cudaStreamSynchronize(st_));
    R_ = n;
    self_ = false;
    for (int i = 0; i < n; i++) self_ = self_ || a[i] == b[i];
}

} // namespace pe
