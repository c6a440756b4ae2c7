// Many LPs packed block-diagonally, each on a thread-block cluster of its own (cluster.cuh): which
// instances go to clusters of which size.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "cluster.cuh"

namespace vajra {
namespace {

// The packed matrices as the clusters read them.
template <typename T>
struct BMats {
    const int64_t* a_ptr; const int32_t* a_idx; const T* a_val;
    const int64_t* at_ptr; const int32_t* at_idx; const T* at_val;
    int group_a, group_at;
    int64_t long_a, long_at;
};
// Instance `inst` of them, by thread 0.
template <typename T>
__device__ __forceinline__ void bmats_of(const BMats<T>& M, const int64_t* roff, const int64_t* coff, int inst, ClMats<T>& out) {
    const int r0 = static_cast<int>(roff[inst]), c0 = static_cast<int>(coff[inst]);
    out.a = ClMat<T>{static_cast<int>(roff[inst + 1]) - r0, M.a_ptr + r0, M.a_idx, M.a_val, c0, M.group_a, M.long_a};
    out.at = ClMat<T>{static_cast<int>(coff[inst + 1]) - c0, M.at_ptr + c0, M.at_idx, M.at_val, r0, M.group_at, M.long_at};
}

// nofit[insts[q]] = 1 where the slices of cluster q do not fit its CTAs.
template <typename T, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1)
k_cluster_fit(const __grid_constant__ BMats<T> M, const int* __restrict__ insts, const int64_t* __restrict__ roff,
              const int64_t* __restrict__ coff, int* __restrict__ nofit, ClLaunch L) {
    __shared__ ClInfo I;
    __shared__ ClMats<T> mats;
    const int inst = insts[blockIdx.x / cl_size()];
    if (threadIdx.x == 0) bmats_of(M, roff, coff, inst, mats);
    __syncthreads();
    ClCore<T, T> core;
    if (!core.begin(mats.a, mats.at, L, I) && threadIdx.x == 0) nofit[inst] = 1;
}

// The instances that run on clusters, by cluster size and threads.
struct ClusterClass {
    int ctas = 0, threads = 0, first = 0, clusters = 0;   // its part of the instance list
    size_t smem = 0;
};
struct ClusterBatch {
    std::vector<int> least;              // per instance: CTAs of its smallest cluster, 0: it has none
    std::vector<int> most;               // per instance: CTAs of the widest that may hold it (set by the first plan)
    std::vector<int> insts;              // the instances of the present plan, by class, largest first
    std::vector<ClusterClass> classes;   // widest clusters first
    DeviceBuffer<int> d_insts, d_on;     // the same list; per instance: runs on a cluster
};

// A stream for every class of a launch, forked from and joined into the caller's.
struct ClusterStreams {
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> events;
    cudaEvent_t ready = nullptr;
    size_t used = 0;
    ~ClusterStreams() {   // (a failed call may leave work on them; buffers declared before outlive it)
        for (auto& s : streams) { cudaStreamSynchronize(s); cudaStreamDestroy(s); }
        for (auto& e : events) cudaEventDestroy(e);
        if (ready) cudaEventDestroy(ready);
    }
    vajra_status create(size_t k) {
        used = k;
        if (!ready) VJ_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
        while (streams.size() < k) {
            cudaStream_t s = nullptr;
            cudaEvent_t e = nullptr;
            VJ_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
            streams.push_back(s);
            VJ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            events.push_back(e);
        }
        return VAJRA_OK;
    }
    vajra_status fork(cudaStream_t st) {
        VJ_CUDA(cudaEventRecord(ready, st));
        for (size_t q = 0; q < used; ++q) VJ_CUDA(cudaStreamWaitEvent(streams[q], ready, 0));
        return VAJRA_OK;
    }
    vajra_status join(cudaStream_t st) {
        for (size_t q = 0; q < used; ++q) {
            VJ_CUDA(cudaEventRecord(events[q], streams[q]));
            VJ_CUDA(cudaStreamWaitEvent(st, events[q], 0));
        }
        return VAJRA_OK;
    }
};

template <typename T>
auto fit_kernel(int threads) -> decltype(&k_cluster_fit<T, 256>) {
    return threads == 256 ? &k_cluster_fit<T, 256> : &k_cluster_fit<T, 512>;
}

// The smallest cluster that holds an instance takes the least of the GPU, since an exchange costs
// no less with more CTAs: 256 threads on one CTA, else CTAs of 512 with at most 4,096 entries of each
// matrix.  `from`: CTAs it has at least.
template <typename T>
int least_cluster(const vajra_lp& L, int group_a, int group_at, int from) {
    auto fits = [&](int c, int t) { return cl_fits(sizeof(T), L.num_rows, L.num_cols, L.nnz, group_a, group_at, c, t); };
    for (int c = from; c <= kClMaxCtas; c *= 2)
        if (fits(c, 512) && (L.nnz <= 4096 * static_cast<int64_t>(c) || c == kClMaxCtas)) return c;
    return 0;
}

// CTAs of the cluster of every instance with open[i] != 0, 0: none.  A plan that leaves half of the SMs
// idle gets clusters of twice the size, as far as their CTAs keep 512 entries.
template <typename T>
std::vector<int> size_clusters(const vajra_lp* lps, int count, const std::vector<int>& open, int group_a, int group_at, ClusterBatch& out) {
    out.most.resize(count, kClMaxCtas);
    std::vector<int> ctas(count);
    int64_t sms_used = 0;
    for (int i = 0; i < count; ++i) {
        ctas[i] = open[i] ? out.least[i] : 0;
        sms_used += ctas[i];
    }
    while (sms_used > 0 && 2 * sms_used <= sm_count()) {
        int64_t used = 0;
        for (int i = 0; i < count; ++i) {
            if (ctas[i] > 0 && ctas[i] < out.most[i] && lps[i].nnz > 1024 * static_cast<int64_t>(ctas[i]) &&
                cl_fits(sizeof(T), lps[i].num_rows, lps[i].num_cols, lps[i].nnz, group_a, group_at, 2 * ctas[i], 512))
                ctas[i] *= 2;
            used += ctas[i];
        }
        if (used == sms_used) break;
        sms_used = used;
    }
    return ctas;
}

// Whether clusters are the faster way for a plan is estimated from measured rates (B200; batches of 1 to 1,024
// equal LPs of 60 to 3,000 rows, 20 entries a row; us an iteration, checks included).  A cluster on 1, 4, 8,
// 16 CTAs of 4,000, 3,000, 2,500, 2,500 entries: 3.8, 4.5, 4.3, 5.3 in FP64, 2.3, 2.9, 2.7, 3.2 in
// FP32; the device holds 148, about 34, 15 and 7 of them, and more of them come one after another.  An
// entry costs a full device 7, 11.5, 15, 20 ps so (FP32: 4, 7.5, 10, 12), the packed iteration 9
// over windows, 9.5 to 12 in lane groups (6.5) beside its 5 to 8 us of launches.
inline double cluster_us(size_t t, int ctas, int64_t nnz) {
    const double entries = static_cast<double>(nnz) / ctas;
    const double step = ctas == 1 ? 0.1 : ctas <= 4 ? 1.65 : ctas == 8 ? 1.9 : 2.95;
    return t == 8 ? step + 0.95e-3 * entries : (ctas == 1 ? 0.1 : 0.7 * step) + 0.54e-3 * entries;
}
struct ClusterLoad {
    double us = 0.0;        // an iteration of all clusters
    double at_once = 0.0;   // the share of the device that they take together, 1: all of it
    int64_t entries = 0, outside = 0;   // of open instances on clusters, and of the others
};
inline ClusterLoad cluster_load(size_t t, const vajra_lp* lps, const std::vector<int>& open, const std::vector<int>& ctas) {
    ClusterLoad L;
    double sum = 0.0, longest = 0.0, widths[5] = {0, 0, 0, 0, 0}, counts[5] = {0, 0, 0, 0, 0}, sums[5] = {0, 0, 0, 0, 0};
    for (size_t i = 0; i < ctas.size(); ++i) {
        if (!open[i]) continue;
        if (!ctas[i]) { L.outside += lps[i].nnz; continue; }
        int k = 0;
        while ((1 << k) < ctas[i]) ++k;
        widths[k] = k == 0 ? sm_count() : std::max(1.0, std::floor(0.82 * sm_count() / ctas[i]));   // clusters the device holds
        const double us = cluster_us(t, ctas[i], lps[i].nnz);
        L.entries += lps[i].nnz;
        L.at_once += 1.0 / widths[k];
        sum += us / widths[k];
        longest = std::max(longest, us);
        counts[k] += 1.0;
        sums[k] += us;
    }
    if (L.at_once <= 1.0) { L.us = longest; return L; }
    L.us = sum + 0.5 * longest;
    for (int k = 0; k < 5; ++k)   // equal clusters leave their last round half empty
        if (counts[k] > 0.0) L.us = std::max(L.us, std::ceil(counts[k] / widths[k]) * sums[k] / counts[k]);
    return L;
}

// Plans the instances with open[i] != 0 for a launch, if `pays` says so of the clusters' load.  `prepare`: what a
// class's launch needs (an error: there is no such cluster on this device).
template <typename T, class Pays, class Prepare>
vajra_status plan_clusters(const vajra_lp* lps, int count, const std::vector<int>& open, const BMats<T>& M, const int64_t* roff,
                           const int64_t* coff, ClusterBatch& out, Pays pays, Prepare prepare, cudaStream_t st) {
    DeviceBuffer<int> nofit;
    VJ_TRY(nofit.alloc(count));
    VJ_TRY(out.d_insts.alloc(count));
    VJ_TRY(out.d_on.alloc(count));
    std::vector<int> threads(count), on(count), h(count);
    auto fits = [&](int i, int c, int t) {
        return cl_fits(sizeof(T), lps[i].num_rows, lps[i].num_cols, lps[i].nnz, M.group_a, M.group_at, c, t);
    };
    for (bool again = true; again;) {
        again = false;
        std::vector<int> ctas = size_clusters<T>(lps, count, open, M.group_a, M.group_at, out);
        if (!pays(cluster_load(sizeof(T), lps, open, ctas))) ctas.assign(count, 0);
        for (int i = 0; i < count; ++i)
            threads[i] = ctas[i] && fits(i, ctas[i], 256) && lps[i].nnz <= 2048 * static_cast<int64_t>(ctas[i]) ? 256 : 512;
        out.classes.clear();
        out.insts.clear();
        for (int c = kClMaxCtas; c >= 1; c /= 2)
            for (int t : {512, 256}) {
                ClusterClass k;
                k.ctas = c;
                k.threads = t;
                k.first = static_cast<int>(out.insts.size());
                size_t most = 0;
                for (int i = 0; i < count; ++i)
                    if (ctas[i] == c && threads[i] == t) {
                        out.insts.push_back(i);
                        most = std::max(most, cl_smem_bytes(sizeof(T), sizeof(T), lps[i].num_rows, lps[i].num_cols, lps[i].nnz, c, t));
                    }
                k.clusters = static_cast<int>(out.insts.size()) - k.first;
                if (!k.clusters) continue;
                std::stable_sort(out.insts.begin() + k.first, out.insts.end(), [&](int x, int y) { return lps[x].nnz > lps[y].nnz; });
                // two CTAs of 256 threads fit an SM when each takes half of its shared memory
                k.smem = t == 256 && most <= kClSmemCap / 2 - 4096 ? kClSmemCap / 2 - 4096 : kClSmemCap;
                out.classes.push_back(k);
            }
        if (out.insts.empty()) break;
        // Uneven rows may not fit after all, or the device may lack such a cluster.  An instance on more
        // CTAs than it needs then goes back to half of them for good; one on its smallest cluster gets a
        // wider one where its rows are uneven, at last none.
        auto refuse = [&](int i, bool uneven) {
            if (ctas[i] > out.least[i]) out.most[i] = ctas[i] / 2;
            else out.least[i] = uneven ? least_cluster<T>(lps[i], M.group_a, M.group_at, 2 * ctas[i]) : 0;
            again = true;
        };
        VJ_CUDA(cudaMemcpyAsync(out.d_insts.get(), out.insts.data(), sizeof(int) * out.insts.size(), cudaMemcpyHostToDevice, st));
        VJ_CUDA(cudaMemsetAsync(nofit.get(), 0, sizeof(int) * count, st));
        for (const ClusterClass& k : out.classes) {
            cudaError_t e = prepare(k);
            if (e == cudaSuccess) e = prepare_clusters(fit_kernel<T>(k.threads), k.ctas, k.threads, k.smem);
            if (e != cudaSuccess) {   // no such cluster on this device
                cudaGetLastError();
                for (int q = k.first; q < k.first + k.clusters; ++q) refuse(out.insts[q], false);
                continue;
            }
            VJ_CUDA(launch_clusters(fit_kernel<T>(k.threads), k.clusters, k.ctas, k.threads, k.smem, st, M, out.d_insts.get() + k.first,
                                    roff, coff, nofit.get(), cl_launch(k.smem)));
        }
        VJ_CUDA(cudaMemcpyAsync(h.data(), nofit.get(), sizeof(int) * count, cudaMemcpyDeviceToHost, st));
        VJ_CUDA(cudaStreamSynchronize(st));
        for (int q : out.insts)
            if (h[q]) refuse(q, true);
    }
    for (int q : out.insts) on[q] = 1;
    VJ_CUDA(cudaMemcpyAsync(out.d_on.get(), on.data(), sizeof(int) * count, cudaMemcpyHostToDevice, st));
    VJ_CUDA(cudaStreamSynchronize(st));   // host vectors above
    return VAJRA_OK;
}

}  // namespace
}  // namespace vajra
