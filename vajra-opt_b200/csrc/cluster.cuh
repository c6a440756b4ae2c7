// Cluster-resident PDHG iterations: one thread-block cluster (1..16 CTAs) keeps an LP in its
// shared memory and runs whole chunks of iterations in one launch.
//
// Why: on an LP of a few 10^4 entries an iteration kernel moves a few hundred KB, a
// microsecond of work, and two launches an iteration cost 5.5 to 6.8 us whatever they do.  Here the
// iterates never leave shared memory, and the only thing an iteration waits for is the
// exchange of x_bar and of y between the CTAs.
//
// Layout.  CTA r of the cluster owns a slice of the columns and a slice of the rows (contiguous,
// cut at equal shares of entries + 16 per row, at multiples of four so that slices are 16-byte
// aligned): a thread owns at most one of each and keeps its vectors in registers.  Shared memory
// holds both matrices' entries of the slices and full copies of x_bar and y, from which the row
// sums gather.
// Exchange.  After each half-iteration a CTA sends its slice of the new vector to every other
// CTA with one bulk copy each (cp.async.bulk, shared memory to shared memory), which signals the
// receiver's mbarrier; a CTA goes on when all slices have arrived.  That is the only barrier of
// a half-iteration.  Measured for 8 CTAs of 512 threads (B200): 0.62 us for 2 KB, 0.64 us for
// 8 KB, 0.95 us for 20 KB; plain remote stores and a cluster barrier took 0.88 to 1.33 us, a copy
// through L2 1.3 to 1.5 us.
// Why no buffer is written early: x_bar and y alternate.  A CTA overwrites a peer's copy of x_bar
// only after it has received that peer's y of the iteration before, which the peer sends after
// its last read of x_bar; the same with the names exchanged.
// Why each vector has its own mbarrier: a CTA that runs ahead sends at most one exchange ahead,
// and that one goes to the other mbarrier, so bytes are never counted in the wrong phase.
// Where a wait runs out, that thread waits, sends and arms no more (a second arrival could fall into a
// phase that is not complete).  A CTA that no longer arms its mbarriers runs out in its other threads,
// one that no longer sends makes its peers run out; each of them is at most one exchange ahead, so no
// mbarrier sees a phase's arrivals twice.  Everybody goes through the remaining steps on garbage, but in
// bounds and with the same decisions, and the kernel reports it.  At the end (ClCore::leave) the cluster then
// stays for the copies still on their way, so that none outlives a CTA.
// Row sums are formed exactly as the grouped-lane kernel forms them (G lanes a row, strided,
// butterfly; rows longer than long_len by 256 threads), so results have the same bits.
#pragma once

#include "common.cuh"
#include "halpern_state.cuh"
#include "spmv.cuh"

namespace vajra {

constexpr int kClThreads = 512;                // most threads of a CTA
constexpr int kClMaxChains = 8;                // chains of a row that one thread may form
constexpr int kClMaxLong = 16;                 // rows summed by 256 threads that a CTA may have
constexpr int kClMaxCtas = 16;
constexpr int kClRowWeight = 16;               // a row's share of the work beside its entries
constexpr size_t kClSmemCap = 216 * 1024;      // dynamic shared memory a CTA may ask for
constexpr int kClWaitTries = 1 << 20;          // bound of every mbarrier wait, unless the environment sets it
constexpr int kClDrainNaps = 2000;             // half microseconds that a failed cluster stays at its end

// Tries of an mbarrier wait: kClWaitTries, or VAJRA_CLUSTER_WAIT_TRIES (read once).
int cluster_wait_tries();

// What a launch tells the kernel of its set-up.
struct ClLaunch {
    uint32_t smem_bytes;
    int wait_tries;
};
inline ClLaunch cl_launch(size_t smem) { return {static_cast<uint32_t>(smem), cluster_wait_tries()}; }

// One matrix of the LP: rows `rows`, indices minus idx_base are local.
template <typename V>
struct ClMat {
    int rows;
    const int64_t* ptr;
    const int32_t* idx;
    const V* val;
    int idx_base;
    int group;          // lanes per row: 1, 2, 4, .. 32
    int64_t long_len;   // rows longer than this are summed by 256 threads
};

__device__ __forceinline__ uint32_t cl_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cl_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// All threads of the cluster; global and shared writes before it are visible after it.
__device__ __forceinline__ void cl_barrier() {
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_map(uint32_t addr, uint32_t rank) {
    uint32_t o;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(addr), "r"(rank));
    return o;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// First row of slice `r` of `parts`: the smallest multiple of four whose rows before it carry
// at least r / parts of the weight (entries + kClRowWeight a row).
__host__ __device__ inline int cl_bound(int rows, const int64_t* ptr, int r, int parts) {
    if (r <= 0) return 0;
    if (r >= parts) return rows;
    const int64_t p0 = ptr[0];
    const int64_t total = ptr[rows] - p0 + static_cast<int64_t>(kClRowWeight) * rows;
    const int64_t target = total * r / parts;
    int lo = 0, hi = (rows + 3) / 4;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        const int j = 4 * mid < rows ? 4 * mid : rows;
        if (ptr[j] - p0 + static_cast<int64_t>(kClRowWeight) * j < target) lo = mid + 1; else hi = mid;
    }
    return 4 * lo < rows ? 4 * lo : rows;
}
inline int64_t pad4(int64_t v) { return (v + 3) / 4 * 4; }

// Shared memory of a CTA: the two full vectors, the larger scratch of dealing a slice, and both
// slices' entries (an equal share of `value` bytes and a 4-byte place each, a half more for
// padding, at least a pair a thread).
inline size_t cl_smem_bytes(size_t t, size_t value, int64_t m, int64_t n, int64_t nnz, int parts, int threads) {
    const size_t share = static_cast<size_t>(nnz + nnz / 2) / parts + 2 * threads;
    return t * (pad4(n + 1) + pad4(m + 1)) + 2 * share * (value + 4) + 8 * threads + 24 * kClMaxLong + 1024;
}

// Whether an LP should fit a cluster of `ctas` CTAs: indices of 16 bits, lane-group row sums, at
// most `threads` rows and columns and kClMaxChains chains a thread in every CTA, and the entries in
// shared memory.  From equal shares and a tenth: a CTA that gets more says so when it deals its
// slices.
inline bool cl_fits(size_t t, int64_t m, int64_t n, int64_t nnz, int group_a, int group_at, int ctas, int threads) {
    if (group_a < 1 || group_a > 32 || group_at < 1 || group_at > 32 || m >= 65535 || n >= 65535) return false;
    const int64_t most = std::max(m, n);
    if (ctas == 1 ? most > threads : (most + most / 10) / ctas + 8 > threads) return false;
    if (std::max(m / ctas * group_a, n / ctas * group_at) / threads >= kClMaxChains) return false;
    return cl_smem_bytes(t, t, m, n, nnz, ctas, threads) <= kClSmemCap;
}

// The dynamic shared memory of a cluster kernel and an array in it.  Arrays are kept as offsets,
// not as pointers, so that every access compiles to a shared-memory instruction.
extern __shared__ __align__(16) unsigned char cl_smem[];
template <typename U>
struct ClArray {
    uint32_t off = 0;
    __device__ __forceinline__ U* ptr() const { return reinterpret_cast<U*>(cl_smem + off); }
    __device__ __forceinline__ U& operator[](int i) const { return ptr()[i]; }
};

// One matrix slice as the iterations read it: every row of the slice has its own threads, so a
// CTA has at most blockDim.x rows and columns, and everything an iteration needs of a row is in
// its owner's registers.
// The grouped-lane kernel gives a row G chains of products (entry k to chain k mod G) and adds
// the chains in a butterfly.  Here tpr (<= G) threads share a row: thread l forms the chains l,
// l + tpr, l + 2 tpr, .. in order, adds them up the butterfly as far as they go, and shuffles do
// the rest.  The rows are sorted by length and dealt to the threads in that order; the entries
// of a warp's 32 tasks lie side by side, two of a task in one load, padded with zero values that
// point at the zero behind the vector.
// (Reading the slice as CSR, with the vectors in shared memory and rounds over the rows, took
// 370 instructions a thread and iteration: with 8 to 16 warps on an SM those instructions, one
// after another, were what an iteration waited for -- 1.9 us on a 60 x 150 LP.)
struct ClSlice {                // uniform over the CTA, in shared memory
    int b0, rows;               // first row, number of rows
    int tpr_shift;              // threads per row, log2
    int n_long;                 // rows longer than long_len (summed by 256 threads), and of
    uint32_t longs;             // each its number, first entry and length
    long long e0;               // first entry
};
struct ClInfo {                 // uniform over the CTA, in shared memory
    unsigned long long bar_x, bar_y;     // mbarriers of the two exchanges
    ClSlice cols, rows;
    int m, n;
    uint32_t rank, size;
    uint32_t bytes_x, bytes_y;           // my slices of x_bar and y
    uint32_t expect_x, expect_y;         // what the peers send
    uint32_t top, end;                   // free dynamic shared memory
    int count;
    int ran_out;                         // a wait ran out somewhere in the cluster (set by `leave`)
};
// Two entries of a task: the vector entries' places in shared memory (bytes) and the values.
template <typename T> struct ClPair;
template <> struct alignas(16) ClPair<float> { uint32_t off0; float val0; uint32_t off1; float val1; };
template <> struct alignas(8) ClPair<double> { uint32_t off0, off1; double val0, val1; };
struct ClTask {                 // a thread's task of one slice
    int row;                    // its row of the slice, -1: none
    int pairs, turn;            // pairs of entries and pairs a chain (the same for all of a warp)
    uint32_t pair;              // its first pair; the next ones follow 32 pairs apart
};

// Bytes of `rows` entries of a vector, rounded up to whole groups of four (the full vectors are
// padded to multiples of four).
template <typename T>
__host__ __device__ inline uint32_t cl_bytes(int rows) { return static_cast<uint32_t>((rows + 3) / 4 * 4 * sizeof(T)); }
// Offset of the full y behind the full x_bar (which starts the dynamic shared memory); each has
// at least one zero after its end.
template <typename T>
__device__ __forceinline__ uint32_t cl_y_offset(int n) { return static_cast<uint32_t>((n / 4 * 4 + 4) * sizeof(T)); }

// Cuts the slices and sets the mbarriers up.  A cluster barrier has to follow before the first
// exchange.
template <typename T, typename V>
__device__ __noinline__ void cl_begin(const ClMat<V>& a, const ClMat<V>& at, uint32_t bytes, ClInfo& I) {
    if (threadIdx.x == 0) {
        const uint32_t rank = cl_rank(), size = cl_size();
        I.rank = rank;
        I.size = size;
        I.m = a.rows;
        I.n = at.rows;
        // arrivals of a phase: my own and one from every peer that has nothing to send
        uint32_t ax = 1, ay = 1;
        int c = 0, r = 0;
#pragma unroll 1
        for (uint32_t q = 0; q < size; ++q) {
            const int c1 = cl_bound(at.rows, at.ptr, q + 1, size), r1 = cl_bound(a.rows, a.ptr, q + 1, size);
            if (q == rank) {
                I.cols.b0 = c; I.cols.rows = c1 - c; I.cols.e0 = at.ptr[c];
                I.rows.b0 = r; I.rows.rows = r1 - r; I.rows.e0 = a.ptr[r];
            } else {
                ax += c1 == c ? 1 : 0;
                ay += r1 == r ? 1 : 0;
            }
            c = c1;
            r = r1;
        }
        I.bytes_x = cl_bytes<T>(I.cols.rows);
        I.bytes_y = cl_bytes<T>(I.rows.rows);
        I.expect_x = cl_bytes<T>(at.rows) - I.bytes_x;
        I.expect_y = cl_bytes<T>(a.rows) - I.bytes_y;
        I.top = cl_y_offset<T>(at.rows) + cl_y_offset<T>(a.rows);
        I.end = bytes;
        I.ran_out = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&I.bar_x)), "r"(ax) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&I.bar_y)), "r"(ay) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 4) {   // the zeros behind the full vectors
        const int n4 = at.rows / 4 * 4 + static_cast<int>(threadIdx.x), m4 = a.rows / 4 * 4 + static_cast<int>(threadIdx.x);
        ClArray<T>{0}[n4] = T(0);
        ClArray<T>{cl_y_offset<T>(at.rows)}[m4] = T(0);
    }
    __syncthreads();
}

// Deals the rows of slice `s` to the threads and lays their entries out; `vec`: where the
// vector they multiply starts, `zero`: the index of the zero behind it.  *ok: false when they do not fit (uniform over the CTA).
template <typename V>
__device__ __noinline__ ClTask cl_deal(const ClMat<V>& mat, ClSlice& s, uint32_t vec, int zero, ClInfo& I, bool* ok) {
    ClTask t{-1, 0, 0, 0};
    *ok = false;
    const int rows = s.rows, tid = threadIdx.x;
    const long long e0 = s.e0;
    const uint32_t base = (I.top + 15) / 16 * 16;
    ClArray<int> longs{base};
    const uint32_t mark = base + 12 * kClMaxLong;   // scratch from here on: given back below
    ClArray<int> off{mark};
    ClArray<uint16_t> perm{mark + 4u * (rows + 1)};
    ClArray<int> first_pair{(mark + 6u * (rows + 1) + 3) / 4 * 4};
    if (rows > static_cast<int>(blockDim.x) || first_pair.off + 4 * 33 > I.end) return t;
    if (tid == 0) I.count = 0;
    __syncthreads();
    for (int r = tid; r <= rows; r += blockDim.x) {
        const int64_t p = mat.ptr[s.b0 + r];
        off[r] = static_cast<int>(p - e0);
        const int64_t len = r < rows ? mat.ptr[s.b0 + r + 1] - p : 0;
        if (len > mat.long_len) {
            const int i = atomicAdd(&I.count, 1);
            if (i < kClMaxLong) {
                longs[3 * i] = r;
                longs[3 * i + 1] = static_cast<int>(p - e0);
                longs[3 * i + 2] = static_cast<int>(len);
            }
        }
    }
    __syncthreads();
    int sh = 0;
    while ((2 << sh) <= mat.group && (rows << (sh + 1)) <= static_cast<int>(blockDim.x)) ++sh;
    const int chains = mat.group >> sh, tpr = 1 << sh;
    if (I.count > kClMaxLong || chains > kClMaxChains) return t;
    auto length = [&](int r) {   // rows for the 256 threads have no tasks
        const int len = off[r + 1] - off[r];
        return len > mat.long_len ? 0 : len;
    };
    if (tid < rows) {
        const int len = length(tid);
        int before = 0;
        for (int q = 0; q < rows; ++q) {
            const int l = length(q);
            before += (l > len || (l == len && q < tid)) ? 1 : 0;
        }
        perm[before] = static_cast<uint16_t>(tid);
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    // a warp's first task is its longest; its pairs come after those of the warps before it
    auto warp_turn = [&](int w) {
        const int p = (32 * w) >> sh;
        return p < rows ? ((length(perm[p]) + mat.group - 1) / mat.group + 1) / 2 : 0;
    };
    int len = 0, first = 0;
    if ((tid >> sh) < rows) {
        t.row = perm[tid >> sh];
        len = length(t.row);
        first = off[t.row];
    }
    t.turn = warp_turn(warp);
    t.pairs = chains * t.turn;
    if (tid == 0) {
        int sum = 0;
        for (int w = 0; w < warps; ++w) { first_pair[w] = sum; sum += chains * warp_turn(w); }
        first_pair[32] = sum;
        s.tpr_shift = sh;
        s.n_long = I.count;
        s.longs = longs.off;
    }
    __syncthreads();
    const int64_t pairs = 32 * static_cast<int64_t>(first_pair[32]);
    const int slot = 32 * first_pair[warp] + lane;
    __syncthreads();   // the scratch is read
    const uint32_t pair0 = (mark + 15) / 16 * 16;
    const int64_t end = pair0 + pairs * static_cast<int64_t>(sizeof(ClPair<V>));
    if (end > static_cast<int64_t>(I.end)) return t;
    t.pair = pair0 + slot * static_cast<uint32_t>(sizeof(ClPair<V>));
    for (int u = 0; u < t.pairs; ++u) {
        uint32_t ii[2];
        V vv[2];
        int chain = 0;   // the place of u's chain, its bits reversed
        for (int q = u / t.turn, c = 1; c < chains; c *= 2, q /= 2) chain = 2 * chain + (q & 1);
        for (int h = 0; h < 2; ++h) {
            const int k = (tid & (tpr - 1)) + tpr * (chain + chains * (2 * (u % t.turn) + h));
            ii[h] = static_cast<uint32_t>(zero);
            vv[h] = V(0);
            if (k < len) {
                ii[h] = static_cast<uint32_t>(mat.idx[e0 + first + k] - mat.idx_base);
                vv[h] = mat.val[e0 + first + k];
            }
        }
        ClPair<V> e;
        e.off0 = vec + ii[0] * static_cast<uint32_t>(sizeof(V));
        e.off1 = vec + ii[1] * static_cast<uint32_t>(sizeof(V));
        e.val0 = vv[0];
        e.val1 = vv[1];
        ClArray<ClPair<V>>{t.pair}[32 * u] = e;
    }
    if (tid == 0) I.top = static_cast<uint32_t>(end);
    __syncthreads();
    *ok = true;
    return t;
}

// My chains of my row, added up the butterfly as far as they go in this thread.  The chains lie
// one after another in the order in which the butterfly pairs them up (0, C/2, C/4, 3C/4, ..), each
// `turn` pairs long; finished sums wait in s0, s1, s2 for their partners like the digits of a
// binary counter.  One form for every number of chains: a form for each, inlined twice, drove the
// iteration's registers into local memory.
// EXACT: products rounded before they are added (the reference's arithmetic); DROP: an entry whose
// vector entry is zero adds nothing, whatever its value.
template <typename T, bool EXACT = false, bool DROP = false>
__device__ __forceinline__ T cl_chains(const ClTask& t) {
    auto add = [](T a, T v, T x) -> T {
        if constexpr (!EXACT) return fma(v, x, a);
        else if constexpr (DROP) return x == T(0) ? a : rn_add(a, rn_mul(v, x));
        else return rn_add(a, rn_mul(v, x));
    };
    constexpr int P = 4;   // pairs taken together: their loads overlap
    const ClArray<ClPair<T>> ep{t.pair};
    T acc = T(0), s0 = T(0), s1 = T(0), s2 = T(0), total = T(0);
    int left = t.turn, k = 0;
#pragma unroll 1
    for (int u = 0; u < t.pairs; u += P) {
        ClPair<T> e[P];
        T xx[2 * P];
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (p == 0 || u + p < t.pairs) e[p] = ep[32 * (u + p)];
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (p == 0 || u + p < t.pairs) {
                xx[2 * p] = *reinterpret_cast<const T*>(cl_smem + e[p].off0);
                xx[2 * p + 1] = *reinterpret_cast<const T*>(cl_smem + e[p].off1);
            }
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (p == 0 || u + p < t.pairs) {
                acc = add(acc, e[p].val0, xx[2 * p]);
                acc = add(acc, e[p].val1, xx[2 * p + 1]);
                if (--left == 0) {   // a chain is done (the same for all of a warp)
                    left = t.turn;
                    total = acc;
                    if (k & 1) {
                        total = s0 + total;
                        if (k & 2) {
                            total = s1 + total;
                            if (k & 4) total = s2 + total; else s2 = total;
                        } else {
                            s1 = total;
                        }
                    } else {
                        s0 = total;
                    }
                    ++k;
                    acc = T(0);
                }
            }
    }
    return total;
}

// The rows longer than long_len, one after another, by 256 threads each, as the grouped-lane
// kernel sums them; their owners' tasks are empty.
template <typename T, typename V>
__device__ __noinline__ T cl_long_sum(const ClMat<V>& mat, const ClSlice& s, int my_row, ClArray<T> vec, T t) {
    __shared__ T red[32];
    __shared__ T total;
    const ClArray<int> longs{s.longs};
    for (int i = 0; i < s.n_long; ++i) {
        const int row = longs[3 * i];
        const int64_t b = s.e0 + longs[3 * i + 1], e = b + longs[3 * i + 2];
        T acc = T(0);
        if (threadIdx.x < kThreads)
            for (int64_t k = b + threadIdx.x; k < e; k += kThreads)
                acc = fma(static_cast<T>(mat.val[k]), vec[mat.idx[k] - mat.idx_base], acc);
        T v[1] = {acc};
        block_reduce<OpSum, T, 1>(v, red);
        if (threadIdx.x == 0) total = v[0];
        __syncthreads();
        if (my_row == row) t = total;
        __syncthreads();
    }
    return t;
}

// The sum of my row in FP64 from FP64 values in global memory (the checks of FP32 iterations);
// any order will do.
template <typename T, typename V>
__device__ __noinline__ double cl_sum64(const ClMat<V>& mat, const ClSlice& s, int my_row, const double* val, ClArray<T> vec) {
    const int tpr = 1 << s.tpr_shift;
    int64_t b = 0, e = 0;
    if (my_row >= 0) { b = mat.ptr[s.b0 + my_row]; e = mat.ptr[s.b0 + my_row + 1]; }
    double acc = 0.0;
#pragma unroll 4
    for (int64_t k = b + (threadIdx.x & (tpr - 1)); k < e; k += tpr)
        acc = fma(__ldg(val + k), static_cast<double>(vec[__ldg(mat.idx + k) - mat.idx_base]), acc);
#pragma unroll 1
    for (int o = tpr >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

// One CTA's half-iterations.  T: vector type, V: value type.  What only some steps need stays in
// the ClInfo in shared memory: kept in registers it pushed the iteration's into local memory.
template <typename T, typename V>
struct ClCore {
    ClTask tc, tr;              // my column's and my row's task
    ClArray<T> yf;              // full y; the full x_bar is at offset 0
    int tpr_c, tpr_r;
    uint32_t size, rank;
    uint32_t peer_x, peer_y, peer_bar_x, peer_bar_y;   // thread t: my slices' places and the mbarriers in CTA t
    uint32_t par_x = 0, par_y = 0;
    int tries;                  // bound of a wait (a kernel parameter: no register)
    bool dead = false;          // a wait ran out: no further waiting, sending or arming

    __device__ __forceinline__ ClArray<T> xb() const { return ClArray<T>{0}; }

    // False when a slice does not fit into this CTA (uniform over the CTA).  A cluster barrier has
    // to follow before the first exchange.
    __device__ __forceinline__ bool begin(const ClMat<V>& a, const ClMat<V>& at, const ClLaunch& L, ClInfo& I) {
        tries = L.wait_tries;
        cl_begin<T, V>(a, at, L.smem_bytes, I);
        size = I.size;
        rank = I.rank;
        yf = ClArray<T>{cl_y_offset<T>(I.n)};
        bool ok = false;
        tc = cl_deal<V>(at, I.cols, yf.off, I.m, I, &ok);
        if (!ok) return false;
        tr = cl_deal<V>(a, I.rows, 0u, I.n, I, &ok);
        const uint32_t peer = threadIdx.x < size ? threadIdx.x : rank;
        peer_x = cl_map(smem_addr(xb().ptr() + I.cols.b0), peer);
        peer_y = cl_map(smem_addr(yf.ptr() + I.rows.b0), peer);
        peer_bar_x = cl_map(smem_addr(&I.bar_x), peer);
        peer_bar_y = cl_map(smem_addr(&I.bar_y), peer);
        tpr_c = 1 << I.cols.tpr_shift;
        tpr_r = 1 << I.rows.tpr_shift;
        return ok;
    }
    // The column / row this thread owns, -1: none.
    __device__ __forceinline__ int my_col(const ClInfo& I) const { return tc.row >= 0 && (threadIdx.x & (tpr_c - 1)) == 0 ? I.cols.b0 + tc.row : -1; }
    __device__ __forceinline__ int my_row(const ClInfo& I) const { return tr.row >= 0 && (threadIdx.x & (tpr_r - 1)) == 0 ? I.rows.b0 + tr.row : -1; }

    // Waits for the mbarrier's phase of that parity.
    __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity) {
        if (dead) return;
#pragma unroll 1
        for (int t = 0; t < tries; ++t) {
            uint32_t ok;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
            if (ok) return;
        }
        dead = true;
    }
    __device__ __forceinline__ static void push(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
        asm volatile(
            "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            ::"r"(dst), "r"(src), "r"(bytes), "r"(bar) : "memory");
    }
    // Sends my slices (of x_bar, of y) to every peer and waits for theirs, on x_bar's or y's
    // mbarrier.  A CTA without a slice of that vector signals the peers all the same, so that
    // nobody runs ahead of it.  All threads; the writes to my slices come before it.
    template <bool X, bool Y>
    __device__ __forceinline__ void exchange(ClInfo& I) {
        if (size == 1) { __syncthreads(); return; }
        const uint32_t bar = smem_addr(Y ? &I.bar_y : &I.bar_x);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < size && !dead) {
            if (threadIdx.x == rank) {
                const uint32_t expect = (X ? I.expect_x : 0u) + (Y ? I.expect_y : 0u);
                asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(expect) : "memory");
            } else {
                const uint32_t there = Y ? peer_bar_y : peer_bar_x;
                const uint32_t bx = X ? I.bytes_x : 0u, by = Y ? I.bytes_y : 0u;
                if (X && bx) push(peer_x, smem_addr(xb().ptr() + I.cols.b0), bx, there);
                if (Y && by) push(peer_y, smem_addr(yf.ptr() + I.rows.b0), by, there);
                if ((Y ? by : bx) == 0u)
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(there) : "memory");
            }
        }
        if constexpr (Y) { wait(bar, par_y); par_y ^= 1; }
        else { wait(bar, par_x); par_x ^= 1; }
    }
    __device__ __forceinline__ void exchange_x(ClInfo& I) { exchange<true, false>(I); }
    __device__ __forceinline__ void exchange_y(ClInfo& I) { exchange<false, true>(I); }
    // Both at once, on y's mbarrier: only between two cluster barriers.
    __device__ __forceinline__ void exchange_both(ClInfo& I) { exchange<true, true>(I); }

    // The end of a kernel, by all threads of the cluster, after the last exchange: no CTA may end
    // while a peer still sends to it or a copy still reads its memory.  Where every wait was met,
    // everything sent has arrived.
    __device__ __forceinline__ void leave(ClInfo& I) {
        if (dead)
            for (uint32_t q = 0; q < size; ++q)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_map(smem_addr(&I.ran_out), q)), "r"(1) : "memory");
        cl_barrier();
        if (!*static_cast<volatile int*>(&I.ran_out)) return;
        // Nobody sends any more, and nobody knows what is on its way (those phases were not armed): all stay
        // for a millisecond, a thousand times as long as a copy takes.
#pragma unroll 1
        for (int t = 0; t < kClDrainNaps; ++t) __nanosleep(500);
        cl_barrier();
    }

    // The sum of my row against `vec`, valid in the row's owner.  All threads.
    __device__ __forceinline__ static T sum(const ClTask& task, int tpr, const ClMat<V>& mat, const ClSlice& s, ClArray<T> vec) {
        T t = cl_chains<T>(task);
#pragma unroll 1
        for (int o = tpr >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (s.n_long) t = cl_long_sum<T, V>(mat, s, task.row, vec, t);
        return t;
    }
    // In the reference's arithmetic (group 1: a thread a row, no long rows); a padding entry of the
    // transpose adds the product of zero and a zero.
    __device__ __forceinline__ T col_sum_exact() { return cl_chains<T, true, false>(tc); }
    __device__ __forceinline__ T row_sum_exact() { return cl_chains<T, true, true>(tr); }
    __device__ __forceinline__ T col_sum(const ClMat<V>& at, const ClInfo& I) { return sum(tc, tpr_c, at, I.cols, yf); }
    __device__ __forceinline__ T row_sum(const ClMat<V>& a, const ClInfo& I) { return sum(tr, tpr_r, a, I.rows, xb()); }
};

// ----- chunks of Halpern iterations ----------------------------------------------------------
// What an iteration and a check need to know of the solver's state, by chunk.
struct ClControl {
    double tau, sigma, inv_sigma, gamma;
    long long k_base;
    int stop;       // no further chunk
    int restart;    // the candidate becomes iterate and anchor
    int wait_error; // a bounded wait ran out somewhere in the cluster
    int no_fit;     // a CTA's slices do not fit its shared memory: nothing was done
};
// The vectors of the LP(s); an instance's rows / columns start at the offsets its runner is given.
template <typename T>
struct ClVectors {
    const T* c; const T* cl; const T* cu; const T* rl; const T* ru;
    T* x; T* x0; T* xc; T* xprev; T* y; T* y0; T* yc; T* yprev;   // xprev, yprev may be null
    double* x_last; double* y_last;
    const double* a64; const double* at64;   // the matrices' FP64 values (entry by entry as V)
};
template <typename T>
struct ClMats { ClMat<T> a, at; };   // in shared memory

constexpr int kClWeights = 128;   // Halpern weights kept ahead

__device__ __forceinline__ unsigned long long ns_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Sums / maxima (MAXES: bit q set) of Q values a thread over the CTA, into part[0, Q): the warps'
// values go to shared memory, then a thread per quantity adds them up.  In a fixed order.
constexpr int kClWarps = kClThreads / 32;
template <int Q, uint32_t MAXES>
__device__ __forceinline__ void cl_reduce(double (&v)[Q], double* red, double* part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        v[q] = (MAXES >> q & 1u) ? warp_reduce<OpMax>(v[q]) : warp_reduce<OpSum>(v[q]);
        if (lane == 0) red[q * kClWarps + warp] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < Q) {
        const bool is_max = MAXES >> threadIdx.x & 1u;
        double t = 0.0;
        for (int w = 0; w < warps; ++w) {
            const double p = red[threadIdx.x * kClWarps + w];
            t = is_max ? fmax(t, p) : t + p;
        }
        part[threadIdx.x] = t;
    }
}
// The same over the CTAs' partials (Q each, in global memory), into red[0, Q).
template <int Q, uint32_t MAXES>
__device__ __forceinline__ void cl_combine(const double* part, int ctas, double* red) {
    if (threadIdx.x < Q) {
        const bool is_max = MAXES >> threadIdx.x & 1u;
        double t = 0.0;
        for (int r = 0; r < ctas; ++r) {
            const double p = __ldcg(part + r * Q + threadIdx.x);
            t = is_max ? fmax(t, p) : t + p;
        }
        red[threadIdx.x] = t;
    }
    __syncthreads();
}

// Up to max_chunks chunks of `K` iterations and a check each (the last one shorter where the
// iteration budget ends), until the solver's control stops the LP.  The arithmetic is that of the
// two-launch iteration: only where the data is differs, and the order of the checks' FP64 sums.
// Pol: `start(ctl)` gives the control of the first chunk (rank 0, all threads), `partials(i, ax,
// j, aty, rank)` stores this CTA's part of a check (i / j: this thread's row / column, -1: none),
// `decide(ctas, len, ns_primal, ns_dual, ctl)` takes the decision (rank 0, all threads) and
// `finish()` puts the state back (rank 0).  Rank 0 hands the control to its peers through *shared,
// in global memory.  Returns false when a slice does not fit.
template <typename T, int NT, class Pol>
__device__ __forceinline__ bool cl_run(const ClVectors<T>& P, const ClMats<T>& M, int row0, int col0, Pol& pol,
                                       ClControl* shared, int K, long long budget, int max_chunks, const ClLaunch& L) {
    __shared__ ClInfo I;
    __shared__ T hw[2 * kClWeights];
    __shared__ ClControl now;
    const int tid = threadIdx.x;
    ClCore<T, T> core;
    const bool fits = core.begin(M.a, M.at, L, I);
    for (int i = tid; i < I.m; i += NT) core.yf[i] = P.y[row0 + i];
    if (core.rank == 0) {
        if (tid == 0) now.wait_error = now.no_fit = now.restart = 0;
        __syncthreads();
        pol.start(now);
        __syncthreads();
        if (tid == 0) *shared = now;
    }
    cl_barrier();
    if (!fits && tid == 0) shared->no_fit = 1;
    cl_barrier();
    auto read_control = [&]() {   // written before a cluster barrier
        constexpr int kWords = sizeof(ClControl) / 4;
        static_assert(sizeof(ClControl) % 4 == 0 && kWords <= NT, "ClControl is copied in words");
        if (tid < kWords) reinterpret_cast<int*>(&now)[tid] = __ldcg(reinterpret_cast<const int*>(shared) + tid);
        __syncthreads();
    };
    read_control();
    if (now.no_fit) return false;
    // My column and my row, if I own one (-1: none).
    const int jl = core.my_col(I), il = core.my_row(I);
    const int j = jl < 0 ? -1 : col0 + jl, i = il < 0 ? -1 : row0 + il;
    T x = T(0), x0 = T(0), c = T(0), cl = T(0), cu = T(0), y = T(0), y0 = T(0), rl = T(0), ru = T(0);
    if (j >= 0) { x = P.x[j]; x0 = P.x0[j]; c = P.c[j]; cl = P.cl[j]; cu = P.cu[j]; }
    if (i >= 0) { y = P.y[i]; y0 = P.y0[i]; rl = P.rl[i]; ru = P.ru[i]; }
    for (int chunk = 0; chunk < max_chunks && budget > 0 && !now.stop; ++chunk) {
        const int len = budget < K ? static_cast<int>(budget) : K;
        budget -= len;
        const T tau = static_cast<T>(now.tau), sigma = static_cast<T>(now.sigma), inv_sigma = static_cast<T>(now.inv_sigma),
                g = static_cast<T>(now.gamma);
        unsigned int t0 = 0, t1 = 0, t2 = 0;
        // Turn kk < len is an iteration.  Turn len forms the check's products: the candidate takes
        // the place of x_bar and y in the full vectors.
#pragma unroll 1
        for (int kk = 0; kk <= len; ++kk) {
            const bool check = kk == len;
            const int slot = kk & (kClWeights - 1);
            if (slot == 0) {   // everyone is past the last use of the old weights
                const long long k_base = now.k_base;
                for (int q = tid; q < kClWeights; q += NT) {
                    const double k = static_cast<double>(k_base + kk + q);
                    hw[2 * q] = static_cast<T>((k + 1.0) / (k + 2.0));
                    hw[2 * q + 1] = static_cast<T>(1.0 / (k + 2.0));
                }
                __syncthreads();
            }
            if (kk == 1) t0 = static_cast<unsigned int>(ns_now());
            if (check) {
                cl_barrier();   // every row sum is done with x_bar
                if (j >= 0) core.xb()[jl] = P.xc[j];
                if (i >= 0) core.yf[il] = P.yc[i];
                core.exchange_both(I);
                if constexpr (sizeof(T) == 4) {   // FP64 values, from global memory
                    const double ax = cl_sum64<T, T>(M.a, I.rows, core.tr.row, P.a64, core.xb());
                    const double aty = cl_sum64<T, T>(M.at, I.cols, core.tc.row, P.at64, core.yf);
                    pol.partials(i, ax, j, aty, core.rank);
                    break;
                }
            }
            const T w1 = hw[2 * slot], w0 = hw[2 * slot + 1];
            const T v = core.col_sum(M.at, I);
            if (!check) {
                if (j >= 0) {
                    const T xo = x;
                    T xp, xbn;
                    halpern_primal(xo, v, c, cl, cu, x0, tau, w1, w0, g, &xp, &xbn, &x);
                    core.xb()[jl] = xbn;
                    if (kk == len - 1) { P.xc[j] = xp; if (P.xprev) P.xprev[j] = xo; }
                }
                core.exchange_x(I);
                if (kk == 1) t1 = static_cast<unsigned int>(ns_now());
            }
            const T w = core.row_sum(M.a, I);
            if (!check) {
                if (i >= 0) {
                    const T yo = y;
                    T yp;
                    halpern_dual(yo, w, rl, ru, y0, sigma, inv_sigma, w1, w0, g, &yp, &y);
                    core.yf[il] = y;
                    if (kk == len - 1) { P.yc[i] = yp; if (P.yprev) P.yprev[i] = yo; }
                }
                if (kk < len - 1) core.exchange_y(I);
                if (kk == 1) t2 = static_cast<unsigned int>(ns_now());
            } else {
                pol.partials(i, static_cast<double>(w), j, static_cast<double>(v), core.rank);
            }
        }
        if (core.dead) shared->wait_error = 1;
        cl_barrier();
        if (core.rank == 0) {
            if (tid == 0) now.wait_error = *static_cast<volatile int*>(&shared->wait_error);
            pol.decide(static_cast<int>(core.size), len, len > 2 ? static_cast<double>(t1 - t0) : 0.0, static_cast<double>(t2 - t1), now);
            __syncthreads();
            if (tid == 0) {
                if (now.wait_error) now.stop = 1;
                *shared = now;
            }
        }
        cl_barrier();
        read_control();
        if (now.restart) {
            if (j >= 0) { x = x0 = P.xc[j]; P.x_last[j] = static_cast<double>(x); }
            if (i >= 0) { y = y0 = P.yc[i]; P.y_last[i] = static_cast<double>(y); }
        }
        if (now.stop) break;
        if (i >= 0) core.yf[il] = y;
        core.exchange_y(I);
    }
    if (j >= 0) { P.x[j] = x; P.x0[j] = x0; }
    if (i >= 0) { P.y[i] = y; P.y0[i] = y0; }
    if (core.rank == 0) pol.finish();
    core.leave(I);
    return true;
}

// Launches `kernel` on `clusters` clusters of `ctas` CTAs; errors are left for cudaGetLastError.
template <typename... Params, typename... Args>
inline cudaError_t launch_clusters(void (*kernel)(Params...), int clusters, int ctas, int threads, size_t smem,
                                   cudaStream_t st, Args&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters) * ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
    note_launch();
    return e;
}
// Grants a kernel the shared memory and the cluster size of a launch; an error when the device has
// no room for one such cluster.
template <typename... Params>
inline cudaError_t prepare_clusters(void (*kernel)(Params...), int ctas, int threads, size_t smem) {
    const void* f = reinterpret_cast<const void*>(kernel);
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kClSmemCap));
    if (e == cudaSuccess && ctas > 8) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess || ctas == 1) return e;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    e = cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg);
    return e != cudaSuccess ? e : fit >= 1 ? cudaSuccess : cudaErrorInvalidConfiguration;
}

// How a single LP is laid over a cluster: CTAs (0: it does not go there), threads, shared memory.
struct ClusterPlan { int ctas = 0, threads = 0; size_t smem = 0; };

// The smallest cluster whose CTAs have at most 256 rows and columns and about 1,000 entries of
// each matrix, else 16 CTAs of up to 512.  Fewer CTAs exchange faster (0.6 us for 8, 0.8 us for
// 16), more share the row sums; 256 threads pass a CTA's barriers faster than 512.  Microseconds
// an iteration (FP32 / FP64; two launches an iteration: 5.5 to 6.8), checks included: 60 x 150 on
// 1 CTA 1.2 / 1.3, on 4 1.7 / 1.7; 301 x 807 on 4 CTAs 1.9 / 2.1, on 8 1.9 / 2.1; 2000 x 5000 on
// 16 CTAs of 512 threads 3.4 / 4.9; 5000 x 12000 (1,024 threads) 8.4 against 7.2, which is why the
// line lies at 512.  Every thread forms at most kClMaxChains chains of a row.
// `from`: CTAs it has at least.  `prepare(ctas, threads)`: what a launch needs (an error: there is
// no such cluster on this device).
template <class Prepare>
inline ClusterPlan plan_one_cluster(size_t t, int64_t m, int64_t n, int64_t nnz, int group_a, int group_at, int from, Prepare prepare) {
    for (int ctas = from; ctas <= kClMaxCtas; ctas *= 2) {
        const int threads = cl_fits(t, m, n, nnz, group_a, group_at, ctas, 256) ? 256 : 512;
        if (!cl_fits(t, m, n, nnz, group_a, group_at, ctas, threads)) continue;
        if (ctas < kClMaxCtas && (threads > 256 || nnz > 1024 * static_cast<int64_t>(ctas))) continue;
        if (prepare(ctas, threads) != cudaSuccess) { cudaGetLastError(); continue; }
        return ClusterPlan{ctas, threads, kClSmemCap};   // all of it: slices may be uneven
    }
    return {};
}

}  // namespace vajra
