// Edge-batch updates of a decomposed graph (methods 5-11 of the reference:
// insert_idea1/insert_idea2, src/scc_incremental.cc:7-27, create_scc_edges,
// src/common_main.h:180-314; delete_idea1, src/scc_decremental.cc:7-24, and
// read_file2, src/common_main.h:343-393).
//
// The reference rebuilds gm_graph on the host and either recomputes
// everything (method 5), decomposes the condensation graph (methods 6, 7, 11),
// or re-runs the pipeline with the SCCs that lost an edge (methods 8-10, only
// SCC index 5 in its code).  Here a batch is applied on the device:
//
//  1. CSR merge: deleted (u,v) pairs remove every copy of that edge, inserted
//     pairs are added (kept sorted, duplicates allowed as add_edge allows
//     them), on the CSR and on the transpose.
//  2. Deletions: only an old SCC that lost an internal edge can split.  Those
//     SCCs become classes and the device recursion re-decomposes them; every
//     other SCC keeps its label.  Afterwards every label class is strongly
//     connected in the new graph.
//  3. Insertions: a merge needs a cycle through an inserted edge (u,v) whose
//     ends are in different classes (the old condensation had no cycle), so
//     every merged SCC lies in R = FW(those v) and BW(those u).  R is a union
//     of classes closed under strong connectivity; SCCs are recomputed inside
//     R only.
#include <algorithm>
#include <string.h>
#include "scc_round.cuh"
#include "scc_sort.cuh"

// ------------------------------------------------------------------ kernels
__global__ void k_upd_keys(int64_t k, const int32_t* __restrict__ a, const int32_t* __restrict__ b, int32_t n,
                           unsigned long long* __restrict__ keys, int* __restrict__ bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t x = a[i], y = b[i];
        if (x < 0 || x >= n || y < 0 || y >= n) { atomicExch(bad, 1); keys[i] = ~0ull; continue; }
        keys[i] = ((unsigned long long)(uint32_t)x << 32) | (uint32_t)y;
    }
}

// The merge of one side (CSR or transpose) treats the adjacency array as one
// ascending sequence of (row, col) keys.  A batch changes it at few places, so
// an old entry only moves by a shift: the inserted keys placed before it minus
// the deleted entries before it, constant between two neighbouring events.
//   k_upd_events   where each event lies in the old array (a search per key)
//   k_upd_offsets  the new offsets: the old ones shifted the same way
//   k_upd_move     the old entries, copied with their shift
//   k_upd_place    the inserted entries
// Every kernel is balanced over entries, vertices or keys.  (One warp per list
// took as long as the largest hub needed: 2.7 ms a side on R-MAT s22, whose
// largest list has 95,000 entries, against 0.16 ms for the copy now; the copy
// is bound by HBM at 4 B read and 4 B written per entry.)

// The number of elements of a[0, k), ascending, that come before `key` (LE: that
// are <= key), searched by the whole warp 33 ways at a time; the same in every lane.
template <bool LE, typename T>
__device__ __forceinline__ int64_t warp_count_before(const T* __restrict__ a, int64_t k, T key) {
    const int lane = threadIdx.x & 31;
    int64_t lo = 0, hi = k;
    while (hi > lo) {
        const int64_t step = (hi - lo + 32) / 33;           // 32 probes split [lo, hi) into 33 parts
        const int64_t at = lo + step * (lane + 1) - 1;
        bool before = false;
        if (at < hi) { const T x = a[at]; before = LE ? x <= key : x < key; }
        const int c = __popc(__ballot_sync(0xFFFFFFFFu, before));   // probes ascend: the true ones come first
        lo += step * c;
        if (c < 32) hi = min(hi, lo + step - 1);            // probe c did not come before
    }
    return lo;
}

// The same inside [lo, hi) for one thread.
template <bool LE, typename T>
__device__ __forceinline__ int32_t count_before(const T* __restrict__ a, int32_t lo, int32_t hi, T key) {
    while (lo < hi) {
        const int32_t mid = lo + ((hi - lo) >> 1);
        const T x = __ldg(a + mid);
        if (LE ? x <= key : x < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Places of the events in the old array.  A deleted key (row, col) is the run
// of its copies, [run_lo, run_lo + run_cnt) (no copy: run_cnt 0); of repeats of
// one key the last has the count, so that the last run starting at or before
// an entry is the one that can cover it.  An inserted key goes behind the old
// entries <= it.  Keys ascend, so run_lo and ins_at do too.
__global__ void k_upd_events(int32_t kdel, const unsigned long long* __restrict__ del, int32_t kins,
                             const unsigned long long* __restrict__ ins, const int32_t* __restrict__ off,
                             const int32_t* __restrict__ adj, int32_t* __restrict__ run_lo,
                             int32_t* __restrict__ run_cnt, int32_t* __restrict__ ins_at) {
    const int64_t total = (int64_t)kdel + kins;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < kdel) {
            const unsigned long long key = del[i];
            const int32_t r = (int32_t)(key >> 32), c = (int32_t)(uint32_t)key;
            const int32_t e = off[r + 1];
            const int32_t lo = count_before<false>(adj, off[r], e, c);
            int32_t cnt = 0;
            if (!(i + 1 < kdel && del[i + 1] == key)) cnt = count_before<true>(adj, lo, e, c) - lo;
            run_lo[i] = lo;
            run_cnt[i] = cnt;
        } else {
            const unsigned long long key = ins[i - kdel];
            const int32_t r = (int32_t)(key >> 32), c = (int32_t)(uint32_t)key;
            ins_at[i - kdel] = count_before<true>(adj, off[r], off[r + 1], c);
        }
    }
}

// new_off[v] = off[v] + inserted keys of rows before v - deleted entries before
// off[v].  A warp takes 128 consecutive offsets: it searches the batch for its
// first and last one together, its lanes only between those two.
#define UPD_OFFS 128
__global__ void k_upd_offsets(int32_t n, const int32_t* __restrict__ off, int32_t kdel,
                              const int32_t* __restrict__ run_lo, const int32_t* __restrict__ run_pref, int32_t kins,
                              const unsigned long long* __restrict__ ins, int32_t* __restrict__ new_off) {
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t groups = ((int64_t)n + UPD_OFFS) / UPD_OFFS;          // n + 1 offsets
    for (int64_t gi = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; gi < groups; gi += nwarps) {
        const int64_t v0 = gi * UPD_OFFS, v1 = min((int64_t)n, v0 + UPD_OFFS - 1);
        const int32_t i0 = (int32_t)warp_count_before<false>(ins, kins, (unsigned long long)v0 << 32);
        const int32_t i1 = i0 + (int32_t)warp_count_before<false>(ins + i0, kins - i0, (unsigned long long)v1 << 32);
        const int32_t d0 = (int32_t)warp_count_before<false>(run_lo, kdel, off[v0]);
        const int32_t d1 = d0 + (int32_t)warp_count_before<false>(run_lo + d0, kdel - d0, off[v1]);
        for (int64_t v = v0 + lane; v <= v1; v += 32) {
            const int32_t o = off[v];
            const int32_t i = i0 == i1 ? i0 : count_before<false>(ins, i0, i1, (unsigned long long)v << 32);
            const int32_t d = d0 == d1 ? d0 : count_before<false>(run_lo, d0, d1, o);
            new_off[v] = o + i - run_pref[d];
        }
    }
}

// Events at or before the first entry of each tile of UPD_TILE old entries, in
// the insert and the delete list (one more for the end): the tile's own events
// lie between its pair and the next one.
#define UPD_ITEMS 16
#define UPD_TILE (32 * UPD_ITEMS)
__global__ void k_upd_bounds(int32_t m, int32_t kdel, const int32_t* __restrict__ run_lo, int32_t kins,
                             const int32_t* __restrict__ ins_at, int32_t tiles, int2* __restrict__ bound) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t <= tiles; t += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = (int32_t)min((int64_t)m, t * UPD_TILE);
        bound[t] = make_int2(count_before<true>(ins_at, 0, kins, i), count_before<true>(run_lo, 0, kdel, i));
    }
}

// Old entries to their new places, a tile per warp.  A tile with no event is
// one shifted copy; in the others each lane searches the tile's own events.  A
// place outside the new array (only a list that was not sorted could give one)
// is skipped.  The bounds come from their own launch: searched here, they put
// four dependent loads before every tile (R-MAT s22, 65 M entries and 100,000
// events, a side: 314 us with the searches and a block per 4,096 entries,
// 159 us so).
__global__ void __launch_bounds__(SCC_THREADS) k_upd_move(int32_t m, const int32_t* __restrict__ adj,
                                                          const int32_t* __restrict__ run_lo,
                                                          const int32_t* __restrict__ run_pref,
                                                          const int32_t* __restrict__ ins_at, int32_t tiles,
                                                          const int2* __restrict__ bound, int64_t new_m,
                                                          int32_t* __restrict__ new_adj) {
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; t < tiles; t += nwarps) {
        const int64_t t0 = t * UPD_TILE + lane;
        int32_t x[UPD_ITEMS];
#pragma unroll
        for (int j = 0; j < UPD_ITEMS; ++j) x[j] = t0 + 32 * j < m ? __ldcs(adj + t0 + 32 * j) : 0;
        const int2 b0 = __ldg(bound + t), b1 = __ldg(bound + t + 1);
        const int32_t dead0 = __ldg(run_pref + b0.y);
        // a run that started at or before the tile may reach into it
        const bool covered = b0.y > 0 && (int64_t)__ldg(run_lo + b0.y - 1) + (dead0 - __ldg(run_pref + b0.y - 1)) > t * UPD_TILE;
        if (b0.x == b1.x && b0.y == b1.y && !covered) {
            const int64_t at = t0 + b0.x - dead0;
#pragma unroll
            for (int j = 0; j < UPD_ITEMS; ++j)
                if (t0 + 32 * j < m && (uint64_t)(at + 32 * j) < (uint64_t)new_m) __stcs(new_adj + at + 32 * j, x[j]);
            continue;
        }
#pragma unroll
        for (int j = 0; j < UPD_ITEMS; ++j) {
            const int64_t i = t0 + 32 * j;
            if (i >= m) continue;
            const int32_t before = count_before<true>(ins_at, b0.x, b1.x, (int32_t)i);
            const int32_t d = count_before<true>(run_lo, b0.y, b1.y, (int32_t)i);
            const int32_t dead = __ldg(run_pref + d);
            if (d > 0 && (int64_t)__ldg(run_lo + d - 1) + (dead - __ldg(run_pref + d - 1)) > i) continue;      // deleted
            const int64_t at = i + before - dead;
            if ((uint64_t)at < (uint64_t)new_m) __stcs(new_adj + at, x[j]);
        }
    }
}

// Inserted entries: behind the old entries <= them and the inserted ones before them.
__global__ void k_upd_place(int32_t kins, const unsigned long long* __restrict__ ins,
                            const int32_t* __restrict__ ins_at, int32_t kdel, const int32_t* __restrict__ run_lo,
                            const int32_t* __restrict__ run_pref, int64_t new_m, int32_t* __restrict__ new_adj) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < kins; j += (int64_t)gridDim.x * blockDim.x) {
        const int32_t at0 = ins_at[j];
        const int64_t at = (int64_t)at0 + j - run_pref[count_before<false>(run_lo, 0, kdel, at0)];
        if ((uint64_t)at < (uint64_t)new_m) new_adj[at] = (int32_t)(uint32_t)ins[j];
    }
}

__global__ void k_upd_fill(int64_t n, int32_t* __restrict__ a, int32_t v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) a[i] = v;
}

// Deleted pairs inside one SCC flag that SCC's representative.
__global__ void k_upd_flag_split(int64_t k, const unsigned long long* __restrict__ keys, const int32_t* __restrict__ scc,
                                 int32_t* __restrict__ flag) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long key = keys[i];
        if (key == ~0ull) continue;
        int32_t u = (int32_t)(key >> 32), w = (int32_t)(uint32_t)key;
        int32_t r = scc[u];
        if (r >= 0 && r == scc[w]) flag[r] = 1;
    }
}

// Vertices of flagged SCCs become live with their old representative as class
// colour; all others are finished.
__global__ void k_upd_colour_flagged(int32_t n, const int32_t* __restrict__ scc, const int32_t* __restrict__ flag,
                                     int32_t* __restrict__ color, int32_t* __restrict__ count) {
    int32_t c = 0;
    int64_t limit = (((int64_t)n + 31) / 32) * 32;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < limit; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < n) {
            int32_t r = scc[i];
            bool live = r >= 0 && flag[r];
            color[i] = live ? r : SCC_COLOR_DONE;
            c += live;
        }
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

// Seeds of the merge region: for inserted (u,v) across classes, FW from v, BW from u.
__global__ void k_upd_seed_region(int64_t k, const unsigned long long* __restrict__ keys, const int32_t* __restrict__ scc,
                                  uint8_t* __restrict__ mark, int32_t* __restrict__ q, int32_t* __restrict__ qlen) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long key = keys[i];
        if (key == ~0ull) continue;
        int32_t u = (int32_t)(key >> 32), v = (int32_t)(uint32_t)key;
        if (scc[u] == scc[v]) continue;
        unsigned sh = (unsigned)(v & 3) * 8u;
        unsigned old = atomicOr(reinterpret_cast<unsigned*>(mark + (v & ~3)), 1u << sh);
        if (!((old >> sh) & 1u)) q[atomicAdd(qlen, 1)] = v;
        sh = (unsigned)(u & 3) * 8u;
        old = atomicOr(reinterpret_cast<unsigned*>(mark + (u & ~3)), 2u << sh);
        if (!((old >> sh) & 2u)) q[atomicAdd(qlen, 1)] = u | (1 << DIR_SHIFT);
    }
}

// R = reached both ways: class 0, live; everything else finished.  Marks cleared.
__global__ void k_upd_colour_region(int32_t n, uint8_t* __restrict__ mark, int32_t* __restrict__ color,
                                    int32_t* __restrict__ count) {
    int32_t c = 0;
    int64_t limit = (((int64_t)n + 31) / 32) * 32;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < limit; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < n) {
            bool in = (mark[i] & 3) == 3;
            color[i] = in ? 0 : SCC_COLOR_DONE;
            mark[i] = 0;
            c += in;
        }
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

// ------------------------------------------------------------------ host helpers
// Stream-ordered scratch: cudaFree would synchronise the whole device and
// serialise updates that run concurrently on other streams.
struct DevBuf {
    void* p = nullptr;
    cudaStream_t st = nullptr;
    ~DevBuf() { if (p) cudaFreeAsync(p, st); }
    template <class T> T* as() { return (T*)p; }
};

static int alloc(DevBuf& b, size_t bytes, cudaStream_t st) {
    b.st = st;
    SCC_CUDA(scc_impl_malloc_async(&b.p, bytes > 0 ? bytes : 16, st));
    return SCC_OK;
}

// Replace a graph's arrays with stream-ordered ones.
static void release_graph_arrays(scc_graph* g, cudaStream_t st) {
    int32_t* arr[4] = {g->begin, g->node_idx, g->r_begin, g->r_node_idx};
    // the first update of a built graph waits for the device, as cudaFree does where
    // its arrays come from cudaMalloc
    if (g->built_arrays) cudaDeviceSynchronize();
    g->built_arrays = false;
    for (int i = 0; i < 4; ++i) {
        if (!arr[i]) continue;
        if (g->async_arrays) cudaFreeAsync(arr[i], st);
        else cudaFree(arr[i]);
    }
}

// The batch's pairs as one list to sort: list 0 inserts (src, dst), 1 inserts
// (dst, src), 2 deletes (src, dst), 3 deletes (dst, src); key = list, row and column in
// 2 + bits + bits bits.  One sort in place of four: a sort's passes are bound by their
// launches at these sizes.
__global__ void k_upd_pack(int64_t ki, const int32_t* __restrict__ is, const int32_t* __restrict__ id, int64_t kd,
                           const int32_t* __restrict__ ds, const int32_t* __restrict__ dd, int32_t n, int bits,
                           unsigned long long* __restrict__ keys, int* __restrict__ bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ki + kd; i += (int64_t)gridDim.x * blockDim.x) {
        const bool del = i >= ki;
        const int64_t j = del ? i - ki : i, k = del ? kd : ki, base = del ? 2 * ki : 0;
        const int32_t x = del ? ds[j] : is[j], y = del ? dd[j] : id[j];
        if (x < 0 || x >= n || y < 0 || y >= n) atomicExch(bad, 1);
        const unsigned long long list = (unsigned long long)(del ? 2 : 0) << (2 * bits);
        keys[base + j] = list | ((unsigned long long)(uint32_t)x << bits) | (uint32_t)y;
        keys[base + k + j] = list | (1ull << (2 * bits)) | ((unsigned long long)(uint32_t)y << bits) | (uint32_t)x;
    }
}

// Sorted keys to (row << 32 | column).
__global__ void k_upd_unpack(int64_t k, int bits, unsigned long long* __restrict__ keys) {
    const unsigned long long mask = (1ull << bits) - 1ull;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long x = keys[i];
        keys[i] = (((x >> bits) & mask) << 32) | (x & mask);
    }
}

// keys (a<<32|b) sorted ascending into out (k entries); invalid ids flagged in *bad.
static int sorted_keys(int64_t k, const int32_t* d_a, const int32_t* d_b, int32_t n, cudaStream_t st,
                       unsigned long long* out, int* d_bad) {
    DevBuf tmpk;
    SCC_TRY(alloc(tmpk, sizeof(unsigned long long) * (size_t)k, st));
    if (k == 0) return SCC_OK;
    k_upd_keys<<<scc_blocks(k), SCC_THREADS, 0, st>>>(k, d_a, d_b, n, tmpk.as<unsigned long long>(), d_bad);
    SCC_CUDA(cudaPeekAtLastError());
    // a < n in the high word: the bits above 32 + log2(n) are zero
    int hb = 1;
    while (hb < 31 && (1LL << hb) < (int64_t)n) hb++;
    return scc_impl_sort_keys_u64(tmpk.as<unsigned long long>(), out, k, 32 + hb, st);
}

// The four sorted lists (see k_upd_pack) one after another in out, and where each begins.
struct BatchKeys {
    DevBuf all;
    unsigned long long *ins = nullptr, *ins_t = nullptr, *del = nullptr, *del_t = nullptr;
};
static int sort_batch(BatchKeys& b, int64_t ki, const int32_t* is, const int32_t* id, int64_t kd, const int32_t* ds,
                      const int32_t* dd, int32_t n, cudaStream_t st, int* d_bad) {
    const int64_t total = 2 * (ki + kd);
    SCC_TRY(alloc(b.all, sizeof(unsigned long long) * (size_t)total, st));
    b.ins = b.all.as<unsigned long long>();
    b.ins_t = b.ins + ki;
    b.del = b.ins_t + ki;
    b.del_t = b.del + kd;
    if (total == 0) return SCC_OK;
    if (total >= (1LL << 31)) {          // beyond one sort: each list by itself
        SCC_TRY(sorted_keys(ki, is, id, n, st, b.ins, d_bad));
        SCC_TRY(sorted_keys(ki, id, is, n, st, b.ins_t, d_bad));
        SCC_TRY(sorted_keys(kd, ds, dd, n, st, b.del, d_bad));
        return sorted_keys(kd, dd, ds, n, st, b.del_t, d_bad);
    }
    int bits = 1;
    while (bits < 31 && (1LL << bits) < (int64_t)n) bits++;
    DevBuf tmpk;
    SCC_TRY(alloc(tmpk, sizeof(unsigned long long) * (size_t)total, st));
    k_upd_pack<<<scc_blocks(ki + kd), SCC_THREADS, 0, st>>>(ki, is, id, kd, ds, dd, n, bits,
                                                           tmpk.as<unsigned long long>(), d_bad);
    SCC_CUDA(cudaPeekAtLastError());
    SCC_TRY(scc_impl_sort_keys_u64(tmpk.as<unsigned long long>(), b.ins, total, 2 * bits + 2, st));
    k_upd_unpack<<<scc_blocks(total), SCC_THREADS, 0, st>>>(total, bits, b.ins);
    SCC_CUDA(cudaPeekAtLastError());
    return SCC_OK;
}

// One side of the merge: where the batch's events lie in the old arrays, then
// the new arrays (NULL until they are allocated; freed on `st` unless taken).
struct MergeSide {
    const int32_t* off; const int32_t* adj;
    const unsigned long long* del; const unsigned long long* ins;
    DevBuf run_lo, run_pref, ins_at;
    int32_t* new_off = nullptr; int32_t* new_adj = nullptr;
    cudaStream_t st = nullptr;
    int32_t dead = 0;               // entries deleted (valid after a synchronisation)
    ~MergeSide() {
        if (new_off) cudaFreeAsync(new_off, st);
        if (new_adj) cudaFreeAsync(new_adj, st);
    }
};

static int merge_events(MergeSide& x, int32_t kdel, int32_t kins, cudaStream_t st) {
    DevBuf cnt;
    x.st = st;
    SCC_TRY(alloc(x.run_lo, sizeof(int32_t) * (size_t)kdel, st));
    SCC_TRY(alloc(cnt, sizeof(int32_t) * ((size_t)kdel + 1), st));
    SCC_TRY(alloc(x.run_pref, sizeof(int32_t) * ((size_t)kdel + 1), st));
    SCC_TRY(alloc(x.ins_at, sizeof(int32_t) * (size_t)kins, st));
    // one extra zero count: its exclusive prefix is the number of deleted entries
    SCC_CUDA(cudaMemsetAsync(cnt.as<int32_t>() + kdel, 0, sizeof(int32_t), st));
    if ((int64_t)kdel + kins > 0) {          // two lists of 2^30 and more pass 2^31 together
        k_upd_events<<<scc_blocks((int64_t)kdel + kins), SCC_THREADS, 0, st>>>(
            kdel, x.del, kins, x.ins, x.off, x.adj, x.run_lo.as<int32_t>(), cnt.as<int32_t>(), x.ins_at.as<int32_t>());
        SCC_CUDA(cudaPeekAtLastError());
    }
    SCC_TRY(scc_impl_scan_i32(cnt.as<int32_t>(), x.run_pref.as<int32_t>(), (int64_t)kdel + 1, false, st));
    SCC_CUDA(cudaMemcpyAsync(&x.dead, x.run_pref.as<int32_t>() + kdel, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    return SCC_OK;
}

static int merge_write(MergeSide& x, int32_t n, int64_t m, int32_t kdel, int32_t kins, cudaStream_t st) {
    const int64_t new_m = m + kins - x.dead;
    SCC_CUDA(scc_impl_malloc_async((void**)&x.new_off, sizeof(int32_t) * ((size_t)n + 1), st));
    SCC_CUDA(scc_impl_malloc_async((void**)&x.new_adj, sizeof(int32_t) * (size_t)(new_m > 0 ? new_m : 1), st));
    k_upd_offsets<<<scc_blocks(((int64_t)n / UPD_OFFS + 1) * 32, SCC_THREADS, 148 * 8), SCC_THREADS, 0, st>>>(
        n, x.off, kdel, x.run_lo.as<int32_t>(), x.run_pref.as<int32_t>(), kins, x.ins, x.new_off);
    SCC_CUDA(cudaPeekAtLastError());
    if (m > 0) {
        const int32_t tiles = (int32_t)((m + UPD_TILE - 1) / UPD_TILE);
        DevBuf bound;
        SCC_TRY(alloc(bound, sizeof(int2) * ((size_t)tiles + 1), st));
        k_upd_bounds<<<scc_blocks((int64_t)tiles + 1), SCC_THREADS, 0, st>>>(
            (int32_t)m, kdel, x.run_lo.as<int32_t>(), kins, x.ins_at.as<int32_t>(), tiles, bound.as<int2>());
        SCC_CUDA(cudaPeekAtLastError());
        k_upd_move<<<scc_blocks((int64_t)tiles * 32), SCC_THREADS, 0, st>>>(
            (int32_t)m, x.adj, x.run_lo.as<int32_t>(), x.run_pref.as<int32_t>(), x.ins_at.as<int32_t>(), tiles,
            bound.as<int2>(), new_m, x.new_adj);
        SCC_CUDA(cudaPeekAtLastError());
    }
    if (kins > 0) {
        k_upd_place<<<scc_blocks(kins), SCC_THREADS, 0, st>>>(kins, x.ins, x.ins_at.as<int32_t>(), kdel,
                                                             x.run_lo.as<int32_t>(), x.run_pref.as<int32_t>(), new_m,
                                                             x.new_adj);
        SCC_CUDA(cudaPeekAtLastError());
    }
    return SCC_OK;
}

// Merge a batch (sorted keys of the CSR, and of the transpose) into g's arrays.
// A failure leaves g as it was.
static int merge_batch(scc_graph* g, const unsigned long long* del, const unsigned long long* del_t, int64_t kdel,
                       const unsigned long long* ins, const unsigned long long* ins_t, int64_t kins, cudaStream_t st) {
    SCC_REQUIRE(kdel < (1LL << 31) && g->m + kins < (1LL << 31) - 1, SCC_ERR_INVALID,
                "batch of %lld inserts and %lld deletes exceeds int32 edge ids", (long long)kins, (long long)kdel);
    MergeSide f, r;
    f.off = g->begin; f.adj = g->node_idx; f.del = del; f.ins = ins;
    r.off = g->r_begin; r.adj = g->r_node_idx; r.del = del_t; r.ins = ins_t;
    SCC_TRY(merge_events(f, (int32_t)kdel, (int32_t)kins, st));
    SCC_TRY(merge_events(r, (int32_t)kdel, (int32_t)kins, st));
    SCC_CUDA(cudaStreamSynchronize(st));
    SCC_TRY(merge_write(f, g->n, g->m, (int32_t)kdel, (int32_t)kins, st));
    SCC_TRY(merge_write(r, g->n, g->m, (int32_t)kdel, (int32_t)kins, st));
    release_graph_arrays(g, st);
    g->begin = f.new_off; g->node_idx = f.new_adj; g->r_begin = r.new_off; g->r_node_idx = r.new_adj;
    f.new_off = f.new_adj = r.new_off = r.new_adj = nullptr;
    g->m = g->m + kins - f.dead;
    g->self_loops = -1;
    g->async_arrays = true;
    return SCC_OK;
}

static RoundArgs update_round_args(const scc_graph* g, scc_state* s) {
    RoundArgs a;
    a.begin = g->begin; a.node_idx = g->node_idx; a.r_begin = g->r_begin; a.r_node_idx = g->r_node_idx;
    a.color = s->color; a.scc = s->scc; a.mark = s->mark;
    a.slot_key = s->slot_key; a.slot_pivot = s->slot_pivot; a.slot_fw = s->slot_fw; a.slot_bw = s->slot_bw;
    a.slot_count = s->slot_count;
    a.colour_cap = s->colour_cap;
    a.ctr = s->ctr;
    a.live = s->live; a.live_count = s->live_count;
    a.only_color = 0; a.use_only = 1;
    a.huge_deg = s->tune.huge_deg;
    a.async_keep = s->tune.async_keep;
    a.async_bail = std::max<int32_t>(8 * s->tune.async_max, 1 << 16);
    a.pivot_salt = 0;
    a.cta_deg = s->tune.cta_deg;
    round_args_adjacency(a, g->node_idx, g->r_node_idx, g->m);
    return a;
}

// Decompose the classes an update left live (colours in [0, n), live list not
// built).  The first round takes them as they are: they come from old SCCs, so
// nearly all of one is still strongly connected, and pivoting it at once costs
// less than peeling and splitting it first; what it leaves is peeled and split by
// the next round.  Fresh colours must lie above every class colour.
static int resolve_update(const scc_graph* g, scc_state* s) {
    s->fresh = false;
    s->prefinished = false;
    s->live_count = -1;
    const int32_t last = g->n - 1;
    SCC_CUDA(cudaMemcpyAsync(s->ctr + CTR_NEXT_COLOR, &last, sizeof(int32_t), cudaMemcpyHostToDevice, s->stream));
    s->h_ctr[CTR_NEXT_COLOR] = last;
    return scc_impl_resolve_all(g, s, true);
}

static double ev_ms(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, a, b) != cudaSuccess) { cudaGetLastError(); return 0.0; }
    return ms;
}

// ------------------------------------------------------------------ C ABI
extern "C" int scc_update_batch(scc_graph* g, scc_state* s, int64_t n_ins, const int32_t* ins_src,
                                const int32_t* ins_dst, int64_t n_del, const int32_t* del_src, const int32_t* del_dst,
                                int on_device, scc_update_stats* stats) {
    SCC_REQUIRE(g && s, SCC_ERR_INVALID, "NULL argument");
    SCC_REQUIRE(s->n == g->n, SCC_ERR_INVALID, "state and graph differ in size");
    SCC_REQUIRE(n_ins >= 0 && n_del >= 0, SCC_ERR_INVALID, "negative batch size");
    SCC_REQUIRE((n_ins == 0 || (ins_src && ins_dst)) && (n_del == 0 || (del_src && del_dst)), SCC_ERR_INVALID,
                "NULL batch arrays");
    SCC_REQUIRE(g->m + n_ins < (1LL << 31) - 1, SCC_ERR_INVALID, "edge count would exceed int32");
    SCC_CUDA(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    scc_update_stats out;
    memset(&out, 0, sizeof(out));
    SCC_CUDA(cudaEventRecord(s->ev[8], st));
    int32_t n = g->n;
    // batch to the device
    DevBuf d_is, d_id, d_ds, d_dd, bad;
    const int32_t *is = ins_src, *id = ins_dst, *ds = del_src, *dd = del_dst;
    if (!on_device) {
        SCC_TRY(alloc(d_is, sizeof(int32_t) * (size_t)n_ins, st)); SCC_TRY(alloc(d_id, sizeof(int32_t) * (size_t)n_ins, st));
        SCC_TRY(alloc(d_ds, sizeof(int32_t) * (size_t)n_del, st)); SCC_TRY(alloc(d_dd, sizeof(int32_t) * (size_t)n_del, st));
        if (n_ins) {
            SCC_CUDA(cudaMemcpyAsync(d_is.p, ins_src, sizeof(int32_t) * (size_t)n_ins, cudaMemcpyHostToDevice, st));
            SCC_CUDA(cudaMemcpyAsync(d_id.p, ins_dst, sizeof(int32_t) * (size_t)n_ins, cudaMemcpyHostToDevice, st));
        }
        if (n_del) {
            SCC_CUDA(cudaMemcpyAsync(d_ds.p, del_src, sizeof(int32_t) * (size_t)n_del, cudaMemcpyHostToDevice, st));
            SCC_CUDA(cudaMemcpyAsync(d_dd.p, del_dst, sizeof(int32_t) * (size_t)n_del, cudaMemcpyHostToDevice, st));
        }
        is = d_is.as<int32_t>(); id = d_id.as<int32_t>(); ds = d_ds.as<int32_t>(); dd = d_dd.as<int32_t>();
    }
    SCC_TRY(alloc(bad, sizeof(int), st));
    SCC_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(int), st));
    BatchKeys keys;
    SCC_TRY(sort_batch(keys, n_ins, is, id, n_del, ds, dd, n, st, bad.as<int>()));
    int hbad = 0;
    SCC_CUDA(cudaMemcpyAsync(&hbad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SCC_CUDA(cudaStreamSynchronize(st));
    SCC_REQUIRE(!hbad, SCC_ERR_INVALID, "batch edge endpoint outside [0, %d)", n);

    // 1. CSR merge, both sides
    SCC_TRY(merge_batch(g, keys.del, keys.del_t, n_del, keys.ins, keys.ins_t, n_ins, st));
    SCC_CUDA(cudaEventRecord(s->ev[9], st));

    // 2. deletions: re-decompose the SCCs that lost an internal edge
    int32_t* flag = reinterpret_cast<int32_t*>(s->cnt);   // scratch, n ints: the peel residue is gone
    s->cnt_valid = false;
    if (n_del > 0) {
        k_upd_fill<<<scc_blocks(n), SCC_THREADS, 0, st>>>(n, flag, 0);
        SCC_LAUNCHED(s);
        k_upd_flag_split<<<scc_blocks(n_del), SCC_THREADS, 0, st>>>(n_del, keys.del, s->scc, flag);
        SCC_LAUNCHED(s);
        SCC_TRY(scc_zero_counters(s, CTR_SPARE0, 1));
        k_upd_colour_flagged<<<scc_blocks(n), SCC_THREADS, 0, st>>>(n, s->scc, flag, s->color, s->ctr + CTR_SPARE0);
        SCC_LAUNCHED(s);
        SCC_TRY(scc_sync_counters(s));
        out.affected_delete = s->h_ctr[CTR_SPARE0];
        if (out.affected_delete > 0) SCC_TRY(resolve_update(g, s));
    }
    SCC_CUDA(cudaEventRecord(s->ev[10], st));

    // 3. insertions: recompute inside R = FW(targets) & BW(sources) of cross-class inserted edges
    if (n_ins > 0) {
        // every vertex one traversal class
        k_upd_fill<<<scc_blocks(n), SCC_THREADS, 0, st>>>(n, s->color, 0);
        SCC_LAUNCHED(s);
        SCC_CUDA(cudaMemsetAsync(s->mark, 0, (size_t)((n + 4) & ~3LL), st));
        SCC_TRY(scc_zero_counters(s, CTR_QLEN, 1));
        k_upd_seed_region<<<scc_blocks(n_ins), SCC_THREADS, 0, st>>>(n_ins, keys.ins, s->scc,
                                                                     s->mark, s->qa, s->ctr + CTR_QLEN);
        SCC_LAUNCHED(s);
        SCC_TRY(scc_sync_counters(s));
        int32_t qlen = s->h_ctr[CTR_QLEN];
        if (qlen > 0) {
            // traversal over all vertices: the live list is every vertex
            SCC_TRY(scc_impl_compact_live(g, s, true));
            RoundArgs a = update_round_args(g, s);
            bool taken = false;
            ReachStart start;
            SCC_TRY(scc_impl_round_coop(g, s, a, COOP_REACH, true, false, &taken, &qlen, &start));
            if (!taken) {
                qlen = s->h_ctr[CTR_QLEN];
                *reinterpret_cast<unsigned long long*>(s->h_ctr + CTR_LIVE_EDGES) = 2ull * (unsigned long long)g->m;
                s->h_ctr[CTR_MAXDEG] = INT32_MAX;      // degrees not scanned here: no shortcut to the drain
            }
            if (qlen > 0) SCC_TRY(scc_impl_reach(g, s, a, qlen, taken ? &start : nullptr));
            SCC_TRY(scc_zero_counters(s, CTR_SPARE0, 1));
            k_upd_colour_region<<<scc_blocks(n), SCC_THREADS, 0, st>>>(n, s->mark, s->color, s->ctr + CTR_SPARE0);
            SCC_LAUNCHED(s);
            SCC_TRY(scc_sync_counters(s));
            out.affected_insert = s->h_ctr[CTR_SPARE0];
            s->fresh = false;
            s->prefinished = false;
            s->live_count = -1;
            if (out.affected_insert > 0) SCC_TRY(resolve_update(g, s));
        } else {
            k_upd_fill<<<scc_blocks(n), SCC_THREADS, 0, st>>>(n, s->color, SCC_COLOR_DONE);
            SCC_LAUNCHED(s);
        }
    }
    SCC_CUDA(cudaEventRecord(s->ev[11], st));
    SCC_CUDA(cudaStreamSynchronize(st));
    SCC_TRY(scc_check_device_error(s));
    out.ms_merge = ev_ms(s->ev[8], s->ev[9]);
    out.ms_delete = ev_ms(s->ev[9], s->ev[10]);
    out.ms_insert = ev_ms(s->ev[10], s->ev[11]);
    out.ms_total = ev_ms(s->ev[8], s->ev[11]);
    out.m_after = g->m;
    int32_t k = 0;
    SCC_TRY(scc_count_sccs(s, &k));
    out.num_sccs = k;
    if (stats) *stats = out;
    return SCC_OK;
}

extern "C" int scc_incremental_insert(scc_graph* g, scc_state* s, int64_t n_ins, const int32_t* src,
                                      const int32_t* dst, scc_update_stats* stats) {
    return scc_update_batch(g, s, n_ins, src, dst, 0, nullptr, nullptr, 0, stats);
}

extern "C" int scc_decremental_delete(scc_graph* g, scc_state* s, int64_t n_del, const int32_t* src,
                                      const int32_t* dst, scc_update_stats* stats) {
    return scc_update_batch(g, s, 0, nullptr, nullptr, n_del, src, dst, 0, stats);
}

// insert_idea1 (src/scc_incremental.cc:7-17): the graph plus the inserted
// edges, decomposed from scratch (method 5).
extern "C" int scc_insert_idea1(scc_graph* g, scc_state* s, int64_t n_ins, const int32_t* src, const int32_t* dst,
                                scc_run_stats* stats) {
    SCC_REQUIRE(g && s, SCC_ERR_INVALID, "NULL argument");
    SCC_REQUIRE(n_ins >= 0 && (n_ins == 0 || (src && dst)), SCC_ERR_INVALID, "bad batch");
    SCC_REQUIRE(g->m + n_ins < (1LL << 31) - 1, SCC_ERR_INVALID, "edge count would exceed int32");
    SCC_CUDA(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    DevBuf d_s, d_d, bad;
    BatchKeys keys;
    SCC_TRY(alloc(d_s, sizeof(int32_t) * (size_t)n_ins, st)); SCC_TRY(alloc(d_d, sizeof(int32_t) * (size_t)n_ins, st));
    if (n_ins) {
        SCC_CUDA(cudaMemcpyAsync(d_s.p, src, sizeof(int32_t) * (size_t)n_ins, cudaMemcpyHostToDevice, st));
        SCC_CUDA(cudaMemcpyAsync(d_d.p, dst, sizeof(int32_t) * (size_t)n_ins, cudaMemcpyHostToDevice, st));
    }
    SCC_TRY(alloc(bad, sizeof(int), st));
    SCC_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(int), st));
    SCC_TRY(sort_batch(keys, n_ins, d_s.as<int32_t>(), d_d.as<int32_t>(), 0, nullptr, nullptr, g->n, st,
                       bad.as<int>()));
    int hbad = 0;
    SCC_CUDA(cudaMemcpyAsync(&hbad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SCC_CUDA(cudaStreamSynchronize(st));
    SCC_REQUIRE(!hbad, SCC_ERR_INVALID, "inserted edge endpoint outside [0, %d)", g->n);
    SCC_TRY(merge_batch(g, keys.del, keys.del_t, 0, keys.ins, keys.ins_t, n_ins, st));
    SCC_TRY(scc_state_reset(s));
    return scc_run(g, s, SCC_METHOD_GLOBAL_WCC_FB, SCC_PIVOT_DEGREE, stats);
}

// create_scc_edges + insert_idea2 (src/common_main.h:180-314,
// src/scc_incremental.cc:19-27): the condensation graph over the SCC ids of
// `labels` (ids < num_sccs), with every cross-SCC edge of g and of the
// inserted batch mapped to (id(u), id(v)); duplicates dropped.
// Condensation edges (create_scc_edges, src/common_main.h:180-314): every
// edge (u, v) becomes (label[u], label[v]); pairs inside one SCC would be
// self-loops the build drops, so only cross-SCC pairs are written, appended
// to a compact list.  Edge-balanced: a block takes COND_CHUNK consecutive
// edges, stages the offsets and labels of the vertices owning them in shared
// memory, and each thread finds its edges' sources there by binary search.
// Adjacency is streamed (evict-first) so the label array stays in L2 for
// the random destination gathers.
#define COND_ITEMS 8
#define COND_CHUNK (SCC_THREADS * COND_ITEMS)
#define COND_TILE_V COND_CHUNK

// largest v in [lo, hi] with off[v] <= k (off[lo] <= k)
__device__ __forceinline__ int32_t cond_owner(const int32_t* off, int32_t lo, int32_t hi, int32_t k) {
    while (lo < hi) {
        int32_t mid = lo + ((hi - lo + 1) >> 1);
        if (off[mid] <= k) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// owner[c] = source vertex of edge c * COND_CHUNK; owner[chunks] = n - 1
__global__ void k_cond_owners(int32_t n, int64_t chunks, const int32_t* __restrict__ off, int32_t* __restrict__ owner) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c <= chunks; c += (int64_t)gridDim.x * blockDim.x)
        owner[c] = c == chunks ? n - 1 : cond_owner(off, 0, n - 1, (int32_t)(c * COND_CHUNK));
}

__global__ void k_cond_check_labels(int32_t n, const int32_t* __restrict__ label, int32_t num_sccs, int* __restrict__ bad) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        int32_t l = label[v];
        if (l < 0 || l >= num_sccs) atomicExch(bad, 1);
    }
}

__global__ void __launch_bounds__(SCC_THREADS) k_cond_cross(int32_t m, int64_t chunks, const int32_t* __restrict__ off,
                                                            const int32_t* __restrict__ adj,
                                                            const int32_t* __restrict__ label,
                                                            const int32_t* __restrict__ owner,
                                                            int32_t* __restrict__ out_src, int32_t* __restrict__ out_dst,
                                                            int32_t* __restrict__ count) {
    __shared__ int32_t scan_w[SCC_THREADS / 32];
    __shared__ int32_t s_off[COND_TILE_V + 1];
    __shared__ int32_t s_lab[COND_TILE_V];
    __shared__ int32_t s_base;
    const bool vec = (((uintptr_t)adj) & 15) == 0;
    for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int32_t e0 = (int32_t)(c * COND_CHUNK);
        const int32_t e1 = (int32_t)min((int64_t)m, (c + 1) * COND_CHUNK);
        const int32_t vs = owner[c], hi = owner[c + 1];   // every source of the chunk lies in [vs, hi]
        const int32_t nv = hi - vs + 1;
        const bool tiled = nv <= COND_TILE_V;
        if (tiled) {
            for (int i = threadIdx.x; i <= nv; i += SCC_THREADS) s_off[i] = off[vs + i];
            for (int i = threadIdx.x; i < nv; i += SCC_THREADS) s_lab[i] = label[vs + i];
        }
        const int32_t k0 = e0 + threadIdx.x * COND_ITEMS;
        int32_t d[COND_ITEMS];
        if (vec && k0 + COND_ITEMS <= e1) {
#pragma unroll
            for (int j = 0; j < COND_ITEMS; j += 4) {
                int4 q = __ldcs((const int4*)(adj + k0 + j));
                d[j] = q.x; d[j + 1] = q.y; d[j + 2] = q.z; d[j + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < COND_ITEMS; j++) d[j] = k0 + j < e1 ? __ldcs(adj + k0 + j) : 0;
        }
#pragma unroll
        for (int j = 0; j < COND_ITEMS; j++) d[j] = k0 + j < e1 ? __ldg(label + d[j]) : 0;
        __syncthreads();
        int32_t sl[COND_ITEMS];
        int keep = 0;
        if (k0 < e1) {
            if (tiled) {
                int32_t i = cond_owner(s_off, 0, nv - 1, k0);
#pragma unroll
                for (int j = 0; j < COND_ITEMS; j++) {
                    sl[j] = 0;
                    if (k0 + j < e1) {   // off[hi + 1] > k0 + j stops the walk inside the tile
                        while (s_off[i + 1] <= k0 + j) i++;
                        sl[j] = s_lab[i];
                    }
                }
            } else {
                int32_t v = cond_owner(off, vs, hi, k0);
#pragma unroll
                for (int j = 0; j < COND_ITEMS; j++) {
                    sl[j] = 0;
                    if (k0 + j < e1) {
                        while (v < hi && off[v + 1] <= k0 + j) v++;
                        sl[j] = label[v];
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < COND_ITEMS; j++)
                if (k0 + j < e1 && sl[j] != d[j]) keep |= 1 << j;
        }
        int32_t total = 0;
        const int32_t pre = scc_block_excl_sum256(__popc(keep), scan_w, &total);
        if (threadIdx.x == 0 && total > 0) s_base = atomicAdd(count, total);
        __syncthreads();
        if (keep) {
            int32_t at = s_base + pre;
#pragma unroll
            for (int j = 0; j < COND_ITEMS; j++)
                if (keep & (1 << j)) { out_src[at] = sl[j]; out_dst[at] = d[j]; at++; }
        }
        __syncthreads();   // shared tiles and scan storage are reused
    }
}

// inserted pairs (insert_idea2, src/scc_incremental.cc:18-27) mapped through
// the labels and appended when they join two SCCs
__global__ void k_cond_batch(int64_t k, const int32_t* __restrict__ a, const int32_t* __restrict__ b,
                             const int32_t* __restrict__ label, int32_t n, int32_t* __restrict__ out_src,
                             int32_t* __restrict__ out_dst, int32_t* __restrict__ count, int* __restrict__ bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t x = a[i], y = b[i];
        if (x < 0 || x >= n || y < 0 || y >= n) { atomicExch(bad, 1); continue; }
        int32_t lx = label[x], ly = label[y];
        if (lx == ly) continue;
        int32_t at = atomicAdd(count, 1);
        out_src[at] = lx;
        out_dst[at] = ly;
    }
}

extern "C" int scc_condensation_graph(const scc_graph* g, const int32_t* labels, int32_t num_sccs, int64_t n_ins,
                                      const int32_t* ins_src, const int32_t* ins_dst, scc_graph** out) {
    SCC_REQUIRE(g && labels && out && num_sccs >= 0, SCC_ERR_INVALID, "NULL argument");
    SCC_REQUIRE(n_ins == 0 || (ins_src && ins_dst), SCC_ERR_INVALID, "NULL batch arrays");
    SCC_REQUIRE(n_ins >= 0 && g->m + n_ins < (1LL << 31) - 1, SCC_ERR_INVALID, "batch of %lld edges too large",
                (long long)n_ins);
    SCC_CUDA(cudaSetDevice(g->device));
    cudaStream_t st;
    SCC_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    const int64_t total = g->m + n_ins;
    const int64_t chunks = (g->m + COND_CHUNK - 1) / COND_CHUNK;
    int rc = SCC_OK;
    {   // buffers are freed on `st` before it is destroyed
    DevBuf lab, osrc, odst, own, bs, bd, ctr;
    if ((rc = alloc(lab, sizeof(int32_t) * (size_t)g->n, st)) == SCC_OK &&
        (rc = alloc(osrc, sizeof(int32_t) * (size_t)total, st)) == SCC_OK &&
        (rc = alloc(odst, sizeof(int32_t) * (size_t)total, st)) == SCC_OK &&
        (rc = alloc(own, sizeof(int32_t) * (size_t)(chunks + 1), st)) == SCC_OK &&
        (rc = alloc(bs, sizeof(int32_t) * (size_t)n_ins, st)) == SCC_OK &&
        (rc = alloc(bd, sizeof(int32_t) * (size_t)n_ins, st)) == SCC_OK &&
        (rc = alloc(ctr, 2 * sizeof(int), st)) == SCC_OK) {
        int* bad = ctr.as<int>();
        int32_t* count = ctr.as<int32_t>() + 1;
        cudaMemsetAsync(ctr.p, 0, 2 * sizeof(int), st);
        cudaMemcpyAsync(lab.p, labels, sizeof(int32_t) * (size_t)g->n, cudaMemcpyHostToDevice, st);
        if (g->n > 0)
            k_cond_check_labels<<<scc_blocks(g->n, SCC_THREADS, 148 * 8), SCC_THREADS, 0, st>>>(
                g->n, lab.as<int32_t>(), num_sccs, bad);
        if (g->m > 0) {
            k_cond_owners<<<scc_blocks(chunks + 1), SCC_THREADS, 0, st>>>(g->n, chunks, g->begin, own.as<int32_t>());
            // one resident wave: a grid-stride loop over chunks with a second
            // wave would leave its blocks a full share of chunks to run late
            int sms = 148, per = 1;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cond_cross, SCC_THREADS, 0);
            k_cond_cross<<<(unsigned)std::min<int64_t>(chunks, (int64_t)sms * std::max(per, 1)), SCC_THREADS, 0, st>>>(
                (int32_t)g->m, chunks, g->begin, g->node_idx, lab.as<int32_t>(), own.as<int32_t>(),
                osrc.as<int32_t>(), odst.as<int32_t>(), count);
        }
        if (n_ins > 0) {
            cudaMemcpyAsync(bs.p, ins_src, sizeof(int32_t) * (size_t)n_ins, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(bd.p, ins_dst, sizeof(int32_t) * (size_t)n_ins, cudaMemcpyHostToDevice, st);
            k_cond_batch<<<scc_blocks(n_ins), SCC_THREADS, 0, st>>>(n_ins, bs.as<int32_t>(), bd.as<int32_t>(),
                                                                    lab.as<int32_t>(), g->n, osrc.as<int32_t>(),
                                                                    odst.as<int32_t>(), count, bad);
        }
        int h[2] = {0, 0};
        cudaError_t e = cudaPeekAtLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h, ctr.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = scc_cuda_status(e, "condensation map", __FILE__, __LINE__);
        else if (h[0]) { scc_set_error("label or inserted endpoint out of range"); rc = SCC_ERR_INVALID; }
        else rc = scc_impl_build_graph_from_device_edges(num_sccs, h[1], osrc.as<int32_t>(), odst.as<int32_t>(),
                                                         SCC_BUILD_DEDUP | SCC_BUILD_NO_SELF_LOOPS, g->device, out);
    }
    }
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return rc;
}
