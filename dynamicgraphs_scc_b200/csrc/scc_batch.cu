// Batched decomposition of many independent small graphs in ONE persistent
// launch: each block takes whole graphs from a device counter (largest
// first) and runs the complete method on each inside the block -- a first
// round of FW-BW from one pivot with its marks in shared memory, then Trim1 to the
// fixpoint and rounds of pivot / FW+BW reachability / classify / peel
// over every class left of that graph at once (the structure of
// do_baseline_global_wcc_fb and start_workers_fw_bw, src/scc_main.cc:272-351,
// src/scc_fb_seq2.cc:292-351) -- with __syncthreads between the steps instead
// of kernel boundaries and host round trips.  One launch per batch, so the
// run is captured once into a CUDA graph and replayed with one host
// submission.  Blocks never wait on one another.
//
// Per graph g with vertices [lo, hi) the block uses only slices of the
// state's arrays: colour/scc/mark/counts [lo, hi), the queue [2lo, 2hi), the
// live lists [lo, hi).  Colours are globally unique without an allocator:
// the graph starts as one class of colour 3*lo, and the FW-only / BW-only
// parts of the class pivoted on p become 3p+1 / 3p+2 (a pivot is finished in
// its round, so it never pivots again).  The per-colour pivot key lives in an
// array indexed by colour (3N entries).
#include <algorithm>
#include "scc_round.cuh"
#include "scc_batch.cuh"
#include "scc_sort.cuh"

struct BatchArgs {
    const int32_t* begin; const int32_t* adj; const int32_t* rbegin; const int32_t* radj;
    const int32_t* offs;        // [G+1] vertex offsets of the graphs
    const int32_t* order;       // [G] graphs, largest first
    int32_t G;
    int32_t* color; int32_t* scc; uint8_t* mark;
    uint32_t* cin; uint32_t* cout;   // live in/out counts within the class
    int32_t* q;                 // [2N] queue slices
    int32_t* live; int32_t* live2;   // [N] live-list slices
    unsigned long long* key;    // [3N] pivot key per colour
    int32_t* ctr;               // BATCH_CTR_* counters
    int32_t warp_deg;           // lists longer than this are expanded by a whole warp
    const int32_t* members;     // class mode: unit k is members[offs[k] .. offs[k+1]); NULL: vertex ids
    int32_t marks_cap;          // graphs of at most this many vertices keep the first round's marks in shared memory
    int32_t vec_adj;            // both adjacency arrays start on a 16-byte boundary
    int64_t adj_len;            // their entries
};

__device__ __forceinline__ int32_t b_fw_colour(int32_t p) { return 3 * p + 1; }
__device__ __forceinline__ int32_t b_bw_colour(int32_t p) { return 3 * p + 2; }

// Warp-aggregated append of `item` (lanes with p) to q[base + tail++], tail in shared memory.
__device__ __forceinline__ void b_append(bool p, int32_t item, int32_t* q, int32_t* s_tail, int32_t cap,
                                         int32_t* err) {
    unsigned bal = __ballot_sync(0xFFFFFFFFu, p);
    if (!bal) return;
    int lane = threadIdx.x & 31;
    int32_t base = 0;
    if (lane == __ffs(bal) - 1) base = atomicAdd(s_tail, __popc(bal));
    base = __shfl_sync(0xFFFFFFFFu, base, __ffs(bal) - 1);
    if (p) {
        int32_t pos = base + __popc(bal & ((1u << lane) - 1u));
        if (pos < cap) q[pos] = item;
        else atomicExch(err, SCC_DEVERR_QUEUE_OVERFLOW);
    }
}

// Block-wide exclusive scan of one int per thread; returns the prefix, *total the sum.
__device__ __forceinline__ int32_t b_scan(int32_t x, int32_t* s_warp, int32_t* total) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int32_t inc = x;
    for (int o = 1; o < 32; o <<= 1) {
        int32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int32_t w = lane < nw ? s_warp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) s_warp[lane] = w;       // inclusive warp totals
    }
    __syncthreads();
    int32_t before = (wid > 0 ? s_warp[wid - 1] : 0) + inc - x;
    *total = s_warp[nw - 1];
    __syncthreads();
    return before;
}

// ------------------------------------------------------------------ peel
// Counts of same-class neighbours (self-loops excluded) of every live vertex;
// vertices with a zero count are trimmed and queued with their class.
__device__ void b_count_and_seed(const BatchArgs& a, const int32_t* live, int32_t nlive, int32_t* q, int32_t* qc,
                                 int32_t* s_tail, int32_t cap) {
    const int lane = threadIdx.x & 31;
    const int nwarps = blockDim.x >> 5, wid = threadIdx.x >> 5;
    for (int32_t base = wid * 32; base < nlive; base += nwarps * 32) {
        int32_t i = base + lane;
        bool valid = i < nlive;
        int32_t v = valid ? live[i] : 0;
        int32_t c = valid ? a.color[v] : SCC_COLOR_DONE;
        uint32_t cnt[2] = {0u, 0u};
        for (int side = 0; side < 2; ++side) {
            const int32_t* off = side ? a.rbegin : a.begin;
            const int32_t* adj = side ? a.radj : a.adj;
            int32_t b = valid ? __ldg(off + v) : 0, e = valid ? __ldg(off + v + 1) : 0;
            int32_t deg = e - b;
            unsigned big = __ballot_sync(0xFFFFFFFFu, deg > a.warp_deg);
            while (big) {
                int l = __ffs(big) - 1;
                big &= big - 1;
                int32_t lb = __shfl_sync(0xFFFFFFFFu, b, l), le = __shfl_sync(0xFFFFFFFFu, e, l);
                int32_t lv = __shfl_sync(0xFFFFFFFFu, v, l), lc = __shfl_sync(0xFFFFFFFFu, c, l);
                uint32_t k = 0;
                for (int32_t j = lb + lane; j < le; j += 32) {
                    int32_t w = __ldg(adj + j);
                    k += (w != lv && a.color[w] == lc) ? 1u : 0u;
                }
                for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(0xFFFFFFFFu, k, o);
                if (lane == l) cnt[side] = k;
            }
            if (deg <= a.warp_deg && c != SCC_COLOR_DONE) {
                uint32_t k = 0;
                for (int32_t j = b; j < e; ++j) {
                    int32_t w = __ldg(adj + j);
                    k += (w != v && a.color[w] == c) ? 1u : 0u;
                }
                cnt[side] = k;
            }
        }
        if (valid && c != SCC_COLOR_DONE) { a.cout[v] = cnt[0]; a.cin[v] = cnt[1]; }
    }
    __syncthreads();
    for (int32_t base = wid * 32; base < nlive; base += nwarps * 32) {
        int32_t i = base + lane;
        bool p = false;
        int32_t v = 0, c = 0;
        if (i < nlive) {
            v = live[i];
            c = a.color[v];
            if (c != SCC_COLOR_DONE && (a.cin[v] == 0u || a.cout[v] == 0u) && atomicCAS(a.color + v, c, SCC_COLOR_DONE) == c) {
                a.scc[v] = v;
                p = true;
            }
        }
        // the queue holds the vertex; its class goes to the parallel slot
        unsigned bal = __ballot_sync(0xFFFFFFFFu, p);
        if (bal) {
            int32_t base2 = 0;
            if (lane == __ffs(bal) - 1) base2 = atomicAdd(s_tail, __popc(bal));
            base2 = __shfl_sync(0xFFFFFFFFu, base2, __ffs(bal) - 1);
            if (p) {
                int32_t pos = base2 + __popc(bal & ((1u << lane) - 1u));
                if (pos < cap) { q[pos] = v; qc[pos] = c; }
                else atomicExch(a.ctr + BATCH_CTR_ERROR, SCC_DEVERR_QUEUE_OVERFLOW);
            }
        }
    }
    __syncthreads();
}

// The trimmed vertex x (class c) leaves its neighbours' counts; a count that
// reaches zero trims that neighbour (once: the colour CAS decides).
__device__ __forceinline__ bool b_peel_edge(const BatchArgs& a, int32_t w, int32_t x, int32_t c, int side) {
    if (w == x || a.color[w] != c) return false;
    uint32_t* cnt = side ? a.cout : a.cin;     // x's out-edge costs w an in-neighbour, and the reverse
    if (atomicSub(cnt + w, 1u) != 1u) return false;
    if (atomicCAS(a.color + w, c, SCC_COLOR_DONE) != c) return false;
    a.scc[w] = w;
    return true;
}

__device__ void b_peel(const BatchArgs& a, int32_t* q, int32_t* qc, int32_t* s_tail, int32_t cap) {
    const int lane = threadIdx.x & 31;
    const int nwarps = blockDim.x >> 5, wid = threadIdx.x >> 5;
    int32_t h = 0;
    while (true) {
        int32_t t = *s_tail;
        if (t > cap) t = cap;
        __syncthreads();          // every warp has read the tail before one appends
        if (h >= t) break;
        for (int32_t base = h + wid * 32; base < t; base += nwarps * 32) {
            int32_t i = base + lane;
            bool valid = i < t;
            int32_t x = valid ? q[i] : 0, c = valid ? qc[i] : 0;
            for (int side = 0; side < 2; ++side) {
                const int32_t* off = side ? a.rbegin : a.begin;
                const int32_t* adj = side ? a.radj : a.adj;
                int32_t b = valid ? __ldg(off + x) : 0, e = valid ? __ldg(off + x + 1) : 0;
                int32_t deg = e - b;
                unsigned big = __ballot_sync(0xFFFFFFFFu, deg > a.warp_deg);
                while (big) {
                    int l = __ffs(big) - 1;
                    big &= big - 1;
                    int32_t lb = __shfl_sync(0xFFFFFFFFu, b, l), le = __shfl_sync(0xFFFFFFFFu, e, l);
                    int32_t lx = __shfl_sync(0xFFFFFFFFu, x, l), lc = __shfl_sync(0xFFFFFFFFu, c, l);
                    for (int32_t j0 = lb; j0 < le; j0 += 32) {
                        int32_t j = j0 + lane;
                        int32_t w = j < le ? __ldg(adj + j) : lx;
                        bool p = j < le && b_peel_edge(a, w, lx, lc, side);
                        unsigned bal = __ballot_sync(0xFFFFFFFFu, p);
                        if (bal) {
                            int32_t pos0 = 0;
                            if (lane == __ffs(bal) - 1) pos0 = atomicAdd(s_tail, __popc(bal));
                            pos0 = __shfl_sync(0xFFFFFFFFu, pos0, __ffs(bal) - 1);
                            if (p) {
                                int32_t pos = pos0 + __popc(bal & ((1u << lane) - 1u));
                                if (pos < cap) { q[pos] = w; qc[pos] = lc; }
                                else atomicExch(a.ctr + BATCH_CTR_ERROR, SCC_DEVERR_QUEUE_OVERFLOW);
                            }
                        }
                    }
                }
                if (valid && deg <= a.warp_deg) {
                    for (int32_t j = b; j < e; ++j) {
                        int32_t w = __ldg(adj + j);
                        if (b_peel_edge(a, w, x, c, side)) {
                            int32_t pos = atomicAdd(s_tail, 1);
                            if (pos < cap) { q[pos] = w; qc[pos] = c; }
                            else atomicExch(a.ctr + BATCH_CTR_ERROR, SCC_DEVERR_QUEUE_OVERFLOW);
                        }
                    }
                }
            }
        }
        h = t;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ a graph's first round
// A whole graph is one class, so its first FW-BW round needs no colours: mark
// bytes in shared memory replace the marks and the colour gathers in global
// memory, and the round comes before the peel, which then only sees what the
// round left.  Narrow frontiers are expanded top down from the queue; from a
// quarter of the vertices on, a sweep over all vertices takes over, whose
// offsets and lists are read in order.  Bound by the barriers and the round trips
// of its levels, and by instruction issue (44 % of the slots on 512 graphs; DRAM
// 1.49 TB/s).
// 4,096 graphs, 63.8 M vertices, 383 M edges, default shape: 23.7 ms with
// colours and marks in global memory and the peel first, 3.35 ms so (3.7 without
// B_LEAF; then, sweeps from a sixteenth on 3.8 ms, from half on 4.4 ms).
#define B_MARKS_MAX (200 * 1024) // vertices of the largest graph whose marks are kept so, a byte each
#define B_BLOCK_DEG 512          // top-down lists longer than this are expanded by the whole block
#define B_BIG 64                 // such items one level sets aside (further ones: by their warp)
#define B_SWEEP 4                // sweep once the frontier (both directions) is this share of the vertices not reached
#define B_STEP 8                 // entries of a short list claimed together
#define B_PROBES 8               // two-chunk probes a lane makes alone before the warp takes the list

// A vertex without out- or without in-edges is a component by itself and on no path
// between others; the pass that finds the pivot sees its degrees and sets it aside.  Without
// this, batches of acyclic and very sparse graphs paid for the first round on top of the
// peel: 5,000 random graphs of 1,000 vertices and 500 edges 0.72 ms, 0.61 with the peel first,
// 0.53 so; 1,000 binary trees of 8,191 0.64, 0.55 and 0.43; the batch below 3.35 ms.
#define B_LEAF 4u

struct FirstRound {
    volatile uint8_t* marks;     // of vertex lo + i: bit 0 FW reached, bit 1 BW reached, B_LEAF
    int32_t lo, ng;
};

// An id outside the graph (a batch whose graphs are not closed) is not claimed.
__device__ __forceinline__ bool b_claim(const FirstRound& r, int dir, int32_t u) {
    const uint32_t i = (uint32_t)(u - r.lo), bit = 1u << dir;
    if (i >= (uint32_t)r.ng || (r.marks[i] & (bit | B_LEAF))) return false;
    const uint32_t sh = (i & 3u) * 8u;
    return !((atomicOr(reinterpret_cast<uint32_t*>(const_cast<uint8_t*>(r.marks) + (i & ~3u)), bit << sh) >> sh) & bit);
}

// Is one of the four entries u at adj[c], ... that lie in [k, e) reached (bit of its mark)?
__device__ __forceinline__ bool b_hit4(const FirstRound& r, uint32_t bit, const int4& u, int32_t c, int32_t k, int32_t e) {
    const int32_t x[4] = {u.x, u.y, u.z, u.w};
    uint32_t m = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t i = (uint32_t)(x[j] - r.lo);
        if ((uint32_t)(c + j - k) < (uint32_t)(e - k) && i < (uint32_t)r.ng) m |= r.marks[i];
    }
    return m & bit;
}

__device__ __forceinline__ int4 b_load4(const BatchArgs& a, const int32_t* __restrict__ adj, int32_t c) {
    if (a.vec_adj && (int64_t)c + 4 <= a.adj_len) return __ldg(reinterpret_cast<const int4*>(adj + c));
    int4 x;      // the array's last entries, or arrays that are not 16-byte aligned
    x.x = c < a.adj_len ? __ldg(adj + c) : 0;
    x.y = c + 1 < a.adj_len ? __ldg(adj + c + 1) : 0;
    x.z = c + 2 < a.adj_len ? __ldg(adj + c + 2) : 0;
    x.w = c + 3 < a.adj_len ? __ldg(adj + c + 3) : 0;
    return x;
}

// Lists still open after a lane's own probes, by the whole warp, 32 entries at a time.
__device__ __forceinline__ bool b_probe_long(const FirstRound& r, uint32_t bit, const int32_t* __restrict__ adj,
                                             int32_t k, int32_t e) {
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    bool hit = false;
    unsigned open = __ballot_sync(full, k < e);
    while (open) {
        const int l = __ffs(open) - 1;
        open &= open - 1;
        const int32_t lk = __shfl_sync(full, k, l), le = __shfl_sync(full, e, l);
        bool found = false;
        for (int32_t j0 = lk; j0 < le && !found; j0 += 32) {
            const int32_t j = j0 + lane;
            const uint32_t i = j < le ? (uint32_t)(__ldg(adj + j) - r.lo) : UINT32_MAX;
            found = __any_sync(full, i < (uint32_t)r.ng && (r.marks[i] & bit));
        }
        if (lane == l) hit = found;
    }
    return hit;
}

// One sweep over the n vertices of `list` (places in the graph; NULL: all of
// them): each one not yet reached looks for a reached in-neighbour (FW) and a
// reached out-neighbour (BW); what it finds joins the queue, and the vertices still
// not reached both ways are listed in `open` for the next sweep, so a sweep
// costs what the one before it left.  A lane per vertex, two aligned int4
// chunks of each direction's list in flight at once (a list of six entries is
// then done in one round trip after its offsets), a list left at its first hit.
// Bound by the round trips of a vertex's loads and by instruction issue.  On the
// batch named above (before B_LEAF): 3.7 ms; all vertices in every sweep 4.4 ms; the
// lists of 32 vertices read end to end, a row of 32 entries at a time 5.7 ms; one
// chunk and one direction at a time 7.1 ms.
__device__ void b_sweep(const BatchArgs& a, const FirstRound& r, const int32_t* list, int32_t n, int32_t* open,
                        int32_t* s_open, int32_t* q, int32_t* s_tail) {
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    for (int32_t at0 = (int32_t)threadIdx.x - lane; at0 < n; at0 += (int32_t)blockDim.x) {
        const bool in = at0 + lane < n;
        const int32_t i = !in ? 0 : list ? list[at0 + lane] : at0 + lane;
        const int32_t v = r.lo + i;
        uint32_t had = in ? r.marks[i] : 3u;
        if (had & B_LEAF) had = 3u;
        int32_t k0 = 0, e0 = 0, k1 = 0, e1 = 0;
        if (!(had & 1u)) { k0 = __ldg(a.rbegin + v); e0 = __ldg(a.rbegin + v + 1); }
        if (!(had & 2u)) { k1 = __ldg(a.begin + v); e1 = __ldg(a.begin + v + 1); }
        bool hit0 = false, hit1 = false;
        for (int t = 0; t < B_PROBES && (k0 < e0 || k1 < e1); ++t) {
            const int32_t c0 = k0 & ~3, c1 = k1 & ~3;
            int4 x0 = {0, 0, 0, 0}, x1 = x0, y0 = x0, y1 = x0;
            if (k0 < e0) x0 = b_load4(a, a.radj, c0);
            if (c0 + 4 < e0) x1 = b_load4(a, a.radj, c0 + 4);
            if (k1 < e1) y0 = b_load4(a, a.adj, c1);
            if (c1 + 4 < e1) y1 = b_load4(a, a.adj, c1 + 4);
            if (k0 < e0) {
                hit0 = b_hit4(r, 1u, x0, c0, k0, e0) || b_hit4(r, 1u, x1, c0 + 4, k0, e0);
                k0 = hit0 ? e0 : c0 + 8;
            }
            if (k1 < e1) {
                hit1 = b_hit4(r, 2u, y0, c1, k1, e1) || b_hit4(r, 2u, y1, c1 + 4, k1, e1);
                k1 = hit1 ? e1 : c1 + 8;
            }
        }
        __syncwarp();
        hit0 = b_probe_long(r, 1u, a.radj, k0, e0) || hit0;
        hit1 = b_probe_long(r, 2u, a.adj, k1, e1) || hit1;
        // the sweep alone writes marks now, each by its own lane
        const uint32_t now = had | (hit0 ? 1u : 0u) | (hit1 ? 2u : 0u);
        if (now != had) r.marks[i] = (uint8_t)now;
        const unsigned n0 = __ballot_sync(full, hit0), n1 = __ballot_sync(full, hit1), no = __ballot_sync(full, now != 3u);
        int32_t at = 0, oat = 0;
        if (lane == 0) {
            if (n0 | n1) at = atomicAdd(s_tail, __popc(n0) + __popc(n1));
            if (no) oat = atomicAdd(s_open, __popc(no));
        }
        at = __shfl_sync(full, at, 0);
        oat = __shfl_sync(full, oat, 0);
        // a vertex enters at most once per direction, so the queue never passes 2 ng
        if (hit0) q[at + __popc(n0 & lt)] = v;
        if (hit1) q[at + __popc(n0) + __popc(n1 & lt)] = v | (1 << DIR_SHIFT);
        if (now != 3u) open[oat + __popc(no & lt)] = i;
    }
}

// One top-down level: the items q[h, t).
__device__ void b_expand(const BatchArgs& a, const FirstRound& r, int32_t* q, int32_t h, int32_t t, int32_t* s_tail,
                         int32_t* s_big, int32_t* s_nbig, int32_t cap) {
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, wid = threadIdx.x >> 5;
    int32_t* err = a.ctr + BATCH_CTR_ERROR;
    for (int32_t base = h + wid * 32; base < t; base += nwarps * 32) {
        const int32_t i = base + lane;
        const bool valid = i < t;
        const int32_t it = valid ? q[i] : 0;
        const int32_t v = it & ITEM_MASK, dir = (it >> DIR_SHIFT) & 1;
        const int32_t* off = dir ? a.rbegin : a.begin;
        const int32_t b = valid ? __ldg(off + v) : 0;
        int32_t e = valid ? __ldg(off + v + 1) : 0;
        if (e - b > B_BLOCK_DEG) {
            const int32_t at = atomicAdd(s_nbig, 1);
            if (at < B_BIG) { s_big[at] = it; e = b; }
        }
        unsigned big = __ballot_sync(full, e - b > a.warp_deg);
        while (big) {
            const int l = __ffs(big) - 1;
            big &= big - 1;
            const int32_t lb = __shfl_sync(full, b, l), le = __shfl_sync(full, e, l), ld = __shfl_sync(full, dir, l);
            const int32_t* adj = ld ? a.radj : a.adj;
            for (int32_t j0 = lb; j0 < le; j0 += 32) {
                const int32_t j = j0 + lane;
                const int32_t u = j < le ? __ldg(adj + j) : 0;
                b_append(j < le && b_claim(r, ld, u), u | (ld << DIR_SHIFT), q, s_tail, cap, err);
            }
        }
        const int32_t mydeg = e - b <= a.warp_deg ? e - b : 0;
        const int32_t maxd = (int32_t)__reduce_max_sync(full, (unsigned)mydeg);
        const int32_t* adj = dir ? a.radj : a.adj;
        // eight entries of every lane's list at a time: loads, then claims, then one
        // append for all of them
        for (int32_t j0 = 0; j0 < maxd; j0 += B_STEP) {
            int32_t u[B_STEP];
            unsigned got[B_STEP];
            int32_t total = 0;
#pragma unroll
            for (int j = 0; j < B_STEP; ++j) u[j] = j0 + j < mydeg ? __ldg(adj + b + j0 + j) : 0;
#pragma unroll
            for (int j = 0; j < B_STEP; ++j) {
                got[j] = __ballot_sync(full, j0 + j < mydeg && b_claim(r, dir, u[j]));
                total += __popc(got[j]);
            }
            if (total == 0) continue;
            int32_t at = 0;
            if (lane == 0) at = atomicAdd(s_tail, total);
            at = __shfl_sync(full, at, 0);
            // claimed once per direction, so the queue never passes 2 ng
#pragma unroll
            for (int j = 0; j < B_STEP; ++j) {
                if ((got[j] >> lane) & 1u) q[at + __popc(got[j] & ((1u << lane) - 1u))] = u[j] | (dir << DIR_SHIFT);
                at += __popc(got[j]);
            }
        }
    }
    __syncthreads();
    const int32_t nbig = min(*s_nbig, B_BIG);
    for (int32_t x = 0; x < nbig; ++x) {
        const int32_t it = s_big[x], v = it & ITEM_MASK, dir = (it >> DIR_SHIFT) & 1;
        const int32_t* off = dir ? a.rbegin : a.begin;
        const int32_t* adj = dir ? a.radj : a.adj;
        const int32_t b = __ldg(off + v), e = __ldg(off + v + 1);
        for (int32_t j0 = b; j0 < e; j0 += (int32_t)blockDim.x) {
            const int32_t j = j0 + (int32_t)threadIdx.x;
            const int32_t u = j < e ? __ldg(adj + j) : 0;
            b_append(j < e && b_claim(r, dir, u), u | (dir << DIR_SHIFT), q, s_tail, cap, err);
        }
    }
}

// The first round of the graph [lo, lo + ng): colours and components of all its
// vertices are written, those it did not resolve are listed in live.  Returns
// their number.  s: 64 ints, s_big: B_BIG ints, marks: ng bytes rounded up to words.
__device__ int32_t b_first_round(const BatchArgs& a, int32_t lo, int32_t ng, int32_t c0, int32_t* s, int32_t* s_big,
                                 uint32_t* marks, int32_t* q, int32_t* live, int32_t* live2, int32_t* levels) {
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    int32_t* s_tail = s;
    int32_t* s_nbig = s + 1;
    unsigned long long* s_key = reinterpret_cast<unsigned long long*>(s + 2);
    int32_t* s_open = s + 4;
    FirstRound r;
    r.marks = reinterpret_cast<uint8_t*>(marks); r.lo = lo; r.ng = ng;
    for (int32_t i = threadIdx.x; i < (ng + 3) >> 2; i += blockDim.x) marks[i] = 0u;
    if (threadIdx.x == 0) { *s_key = 0ull; *s_nbig = 0; *s_open = 0; }
    __syncthreads();
    unsigned long long best = 0ull;
#pragma unroll 4
    for (int32_t i = threadIdx.x; i < ng; i += blockDim.x) {
        const unsigned long long k = pivot_key(a.begin, a.rbegin, lo + i);
        best = k > best ? k : best;
        if (k >> 32 == 1u) r.marks[i] = B_LEAF;          // in x out is 0
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(full, best, o);
        best = y > best ? y : best;
    }
    if (lane == 0) atomicMax(s_key, best);
    __syncthreads();
    const int32_t p = pivot_unhash((uint32_t)*s_key);
    if (threadIdx.x == 0) {
        r.marks[p - lo] = 3;
        q[0] = p;
        q[1] = p | (1 << DIR_SHIFT);
        *s_tail = 2;
    }
    __syncthreads();
    int32_t h = 0;
    const int32_t* list = nullptr;      // what the last sweep left open (NULL: no sweep yet)
    int32_t nopen = ng;
    while (true) {
        const int32_t t = min(*s_tail, 2 * ng);
        __syncthreads();          // every warp has read the tail before one appends
        if (h >= t) break;
        ++*levels;
        if ((t - h) * (int64_t)B_SWEEP >= nopen) {
            int32_t* out = list == live ? live2 : live;
            b_sweep(a, r, list, nopen, out, s_open, q, s_tail);
            __syncthreads();
            list = out;
            nopen = *s_open;
            __syncthreads();
            if (threadIdx.x == 0) *s_open = 0;
        } else {
            b_expand(a, r, q, h, t, s_tail, s_big, s_nbig, 2 * ng);
            __syncthreads();
            if (threadIdx.x == 0) *s_nbig = 0;
        }
        h = t;
        __syncthreads();
    }
    if (threadIdx.x == 0) *s_tail = 0;
    __syncthreads();
    for (int32_t i0 = threadIdx.x - lane; i0 < ng; i0 += blockDim.x) {
        const int32_t i = i0 + lane, v = lo + i;
        uint32_t m = i < ng ? r.marks[i] : 3u;
        const bool leaf = (m & B_LEAF) != 0u;
        if (leaf) m = 3u;
        if (i < ng) {
            a.scc[v] = m == 3u ? (leaf ? v : p) : SCC_NIL_NODE;
            a.color[v] = m == 3u ? SCC_COLOR_DONE : m == 1u ? b_fw_colour(p) : m == 2u ? b_bw_colour(p) : c0;
            if (m != 3u) a.mark[v] = 0;
        }
        b_append(m != 3u, v, live, s_tail, ng, a.ctr + BATCH_CTR_ERROR);
    }
    __syncthreads();
    const int32_t left = *s_tail;
    __syncthreads();
    return left;
}

// ------------------------------------------------------------------ one graph
__device__ void b_graph(const BatchArgs& a, int32_t gi, int32_t* s, int32_t* s_big, uint32_t* marks) {
    int32_t* s_tail = s;          // queue tail
    int32_t* s_warp = s + 32;     // scan scratch (32 ints)
    const int32_t lo = a.offs[gi], hi = a.offs[gi + 1];
    const int32_t ng = hi - lo;
    if (ng <= 0) return;
    int32_t* q = a.q + 2LL * lo;          // [2 ng]: peel queue (vertices | classes) or BFS items
    int32_t* live = a.live + lo;
    int32_t* live2 = a.live2 + lo;
    // one class per unit: colour 3 x its first vertex (a multiple of 3, so it
    // never meets the 3p+1 / 3p+2 colours of a pivot's parts)
    const int32_t c0 = 3 * (a.members ? a.members[lo] : lo);
    int32_t nlive = ng;
    int32_t rounds = 0, levels = 0;
    if (!a.members && ng <= a.marks_cap) {
        nlive = b_first_round(a, lo, ng, c0, s, s_big, marks, q, live, live2, &levels);
        rounds = 1;
    } else {
        for (int32_t i = threadIdx.x; i < ng; i += blockDim.x) {
            int32_t v = a.members ? a.members[lo + i] : lo + i;
            a.color[v] = c0;
            a.scc[v] = SCC_NIL_NODE;
            a.mark[v] = 0;
            live[i] = v;
        }
        __syncthreads();
    }
    while (nlive > 0) {
        // peel inside the classes
        if (threadIdx.x == 0) *s_tail = 0;
        __syncthreads();
        b_count_and_seed(a, live, nlive, q, q + ng, s_tail, ng);
        b_peel(a, q, q + ng, s_tail, ng);
        // compact the live list
        int32_t kept = 0;
        for (int32_t base = 0; base < nlive; base += blockDim.x) {
            int32_t i = base + threadIdx.x;
            int32_t v = i < nlive ? live[i] : 0;
            int32_t keep = (i < nlive && a.color[v] != SCC_COLOR_DONE) ? 1 : 0;
            int32_t tot = 0;
            int32_t pos = b_scan(keep, s_warp, &tot);
            if (keep) live2[kept + pos] = v;
            kept += tot;
        }
        { int32_t* t = live; live = live2; live2 = t; }
        nlive = kept;
        __syncthreads();
        if (nlive == 0) break;
        if (++rounds > ng + 2) {
            if (threadIdx.x == 0) atomicExch(a.ctr + BATCH_CTR_ERROR, SCC_DEVERR_WAIT_LIMIT);
            break;
        }
        // pivot of every class: largest in x out degree, ties by the id hash
        for (int32_t i = threadIdx.x; i < nlive; i += blockDim.x) a.key[a.color[live[i]]] = 0ull;
        __syncthreads();
        for (int32_t i = threadIdx.x; i < nlive; i += blockDim.x) {
            int32_t v = live[i];
            atomicMax(a.key + a.color[v], pivot_key(a.begin, a.rbegin, v));
        }
        __syncthreads();
        if (threadIdx.x == 0) *s_tail = 0;
        __syncthreads();
        for (int32_t base = 0; base < nlive; base += blockDim.x) {
            int32_t i = base + threadIdx.x;
            bool p = false;
            int32_t v = 0;
            if (i < nlive) {
                v = live[i];
                if (pivot_unhash((uint32_t)a.key[a.color[v]]) == v) { p = true; a.mark[v] = 3; }
            }
            b_append(p, v, q, s_tail, 2 * ng, a.ctr + BATCH_CTR_ERROR);
            b_append(p, v | (1 << DIR_SHIFT), q, s_tail, 2 * ng, a.ctr + BATCH_CTR_ERROR);
        }
        __syncthreads();
        // FW and BW of every class, level by level
        int32_t h = 0;
        const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, wid = threadIdx.x >> 5;
        while (true) {
            int32_t t = min(*s_tail, 2 * ng);
            __syncthreads();      // every warp has read the tail before one appends
            if (h >= t) break;
            ++levels;
            for (int32_t base = h + wid * 32; base < t; base += nwarps * 32) {
                int32_t i = base + lane;
                bool valid = i < t;
                int32_t it = valid ? q[i] : 0;
                int32_t v = it & ITEM_MASK, dir = (it >> DIR_SHIFT) & 1;
                const int32_t* off = dir ? a.rbegin : a.begin;
                int32_t b = valid ? __ldg(off + v) : 0, e = valid ? __ldg(off + v + 1) : 0;
                int32_t c = valid ? a.color[v] : 0;
                int32_t deg = e - b;
                unsigned big = __ballot_sync(0xFFFFFFFFu, deg > a.warp_deg);
                while (big) {
                    int l = __ffs(big) - 1;
                    big &= big - 1;
                    int32_t lb = __shfl_sync(0xFFFFFFFFu, b, l), le = __shfl_sync(0xFFFFFFFFu, e, l);
                    int32_t lc = __shfl_sync(0xFFFFFFFFu, c, l), ld = __shfl_sync(0xFFFFFFFFu, dir, l);
                    const int32_t* ladj = ld ? a.radj : a.adj;
                    const unsigned bit = 1u << ld;
                    for (int32_t j0 = lb; j0 < le; j0 += 32) {
                        int32_t j = j0 + lane;
                        bool p = false;
                        int32_t w = 0;
                        if (j < le) {
                            w = __ldg(ladj + j);
                            if (!(*(volatile uint8_t*)(a.mark + w) & bit) && a.color[w] == lc) {
                                unsigned sh = (unsigned)(w & 3) * 8u;
                                p = !((atomicOr(reinterpret_cast<unsigned*>(a.mark + (w & ~3)), bit << sh) >> sh) & bit);
                            }
                        }
                        b_append(p, w | (ld << DIR_SHIFT), q, s_tail, 2 * ng, a.ctr + BATCH_CTR_ERROR);
                    }
                }
                int32_t mydeg = (valid && deg <= a.warp_deg) ? deg : 0;
                int32_t maxd = (int32_t)__reduce_max_sync(0xFFFFFFFFu, (unsigned)mydeg);
                const int32_t* adj = dir ? a.radj : a.adj;
                const unsigned bit = 1u << dir;
                for (int32_t j = 0; j < maxd; ++j) {
                    bool p = false;
                    int32_t w = 0;
                    if (j < mydeg) {
                        w = __ldg(adj + b + j);
                        if (!(*(volatile uint8_t*)(a.mark + w) & bit) && a.color[w] == c) {
                            unsigned sh = (unsigned)(w & 3) * 8u;
                            p = !((atomicOr(reinterpret_cast<unsigned*>(a.mark + (w & ~3)), bit << sh) >> sh) & bit);
                        }
                    }
                    b_append(p, w | (dir << DIR_SHIFT), q, s_tail, 2 * ng, a.ctr + BATCH_CTR_ERROR);
                }
            }
            h = t;
            __syncthreads();
        }
        // classify: FW&BW -> SCC of the pivot, FW only / BW only -> the pivot's new classes
        for (int32_t i = threadIdx.x; i < nlive; i += blockDim.x) {
            int32_t v = live[i];
            uint8_t m = a.mark[v];
            if (!m) continue;
            int32_t p = pivot_unhash((uint32_t)a.key[a.color[v]]);
            if (m == 3) { a.scc[v] = p; a.color[v] = SCC_COLOR_DONE; }
            else a.color[v] = (m & 1) ? b_fw_colour(p) : b_bw_colour(p);
            a.mark[v] = 0;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        atomicAdd(a.ctr + BATCH_CTR_ROUNDS, rounds);
        atomicAdd(a.ctr + BATCH_CTR_LEVELS, levels);
        atomicMax(a.ctr + BATCH_CTR_MAX_ROUNDS, rounds);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(1024, 1) k_batch_scc(BatchArgs a) {
    __shared__ __align__(8) int32_t s[64];
    __shared__ int32_t s_big[B_BIG];
    __shared__ int32_t s_gi;
    extern __shared__ uint32_t s_marks[];
    while (true) {
        if (threadIdx.x == 0) {
            // a device error anywhere ends every block (read by one thread, so the block agrees)
            s_gi = *(volatile int32_t*)(a.ctr + BATCH_CTR_ERROR) ? a.G : atomicAdd(a.ctr + BATCH_CTR_NEXT, 1);
        }
        __syncthreads();
        int32_t k = s_gi;
        __syncthreads();
        if (k >= a.G) break;
        b_graph(a, a.order[k], s, s_big, s_marks);
    }
}

// ------------------------------------------------------------------ host side
struct scc_batch_plan {
    const scc_graph* g = nullptr;
    scc_state* s = nullptr;
    int32_t G = 0;
    int32_t* d_offs = nullptr;
    int32_t* d_order = nullptr;
    unsigned long long* d_key = nullptr;
    int32_t* d_live2 = nullptr;
    int32_t* d_ctr = nullptr;
    int32_t* h_ctr = nullptr;
    int32_t marks_n = 0;        // vertices of the largest graph whose marks fit shared memory
    scc_batch_tuning tune;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t ev[2];
};

static int batch_enqueue(scc_batch_plan* p, int sms) {
    scc_state* s = p->s;
    const scc_graph* g = p->g;
    BatchArgs a;
    a.begin = g->begin; a.adj = g->node_idx; a.rbegin = g->r_begin; a.radj = g->r_node_idx;
    a.offs = p->d_offs; a.order = p->d_order; a.G = p->G;
    a.color = s->color; a.scc = s->scc; a.mark = s->mark;
    a.cin = reinterpret_cast<uint32_t*>(s->cnt);
    a.cout = reinterpret_cast<uint32_t*>(s->cnt) + s->n;
    a.q = s->qa;
    a.live = s->live; a.live2 = p->d_live2;
    a.key = p->d_key;
    a.ctr = p->d_ctr;
    a.warp_deg = p->tune.warp_deg;
    a.members = nullptr;
    // Marks of the largest graph that fits B_MARKS_MAX; larger graphs take the
    // rounds over global marks from the start and ask for none: 300 graphs of 210,000
    // vertices on one block an SM with 200 KB each take 79 ms, on two
    // without 47.  Where the marks leave fewer blocks resident than asked
    // for, the others follow: no block waits for another.
    const int32_t smem = (p->marks_n + 3) & ~3;
    a.marks_cap = smem;
    a.vec_adj = ((reinterpret_cast<uintptr_t>(g->node_idx) | reinterpret_cast<uintptr_t>(g->r_node_idx)) & 15u) == 0;
    a.adj_len = g->m;
    SCC_CUDA(cudaFuncSetAttribute(k_batch_scc, cudaFuncAttributeMaxDynamicSharedMemorySize, B_MARKS_MAX));
    SCC_CUDA(cudaMemsetAsync(p->d_ctr, 0, sizeof(int32_t) * BATCH_CTR_WORDS, s->stream));
    k_batch_scc<<<sms * p->tune.blocks_per_sm, p->tune.threads, smem, s->stream>>>(a);
    SCC_CUDA(cudaPeekAtLastError());
    SCC_CUDA(cudaMemcpyAsync(p->h_ctr, p->d_ctr, sizeof(int32_t) * BATCH_CTR_WORDS, cudaMemcpyDeviceToHost,
                             s->stream));
    return SCC_OK;
}

static void batch_release(scc_batch_plan* p) {
    if (!p) return;
    if (p->exec) cudaGraphExecDestroy(p->exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    cudaFree(p->d_offs); cudaFree(p->d_order); cudaFree(p->d_key); cudaFree(p->d_live2); cudaFree(p->d_ctr);
    if (p->h_ctr) cudaFreeHost(p->h_ctr);
    cudaEventDestroy(p->ev[0]); cudaEventDestroy(p->ev[1]);
    delete p;
}

static bool batch_tuning_ok(const scc_batch_tuning* t) {
    return t->threads >= 64 && t->threads <= 1024 && (t->threads & 31) == 0 && t->blocks_per_sm >= 1 &&
           t->blocks_per_sm <= 8 && t->warp_deg >= 1;
}

extern "C" int scc_batch_default_tuning(scc_batch_tuning* t) {
    SCC_REQUIRE(t, SCC_ERR_INVALID, "NULL argument");
    t->threads = 512;
    t->blocks_per_sm = 2;
    t->warp_deg = 32;
    return SCC_OK;
}

extern "C" int scc_batch_plan_create(const scc_graph* g, scc_state* s, const int32_t* offsets, int32_t num_graphs,
                                     const scc_batch_tuning* tuning, scc_batch_plan** out) {
    SCC_REQUIRE(g && s && offsets && out && num_graphs >= 0, SCC_ERR_INVALID, "bad argument");
    SCC_REQUIRE(s->n == g->n, SCC_ERR_INVALID, "state of another graph");
    SCC_REQUIRE(offsets[0] == 0 && offsets[num_graphs] <= g->n, SCC_ERR_INVALID,
                "offsets must run from 0 to at most the graph's %d vertices", g->n);
    for (int32_t i = 0; i < num_graphs; ++i)
        SCC_REQUIRE(offsets[i + 1] >= offsets[i], SCC_ERR_INVALID, "offsets decrease at graph %d", i);
    SCC_REQUIRE((int64_t)g->n * 3 < (int64_t)INT32_MAX, SCC_ERR_INVALID, "too many vertices for batch colours");
    SCC_CUDA(cudaSetDevice(s->device));
    scc_batch_plan* p = new scc_batch_plan();
    p->g = g; p->s = s; p->G = num_graphs;
    for (int32_t i = 0; i < num_graphs; ++i) {
        const int32_t ng = offsets[i + 1] - offsets[i];
        if (ng <= B_MARKS_MAX) p->marks_n = std::max(p->marks_n, ng);
    }
    if (tuning) p->tune = *tuning; else scc_batch_default_tuning(&p->tune);
    if (!batch_tuning_ok(&p->tune)) { delete p; scc_set_error("bad batch tuning"); return SCC_ERR_INVALID; }
    cudaEventCreate(&p->ev[0]); cudaEventCreate(&p->ev[1]);
    // graphs by decreasing size: the largest start first, the small ones fill in
    std::vector<int32_t> order((size_t)num_graphs);
    for (int32_t i = 0; i < num_graphs; ++i) order[(size_t)i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
        return offsets[x + 1] - offsets[x] > offsets[y + 1] - offsets[y];
    });
    int rc = SCC_OK;
    int sms = 148;
#define BATCH_TRY(call) do { cudaError_t _e = (call); if (_e != cudaSuccess) { rc = scc_cuda_status(_e, #call, __FILE__, __LINE__); goto fail; } } while (0)
    BATCH_TRY(cudaMalloc(&p->d_offs, sizeof(int32_t) * ((size_t)num_graphs + 1)));
    BATCH_TRY(cudaMalloc(&p->d_order, sizeof(int32_t) * std::max<size_t>(1, (size_t)num_graphs)));
    BATCH_TRY(cudaMalloc(&p->d_key, sizeof(unsigned long long) * (3 * (size_t)std::max(g->n, 1) + 3)));
    BATCH_TRY(cudaMalloc(&p->d_live2, sizeof(int32_t) * (size_t)std::max(g->n, 1)));
    BATCH_TRY(cudaMalloc(&p->d_ctr, sizeof(int32_t) * BATCH_CTR_WORDS));
    BATCH_TRY(cudaMallocHost(&p->h_ctr, sizeof(int32_t) * BATCH_CTR_WORDS));
    BATCH_TRY(cudaMemcpy(p->d_offs, offsets, sizeof(int32_t) * ((size_t)num_graphs + 1), cudaMemcpyHostToDevice));
    if (num_graphs > 0)
        BATCH_TRY(cudaMemcpy(p->d_order, order.data(), sizeof(int32_t) * (size_t)num_graphs, cudaMemcpyHostToDevice));
    // the whole run -- counter reset, the persistent launch, counters back --
    // captured once; every run is one graph launch
    BATCH_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
    BATCH_TRY(cudaStreamSynchronize(s->stream));
    BATCH_TRY(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    rc = batch_enqueue(p, sms);
    {
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamEndCapture(s->stream, &graph);
        if (rc != SCC_OK) { if (graph) cudaGraphDestroy(graph); goto fail; }
        BATCH_TRY(e);
        p->graph = graph;
    }
    BATCH_TRY(cudaGraphInstantiate(&p->exec, p->graph, 0));
#undef BATCH_TRY
    *out = p;
    return SCC_OK;
fail:
    batch_release(p);
    return rc;
}

extern "C" int scc_batch_plan_run(scc_batch_plan* p, scc_batch_stats* stats) {
    SCC_REQUIRE(p, SCC_ERR_INVALID, "NULL plan");
    scc_state* s = p->s;
    SCC_CUDA(cudaSetDevice(s->device));
    SCC_CUDA(cudaEventRecord(p->ev[0], s->stream));
    SCC_CUDA(cudaGraphLaunch(p->exec, s->stream));
    SCC_CUDA(cudaEventRecord(p->ev[1], s->stream));
    SCC_CUDA(cudaStreamSynchronize(s->stream));
    float ms = 0.f;
    SCC_CUDA(cudaEventElapsedTime(&ms, p->ev[0], p->ev[1]));
    s->live_count = -1;      // the live list slices no longer describe the whole graph
    s->fresh = false;
    s->prefinished = false;
    s->cnt_valid = false;
    if (p->h_ctr[BATCH_CTR_ERROR]) {
        scc_set_error("batched run: device error %d", p->h_ctr[BATCH_CTR_ERROR]);
        return p->h_ctr[BATCH_CTR_ERROR] == SCC_DEVERR_WAIT_LIMIT ? SCC_ERR_TIMEOUT : SCC_ERR_OOM;
    }
    if (stats) {
        stats->ms_total = ms;
        stats->graphs = p->G;
        stats->rounds = p->h_ctr[BATCH_CTR_ROUNDS];
        stats->levels = p->h_ctr[BATCH_CTR_LEVELS];
        stats->max_rounds = p->h_ctr[BATCH_CTR_MAX_ROUNDS];
        stats->host_submissions = 1;
        stats->kernels = 1;
    }
    return SCC_OK;
}

extern "C" int scc_batch_plan_free(scc_batch_plan* p) {
    if (!p) return SCC_OK;
    cudaSetDevice(p->s->device);
    batch_release(p);
    return SCC_OK;
}

// ------------------------------------------------------------------ autotuner
// Successive halving: every candidate runs on the first eighth of the graphs
// (ids are in generation order, so a prefix is a fair sample of the sizes),
// the faster half goes on to a quarter, then half, then the whole batch.
static int batch_time(const scc_graph* g, scc_state* s, const int32_t* offsets, int32_t k,
                      const scc_batch_tuning& t, double* ms) {
    scc_batch_plan* p = nullptr;
    SCC_TRY(scc_batch_plan_create(g, s, offsets, k, &t, &p));
    scc_batch_stats st;
    int rc = scc_batch_plan_run(p, &st);            // warm-up
    if (rc == SCC_OK) rc = scc_batch_plan_run(p, &st);
    *ms = st.ms_total;
    scc_batch_plan_free(p);
    return rc;
}

extern "C" int scc_batch_autotune(const scc_graph* g, scc_state* s, const int32_t* offsets, int32_t num_graphs,
                                  scc_batch_tuning* best, double* best_ms) {
    SCC_REQUIRE(g && s && offsets && num_graphs > 0, SCC_ERR_INVALID, "bad argument");
    std::vector<scc_batch_tuning> cand;
    const int32_t threads[] = {256, 512, 1024};
    const int32_t per_sm[] = {1, 2, 4};
    const int32_t warp_deg[] = {8, 16, 32, 64};
    for (int32_t t : threads)
        for (int32_t b : per_sm)
            for (int32_t w : warp_deg)
                if (t * b <= 2048) cand.push_back(scc_batch_tuning{t, b, w});
    std::vector<double> ms(cand.size());
    for (int stage = 3; stage >= 0; --stage) {
        int32_t k = std::max<int32_t>(1, num_graphs >> stage);
        for (size_t i = 0; i < cand.size(); ++i) SCC_TRY(batch_time(g, s, offsets, k, cand[i], &ms[i]));
        std::vector<size_t> idx(cand.size());
        for (size_t i = 0; i < idx.size(); ++i) idx[i] = i;
        std::sort(idx.begin(), idx.end(), [&](size_t x, size_t y) { return ms[x] < ms[y]; });
        size_t keep = stage > 0 ? std::max<size_t>(1, (cand.size() + 1) / 2) : 1;
        std::vector<scc_batch_tuning> next;
        std::vector<double> next_ms;
        for (size_t i = 0; i < keep; ++i) { next.push_back(cand[idx[i]]); next_ms.push_back(ms[idx[i]]); }
        cand.swap(next);
        ms.swap(next_ms);
    }
    if (best) *best = cand[0];
    if (best_ms) *best_ms = ms[0];
    return SCC_OK;
}

// ------------------------------------------------------------------ the recursion's tail
// Once few vertices are left (tail_live), every remaining class is an
// independent subproblem: the live vertices are grouped by class (a stable
// sort of (colour, vertex)), and one persistent launch decomposes each class
// inside a block, as for a batch of graphs, instead of further rounds of many
// launches and host round trips.  Classes are unions of SCCs, so the labels
// are the same.  Skipped (nothing done) when a class is larger than
// tail_class, which one block would take too long to finish alone.
__global__ void k_tail_keys(const int32_t* __restrict__ live, int32_t nl, const int32_t* __restrict__ color,
                            uint32_t* __restrict__ keys) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nl; i += (int64_t)gridDim.x * blockDim.x)
        keys[i] = (uint32_t)color[live[i]];
}

// Every member's place in the grouped list, and one colour per class that no
// pivot's part can meet (3 x its first member, see the top of the file): all
// classes at once, so that no block sees another class's old colour.
__global__ void k_tail_classes(const int32_t* __restrict__ members, int32_t nl, const int32_t* __restrict__ starts,
                               int32_t G, int32_t* __restrict__ place, int32_t* __restrict__ color) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nl; k += (int64_t)gridDim.x * blockDim.x) {
        int32_t lo = 0, hi = G - 1;                     // the last class that starts at or before k
        while (lo < hi) {
            const int32_t mid = (lo + hi + 1) >> 1;
            if (starts[mid] <= k) lo = mid; else hi = mid - 1;
        }
        const int32_t v = members[k];
        place[v] = (int32_t)k;
        color[v] = 3 * members[starts[lo]];
    }
}

// A small class in shared memory: its members' lists, cut to the class and in
// local numbers, are read once; peel, pivots, FW+BW levels and classification
// then run as in b_graph on local arrays, so that a step costs tens of
// nanoseconds instead of a chain of global loads.  Classes with a list of more
// than TAIL_LIST entries or more than TAIL_EDGES x the capacity edges go to b_graph.
// The tail of R-MAT s20 with a 1024 x 1024 grid (48,000 vertices in 3,200
// classes, largest 667): 490 us with b_graph, 147 us so (128 threads 170, 64 threads 203).
#define TAIL_LIST 256
#define TAIL_EDGES 4
#define TAIL_THREADS 256
#define TAIL_MAX 1024                // members of the largest class handled so

// Bytes of shared memory for classes of up to cap members.
__host__ __device__ __forceinline__ int32_t tail_smem(int32_t cap) {
    return 8 * (4 * cap + 3) + 4 * (7 * cap + 2) + 2 * ((2 * TAIL_EDGES + 9) * cap + 3) + 64;
}

struct TailClass {
    int32_t cap;
    unsigned long long *pk, *key;    // pivot key of a member; best key of a local class
    int32_t *vid, *off0, *lab, *mark, *cnt0;
    uint16_t *adj0, *piv, *scc, *q, *qc, *live, *live2;
    __device__ __forceinline__ TailClass(void* sm, int32_t c) : cap(c) {
        pk = (unsigned long long*)sm; key = pk + cap;
        vid = (int32_t*)(key + 3 * cap + 3);
        off0 = vid + cap;
        lab = off0 + 2 * (cap + 1); mark = lab + cap;
        cnt0 = mark + cap;
        adj0 = (uint16_t*)(cnt0 + 2 * cap);
        piv = adj0 + 2 * TAIL_EDGES * cap; scc = piv + 3 * cap + 3;
        q = scc + cap; qc = q + 2 * cap; live = qc + cap; live2 = live + cap;
    }
    // direction 0: out-neighbours, 1: in-neighbours
    __device__ __forceinline__ int32_t* off(int d) const { return off0 + d * (cap + 1); }
    __device__ __forceinline__ uint16_t* adj(int d) const { return adj0 + d * TAIL_EDGES * cap; }
    __device__ __forceinline__ int32_t* cnt(int d) const { return cnt0 + d * cap; }
};

// Returns false, with nothing changed, when the class does not fit.
__device__ bool b_class_small(const BatchArgs& a, int32_t lo, int32_t ng, int32_t cap, const int32_t* __restrict__ place,
                              int32_t* s, void* sm) {
    TailClass t(sm, cap);
    int32_t* s_tail = s;
    int32_t* s_n = s + 1;
    int32_t* s_warp = s + 32;
    const int32_t T = blockDim.x;
    for (int d = 0; d < 2; ++d) {
        const int32_t* off = d ? a.rbegin : a.begin;
        const int32_t* adj = d ? a.radj : a.adj;
        // count the class's entries per member, place the lists, then fill them
        int32_t base = 0;
        bool fits = true;
        for (int32_t i0 = 0; i0 < ng; i0 += T) {
            const int32_t i = i0 + threadIdx.x;
            int32_t k = 0;
            bool small = true;
            if (i < ng) {
                const int32_t v = a.members[lo + i], b = __ldg(off + v), e = __ldg(off + v + 1);
                small = e - b <= TAIL_LIST;
                if (small)
                    for (int32_t j = b; j < e; ++j) {
                        const int32_t w = __ldg(adj + j), at = __ldg(place + w) - lo;
                        k += w != v && (uint32_t)at < (uint32_t)ng && a.members[lo + at] == w;
                    }
            }
            fits = __syncthreads_and(small) && fits;
            int32_t tot = 0;
            const int32_t before = b_scan(k, s_warp, &tot);
            if (i < ng) t.off(d)[i] = base + before;
            base += tot;
        }
        if (!fits || base > TAIL_EDGES * cap) return false;          // the same in every thread
        if (threadIdx.x == 0) t.off(d)[ng] = base;
        for (int32_t i = threadIdx.x; i < ng; i += T) {
            const int32_t v = a.members[lo + i], b = __ldg(off + v), e = __ldg(off + v + 1);
            int32_t at0 = t.off(d)[i];
            for (int32_t j = b; j < e; ++j) {
                const int32_t w = __ldg(adj + j), at = __ldg(place + w) - lo;
                if (w != v && (uint32_t)at < (uint32_t)ng && a.members[lo + at] == w) t.adj(d)[at0++] = (uint16_t)at;
            }
        }
    }
    for (int32_t i = threadIdx.x; i < ng; i += T) {
        const int32_t v = a.members[lo + i];
        t.vid[i] = v;
        t.pk[i] = pivot_key(a.begin, a.rbegin, v);
        t.lab[i] = 0;
        t.mark[i] = 0;
        t.live[i] = (uint16_t)i;
    }
    __syncthreads();
    int32_t nlive = ng, rounds = 0, levels = 0;
    uint16_t *live = t.live, *live2 = t.live2;
    while (true) {
        // peel inside the local classes
        for (int32_t x = threadIdx.x; x < nlive; x += T) {
            const int32_t i = live[x], c = t.lab[i];
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                int32_t k = 0;
                for (int32_t j = t.off(d)[i]; j < t.off(d)[i + 1]; ++j) k += t.lab[t.adj(d)[j]] == c;
                t.cnt(d)[i] = k;
            }
        }
        if (threadIdx.x == 0) *s_tail = 0;
        __syncthreads();
        for (int32_t x = threadIdx.x; x < nlive; x += T) {
            const int32_t i = live[x];
            if (t.cnt(0)[i] == 0 || t.cnt(1)[i] == 0) {
                const int32_t at = atomicAdd(s_tail, 1);
                t.q[at] = (uint16_t)i;
                t.qc[at] = (uint16_t)t.lab[i];
                t.lab[i] = SCC_COLOR_DONE;
                t.scc[i] = (uint16_t)i;
            }
        }
        __syncthreads();
        int32_t h = 0;
        while (true) {
            const int32_t n = *s_tail;
            __syncthreads();
            if (h >= n) break;
            for (int32_t x = h + threadIdx.x; x < n; x += T) {
                const int32_t i = t.q[x], c = t.qc[x];
#pragma unroll
                for (int d = 0; d < 2; ++d)           // an out-edge costs the neighbour an in-neighbour, and the reverse
                    for (int32_t j = t.off(d)[i]; j < t.off(d)[i + 1]; ++j) {
                        const int32_t w = t.adj(d)[j];
                        if (*(volatile int32_t*)(t.lab + w) != c || atomicSub(t.cnt(d ^ 1) + w, 1) != 1) continue;
                        if (atomicCAS(t.lab + w, c, SCC_COLOR_DONE) != c) continue;
                        t.scc[w] = (uint16_t)w;
                        const int32_t at = atomicAdd(s_tail, 1);
                        t.q[at] = (uint16_t)w;
                        t.qc[at] = (uint16_t)c;
                    }
            }
            h = n;
            __syncthreads();
        }
        if (threadIdx.x == 0) *s_n = 0;
        __syncthreads();
        for (int32_t x = threadIdx.x; x < nlive; x += T) {
            const int32_t i = live[x];
            if (t.lab[i] != SCC_COLOR_DONE) {
                live2[atomicAdd(s_n, 1)] = (uint16_t)i;
                t.key[t.lab[i]] = 0ull;
            }
        }
        __syncthreads();
        nlive = *s_n;
        uint16_t* tmp = live; live = live2; live2 = tmp;
        if (nlive == 0) break;
        if (++rounds > ng + 2) {
            if (threadIdx.x == 0) atomicExch(a.ctr + BATCH_CTR_ERROR, SCC_DEVERR_WAIT_LIMIT);
            break;
        }
        // pivot of every local class, then FW and BW level by level
        for (int32_t x = threadIdx.x; x < nlive; x += T) atomicMax(t.key + t.lab[live[x]], t.pk[live[x]]);
        if (threadIdx.x == 0) *s_tail = 0;
        __syncthreads();
        for (int32_t x = threadIdx.x; x < nlive; x += T) {
            const int32_t i = live[x];
            if (t.pk[i] != t.key[t.lab[i]]) continue;
            t.mark[i] = 3;
            t.piv[t.lab[i]] = (uint16_t)i;
            const int32_t at = atomicAdd(s_tail, 2);
            t.q[at] = (uint16_t)i;
            t.q[at + 1] = (uint16_t)(i | 0x8000);
        }
        __syncthreads();
        h = 0;
        while (true) {
            const int32_t n = *s_tail;
            __syncthreads();
            if (h >= n) break;
            ++levels;
            for (int32_t x = h + threadIdx.x; x < n; x += T) {
                const int32_t it = t.q[x], i = it & 0x7FFF, d = it >> 15, c = t.lab[i];
                for (int32_t j = t.off(d)[i]; j < t.off(d)[i + 1]; ++j) {
                    const int32_t w = t.adj(d)[j];
                    if (t.lab[w] != c || ((atomicOr(t.mark + w, 1 << d) >> d) & 1)) continue;
                    t.q[atomicAdd(s_tail, 1)] = (uint16_t)(w | (d << 15));
                }
            }
            h = n;
            __syncthreads();
        }
        for (int32_t x = threadIdx.x; x < nlive; x += T) {
            const int32_t i = live[x], m = t.mark[i];
            if (!m) continue;
            const int32_t p = t.piv[t.lab[i]];
            if (m == 3) { t.scc[i] = (uint16_t)p; t.lab[i] = SCC_COLOR_DONE; }
            else t.lab[i] = 3 * p + ((m & 1) ? 1 : 2);
            t.mark[i] = 0;
        }
        __syncthreads();
    }
    for (int32_t i = threadIdx.x; i < ng; i += T) {
        a.scc[t.vid[i]] = t.vid[t.scc[i]];
        a.color[t.vid[i]] = SCC_COLOR_DONE;
    }
    if (threadIdx.x == 0) {
        atomicAdd(a.ctr + BATCH_CTR_ROUNDS, rounds);
        atomicAdd(a.ctr + BATCH_CTR_LEVELS, levels);
        atomicMax(a.ctr + BATCH_CTR_MAX_ROUNDS, rounds);
    }
    __syncthreads();
    return true;
}

__global__ void __launch_bounds__(512, 1) k_tail_scc(BatchArgs a, int32_t cap, const int32_t* __restrict__ place) {
    __shared__ __align__(8) int32_t s[64];
    __shared__ int32_t s_big[B_BIG];
    __shared__ int32_t s_gi;
    extern __shared__ __align__(16) unsigned char s_class[];
    while (true) {
        if (threadIdx.x == 0)
            s_gi = *(volatile int32_t*)(a.ctr + BATCH_CTR_ERROR) ? a.G : atomicAdd(a.ctr + BATCH_CTR_NEXT, 1);
        __syncthreads();
        const int32_t k = s_gi;
        __syncthreads();
        if (k >= a.G) break;
        const int32_t gi = a.order[k], lo = a.offs[gi], ng = a.offs[gi + 1] - lo;
        if (ng > cap || !b_class_small(a, lo, ng, cap, place, s, s_class)) b_graph(a, gi, s, s_big, nullptr);
    }
}

// Classes of at most TAIL_ONE_BLOCK grouped members: where each begins, their
// number, the largest, and an order to take them in, by one block.
#define TAIL_ONE_BLOCK 4096
__global__ void __launch_bounds__(256) k_tail_starts(const uint32_t* __restrict__ keys, int32_t nl,
                                                     int32_t* __restrict__ starts, int32_t* __restrict__ order,
                                                     int32_t* __restrict__ out) {
    __shared__ int32_t s_warp[32];
    __shared__ int32_t s_big;
    if (threadIdx.x == 0) s_big = 0;
    int32_t base = 0;
    for (int32_t i0 = 0; i0 < nl; i0 += 256) {
        const int32_t i = i0 + threadIdx.x;
        const int32_t first = i < nl && (i == 0 || keys[i] != keys[i - 1]);
        int32_t tot = 0;
        const int32_t before = b_scan(first, s_warp, &tot);
        if (first) { starts[base + before] = i; order[base + before] = base + before; }
        base += tot;
    }
    if (threadIdx.x == 0) starts[base] = nl;
    __syncthreads();
    int32_t big = 0;
    for (int32_t k = threadIdx.x; k < base; k += 256) big = max(big, starts[k + 1] - starts[k]);
    atomicMax(&s_big, big);
    __syncthreads();
    if (threadIdx.x == 0) { out[0] = base; out[1] = s_big; }
}

int scc_impl_resolve_tail(const scc_graph* g, scc_state* s, bool* taken) {
    *taken = false;
    const int32_t nl = s->live_count;
    if (nl <= 0) return SCC_OK;
    cudaStream_t st = s->stream;
    struct Pool {
        cudaStream_t st;
        std::vector<void*> v;
        ~Pool() { for (void* p : v) cudaFreeAsync(p, st); }
        cudaError_t get(void** p, size_t b) { cudaError_t e = scc_impl_malloc_async(p, b, st); if (e == cudaSuccess) v.push_back(*p); return e; }
    } pool{st, {}};
    uint32_t *keys = nullptr, *skeys = nullptr;
    int32_t *members = nullptr, *starts = nullptr, *order = nullptr, *ctr = nullptr;
    SCC_CUDA(pool.get((void**)&keys, sizeof(uint32_t) * (size_t)nl));
    SCC_CUDA(pool.get((void**)&skeys, sizeof(uint32_t) * (size_t)nl));
    SCC_CUDA(pool.get((void**)&members, sizeof(int32_t) * (size_t)nl));
    SCC_CUDA(pool.get((void**)&starts, sizeof(int32_t) * ((size_t)nl + 1)));
    k_tail_keys<<<scc_blocks(nl), SCC_THREADS, 0, st>>>(s->live, nl, s->color, keys);
    SCC_LAUNCHED(s);
    // colours are at most the last one handed out (the host mirror is current here)
    int bits = 1;
    while (bits < 32 && (1LL << bits) <= (int64_t)s->h_ctr[CTR_NEXT_COLOR]) bits++;
    SCC_TRY(scc_impl_sort_pairs_u32(keys, skeys, s->live, members, nl, bits, st));
    int64_t G = 0;
    int32_t biggest = 0;
    SCC_CUDA(pool.get((void**)&ctr, sizeof(int32_t) * BATCH_CTR_WORDS));
    if (nl <= TAIL_ONE_BLOCK) {
        SCC_CUDA(pool.get((void**)&order, sizeof(int32_t) * (size_t)nl));
        k_tail_starts<<<1, 256, 0, st>>>(skeys, nl, starts, order, s->ctr + CTR_QLEN);     // CTR_QLEN, CTR_QLEN2
        SCC_LAUNCHED(s);
        SCC_TRY(scc_sync_counters(s));
        G = s->h_ctr[CTR_QLEN];
        biggest = s->h_ctr[CTR_QLEN2];
        if (biggest > s->tune.tail_class) return SCC_OK;
    } else {
        SCC_TRY(scc_impl_segment_starts(skeys, nl, starts, &G, st));
        std::vector<int32_t> h((size_t)G + 1);
        SCC_CUDA(cudaMemcpyAsync(h.data(), starts, sizeof(int32_t) * (size_t)G, cudaMemcpyDeviceToHost, st));
        SCC_CUDA(cudaStreamSynchronize(st));
        h[(size_t)G] = nl;
        for (int64_t k = 0; k < G; ++k) biggest = std::max(biggest, h[(size_t)k + 1] - h[(size_t)k]);
        if (biggest > s->tune.tail_class) return SCC_OK;
        // largest first
        std::vector<int32_t> ord((size_t)G);
        for (int64_t k = 0; k < G; ++k) ord[(size_t)k] = (int32_t)k;
        std::stable_sort(ord.begin(), ord.end(), [&](int32_t x, int32_t y) { return h[x + 1] - h[x] > h[y + 1] - h[y]; });
        SCC_CUDA(pool.get((void**)&order, sizeof(int32_t) * (size_t)std::max<int64_t>(G, 1)));
        SCC_CUDA(cudaMemcpyAsync(starts + G, &nl, sizeof(int32_t), cudaMemcpyHostToDevice, st));
        SCC_CUDA(cudaMemcpyAsync(order, ord.data(), sizeof(int32_t) * (size_t)G, cudaMemcpyHostToDevice, st));
    }
    if (!s->bkey) SCC_CUDA(cudaMalloc(&s->bkey, sizeof(unsigned long long) * (3 * (size_t)std::max(s->n, 1) + 3)));
    SCC_CUDA(cudaMemsetAsync(ctr, 0, sizeof(int32_t) * BATCH_CTR_WORDS, st));
    BatchArgs a;
    a.begin = g->begin; a.adj = g->node_idx; a.rbegin = g->r_begin; a.radj = g->r_node_idx;
    a.offs = starts; a.order = order; a.G = (int32_t)G;
    a.color = s->color; a.scc = s->scc; a.mark = s->mark;
    a.cin = reinterpret_cast<uint32_t*>(s->cnt);
    a.cout = reinterpret_cast<uint32_t*>(s->cnt) + s->n;
    a.q = s->qa;
    a.live = s->live; a.live2 = s->live_tmp;
    a.key = s->bkey;
    a.ctr = ctr;
    a.warp_deg = 32;
    a.members = members;
    a.marks_cap = 0;
    a.vec_adj = 0;
    a.adj_len = g->m;
    int sms = 148;
    SCC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
    int32_t* place = s->aux;          // free here
    k_tail_classes<<<scc_blocks(nl), SCC_THREADS, 0, st>>>(members, nl, starts, (int32_t)G, place, s->color);
    SCC_LAUNCHED(s);
    // shared memory for the largest class, as many blocks as that leaves room for
    const int32_t cap = std::min(biggest, TAIL_MAX);
    const int32_t smem = tail_smem(cap);
    const bool all_small = biggest <= TAIL_MAX;
    const int per_sm = std::max(1, std::min(8, 200 * 1024 / smem));
    SCC_CUDA(cudaFuncSetAttribute(k_tail_scc, cudaFuncAttributeMaxDynamicSharedMemorySize, tail_smem(TAIL_MAX)));
    k_tail_scc<<<(unsigned)std::min<int64_t>(G, (int64_t)sms * per_sm), all_small ? TAIL_THREADS : 512, smem, st>>>(a, cap,
                                                                                                            place);
    SCC_LAUNCHED(s);
    int32_t h_ctr[BATCH_CTR_WORDS];
    SCC_CUDA(cudaMemcpyAsync(h_ctr, ctr, sizeof(h_ctr), cudaMemcpyDeviceToHost, st));
    SCC_CUDA(cudaStreamSynchronize(st));
    if (h_ctr[BATCH_CTR_ERROR]) {
        scc_set_error("tail decomposition: device error %d", h_ctr[BATCH_CTR_ERROR]);
        return h_ctr[BATCH_CTR_ERROR] == SCC_DEVERR_WAIT_LIMIT ? SCC_ERR_TIMEOUT : SCC_ERR_OOM;
    }
    s->fb_rounds += h_ctr[BATCH_CTR_MAX_ROUNDS];
    s->cnt_valid = false;
    s->live_count = 0;
    *taken = true;
    if (scc_trace_on())
        fprintf(stderr, "[scc] tail: %d live vertices in %lld classes (largest %d) in one launch, up to %d rounds\n", nl,
                (long long)G, biggest, h_ctr[BATCH_CTR_MAX_ROUNDS]);
    return SCC_OK;
}
