// Record drain: the asynchronous reachability drain (k_reach_async in
// scc_reach.cu) for sparse rounds whose narrow wave still has far to go, such
// as grids, meshes and long cycles (the traversal under fw_trim_global /
// bw_trim_global, src/scc_fb_global.cc:32-130).
//
// A wave through a long-diameter class is a chain of dependent memory round
// trips, so what counts is how far one round trip gets.  The plain drain takes
// two per hop: a neighbour's mark, colour and offsets, then its claim and its
// list.  Here a pass over the round's live vertices first writes, for every
// vertex and direction, a record of up to REC_W vertices it reaches inside its
// class:
//   * vertices are named by their place in the live list, so marks, records
//     and queue items of the round are dense, and only class members appear:
//     the drain reads no colour, offset or adjacency;
//   * the record starts as the vertex's neighbours and grows breadth first: an
//     entry's own neighbours join it while they all fit, and the entry is then
//     covered.  An entry that is not covered is on the record's boundary.
// Expanding a vertex claims all entries of its record in one round trip, an
// atomic per entry, while the boundary entries' records are loaded with it.  A
// claimed boundary entry is expanded next; a covered one needs no expansion,
// since its neighbours are claimed along with it.  Everything claimed is
// reached, and the neighbours of everything claimed are claimed in the end,
// which is the closure the plain drain computes.  One round trip advances a
// grid's wave about two hops, a chain's by eight.
//
// C2's wave (the 4096 x 4096 grid's giant class, 13.1 M live vertices): 18.7 ms
// in the plain drain; 1.0 ms of building and 4.2 ms here.  2501 x 2501 grid:
// 10.9 ms against 0.4 + 2.4 ms.  Both waves are bound by the latency of an
// iteration (about 1 us: one round trip and the instructions around it on two
// warps per scheduler; one warp per scheduler 6.8 ms on C2, four no faster).
//
// The work count and the bounded waits are the plain drain's.  A
// vertex of more than REC_W class neighbours, or of a neighbour outside the live
// list, has a LONG record: the warp that takes it walks its adjacency list with
// the colour test; a claimed neighbour outside the live list goes to the host's
// next frontier, as such a vertex does that is in the frontier already.  What a warp
// shares after the idle ones gave up their tickets is collected by the host.
#include <algorithm>
#include "scc_record.cuh"

#define REC_W 8                       // entries of a record (32 bytes)
#define REC_LONG (-2)                 // first entry of a record that is no list
#define REC_NONE (-1)                 // empty entry
#define REC_MANY (-3)                 // first neighbour of a vertex that has more than four
#define REC_DIR 29                    // direction bit of an entry (places stay below 2^29, as vertex ids do)
#define REC_EDGE 30                   // the entry is on the boundary
#define REC_PLACE 0x1FFFFFFF
#define REC_SCAN 64                   // a list longer than this is LONG without being read
#define REC_THREADS 256
#define REC_WARPS (REC_THREADS / 32)
#define REC_ITEMS (32 / REC_W)        // items a warp expands at once
#define REC_BUF 128                   // a warp's own list, in items
#define REC_KEEP 8                    // items a warp keeps when it shares
#define REC_IDLE_LIMIT (1 << 22)      // polls without progress anywhere before the bounded wait gives up

// ------------------------------------------------------------------ building
__global__ void k_rec_places(const int32_t* __restrict__ live, int32_t n, const uint8_t* __restrict__ mark,
                             int32_t* __restrict__ place, uint8_t* __restrict__ pm) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = live[i];
        place[v] = (int32_t)i;
        pm[i] = mark[v];
    }
}

// The class neighbours of every live vertex in both directions, number 2 i +
// dir for the vertex at place i.  Self-loops and repeats (lists are sorted) are
// left out.  Up to four go to nbr, from which k_rec_grow makes the record;
// a vertex of more has REC_MANY there and its record, its neighbours or LONG, is
// written here.
__global__ void __launch_bounds__(SCC_THREADS) k_rec_neighbours(RoundArgs a, const int32_t* __restrict__ place,
                                                                int4* __restrict__ nbr, int4* __restrict__ rec) {
    __shared__ int32_t s[REC_W][SCC_THREADS];
    const int64_t total = 2LL * a.live_count;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int dir = (int)(t & 1);
        const int32_t v = a.live[t >> 1], c = __ldg(a.color + v);
        const int32_t* off = dir ? a.r_begin : a.begin;
        const int32_t* adj = dir ? a.r_node_idx : a.node_idx;
        const int32_t b = __ldg(off + v), e = __ldg(off + v + 1);
        bool is_long = c != SCC_COLOR_DONE && e - b > REC_SCAN;
        int n = 0;
        int32_t last = v;
        if (c != SCC_COLOR_DONE && !is_long) {
            for (int32_t k = b; k < e; k += 4) {
                int32_t w[4], col[4], p[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = k + j < e ? __ldg(adj + k + j) : v;
#pragma unroll
                for (int j = 0; j < 4; ++j) { col[j] = __ldg(a.color + w[j]); p[j] = __ldg(place + w[j]); }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (w[j] == v || w[j] == last || col[j] != c) continue;
                    last = w[j];
                    if ((uint32_t)p[j] >= (uint32_t)a.live_count || a.live[p[j]] != w[j] || n == REC_W) {
                        is_long = true;
                        continue;
                    }
                    s[n++][threadIdx.x] = p[j];
                }
            }
        }
        if (n <= 4 && !is_long) {
            int32_t x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = j < n ? s[j][threadIdx.x] : REC_NONE;
            nbr[t] = make_int4(x[0], x[1], x[2], x[3]);
        } else {
            int32_t x[REC_W];
#pragma unroll
            for (int j = 0; j < REC_W; ++j)
                x[j] = j < n && !is_long ? s[j][threadIdx.x] | (dir << REC_DIR) | (1 << REC_EDGE) : REC_NONE;
            if (is_long) x[0] = REC_LONG;
            nbr[t] = make_int4(REC_MANY, REC_NONE, REC_NONE, REC_NONE);
            rec[2 * t] = make_int4(x[0], x[1], x[2], x[3]);
            rec[2 * t + 1] = make_int4(x[4], x[5], x[6], x[7]);
        }
    }
}

// Records grown from the neighbour lists, breadth first, as far as REC_W
// entries go; an entry may come twice, which costs its place and a claim that
// fails.  Bound by instruction issue (divergent lanes).  C2's grid, 13.1 M
// vertices: 0.60 ms, and the drain after it 4.2 ms; with each entry looked up
// among the others first, 1.45 ms and 0.3 ms less in the drain, or branch-free in
// registers 0.94 ms and 0.25 ms less.
__global__ void __launch_bounds__(SCC_THREADS) k_rec_grow(int32_t live_count, const int4* __restrict__ nbr,
                                                          int4* __restrict__ rec) {
    __shared__ int32_t s[REC_W][SCC_THREADS];
    const int tid = threadIdx.x;
    const int64_t total = 2LL * live_count;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + tid; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int dir = (int)(t & 1);
        const int32_t self = (int32_t)(t >> 1);
        const int4 own = __ldg(nbr + t);
        if (own.x == REC_MANY) continue;         // written already
        s[0][tid] = own.x; s[1][tid] = own.y; s[2][tid] = own.z; s[3][tid] = own.w;
        int n = (own.x >= 0) + (own.y >= 0) + (own.z >= 0) + (own.w >= 0);
        unsigned covered = 0u;
        for (int i = 0; i < n && n < REC_W; ++i) {
            const int4 z = __ldg(nbr + 2LL * s[i][tid] + dir);
            if (z.x == REC_MANY) continue;
            // the entry is covered when all its neighbours fit
            const int32_t y[4] = {z.x, z.y, z.z, z.w};
            int m = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) m += y[j] >= 0 && y[j] != self;
            if (n + m > REC_W) continue;
            covered |= 1u << i;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (y[j] >= 0 && y[j] != self) s[n++][tid] = y[j];
        }
        int32_t x[REC_W];
#pragma unroll
        for (int j = 0; j < REC_W; ++j)
            x[j] = j < n ? s[j][tid] | (dir << REC_DIR) | (((covered >> j) & 1u) ? 0 : 1 << REC_EDGE) : REC_NONE;
        rec[2 * t] = make_int4(x[0], x[1], x[2], x[3]);
        rec[2 * t + 1] = make_int4(x[4], x[5], x[6], x[7]);
    }
}

// Frontier items (vertex | direction << DIR_SHIFT) to places, and back.  Of the
// n items of q, those of listed vertices are appended to out (count *listed, and the
// drain's *work with it); a class vertex that the live list does not hold has no
// place -- whatever is read for it is some earlier use's -- and goes to the host's next frontier.
__global__ void k_rec_items_in(const int32_t* __restrict__ q, int32_t n, const int32_t* __restrict__ live,
                               int32_t live_count, const int32_t* __restrict__ place, int32_t* __restrict__ out,
                               int32_t* __restrict__ listed, int32_t* __restrict__ work,
                               int32_t* __restrict__ outside, int32_t* __restrict__ outside_count) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xFFFFFFFFu, lt = (1u << lane) - 1u;
    const int64_t limit = ((int64_t)n + 31) / 32 * 32;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < limit; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t it = i < n ? q[i] : 0, v = it & ITEM_MASK;
        const int32_t p = i < n ? place[v] : -1;
        const bool in = (uint32_t)p < (uint32_t)live_count && live[p] == v;
        const unsigned bin = __ballot_sync(full, in), bout = __ballot_sync(full, i < n && !in);
        int32_t at = 0, oat = 0;
        if (lane == 0) {
            if (bin) { at = atomicAdd(listed, __popc(bin)); atomicAdd(work, __popc(bin)); }
            if (bout) oat = atomicAdd(outside_count, __popc(bout));
        }
        at = __shfl_sync(full, at, 0);
        oat = __shfl_sync(full, oat, 0);
        if (in) out[at + __popc(bin & lt)] = p | (((it >> DIR_SHIFT) & 1) << REC_DIR);
        else if (i < n) outside[oat + __popc(bout & lt)] = it;
    }
}
// What a hand-back left anywhere in the queue, appended to out; the queue is kept empty between uses.
__global__ void k_rec_items_out(int32_t* __restrict__ q, int32_t n, const int32_t* __restrict__ live,
                                int32_t* __restrict__ out, int32_t* __restrict__ count) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t x = q[i];
        if (x == -1) continue;
        out[atomicAdd(count, 1)] = live[x & REC_PLACE] | (((x >> REC_DIR) & 1) << DIR_SHIFT);
        q[i] = -1;
    }
}
__global__ void k_rec_marks_out(const int32_t* __restrict__ live, int32_t n, const uint8_t* __restrict__ pm,
                                uint8_t* __restrict__ mark) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        mark[live[i]] = pm[i];
}

// ------------------------------------------------------------------ the drain
__device__ __forceinline__ int32_t rec_ld(const int32_t* p) { return *(const volatile int32_t*)p; }

// A warp's own items, newest last: their records and, for sharing, their names.
struct RecList {
    int4* buf;
    int32_t* id;
    int32_t count;         // warp-uniform
    // Warp-collective: lanes with p add an item of record (r0, r1).  Returns their number.
    __device__ __forceinline__ int32_t push(bool p, int32_t item, const int4& r0, const int4& r1) {
        const int lane = threadIdx.x & 31;
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, p);
        if (p) {
            const int at = count + __popc(bal & ((1u << lane) - 1u));
            buf[2 * at] = r0;
            buf[2 * at + 1] = r1;
            id[at] = item;
        }
        count += __popc(bal);
        return __popc(bal);
    }
};

// Claims entry ent (place | direction | boundary), its record loaded in the
// same round trip when it is on the boundary; true if it is to be expanded.
__device__ __forceinline__ bool rec_claim(const int4* __restrict__ rec, uint8_t* pm, int32_t ent, bool act, int4& r0,
                                          int4& r1) {
    const int32_t p = ent & REC_PLACE, dir = (ent >> REC_DIR) & 1;
    const bool edge = act && ((ent >> REC_EDGE) & 1);
    const unsigned bit = 1u << (dir + (p & 3) * 8);
    unsigned old = bit;
    r0 = make_int4(REC_NONE, REC_NONE, REC_NONE, REC_NONE);
    r1 = r0;
    if (act) old = atomicOr(reinterpret_cast<unsigned*>(pm + (p & ~3)), bit);
    if (edge) {
        const int4* at = rec + (2LL * p + dir) * 2;
        r0 = __ldg(at);
        r1 = __ldg(at + 1);
    }
    return edge && !(old & bit) && r0.x != REC_NONE;
}

// A warp expands REC_ITEMS items at once, a lane per entry; an iteration is one
// pop from shared memory, one round trip (claims and records together) and one
// push.  Nothing else may wait on memory in a busy warp's iteration:
//   * a warp without items takes REC_ITEMS tickets, the next places of the
//     shared queue, and polls those places alone (592 warps popping a head
//     counter by compare-and-swap took four items a round trip between them:
//     166 ms for C2's grid wave);
//   * a warp with more than REC_KEEP items shares the newest: it asks for the
//     queue places and publishes its work count in one iteration and writes
//     the items in the next, when both atomics have long answered.
// work counts the items not expanded.  A warp publishes its net change before
// its items become visible and before it waits, so the count reaches zero only
// when nothing is left.
__global__ void __launch_bounds__(REC_THREADS, 1) k_reach_records(RoundArgs a, const int4* __restrict__ rec, uint8_t* pm,
                                                                  const int32_t* __restrict__ place,
                                                                  int32_t* __restrict__ q, int64_t qcap,
                                                                  int32_t* __restrict__ outside, int idle_limit) {
    static_assert(REC_W == 8, "a record is two int4 and eight lanes wide");
    const unsigned full = 0xFFFFFFFFu;
    __shared__ int4 s_buf[REC_WARPS][2 * REC_BUF];
    __shared__ int32_t s_id[REC_WARPS][REC_BUF];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane / REC_W;
    int32_t* head = a.ctr + CTR_AHEAD;
    int32_t* tail = a.ctr + CTR_ATAIL;
    int32_t* work = a.ctr + CTR_AWORK;
    int32_t* err = a.ctr + CTR_ERROR;
    int32_t* bail = a.ctr + CTR_ABAIL;
    RecList list{s_buf[wid], s_id[wid], 0};
    int32_t net = 0;                 // items pushed - expanded, not yet published (uniform)
    unsigned ticket = 0;             // tickets not served yet, one bit each; lane j < REC_ITEMS polls ticket_at + j
    int32_t ticket_at = 0;
    int32_t give = 0, give_id = 0;   // items being shared (uniform) and this lane's one
    int32_t give_at = 0, give_work = 0, stop = 0;     // answers of lane 0's atomics and load
    int idle = 0;
    uint32_t iter = 0;
    int32_t last_work = -1;
    uint32_t my_items = 0;                            // uniform; the ledger's totals
    uint32_t my_edges = 0;                            // this lane's
    while (true) {
        if (list.count == 0 && ticket == 0) {
            int32_t at = 0;
            if (lane == 0) at = atomicAdd(head, REC_ITEMS);
            ticket_at = __shfl_sync(full, at, 0);
            ticket = (1u << REC_ITEMS) - 1u;
        }
        int32_t came = -1;
        if (((ticket >> lane) & 1u) && (int64_t)ticket_at + lane < qcap) came = rec_ld(q + ticket_at + lane);
        // expand
        const int32_t k = min(REC_ITEMS, list.count), first = list.count - k;
        const int32_t ent = g < k ? reinterpret_cast<const int32_t*>(list.buf)[(first + g) * REC_W + (lane & (REC_W - 1))]
                                  : REC_NONE;
        // the claims and record loads go out first; the bookkeeping runs while they are under way
        const int32_t dir = (ent >> REC_DIR) & 1;
        const unsigned bit = 1u << (dir + (ent & 3) * 8);
        const bool edge = ent >= 0 && ((ent >> REC_EDGE) & 1);
        unsigned old = bit;
        if (ent >= 0) old = atomicOr(reinterpret_cast<unsigned*>(pm + (ent & (REC_PLACE & ~3))), bit);
        int4 r0 = make_int4(REC_NONE, REC_NONE, REC_NONE, REC_NONE), r1 = r0;
        if (edge) {
            const int4* at = rec + (2LL * (ent & REC_PLACE) + dir) * 2;
            r0 = __ldg(at);
            r1 = __ldg(at + 1);
        }
        unsigned longs = __ballot_sync(full, ent == REC_LONG);
        int32_t long_id = 0;
        if (longs) {
            if (ent == REC_LONG) long_id = list.id[first + g];
            __syncwarp();
        }
        list.count = first;
        net -= k;
        my_items += k;
        my_edges += ent >= 0;
        // hand over what the last iteration prepared
        if (give) {
            // both answers are here: the count is published before the items are
            const int32_t at = __shfl_sync(full, give_at, 0), w = __shfl_sync(full, give_work, 0);
            if (lane < give && (int64_t)at + lane < qcap) *(volatile int32_t*)(q + at + lane) = give_id;
            if (lane == 0) {
                if ((int64_t)at + give > qcap) atomicExch(err, SCC_DEVERR_QUEUE_OVERFLOW);
                // a frontier that has grown wide goes back to the level-synchronous kernels
                if (w > a.async_bail) atomicExch(bail, 1);
            }
            give = 0;
        }
        net += list.push(edge && !(old & bit) && r0.x != REC_NONE, ent & ~(1 << REC_EDGE), r0, r1);
        while (longs) {
            const int l = __ffs(longs) - 1;
            longs &= longs - 1;
            const int32_t item = __shfl_sync(full, long_id, l);
            const int32_t v = a.live[item & REC_PLACE], ldir = (item >> REC_DIR) & 1;
            const int32_t c = __ldg(a.color + v);
            const int32_t* off = ldir ? a.r_begin : a.begin;
            const int32_t* adj = ldir ? a.r_node_idx : a.node_idx;
            const int32_t b = __ldg(off + v), e = __ldg(off + v + 1);
            if (lane == 0) my_edges += (uint32_t)(e - b);
            for (int32_t k0 = b; k0 < e; k0 += 32) {
                const int32_t w = k0 + lane < e ? __ldg(adj + k0 + lane) : v;
                const bool mine = w != v && __ldg(a.color + w) == c;
                const int32_t at = mine ? __ldg(place + w) : 0;
                const bool in = mine && (uint32_t)at < (uint32_t)a.live_count && a.live[at] == w;
                if (mine && !in) {
                    // not in the live list: the host's next frontier takes it
                    const unsigned mbit = 1u << (ldir + (w & 3) * 8);
                    if (!(atomicOr(reinterpret_cast<unsigned*>(a.mark + (w & ~3)), mbit) & mbit))
                        outside[atomicAdd(a.ctr + CTR_QLEN, 1)] = w | (ldir << DIR_SHIFT);
                }
                const int32_t x = at | (ldir << REC_DIR);
                const bool p2 = rec_claim(rec, pm, x | (1 << REC_EDGE), in, r0, r1);
                net += list.push(p2, x, r0, r1);
                if (list.count > REC_BUF - 64) {
                    // no room for the next 32: share the newest 32 at once
                    __syncwarp();
                    int32_t at2 = 0, w2 = 0;
                    if (lane == 0) { w2 = atomicAdd(work, net); at2 = atomicAdd(tail, 32); }
                    w2 = __shfl_sync(full, w2, 0);
                    at2 = __shfl_sync(full, at2, 0);
                    net = 0;
                    list.count -= 32;
                    if ((int64_t)at2 + 32 <= qcap) *(volatile int32_t*)(q + at2 + lane) = list.id[list.count + lane];
                    else if (lane == 0) atomicExch(err, SCC_DEVERR_QUEUE_OVERFLOW);
                    __syncwarp();
                }
            }
        }
        __syncwarp();
        if (list.count > REC_KEEP) {
            give = min(32, list.count - REC_KEEP);
            list.count -= give;
            give_id = lane < give ? list.id[list.count + lane] : 0;
            if (lane == 0) {
                give_work = atomicAdd(work, net) + net;
                give_at = atomicAdd(tail, give);
            }
            net = 0;
            __syncwarp();
        }
        // items that came for the tickets; on top of the list, so the next iteration
        // expands them: an item passes the queue once, which bounds the queue
        const unsigned got = __ballot_sync(full, came != -1);
        if (got) {
            if (came != -1) {
                *(volatile int32_t*)(q + ticket_at + lane) = -1;
                const int4* at = rec + (2LL * (came & REC_PLACE) + ((came >> REC_DIR) & 1)) * 2;
                r0 = __ldg(at);
                r1 = __ldg(at + 1);
            }
            ticket &= ~got;
            list.push(came != -1, came, r0, r1);      // already counted as work
        }
        __syncwarp();
        if (k == 0 && !got) {
            // nothing to do: publish, then wait for the tickets, the end, an error or a hand-back
            if (net != 0) {
                if (lane == 0) atomicAdd(work, net);
                net = 0;
            }
            ++idle;
            if ((idle & 7) == 1) {
                int32_t w = 1, e = 0, bl = 0;
                if (lane == 0) { w = rec_ld(work); e = rec_ld(err); bl = rec_ld(bail); }
                w = __shfl_sync(full, w, 0);
                e = __shfl_sync(full, e, 0);
                bl = __shfl_sync(full, bl, 0);
                if (w == 0 || e != 0 || bl != 0) break;
                if (w != last_work) { last_work = w; idle = 1; }     // progress elsewhere resets the limit
            }
            if (idle > idle_limit) {
                if (lane == 0) { atomicExch(err, SCC_DEVERR_WAIT_LIMIT); atomicExch(a.ctr + CTR_ERROR_INFO, 1); }
                break;
            }
            __nanosleep(idle < 64 ? 40 : 200);
            continue;
        }
        idle = 0;
        // the bail word, read every eighth iteration and looked at one later
        if ((++iter & 7) == 1 && __shfl_sync(full, stop, 0)) {
            // hand everything back: what is being shared to the queue, which the host
            // collects, the list straight to the host's frontier
            if (give) {
                const int32_t at = __shfl_sync(full, give_at, 0);
                if (lane < give && (int64_t)at + lane < qcap) *(volatile int32_t*)(q + at + lane) = give_id;
            }
            int32_t at = 0;
            if (lane == 0) at = atomicAdd(a.ctr + CTR_QLEN, list.count);
            at = __shfl_sync(full, at, 0);
            for (int32_t j = lane; j < list.count; j += 32)
                outside[at + j] = a.live[list.id[j] & REC_PLACE] | (((list.id[j] >> REC_DIR) & 1) << DIR_SHIFT);
            break;
        }
        if ((iter & 7) == 0 && lane == 0) stop = rec_ld(bail);
    }
    unsigned long long edges = my_edges;
    for (int o = 16; o > 0; o >>= 1) edges += __shfl_down_sync(full, edges, o);
    if (lane == 0) {
        atomicAdd(reinterpret_cast<unsigned long long*>(a.ctr + CTR_ASYNC_ITEMS), (unsigned long long)my_items);
        atomicAdd(reinterpret_cast<unsigned long long*>(a.ctr + CTR_ASYNC_EDGES), edges);
    }
}

// ------------------------------------------------------------------ host side
bool scc_impl_records_pay(const RoundArgs& a, const RecordSet& rs, int64_t left, unsigned long long live_edges,
                          int32_t maxdeg) {
    return !rs.unusable && !rs.outside && left >= REC_MIN_LEFT && maxdeg <= a.huge_deg &&
           live_edges <= REC_SPARSE * (unsigned long long)a.live_count;
}

static int rec_blocks(int device) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms;      // one block per SM, all resident: warps wait on one another's items
}

int scc_impl_reach_records(scc_state* s, RoundArgs& a, RecordSet& rs, const int32_t* qin, int32_t qlen, int32_t* qout,
                           int32_t* handed_back) {
    *handed_back = 0;
    cudaStream_t st = s->stream;
    const int32_t L = a.live_count;
    const size_t rec_bytes = sizeof(int32_t) * REC_W * 2 * (size_t)L;
    int32_t* place = s->aux;          // free during a traversal
    if (!rs.rec) {
        rs.st = st;
        void* nbr = nullptr;
        static_assert(REC_W == 8, "scc_record_bytes");
        if (s->drain_scratch >= 0 && scc_record_bytes(L) > s->drain_scratch) {
            rs.unusable = true;
            return SCC_OK;
        }
        if (scc_impl_malloc_async((void**)&rs.rec, rec_bytes, st) != cudaSuccess ||
            scc_impl_malloc_async((void**)&rs.pm, ((size_t)L + 3) & ~(size_t)3, st) != cudaSuccess ||
            scc_impl_malloc_async(&nbr, rec_bytes / 2, st) != cudaSuccess) {
            cudaGetLastError();
            rs.unusable = true;
            return SCC_OK;
        }
        k_rec_places<<<scc_blocks(L), SCC_THREADS, 0, st>>>(a.live, L, a.mark, place, rs.pm);
        SCC_LAUNCHED(s);
        k_rec_neighbours<<<scc_blocks(2LL * L), SCC_THREADS, 0, st>>>(a, place, (int4*)nbr, rs.rec);
        SCC_LAUNCHED(s);
        k_rec_grow<<<scc_blocks(2LL * L), SCC_THREADS, 0, st>>>(L, (const int4*)nbr, rs.rec);
        SCC_LAUNCHED(s);
        SCC_CUDA(cudaFreeAsync(nbr, st));
    } else {
        k_rec_places<<<scc_blocks(L), SCC_THREADS, 0, st>>>(a.live, L, a.mark, place, rs.pm);
        SCC_LAUNCHED(s);
    }
    const int64_t qcap = 2LL * s->n + 64;
    int32_t init[CTR_AWORK - CTR_AHEAD + 1] = {0};   // head, tail, work on separate lines
    // an injected failure announces one item that is never written: slot 0 stays empty
    const int32_t hole = scc_impl_take_wait_injection() ? 1 : 0;
    init[CTR_ATAIL - CTR_AHEAD] = hole;
    init[CTR_AWORK - CTR_AHEAD] = hole;
    SCC_CUDA(cudaMemcpyAsync(s->ctr + CTR_AHEAD, init, sizeof(init), cudaMemcpyHostToDevice, st));
    SCC_TRY(scc_zero_list(s, {CTR_ASYNC_ITEMS, CTR_ASYNC_ITEMS + 1, CTR_ASYNC_EDGES, CTR_ASYNC_EDGES + 1, CTR_ABAIL,
                              CTR_QLEN}));
    k_rec_items_in<<<scc_blocks(qlen), SCC_THREADS, 0, st>>>(qin, qlen, a.live, L, place, s->aq, s->ctr + CTR_ATAIL,
                                                            s->ctr + CTR_AWORK, qout, s->ctr + CTR_QLEN);
    SCC_LAUNCHED(s);
    if (s->ledger_on) SCC_CUDA(cudaEventRecord(s->lev[0], st));
    const int idle_polls = scc_impl_take_idle_injection();
    k_reach_records<<<rec_blocks(s->device), REC_THREADS, 0, st>>>(a, rs.rec, rs.pm, place, s->aq, qcap, qout,
                                                                  idle_polls > 0 ? idle_polls : REC_IDLE_LIMIT);
    SCC_LAUNCHED(s);
    if (s->ledger_on) SCC_CUDA(cudaEventRecord(s->lev[1], st));
    k_rec_marks_out<<<scc_blocks(L), SCC_THREADS, 0, st>>>(a.live, L, rs.pm, a.mark);
    SCC_LAUNCHED(s);
    s->traversal_steps++;
    SCC_TRY(scc_sync_counters(s));
    if (s->ledger_on) {
        float ms = 0.f;
        SCC_CUDA(cudaEventElapsedTime(&ms, s->lev[0], s->lev[1]));
        s->ledger_ms += ms;
        s->ledger_launches++;
        s->ledger_items += *reinterpret_cast<long long*>(s->h_ctr + CTR_ASYNC_ITEMS);
        s->ledger_edges += *reinterpret_cast<long long*>(s->h_ctr + CTR_ASYNC_EDGES);
    }
    int32_t items = s->h_ctr[CTR_QLEN];           // already in qout
    // class vertices outside the live list: the plain drain, which goes by vertex, does the rest
    if (items > 0 && !s->h_ctr[CTR_ABAIL]) rs.outside = true;
    const bool gave_up = s->h_ctr[CTR_ERROR] == SCC_DEVERR_WAIT_LIMIT && s->h_ctr[CTR_ERROR_INFO] == 1;
    if ((s->h_ctr[CTR_ABAIL] || (gave_up && s->h_ctr[CTR_AWORK] != 0)) && s->h_ctr[CTR_ATAIL] > 0) {
        const int32_t work = s->h_ctr[CTR_AWORK], tail = (int32_t)std::min<int64_t>(s->h_ctr[CTR_ATAIL], qcap);
        k_rec_items_out<<<scc_blocks(tail), SCC_THREADS, 0, st>>>(s->aq, tail, a.live, qout, s->ctr + CTR_QLEN);
        SCC_LAUNCHED(s);
        SCC_TRY(scc_sync_counters(s));
        // Idle warps gave up beside one warp's long chain, on which the work count
        // sits still; they held tickets, so what that warp shared afterwards
        // lies at places that nobody reads.  If that is all the work there is, it is handed back.
        if (!s->h_ctr[CTR_ABAIL] && s->h_ctr[CTR_QLEN] - items == work) s->h_ctr[CTR_AWORK] = 0;
        items = s->h_ctr[CTR_QLEN];
    }
    if (gave_up && (s->h_ctr[CTR_AWORK] == 0 || s->h_ctr[CTR_ABAIL])) {
        // the traversal is complete, or handed back, all the same: see the plain drain
        s->h_ctr[CTR_ERROR] = 0;
        SCC_CUDA(cudaMemsetAsync(s->ctr + CTR_ERROR, 0, sizeof(int32_t) * 2, st));
    }
    if (s->h_ctr[CTR_ERROR]) {
        SCC_CUDA(cudaMemsetAsync(s->aq, 0xFF, sizeof(int32_t) * (size_t)qcap, st));
        return scc_check_device_error(s);
    }
    *handed_back = items;
    if (scc_trace_on())
        fprintf(stderr, "[scc] reach records live=%d seeds=%d spilled=%d handed_back=%d items=%lld\n", L, qlen,
                s->h_ctr[CTR_ATAIL], items, *reinterpret_cast<long long*>(s->h_ctr + CTR_ASYNC_ITEMS));
    return SCC_OK;
}
