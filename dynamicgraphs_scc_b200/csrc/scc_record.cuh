// Record drain (scc_record.cu): interface for the traversal driver in scc_reach.cu.
#pragma once
#include "scc_round.cuh"

// Records cost a pass over the live vertices (96 bytes written and a few gathers
// each), so they pay where the wave still has far to go: a sparse round (a dense
// one ends in a few levels), no hub among its vertices (a warp would walk its
// LONG record alone), and at least REC_MIN_LEFT items to reach.
#define REC_SPARSE 10ull
#define REC_MIN_LEFT (1 << 14)

// One round's records, built at its first narrow frontier and kept until the
// round's traversal ends.  Scratch comes from the library's pool on the state's
// stream.
struct RecordSet {
    cudaStream_t st = nullptr;
    int4* rec = nullptr;          // [2 x live] records, REC_W entries each
    uint8_t* pm = nullptr;        // [live] marks by place in the live list
    bool unusable = false;        // scratch could not be had: the round keeps to the plain drain
    bool outside = false;         // the wave met class vertices outside the live list: so does the rest of the round
    ~RecordSet() {
        if (rec) cudaFreeAsync(rec, st);
        if (pm) cudaFreeAsync(pm, st);
    }
};

// Does a narrow frontier of this round go to the record drain?  left: items
// (vertices x directions) not reached yet; live_edges, maxdeg: total and
// largest in+out degree of the live vertices.
bool scc_impl_records_pay(const RoundArgs& a, const RecordSet& rs, int64_t left, unsigned long long live_edges,
                          int32_t maxdeg);
// Bytes of pool scratch a round of `live` vertices takes: records, their marks and, while they are made, neighbours.
static inline int64_t scc_record_bytes(int64_t live) { return 96 * live + ((live + 3) & ~3LL); }
// Drains the qlen items of qin.  On return either the traversal is complete
// (*handed_back = 0) or its *handed_back unexpanded items are in qout.  When
// rs.unusable comes back set, nothing was done.
int scc_impl_reach_records(scc_state* s, RoundArgs& a, RecordSet& rs, const int32_t* qin, int32_t qlen, int32_t* qout,
                           int32_t* handed_back);
