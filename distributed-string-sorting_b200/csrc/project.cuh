// The PEs' local orders, distinguishing prefixes, splitters and merged
// sequences as projections of one global sorted order; see project.cu.
#pragma once
#include "internal.cuh"

namespace dsss {

// One string set of the call: its positions [begin, end) in the global order
// and its splitters (nspl <= p - 1, the k-th the sample of sorted rank k * dist).
struct SetSplit {
    uint64_t begin, end;
    uint32_t nspl, dist;
};

struct ProjectLayout {
    uint32_t* hist;      // PE counts per tile of the global order, PE-major
    uint32_t* off;       // their exclusive scan
    void* scan;
    uint64_t* pb;        // npe + 1 PE bounds
    SetSplit* sets;
    uint32_t* bounds;    // npe x (p + 1): where PE g's strings for receiver r start
    uint32_t* start;     // global position where receiver (set, k)'s strings start
    uint32_t* flags;     // [0] a guard tripped, [1] ties cross a splitter (project_buckets)
    uint64_t tiles;
};

// n positions, nsets sets of p PEs.
void layout_project(Carve& c, ProjectLayout& L, uint64_t n, uint32_t nsets, uint32_t p);

// Pinned host bytes project_setup and project_read need.
uint64_t project_pin_bytes(uint32_t nsets, uint32_t p);

// Copies the PE bounds and the sets' splitter ranks (factor (p - 1) samples
// per PE) to the device through pin.
int project_setup(const ProjectLayout& L, uint32_t nsets, uint32_t p, const uint64_t* pb, uint32_t factor, void* pin,
                  cudaStream_t st);

// Local orders: pe[g] (the PE of global position g inside its set) and, with
// several sets, bucket[g] (set * p + pe), local_order, rank[g] (position in
// the PE's local order), and either the distinguishing prefixes in local order
// (dp) or, dp == nullptr, *lcp_sum += the sum of the PEs' local LCPs (edges:
// scratch of project_edge_words).  bucket may be pe itself with one set.
int project_local(const ProjectLayout& L, const ArenaDev& a, uint64_t n, uint32_t nsets, uint32_t p,
                  const uint32_t* ord, const uint32_t* lcp, const LenStats* stats, uint32_t* pe, uint32_t* bucket,
                  uint32_t* local_order, uint32_t* rank, uint32_t* dp, uint32_t* edges, unsigned long long* lcp_sum,
                  cudaStream_t st);
uint64_t project_edge_words(uint64_t n, uint32_t npe);

// Splitters and every PE's bounds against them (computePartition), from the
// global order.  Samples are cut to their distinguishing prefixes (cut ==
// nullptr) or to 200 (*cut / n + 5) bytes (the merge-sort path: *cut the sum
// of the local LCPs).  indexed: the sampler whose ties compare by index.
// merged (optional): the global LCPs, set to 0 where a receiver's strings
// start unless flags[1] is raised.
int project_partition(const ProjectLayout& L, const ArenaDev& a, uint64_t n, uint32_t nsets, uint32_t p,
                      uint32_t factor, int indexed, const unsigned long long* cut, const uint32_t* ord,
                      const uint32_t* lcp, const uint32_t* bucket, const uint32_t* rank, uint32_t* merged,
                      cudaStream_t st);

// Enqueues the read-back of the bounds and flags, and, after the stream is
// synchronised, turns them into intervals and receive counts (0: a guard
// tripped; ties: flags[1]).
int project_read_async(const ProjectLayout& L, uint32_t nsets, uint32_t p, void* pin, cudaStream_t st);
int project_read(uint32_t nsets, uint32_t p, const void* pin, uint64_t* intervals, uint64_t* recv_counts,
                 bool* ties);

// Receiver of every position (set * p + r), for the multisplit when equal
// strings on different PEs fall on different sides of a splitter.
int project_buckets(const ProjectLayout& L, uint64_t n, uint32_t p, const uint32_t* bucket, const uint32_t* rank,
                    uint32_t* dest_bucket, cudaStream_t st);

}  // namespace dsss
