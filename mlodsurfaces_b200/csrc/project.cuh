// project.cuh -- launch interface of the MLoD projection kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "mlods_internal.cuh"

namespace mlods
{

#ifndef MLODS_PROJECT_MIN_BLOCKS
#define MLODS_PROJECT_MIN_BLOCKS 10
#endif
#ifndef MLODS_PROJECT_STACK_CAP
#define MLODS_PROJECT_STACK_CAP 160
#endif
#ifndef MLODS_PROJECT_PAIR_MIN_BLOCKS
#define MLODS_PROJECT_PAIR_MIN_BLOCKS 7
#endif
#ifndef MLODS_PROJECT_PAIR_STACK_CAP
#define MLODS_PROJECT_PAIR_STACK_CAP 128
#endif
constexpr int kProjectThreads = 128;                          // 4 warps per block, one walk per warp at a time
constexpr int kProjectMinBlocks = MLODS_PROJECT_MIN_BLOCKS;  // 10 -> 40 warps per SM, <= 48 registers
constexpr int kProjectStackCap = MLODS_PROJECT_STACK_CAP;    // sibling ranges per warp (24 bytes each)
// the paired walk (two queries per warp): more registers and a wider stack entry
constexpr int kProjectPairMinBlocks = MLODS_PROJECT_PAIR_MIN_BLOCKS;
constexpr int kProjectPairStackCap = MLODS_PROJECT_PAIR_STACK_CAP;

// the wide walk (one query per warp, two nodes a lane): 128 registers, a stack
// of whole 64-node rounds (24 bytes a range)
constexpr int kWideMinBlocks = 4;
constexpr int kWideCap = 288;

// One tree and its projection settings, plus the query buffers it serves.
struct CloudArgs {
    NodeArrays nodes;
    double o0, o1, o2;      // local frame origin
    KernelConsts kc;
    float cutoff;
    int min_depth;
    float step_max;
    int rule;               // MLODS_BLEND_*
    int n_iter;
    int conv_mode;          // MLODS_CONVERGE_*
    float conv_tol;
    const float* q_in;      // world xyz
    float* out_p;           // world xyz (may alias q_in), or relative to the origin with local_out
    float* out_n;
    int local_out;          // 1: out_p holds the result relative to (o0, o1, o2)
    int qpw;                // the tree's walk schedule (queries per warp) for launches of its own
    int64_t n_pts;          // points of the tree
    int64_t n_nodes;        // and its nodes
    int64_t n_call;         // queries of the whole call or request on this tree
    float prune_thr;        // > 0: kernel-weight pruning threshold (prune_tol * w(0) * mean sample area)
};

// Whether a projection may take another form than the narrow walk.  Not with one
// iteration: that is the projection behind the dual-contouring field and the
// cell grids, whose signs and cells are whole numbers that follow the float
// sums of the narrow walk bit for bit; and not with pruning, which is a variant
// of the narrow walk.
inline bool walks_freely(const CloudArgs& c) { return c.n_iter >= 2 && !(c.prune_thr > 0.f); }

// Whether a one-query-per-warp projection takes the wide walk.  Where it does not
// fill its 64 lanes the narrow one is faster (100k queries on 100k points, 3
// iterations but where said, narrow / wide, ms), but for calls that it holds in
// flight at once (2,368 queries) later than for others:
//  - its stack holds fewer ranges than the narrow walk's for twice the nodes, and
//    near its end it pops one range a round: cutoff 6 10.3 / 9.7 and 6.6 / 6.1,
//    9 19.3 / 23.9, 14 39 / 68; min_depth 4 9.6 / 8.3, 5 30.7 / 31.6, 6 110 / 230; 1k
//    queries cutoff 9 0.61 / 0.44, 14 1.06 / 1.05, min_depth 5 1.00 / 0.63, 6 2.4 / 2.6;
//  - it takes 32 of the points of a leaf of more a round: 10.2 points a node
//    11.3 / 10.9, 15.4 11.9 / 13.9, 25 25.0 / 30.7, 87 53 / 78; 25 1k queries 1.29 /
//    0.79, 3k 1.50 / 1.45, 4k 1.69 / 1.66, 62 1k 2.27 / 1.63, 4k 2.67 / 2.95;
//  - short walks spend their time in rounds of a few nodes (10 iterations):
//    cutoff 2.5 6.0 / 6.0 and 8.4 / 7.8, 2 4.6 / 5.0 and 6.1 / 5.9, 1 3.4 / 4.4;
//    calls of few queries, which are bound by the number of rounds, gain all the
//    same: cutoff 2 6k queries 0.46 / 0.38, 14k 0.77 / 0.76, 20k 0.98 / 1.01, 50k
//    2.31 / 2.49; cutoff 1 6k 0.39 / 0.34, 8k 0.44 / 0.44, 14k 0.63 / 0.69.
// The rule looks at nothing that a batch or a server changes, so a query's result
// does not depend on what it is projected with, but for the number of queries.
inline bool walks_wide(const CloudArgs& c)
{
    if (!walks_freely(c)) return false;
    const bool few = c.n_call <= 2368;
    if (c.cutoff > (few ? 9.f : 6.f) || c.min_depth > (few ? 5 : 4)) return false;
    if (!few && c.n_pts > 10 * c.n_nodes) return false;
    return c.cutoff >= 2.5f || c.n_call <= (c.cutoff < 2.f ? 8192 : 16384);
}

struct ProjectArgs {
    CloudArgs cloud;
    const uint32_t* order;  // processing order (Morton), or nullptr
    int64_t nq;
    unsigned int* counter;  // work counter, zero before launch
    int64_t* stats;         // [0] query-node visits, [1] max stack, [2] overflows, [3] counter, [4] rounds,
                            // [5] query-iterations, [6] lane visits (a node shared by a warp's queries once)
    int queries_per_warp = 1;  // 1, or 2: consecutive queries of `order` share one walk
    uint32_t order_base = 0;   // subtracted from every entry of `order` (a tree's slice of a batch order)
};

// The surroundings of a tree's root box, widened by half its largest extent.
struct QueryBox {
    float lo[3], hi[3];
    float extent;  // the root box's largest
};
__host__ __device__ inline bool in_box(const QueryBox& b, const float* q)
{
    return q[0] >= b.lo[0] && q[0] <= b.hi[0] && q[1] >= b.lo[1] && q[1] <= b.hi[1] && q[2] >= b.lo[2] && q[2] <= b.hi[2];
}
// Whether queries of which `outside` lie outside that box walk in packets where
// walks_in_packets allows it.  Far from the cloud neighbours in Morton order are
// no neighbours, and a few packets of queries strewn over the cloud run long after
// the others: 400k queries on 400k points, 3 iterations, with 0 / 12 / 24 / 35 / 44 /
// 49 / 70 / 96 % outside in packets 11.7 / 12.3 / 11.6 / 11.8 / 11.2 / 11.3 / 11.6 / 9.4 ms,
// one query per warp 15.5 / 14.2 / 12.3 / 12.1 / 10.4 / 10.3 / 8.7 / 2.8; 350k on 700k
// points 12.6 / 13.5 / 12.5 / 12.8 / 12.1 / 12.6 / 13.4 / 11.0, not 14.6 / 13.3 / 11.5 / 11.4 / 9.8 /
// 9.7 / 8.2 / 2.6; 1M on 1M points, two queries per warp, at 0 / 12 / 18 % 28.4 / 28.6 / 29.6,
// not 30.0 / 29.1 / 28.3.
__host__ __device__ inline bool packets_pay(unsigned int outside, int64_t nq) { return 8 * int64_t(outside) <= nq; }

// Many trees in ONE persistent launch.  The queries of cloud c occupy the
// global range [base[c], base[c] + len[c]) of the concatenated buffers, and
// the same range of slots of the batch order: order[slot] is the global
// index of the query processed at that slot (nullptr: slot = query index).
// The warps of the queue kernel take queries_per_warp consecutive slots of
// one cloud at a time from a device counter, as the single-tree kernel does
// over one cloud.
struct QueueArgs {
    const CloudArgs* clouds;   // host array: each cloud's q_in / out_p / out_n address its own range
    const int64_t* base;       // host array: first global query of each cloud
    const int64_t* len;        // host array: its query count
    int n_clouds;
    const uint32_t* order;     // device
    unsigned long long* counters;  // device: one 64-bit slot counter per launch group, zero before launch
    int64_t* stats;            // device, as ProjectArgs::stats
    int line_order = 0;        // kQueueMostWorkFirst or kQueueBySpecialisation
};

// The order of the clouds along a launch's slot line: the clouds with the
// most work (queries x iterations) first, or grouped by walk specialisation
// (kernel family, terms, blend rule; the groups with the most work first,
// the clouds inside each group likewise), so that the warps working at any
// moment run the same code.
constexpr int kQueueMostWorkFirst = 0;
constexpr int kQueueBySpecialisation = 1;

// Clouds per launch of the queue kernel: their launch arguments travel by
// value in the kernel's parameters (within the 32 KB parameter limit); a
// batch of more clouds runs as consecutive launches of up to this many.
constexpr int kQueueMaxClouds = 80;
// (clouds that walk wide and clouds that do not are grouped apart: a mixed
// batch uses at most one group, and one counter, more)
inline int queue_groups(int n_clouds) { return (n_clouds + kQueueMaxClouds - 1) / kQueueMaxClouds; }

// The queue kernel over every group of clouds (usually one launch); every
// cloud is walked queries_per_warp (1 or 2) queries at a time, the pairs
// aligned to the cloud's first slot, so that results equal per-tree
// launches with the same schedule bit for bit.
cudaError_t launch_mlod_queue(const QueueArgs& a, int queries_per_warp, int sm_count, int grid_pct, cudaStream_t s);

// Queries the single-tree walk holds in flight when every SM runs its
// blocks (resident warps x queries per warp); wide: one query per warp in the
// wide walk.
int64_t project_resident_queries(int queries_per_warp, bool wide, int sm_count);

// Per-cloud frame used to key queries: the cloud's rank in the batch order
// (clouds of a batch keep their own rank: their slots are their query range)
// and its Morton frame.
struct BatchFrame {
    double o0, o1, o2;
    float inv_ext;
    uint32_t rank;
};

// Whether a projection of n queries runs in packets of 32 (packet.cu).  Where
// the packets fill the GPU several times over (148 SMs x 28 warps x 32 queries =
// 133k; the last packets run alone for about 3 ms) and the queries lie about as
// close as the points, so that neighbours need the same nodes.  10 iterations on
// the torus / blobs (four Gaussians) / knot (rational), packets, not one query per
// warp: 350k queries on 350k points 34.0 / 25.5 / 14.1 ms, not 40.3 / 30.4 / 18.4, on
// 700k points 42.1 / 31.8 / 16.9, not 43.7 / 32.8 / 19.6, but 150k on 150k 18.0 / 12.8 /
// 7.2, not 15.7 / 12.0 / 7.4, 200k on 600k 27.9 / 24.0 / 12.4, not 24.6 / 18.5 / 11.1.
// Two or four queries per warp already share nodes: 800k on 800k 74.3 / 53.5 / 29.5,
// not 76.2 / 55.4 / 33.5 with two, 1M on 1M 93.0 / 66.4 / 35.9, not 98.3 / 71.4 / 42.8, but
// 400k on 500k 41.1 / 30.5 / 16.3, not 36.1 / 26.3 / 16.2, 500k on 2M 71.9 / 51.8 / 29.2,
// not 56.7 / 41.3 / 24.2; 650k on 650k 60.1 / 45.1 / 24.2, not 60.2 / 43.7 / 26.7.  Not
// with one iteration (walks_freely gives the reason), with pruning, or stopping at a tolerance (a
// query's end does not fit the state kept between the launches); exact
// convergence returns the bits of a run without it, which is promised with one
// query per warp, so there it follows; and so does a call without Morton order
// (ordered: whether the call asks for it), whose results are promised to be the
// same: the packets order the queries themselves.
constexpr int64_t kPacketMinQueries = 350000;
inline bool walks_in_packets(const CloudArgs& c, int qpw, int64_t n, bool ordered)
{
    if (!walks_freely(c) || n >= (int64_t(1) << 32) - 64) return false;
    if (c.conv_mode != MLODS_CONVERGE_OFF && !(c.conv_mode == MLODS_CONVERGE_EXACT && qpw == 1)) return false;
    return qpw == 1 ? n >= kPacketMinQueries && 2 * n >= c.n_pts : ordered && n >= 800000 && 4 * n >= 3 * c.n_pts;
}
// The whole projection in packets: a's launch arguments; the order of the
// queries (made here where a.order is null) is rewritten after the first
// iteration (order: a.nq entries, may be a.order; order_temp:
// query_order_temp_bytes(a.nq) bytes).  Where too many queries lie outside `box`
// the walk of the setting runs instead, which the device decides (a.counter[1]:
// their number, zero before launch), unless `near` says that they do not.
cudaError_t launch_mlod_packets(const ProjectArgs& a, uint32_t* order, void* order_temp, const QueryBox& box, bool near,
                                int sm_count, cudaStream_t s);

cudaError_t launch_mlod_project(const ProjectArgs& a, int ktype, int rule, int sm_count, cudaStream_t s);

// Swaps query points invalid[i] and end_valid-1-i (GPUUtils.cu:413-424).
cudaError_t launch_reorganize(float* d_q, const uint32_t* d_invalid, int64_t n_invalid, uint32_t end_valid,
                              cudaStream_t s);

// Morton order of queries on a 1024^3 grid over the root box (the reference
// orders its queries on a 64^3 grid, Pn.cpp:388-445).  d_order receives the
// query indices in processing order.
size_t query_order_temp_bytes(int64_t n);
cudaError_t compute_query_order(const float* d_q, int64_t n, const double origin[3], float extent, uint32_t* d_order,
                                void* temp, cudaStream_t s);
// Same for a batch: grouped by cloud rank, Morton order inside each cloud
// (input order when morton is false).
cudaError_t compute_batch_order(const float* d_q, int64_t n, const int64_t* d_q_offsets, int n_clouds,
                                const BatchFrame* d_frames, bool morton, uint32_t* d_order, void* temp,
                                cudaStream_t s);

}  // namespace mlods
