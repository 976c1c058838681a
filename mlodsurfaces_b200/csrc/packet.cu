// packet.cu -- MLoD projection of many queries: a warp walks the tree once for
// a packet of 32 neighbouring queries, lanes = queries.
//
// The walks of project.cu give a warp one, two or four queries and its lanes the
// nodes.  With enough queries to fill the GPU the other assignment costs fewer
// instructions and a fraction of the loads: 32 queries that are neighbours in
// Morton order share one depth-first walk of the union of their nodes, every
// lane evaluating the same node for its own query.  There is no scan, no
// shuffle and no segmented sum: the recursion
//     R(n) = sum_c [beta_c R(c) + (1 - beta_c) rho_c w_n S_n]
// (project.cu) is summed in its own form, an opened node adding
// f_n w_n sum_c (1 - beta_c) rho_c times its own moments S_n once its children
// have been evaluated.
//
// Of a packet's 32 queries 0.71 need the node they evaluate; 5.9 instructions of
// a warp for each query that does, all in all (80 % of the issue slots), against
// 6.8 with two queries per warp and 8.1 in the wide walk: 2M four-Gaussian
// queries, 10 iterations, 138 ms (two per warp 158, one 212); 500k rational, 5
// iterations, 8.3 ms (9.4, 12.8).  Two queries or two children a lane in packed
// f32x2 instructions issue as many (the operands' pairs cost the moves) and ran at
// 160-210 ms.
//
// A query's sums depend on its own walk only: the union's depth-first order
// restricted to the nodes a query needs is that query's depth-first order, and
// lanes for which a range is not live add nothing.  Results therefore do not
// depend on which queries share a warp, nor on the order the queries are in.
#include <algorithm>
#include <cmath>

#include "project.cuh"
#include "tree.cuh"
#include "walk.cuh"

namespace mlods
{
namespace
{
constexpr uint32_t kFull = 0xffffffffu;
// Stack entry: {first child, count | level | flags, live queries, node}.
constexpr int kPkLevelShift = 24;
constexpr uint32_t kPkLevelMask = 0xFu;
// A lane adds about 1200 terms an iteration.  It keeps them in blocks, ended by
// the ranges up to this level that its query needs, and the next block starts
// from what rounding left out of the total (the fast two-sum's error term), so
// that only the roundings within a block stay.  Normals off FP64 (rms, 1e-7) for
// one sum / two plain levels of blocks / this one at 5, 6, 7, 8, every level,
// beside one query per warp: 400k four-Gaussian queries - / 3.04 / 2.11, 1.71,
// 1.95, 1.60, 1.60 beside 1.63; 500k rational - / 2.81 / 2.75, 2.64, 2.60, 2.58,
// 2.58 beside 2.59; 200k four-Gaussian 3.8 in one sum beside 1.7.  2M queries at
// 5, 6, 7, 8, every level: 135.8, 136.6, 137.1, 138.2, 140.7 ms.
constexpr uint32_t kPkBlockLevel = 8;
constexpr uint32_t kPkNoBlend = 1u << 31;
constexpr uint32_t kPkLastOnly = 1u << 30;  // CPU rule multi-point leaf: only the last point is weighted
// A range holds at most 8 nodes (a multi-point leaf's points push nothing) and
// the walk is depth first: at most 7 entries wait per level above the deepest.
constexpr int kPkCap = 7 * kMaxTreeDepth + 4;
// The factors f of the bottom entries live in shared memory, those above (an
// eighth of the pops) in local memory: a full-height stack in shared memory would halve
// the resident warps.
constexpr int kPkRows = 24;
constexpr int kPkThreads = 128;
// 7 blocks of 4 warps (72 registers): the walk is bound by issue (80 % of the
// slots at 6.7 warps a scheduler) and by the latency of its dependent chains (70 %
// at 5.2).  2M four-Gaussian / 500k rational workload at 6 / 7 / 8 blocks: 155 /
// 138 / 141 and 9.2 / 8.3 / 8.8 ms.
constexpr int kPkMinBlocks = 7;
// State of a query between two launches of one projection, kept in the output
// buffers: the iterate in the local frame, or (this pattern in the normal's
// first word) a query whose result is final.
constexpr uint32_t kPkFailed = 0x7fc0dead;

// One launch over queries that consecutive places of `order` name.
struct PacketArgs {
    CloudArgs cloud;
    const uint32_t* order;
    uint32_t order_base;    // subtracted from every entry of `order`
    int64_t nq;
    unsigned int* counter;  // work counter, zero before launch
    int64_t* stats;         // as ProjectArgs::stats
    int n_iter;             // iterations of this launch
    int resume;             // 1: an earlier launch of this projection left the queries' state in the outputs
    int more;               // 1: another launch goes on from the state this one leaves
    const unsigned int* outside;  // if set: the launch walks only where packets_pay(*outside, nq)
};

struct __align__(16) PacketWarp {
    float4 rec[32];  // the range's records: geom, pm, nc, aux of up to 8 children
    float4 par[4];   // those of the node above
    uint4 ent[kPkCap];
    float f[kPkRows][32];
};

struct Moments {
    float v[9];
    __device__ __forceinline__ void add(float coef, float m, float px, float py, float pz, float d2, float4 n4, float cpp)
    {
        const float cm = coef * m;
        v[0] += cm;
        v[1] = fmaf(coef, n4.x, v[1]);
        v[2] = fmaf(coef, n4.y, v[2]);
        v[3] = fmaf(coef, n4.z, v[3]);
        v[4] = fmaf(cm, px, v[4]);
        v[5] = fmaf(cm, py, v[5]);
        v[6] = fmaf(cm, pz, v[6]);
        v[7] = fmaf(coef, fmaf(px, n4.x, fmaf(py, n4.y, fmaf(pz, n4.z, n4.w))), v[7]);
        v[8] = fmaf(coef, fmaf(d2, m, cpp), v[8]);
    }
};

// Queries outside the box.
__global__ void count_outside_kernel(const float* __restrict__ q, int64_t n, QueryBox box, unsigned int* __restrict__ outside)
{
    unsigned int c = 0;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const float p[3] = {q[3 * i], q[3 * i + 1], q[3 * i + 2]};
        c += in_box(box, p) ? 0u : 1u;
    }
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(outside, c);
}

// The other walk's work counter: at its end, so that its warps find nothing to
// do, where the packets will walk (a look at `outside` in those kernels cost calls
// of a thousand queries 1 %).
__global__ void end_counter_kernel(const unsigned int* __restrict__ outside, int64_t nq, unsigned int* __restrict__ counter)
{
    *counter = packets_pay(*outside, nq) ? (unsigned int)nq : 0u;
}

template <int KTYPE, int NSIG, int RULE>
__global__ void __launch_bounds__(kPkThreads, kPkMinBlocks) mlod_packet_kernel(PacketArgs a)
{
    if (a.outside && !packets_pay(*a.outside, a.nq)) return;
    constexpr bool gpu_rule = RULE == MLODS_BLEND_GPU;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PacketWarp& sm = reinterpret_cast<PacketWarp*>(smem_raw)[threadIdx.x >> 5];
    const CloudArgs& c = a.cloud;
    const int lane = threadIdx.x & 31;
    const float cutoff = c.cutoff;
    const int min_depth = c.min_depth;
    // the lane's share of a range's records: array lane >> 3 of child lane & 7
    const int arr = lane >> 3, kid = lane & 7;
    const float4* const my_arr = arr == 0 ? c.nodes.geom : (arr == 1 ? c.nodes.pm : (arr == 2 ? c.nodes.nc : c.nodes.aux));
    const float4* const par_arr = lane == 0 ? c.nodes.geom : (lane == 1 ? c.nodes.pm : (lane == 2 ? c.nodes.nc : c.nodes.aux));
    float f_high[kPkCap - kPkRows];
    unsigned long long visits = 0, evals = 0, rounds = 0, iterations = 0;
    int max_top = 0;

    for (;;) {
        unsigned int qs = 0;
        if (lane == 0) qs = atomicAdd(a.counter, 32u);
        qs = __shfl_sync(kFull, qs, 0);
        if (int64_t(qs) >= a.nq) break;
        const bool mine = int64_t(qs) + lane < a.nq;
        uint32_t my_q = qs + uint32_t(mine ? lane : 0);
        if (a.order) my_q = __ldg(a.order + my_q) - a.order_base;
        double qd[3];
        float nrm[3] = {0.f, 0.f, 0.f};
        bool failed = false, done = !mine;
        bool keep = false;  // final before this launch: nothing but the normal is left to write
        if (a.resume) {
            const float* ip = c.out_p + 3 * int64_t(my_q);
            qd[0] = ip[0];
            qd[1] = ip[1];
            qd[2] = ip[2];
            if (__float_as_uint(c.out_n[3 * int64_t(my_q)]) == kPkFailed) keep = done = failed = true;
        } else {
            const float* ip = c.q_in + 3 * int64_t(my_q);
            qd[0] = double(ip[0]) - c.o0;
            qd[1] = double(ip[1]) - c.o1;
            qd[2] = double(ip[2]) - c.o2;
        }
        for (int it = 0; it < a.n_iter; ++it) {
            const float qx = float(qd[0]), qy = float(qd[1]), qz = float(qd[2]);
            // a NaN iterate would open every node and fail; it fails at once
            if (!done && !(qx == qx && qy == qy && qz == qz)) failed = done = true;
            const uint32_t live_all = __ballot_sync(kFull, !done);
            if (live_all == 0u) break;
            Moments acc;
            float sum[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) acc.v[k] = sum[k] = 0.f;
            uint32_t n_visits = 0, n_evals = 0, n_rounds = 0;
            int top = 1;
            if (lane == 0) sm.ent[0] = make_uint4(0u, 1u | kPkNoBlend, live_all, 0u);  // the root alone
            sm.f[0][lane] = 1.f;
            __syncwarp();
            while (top > 0) {
                --top;
                const uint4 e = sm.ent[top];
                const float f_par = top < kPkRows ? sm.f[top][lane] : f_high[top - kPkRows];
                uint32_t first = e.x;
                int left = int(e.y & kCountMask);
                const bool blend = !(e.y & kPkNoBlend);
                const bool live = (e.z >> lane) & 1u;
                float4 v = __ldg(my_arr + first + uint32_t(min(kid, left - 1)));
                float4 pv = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < 4) pv = __ldg(par_arr + e.w);
                const uint32_t level = (e.y >> kPkLevelShift) & kPkLevelMask;
                if (level <= kPkBlockLevel && live) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        const float t = sum[k] + acc.v[k];
                        acc.v[k] -= t - sum[k];  // what the sum's rounding left out
                        sum[k] = t;
                    }
                }
                n_visits += uint32_t(__popc(e.z) * left);
                n_evals += uint32_t(left);
                ++n_rounds;
                float g = 0.f, dP = 0.f, pdP = 0.f, K = 0.f;
                const float n_range = float(left);
                for (;;) {
                    const int m = left < 8 ? left : 8;
                    // ---- stage the records; a child's distance beyond which it
                    // ends a query's walk (none for a leaf; infinite for what is
                    // opened whatever its distance, the points of a multi-point
                    // leaf and the children of a node above min_depth) takes the
                    // place of its parent index
                    if (arr == 0) v.w *= cutoff;
                    const float cr = __shfl_sync(kFull, v.w, kid);
                    const uint32_t info_s = __float_as_uint(v.z);
                    const bool leaf_s = (info_s & kLeafBit) != 0;
                    const bool all_s = leaf_s ? (info_s & kMultiBit) != 0 : node_depth(info_s) < min_depth;
                    if (arr == 3) v.w = all_s ? INFINITY : (leaf_s ? -1.f : cr);
                    __syncwarp();  // every lane is done with the previous records
                    sm.rec[lane] = v;
                    if (lane < 4) sm.par[lane] = pv;
                    __syncwarp();
                    if (blend) {
                        const float4 g4 = sm.par[0], p4 = sm.par[1];
                        const float cx = g4.x - qx, cy = g4.y - qy, cz = g4.z - qz;
                        dP = cutoff * g4.w - sqrtf(fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
                        pdP = kPiRef * dP;
                        const float px = p4.x - qx, py = p4.y - qy, pz = p4.z - qz;
                        const float w = weight_n<KTYPE, NSIG>(c.kc, fmaf(px, px, fmaf(py, py, pz * pz)));
                        g = f_par * w * rcp_fast(gpu_rule ? p4.w : n_range);
                    }
                    const float fh = 0.5f * f_par;
                    for (int ch = 0; ch < m; ++ch) {
                        const float4 g4 = sm.rec[ch], p4 = sm.rec[8 + ch], x4 = sm.rec[24 + ch];
                        const float cx = g4.x - qx, cy = g4.y - qy, cz = g4.z - qz;
                        const float dist = sqrtf(fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
                        float f = f_par;
                        if (blend) {
                            // beta = (1 - cos) / 2
                            const float h = __cosf(pdP * rcp_fast(dP + fmaxf(dist - g4.w, 0.f)));
                            f = fmaf(-fh, h, fh);
                            const float b1 = fmaf(0.5f, h, 0.5f);
                            K = gpu_rule ? fmaf(b1, p4.w, K) : K + b1;
                        } else if (!gpu_rule && (e.y & kPkLastOnly)) {
                            if (left > 8 || ch != m - 1) f = 0.f;
                        }
                        const bool far = dist > x4.w;
                        const uint32_t nb = __ballot_sync(kFull, live && !far);
                        const float4 n4 = sm.rec[16 + ch];
                        const float px = p4.x - qx, py = p4.y - qy, pz = p4.z - qz;
                        const float d2 = fmaf(px, px, fmaf(py, py, pz * pz));
                        float coef = f * weight_n<KTYPE, NSIG>(c.kc, d2);
                        coef = live && far ? coef : 0.f;
                        acc.add(coef, p4.w, px, py, pz, d2, n4, x4.x);
                        if (nb) {
                            const uint32_t info = __float_as_uint(x4.z);
                            const bool leaf = (info & kLeafBit) != 0;
                            const uint32_t flags = leaf || node_depth(info) < min_depth
                                                       ? kPkNoBlend | (leaf && !gpu_rule ? kPkLastOnly : 0u)
                                                       : 0u;
                            if (lane == 0)
                                sm.ent[top] = make_uint4(__float_as_uint(x4.y),
                                                         node_count(info) | ((level + 1u) << kPkLevelShift) | flags, nb,
                                                         first + uint32_t(ch));
                            if (top < kPkRows) sm.f[top][lane] = f;
                            else f_high[top - kPkRows] = f;
                            ++top;
                        }
                    }
                    left -= m;
                    if (left <= 0) break;
                    first += 8u;  // the next points of a multi-point leaf
                    v = __ldg(my_arr + first + uint32_t(min(kid, left - 1)));
                }
                if (blend) {
                    const float4 p4 = sm.par[1], n4 = sm.par[2], x4 = sm.par[3];
                    const float px = p4.x - qx, py = p4.y - qy, pz = p4.z - qz;
                    acc.add(live ? K * g : 0.f, p4.w, px, py, pz, fmaf(px, px, fmaf(py, py, pz * pz)), n4, x4.x);
                }
                max_top = max(max_top, top);
                __syncwarp();
            }
            visits += n_visits;
            evals += n_evals;
            rounds += n_rounds;
            iterations += __popc(live_all);
#pragma unroll
            for (int k = 0; k < 9; ++k) sum[k] += acc.v[k];
            if (!done) {
                double xr[3] = {0.0, 0.0, 0.0};
                if (!fit_sphere(sum, double(c.step_max), gpu_rule, xr, nrm)) {
                    failed = done = true;
                } else {
                    qd[0] = double(qx) + xr[0];
                    qd[1] = double(qy) + xr[1];
                    qd[2] = double(qz) + xr[2];
                    if (c.conv_mode == MLODS_CONVERGE_EXACT) {
                        done = float(qd[0]) == qx && float(qd[1]) == qy && float(qd[2]) == qz;
                    } else if (c.conv_mode == MLODS_CONVERGE_TOL) {
                        done = xr[0] * xr[0] + xr[1] * xr[1] + xr[2] * xr[2] < double(c.conv_tol) * double(c.conv_tol);
                    }
                }
            }
        }
        if (mine) {
            float* op = c.out_p + 3 * int64_t(my_q);
            float* on = c.out_n + 3 * int64_t(my_q);
            if (!keep) {
                // a query that goes on in another launch keeps the float
                // iterate that launch would evaluate
                const bool local = c.local_out || (a.more && !failed);
                op[0] = float(local ? qd[0] : qd[0] + c.o0);
                op[1] = float(local ? qd[1] : qd[1] + c.o1);
                op[2] = float(local ? qd[2] : qd[2] + c.o2);
            }
            on[0] = failed ? (a.more ? __uint_as_float(kPkFailed) : 0.f) : nrm[0];
            on[1] = failed ? 0.f : nrm[1];
            on[2] = failed ? 0.f : nrm[2];
        }
    }
    if (lane == 0 && a.stats) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[0]), visits);
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[4]), rounds);
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[5]), iterations);
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.stats[6]), evals);
        atomicMax(reinterpret_cast<unsigned long long*>(&a.stats[1]), (unsigned long long)max_top);
    }
}

template <int KTYPE, int NSIG, int RULE>
cudaError_t launch_packet_typed(const PacketArgs& a, int sm_count, cudaStream_t s)
{
    auto kern = mlod_packet_kernel<KTYPE, NSIG, RULE>;
    const size_t smem = sizeof(PacketWarp) * (kPkThreads / 32);
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPkThreads, smem);
    if (e != cudaSuccess) return e;
    const int64_t grid = std::min<int64_t>(int64_t(std::max(per_sm, 1)) * sm_count, (a.nq + kPkThreads - 1) / kPkThreads);
    kern<<<unsigned(std::max<int64_t>(grid, 1)), kPkThreads, smem, s>>>(a);
    note_launch();
    return cudaGetLastError();
}

template <int RULE>
cudaError_t launch_packet_rule(const PacketArgs& a, int sm_count, cudaStream_t s)
{
    const KernelConsts& kc = a.cloud.kc;
    if (kc.type == MLODS_GAUSSIAN) return launch_packet_typed<MLODS_GAUSSIAN, 0, RULE>(a, sm_count, s);
    if (kc.type == MLODS_SINGULAR) return launch_packet_typed<MLODS_SINGULAR, 0, RULE>(a, sm_count, s);
    switch (kc.nsig) {
    case 2: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 2, RULE>(a, sm_count, s);
    case 3: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 3, RULE>(a, sm_count, s);
    case 4: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 4, RULE>(a, sm_count, s);
    case 5: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 5, RULE>(a, sm_count, s);
    case 6: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 6, RULE>(a, sm_count, s);
    case 8: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 8, RULE>(a, sm_count, s);
    default: return launch_packet_typed<MLODS_GAUSSIAN_MULTIPLE, 0, RULE>(a, sm_count, s);
    }
}
}  // namespace

// One iteration, the order of the queries where it has left them -- on the
// surface, where neighbours stay neighbours -- and the other iterations: of the
// union's nodes 0.74 instead of 0.52 are then needed by a query.
cudaError_t launch_mlod_packets(const ProjectArgs& a, uint32_t* order, void* order_temp, const QueryBox& box, bool near,
                                int sm_count, cudaStream_t s)
{
    auto launch = [&](const PacketArgs& p) {
        return p.cloud.rule == MLODS_BLEND_GPU ? launch_packet_rule<MLODS_BLEND_GPU>(p, sm_count, s)
                                               : launch_packet_rule<MLODS_BLEND_CPU>(p, sm_count, s);
    };
    PacketArgs p;
    p.cloud = a.cloud;
    p.order = a.order;
    p.order_base = a.order_base;
    p.nq = a.nq;
    p.counter = a.counter;
    p.stats = a.stats;
    p.n_iter = 1;
    p.resume = 0;
    p.more = 1;
    p.outside = nullptr;
    cudaError_t e = cudaSuccess;
    if (!p.order) {
        const double origin[3] = {a.cloud.o0, a.cloud.o1, a.cloud.o2};
        e = compute_query_order(a.cloud.q_in, a.nq, origin, box.extent, order, order_temp, s);
        p.order = order;
        p.order_base = 0;
    }
    if (e == cudaSuccess && !near) {
        count_outside_kernel<<<unsigned(sm_count) * 4, 256, 0, s>>>(a.cloud.q_in, a.nq, box, a.counter + 1);
        note_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        p.outside = a.counter + 1;
        end_counter_kernel<<<1, 1, 0, s>>>(p.outside, a.nq, a.counter);
        note_launch();
        e = cudaGetLastError();
        ProjectArgs w = a;
        w.order = p.order;
        w.order_base = p.order_base;
        if (e == cudaSuccess) e = launch_mlod_project(w, w.cloud.kc.type, w.cloud.rule, sm_count, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned int), s);
    }
    if (e == cudaSuccess) e = launch(p);
    const double frame[3] = {0.0, 0.0, 0.0};  // the state is in the tree's frame
    if (e == cudaSuccess) e = compute_query_order(a.cloud.out_p, a.nq, frame, box.extent, order, order_temp, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    p.order = order;
    p.order_base = 0;
    p.n_iter = a.cloud.n_iter - 1;
    p.resume = 1;
    p.more = 0;
    return launch(p);
}

}  // namespace mlods
