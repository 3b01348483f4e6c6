// Routing, deterministic dispatch and the activation quantiser.
#include <cooperative_groups.h>
#include <stdio.h>

#include "common.cuh"
#include "kernels.cuh"
#include "tc_plan.cuh"

namespace q36 {

// ---------------------------------------------------------------- router
// One warp per token row; each lane holds n_expert/32 logits in registers.
// Same selection rule as k_router_topk (q36_ops.cuh:397-431): arg-max on the
// raw logits, ties to the lower expert id, k rounds with the winner masked.
//
// Bound by instruction issue once a few tokens share an SM (two dependent warp reductions and a scan of the lane's eight
// values per round).  The k-th largest of the 32 lane maxima is a lower bound of the k-th largest logit, and only a
// dozen logits reach it: those are compacted to one per lane, in expert order, and the rounds run on one value per lane.
// (Rounds over all eight values per lane: see launch_front for the figures.)
typedef unsigned long long RouteSlots[32];      // shared memory of a warp: its candidates, key << 32 | expert id

// order-preserving integer key of a float (-0 -> +0: equal floats, equal keys) and back
__device__ __forceinline__ uint32_t key_of(float v) {
    const uint32_t b = __float_as_uint(v + 0.f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

template <int PER_LANE>
__device__ __forceinline__ void route_row(const float *__restrict__ l, int k, int *idx, float *wt,
                                          float scale, int renorm, int lane, RouteSlots &slots) {
    constexpr uint32_t ALL = 0xffffffffu;
    const float NONE = -1e30f;           // logits at or below this are never chosen (and -1e30 stands for "no more experts")
    const uint32_t none = key_of(NONE);
    float v[PER_LANE];
    uint32_t key[PER_LANE];
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) v[j] = l[lane + j * 32];
    uint32_t top = none;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) {
        key[j] = v[j] > NONE ? key_of(v[j]) : none;      // (a NaN is not chosen either)
        top = max(top, key[j]);
    }
    const uint32_t kfirst = __reduce_max_sync(ALL, top);
    const float m = value_of(kfirst);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) s += expf(v[j] - m);
    s = warp_sum(s);
    // the k-th largest lane maximum (several lanes with the same one count as many)
    uint32_t thr = kfirst;
    if (PER_LANE > 1) {
        uint32_t cur = top;
        for (int left = k; left > 0;) {
            thr = __reduce_max_sync(ALL, cur);
            const bool hit = cur == thr;
            left -= __popc(__ballot_sync(ALL, hit));
            if (hit) cur = 0;
        }
    } else {
        thr = 0;                         // one value per lane: everybody is a candidate
    }
    int base = 0;
#pragma unroll
    for (int j = 0; j < PER_LANE; j++) { // slot order = expert order
        const bool in = key[j] >= thr;
        const uint32_t mask = __ballot_sync(ALL, in);
        const int slot = base + __popc(mask & ((1u << lane) - 1u));
        if (in && slot < 32) slots[slot] = (unsigned long long)key[j] << 32 | (uint32_t)(lane + 32 * j);
        base += __popc(mask);
    }
    __syncwarp();
    uint32_t k_keep = 0;                 // lane r keeps the choice of round r
    int i_keep = 0;
    if (base <= 32) {
        const unsigned long long c = lane < base ? slots[lane] : 0ull;
        uint32_t cur = (uint32_t)(c >> 32);
        int src = 0;
        for (int r = 0; r < k; r++) {
            const uint32_t kmax = __reduce_max_sync(ALL, cur);
            const int who = __ffs(__ballot_sync(ALL, cur == kmax)) - 1;     // the lowest slot = the lowest expert id
            if (lane == r) src = who;
            if (lane == who) cur = 0;
        }
        k_keep = __shfl_sync(ALL, (uint32_t)(c >> 32), src);
        i_keep = (int)__shfl_sync(ALL, (uint32_t)c, src);
    } else {                             // (more than 32 logits tie at the bound: all values, round by round)
        for (int r = 0; r < k; r++) {
            uint32_t bk = 0;
            int bj = 0;
#pragma unroll
            for (int j = 0; j < PER_LANE; j++)
                if (key[j] > bk) { bk = key[j]; bj = j; }
            const uint32_t kmax = __reduce_max_sync(ALL, bk);
            const int wi = (int)__reduce_min_sync(ALL, bk == kmax ? (uint32_t)(lane + bj * 32) : ALL);
            if (lane == r) { k_keep = kmax; i_keep = wi; }
            if (lane == (wi & 31)) {
#pragma unroll
                for (int j = 0; j < PER_LANE; j++)
                    if (j == (wi >> 5)) key[j] = 0;
            }
        }
    }
    __syncwarp();                        // (the slots are read: the warp's next row may overwrite them)
    // the k weights at once, one lane each; their sum in round order
    const float w_keep = expf(value_of(k_keep) - m) / s;
    float wsum = 0.f;
    for (int r = 0; r < k; r++) wsum += __shfl_sync(ALL, w_keep, r);
    if (lane < k) {
        idx[lane] = k_keep > none ? i_keep : 0;
        wt[lane] = renorm ? (w_keep / wsum * scale) : (w_keep * scale);
    }
}
// the row function of a given expert count (32, 64, 128 or 256)
__device__ __forceinline__ void route_row_of(int n_expert, const float *__restrict__ l, int k, int *idx, float *wt, float scale,
                                             int renorm, int lane, RouteSlots &slots) {
    if (n_expert == 256) route_row<8>(l, k, idx, wt, scale, renorm, lane, slots);
    else if (n_expert == 128) route_row<4>(l, k, idx, wt, scale, renorm, lane, slots);
    else if (n_expert == 64) route_row<2>(l, k, idx, wt, scale, renorm, lane, slots);
    else route_row<1>(l, k, idx, wt, scale, renorm, lane, slots);
}

__global__ void k_router_topk(const float *__restrict__ logits, int n_expert, int k, int *idx,
                              float *wt, float scale, int renorm, int T, int row_stride) {
    Q36_GDS();
    __shared__ RouteSlots slots[8];
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= T) return;
    const float *l = logits + (size_t)warp * row_stride;
    route_row_of(n_expert, l, k, idx + (size_t)warp * k, wt + (size_t)warp * k, scale, renorm, lane, slots[threadIdx.x >> 5]);
}

// -------------------------------------------------------------- dispatch
// Stable counting sort of entry ids by expert in two or three launches.  Entries are cut into chunks of at most DISPATCH_CHUNK;
// inside a chunk warp w owns entries [32w, 32w+32).
//   k_dispatch_count      : per (expert, chunk) counts and each entry's rank among the chunk's earlier entries of the
//                           same expert; with ROUTE the chunk's tokens are routed by the same block first
//   k_dispatch_scan_place : one cluster: per expert exclusive scan over its chunks (a warp per expert), scan over the
//                           experts, then elist / pos of every entry; its first CTA writes the tensor-core work plan
// A third one places the entries when they are many (k_dispatch_place), or the row quantiser does (k_quant_rows).
// The order inside a bucket is ascending entry id, one of the orders the
// engine's atomic k_moe_dispatch (q36_engine.cu:3387-3392) can produce.
// Bound by latency at every size that matters (12 B per entry).  One block that scanned, and separate router and place
// launches around it, took 46 us at 4096 tokens and 96 at 32,768; see launch_front for the figures now.
constexpr int DISPATCH_CHUNK = 512;
constexpr int DISPATCH_MAX_E = 512;
constexpr int DISPATCH_CLUSTER = 8;

// entries per chunk when the router runs in the same block: one token per warp of the block (4096 tokens are then 128
// blocks; two tokens per warp left half of the chip idle), as far as the chunk holds them
static inline int route_chunk(int k) { return min(32, DISPATCH_CHUNK / k) * k; }

template <bool ROUTE>
__global__ void __launch_bounds__(1024)
k_dispatch_count(const float *__restrict__ logits, int row_stride, int k, float scale, int T, int *__restrict__ idx,
                 float *__restrict__ wt, const int *__restrict__ eid, int n, int per_chunk, int n_expert, int se0, int se1,
                 int *__restrict__ cnt_ec, int n_chunk, unsigned short *__restrict__ lrank) {
    // synchronise first, then let the next grid start: see k_quant_rows
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    __shared__ unsigned short cnt[DISPATCH_CHUNK / 32][DISPATCH_MAX_E];
    __shared__ int s_idx[DISPATCH_CHUNK];
    __shared__ float s_wt[DISPATCH_CHUNK];
    __shared__ RouteSlots slots[ROUTE ? 32 : 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, i0 = blockIdx.x * per_chunk;
    const int ne = min(per_chunk, n - i0), i = i0 + tid;          // entries of this chunk, one thread each (the upper half idles)
    for (int x = tid; x < (DISPATCH_CHUNK / 32) * DISPATCH_MAX_E / 2; x += blockDim.x) reinterpret_cast<uint32_t *>(&cnt[0][0])[x] = 0;
    if (ROUTE) {
        const int t0 = i0 / k, nt = ne / k;
        for (int t = warp; t < nt; t += 32)
            route_row_of(n_expert, logits + (size_t)(t0 + t) * row_stride, k, s_idx + t * k, s_wt + t * k, scale, 1, lane, slots[warp]);
    }
    __syncthreads();
    int e = -1;
    if (tid < ne) {
        e = ROUTE ? s_idx[tid] : eid[i];
        if (ROUTE) { idx[i] = e; wt[i] = s_wt[tid]; }
        if (e < 0 || e < se0 || e >= se1 || e >= n_expert) e = -1;
    }
    int r_in_warp = 0;
    if (warp < DISPATCH_CHUNK / 32) {
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        r_in_warp = __popc(peers & ((1u << lane) - 1u));
        if (e >= 0 && r_in_warp == 0) cnt[warp][e] = (unsigned short)__popc(peers);
    }
    __syncthreads();
    for (int x = tid; x < n_expert; x += blockDim.x) {
        int run = 0;
#pragma unroll
        for (int w = 0; w < DISPATCH_CHUNK / 32; w++) {
            const int c = cnt[w][x];
            cnt[w][x] = (unsigned short)run;
            run += c;
        }
        cnt_ec[(size_t)x * n_chunk + blockIdx.x] = run;
    }
    __syncthreads();
    if (tid < ne) lrank[i] = (e >= 0) ? (unsigned short)(cnt[warp][e] + r_in_warp) : (unsigned short)0xffff;
}

// exclusive block scan of one value per thread (1024 threads); s_w: 32 values of shared memory.  All threads call.
template <typename V>
__device__ __forceinline__ V block_scan_excl(V val, V *s_w, V *total) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    V incl = val;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const V u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    V before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < 32; w++) { const V u = s_w[w]; if (w < warp) before += u; all += u; }
    *total = all;
    return before + incl - val;
}

__global__ void __launch_bounds__(1024)
k_dispatch_scan_place(const int *__restrict__ eid, int n, int per_chunk, int n_expert, int *cnt_ec, int n_chunk,
                      const unsigned short *__restrict__ lrank, int *__restrict__ ecount, int *__restrict__ eoffs,
                      int *__restrict__ elist, int *__restrict__ pos, int *__restrict__ soffs, int s0, int s1, TcPlan *plan, int se0,
                      int se1, int mt_gu, int mt_dn, int plan_tile_rows) {
    // elist == nullptr: a launch behind this one places the entries (k_quant_rows or k_dispatch_place)
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_arrive();                 // every CTA has started before anyone writes into its shared memory
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    __shared__ int s_tot[DISPATCH_MAX_E], s_eoffs[DISPATCH_MAX_E + 1], s_w[32];
    __shared__ int scratch[4 * (DISPATCH_MAX_GROUPS + 1)];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster.block_rank();
    cluster.barrier_wait();
    // a warp per expert: exclusive scan over the chunks, in place
    const int per = (n_expert + DISPATCH_CLUSTER - 1) / DISPATCH_CLUSTER;
    for (int x = rank * per + warp; x < min(n_expert, (rank + 1) * per); x += 32) {
        int *row = cnt_ec + (size_t)x * n_chunk;
        int run = 0;
        for (int c0 = 0; c0 < n_chunk; c0 += 128) {               // four loads in flight per lane
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = c0 + 32 * j + lane < n_chunk ? row[c0 + 32 * j + lane] : 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                int incl = v[j];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
                if (c0 + 32 * j + lane < n_chunk) row[c0 + 32 * j + lane] = run + incl - v[j];
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        if (lane < DISPATCH_CLUSTER) *cluster.map_shared_rank(&s_tot[x], lane) = run;
    }
    cluster.sync();   // the totals of every expert are in every CTA; the scanned rows are visible in the cluster
    int all;
    const int tot = tid < n_expert ? s_tot[tid] : 0;
    const int row0 = block_scan_excl(tot, s_w, &all);
    if (tid < n_expert) s_eoffs[tid] = row0;
    if (tid == 0) s_eoffs[n_expert] = all;
    __syncthreads();
    if (rank == 0) {   // the tables, and the work plan, which depends on nothing else
        if (tid < n_expert) ecount[tid] = tot;
        if (tid <= n_expert) eoffs[tid] = s_eoffs[tid];
        if (tid == 0 && soffs) { soffs[0] = s0; soffs[1] = s1; }
        if (plan) tc_plan_block(s_eoffs + se0, se1 - se0, s1 > s0, s0, s1, plan, mt_gu, mt_dn, scratch, true, plan_tile_rows);
        return;        // (its shared memory is written by the others before the barrier only)
    }
    if (!elist) return;
    constexpr int U = 4, STEP = (DISPATCH_CLUSTER - 1) * 1024;
    for (int i0 = (rank - 1) * 1024 + tid; i0 < n; i0 += U * STEP) {
        int e[U], r[U], b[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * STEP;
            r[u] = i < n ? (int)lrank[i] : 0xffff;
            e[u] = i < n ? eid[i] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            b[u] = r[u] != 0xffff ? __ldcg(cnt_ec + (size_t)e[u] * n_chunk + (i0 + u * STEP) / per_chunk) : 0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * STEP;
            if (i >= n) continue;
            if (r[u] == 0xffff) { pos[i] = -1; continue; }
            const int p = s_eoffs[e[u]] + b[u] + r[u];
            elist[p] = i;
            pos[i] = p;
        }
    }
}

// elist / pos of many entries, by the whole chip instead of the seven SMs above (see dispatch_launches)
__global__ void __launch_bounds__(256)
k_dispatch_place(const int *__restrict__ eid, int n, int per_chunk, const int *__restrict__ cnt_ec, int n_chunk,
                 const unsigned short *__restrict__ lrank, const int *__restrict__ eoffs, int *__restrict__ elist, int *__restrict__ pos) {
    Q36_GDS();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int r = lrank[i], e = eid[i];
    if (r == 0xffff) { pos[i] = -1; return; }
    const int p = eoffs[e] + cnt_ec[(size_t)e * n_chunk + i / per_chunk] + r;
    elist[p] = i;
    pos[i] = p;
}

// ------------------------------------------------------------- quantiser
// One warp per (row, 32-block), one lane per element, as k_quant_e4m3 does
// (q36_engine.cu:2412-2428).  SCATTER = false: logical order into Xq[T][K].
// SCATTER = true: hw order into every row of the sorted space the token feeds.
// one (row, 32-block) task of a warp: lane = element
__device__ __forceinline__ float quant_load(const void *__restrict__ X, bool bf16, int t, int b, int K, int lane) {
    const size_t off = (size_t)t * K + (size_t)b * Q36_QK + lane;
    return bf16 ? __bfloat162float(((const __nv_bfloat16 *)X)[off]) : ((const float *)X)[off];
}
template <bool SCATTER>
__device__ __forceinline__ void quant_task(float v, uint8_t *__restrict__ Xq, uint8_t *__restrict__ Xs, int t, int b,
                                           int K, const int *pos, int k, int shared_row0, int lane) {
    const int nb = K / Q36_QK;
    const size_t off = (size_t)t * K + (size_t)b * Q36_QK + lane;
    const float a = warp_max(fabsf(v));
    const int e2 = e2_of_amax(a);
    const uint8_t q = f32_to_e4m3(v * inv_scale_of_e2(e2));
    if (!SCATTER) {
        Xq[off] = q;
        if (lane == 0) Xs[(size_t)t * nb + b] = (uint8_t)(127 + e2);
    } else {
        // gather the block's 32 codes in hw order: lane p receives the code of
        // the element that lives at position p
        const int src = (lane & 1) ? (16 + (lane >> 1)) : (lane >> 1);
        const uint32_t qp = __shfl_sync(0xffffffffu, (uint32_t)q, src);
        // pack 4 positions per lane (lanes 0..7 hold the 32 bytes)
        uint32_t w = qp;
        w |= __shfl_down_sync(0xffffffffu, qp, 1) << 8;
        w |= __shfl_down_sync(0xffffffffu, qp, 2) << 16;
        w |= __shfl_down_sync(0xffffffffu, qp, 3) << 24;
        const uint32_t word = __shfl_sync(0xffffffffu, w, (lane & 7) * 4);
        // lane l writes word (l & 7) of destination (l >> 3), 4 destinations a pass
        const int n_dst = k + (shared_row0 >= 0 ? 1 : 0);
        for (int d0 = 0; d0 < n_dst; d0 += 4) {
            const int d = d0 + (lane >> 3);
            if (d < n_dst) {
                const int row = (d < k) ? pos[(size_t)t * k + d] : (shared_row0 + t);
                if (row >= 0) {
                    ((uint32_t *)(Xq + (size_t)row * K + (size_t)b * Q36_QK))[lane & 7] = word;
                    if ((lane & 7) == 0) Xs[(size_t)row * nb + b] = (uint8_t)(127 + e2);
                }
            }
        }
    }
}


// ------------------------------------------- quantiser, one lane per 32-block
// The same arithmetic as quant_task, laid out for rows that are scattered to several destinations: a lane
// owns a whole 32-block (64 B of bf16 or 128 B of f32 in, its amax needs no shuffle), a warp 32 consecutive
// blocks of one token row, so every destination row receives 1 KB of codes and 32 scale bytes per warp in
// full sectors.  (One warp per block writes 32 B and one scale byte per destination: at 4096 tokens the
// single-byte stores alone are 2.4 M partial-sector writes.)
struct QBlock { uint4 lo, hi; int e2; };   // the block's 32 codes in hw order (element j at 2j, j+16 at 2j+1)

template <bool BF16>
__device__ __forceinline__ QBlock quant_block_lane(const void *__restrict__ X, size_t off) {
    float v[32];
    if (BF16) {
        const uint4 *p = reinterpret_cast<const uint4 *>((const __nv_bfloat16 *)X + off);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 u = p[i];
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                v[8 * i + 2 * j] = __uint_as_float(w[j] << 16);
                v[8 * i + 2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
            }
        }
    } else {
        const float4 *p = reinterpret_cast<const float4 *>((const float *)X + off);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float4 u = p[i];
            v[4 * i] = u.x; v[4 * i + 1] = u.y; v[4 * i + 2] = u.z; v[4 * i + 3] = u.w;
        }
    }
    float a = 0.f;
#pragma unroll
    for (int i = 0; i < 32; i++) a = fmaxf(a, fabsf(v[i]));
    QBlock r;
    r.e2 = e2_of_amax(a);
    const float inv = inv_scale_of_e2(r.e2);
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {   // bytes 4i..4i+3 = elements 2i, 2i+16, 2i+1, 2i+17
        w[i] = (uint32_t)f32_to_e4m3(v[2 * i] * inv) | ((uint32_t)f32_to_e4m3(v[2 * i + 16] * inv) << 8) |
               ((uint32_t)f32_to_e4m3(v[2 * i + 1] * inv) << 16) | ((uint32_t)f32_to_e4m3(v[2 * i + 17] * inv) << 24);
    }
    r.lo = make_uint4(w[0], w[1], w[2], w[3]);
    r.hi = make_uint4(w[4], w[5], w[6], w[7]);
    return r;
}
// Lane pairs swap halves so that each of the two store instructions of a warp covers 512 contiguous bytes (whole
// sectors); a lane storing its own two halves would leave every sector half-written twice.  All 32 lanes call.
struct QStore { uint4 first, second; };   // what this lane stores at byte 64 * (lane / 2) + 16 * (lane & 1) and + 32
__device__ __forceinline__ QStore quant_block_pair(const QBlock &q, int lane) {
    const bool odd = lane & 1;
    // even lane keeps lo, gives hi; odd lane keeps hi, gives lo
    const uint4 give = odd ? q.lo : q.hi;
    uint4 got;
    got.x = __shfl_xor_sync(0xffffffffu, give.x, 1); got.y = __shfl_xor_sync(0xffffffffu, give.y, 1);
    got.z = __shfl_xor_sync(0xffffffffu, give.z, 1); got.w = __shfl_xor_sync(0xffffffffu, give.w, 1);
    QStore r;
    r.first = odd ? got : q.lo;     // block 2i:   [lo_2i | hi_2i]     <- lanes 2i, 2i+1
    r.second = odd ? q.hi : got;    // block 2i+1: [lo_2i+1 | hi_2i+1] <- lanes 2i, 2i+1
    return r;
}
// blk0 = first block of the warp's run of 32
__device__ __forceinline__ void quant_block_put(const QStore &qs, int e2, uint8_t *__restrict__ Xq, uint8_t *__restrict__ Xs,
                                                int row, int blk0, int lane, int K) {
    uint8_t *base = Xq + (size_t)row * K + (size_t)blk0 * Q36_QK + 64 * (lane >> 1) + 16 * (lane & 1);
    *reinterpret_cast<uint4 *>(base) = qs.first;
    *reinterpret_cast<uint4 *>(base + 32) = qs.second;
    Xs[(size_t)row * (K / Q36_QK) + blk0 + lane] = (uint8_t)(127 + e2);
}

// warp = (token, run of 32 blocks); K must be a multiple of 1024.
// The rows' positions are loaded ahead of the token row unless they are not there yet: 4096 tokens 14.3 us, 15.1 with the loads
// behind the quantising or with one load per lane and shuffles.
// early: the token row is read and quantised BEFORE the grid dependency resolves, only its row positions after.  Only
// for a launch whose predecessor in the stream lets its successor start after it has itself seen everything before it
// complete (the dispatch kernels above do): the rows were then written by something that is over.
// PLACE: the kernel also turns every entry's rank into its row (what k_dispatch_scan_place does for callers without this
// launch): the seven SMs of that cluster took 60 us for the 262,144 entries of 32,768 tokens.
struct PlaceArgs { const int *idx, *cnt_ec, *eoffs; const unsigned short *lrank; int n_chunk, per_chunk; };
template <bool BF16, bool PLACE>
__global__ void __launch_bounds__(256)
k_quant_rows(const void *__restrict__ X, uint8_t *__restrict__ Xq, uint8_t *__restrict__ Xs, int T, int K,
             int *__restrict__ pos, int k, int shared_row0, int early, const PlaceArgs pl) {
    cudaTriggerProgrammaticLaunchCompletion();
    if (!early) cudaGridDependencySynchronize();
    const int runs = K / (32 * Q36_QK);
    const long gwarp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const bool mine = gwarp < (long)T * runs;
    const int t = mine ? (int)(gwarp / runs) : 0, run = mine ? (int)(gwarp % runs) : 0, blk = run * 32 + lane;
    int rows[9];
    auto entry_rows = [&] {
#pragma unroll
        for (int d = 0; d < 8; d++) rows[d] = d < k ? pos[(size_t)t * k + d] : -1;
    };
    if (!PLACE && !early) entry_rows();              // (issued before the row is read)
    rows[8] = shared_row0 >= 0 ? shared_row0 + t : -1;
    const QBlock q = quant_block_lane<BF16>(X, (size_t)t * K + (size_t)blk * Q36_QK);
    const QStore qs = quant_block_pair(q, lane);
    if (early) cudaGridDependencySynchronize();
    if (!mine) return;
    if (PLACE) {                                     // lane d: the row of the token's entry d
        int p = -1;
        if (lane < k) {
            const int i = t * k + lane, r = pl.lrank[i], e = pl.idx[i];
            if (r != 0xffff) p = pl.eoffs[e] + pl.cnt_ec[(size_t)e * pl.n_chunk + i / pl.per_chunk] + r;
            if (run == 0) pos[i] = p;
        }
#pragma unroll
        for (int d = 0; d < 8; d++) rows[d] = __shfl_sync(0xffffffffu, p, d);
    } else if (early) {
        entry_rows();
    }
#pragma unroll
    for (int d = 0; d < 9; d++)
        if (rows[d] >= 0) quant_block_put(qs, q.e2, Xq, Xs, rows[d], blk - lane, lane, K);
}

template <bool BF16, bool SCATTER>
__global__ void k_quant_e4m3(const void *__restrict__ X, uint8_t *__restrict__ Xq,
                             uint8_t *__restrict__ Xs, int T, int K, const int *__restrict__ pos,
                             int k, int shared_row0) {
    Q36_GDS();
    const int nb = K / Q36_QK;
    const long gwarp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gwarp >= (long)T * nb) return;
    const int t = (int)(gwarp / nb), b = (int)(gwarp % nb);
    quant_task<SCATTER>(quant_load(X, BF16, t, b, K, lane), Xq, Xs, t, b, K, pos, k, shared_row0, lane);
}

// ---------------------------------------------------- one-block dispatch of received slots
constexpr int FRONT_MAX_ENTRIES = 1024;

// Block-wide stable bucketing of up to FRONT_MAX_ENTRIES entries by expert (thread i owns entry i, e = its expert
// id or anything outside [se0, se1) for "not resident"), then the tensor-core work plan.  Shared arrays come from
// the caller.  All threads of the block call; ends with every output written (no trailing barrier).
struct SortSmem {
    unsigned short cnt[FRONT_MAX_ENTRIES / 32][DISPATCH_MAX_E];   // 32 KB: per (entry warp, expert) count, then base
    int s_eoffs[DISPATCH_MAX_E + 1];
    int scratch[4 * (DISPATCH_MAX_GROUPS + 1)];
};
__device__ __forceinline__ void sort_entries_block(SortSmem &sm, int e, int n, int n_expert, int se0, int se1,
                                                   int *__restrict__ ecount, int *__restrict__ eoffs, int *__restrict__ elist,
                                                   int *__restrict__ pos, int *__restrict__ soffs, int s0, int s1, TcPlan *plan,
                                                   int mt_gu, int mt_dn, int plan_tile_rows) {
    // precondition: sm.cnt rows [0, (n + 31) / 32) are zero and a barrier separates that from this call
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int used_warps = (n + 31) / 32;          // only the warps that own entries contribute counts
    if (tid >= n || e < 0 || e < se0 || e >= se1 || e >= n_expert) e = -1;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int r_in_warp = __popc(peers & ((1u << lane) - 1u));
    if (e >= 0 && r_in_warp == 0) sm.cnt[warp][e] = (unsigned short)__popc(peers);
    __syncthreads();
    for (int x = tid; x < n_expert; x += blockDim.x) {
        int run = 0;
        for (int w = 0; w < used_warps; w++) {
            const int c = sm.cnt[w][x];
            sm.cnt[w][x] = (unsigned short)run;
            run += c;
        }
        ecount[x] = run;
        sm.s_eoffs[x] = run;
    }
    __syncthreads();
    if (warp == 0) {   // exclusive scan of the expert totals: lane owns a contiguous run
        const int per = (n_expert + 31) / 32;
        int sum = 0;
        for (int j = 0; j < per; j++) { const int x = lane * per + j; if (x < n_expert) sum += sm.s_eoffs[x]; }
        int incl = sum;
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        int run = incl - sum;
        for (int j = 0; j < per; j++) {
            const int x = lane * per + j;
            if (x < n_expert) { const int c = sm.s_eoffs[x]; sm.s_eoffs[x] = run; run += c; }
        }
        if (lane == 31) sm.s_eoffs[n_expert] = run;
    }
    __syncthreads();
    for (int x = tid; x <= n_expert; x += blockDim.x) eoffs[x] = sm.s_eoffs[x];
    if (tid == 0 && soffs) { soffs[0] = s0; soffs[1] = s1; }
    if (tid < n) {
        if (e >= 0) {
            const int p = sm.s_eoffs[e] + sm.cnt[warp][e] + r_in_warp;
            elist[p] = tid;
            pos[tid] = p;
        } else pos[tid] = -1;
    }
    // groups here hold at most a few token tiles: ranking by size would buy nothing
    if (plan) tc_plan_block(sm.s_eoffs + se0, se1 - se0, s1 > s0, s0, s1, plan, mt_gu, mt_dn, sm.scratch, false, plan_tile_rows);
}

// ------------------------------------------------- front end of up to 512 tokens of 8 entries, 768 of fewer: one cluster
// Router -> stable dispatch -> work plan in ONE launch.  CTA r of the cluster routes the tokens [r tpc, (r + 1) tpc) and
// counts its entries per expert; the counts (2 B each) go to every CTA's shared memory, so that each of them knows every
// expert's offset after one cluster barrier and places its own entries.
// Bound by latency: logits (one read), eight dependent selection rounds, three block barriers and a cluster barrier.
// One block that did all of it took 21 us at 33 tokens and 23 at 96 (the k_front_small this replaces), five launches
// 28 us at 300; see launch_front for the figures now.
constexpr int FM_CLUSTER = 8;
constexpr int FM_ENTRIES = 512;                       // per CTA
constexpr int FM_MAX_E = 256;                         // what the router takes

__global__ void __launch_bounds__(1024)
k_front_mid(const float *__restrict__ logits, int n_expert, int k, float scale, int T, int row_stride, int se0, int se1,
            int *__restrict__ idx, float *__restrict__ wt, int *__restrict__ ecount, int *__restrict__ eoffs,
            int *__restrict__ elist, int *__restrict__ pos, int *__restrict__ soffs, int s0, int s1, TcPlan *plan, int mt_gu,
            int mt_dn, int plan_tile_rows) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_arrive();                 // every CTA has started before anyone writes into its shared memory
    // synchronise first, then let the next grid start: see k_quant_rows
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    __shared__ unsigned short cnt[FM_ENTRIES / 32][FM_MAX_E];    // per (entry warp, expert): count, then base
    __shared__ unsigned short s_cta[FM_CLUSTER][FM_MAX_E];       // entries of every CTA per expert
    __shared__ int s_idx[FM_ENTRIES], s_base[FM_MAX_E];
    __shared__ float s_wt[FM_ENTRIES];
    __shared__ RouteSlots slots[32];
    __shared__ unsigned long long s_w[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster.block_rank();
    const int tpc = (T + FM_CLUSTER - 1) / FM_CLUSTER, t0 = min(T, rank * tpc), nt = min(tpc, T - t0), ne = nt * k;
    const int used_warps = (ne + 31) / 32;
    for (int x = tid; x < used_warps * FM_MAX_E / 2; x += 1024) reinterpret_cast<uint32_t *>(&cnt[0][0])[x] = 0;
    for (int t = warp; t < nt; t += 32)
        route_row_of(n_expert, logits + (size_t)(t0 + t) * row_stride, k, s_idx + t * k, s_wt + t * k, scale, 1, lane, slots[warp]);
    __syncthreads();
    int e = -1;
    const int i = t0 * k + tid;
    if (tid < ne) {
        e = s_idx[tid];
        idx[i] = e;
        wt[i] = s_wt[tid];
        if (e < se0 || e >= se1 || e >= n_expert) e = -1;
    }
    int r_in_warp = 0;
    if (warp < used_warps) {
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        r_in_warp = __popc(peers & ((1u << lane) - 1u));
        if (e >= 0 && r_in_warp == 0) cnt[warp][e] = (unsigned short)__popc(peers);
    }
    __syncthreads();
    cluster.barrier_wait();
    if (tid < n_expert) {
        int run = 0;
        for (int w = 0; w < used_warps; w++) {
            const int c = cnt[w][tid];
            cnt[w][tid] = (unsigned short)run;
            run += c;
        }
#pragma unroll
        for (int r = 0; r < FM_CLUSTER; r++) *cluster.map_shared_rank(&s_cta[rank][tid], r) = (unsigned short)run;
    }
    cluster.sync();
    // rows, gate/up token tiles and down token tiles before every expert, in one scan
    const int tr_gu = plan_tile_rows ? plan_tile_rows : TC_N_GATEUP, tr_dn = plan_tile_rows ? plan_tile_rows : TC_N_DOWN;
    int tot = 0, mine = 0;
    if (tid < n_expert) {
#pragma unroll
        for (int r = 0; r < FM_CLUSTER; r++) {
            const int c = s_cta[r][tid];
            if (r < rank) mine += c;
            tot += c;
        }
    }
    typedef unsigned long long u64;
    u64 all;
    const u64 excl = block_scan_excl<u64>((u64)tot | (u64)((tot + tr_gu - 1) / tr_gu) << 20 | (u64)((tot + tr_dn - 1) / tr_dn) << 40, s_w, &all);
    const int row0 = (int)(excl & 0xfffff);
    if (tid < n_expert) s_base[tid] = row0 + mine;
    __syncthreads();
    if (tid < ne) {
        int p = -1;
        if (e >= 0) {
            p = s_base[e] + cnt[warp][e] + r_in_warp;
            elist[p] = i;
        }
        pos[i] = p;
    }
    if (rank != 0) return;
    if (tid < n_expert) {
        ecount[tid] = tot;
        eoffs[tid] = row0;
        if (plan && tid >= se0 && tid < se1) {
            // (groups in expert order: ranking them by size takes a scan of its own, which did not pay at these sizes, skewed routing
            // included: see front_mid_takes, the other side of which ranks them)
            const int g = tid - se0;
            plan->row0[g] = row0; plan->cnt[g] = tot; plan->done[g] = 0; plan->order[g] = g;
            plan->base[0][g] = (int)(excl >> 20 & 0xfffff) * mt_gu; plan->base[1][g] = (int)(excl >> 40) * mt_dn;
        }
    }
    if (tid == 0) {
        eoffs[n_expert] = (int)(all & 0xfffff);
        if (soffs) { soffs[0] = s0; soffs[1] = s1; }
        if (plan) {
            int G = se1 - se0, ta = (int)(all >> 20 & 0xfffff) * mt_gu, tb = (int)(all >> 40) * mt_dn;
            if (s1 > s0) {                       // the shared expert's rows are one more group
                plan->row0[G] = s0; plan->cnt[G] = s1 - s0; plan->done[G] = 0; plan->order[G] = G;
                plan->base[0][G] = ta; plan->base[1][G] = tb;
                ta += (s1 - s0 + tr_gu - 1) / tr_gu * mt_gu;
                tb += (s1 - s0 + tr_dn - 1) / tr_dn * mt_dn;
                G++;
            }
            plan->base[0][G] = ta; plan->base[1][G] = tb;
            plan->n_tiles[0] = ta; plan->n_tiles[1] = tb; plan->n_groups = G; plan->gu_done = 0; plan->tile_rows = plan_tile_rows;
        }
    }
}

// ---------------------------------------- expert-parallel: received slots -> local plan
// The slots a rank received sit in its exchange window as [world sources][cap slots][row_bytes]; source s filled
// the first count_s of its slots and then published (count_s, epoch) in hdr[s].  One block waits (bounded) for
// every source's header of this call, then buckets the valid slots by local expert and writes the work plan:
// the dispatch step of the layer applied to what arrived.  world * cap <= FRONT_MAX_ENTRIES.
__device__ __forceinline__ unsigned long long ld_acquire_sys_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// hdr word = count | epoch << 32.  Returns the count, or -1 after `limit` polls (status receives `where`).
__device__ __forceinline__ int ep_wait_hdr(const unsigned long long *hdr, unsigned epoch, unsigned limit, int *status, int where) {
    for (unsigned i = 0; i < limit; i++) {
        const unsigned long long v = ld_acquire_sys_u64(hdr);
        if ((unsigned)(v >> 32) == epoch) return (int)(unsigned)v;
        if (i > 64) __nanosleep(i < 4096 ? 32 : 256);
    }
    atomicCAS(status, 0, where);
    return -1;
}

__global__ void __launch_bounds__(1024)
k_ep_recv_plan(const uint8_t *__restrict__ win, uint64_t off_hdr0, uint64_t off_hdr1, uint64_t off_rows0, uint64_t off_rows1,
               const int *__restrict__ ctr, int world, int cap, int row_bytes, int eid_off, unsigned limit, int *status,
               int n_expert, int se0, int se1, int *__restrict__ ecount, int *__restrict__ eoffs, int *__restrict__ elist,
               int *__restrict__ pos, int *__restrict__ soffs, int s0, int s1, TcPlan *plan, int mt_gu, int mt_dn,
               int plan_tile_rows, int *__restrict__ counts_out) {
    Q36_GDS();
    Q36_TR_BEGIN(status, 2)
    __shared__ SortSmem sm;
    __shared__ int s_cnt[64];
    const int tid = threadIdx.x;
    const int n = world * cap;
    const unsigned epoch = (unsigned)ctr[1] + 1u;   // (this rank's phase-1 call counter)
    const bool odd = epoch & 1u;
    const int used_warps = (n + 31) / 32;
    for (int i = tid; i < used_warps * DISPATCH_MAX_E; i += blockDim.x) (&sm.cnt[0][0])[i] = 0;
    if (tid < world) {
        const unsigned long long *hdr = reinterpret_cast<const unsigned long long *>(win + (odd ? off_hdr1 : off_hdr0)) + tid;
        const int c = ep_wait_hdr(hdr, epoch, limit, status, 0xB00 + tid);
        s_cnt[tid] = max(0, min(c, cap));
        counts_out[tid] = s_cnt[tid];
    }
    __syncthreads();
    int e = -1;
    if (tid < n && (tid % cap) < s_cnt[tid / cap])
        e = *reinterpret_cast<const int *>(win + (odd ? off_rows1 : off_rows0) + (size_t)tid * row_bytes + eid_off);
    sort_entries_block(sm, e, n, n_expert, se0, se1, ecount, eoffs, elist, pos, soffs, s0, s1, plan, mt_gu, mt_dn, plan_tile_rows);
    Q36_TR_END(status, 2)
}

int launch_ep_recv_plan(const void *win, uint64_t off_hdr0, uint64_t off_hdr1, uint64_t off_rows0, uint64_t off_rows1, const int *ctr,
                        int world, int cap, int row_bytes, int eid_off, unsigned limit, int *status, int n_expert, int se0, int se1,
                        int *ecount, int *eoffs, int *elist, int *pos, int *soffs, int s0, int s1, void *plan, int D, int FF,
                        int plan_tile_rows, int *counts_out, cudaStream_t st) {
    if (world * cap > FRONT_MAX_ENTRIES || world > 64 || n_expert > DISPATCH_MAX_E) return Q36_MOE_EINVAL;
    launch_k(k_ep_recv_plan, dim3(1), dim3(1024), 0, st, (const uint8_t *)win, off_hdr0, off_hdr1, off_rows0, off_rows1, ctr, world, cap,
             row_bytes, eid_off, limit, status, n_expert, se0, se1, ecount, eoffs, elist, pos, soffs, s0, s1, (TcPlan *)plan,
             FF / TC_M, D / TC_M, plan_tile_rows, counts_out);
    return check_launch();
}

// Tokens bound it as well as entries: its eight SMs route them.  us per layer (256 experts, uniform / skewed routing) through this
// launch and through the two of launch_route_dispatch: top-4 513 tokens 106.8 / 76.2 and 108.9 / 78.5, 700 tokens 120.5 / 96.4 and
// 121.5 / 97.8, 800 tokens 134.6 / 108.3 and 135.1 / 107.2, 1024 tokens 151.9 / 90.6 and 149.5 / 90.1; top-1 800 tokens 106.9 / 55.2
// and 106.7 / 57.0, 1500 tokens 130.6 / 87.9 and 125.7 / 83.8, 4096 tokens 195.5 / 132.4 and 173.1 / 111.4.
constexpr int FM_MAX_T = 768;
bool front_mid_takes(int T, int k, int n_expert) {
    return T <= FM_MAX_T && k >= 1 && k <= 8 && n_expert <= FM_MAX_E && (T + FM_CLUSTER - 1) / FM_CLUSTER * k <= FM_ENTRIES;
}
int launch_front_mid(const float *logits, int n_expert, int k, float scale, int T, int row_stride, int se0, int se1,
                     int *idx, float *wt, int *ecount, int *eoffs, int *elist, int *pos, int *soffs, int s0, int s1,
                     void *plan, int D, int FF, int plan_tile_rows, cudaStream_t st) {
    if (!front_mid_takes(T, k, n_expert)) return Q36_MOE_EINVAL;
    launch_k_cluster(k_front_mid, dim3(1, 1, FM_CLUSTER), dim3(1024), FM_CLUSTER, st, logits, n_expert, k, scale, T, row_stride, se0, se1,
                     idx, wt, ecount, eoffs, elist, pos, soffs, s0, s1, (TcPlan *)plan, FF / TC_M, D / TC_M, plan_tile_rows);
    return check_launch();
}


// ----------------------------------------------- decode front end: one cluster
// At most 16 tokens (T * k <= 128 entries), all experts resident.  One thread-block cluster, one launch:
//   CTA 0        router -> stable dispatch -> work plan of the fused tensor-core kernel
//   CTAs 1..7    quantise the token rows (needs no routing result), wait at the cluster barrier for CTA 0's
//                row positions, then write every block to the k + 1 rows it feeds.
// Same results as k_front_mid + k_quant_rows: the same route_row, the same ascending-entry order inside an expert's
// bucket, the same quantiser.  The plan is cut in the decode kernel's 16-row token tiles, whatever launch follows.
constexpr int FD_CLUSTER = 8;
constexpr int FD_THREADS = 1024;
constexpr int FD_MAX_ENTRIES = 128;
constexpr int FD_QWARPS = (FD_CLUSTER - 1) * (FD_THREADS / 32);   // one (token, run of 32 blocks) per quantising warp

__global__ void __launch_bounds__(FD_THREADS)
k_front_decode(const float *__restrict__ logits, int n_expert, int k, float scale, int T, int row_stride,
               int *__restrict__ idx, float *__restrict__ wt, int *__restrict__ ecount, int *__restrict__ eoffs,
               int *__restrict__ elist, int *__restrict__ pos, int *__restrict__ soffs, int s0, int s1, TcPlan *plan,
               int mt_gu, int mt_dn, int *status, const void *__restrict__ X, int x_is_bf16, uint8_t *__restrict__ Xq,
               uint8_t *__restrict__ Xs, int D, int shared_row0, int put_k, const EpSendArgs ep) {
    // put_k: k for the sorted row space of a single-GPU layer; 0 when only the token-order rows (shared_row0 + t)
    // are wanted, as in the expert-parallel step
    Q36_GDS();
    Q36_TR_BEGIN(status, 0)
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = T * k;
    __shared__ int s_pos[FD_MAX_ENTRIES];          // row of every entry; CTA 0 writes it into every CTA of the cluster
    // expert-parallel: where every entry's row goes, (destination rank << 20) | slot, or -1 (beyond the capacity)
    __shared__ int s_slot[FD_MAX_ENTRIES];
    const unsigned ep_epoch = ep.peers ? (unsigned)ep.ctl[0] + 1u : 0u;
    if (cluster.block_rank() != 0) {
        // ---- quantise now (warp = token x run of 32 blocks, lane = block), place after the barrier
        // (units are dealt across the CTAs first: one SM's store path would take microseconds for all rows)
        const int runs = D / (32 * Q36_QK);
        const int unit = ((int)cluster.block_rank() - 1) + (FD_CLUSTER - 1) * warp;
        const int t = unit / runs, blk0 = (unit % runs) * 32;
        const bool mine = unit < T * runs;
        QBlock q;
        QStore qs;
        if (mine) {
            q = x_is_bf16 ? quant_block_lane<true>(X, (size_t)t * D + (size_t)(blk0 + lane) * Q36_QK)
                          : quant_block_lane<false>(X, (size_t)t * D + (size_t)(blk0 + lane) * Q36_QK);
            qs = quant_block_pair(q, lane);
        }
        cluster.sync();
        if (mine) {
            for (int d = 0; d < put_k; d++) {
                const int row = s_pos[t * k + d];
                if (row >= 0) quant_block_put(qs, q.e2, Xq, Xs, row, blk0, lane, D);
            }
            if (shared_row0 >= 0) quant_block_put(qs, q.e2, Xq, Xs, shared_row0 + t, blk0, lane, D);
            if (ep.peers) {   // the same blocks straight into the windows of the ranks that own the token's experts
                const int row_bytes = D + D / Q36_QK + 16;
                for (int d = 0; d < k; d++) {
                    const int code = s_slot[t * k + d];
                    if (code < 0) continue;
                    const int r = code >> 20, j = code & 0xfffff;
                    uint8_t *rowbase = ep.peers[r] + ((ep_epoch & 1u) ? ep.rows1 : ep.rows0) +
                                       ((size_t)(ep.slot_major ? r : ep.me) * ep.cap + j) * row_bytes;
                    quant_block_put(qs, q.e2, rowbase, rowbase + D, 0, blk0, lane, D);
                }
            }
        }
        if (ep.peers) cluster.sync();   // every CTA's remote stores before CTA 0 publishes the headers
        return;
    }
    // ---- CTA 0: route, sort, plan
    __shared__ unsigned short cnt[FD_MAX_ENTRIES / 32][DISPATCH_MAX_E];   // per (entry warp, expert): count, then base
    __shared__ int s_idx[FD_MAX_ENTRIES];
    __shared__ float s_wt[FD_MAX_ENTRIES];
    __shared__ RouteSlots slots[16];                                      // one warp per token, at most 16
    __shared__ int s_eoffs[DISPATCH_MAX_E + 1];
    __shared__ int s_wsum[FD_THREADS / 32];
    const int used_warps = (n + 31) / 32;
    if (warp < T) {
        const float *l = logits + (size_t)warp * row_stride;
        route_row_of(n_expert, l, k, s_idx + warp * k, s_wt + warp * k, scale, 1, lane, slots[warp]);
    } else {
        for (int i = tid - 32 * T; i < used_warps * DISPATCH_MAX_E; i += FD_THREADS - 32 * T) (&cnt[0][0])[i] = 0;
    }
    __syncthreads();
    int e = -1;
    if (tid < n) {
        e = s_idx[tid];
        idx[tid] = e;
        wt[tid] = s_wt[tid];
        if (e < 0 || e >= n_expert) e = -1;
    }
    int r_in_warp = 0;
    if (warp < used_warps) {
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        r_in_warp = __popc(peers & ((1u << lane) - 1u));
        if (e >= 0 && r_in_warp == 0) cnt[warp][e] = (unsigned short)__popc(peers);
    }
    __syncthreads();
    // per expert: rows, and (one scan for both) rows before it | token tiles of 16 rows before it << 16 (16 tokens with several
    // entries of one expert each, as rows with fewer than k eligible logits have, are more than one tile)
    int tot = 0;
    if (tid < n_expert) {
        for (int w = 0; w < used_warps; w++) {
            const int c = cnt[w][tid];
            cnt[w][tid] = (unsigned short)tot;
            tot += c;
        }
    }
    const int val = tot | ((tot + 15) / 16 << 16);
    int incl = val;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; w++) before += s_wsum[w];
    const int excl = before + incl - val;
    if (tid < n_expert) {
        const int row0 = excl & 0xffff, ne = excl >> 16;
        s_eoffs[tid] = row0;
        ecount[tid] = tot;
        eoffs[tid] = row0;
        if (plan) {
            plan->row0[tid] = row0; plan->cnt[tid] = tot; plan->done[tid] = 0; plan->order[tid] = tid;
            plan->base[0][tid] = ne * mt_gu; plan->base[1][tid] = ne * mt_dn;
        }
        if (tid == n_expert - 1) {
            const int total = (excl + val) & 0xffff, ne_all = (excl + val) >> 16;
            eoffs[n_expert] = total;
            s_eoffs[n_expert] = total;
            if (soffs) { soffs[0] = s0; soffs[1] = s1; }
            if (plan) {
                const bool extra = s1 > s0;
                int G = n_expert;
                int ta = ne_all * mt_gu, tb = ne_all * mt_dn;
                if (extra) {   // the shared expert's rows are one more group: T <= 16 rows, one token tile
                    plan->row0[G] = s0; plan->cnt[G] = s1 - s0; plan->done[G] = 0; plan->order[G] = G;
                    plan->base[0][G] = ta; plan->base[1][G] = tb;
                    ta += mt_gu; tb += mt_dn;
                    G++;
                }
                plan->base[0][G] = ta; plan->base[1][G] = tb;
                plan->n_tiles[0] = ta; plan->n_tiles[1] = tb; plan->n_groups = G; plan->gu_done = 0; plan->tile_rows = 16;
            }
        }
    }
    __syncthreads();
    if (tid < n) {
        int p = -1;
        if (e >= 0) {
            p = s_eoffs[e] + cnt[warp][e] + r_in_warp;
            elist[p] = tid;
        }
        pos[tid] = p;
        for (int r = 1; r < FD_CLUSTER; r++) *cluster.map_shared_rank(&s_pos[tid], r) = p;   // no L2 round trip for the scatter
        if (ep.peers) {
            int code = -1;
            if (e >= 0) {
                const int dr = e / ep.per, j = p - s_eoffs[dr * ep.per];
                if (j < ep.cap) {
                    code = (dr << 20) | j;
                    const int row_bytes = D + D / Q36_QK + 16;
                    uint8_t *rowbase = ep.peers[dr] + ((ep_epoch & 1u) ? ep.rows1 : ep.rows0) +
                                       ((size_t)(ep.slot_major ? dr : ep.me) * ep.cap + j) * row_bytes;
                    *reinterpret_cast<int4 *>(rowbase + D + D / Q36_QK) = make_int4(e, 0, 0, 0);     // the row's tail: its expert
                    ep.ypos[tid] = dr * ep.cap + j;
                } else {
                    ep.ypos[tid] = -1;                       // beyond the window's capacity: dropped, and reported
                    if (status) atomicCAS(status, 0, 0xD00);
                }
            } else ep.ypos[tid] = -1;
            for (int r = 1; r < FD_CLUSTER; r++) *cluster.map_shared_rank(&s_slot[tid], r) = code;
        }
    }
    cluster.sync();   // (release/acquire at cluster scope: the remote stores above are visible to their CTAs)
    if (ep.peers) {
        cluster.sync();   // the quantising CTAs have stored their blocks into the peers' windows
        if (tid < ep.world) {
            const int cnt = min(ep.cap, s_eoffs[(tid + 1) * ep.per] - s_eoffs[tid * ep.per]);
            unsigned long long *h = reinterpret_cast<unsigned long long *>(ep.peers[tid] + ((ep_epoch & 1u) ? ep.hdr1 : ep.hdr0)) +
                                    (ep.slot_major ? tid : ep.me);
            const unsigned long long v = (unsigned long long)(unsigned)cnt | ((unsigned long long)ep_epoch << 32);
            asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(h), "l"(v) : "memory");
        }
        __syncthreads();
        if (tid == 0) ep.ctl[0] = (int)ep_epoch;      // phase 0 of this call is over (every CTA read the counter before the barriers above)
    }
    Q36_TR_END(status, 0)
}

// 0 when this front end applies, else the caller takes the general kernels
int launch_front_decode(const float *logits, int n_expert, int k, float scale, int T, int row_stride, int *idx, float *wt,
                        int *ecount, int *eoffs, int *elist, int *pos, int *soffs, int s0, int s1, void *plan, int D, int FF,
                        int *status, const void *X, int x_is_bf16, uint8_t *Xq, uint8_t *Xs, int shared_row0, int put_k,
                        cudaStream_t st, const EpSendArgs *ep) {
    if (T > 16 || T * k > FD_MAX_ENTRIES || n_expert > DISPATCH_MAX_E || n_expert > FD_THREADS || D % (32 * Q36_QK) ||
        T * (D / (32 * Q36_QK)) > FD_QWARPS || s1 - s0 > 16)
        return Q36_MOE_EINVAL;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(FD_CLUSTER);
    cfg.blockDim = dim3(FD_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = FD_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k_front_decode, logits, n_expert, k, scale, T, row_stride, idx, wt, ecount, eoffs, elist, pos,
                       soffs, s0, s1, (TcPlan *)plan, FF / TC_M, D / TC_M, status, X, x_is_bf16, Xq, Xs, D, shared_row0, put_k,
                       ep ? *ep : EpSendArgs{nullptr, 0, 0, 0, 0, nullptr, nullptr, 0, 0, 1, 0, 0});
    return check_launch();
}

// -------------------------------------------------------------- launchers
int launch_router_topk(const float *logits, int n_expert, int k, int *idx, float *wt, float scale,
                       int renorm, int T, int row_stride, cudaStream_t st) {
    if (T <= 0) return Q36_MOE_OK;
    launch_k(k_router_topk, dim3((T + 7) / 8), dim3(256), 0, st, logits, n_expert, k, idx, wt, scale, renorm, T, row_stride);
    return check_launch();
}

// [expert][chunk] counts, then the entries' ranks
uint64_t dispatch_ws_bytes(int n_entries, int n_expert) {
    const uint64_t n_chunk = ((uint64_t)n_entries + DISPATCH_CHUNK - 1) / DISPATCH_CHUNK;
    return n_chunk * n_expert * sizeof(int) + (uint64_t)n_entries * sizeof(unsigned short) + 256;
}
uint64_t route_dispatch_ws_bytes(int T, int k, int n_expert) {
    k = min(k, 8);   // (the layers refuse a larger k; the size queries answer for any, and a chunk holds no token of 513 entries)
    const uint64_t n_chunk = ((uint64_t)T * k + route_chunk(k) - 1) / route_chunk(k);
    return n_chunk * n_expert * sizeof(int) + (uint64_t)T * k * sizeof(unsigned short) + 256;
}

// Entries up to which the scan's own cluster places them: beyond, a launch over the whole chip costs less than its seven SMs take.
// us of a dispatch of 256 experts with the placement in the cluster / in a launch of its own (and, before either, with a scan by one
// block): 512 entries 6.1 / 6.6 (6.0), 4096 entries 7.3 / 7.5 (7.3), 8192 entries 8.7 / 7.6 (7.7), 32,768 entries 12.9 / 9.0 (9.8),
// 262,144 entries 57.5 / 16.0 (34.2).
constexpr int PLACE_IN_CLUSTER = 4096;
// eid == nullptr: the entries are the top-k experts of `logits`, written to idx / wt (per_chunk: whole tokens)
static int dispatch_launches(const float *logits, int row_stride, int k, float scale, int T, int *idx, float *wt, const int *eid, int n,
                             int n_expert, int se0, int se1, int *ecount, int *eoffs, int *elist, int *pos, void *ws, int *soffs, int s0,
                             int s1, cudaStream_t st, void *plan, int D, int FF, int plan_tile_rows) {
    const int per_chunk = eid ? DISPATCH_CHUNK : route_chunk(k), n_chunk = (n + per_chunk - 1) / per_chunk;
    int *cnt_ec = (int *)ws;
    unsigned short *lrank = (unsigned short *)(cnt_ec + (size_t)n_chunk * n_expert);
    if (n > 0) {
        if (eid) launch_k(k_dispatch_count<false>, dim3(n_chunk), dim3(1024), 0, st, logits, row_stride, k, scale, T, idx, wt, eid, n, per_chunk,
                          n_expert, se0, se1, cnt_ec, n_chunk, lrank);
        else launch_k(k_dispatch_count<true>, dim3(n_chunk), dim3(1024), 0, st, logits, row_stride, k, scale, T, idx, wt, eid, n, per_chunk,
                      n_expert, se0, se1, cnt_ec, n_chunk, lrank);
    }
    const bool spread = elist && n > PLACE_IN_CLUSTER;
    if (!eid) eid = idx;
    launch_k_cluster(k_dispatch_scan_place, dim3(1, 1, DISPATCH_CLUSTER), dim3(1024), DISPATCH_CLUSTER, st, eid, n, per_chunk, n_expert, cnt_ec,
                     n_chunk, (const unsigned short *)lrank, ecount, eoffs, spread ? nullptr : elist, pos, soffs, s0, s1, (TcPlan *)plan, se0,
                     se1, plan ? FF / TC_M : 0, plan ? D / TC_M : 0, plan_tile_rows);
    if (spread) launch_k(k_dispatch_place, dim3((n + 255) / 256), dim3(256), 0, st, eid, n, per_chunk, (const int *)cnt_ec, n_chunk,
                         (const unsigned short *)lrank, (const int *)eoffs, elist, pos);
    return check_launch();
}
int launch_dispatch(const int *eid, int n, int n_expert, int se0, int se1, int *ecount, int *eoffs,
                    int *elist, int *pos, void *ws, int *soffs, int s0, int s1, cudaStream_t st, void *plan, int D, int FF,
                    int plan_tile_rows) {
    return dispatch_launches(nullptr, 0, 1, 0.f, 0, nullptr, nullptr, eid, n, n_expert, se0, se1, ecount, eoffs, elist, pos, ws, soffs, s0,
                             s1, st, plan, D, FF, plan_tile_rows);
}
int launch_route_dispatch(const float *logits, int n_expert, int k, float scale, int T, int row_stride, int se0, int se1, int *idx,
                          float *wt, int *ecount, int *eoffs, int *elist, int *pos, void *ws, int *soffs, int s0, int s1,
                          cudaStream_t st, void *plan, int D, int FF, int plan_tile_rows) {
    return dispatch_launches(logits, row_stride, k, scale, T, idx, wt, nullptr, T * k, n_expert, se0, se1, ecount, eoffs, elist, pos, ws,
                             soffs, s0, s1, st, plan, D, FF, plan_tile_rows);
}

static bool quant_rows_takes(int K, int k) { return K % (32 * Q36_QK) == 0 && k <= 8; }
template <bool PLACE>
static void launch_quant_rows(const void *X, int bf16, uint8_t *Xq, uint8_t *Xs, int T, int K, int *pos, int k, int shared_row0,
                              bool early, const PlaceArgs &pl, cudaStream_t st) {
    const unsigned grid = (unsigned)(((long)T * (K / (32 * Q36_QK)) + 7) / 8);
    if (bf16) launch_k(k_quant_rows<true, PLACE>, dim3(grid), dim3(256), 0, st, X, Xq, Xs, T, K, pos, k, shared_row0, early ? 1 : 0, pl);
    else launch_k(k_quant_rows<false, PLACE>, dim3(grid), dim3(256), 0, st, X, Xq, Xs, T, K, pos, k, shared_row0, early ? 1 : 0, pl);
}
// Router, dispatch, plan and the scattered row quantiser of a batch of any size.  What front_mid_takes: one cluster (k_front_mid)
// in front of the quantiser, else the routing count, the scan and the quantiser, which places the entries.
// Measured (us, router to quantised rows, 256 experts, top-8): 33 tokens 9 against 18 with the kernels this replaces, 96
// tokens 8 against 22, 300 tokens 15 against 24, 1001 tokens 23 against 31, 4096 tokens 33 against 47.
int launch_front(const float *logits, int n_expert, int k, float scale, int T, int row_stride, int se0, int se1, int *idx, float *wt,
                 int *ecount, int *eoffs, int *elist, int *pos, void *ws, int *soffs, int s0, int s1, void *plan, int D, int FF,
                 int plan_tile_rows, const void *X, int x_is_bf16, uint8_t *Xq, uint8_t *Xs, int shared_row0, cudaStream_t st) {
    int rc;
    if (front_mid_takes(T, k, n_expert)) {
        if ((rc = launch_front_mid(logits, n_expert, k, scale, T, row_stride, se0, se1, idx, wt, ecount, eoffs, elist, pos, soffs, s0, s1,
                                   plan, D, FF, plan_tile_rows, st)))
            return rc;
        return launch_quant(X, x_is_bf16, Xq, Xs, T, D, pos, k, shared_row0, true, st, true);
    }
    const bool place = quant_rows_takes(D, k);
    if ((rc = launch_route_dispatch(logits, n_expert, k, scale, T, row_stride, se0, se1, idx, wt, ecount, eoffs, place ? nullptr : elist,
                                    pos, ws, soffs, s0, s1, st, plan, D, FF, plan_tile_rows)))
        return rc;
    if (!place) return launch_quant(X, x_is_bf16, Xq, Xs, T, D, pos, k, shared_row0, true, st, true);
    const int per_chunk = route_chunk(k), n_chunk = (T * k + per_chunk - 1) / per_chunk;
    const int *cnt_ec = (const int *)ws;
    launch_quant_rows<true>(X, x_is_bf16, Xq, Xs, T, D, pos, k, shared_row0, true,
                            PlaceArgs{idx, cnt_ec, eoffs, (const unsigned short *)(cnt_ec + (size_t)n_chunk * n_expert), n_chunk, per_chunk}, st);
    return check_launch();
}

int launch_quant(const void *X, int bf16, uint8_t *Xq, uint8_t *Xs, int T, int K, const int *pos,
                 int k, int shared_row0, bool scatter, cudaStream_t st, bool early) {
    if (T <= 0) return Q36_MOE_OK;
    const long warps = (long)T * (K / Q36_QK);
    const unsigned grid = (unsigned)((warps + 7) / 8);
    if (scatter && quant_rows_takes(K, k)) {
        launch_quant_rows<false>(X, bf16, Xq, Xs, T, K, const_cast<int *>(pos), k, shared_row0, early, PlaceArgs{}, st);
    } else if (scatter) {
        if (bf16) launch_k(k_quant_e4m3<true, true>, dim3(grid), dim3(256), 0, st, X, Xq, Xs, T, K, pos, k, shared_row0);
        else launch_k(k_quant_e4m3<false, true>, dim3(grid), dim3(256), 0, st, X, Xq, Xs, T, K, pos, k, shared_row0);
    } else {
        if (bf16) launch_k(k_quant_e4m3<true, false>, dim3(grid), dim3(256), 0, st, X, Xq, Xs, T, K, nullptr, 0, -1);
        else launch_k(k_quant_e4m3<false, false>, dim3(grid), dim3(256), 0, st, X, Xq, Xs, T, K, nullptr, 0, -1);
    }
    return check_launch();
}

}  // namespace q36

// ------------------------------------------------- dispatch without a workspace
// Scratch of q36_moe_dispatch_noalloc: the per-(chunk, expert) counters and the per-entry ranks of the
// dispatch kernels for at most Q36_MOE_NOALLOC_MAX_ENTRIES entries and 512 experts.  It lives in the library
// image: every GPU that loads the library carries these 96 KiB until the process exits.
static constexpr int NOALLOC_MAX_ENTRIES = 16384;
static constexpr int NOALLOC_MAX_EXPERTS = q36::DISPATCH_MAX_E;
static constexpr size_t NOALLOC_SCRATCH_INTS =
    (size_t)(NOALLOC_MAX_ENTRIES / q36::DISPATCH_CHUNK) * NOALLOC_MAX_EXPERTS + NOALLOC_MAX_ENTRIES / 2;
static __device__ __align__(256) int g_noalloc_scratch[NOALLOC_SCRATCH_INTS];

// Device address of the array above, looked up once per device.  In host code the symbol is only a
// stand-in: kernels must be given the address cudaGetSymbolAddress returns for the CURRENT device.
static int *g_noalloc_ptr[64] = {nullptr};

extern "C" int q36_moe_dispatch_noalloc(const int *expert_of_entry, int n_entries, int n_expert, int se0, int se1,
                                        int *ecount, int *eoffs, int *elist, int *pos, void *stream) {
    if (!ecount || !eoffs || n_entries < 0) return Q36_MOE_EINVAL;
    if (n_entries > 0 && (!expert_of_entry || !elist || !pos)) return Q36_MOE_EINVAL;   // no entries: nothing to read or place
    if (n_expert <= 0 || se0 < 0 || se0 > se1 || se1 > n_expert) return Q36_MOE_EINVAL;
    if (n_entries > NOALLOC_MAX_ENTRIES || n_expert > NOALLOC_MAX_EXPERTS) {
        fprintf(stderr,
                "q36_moe_dispatch_noalloc: %d entries / %d experts exceed the built-in scratch (max %d entries, %d "
                "experts); use q36_moe_dispatch with a caller workspace\n",
                n_entries, n_expert, NOALLOC_MAX_ENTRIES, NOALLOC_MAX_EXPERTS);
        return Q36_MOE_ENOSPACE;
    }
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { q36::last_cuda_error() = (int)e; return Q36_MOE_ECUDA; }
    if (dev < 0 || dev >= 64) {
        fprintf(stderr, "q36_moe_dispatch_noalloc: device ordinal %d is beyond the 64 this entry keeps an address for\n", dev);
        return Q36_MOE_EINVAL;
    }
    if (!g_noalloc_ptr[dev]) {   // first call on this device: resolve the array's device address
        int *p = nullptr;
        e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) { q36::last_cuda_error() = (int)e; return Q36_MOE_ECUDA; }
        g_noalloc_ptr[dev] = p;
    }
    // Nothing in the scratch has to start at zero: k_dispatch_count writes every counter of every chunk it
    // covers and the rank of every entry before the later kernels read them.
    return q36::launch_dispatch(expert_of_entry, n_entries, n_expert, se0, se1, ecount, eoffs, elist, pos,
                                g_noalloc_ptr[dev], nullptr, 0, 0, (cudaStream_t)stream, nullptr, 0, 0, 0);
}
