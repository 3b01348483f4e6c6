// The steps either side of the expert computation, so that a block can be driven from the residual stream:
//
//   before  h += a; x = rmsnorm(h) * w; logits = router_w . x
//           k_add_rmsnorm (q36_engine.cu:696-706) + k_matvec_f32_row (q36_ops.cuh:331-342) at decode,
//           k_rmsnorm_b + pf_gemm(f32 router) + pf_gemm(shared gate) when batched (q36_engine.cu:3426-3427, 3469)
//   after   moe = combine(...); h += moe; x_next = rmsnorm(h) * w_next
//           k_moe_combine(_pf) (q36_engine.cu:785-791, 3393-3401) + k_add_rmsnorm (:696-706, :1966)
//
// The router logits are f32 dot products at every batch size (the engine's batched path rounds both operands to fp16 for its
// wmma GEMM).  The order of a dot product's additions follows the batch: one up to 16 tokens, K cut in eight or four pieces in
// the split kernel (and over two groups of warps from 1025 tokens on), one run over K beyond 2.2 tiles per SM.  So the same token
// may get logits that differ in the last bits in two batches, and another expert where two tie to these.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.cuh"

namespace q36 {

__device__ __forceinline__ float block_sum_256(float v, float *part) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) part[wid] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) s += part[i];   // every thread adds the eight partials in the same order
    __syncthreads();
    return s;
}

// ------------------------------------------------------------------ before
// One block per token row.  Also computes the extra logit column `gate_row` (the shared-expert gate: one more
// router row) while the normalised row is in registers.  D <= 256 * 4 * ROW_F4 floats.
constexpr int ROW_F4 = 4;   // float4 per thread: rows up to 4096 floats
__global__ void __launch_bounds__(256)
k_add_rmsnorm_rows(float *__restrict__ h, const float *__restrict__ a, const float *__restrict__ w, float eps,
                   float *__restrict__ x, const float *__restrict__ gate_row, float *__restrict__ logits, int logit_stride,
                   int gate_col, int D) {
    // synchronise FIRST: the next grid (k_router_logits_small) reads the router matrix before its own wait
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    __shared__ float part[8];
    const int t = blockIdx.x, n4 = D / 4;
    float4 *hr = reinterpret_cast<float4 *>(h + (size_t)t * D);
    const float4 *ar = a ? reinterpret_cast<const float4 *>(a + (size_t)t * D) : nullptr;
    float4 v[ROW_F4];
    float loc = 0.f;
#pragma unroll
    for (int j = 0; j < ROW_F4; j++) {
        const int i = threadIdx.x + j * 256;
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n4) {
            v[j] = hr[i];
            if (ar) {
                const float4 b = ar[i];
                v[j].x += b.x; v[j].y += b.y; v[j].z += b.z; v[j].w += b.w;
                hr[i] = v[j];
            }
            loc += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
        }
    }
    const float ss = rsqrtf(block_sum_256(loc, part) / (float)D + eps);
    float gdot = 0.f;
#pragma unroll
    for (int j = 0; j < ROW_F4; j++) {
        const int i = threadIdx.x + j * 256;
        if (i < n4) {
            const float4 ww = reinterpret_cast<const float4 *>(w)[i];
            float4 o;
            o.x = v[j].x * ss * ww.x; o.y = v[j].y * ss * ww.y; o.z = v[j].z * ss * ww.z; o.w = v[j].w * ss * ww.w;
            reinterpret_cast<float4 *>(x + (size_t)t * D)[i] = o;
            if (gate_row) {
                const float4 g = reinterpret_cast<const float4 *>(gate_row)[i];
                gdot += o.x * g.x + o.y * g.y + o.z * g.z + o.w * g.w;
            }
        }
    }
    if (gate_row) {
        gdot = block_sum_256(gdot, part);
        if (threadIdx.x == 0) logits[(size_t)t * logit_stride + gate_col] = gdot;
    }
}

// Router logits for a handful of tokens (T <= 16): a block per two router rows, the rows in registers.
// Latency-bound: 2.1 MB of router matrix and T * 8 KB of activations are nothing next to the chain load -> FMA ->
// reduce.  So every thread holds its 8 elements of both rows, loaded BEFORE the grid dependency resolves (the
// predecessor k_add_rmsnorm_rows lets this grid start only after it has itself seen everything before it complete, so
// the router matrix is as settled here as after the wait), all token loads are independent, and the 2 * TT partial sums
// of a warp are reduced together by halving exchanges (31 shuffles for 32 sums instead of 160).
// The previous form (a warp per row walking K in 16 dependent steps) took 18.6 us at T = 5, D = 2048; see the launcher.
constexpr int RL_T = 16;
template <int TT>
__global__ void __launch_bounds__(256)
k_router_logits_small(const float *__restrict__ W, const float *__restrict__ x, float *__restrict__ logits, int logit_stride,
                      int n_rows, int T, int D) {
    constexpr int V = 2 * TT;
    const int n4 = D / 4, tid = threadIdx.x, lane = tid & 31, row0 = blockIdx.x * 2;
    float4 w[2][ROW_F4];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int j = 0; j < ROW_F4; j++) {
            const int i = tid + j * 256;
            w[r][j] = (i < n4 && row0 + r < n_rows) ? __ldg(reinterpret_cast<const float4 *>(W + (size_t)(row0 + r) * D) + i)
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    float v[V];
#pragma unroll
    for (int i = 0; i < V; i++) v[i] = 0.f;
#pragma unroll
    for (int t = 0; t < TT; t++) {
        if (t >= T) break;
#pragma unroll
        for (int j = 0; j < ROW_F4; j++) {
            const int i = tid + j * 256;
            if (i < n4) {
                const float4 xv = reinterpret_cast<const float4 *>(x + (size_t)t * D)[i];
#pragma unroll
                for (int r = 0; r < 2; r++)
                    v[2 * t + r] += w[r][j].x * xv.x + w[r][j].y * xv.y + w[r][j].z * xv.z + w[r][j].w * xv.w;
            }
        }
    }
    // halving exchange: after the step over lane bit o a lane holds the sums of its half of the values
    int n = V;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < V / 2; i++)
                if (i < n) {
                    const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    __shared__ float part[8][V];
    constexpr int PER = 32 / V;                    // lanes that hold the same sum
    if (lane % PER == 0) part[tid >> 5][lane / PER] = v[0];
    __syncthreads();
    if (tid < V) {
        const int t = tid >> 1, r = row0 + (tid & 1);
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) s += part[i][tid];
        if (t < T && r < n_rows) logits[(size_t)t * logit_stride + r] = s;
    }
}

// Router logits for a batch: logits[t][r] = x[t][:] . W[r][:] in f32 FMAs, BT tokens x 64 rows per block, 8 x TJ outputs
// per thread, K in chunks of 16 through a ring of cp.async stages.  Both operands stay row-major in shared memory; rows
// of 80 B and interleaved row ownership keep the 16-byte reads of a quarter warp in different bank groups.
// T * 256 outputs are few tiles (300 tokens: 20), so the K axis is split over the `gridDim.z` CTAs of a cluster and the
// partial tiles are added through distributed shared memory in rank order (the same bits from run to run): 20.9 us at 300
// tokens where one CTA per tile took 135.  With full chips it is bound by shared-memory reads beside the FMAs: 8 x 8
// outputs per thread and two groups of warps over a chunk's k range from 1025 tokens on (2000 tokens: 77 us against 86
// with 8 x 4, which keeps more warps busy below that: 1000 tokens 37 against 41).
constexpr int RG_BR = 64, RG_BK = 16, RG_LD = RG_BK + 4;
template <int BT, int TJ, int KG>
struct RouterGemm {
    static constexpr int TX = RG_BR / TJ, TY = BT / 8, GROUP = TX * TY, THREADS = GROUP * KG;
    static constexpr int ROWS = BT + RG_BR, STAGES = BT == 128 ? 3 : 4;
    static constexpr int LOADS = ROWS * 4 / THREADS;          // 16-byte copies per thread and stage
    static constexpr int KSTEPS = RG_BK / 4 / KG;             // 4-element k steps of a chunk per warp group
    static_assert(GROUP % 32 == 0 && ROWS * 4 % THREADS == 0 && BT * RG_BR <= STAGES * ROWS * RG_LD, "shape");
};
template <int BT, int TJ, int KG>
__global__ void __launch_bounds__(RouterGemm<BT, TJ, KG>::THREADS, 512 / RouterGemm<BT, TJ, KG>::THREADS)
k_router_logits_gemm(const float *__restrict__ W, const float *__restrict__ x, float *__restrict__ logits, int logit_stride,
                     int n_rows, int T, int D) {
    using C = RouterGemm<BT, TJ, KG>;
    Q36_GDS();
    namespace cg = cooperative_groups;
    __shared__ __align__(16) float stage[C::STAGES][C::ROWS][RG_LD];     // rows [0, BT) tokens, then router rows
    float (*part)[RG_BR] = reinterpret_cast<float (*)[RG_BR]>(&stage[0][0][0]);   // later: this CTA's sums over its share of K
    const int t0 = blockIdx.y * BT, r0 = blockIdx.x * RG_BR, tid = threadIdx.x;
    const int nz = gridDim.z, chunks = D / RG_BK;
    const int c_begin = (int)((long)chunks * blockIdx.z / nz), c_end = (int)((long)chunks * (blockIdx.z + 1) / nz);
    const int kg = tid / C::GROUP, tx = tid % C::TX, ty = (tid % C::GROUP) / C::TX;   // tokens ty + TY i, rows tx + TX j
    auto load = [&](int c, int s) {
#pragma unroll
        for (int i = 0; i < C::LOADS; i++) {
            const int id = tid + i * C::THREADS, row = id >> 2, k4 = (id & 3) * 4;
            const bool tok = row < BT;
            const int g = tok ? t0 + row : r0 + row - BT;
            const bool in = tok ? g < T : g < n_rows;
            const float *src = (tok ? x : W) + (size_t)(in ? g : 0) * D + c * RG_BK + k4;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&stage[s][row][k4]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
        }
    };
    float acc[8][TJ];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TJ; j++) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < C::STAGES - 1; s++) {
        if (c_begin + s < c_end) load(c_begin + s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int c = c_begin; c < c_end; c++) {
        const int s = (c - c_begin) % C::STAGES;
        asm volatile("cp.async.wait_group %0;" ::"n"(C::STAGES - 2) : "memory");
        __syncthreads();                                            // chunk c has landed, and chunk c - 1 is used up
        if (c + C::STAGES - 1 < c_end) load(c + C::STAGES - 1, (c - c_begin + C::STAGES - 1) % C::STAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int q = 0; q < C::KSTEPS; q++) {
            const int k4 = (kg * C::KSTEPS + q) * 4;
            float4 wv[TJ];
#pragma unroll
            for (int j = 0; j < TJ; j++) wv[j] = *reinterpret_cast<const float4 *>(&stage[s][BT + tx + C::TX * j][k4]);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 xv = *reinterpret_cast<const float4 *>(&stage[s][ty + C::TY * i][k4]);
#pragma unroll
                for (int j = 0; j < TJ; j++) {
                    acc[i][j] = fmaf(xv.x, wv[j].x, acc[i][j]); acc[i][j] = fmaf(xv.y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(xv.z, wv[j].z, acc[i][j]); acc[i][j] = fmaf(xv.w, wv[j].w, acc[i][j]);
                }
            }
        }
    }
    for (int g = 0; g < KG; g++) {                                   // the warp groups add their sums in turn
        __syncthreads();
        if (kg == g) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < TJ; j++) {
                    float &d = part[ty + C::TY * i][tx + C::TX * j];
                    d = g ? d + acc[i][j] : acc[i][j];
                }
        }
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    // CTA z of the cluster adds and writes its share of the token rows
    const int z = blockIdx.z, tok0 = BT * z / nz, tok_per = BT * (z + 1) / nz - tok0;
    for (int i = tid; i < tok_per * (RG_BR / 4); i += C::THREADS) {
        const int tt = tok0 + i / (RG_BR / 4), rr = (i % (RG_BR / 4)) * 4, t = t0 + tt;
        float4 v[8];                                                // (all remote reads in flight before the first add)
#pragma unroll
        for (int p = 0; p < 8; p++)
            v[p] = p < nz ? *reinterpret_cast<const float4 *>(cluster.map_shared_rank(&part[tt][rr], p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 s = v[0];
#pragma unroll
        for (int p = 1; p < 8; p++) { s.x += v[p].x; s.y += v[p].y; s.z += v[p].z; s.w += v[p].w; }
        const float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (t < T && r0 + rr + j < n_rows) logits[(size_t)t * logit_stride + r0 + rr + j] = sv[j];
    }
    cluster.sync();   // nobody leaves while its partial tile may still be read
}

// The same for very many tokens: 128 tokens x 64 rows per block, K in chunks of 16 through shared memory (register-prefetched,
// k-major), 8 x 4 outputs per thread.  With more than two tiles per SM the SMs are full without a split of K, and what counts is
// warps in flight beside a short inner loop: 79 registers a thread leave room for three blocks, 128 of the kernel above for two.  The rule
// is in the launcher.
constexpr int RM_BT = 128;
__global__ void __launch_bounds__(256)
k_router_logits_many(const float *__restrict__ W, const float *__restrict__ x, float *__restrict__ logits, int logit_stride,
                     int n_rows, int T, int D) {
    Q36_GDS();
    __shared__ float sx[RG_BK][RM_BT + 4];   // [k][token]
    __shared__ float sw[RG_BK][RG_BR + 4];   // [k][row]
    const int t0 = blockIdx.y * RM_BT, r0 = blockIdx.x * RG_BR, tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;   // thread tile: tokens ty * 8 .. + 8, rows tx * 4 .. + 4
    // loaders: x tile 128 x 16 floats = 512 float4 (2 per thread), W tile 64 x 16 = 256 float4 (1 per thread)
    const int lx_t = tid >> 2, lx_k = (tid & 3) * 4;          // tokens lx_t and lx_t + 64
    const int lw_r = tid >> 2, lw_k = (tid & 3) * 4;
    float4 px0, px1, pw;
    auto fetch = [&](int k0) {
        const int ta = t0 + lx_t, tb = ta + 64, r = r0 + lw_r;
        px0 = (ta < T) ? *reinterpret_cast<const float4 *>(x + (size_t)ta * D + k0 + lx_k) : make_float4(0.f, 0.f, 0.f, 0.f);
        px1 = (tb < T) ? *reinterpret_cast<const float4 *>(x + (size_t)tb * D + k0 + lx_k) : make_float4(0.f, 0.f, 0.f, 0.f);
        pw = (r < n_rows) ? *reinterpret_cast<const float4 *>(W + (size_t)r * D + k0 + lw_k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto stash = [&]() {
        sx[lx_k][lx_t] = px0.x; sx[lx_k + 1][lx_t] = px0.y; sx[lx_k + 2][lx_t] = px0.z; sx[lx_k + 3][lx_t] = px0.w;
        sx[lx_k][lx_t + 64] = px1.x; sx[lx_k + 1][lx_t + 64] = px1.y; sx[lx_k + 2][lx_t + 64] = px1.z; sx[lx_k + 3][lx_t + 64] = px1.w;
        sw[lw_k][lw_r] = pw.x; sw[lw_k + 1][lw_r] = pw.y; sw[lw_k + 2][lw_r] = pw.z; sw[lw_k + 3][lw_r] = pw.w;
    };
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    fetch(0);
    for (int k0 = 0; k0 < D; k0 += RG_BK) {
        stash();
        __syncthreads();
        if (k0 + RG_BK < D) fetch(k0 + RG_BK);
#pragma unroll
        for (int kk = 0; kk < RG_BK; kk++) {
            const float4 xa = *reinterpret_cast<const float4 *>(&sx[kk][ty * 8]);
            const float4 xb = *reinterpret_cast<const float4 *>(&sx[kk][ty * 8 + 4]);
            const float4 wv = *reinterpret_cast<const float4 *>(&sw[kk][tx * 4]);
            const float xs[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
            const float ws[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(xs[i], ws[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int t = t0 + ty * 8 + i;
        if (t >= T) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = r0 + tx * 4 + j;
            if (r < n_rows) logits[(size_t)t * logit_stride + r] = acc[i][j];
        }
    }
}

// ------------------------------------------------------------------- after
// One block per token: the weighted combine in slot order (as k_combine), then the residual add and the next
// RMSNorm while the row is in registers.  EARLY_META: see k_combine (moe_gemv.cu).
template <bool EARLY_META>
__global__ void __launch_bounds__(256)
k_combine_add_rmsnorm(float *__restrict__ moe_out, const float *__restrict__ Y, const int *__restrict__ pos,
                      const float *__restrict__ wt, const float *__restrict__ SH, const float *__restrict__ shgate,
                      int shgate_stride, float *__restrict__ h, const float *__restrict__ w_next, float eps,
                      float *__restrict__ x_next, int D, int k, int y_bf16) {
    if (!EARLY_META) Q36_GDS();
    else cudaTriggerProgrammaticLaunchCompletion();
    __shared__ float part[8];
    const int t = blockIdx.x, n4 = D / 4;
    constexpr int KMAX = 8;
    int p[KMAX];
    float wgt[KMAX];
#pragma unroll
    for (int s = 0; s < KMAX; s++) {
        p[s] = (s < k) ? pos[(size_t)t * k + s] : -1;
        wgt[s] = (s < k) ? wt[(size_t)t * k + s] : 0.f;
    }
    const float gs = (SH && shgate) ? sigm_f(shgate[(size_t)t * shgate_stride]) : 1.f;
    if (EARLY_META) cudaGridDependencySynchronize();
    float4 acc[ROW_F4];
    float loc = 0.f;
#pragma unroll
    for (int j = 0; j < ROW_F4; j++) {
        const int i = threadIdx.x + j * 256;
        acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= n4) continue;
        float4 y[KMAX];
        float4 ysh = make_float4(0.f, 0.f, 0.f, 0.f);
        if (SH) ysh = ld_y4(SH, (size_t)t * D + 4 * (size_t)i, y_bf16);
#pragma unroll
        for (int s = 0; s < KMAX; s++)
            y[s] = (p[s] >= 0) ? ld_y4(Y, (size_t)p[s] * D + 4 * (size_t)i, y_bf16) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 hv = reinterpret_cast<const float4 *>(h + (size_t)t * D)[i];
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < KMAX; s++) {
            if (p[s] < 0) continue;
            m.x = fmaf(wgt[s], y[s].x, m.x); m.y = fmaf(wgt[s], y[s].y, m.y);
            m.z = fmaf(wgt[s], y[s].z, m.z); m.w = fmaf(wgt[s], y[s].w, m.w);
        }
        if (SH) { m.x = fmaf(gs, ysh.x, m.x); m.y = fmaf(gs, ysh.y, m.y); m.z = fmaf(gs, ysh.z, m.z); m.w = fmaf(gs, ysh.w, m.w); }
        if (moe_out) __stcs(reinterpret_cast<float4 *>(moe_out + (size_t)t * D) + i, m);
        float4 r = make_float4(hv.x + m.x, hv.y + m.y, hv.z + m.z, hv.w + m.w);
        reinterpret_cast<float4 *>(h + (size_t)t * D)[i] = r;
        acc[j] = r;
        loc += r.x * r.x + r.y * r.y + r.z * r.z + r.w * r.w;
    }
    const float ss = rsqrtf(block_sum_256(loc, part) / (float)D + eps);
#pragma unroll
    for (int j = 0; j < ROW_F4; j++) {
        const int i = threadIdx.x + j * 256;
        if (i >= n4) continue;
        const float4 ww = reinterpret_cast<const float4 *>(w_next)[i];
        float4 o;
        o.x = acc[j].x * ss * ww.x; o.y = acc[j].y * ss * ww.y; o.z = acc[j].z * ss * ww.z; o.w = acc[j].w * ss * ww.w;
        reinterpret_cast<float4 *>(x_next + (size_t)t * D)[i] = o;
    }
}

// ---------------------------------------------------------------- launchers
int launch_pre_norm_router(float *h, const float *a, const float *norm_w, float eps, const float *router_w, int n_rows,
                           int gate_row, float *x, float *logits, int logit_stride, int T, int D, cudaStream_t st) {
    if (T <= 0) return Q36_MOE_OK;
    if (D % 4 || D > 256 * 4 * ROW_F4 || n_rows <= 0 || logit_stride < n_rows) return Q36_MOE_EINVAL;
    // the shared-gate row (one extra router row) is taken by the norm kernel itself when batched; the decode-sized
    // logits kernel reads every row once for all tokens and takes it along
    const bool small = T <= RL_T;
    const float *gate = (!small && gate_row >= 0) ? router_w + (size_t)gate_row * D : nullptr;
    launch_k(k_add_rmsnorm_rows, dim3(T), dim3(256), 0, st, h, a, norm_w, eps, x, gate, logits, logit_stride, gate_row, D);
    if (small) {
        const dim3 grid((n_rows + 1) / 2), block(256);
        const float *xc = x;
        if (T == 1) launch_k(k_router_logits_small<1>, grid, block, 0, st, router_w, xc, logits, logit_stride, n_rows, T, D);
        else if (T == 2) launch_k(k_router_logits_small<2>, grid, block, 0, st, router_w, xc, logits, logit_stride, n_rows, T, D);
        else if (T <= 4) launch_k(k_router_logits_small<4>, grid, block, 0, st, router_w, xc, logits, logit_stride, n_rows, T, D);
        else if (T <= 8) launch_k(k_router_logits_small<8>, grid, block, 0, st, router_w, xc, logits, logit_stride, n_rows, T, D);
        else launch_k(k_router_logits_small<16>, grid, block, 0, st, router_w, xc, logits, logit_stride, n_rows, T, D);
    } else {
        if (D % RG_BK) return Q36_MOE_EINVAL;
        const int rows = (gate_row == n_rows - 1) ? n_rows - 1 : n_rows;   // the gate row is done already when it is the last one
        if (gate_row >= 0 && gate_row != n_rows - 1) return Q36_MOE_EINVAL;
        // Tile and split of K: small tiles and eight CTAs per tile until the tiles alone fill the chip; the tiles of a larger batch
        // are still split in four so that the last wave is short (T = 8192: 256 tiles on 148 SMs).  From 2.2 tiles per SM on the
        // unsplit kernel with more warps: us with the split one / with that one at 257 rows: 9600 tokens (300 tiles) 330 / 360,
        // 10,500 (332) 367 / 362, 12,000 402 / 366, 16,384 545 / 494, 20,000 659 / 602, 65,536 2092 / 1674.
        const int bt = T <= 128 ? 32 : T <= 1024 ? 64 : 128, row_tiles = (rows + RG_BR - 1) / RG_BR;
        const long tiles = (long)row_tiles * ((T + bt - 1) / bt);
        if (bt == RM_BT && tiles * 5 > (long)sm_count() * 11) {
            launch_k(k_router_logits_many, dim3(row_tiles, (T + bt - 1) / bt), dim3(256), 0, st, router_w, (const float *)x, logits, logit_stride,
                     rows, T, D);
            return check_launch();
        }
        const int chunks = D / RG_BK, z = tiles <= sm_count() && chunks >= 8 ? 8 : chunks >= 4 ? 4 : 1;
        const dim3 grid(row_tiles, (T + bt - 1) / bt, z);
        const float *xc = x;
        if (bt == 32) launch_k_cluster(k_router_logits_gemm<32, 4, 1>, grid, dim3(64), z, st, router_w, xc, logits, logit_stride, rows, T, D);
        else if (bt == 64) launch_k_cluster(k_router_logits_gemm<64, 4, 1>, grid, dim3(128), z, st, router_w, xc, logits, logit_stride, rows, T, D);
        else launch_k_cluster(k_router_logits_gemm<128, 8, 2>, grid, dim3(256), z, st, router_w, xc, logits, logit_stride, rows, T, D);
    }
    return check_launch();
}

int launch_combine_add_rmsnorm(float *moe_out, const float *Y, const int *pos, const float *wt, const float *SH,
                               const float *shgate, int shgate_stride, float *h, const float *w_next, float eps, float *x_next,
                               int D, int k, int T, bool early_meta, cudaStream_t st, int y_bf16) {
    if (T <= 0) return Q36_MOE_OK;
    if (k <= 0 || k > 8 || D % 4 || D > 256 * 4 * ROW_F4) return Q36_MOE_EINVAL;
    if (early_meta)
        launch_k(k_combine_add_rmsnorm<true>, dim3(T), dim3(256), 0, st, moe_out, Y, pos, wt, SH, shgate, shgate_stride, h, w_next,
                 eps, x_next, D, k, y_bf16);
    else
        launch_k(k_combine_add_rmsnorm<false>, dim3(T), dim3(256), 0, st, moe_out, Y, pos, wt, SH, shgate, shgate_stride, h, w_next,
                 eps, x_next, D, k, y_bf16);
    return check_launch();
}

}  // namespace q36
