// Mean-field relaxation kernels (see anc_meanfield.cuh for the recurrence): the J x m GEMM on tcgen05 (kind::f16,
// BF16 operands, f32 accumulation in TMEM) and the fused forward / adjoint elementwise steps.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "anc_meanfield.cuh"
#include "anc_ptx.cuh"
#include "anc_tensor.cuh"

namespace anc {

namespace {
struct PsForm;
}

struct MfContext {
    int n = 0, npad = 0;
    __nv_bfloat16* J = nullptr;       // [npad][npad] (zero padded)
    float* bias = nullptr;            // [npad]
    float* partial = nullptr;         // [npad / 256][64][npad] split-K partial products
    float* mring = nullptr;           // forward ring: 3 x [64][npad]
    __nv_bfloat16* xm = nullptr;      // [3][64][npad]: hi / mid / lo of the m operand (twice in the persistent form)
    __nv_bfloat16* xp = nullptr;      // [3][64][npad]: hi / mid / lo of the adjoint operand (likewise)
    float* seg_m = nullptr;           // [kMfCheckpoint + 2][64][npad]: m_{t0-1} .. m_{t0+16} of a segment
    float* seg_P = nullptr;           // [kMfCheckpoint][64][npad]
    float* pbar = nullptr;            // [3][64][npad] ring of pbar_t
    float* svec = nullptr;            // [3][nch][64] ring of s_t, per 256-column chunk
    Workspace steps;                  // nbuf and gparts
    float* nbuf = nullptr;            // [S + 1][nch][64] soft counts n_t, per 256-column chunk
    float* gparts = nullptr;          // [S][4][nch][64] per-chunk schedule-gradient sums
    int nbuf_steps = 0;
    int* err = nullptr;               // device error word
    const PsForm* form = nullptr;   // the persistent form, null: the launch sequences
    bool loaded[2] = {false, false};  // its forward and adjoint kernels' attributes are set
    unsigned* cnt = nullptr;          // the persistent form's counters
    uint64_t wait_ns = ptx::kWaitNs;  // limit of each device wait before the kernel gives up (recorded in the graphs)
    CUtensorMap mapJ, mapXm[3], mapXp[3];
    // CUDA graphs of the forward and adjoint launch sequences (one step count each), captured on internal buffers:
    // the caller's inputs are copied in and the outputs copied out around each graph launch
    cudaStream_t cap = nullptr;
    cudaGraphExec_t fwd_exec = nullptr, bwd_exec = nullptr;
    int fwd_S = 0, bwd_S = 0, io_steps = 0;
    float* sched_i = nullptr;         // [4][S]
    float* m0_i = nullptr;            // [64][npad]
    float* mprev_i = nullptr;
    float* mout_i = nullptr;
    float* gm_i = nullptr;
    float* ckpt_i = nullptr;          // [ceil(S/16)][2][64][npad]
    float* gs_i = nullptr;            // [S][4][64]
};

namespace {

using namespace ptx;

// Programmatic dependent launch. Every kernel of a step sequence lets the next one in the stream launch right away
// (pdl_trigger), so that kernel's prologue -- TMEM allocation, barrier set-up, the TMA load of its J tile -- overlaps
// this kernel; it then waits for this kernel to complete, with its memory visible (pdl_wait), before reading anything
// this kernel wrote. Both are no-ops in a kernel launched without the programmatic-serialization attribute.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

constexpr int kRows = 128;                 // rows of J per CTA (MMA M)
constexpr int kRep = kMfReplicas;          // MMA N
constexpr int kKC = 256;                   // K per CTA: 4 swizzle atoms of 64 BF16
constexpr int kGemmThreads = 128;
constexpr int kElemThreads = 256;
constexpr int kErrFull = 11, kErrDone = 12;
constexpr uint32_t kATile = kRows * 128;   // 16 KB: 128 rows x 64 BF16
constexpr uint32_t kBTile = kRep * 128;    // 8 KB: 64 rows x 64 BF16

size_t gemm_smem() { return 1024 + 4 * size_t(kATile) + 12 * size_t(kBTile) + 64; }

// partial[ks][r][y] = sum_{x in [256 ks, 256 ks + 256)} J[y][x] * (X0 + X1 + X2)[r][x], X = the three BF16 terms of
// an f32 operand (24 significant bits; J is exact in BF16, so every product is exact); grid (npad / 128, npad / 256).
__global__ void __launch_bounds__(kGemmThreads, 1)
    mf_gemm_kernel(const __grid_constant__ CUtensorMap mapJ, const __grid_constant__ CUtensorMap mapXh,
                   const __grid_constant__ CUtensorMap mapXm, const __grid_constant__ CUtensorMap mapXl,
                   float* __restrict__ partial, int npad, int* err, uint64_t wait_ns) {
    // kind::f16 instruction descriptor: f32 accumulator, BF16 A and B, both K-major, N = 64, M = 128
    constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(kRep >> 3) << 17) | (uint32_t(kRows >> 4) << 24);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sa = smem;
    uint8_t* sbh = sa + 4 * kATile;
    uint8_t* sbm = sbh + 4 * kBTile;
    uint8_t* sbl = sbm + 4 * kBTile;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sbl + 4 * kBTile);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int y0 = blockIdx.x * kRows, k0 = blockIdx.y * kKC;
    const uint32_t bar_full = smem_u32(bars), bar_done = smem_u32(bars + 1);
    pdl_trigger();
    if (tid == 0) {
        mbar_init(bar_full, 1);
        mbar_init(bar_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    if (tid == 0) {
        mbar_arrive_expect_tx(bar_full, 4 * (kATile + 3 * kBTile));
        for (int a = 0; a < 4; ++a) tma_load_2d(smem_u32(sa + a * kATile), &mapJ, k0 + 64 * a, y0, bar_full);
        // the operand terms come from the previous kernel; the partials this CTA writes are read by the previous
        // step's elementwise kernel: both only after it completed. The other threads write only after bar_done,
        // which follows this wait.
        pdl_wait();
        for (int a = 0; a < 4; ++a) {
            tma_load_2d(smem_u32(sbh + a * kBTile), &mapXh, k0 + 64 * a, 0, bar_full);
            tma_load_2d(smem_u32(sbm + a * kBTile), &mapXm, k0 + 64 * a, 0, bar_full);
            tma_load_2d(smem_u32(sbl + a * kBTile), &mapXl, k0 + 64 * a, 0, bar_full);
        }
        // a wait that gives up (after wait_ns) records the error, then waits once more, bounded by kWaitNs, for the
        // copies it issued, so that none is in flight when the CTA skips its MMAs and exits
        const bool ok = mbar_wait_for(bar_full, 0u, err, kErrFull, wait_ns);
        if (!ok) mbar_wait_for(bar_full, 0u, nullptr, 0, kWaitNs);
        tc_fence_after();
        if (ok) {
            // The tensor core's f32 accumulation truncates toward zero each time an MMA adds into an accumulator, a
            // bias of up to half an ulp of the accumulator per add. Keeping the leading-term products of each 64-wide
            // K atom in their own accumulator (columns 64a .. 64a + 63) and the small mid / lo products in a fifth
            // (columns 256 ..) keeps the accumulators small and the adds per accumulator few; the epilogue sums them
            // with round-to-nearest.
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_f16(tmem + uint32_t(64 * a), sw128_desc(smem_u32(sa + a * kATile) + 32 * kk),
                            sw128_desc(smem_u32(sbh + a * kBTile) + 32 * kk), IDESC, kk != 0 ? 1u : 0u);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    mma_f16(tmem + 256u, sw128_desc(smem_u32(sa + a * kATile) + 32 * kk),
                            sw128_desc(smem_u32(sbm + a * kBTile) + 32 * kk), IDESC, (a | kk) != 0 ? 1u : 0u);
                    mma_f16(tmem + 256u, sw128_desc(smem_u32(sa + a * kATile) + 32 * kk),
                            sw128_desc(smem_u32(sbl + a * kBTile) + 32 * kk), IDESC, 1u);
                }
        }
        mma_commit(bar_done);
    }
    __syncwarp();
    if (!mbar_wait_for(bar_done, 0u, err, kErrDone, wait_ns)) mbar_wait_for(bar_done, 0u, nullptr, 0, kWaitNs);
    tc_fence_after();
    // warp w reads TMEM lanes 32w .. 32w + 31 = rows y0 + 32w + lane; columns = replicas
    const int y = y0 + warp * 32 + lane;
    float* dst = partial + size_t(blockIdx.y) * kRep * npad + y;
    const uint32_t tl = tmem + (uint32_t(warp * 32) << 16);
    uint32_t v[32];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float s01[32], s23[32];
        tmem_ld32(tl + uint32_t(32 * h), v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) s01[e] = __uint_as_float(v[e]);
        tmem_ld32(tl + uint32_t(64 + 32 * h), v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) s01[e] += __uint_as_float(v[e]);
        tmem_ld32(tl + uint32_t(128 + 32 * h), v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) s23[e] = __uint_as_float(v[e]);
        tmem_ld32(tl + uint32_t(192 + 32 * h), v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) s23[e] += __uint_as_float(v[e]);
        tmem_ld32(tl + uint32_t(256 + 32 * h), v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) dst[size_t(32 * h + e) * npad] = (s01[e] + s23[e]) + __uint_as_float(v[e]);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// v = x[0] + x[1] + x[2] + O(2^-24 |v|): three BF16 terms, each rounding the remainder of the previous ones.
__device__ __forceinline__ void split_bf16(float v, __nv_bfloat16* x, size_t plane) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    const float r1 = v - __bfloat162float(h);
    const __nv_bfloat16 m = __float2bfloat16_rn(r1);
    x[0] = h;
    x[plane] = m;
    x[2 * plane] = __float2bfloat16_rn(r1 - __bfloat162float(m));
}

// Deterministic block sum (fixed shuffle tree, then warp 0 over the warp partials); the result is valid in warp 0.
template <int NV>
__device__ __forceinline__ void block_sum(float (&v)[NV], float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[k * 32 + warp] = v[k];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            float x = lane < nw ? red[k * 32 + lane] : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            v[k] = x;
        }
    }
}

// Sum of replica r's per-chunk partials parts[ch][r], in chunk order (deterministic).
__device__ __forceinline__ float sum_parts(const float* __restrict__ parts, int nch, int r) {
    float v = 0.f;
    for (int ch = 0; ch < nch; ++ch) v += parts[ch * kRep + r];
    return v;
}

// Elementwise kernels run on a (replica, 256-column chunk) grid, one element per thread; per-replica sums are
// written per chunk (parts[chunk][replica]) and summed in chunk order by their readers.

// Soft count partials n[ch][r] = sum_{i in chunk, i < n} (1 - m[r,i]^2) and the BF16 terms of m.
__global__ void __launch_bounds__(kElemThreads) mf_prep_kernel(const float* __restrict__ m, int n, int npad,
                                                               float* __restrict__ nout, __nv_bfloat16* __restrict__ x) {
    __shared__ float red[32];
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x, i = blockIdx.y * kElemThreads + threadIdx.x;
    const size_t idx = size_t(r) * npad + i;
    const float v = m[idx];
    split_bf16(v, x + idx, size_t(kRep) * npad);
    float acc[1] = {i < n ? 1.f - v * v : 0.f};
    block_sum(acc, red);
    if (threadIdx.x == 0) nout[blockIdx.y * kRep + r] = acc[0];
}

struct FwdArgs {
    const float* partial;
    int ksplit, npad, n, t;
    const float* bias;
    const float *beta, *q, *u, *w;
    const float* m_cur;
    const float* m_prev;
    const float* n_cur;      // [nch][64] partials of n_t
    float* m_next;
    __nv_bfloat16* x;        // BF16 terms of m_next [3][64][npad]
    float* n_next;           // [nch][64] partials of n_{t+1}
    float* P_out;            // [64][npad] or null
};

__global__ void __launch_bounds__(kElemThreads) mf_fwd_kernel(const FwdArgs a) {
    __shared__ float red[32];
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x, npad = a.npad, nch = gridDim.y, i = blockIdx.y * kElemThreads + threadIdx.x;
    const float beta = a.beta[a.t], q = a.q[a.t];
    const float gamma = a.u[a.t] * sum_parts(a.n_cur, nch, r) + a.w[a.t];
    const size_t idx = size_t(r) * npad + i;
    float H = 0.f;
    for (int ks = 0; ks < a.ksplit; ++ks) H += a.partial[(size_t(ks) * kRep + r) * npad + i];
    const float P = H + a.bias[i] + q * a.m_cur[idx] - gamma * a.m_prev[idx];
    const float mn = i < a.n ? tanhf(beta * P) : 0.f;
    a.m_next[idx] = mn;
    split_bf16(mn, a.x + idx, size_t(kRep) * npad);
    if (a.P_out) a.P_out[idx] = P;
    float acc[1] = {i < a.n ? 1.f - mn * mn : 0.f};
    block_sum(acc, red);
    if (threadIdx.x == 0) a.n_next[blockIdx.y * kRep + r] = acc[0];
}

struct BwdArgs {
    const float* partial;      // J pbar_{t+1} split-K partials, or null when t = S - 1
    int ksplit, npad, n, t, S;
    const float* g_final;      // dL/dm_S (used when t = S - 1)
    const float* pbar_next;    // pbar_{t+1} or null
    const float* pbar_next2;   // pbar_{t+2} or null
    const float* s_next;       // partials of s_{t+1} [nch][64], or null
    const float* n_next2;      // partials of n_{t+2} [nch][64], or null
    const float *beta, *q, *u, *w;
    const float* m_next;       // m_{t+1}
    const float* m_cur;        // m_t
    const float* m_prev;       // m_{t-1}
    const float* P;            // P_t
    const float* n_cur;        // partials of n_t [nch][64]
    float* pbar;               // out: pbar_t
    __nv_bfloat16* x;          // out: BF16 terms of pbar_t [3][64][npad]
    float* s_out;              // out: partials of s_t [nch][64]
    float* gparts;             // out: [S][4][nch][64] partials
};

// One adjoint step t:
//   G      = dL/dm_{t+1} = J pbar_{t+1} + q_{t+1} pbar_{t+1} + 2 u_{t+1} s_{t+1} m_{t+1} - gamma_{t+2} pbar_{t+2}
//            (dL/dm_S given at t = S - 1)
//   abar_t = G (1 - m_{t+1}^2),  pbar_t = beta_t abar_t,  s_t = sum_i pbar_t m_{t-1}
//   dL/dbeta_t += sum abar_t P_t, dL/dq_t += sum pbar_t m_t, dL/du_t += -s_t n_t, dL/dw_t += -s_t
__global__ void __launch_bounds__(kElemThreads) mf_bwd_kernel(const BwdArgs a) {
    __shared__ float red[3 * 32];
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x, npad = a.npad, t = a.t, nch = gridDim.y, ch = blockIdx.y;
    const int i = ch * kElemThreads + threadIdx.x;
    const float beta = a.beta[t];
    const bool last = t == a.S - 1;
    const float q1 = last ? 0.f : a.q[t + 1];
    const float us = last ? 0.f : 2.f * a.u[t + 1] * sum_parts(a.s_next, nch, r);
    const float g2 = a.pbar_next2 ? a.u[t + 2] * sum_parts(a.n_next2, nch, r) + a.w[t + 2] : 0.f;
    const size_t idx = size_t(r) * npad + i;
    float G;
    if (last) {
        G = a.g_final[idx];
    } else {
        float H = 0.f;
        for (int ks = 0; ks < a.ksplit; ++ks) H += a.partial[(size_t(ks) * kRep + r) * npad + i];
        G = H + q1 * a.pbar_next[idx] + us * a.m_next[idx];
        if (a.pbar_next2) G -= g2 * a.pbar_next2[idx];
    }
    const float mn = a.m_next[idx];
    const float abar = i < a.n ? G * (1.f - mn * mn) : 0.f;
    const float pb = beta * abar;
    a.pbar[idx] = pb;
    split_bf16(pb, a.x + idx, size_t(kRep) * npad);
    float acc[3] = {abar * a.P[idx], pb * a.m_cur[idx], pb * a.m_prev[idx]};   // abar P, pbar m_t, pbar m_{t-1}
    block_sum(acc, red);
    if (threadIdx.x == 0) {
        a.s_out[ch * kRep + r] = acc[2];
        float* g = a.gparts + size_t(t) * 4 * nch * kRep;
        g[(0 * nch + ch) * kRep + r] = acc[0];
        g[(1 * nch + ch) * kRep + r] = acc[1];
        g[(2 * nch + ch) * kRep + r] = -acc[2] * sum_parts(a.n_cur, nch, r);
        g[(3 * nch + ch) * kRep + r] = -acc[2];
    }
}

// gsched[t][k][r] = sum over chunks of gparts[t][k][ch][r] (chunk order); one thread per (t, k, r).
__global__ void mf_gsum_kernel(const float* __restrict__ gparts, int S, int nch, float* __restrict__ gsched) {
    pdl_trigger();
    pdl_wait();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= S * 4 * kRep) return;
    const int r = e % kRep, tk = e / kRep;
    float v = 0.f;
    for (int ch = 0; ch < nch; ++ch) v += gparts[(size_t(tk) * nch + ch) * kRep + r];
    gsched[e] = v;
}

// ---------------------------------------------------------------------------------------------- persistent form
// The whole forward pass, or the whole adjoint, in one cooperative launch up to 12 chunks of 256 columns: every CTA keeps its
// tile of J on chip and walks through the steps, where the launch sequences below reload J and pay two launches a step. The
// arithmetic is that of the kernels above, operation for operation and in their order, so the results are bit-identical.
//
// The NR = 64, 32 or 16 replicas of a replica group never meet those of another. Within a group, CTA (MB = 1 or 2 blocks of
// 128 rows, K chunk j) keeps its first block's tile of J in TMEM, so that an MMA reads only its B tile from shared memory, and
// a second block's (from nine chunks on, the two blocks of a chunk) in shared memory. The nch CTAs of the same rows are a
// team: replica k of the group is summed by its member k mod nch, 128 rows to a quarter of its 512 threads. Two kinds of
// counters replace the launch boundaries: a_cnt[team], the team's GEMMs done (its partials may be summed), and b_cnt[chunk],
// the elementwise steps of the chunk's teams done (its BF16 terms may be multiplied). The sizes are compile-time constants.
//
// A soft count needs the sum over a chunk's two row blocks, which with MB = 1 two teams hold: the warps publish their sums of
// 32 rows ([replica][chunk][warp of the chunk]) and each reader applies block_sum's tree over them, bit for bit. Those sums and
// the thread's own values are loaded while the MMAs run.
// Before its MMAs a CTA has seen every chunk's last elementwise step, so partials, terms and sums of the step before that have
// all been read: one buffer of partials and two of terms are enough.
// Bound: the chain of a step, about 11000 cycles at n = 2000: counter 800, terms from L2 1450, MMAs 2200 (the mid and low
// terms' 32 in one chain, 45 cycles each), epilogue and store 1000, release and counter 2500, partials 1000, tanh, terms and
// sums 1000, release 1000. 512 threads with up to 128 registers, because 1024 spilled and left each thread one serial chain.
constexpr int kCntStride = 32;             // counters in lines of their own
constexpr int kErrA = 13, kErrB = 14;

struct PsArgs {
    int n, S;
    const float *bias, *beta, *q, *u, *w;
    float* partial;            // [row block][64][nch][128]
    __nv_bfloat16* xm;         // [2][nch][64][3][256] terms of m: chunk, replica, term, column
    __nv_bfloat16* xp;         // [2][nch][64][3][256] terms of pbar (adjoint)
    float* nbuf;               // [S + 1][64][nch][8] soft counts per warp of 32 rows
    unsigned* cnt;             // per replica group b_cnt[nch], a_cnt[teams] (zeroed)
    int* err;
    uint64_t wait_ns;
    const __nv_bfloat16* J;
    // forward
    const float *m0, *mprev;
    float *ring, *ckpt, *m_out;
    // adjoint
    const float *ckpt_in, *g_m;
    float *seg_m, *seg_P, *pbar;
    float* svec;               // [3][64][nch][8] s_t
    float* gparts;             // [S][3][64][nch][8]
};

__device__ __forceinline__ void mma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void ps_ld(uint32_t taddr, uint32_t (&x)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void ps_ld(uint32_t taddr, uint32_t (&x)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3])
                 : "r"(taddr));
}

constexpr int kTmChunks = 12;     // at most: nch^2 CTAs of two row blocks, one per SM
constexpr int kTmThreads = 512;

// block_sum's tree over the 8 warp sums of a chunk
__device__ __forceinline__ float warps_tree(const float* parts) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(parts)), b = __ldcg(reinterpret_cast<const float4*>(parts) + 1);
    return ((a.x + b.x) + (a.z + b.z)) + ((a.y + b.y) + (a.w + b.w));
}

template <int NCH>
struct TmSplit {
    static constexpr int mb = NCH <= 8 ? 1 : 2;                             // row blocks per CTA
    // replicas per group: as few as one CTA per SM allows
    static constexpr int nr = NCH <= 4 ? 16 : NCH <= 6 ? 32 : 64;
    static constexpr int rp = (nr + NCH - 1) / NCH;                         // replicas that a CTA sums, at most
    static constexpr int grid = 2 / mb * NCH * NCH * (kRep / nr);
    // more than half of an SM's shared memory: each CTA allocates all of its SM's TMEM
    static constexpr size_t need = 1024 + (mb - 1) * 4 * size_t(kATile) + 12 * size_t(nr) * 128 + 64;
    static constexpr size_t smem = need > 120 * 1024 ? need : 120 * 1024;
};

template <int NCH, bool ADJOINT>
__global__ void __launch_bounds__(kTmThreads, 1) mf_tmem_kernel(const __grid_constant__ CUtensorMap mapJ, const __grid_constant__ PsArgs A) {
    using Split = TmSplit<NCH>;
    constexpr int MB = Split::mb, NR = Split::nr, rp = Split::rp, nch = NCH, npad = NCH * kKC;
    constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(NR >> 3) << 17) | (uint32_t(kRows >> 4) << 24);
    constexpr int BT = NR * 128, CW = NR / 4;                   // bytes of a B atom; columns per epilogue warp
    constexpr uint32_t kACol = 320;                             // TMEM columns: 5 x NR accumulators, J from 320
    constexpr int UK = 4 / MB, P = (rp + UK - 1) / UK;          // quarters per 128 rows; replicas per quarter
    constexpr int GL = NCH <= 8 ? 8 : 16;                       // lanes per array in sums()
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ int s_ok;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, unit = tid >> 7, ut = tid & 127;
    const int n = A.n, S = A.S;
    const int j = int(blockIdx.x) % NCH, team = int(blockIdx.x) / NCH % (2 / MB * NCH), rg = int(blockIdx.x) / NCH / (2 / MB * NCH);
    const int c = MB == 1 ? team >> 1 : team;                   // own chunk
    const int half = MB == 1 ? team & 1 : unit & 1;             // of the chunk's rows: this quarter's
    const int row0 = MB == 1 ? team : 2 * team;                 // the CTA's first row block
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sa = smem;                                         // [4] J atoms of a second row block
    uint8_t* sb = sa + (MB - 1) * 4 * kATile;                   // [3 terms][4] operand atoms
    uint64_t* bars = reinterpret_cast<uint64_t*>(sb + 12 * BT);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
    const uint32_t bar_done = smem_u32(bars), bar_j = smem_u32(bars + 1);
    constexpr size_t plane = size_t(kRep) * npad;
    unsigned* const b_cnt = A.cnt + rg * 3 * NCH * kCntStride;  // per replica group: b_cnt[nch], a_cnt[up to 2 nch]
    unsigned* const a_cnt = b_cnt + (NCH + team) * kCntStride;
    constexpr unsigned b_all = unsigned(2 / MB * NCH);          // arrivals per step at a b_cnt

    if (tid == 0) {
        s_ok = 1;
        mbar_init(bar_done, 2);
        mbar_init(bar_j, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot, tlane = tmem + (uint32_t((warp & 3) * 32) << 16);
    {
        // warp w: rows 32 (w % 4) .., BF16 columns 64 (w / 4) .. of the tile, two to a TMEM column
        const uint4* src = reinterpret_cast<const uint4*>(A.J + size_t(row0 * kRows + (warp & 3) * 32 + lane) * npad + j * kKC +
                                                          64 * (warp >> 2));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t v[16];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint4 x = __ldg(src + 4 * h + k);
                v[4 * k] = x.x;
                v[4 * k + 1] = x.y;
                v[4 * k + 2] = x.z;
                v[4 * k + 3] = x.w;
            }
            tmem_st16(tlane + kACol + uint32_t(32 * (warp >> 2) + 16 * h), v);
        }
        tmem_wait_st();
        tc_fence_before();
    }
    if (MB == 2 && tid == 0) {
        mbar_arrive_expect_tx(bar_j, 4 * kATile);
        for (int a = 0; a < 4; ++a) tma_load_2d(smem_u32(sa + a * kATile), &mapJ, j * kKC + 64 * a, (row0 + 1) * kRows, bar_j);
        if (!mbar_wait_for(bar_j, 0u, A.err, kErrFull, A.wait_ns)) {
            mbar_wait_for(bar_j, 0u, nullptr, 0, kWaitNs);
            s_ok = 0;
        }
    }
    unsigned ng = 0, nb = 0;                              // GEMMs and elementwise steps so far
    uint32_t done_ph = 0u;

    // Bounded wait for a counter; after a wait that gave up the CTA waits for nothing more and walks on, so that its peers
    // still see every arrival.
    auto poll = [&](const unsigned* p, unsigned target, int code) {
        if (!*const_cast<volatile int*>(&s_ok)) return;
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= target) return;
        const uint64_t t0 = globaltimer();
        for (uint32_t k = 1;; ++k) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
            if (v >= target) return;
            if (((k & 63u) == 0 || A.wait_ns == 0) && (globaltimer() - t0 >= A.wait_ns || err_set(A.err))) {
                atomicCAS(A.err, 0, code);
                *const_cast<volatile int*>(&s_ok) = 0;
                return;
            }
        }
    };
    auto arrive = [&](unsigned* p) {
        __syncthreads();
        if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
    };
    // This thread's 16-byte pieces of the operand: piece tid % 32 of rows (replicas) tid / 32 + 16 k of each term
    constexpr int PIECES = NR / 16;
    const uint32_t b_dst = smem_u32(sb) + uint32_t((lane >> 3) * BT + warp * 128 + (((lane & 7) ^ (warp & 7)) << 4));
    const size_t b_src = (size_t(j * kRep + rg * NR + warp) * 3) * kKC + lane * 8;
    // partials are [row block][replica][K chunk][128 rows]: where this thread's accumulator columns go, and the sums' first
    float* const part_out = A.partial + (size_t(row0 * kRep + rg * NR + CW * (warp >> 2)) * NCH + j) * kRows + (warp & 3) * 32 + lane;
    const float* const part_in = A.partial + size_t((2 * c + half) * kRep) * (NCH * kRows) + ut;
    // partials of J tile x the three terms x[..][chunk j], of the whole team when it returns; `ahead` runs while the MMAs do
    auto gemm = [&](const __nv_bfloat16* x, auto ahead) {
        if (tid == 0) poll(b_cnt + j * kCntStride, nb * b_all, kErrB);
        __syncthreads();
        const __nv_bfloat16* src = x + b_src;
#pragma unroll
        for (int term = 0; term < 3; ++term) {
#pragma unroll
            for (int k = 0; k < PIECES; ++k)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(b_dst + uint32_t(term * 4 * BT + k * 16 * 128)),
                             "l"(src + (k * 16 * 3 + term) * kKC)
                             : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        // every chunk's step, for the sums that `ahead` reads
        if (warp == 15 && lane < nch) poll(b_cnt + lane * kCntStride, nb * b_all, kErrB);
        const uint32_t ut0 = __shfl_sync(0xffffffffu, tmem, 0);
        const uint64_t da = sw128_desc(smem_u32(sa)), db = sw128_desc(smem_u32(sb));
        auto mma = [&](int mb, uint32_t d, int term, int a, int kk, uint32_t acc) {
            const uint64_t b = db + uint64_t((term * 4 + a) * (BT >> 4) + 2 * kk);
            if (mb == 0)
                mma_f16_ta(ut0 + d, ut0 + kACol + uint32_t(8 * (4 * a + kk)), b, IDESC, acc);
            else
                mma_f16(ut0 + d, da + uint64_t(a * (kATile >> 4) + 2 * kk), b, IDESC, acc);
        };
        auto leading = [&](int mb) {
            if (elect_one()) {
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) mma(mb, uint32_t(NR * a), 0, a, kk, kk != 0 ? 1u : 0u);
                mma_commit(bar_done);
            }
            __syncwarp();
        };
        auto others = [&](int mb) {
            if (elect_one()) {
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        mma(mb, uint32_t(4 * NR), 1, a, kk, (a | kk) != 0 ? 1u : 0u);
                        mma(mb, uint32_t(4 * NR), 2, a, kk, 1u);
                    }
                mma_commit(bar_done);
            }
            __syncwarp();
        };
        // the leading term's products while the other two terms are on their way; one warp issues them, another the others
        asm volatile("cp.async.wait_group 2;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        tc_fence_after();
        if (warp == 0) leading(0);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == 1) others(0);
        ahead();
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
            if (mb) {
                __syncthreads();                          // the accumulators of the first block have been read
                tc_fence_after();
                if (warp == 0) leading(1);
                if (warp == 1) others(1);
            }
            if (!mbar_wait_for(bar_done, done_ph & 1u, A.err, kErrDone, A.wait_ns)) {
                mbar_wait_for(bar_done, done_ph & 1u, nullptr, 0, kWaitNs);
                s_ok = 0;
            }
            ++done_ph;
            tc_fence_after();
            const uint32_t tl = tlane + uint32_t(CW * (warp >> 2));
            constexpr int EW = CW < 8 ? CW : 8;
#pragma unroll
            for (int h = 0; h < CW / EW; ++h) {
                uint32_t v[5][EW];
#pragma unroll
                for (int a = 0; a < 5; ++a) ps_ld(tl + uint32_t(NR * a + EW * h), v[a]);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < EW; ++e) {
                    const float s01 = __uint_as_float(v[0][e]) + __uint_as_float(v[1][e]);
                    const float s23 = __uint_as_float(v[2][e]) + __uint_as_float(v[3][e]);
                    __stcg(part_out + (mb * kRep + EW * h + e) * (NCH * kRows), (s01 + s23) + __uint_as_float(v[4][e]));
                }
            }
            tc_fence_before();
        }
        ++ng;
        arrive(a_cnt);
        if (tid == 0) poll(a_cnt, ng * unsigned(NCH), kErrA);
        __syncthreads();
    };
    // sums of the split-K partials of the last GEMM for this thread's row and replicas, in chunk order
    auto field = [&](const int (&r)[P], float (&H)[P]) {
        float v[P][NCH];
#pragma unroll
        for (int h = 0; h < P; ++h)
#pragma unroll
            for (int ks = 0; ks < NCH; ++ks) v[h][ks] = __ldcg(part_in + (r[h] * NCH + ks) * kRows);
#pragma unroll
        for (int h = 0; h < P; ++h) {
            H[h] = 0.f;
#pragma unroll
            for (int ks = 0; ks < NCH; ++ks) H[h] += v[h][ks];
        }
    };
    const int i = c * kKC + half * kRows + ut;                      // this thread's column of m
    const bool in = i < n;
    const float bias = A.bias[i];
    // This thread's replicas. Where the last of them is none (on[P - 1] false) it repeats the first, to be computed and not
    // stored.
    int r[P];
    bool on[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int k = unit / MB + UK * p;
        on[p] = k < rp && k * NCH + j < NR;
        r[p] = rg * NR + (on[p] ? k : unit / MB) * NCH + j;
    }
    auto terms = [&](float v, __nv_bfloat16* x, int r) {
        split_bf16(v, x + (c * kRep + r) * (3 * kKC) + half * kRows + ut, kKC);
    };
    // a replica's raw sums are [chunk][warp of the chunk]
    const int wslot = c * 8 + half * 4 + (warp & 3);
    auto put = [&](float* base, float (&v)[P]) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int h = 0; h < P; ++h) v[h] += __shfl_xor_sync(0xffffffffu, v[h], o);
#pragma unroll
        for (int h = 0; h < P; ++h)
            if (lane == 0 && on[h]) __stcg(base + r[h] * (8 * NCH) + wslot, v[h]);
    };
    // sums over the chunks, in chunk order, of the arrays that each GL lanes are given
    auto sums = [&](const float* mine, float (&v)[P]) {
        const int ch0 = min(lane & (GL - 1), NCH - 1);
        float tree[P];
#pragma unroll
        for (int h = 0; h < P; ++h) {
            tree[h] = warps_tree(mine + (r[h] * NCH + ch0) * 8);
            v[h] = 0.f;
        }
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch)
#pragma unroll
            for (int h = 0; h < P; ++h) v[h] += __shfl_sync(0xffffffffu, tree[h], (lane & ~(GL - 1)) + ch);
    };
    constexpr size_t xbuf = 3 * plane, sstep = size_t(kRep) * 8 * NCH;
    // the BF16 terms and the soft count sums of m_t (mf_prep_kernel), from `m`
    auto prep = [&](const float* m, int t, __nv_bfloat16* x) {
        {
            float acc[P];
#pragma unroll
            for (int h = 0; h < P; ++h) {
                const float v = m[r[h] * npad + i];
                if (on[h]) terms(v, x, r[h]);
                acc[h] = in ? fmaf(-v, v, 1.f) : 0.f;
            }
            put(A.nbuf + size_t(t) * sstep, acc);
        }
        ++nb;
        arrive(b_cnt + c * kCntStride);
    };
    auto copy2 = [&](const float* a, const float* b, float* x, float* y) {
        {
#pragma unroll
            for (int h = 0; h < P; ++h)
                if (on[h]) {
                    x[r[h] * npad + i] = a[r[h] * npad + i];
                    y[r[h] * npad + i] = b[r[h] * npad + i];
                }
        }
    };
    // one forward step t (mf_fwd_kernel): m_{t+1} into m_next, its terms into x, P_t into P_out when that is not null
    auto forward = [&](int t, const __nv_bfloat16* xin, const float* m_cur, const float* m_prev, float* m_next, float* also,
                       __nv_bfloat16* x, float* P_out) {
        const float beta = __ldg(A.beta + t), q = __ldg(A.q + t), u = __ldg(A.u + t), w = __ldg(A.w + t);
        float ns[P], mc[P], mp[P];
        gemm(xin, [&]() {
            {
#pragma unroll
                for (int h = 0; h < P; ++h) {
                    mc[h] = m_cur[r[h] * npad + i];
                    mp[h] = m_prev[r[h] * npad + i];
                }
                sums(A.nbuf + size_t(t) * sstep, ns);
            }
        });
        {
            float H[P], mn[P], Pv[P], acc[P];
            field(r, H);
#pragma unroll
            for (int h = 0; h < P; ++h) {
                const float gamma = fmaf(u, ns[h], w);
                Pv[h] = fmaf(-gamma, mp[h], fmaf(q, mc[h], H[h] + bias));
                mn[h] = in ? tanhf(beta * Pv[h]) : 0.f;
            }
#pragma unroll
            for (int h = 0; h < P; ++h) {
                const int idx = r[h] * npad + i;
                if (on[h]) {
                    terms(mn[h], x, r[h]);
                    m_next[idx] = mn[h];
                    if (also) also[idx] = mn[h];
                    if (P_out) P_out[idx] = Pv[h];
                }
                acc[h] = in ? fmaf(-mn[h], mn[h], 1.f) : 0.f;
            }
            put(A.nbuf + size_t(t + 1) * sstep, acc);
        }
        ++nb;
        arrive(b_cnt + c * kCntStride);
    };
    __syncthreads();
    tc_fence_after();

    if constexpr (!ADJOINT) {
        // m_t in ring slot (t + 1) % 3, touched by its owner threads only; checkpoints of (m_{t-1}, m_t) every 16 steps
        copy2(A.mprev, A.m0, A.ring, A.ring + plane);
        prep(A.m0, 0, A.xm);
        for (int t = 0; t < S; ++t) {
            const float *prev = A.ring + size_t(t % 3) * plane, *cur = A.ring + size_t((t + 1) % 3) * plane;
            if (t % kMfCheckpoint == 0) {
                float* ck = A.ckpt + size_t(t / kMfCheckpoint) * 2 * plane;
                copy2(prev, cur, ck, ck + plane);
            }
            forward(t, A.xm + size_t(t & 1) * xbuf, cur, prev, A.ring + size_t((t + 2) % 3) * plane,
                    t == S - 1 ? A.m_out : nullptr, A.xm + size_t((t + 1) & 1) * xbuf, nullptr);
        }
    } else {
        unsigned pbn = 0;                                 // adjoint steps so far: the buffer of their terms
        for (int seg = (S + kMfCheckpoint - 1) / kMfCheckpoint - 1; seg >= 0; --seg) {
            const int t0 = seg * kMfCheckpoint, t1 = min(S, t0 + kMfCheckpoint);
            // seg_m slot k holds m_{t0 - 1 + k}
            const float* ck = A.ckpt_in + size_t(seg) * 2 * plane;
            copy2(ck, ck + plane, A.seg_m, A.seg_m + plane);
            prep(ck + plane, t0, A.xm);
            for (int t = t0; t < t1; ++t) {
                const int s = t - t0;
                forward(t, A.xm + size_t(s & 1) * xbuf, A.seg_m + size_t(s + 1) * plane, A.seg_m + size_t(s) * plane,
                        A.seg_m + size_t(s + 2) * plane, nullptr, A.xm + size_t((s + 1) & 1) * xbuf, A.seg_P + size_t(s) * plane);
            }
            for (int t = t1 - 1; t >= t0; --t) {
                const int s = t - t0;
                const bool last = t == S - 1, far = t + 2 < S;
                // one adjoint step (mf_bwd_kernel)
                const float beta = __ldg(A.beta + t), q1 = last ? 0.f : __ldg(A.q + t + 1), u1 = last ? 0.f : __ldg(A.u + t + 1);
                const float u2 = far ? __ldg(A.u + t + 2) : 0.f, w2 = far ? __ldg(A.w + t + 2) : 0.f;
                float s1[P], n2[P], mn[P], p1[P], p2[P], Pt[P], mc[P], mp[P];
                auto ahead = [&]() {
                    {
#pragma unroll
                        for (int h = 0; h < P; ++h) {
                            const int idx = r[h] * npad + i;
                            mn[h] = A.seg_m[size_t(s + 2) * plane + idx];
                            mc[h] = A.seg_m[size_t(s + 1) * plane + idx];
                            mp[h] = A.seg_m[size_t(s) * plane + idx];
                            Pt[h] = A.seg_P[size_t(s) * plane + idx];
                            p1[h] = last ? A.g_m[idx] : A.pbar[size_t((t + 1) % 3) * plane + idx];
                            p2[h] = far ? A.pbar[size_t((t + 2) % 3) * plane + idx] : 0.f;
                        }
                        float v[P];
                        // lanes 0 .. GL - 1: s_{t+1}, the others: n_{t+2}; at the last steps other values, which are not used
                        sums(lane < GL ? A.svec + size_t((t + 1) % 3) * sstep : A.nbuf + size_t(far ? t + 2 : t) * sstep, v);
#pragma unroll
                        for (int h = 0; h < P; ++h) {
                            s1[h] = __shfl_sync(0xffffffffu, v[h], 0);
                            n2[h] = __shfl_sync(0xffffffffu, v[h], GL);
                        }
                    }
                };
                if (last)
                    ahead();
                else
                    gemm(A.xp + size_t((pbn - 1u) & 1u) * xbuf, ahead);
                {
                    float H[P], a0[P], a1[P], a2[P];
                    if (!last) field(r, H);
#pragma unroll
                    for (int h = 0; h < P; ++h) {
                        const float us = last ? 0.f : 2.f * u1 * s1[h];
                        const float g2 = far ? fmaf(u2, n2[h], w2) : 0.f;
                        const int idx = r[h] * npad + i;
                        float G = p1[h];                  // dL/dm_S at the last step
                        if (!last) {
                            G = fmaf(us, mn[h], fmaf(q1, p1[h], H[h]));
                            if (far) G = fmaf(-g2, p2[h], G);
                        }
                        const float abar = in ? G * fmaf(-mn[h], mn[h], 1.f) : 0.f;
                        const float pb = beta * abar;
                        if (on[h]) {
                            terms(pb, A.xp + size_t(pbn & 1u) * xbuf, r[h]);
                            A.pbar[size_t(t % 3) * plane + idx] = pb;
                        }
                        a0[h] = __fmul_rn(abar, Pt[h]);
                        a1[h] = __fmul_rn(pb, mc[h]);
                        a2[h] = __fmul_rn(pb, mp[h]);
                    }
                    float* g = A.gparts + size_t(t) * 3 * sstep;
                    put(g, a0);
                    put(g + sstep, a1);
                    put(A.svec + size_t(t % 3) * sstep, a2);
#pragma unroll
                    for (int h = 0; h < P; ++h)
                        if (lane == 0 && on[h]) __stcg(g + 2 * sstep + r[h] * (8 * NCH) + wslot, a2[h]);
                }
                ++pbn;
                ++nb;
                arrive(b_cnt + c * kCntStride);
            }
            if (t1 - t0 == 1 && seg > 0) {
                // a last segment of one step had no GEMM behind its forward step: its terms may still be read
                if (tid < NCH) poll(b_cnt + tid * kCntStride, nb * b_all, kErrB);
                __syncthreads();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// J as int8 [n][n] -> its transpose in BF16, padded with zeros to [npad][npad].
__global__ void mf_pack_kernel(const int8_t* __restrict__ J, int n, int npad, __nv_bfloat16* __restrict__ out) {
    __shared__ int8_t tile[32][33];
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, tx = threadIdx.x;
    for (int i = threadIdx.y; i < 32; i += 8)
        tile[i][tx] = x0 + i < n && y0 + tx < n ? J[size_t(x0 + i) * n + y0 + tx] : int8_t(0);
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += 8) out[size_t(y0 + i) * npad + x0 + tx] = __float2bfloat16(float(tile[tx][i]));
}

// The schedule gradients from mf_tmem_kernel's warp sums, one warp per (step, replica): the halves of the warp hold the chunks
// of s_t and n_t, then those of sum abar P and sum pbar m_t; the same sums as mf_bwd_kernel's and mf_gsum_kernel's.
__global__ void mf_gsum_raw_kernel(const float* __restrict__ gparts, const float* __restrict__ nbuf, int S, int nch, float* __restrict__ gsched) {
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, hi = lane >> 4;
    if (e >= S * kRep) return;
    const int r = e % kRep, t = e / kRep, ch0 = min(lane & 15, nch - 1);
    const size_t sstep = size_t(kRep) * 8 * nch, at = size_t(r * nch + ch0) * 8;
    const float tree = warps_tree((hi ? nbuf + size_t(t) * sstep : gparts + (size_t(t) * 3 + 2) * sstep) + at);
    const float prod = warps_tree(gparts + (size_t(t) * 3 + hi) * sstep + at);
    float n = 0.f, v = 0.f, g2 = 0.f, g3 = 0.f;
    for (int ch = 0; ch < nch; ++ch) {
        n += __shfl_sync(0xffffffffu, tree, 16 + ch);
        v += __shfl_sync(0xffffffffu, prod, (lane & 16) + ch);
    }
    for (int ch = 0; ch < nch; ++ch) {
        const float s = __shfl_sync(0xffffffffu, tree, ch);
        g2 = __fadd_rn(g2, __fmul_rn(-s, n));
        g3 += -s;
    }
    float* const out = gsched + size_t(t) * 4 * kRep + r;
    if ((lane & 15) == 0) {
        out[hi * kRep] = v;
        out[(2 + hi) * kRep] = hi ? g3 : g2;
    }
}

bool check(cudaError_t e, const char* what, std::string* why) {
    if (e == cudaSuccess) return true;
    if (why) *why = std::string(what) + ": " + cudaGetErrorString(e);
    return false;
}

// Launch with programmatic stream serialization (see pdl_trigger / pdl_wait): the kernel may start while the previous
// kernel in the stream still runs, and waits for it where it reads that kernel's outputs.
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

int gemm(MfContext* c, const CUtensorMap (&mx)[3], cudaStream_t st, std::string* why) {
    const cudaError_t e = launch_pdl(mf_gemm_kernel, dim3(c->npad / kRows, c->npad / kKC), dim3(kGemmThreads),
                                     gemm_smem(), st, c->mapJ, mx[0], mx[1], mx[2], c->partial, c->npad, c->err,
                                     c->wait_ns);
    return check(e, "mean-field GEMM launch", why) ? 0 : -2;
}

float* mslot(float* base, int k, int npad) { return base + size_t(k) * kRep * npad; }

// 256-column chunks of the elementwise grid.
int nch(const MfContext* c) { return c->npad / kElemThreads; }

// Forward steps t = t0 .. t1 - 1: m_t = cur(t), m_{t-1} = prev(t); writes m_{t+1} to next(t) and P_t to pout(t)
// when that is not null. The BF16 terms of m_t must already be in c->xm.
template <class CurFn, class PrevFn, class NextFn, class PFn>
int run_steps(MfContext* c, int t0, int t1, const float* beta, const float* q, const float* u, const float* w,
              CurFn cur, PrevFn prev, NextFn next, PFn pout, cudaStream_t st, std::string* why) {
    const int npad = c->npad;
    for (int t = t0; t < t1; ++t) {
        int rc = gemm(c, c->mapXm, st, why);
        if (rc) return rc;
        FwdArgs a{};
        a.partial = c->partial;
        a.ksplit = npad / kKC;
        a.npad = npad;
        a.n = c->n;
        a.t = t;
        a.bias = c->bias;
        a.beta = beta;
        a.q = q;
        a.u = u;
        a.w = w;
        a.m_cur = cur(t);
        a.m_prev = prev(t);
        a.n_cur = c->nbuf + size_t(t) * nch(c) * kRep;
        a.m_next = next(t);
        a.x = c->xm;
        a.n_next = c->nbuf + size_t(t + 1) * nch(c) * kRep;
        a.P_out = pout(t);
        if (!check(launch_pdl(mf_fwd_kernel, dim3(kRep, nch(c)), dim3(kElemThreads), 0, st, a), "mean-field forward step",
                   why))
            return -2;
    }
    return 0;
}

using PsKernel = void (*)(const CUtensorMap, const PsArgs);
struct PsForm {
    int grid;
    size_t smem;
    PsKernel fwd, adj;
};
template <int NCH>
constexpr PsForm tm_form() {
    return {TmSplit<NCH>::grid, TmSplit<NCH>::smem, mf_tmem_kernel<NCH, false>, mf_tmem_kernel<NCH, true>};
}
const PsForm kPsForms[kTmChunks] = {tm_form<1>(), tm_form<2>(), tm_form<3>(), tm_form<4>(),  tm_form<5>(),  tm_form<6>(),
                                    tm_form<7>(), tm_form<8>(), tm_form<9>(), tm_form<10>(), tm_form<11>(), tm_form<12>()};

size_t ps_cnt_bytes(int nch) { return size_t(12 * nch + 1) * kCntStride * sizeof(unsigned); }

// The persistent form for npad columns, or null (the launch sequences) beyond twelve chunks or where its CTAs do not all fit,
// one per SM. Measured, a forward / an adjoint step in us, launch sequences -> persistent: n = 200 8.4 / 15.2 -> 5.8 / 11.2,
// n = 700 10.0 / 18.7 -> 5.8 / 10.4, n = 2000 9.3 / 19.4 -> 6.0 / 12.4, n = 2500 15.8 / 30.9 -> 10.8 / 20.9, n = 3072
// 16.8 / 32.7 -> 10.6 / 20.4. With one or two tiles of J per CTA more chunks do not fit one CTA per SM; three would fit 13 and
// 14 chunks and are not compiled.
const PsForm* ps_form(int npad) {
    const int nch = npad / kKC;
    int dev = 0, sms = 0, coop = 0, optin = 0;
    if (nch > kTmChunks || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
        return nullptr;
    // the launch bounds leave each CTA the registers of its SM; 1 KB for the kernels' static shared memory
    const PsForm& f = kPsForms[nch - 1];
    return f.grid <= sms && f.smem + 1024 <= size_t(optin) ? &f : nullptr;
}

PsArgs ps_args(MfContext* c, int S, const float* beta, const float* q, const float* u, const float* w) {
    PsArgs a{};
    a.n = c->n;
    a.S = S;
    a.J = c->J;
    a.bias = c->bias;
    a.beta = beta;
    a.q = q;
    a.u = u;
    a.w = w;
    a.partial = c->partial;
    a.xm = c->xm;
    a.xp = c->xp;
    a.nbuf = c->nbuf;
    a.cnt = c->cnt;
    a.err = c->err;
    a.wait_ns = c->wait_ns;
    return a;
}

// Soft counts and gradient sums for S steps of a launch on st, in one block.
int ensure_steps(MfContext* c, int S, cudaStream_t st, std::string* why) {
    const int cap = std::max(S, c->nbuf_steps);
    const size_t nbytes = size_t(cap + 1) * (c->form ? 8 : 1) * nch(c) * kRep * sizeof(float);
    const size_t gbytes = size_t(cap) * (c->form ? 24 : 4) * nch(c) * kRep * sizeof(float);
    const cudaError_t e = c->steps.ensure(nbytes + gbytes, st);
    if (e != cudaSuccess) {
        if (!c->steps.p) c->nbuf_steps = 0;
        setup_code(e);
        return check(e, "cudaMalloc", why) ? 0 : -2;
    }
    c->nbuf = reinterpret_cast<float*>(c->steps.p);
    c->gparts = reinterpret_cast<float*>(c->steps.p + nbytes);
    c->nbuf_steps = cap;
    return 0;
}

int ps_launch(MfContext* c, PsKernel kernel, PsArgs& a, cudaStream_t st, std::string* why) {
    void* args[] = {&c->mapJ, &a};
    // a size's kernel is loaded by a context's first launch of it, not with every context (3 ms each)
    bool& loaded = c->loaded[kernel == c->form->adj];
    if (!loaded && !check(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(c->form->smem)),
                          "kernel attributes", why))
        return -2;
    loaded = true;
    if (!check(cudaMemsetAsync(c->cnt, 0, ps_cnt_bytes(nch(c)), st), "clear counters", why) ||
        !check(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(c->form->grid), dim3(kTmThreads),
                                           args, c->form->smem, st),
               "mean-field steps launch", why))
        return -2;
    return 0;
}

}  // namespace

int mf_npad(const MfContext* c) { return c->npad; }

int mf_create(const int8_t* J, const int32_t* bias, int n, MfContext** out, std::string* why) {
    if (!J || n < 1 || !out) {
        if (why) *why = "J, n >= 1 and an output handle are required";
        return -1;
    }
    auto* c = new MfContext();
    c->n = n;
    c->npad = ((n + 255) / 256) * 256;
    const int npad = c->npad;
    std::vector<float> bh(npad, 0.f);
    if (bias)
        for (int i = 0; i < n; ++i) bh[i] = float(bias[i]);
    const size_t plane = size_t(kRep) * npad;
    c->form = ps_form(npad);
    const size_t nbuf = c->form ? 2 : 1, kch = npad / kKC;
    const size_t pbytes = kch * plane * sizeof(float);
    const size_t sbytes = 3 * (c->form ? 8 : 1) * kch * kRep * sizeof(float);
    bool ok = check(cudaMalloc(&c->J, size_t(npad) * npad * sizeof(__nv_bfloat16)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->bias, npad * sizeof(float)), "cudaMalloc", why) &&
              check(cudaMemcpy(c->bias, bh.data(), npad * sizeof(float), cudaMemcpyHostToDevice), "upload bias", why) &&
              check(cudaMalloc(&c->partial, pbytes), "cudaMalloc", why) &&
              check(cudaMalloc(&c->mring, 3 * plane * sizeof(float)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->xm, nbuf * 3 * plane * sizeof(__nv_bfloat16)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->xp, nbuf * 3 * plane * sizeof(__nv_bfloat16)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->seg_m, (kMfCheckpoint + 2) * plane * sizeof(float)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->seg_P, kMfCheckpoint * plane * sizeof(float)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->pbar, 3 * plane * sizeof(float)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->svec, sbytes), "cudaMalloc", why) &&
              check(cudaMalloc(&c->cnt, ps_cnt_bytes(kch)), "cudaMalloc", why) &&
              check(cudaMalloc(&c->err, sizeof(int)), "cudaMalloc", why) &&
              check(cudaMemset(c->err, 0, sizeof(int)), "cudaMemset", why);
    // J goes up as it is, into `partial` (npad^2 bytes), and is padded and transposed there
    int8_t* raw = reinterpret_cast<int8_t*>(c->partial);
    ok = ok && check(cudaMemcpy(raw, J, size_t(n) * n, cudaMemcpyHostToDevice), "upload J", why);
    if (ok) {
        mf_pack_kernel<<<dim3(npad / 32, npad / 32), dim3(32, 8)>>>(raw, n, npad, c->J);
        ok = check(cudaGetLastError(), "pack J", why) && check(cudaStreamSynchronize(nullptr), "pack J", why);
    }
    if (ok) {
        ok = make_map_2d(&c->mapJ, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c->J, npad, npad, 64, kRows);
        for (int k = 0; k < 3 && ok; ++k)
            ok = make_map_2d(&c->mapXm[k], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c->xm + k * plane, npad, kRep, 64, kRep) &&
                 make_map_2d(&c->mapXp[k], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c->xp + k * plane, npad, kRep, 64, kRep);
        if (!ok && why) *why = "cuTensorMapEncodeTiled failed";
    }
    if (ok && !c->form)
        ok = check(cudaFuncSetAttribute(mf_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemm_smem())),
                   "GEMM attributes", why) &&
             check(cudaStreamCreateWithFlags(&c->cap, cudaStreamNonBlocking), "capture stream", why);
    if (!ok) {
        mf_destroy(c);
        return -2;
    }
    *out = c;
    return 0;
}

namespace {

// The forward launch sequence on explicit buffers (recorded into the forward graph).
int forward_body(MfContext* c, int S, const float* beta, const float* q, const float* u, const float* w,
                 const float* m0, const float* mprev, float* ckpt, float* m_out, cudaStream_t st, std::string* why) {
    int rc = 0;
    const int npad = c->npad;
    const size_t plane = size_t(kRep) * npad;
    float* ring = c->mring;
    if (!check(cudaMemcpyAsync(mslot(ring, 0, npad), mprev, plane * 4, cudaMemcpyDeviceToDevice, st), "copy", why) ||
        !check(cudaMemcpyAsync(mslot(ring, 1, npad), m0, plane * 4, cudaMemcpyDeviceToDevice, st), "copy", why))
        return -2;
    mf_prep_kernel<<<dim3(kRep, nch(c)), kElemThreads, 0, st>>>(mslot(ring, 1, npad), c->n, npad, c->nbuf, c->xm);
    if (!check(cudaGetLastError(), "mean-field prep", why)) return -2;
    // m_t lives in ring slot (t + 1) % 3, m_{t-1} in slot t % 3
    for (int t0 = 0; t0 < S; t0 += kMfCheckpoint) {
        float* ck = ckpt + size_t(t0 / kMfCheckpoint) * 2 * plane;
        if (!check(cudaMemcpyAsync(ck, mslot(ring, t0 % 3, npad), plane * 4, cudaMemcpyDeviceToDevice, st), "ckpt",
                   why) ||
            !check(cudaMemcpyAsync(ck + plane, mslot(ring, (t0 + 1) % 3, npad), plane * 4, cudaMemcpyDeviceToDevice, st),
                   "ckpt", why))
            return -2;
        const int t1 = std::min(S, t0 + kMfCheckpoint);
        rc = run_steps(
            c, t0, t1, beta, q, u, w, [&](int t) { return mslot(ring, (t + 1) % 3, npad); },
            [&](int t) { return mslot(ring, t % 3, npad); }, [&](int t) { return mslot(ring, (t + 2) % 3, npad); },
            [](int) { return static_cast<float*>(nullptr); }, st, why);
        if (rc) return rc;
    }
    if (!check(cudaMemcpyAsync(m_out, mslot(ring, (S + 1) % 3, npad), plane * 4, cudaMemcpyDeviceToDevice, st), "copy",
               why))
        return -2;
    return 0;
}

// The adjoint launch sequence on explicit buffers (recorded into the adjoint graph).
int backward_body(MfContext* c, int S, const float* beta, const float* q, const float* u, const float* w,
                  const float* ckpt, const float* g_m, float* gsched, cudaStream_t st, std::string* why) {
    int rc = 0;
    const int npad = c->npad;
    const size_t plane = size_t(kRep) * npad;
    const int nseg = (S + kMfCheckpoint - 1) / kMfCheckpoint;
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int t0 = seg * kMfCheckpoint, t1 = std::min(S, t0 + kMfCheckpoint);
        // segment buffer slot k holds m_{t0 - 1 + k}
        const float* ck = ckpt + size_t(seg) * 2 * plane;
        if (!check(cudaMemcpyAsync(mslot(c->seg_m, 0, npad), ck, 2 * plane * 4, cudaMemcpyDeviceToDevice, st), "copy",
                   why))
            return -2;
        mf_prep_kernel<<<dim3(kRep, nch(c)), kElemThreads, 0, st>>>(mslot(c->seg_m, 1, npad), c->n, npad,
                                                                   c->nbuf + size_t(t0) * nch(c) * kRep, c->xm);
        if (!check(cudaGetLastError(), "mean-field prep", why)) return -2;
        rc = run_steps(
            c, t0, t1, beta, q, u, w, [&](int t) { return mslot(c->seg_m, t - t0 + 1, npad); },
            [&](int t) { return mslot(c->seg_m, t - t0, npad); },
            [&](int t) { return mslot(c->seg_m, t - t0 + 2, npad); },
            [&](int t) { return mslot(c->seg_P, t - t0, npad); }, st, why);
        if (rc) return rc;
        for (int t = t1 - 1; t >= t0; --t) {
            const bool last = t == S - 1;
            if (!last) {
                rc = gemm(c, c->mapXp, st, why);
                if (rc) return rc;
            }
            BwdArgs a{};
            a.partial = last ? nullptr : c->partial;
            a.ksplit = npad / kKC;
            a.npad = npad;
            a.n = c->n;
            a.t = t;
            a.S = S;
            a.g_final = g_m;
            a.pbar_next = last ? nullptr : mslot(c->pbar, (t + 1) % 3, npad);
            a.pbar_next2 = t + 2 < S ? mslot(c->pbar, (t + 2) % 3, npad) : nullptr;
            a.s_next = last ? nullptr : c->svec + size_t((t + 1) % 3) * nch(c) * kRep;
            a.n_next2 = t + 2 < S ? c->nbuf + size_t(t + 2) * nch(c) * kRep : nullptr;
            a.beta = beta;
            a.q = q;
            a.u = u;
            a.w = w;
            a.m_next = mslot(c->seg_m, t - t0 + 2, npad);
            a.m_cur = mslot(c->seg_m, t - t0 + 1, npad);
            a.m_prev = mslot(c->seg_m, t - t0, npad);
            a.P = mslot(c->seg_P, t - t0, npad);
            a.n_cur = c->nbuf + size_t(t) * nch(c) * kRep;
            a.pbar = mslot(c->pbar, t % 3, npad);
            a.x = c->xp;
            a.s_out = c->svec + size_t(t % 3) * nch(c) * kRep;
            a.gparts = c->gparts;
            if (!check(launch_pdl(mf_bwd_kernel, dim3(kRep, nch(c)), dim3(kElemThreads), 0, st, a),
                       "mean-field adjoint step", why))
                return -2;
        }
    }
    const int ne = S * 4 * kRep;
    mf_gsum_kernel<<<(ne + 255) / 256, 256, 0, st>>>(c->gparts, S, nch(c), gsched);
    if (!check(cudaGetLastError(), "mean-field gradient sum", why)) return -2;
    return 0;
}

// Internal buffers for S steps (allocated outside any capture; graphs recorded on older buffers are dropped).
int ensure_io(MfContext* c, int S, cudaStream_t st, std::string* why) {
    int rc = ensure_steps(c, S, st, why);
    if (rc) return rc;
    if (S <= c->io_steps) return 0;
    for (float** p : {&c->sched_i, &c->m0_i, &c->mprev_i, &c->mout_i, &c->gm_i, &c->ckpt_i, &c->gs_i}) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    for (cudaGraphExec_t* g : {&c->fwd_exec, &c->bwd_exec}) {
        if (*g) cudaGraphExecDestroy(*g);
        *g = nullptr;
    }
    c->fwd_S = c->bwd_S = c->io_steps = 0;
    const size_t plane = size_t(kRep) * c->npad;
    const size_t nseg = (S + kMfCheckpoint - 1) / kMfCheckpoint;
    const bool ok = check(cudaMalloc(&c->sched_i, 4 * size_t(S) * 4), "cudaMalloc", why) &&
                    check(cudaMalloc(&c->m0_i, plane * 4), "cudaMalloc", why) &&
                    check(cudaMalloc(&c->mprev_i, plane * 4), "cudaMalloc", why) &&
                    check(cudaMalloc(&c->mout_i, plane * 4), "cudaMalloc", why) &&
                    check(cudaMalloc(&c->gm_i, plane * 4), "cudaMalloc", why) &&
                    check(cudaMalloc(&c->ckpt_i, nseg * 2 * plane * 4), "cudaMalloc", why) &&
                    check(cudaMalloc(&c->gs_i, size_t(S) * 4 * kRep * 4), "cudaMalloc", why);
    if (!ok) return -2;
    c->io_steps = S;
    return 0;
}

// Copy the four schedule vectors into sched_i rows [4][S].
bool copy_sched(MfContext* c, int S, const float* beta, const float* q, const float* u, const float* w, cudaStream_t st,
                std::string* why) {
    const float* v[4] = {beta, q, u, w};
    for (int k = 0; k < 4; ++k)
        if (!check(cudaMemcpyAsync(c->sched_i + size_t(k) * S, v[k], size_t(S) * 4, cudaMemcpyDeviceToDevice, st),
                   "copy schedule", why))
            return false;
    return true;
}

// Record body(cap stream) into *exec once per step count.
template <class Body>
int ensure_graph(MfContext* c, cudaGraphExec_t* exec, int* exec_S, int S, Body body, std::string* why) {
    if (*exec && *exec_S == S) return 0;
    if (*exec) cudaGraphExecDestroy(*exec);
    *exec = nullptr;
    cudaGraph_t g = nullptr;
    if (!check(cudaStreamBeginCapture(c->cap, cudaStreamCaptureModeThreadLocal), "begin capture", why)) return -2;
    const int rc = body(c->cap);
    const cudaError_t e = cudaStreamEndCapture(c->cap, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (!check(e, "end capture", why)) return -2;
    const cudaError_t ei = cudaGraphInstantiate(exec, g, 0);
    cudaGraphDestroy(g);
    if (!check(ei, "instantiate graph", why)) return -2;
    *exec_S = S;
    return 0;
}

}  // namespace

int mf_forward(MfContext* c, int S, const float* beta, const float* q, const float* u, const float* w, const float* m0,
               const float* mprev, float* ckpt, float* m_out, cudaStream_t st, std::string* why) {
    if (!c || S < 1 || !beta || !q || !u || !w || !m0 || !mprev || !ckpt || !m_out) {
        if (why) *why = "invalid mean-field forward arguments";
        return -1;
    }
    if (c->form) {
        int rc = ensure_steps(c, S, st, why);
        if (rc) return rc;
        PsArgs a = ps_args(c, S, beta, q, u, w);
        a.m0 = m0;
        a.mprev = mprev;
        a.ring = c->mring;
        a.ckpt = ckpt;
        a.m_out = m_out;
        return ps_launch(c, c->form->fwd, a, st, why);
    }
    int rc = ensure_io(c, S, st, why);
    if (rc) return rc;
    const size_t plane = size_t(kRep) * c->npad, nseg = (S + kMfCheckpoint - 1) / kMfCheckpoint;
    rc = ensure_graph(c, &c->fwd_exec, &c->fwd_S, S, [&](cudaStream_t cs) {
        const float* sb = c->sched_i;
        return forward_body(c, S, sb, sb + S, sb + 2 * size_t(S), sb + 3 * size_t(S), c->m0_i, c->mprev_i, c->ckpt_i,
                            c->mout_i, cs, why);
    }, why);
    if (rc) return rc;
    if (!copy_sched(c, S, beta, q, u, w, st, why) ||
        !check(cudaMemcpyAsync(c->m0_i, m0, plane * 4, cudaMemcpyDeviceToDevice, st), "copy m0", why) ||
        !check(cudaMemcpyAsync(c->mprev_i, mprev, plane * 4, cudaMemcpyDeviceToDevice, st), "copy mprev", why) ||
        !check(cudaGraphLaunch(c->fwd_exec, st), "forward graph launch", why) ||
        !check(cudaMemcpyAsync(ckpt, c->ckpt_i, nseg * 2 * plane * 4, cudaMemcpyDeviceToDevice, st), "copy ckpt", why) ||
        !check(cudaMemcpyAsync(m_out, c->mout_i, plane * 4, cudaMemcpyDeviceToDevice, st), "copy m_S", why))
        return -2;
    return 0;
}

int mf_backward(MfContext* c, int S, const float* beta, const float* q, const float* u, const float* w,
                const float* ckpt, const float* g_m, float* gsched, cudaStream_t st, std::string* why) {
    if (!c || S < 1 || !beta || !q || !u || !w || !ckpt || !g_m || !gsched) {
        if (why) *why = "invalid mean-field backward arguments";
        return -1;
    }
    if (c->form) {
        int rc = ensure_steps(c, S, st, why);
        if (rc) return rc;
        PsArgs a = ps_args(c, S, beta, q, u, w);
        a.ckpt_in = ckpt;
        a.g_m = g_m;
        a.seg_m = c->seg_m;
        a.seg_P = c->seg_P;
        a.pbar = c->pbar;
        a.svec = c->svec;
        a.gparts = c->gparts;
        rc = ps_launch(c, c->form->adj, a, st, why);
        if (rc) return rc;
        mf_gsum_raw_kernel<<<(S * kRep + 7) / 8, 256, 0, st>>>(c->gparts, c->nbuf, S, nch(c), gsched);
        return check(cudaGetLastError(), "mean-field gradient sum", why) ? 0 : -2;
    }
    int rc = ensure_io(c, S, st, why);
    if (rc) return rc;
    const size_t plane = size_t(kRep) * c->npad, nseg = (S + kMfCheckpoint - 1) / kMfCheckpoint;
    rc = ensure_graph(c, &c->bwd_exec, &c->bwd_S, S, [&](cudaStream_t cs) {
        const float* sb = c->sched_i;
        return backward_body(c, S, sb, sb + S, sb + 2 * size_t(S), sb + 3 * size_t(S), c->ckpt_i, c->gm_i, c->gs_i, cs,
                             why);
    }, why);
    if (rc) return rc;
    if (!copy_sched(c, S, beta, q, u, w, st, why) ||
        !check(cudaMemcpyAsync(c->ckpt_i, ckpt, nseg * 2 * plane * 4, cudaMemcpyDeviceToDevice, st), "copy ckpt", why) ||
        !check(cudaMemcpyAsync(c->gm_i, g_m, plane * 4, cudaMemcpyDeviceToDevice, st), "copy dL/dm", why) ||
        !check(cudaGraphLaunch(c->bwd_exec, st), "adjoint graph launch", why) ||
        !check(cudaMemcpyAsync(gsched, c->gs_i, size_t(S) * 4 * kRep * 4, cudaMemcpyDeviceToDevice, st), "copy grads",
               why))
        return -2;
    return 0;
}

int mf_set_wait_ns(MfContext* c, uint64_t ns) {
    if (!c) return -1;
    if (ns == c->wait_ns) return 0;
    c->wait_ns = ns;
    for (cudaGraphExec_t* g : {&c->fwd_exec, &c->bwd_exec}) {   // the limit is a kernel argument: record again
        if (*g) cudaGraphExecDestroy(*g);
        *g = nullptr;
    }
    c->fwd_S = c->bwd_S = 0;
    return 0;
}

int mf_check_error(MfContext* c, cudaStream_t st, std::string* why) {
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, c->err, 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (!check(e, "mean-field error word", why)) return -2;
    if (h) {
        if (why) *why = "a bounded device wait expired in the mean-field GEMM (code " + std::to_string(h) + ")";
        cudaMemsetAsync(c->err, 0, 4, st);
        return -3;
    }
    return 0;
}

void mf_destroy(MfContext* c) {
    if (!c) return;
    if (c->fwd_exec) cudaGraphExecDestroy(c->fwd_exec);
    if (c->bwd_exec) cudaGraphExecDestroy(c->bwd_exec);
    if (c->cap) cudaStreamDestroy(c->cap);
    for (void* p : {static_cast<void*>(c->sched_i), static_cast<void*>(c->m0_i), static_cast<void*>(c->mprev_i),
                    static_cast<void*>(c->mout_i), static_cast<void*>(c->gm_i), static_cast<void*>(c->ckpt_i),
                    static_cast<void*>(c->gs_i)})
        if (p) cudaFree(p);
    for (void* p : {static_cast<void*>(c->J), static_cast<void*>(c->bias), static_cast<void*>(c->partial),
                    static_cast<void*>(c->mring), static_cast<void*>(c->xm), static_cast<void*>(c->xp),
                    static_cast<void*>(c->seg_m), static_cast<void*>(c->seg_P), static_cast<void*>(c->pbar),
                    static_cast<void*>(c->svec),
                    static_cast<void*>(c->cnt), static_cast<void*>(c->err)})
        if (p) cudaFree(p);
    delete c;
}

}  // namespace anc
