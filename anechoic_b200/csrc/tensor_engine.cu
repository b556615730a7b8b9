// Batched SCA engine for replicas that share J: the field update is a dense int8 contraction on the tcgen05 tensor
// cores, exact with int32 accumulation in TMEM.
//
// Per step of the reference algorithm (sca::run_trial_bias, gpu/multibit_bias_20261008/src/sca_ref_bias.hpp:44-68):
//   h_y += sum_x D_x J_xy  with  D_x = 2 s'_x for flipped x and 0 otherwise  (D = s0 with factor 1 for h(0) = b + J s0).
// Layout: a thread-block cluster of C = 16 CTAs runs a group of 128 replicas (one TMEM lane each). Spin slot
// i = k*256 + l (RNG lane l, round k) is owned by CTA c = l / 16 and held at permuted index
// p(i) = c*NC + (l % 16)*R + k (NC = NP/16 slots per CTA, R = NP/256 rounds); J is stored permuted the same way
// (J_perm[p(x)][p(y)] = J_xy), so CTA c's slots are the contiguous column slice [c*NC, (c+1)*NC).
//   * 16 decision warps: thread (replica r, quarter q) owns RNG lanes 16c + 4q .. 16c + 4q + 3 of replica r, i.e.
//     4R slots = TMEM columns [4Rq, 4R(q+1)). It reads h with tcgen05.ld, decides exactly as the golden model
//     (Q16.16 integer threshold from the replica's own xoshiro128** stream, counted / temperature-scaled correction),
//     and writes its D bytes to a global exchange buffer D[group][parity][r][p]; n_lin partials go to a small buffer.
//   * barrier.cluster (release / acquire) publishes every CTA's slice of D and n_lin.
//   * 1 TMA warp streams K-chunks of 128: A = D[group][parity][0..127][chunk] (128 x 128 B) and
//     B = J_perm[c*NC .. +NC][chunk] (NC x 128 B), 128-byte swizzled, into a 4-stage shared-memory ring
//     (no multicast anywhere).
//   * 1 MMA thread issues tcgen05.mma.cta_group::1.kind::i8 (M = 128, N = NC, K = 32) accumulating into h in TMEM,
//     frees each stage with tcgen05.commit, and signals "h ready" after the last chunk.
// Every mbarrier wait is bounded by %globaltimer: on expiry the kernel records an error code, skips the remaining
// work but keeps every cluster barrier, so all CTAs finish; the host reports ANC_ETIMEOUT.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "anc_ptx.cuh"
#include "anc_tensor.cuh"

namespace anc {
namespace {

using namespace ptx;

constexpr int kC = 16;                  // CTAs per cluster (replica group)
constexpr int kM = 128;                 // replicas per group (MMA M, TMEM lanes)
constexpr int kDW = 16;                 // decision warps
constexpr int kThreads = (kDW + 2) * 32;
constexpr int kTmaWarp = kDW, kMmaWarp = kDW + 1;
constexpr int kStages = 4;
constexpr int kKChunk = 128;            // bytes (= int8 elements) of K per stage

// error codes written to the run's error word
constexpr int kErrFull = 1, kErrEmpty = 2, kErrHready = 3;

struct TensorParams {
    int n, np, R, nc;                   // active spins, padded, rounds, slots per CTA
    int S;
    const int32_t* fourT;
    const int32_t* q;
    const int64_t* kcorr;
    const int32_t* kconst;
    int32_t hclamp;
    const int32_t* bias_perm;           // [np] bias at permuted index, or null
    uint64_t seed;
    uint32_t trial_offset;
    int nchains;
    int8_t* dbuf;                       // [groups][2][128][np]
    int32_t* nlbuf;                     // [groups][2][16][128]
    uint32_t* out_spins;                // [nchains][np/32] (zeroed by the host)
    unsigned long long* out_sum_sh;     // [nchains] (zeroed)
    unsigned long long* out_sum_bs;     // [nchains] (zeroed)
    unsigned long long* out_flips;      // [nchains] (zeroed)
    int32_t* out_trace;                 // [nchains][S] or null
    int32_t* out_h;                     // [nchains][n] or null
    int* err;                           // error word (zeroed)
    long long* prof;                    // [gridDim.x][kProfSlots] clock64 phase totals, or null (off)
};

// opt-in phase profile (clock64 cycles summed over the steps, per CTA):
//   0 decision warps waiting for h   1 TMEM load + decide + D store   2 named barrier + n_lin publish
//   3 cluster barrier   4 n_lin read   5 MMA thread waiting for stages
//   6 MMA thread: barrier end -> last commit issued   7 TMA thread waiting for free stages   8 whole step loop
constexpr int kProfSlots = kTensorProfSlots;

// ------------------------------------------------------------------------------------------------ helpers
__device__ __forceinline__ void flag_publish(uint32_t* p, uint32_t v) {
    asm volatile("fence.acq_rel.gpu;\n\tst.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_id_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}

// ------------------------------------------------------------------------------------------------ the kernel
template <int R>
__global__ void __launch_bounds__(kThreads, 1)
    tensor_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                  const __grid_constant__ TensorParams P) {
    constexpr int NC = 16 * R;            // slots (TMEM columns) per CTA
    constexpr int COLS = 4 * R;           // columns per decision thread (4 RNG lanes x R rounds)
    constexpr int NCHUNK = 2 * R;         // K chunks of 128 over NP = 256 R
    constexpr uint32_t A_BYTES = kM * kKChunk;
    constexpr uint32_t B_BYTES = NC * kKChunk;
    constexpr uint32_t STAGE = A_BYTES + B_BYTES;
    constexpr int TMEM_COLS = NC <= 32 ? 32 : NC <= 64 ? 64 : NC <= 128 ? 128 : 256;
    constexpr uint32_t IDESC = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(NC >> 3) << 17) | (uint32_t(kM >> 4) << 24);

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* stages = smem;                                        // kStages x STAGE, 1024-aligned
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * STAGE);
    // bars: full[kStages], empty[kStages], hready
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);
    int* nl_s = reinterpret_cast<int*>(tmem_slot + 4);           // [128] n_lin partial of this CTA per replica

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c = int(cluster_rank());
    const int g = int(cluster_id_x());                            // replica group
    const int n = P.n, S = P.S;
    int* err = P.err;

    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + kStages);
    const uint32_t bar_h = smem_u32(bars + 2 * kStages);

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_h, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid < kM) nl_s[tid] = 0;
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // ---------------- decision warps ----------------
    // replica r = lane quarter (warp % 4) * 32 + lane; column quarter qq = warp / 4
    const int r = (warp & 3) * 32 + lane;
    const int qq = warp >> 2;
    const int chain = g * kM + r;
    const bool writer = chain < P.nchains;
    Xoshiro rng[4];
    uint32_t sw[2] = {0u, 0u}, dw[2] = {0u, 0u};   // spin (1 = +1) and flipped-last-step bits of the COLS slots
    long long flips = 0;
    int32_t nlin_prev = 0;
    const uint32_t taddr = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(qq * COLS);
    int8_t* drow0 = P.dbuf + (size_t(g) * 2 * kM + r) * P.np + size_t(c) * NC + size_t(qq) * COLS;
    const size_t dpar_stride = size_t(kM) * P.np;

    // slot of column col (= j*R + k) of this thread: RNG lane l = 16c + 4qq + j, round k, i = k*256 + l
    auto slot_of = [&](int col) { return (col % R) * 256 + 16 * c + 4 * qq + col / R; };

    if (warp < kDW) {
        // seeds, initial spins (draw >> 31, padding +1), s_prev = +1 (so "flipped" = [s0 = -1]); h := bias
        for (int j = 0; j < 4; ++j) rng_seed(rng[j], P.seed, P.trial_offset + uint32_t(chain), uint32_t(16 * c + 4 * qq + j));
        uint32_t dbytes[COLS / 4];
#pragma unroll
        for (int w = 0; w < COLS / 4; ++w) dbytes[w] = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int col = j * R + k;
                const uint32_t rv = rng_next(rng[j]);
                const int i = k * 256 + 16 * c + 4 * qq + j;
                const bool valid = i < n;
                const uint32_t up = valid ? (rv >> 31) : 1u;
                sw[col >> 5] |= up << (col & 31);
                if (valid && !up) dw[col >> 5] |= 1u << (col & 31);
                const uint32_t b = valid ? (up ? 0x01u : 0xFFu) : 0u;
                dbytes[col >> 2] |= b << (8 * (col & 3));
            }
        // D(-1) = s0 into parity 1 (the step index -1 is odd)
        int8_t* drow = drow0 + dpar_stride;
#pragma unroll
        for (int w = 0; w < COLS / 16; ++w)
            reinterpret_cast<uint4*>(drow)[w] = make_uint4(dbytes[4 * w], dbytes[4 * w + 1], dbytes[4 * w + 2], dbytes[4 * w + 3]);
        // TMEM h := bias (per column)
#pragma unroll
        for (int cb = 0; cb < COLS; cb += 16) {
            uint32_t v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const int col = qq * COLS + cb + e;
                v[e] = P.bias_perm ? uint32_t(P.bias_perm[c * NC + col]) : 0u;
            }
            tmem_st16(taddr + cb, v);
        }
        tmem_wait_st();
        if (qq == 0) P.nlbuf[((size_t(g) * 2 + 1) * kC + c) * kM + r] = 0;
        asm volatile("fence.proxy.async.global;" ::: "memory");
        tc_fence_before();
    }

    // step index m = -1 (initial field), 0 .. S-1; after each: cluster barrier, then the MMA applies D(m)
    uint32_t stage_it = 0;                     // running stage counter (TMA and MMA threads)
    const bool prof = P.prof != nullptr;
    long long pr[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    long long tq = clock64();
    const long long t_loop0 = tq;
    auto mark = [&](int slot) {
        if (prof) {
            const long long now = clock64();
            pr[slot] += now - tq;
            tq = now;
        }
    };
    for (int m = -1; m < S; ++m) {
        const int par = m & 1;
        if (m >= 0 && warp < kDW) {
            // wait for h (after D(m-1)), read it, decide step m
            if (prof) tq = clock64();
            if (!err_set(err)) mbar_wait(bar_h, uint32_t(m & 1), err, kErrHready);
            tc_fence_after();
            mark(0);
            const int t = m;
            const int32_t fourT = __ldg(P.fourT + t), twoT = fourT >> 1, qv = __ldg(P.q + t);
            const int32_t corr = step_corr(nlin_prev, __ldg(P.kcorr + t), __ldg(P.kconst + t));
            const uint32_t lw = uint32_t(2 * twoT - 1);
            const int32_t hcl = P.hclamp;
            uint32_t dbytes[COLS / 4];
#pragma unroll
            for (int w = 0; w < COLS / 4; ++w) dbytes[w] = 0u;
            int nl = 0;
            uint32_t nsw[2] = {sw[0], sw[1]}, ndw[2] = {0u, 0u};
#pragma unroll
            for (int cb = 0; cb < COLS; cb += 16) {
                uint32_t hv[16];
                tmem_ld16(taddr + cb, hv);
                tmem_wait_ld();
                // draws follow each lane's round order: columns are j*R + k, so 16-column blocks taken in order
                // visit every lane's rounds in increasing k
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int col = cb + e;
                    const int j = col / R, k = col % R;
                    const uint32_t u = rng_next(rng[j]);
                    const int i = k * 256 + 16 * c + 4 * qq + j;
                    const bool valid = i < n;
                    const bool up = (sw[col >> 5] >> (col & 31)) & 1u;
                    const bool dif = (dw[col >> 5] >> (col & 31)) & 1u;
                    const int32_t h = int32_t(hv[e]);
                    int32_t hs = up ? h : -h;
                    if (hcl > 0) hs = max(-hcl, min(hs, hcl));
                    const int32_t x = qv + (dif ? corr : -corr);
                    const int32_t zt = hs * 65536 + x;
                    const int32_t thr = threshold16(u, fourT);
                    const bool fl = valid && (zt - thr < 0);
                    nl += (valid && (uint32_t(zt + twoT - 1) < lw)) ? 1 : 0;
                    if (fl) {
                        nsw[col >> 5] ^= 1u << (col & 31);
                        ndw[col >> 5] |= 1u << (col & 31);
                        dbytes[col >> 2] |= (up ? 0xFEu : 0x02u) << (8 * (col & 3));   // 2 * s' with s' = -s
                        ++flips;
                    }
                }
            }
            sw[0] = nsw[0]; sw[1] = nsw[1];
            dw[0] = ndw[0]; dw[1] = ndw[1];
            int8_t* drow = drow0 + size_t(par) * dpar_stride;
#pragma unroll
            for (int w = 0; w < COLS / 16; ++w)
                reinterpret_cast<uint4*>(drow)[w] =
                    make_uint4(dbytes[4 * w], dbytes[4 * w + 1], dbytes[4 * w + 2], dbytes[4 * w + 3]);
            mark(1);
            atomicAdd(&nl_s[r], nl);
            tc_fence_before();
            asm volatile("bar.sync 1, %0;" ::"r"(kDW * 32) : "memory");
            if (qq == 0) {
                P.nlbuf[((size_t(g) * 2 + par) * kC + c) * kM + r] = nl_s[r];
                nl_s[r] = 0;
            }
            asm volatile("fence.proxy.async.global;" ::: "memory");
            mark(2);
        }
        if (prof) tq = clock64();
        cluster_sync();
        asm volatile("fence.proxy.async.global;" ::: "memory");
        if (warp < kDW) mark(3);
        else if (prof) tq = clock64();
        if (warp < kDW && m >= 0) {
            // n_lin of step m for replica r: sum of the 16 CTAs' partials
            const int32_t* nlp = P.nlbuf + (size_t(g) * 2 + par) * kC * kM + r;
            int32_t tot = 0;
#pragma unroll
            for (int cc = 0; cc < kC; ++cc) tot += __ldcg(nlp + cc * kM);
            nlin_prev = tot;
            if (c == 0 && qq == 0 && writer && P.out_trace) P.out_trace[size_t(chain) * S + m] = tot;
            mark(4);
        }
        if (warp == kTmaWarp) {
            if (lane == 0) {
                const int ay = (g * 2 + (par & 1)) * kM;
                for (int kc = 0; kc < NCHUNK; ++kc, ++stage_it) {
                    const int s = int(stage_it % kStages);
                    const uint32_t ph = (stage_it / kStages) & 1u;
                    if (err_set(err)) continue;   // after a failed wait: issue nothing more
                    const long long w0 = prof ? clock64() : 0;
                    if (stage_it >= kStages && !mbar_wait(bar_empty + 8 * s, ph ^ 1u, err, kErrEmpty)) continue;
                    if (prof) pr[7] += clock64() - w0;
                    const uint32_t dst = smem_u32(stages + size_t(s) * STAGE);
                    mbar_arrive_expect_tx(bar_full + 8 * s, STAGE);
                    tma_load_2d(dst, &mapA, kc * kKChunk, ay, bar_full + 8 * s);
                    tma_load_2d(dst + A_BYTES, &mapB, kc * kKChunk, c * NC, bar_full + 8 * s);
                }
            } else {
                stage_it += NCHUNK;
            }
            __syncwarp();
        } else if (warp == kMmaWarp) {
            if (lane == 0) {
                tc_fence_after();
                for (int kc = 0; kc < NCHUNK; ++kc, ++stage_it) {
                    const int s = int(stage_it % kStages);
                    const uint32_t ph = (stage_it / kStages) & 1u;
                    const long long w0 = prof ? clock64() : 0;
                    const bool ok = !err_set(err) && mbar_wait(bar_full + 8 * s, ph, err, kErrFull);
                    if (prof) pr[5] += clock64() - w0;
                    tc_fence_after();
                    if (ok) {
                        const uint32_t a0 = smem_u32(stages + size_t(s) * STAGE), b0 = a0 + A_BYTES;
#pragma unroll
                        for (int kk = 0; kk < kKChunk / 32; ++kk)
                            mma_i8(tmem, sw128_desc(a0 + 32 * kk), sw128_desc(b0 + 32 * kk), IDESC, 1u);
                    }
                    mma_commit(bar_empty + 8 * s);     // frees the stage once the MMAs above have read it
                }
                mma_commit(bar_h);                     // h ready for the next decision
                mark(6);
            } else {
                stage_it += NCHUNK;
            }
            __syncwarp();
        }
    }
    if (prof) {
        pr[8] = clock64() - t_loop0;
        long long* dst = P.prof + size_t(blockIdx.x) * kProfSlots;
        if (warp == 0 && lane == 0)
            for (int s = 0; s < 5; ++s) dst[s] = pr[s];
        if (warp == kMmaWarp && lane == 0) { dst[5] = pr[5]; dst[6] = pr[6]; dst[8] = pr[8]; }
        if (warp == kTmaWarp && lane == 0) dst[7] = pr[7];
    }

    // ---------------- final fields and outputs ----------------
    if (warp < kDW) {
        if (!err_set(err)) mbar_wait(bar_h, uint32_t(S & 1), err, kErrHready);
        tc_fence_after();
        long long sh = 0, bs = 0;
        const int words = P.np / 32;
#pragma unroll
        for (int cb = 0; cb < COLS; cb += 16) {
            uint32_t hv[16];
            tmem_ld16(taddr + cb, hv);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const int col = cb + e;
                const int i = slot_of(col);
                if (i >= n) continue;
                const bool up = (sw[col >> 5] >> (col & 31)) & 1u;
                const int32_t h = int32_t(hv[e]);
                sh += up ? h : -h;
                if (P.bias_perm) {
                    const int32_t b = P.bias_perm[c * NC + qq * COLS + col];
                    bs += up ? b : -b;
                }
                if (writer) {
                    if (up) atomicOr(P.out_spins + size_t(chain) * words + (i >> 5), 1u << (i & 31));
                    if (P.out_h) P.out_h[size_t(chain) * n + i] = h;
                }
            }
        }
        if (writer) {
            atomicAdd(P.out_sum_sh + chain, static_cast<unsigned long long>(sh));
            atomicAdd(P.out_sum_bs + chain, static_cast<unsigned long long>(bs));
            atomicAdd(P.out_flips + chain, static_cast<unsigned long long>(flips));
        }
        tc_fence_before();
    }
    __syncthreads();
    cluster_sync();   // no CTA leaves while a peer may still read its D slice through L2 (and keeps TMEM until done)
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------ resident-J kernel
// For NP = 2048 (n <= 2048): a cooperative persistent grid of 32 y-slices x P group-pairs. CTA (pair slot gp,
// slice cs) owns spin slots with RNG lanes 8cs .. 8cs+7 (64 columns at permuted indices p = 8l + k) and keeps its
// J column slice (2048 x 64 int8 = 128 KB, 128-byte swizzled) resident in shared memory for the whole launch.
// It runs TWO replica groups of 128 (a pair) and alternates between them, so the decisions of one group overlap
// the tensor-core update of the other:
//   decision warps (16): for group g: wait "h ready", tcgen05.ld 16 field columns + the n_lin accumulator, decide,
//     write D(m) (16 bytes) and the thread's n_lin partial (1 byte) to the exchange buffers, then one thread
//     publishes flag[g][cs] = m + 2 (st.release.gpu).
//   producer warps (4): for every K chunk (128 x-values = two source slices) wait for both slices' flags
//     (ld.acquire.gpu), then TMA the 128 x 128-byte D tile into the stage ring; a 17th chunk carries the 128
//     n_lin partials of all slices. Each warp issues every fourth chunk: one thread's bulk copies are serviced one
//     at a time, so four issuers keep four copies in flight.
//   MMA thread: per chunk 4 x tcgen05.mma.kind::i8 (M 128, N 64, K 32) into the group's field accumulator with B
//     = the resident J chunk; the n_lin chunk is multiplied by a ones row (N 16) into a per-group accumulator,
//     so sum_slices n_lin partials comes out of the tensor core with the fields.
// No cluster barrier exists: the flags make the exchange a dataflow, chunks are consumed as slices finish.
constexpr int kResSlices = 32;            // y-slices for NP = 2048
constexpr int kResYS = 64;                // columns per slice (MMA N)
constexpr int kResPW = 4;                 // producer warps
constexpr int kResStages = 5;
constexpr int kResMmaWarp = kDW + kResPW;
constexpr int kResThreads = (kDW + kResPW + 1) * 32;
constexpr int kResChunks = 17;            // 16 D chunks + 1 n_lin chunk per (step, group)
constexpr int kErrFlag = 4, kErrJ = 5, kErrInit = 6, kErrRead = 7;

struct ResParams {
    int n, S, npairs;
    const int32_t* fourT;
    const int32_t* q;
    const int64_t* kcorr;
    const int32_t* kconst;
    int32_t hclamp;
    const int32_t* bias_perm;           // [2048] or null
    uint64_t seed;
    uint32_t trial_offset;
    int nchains;
    uint32_t* flags;                    // [2 * npairs][32] (zeroed)
    int8_t* dbuf;                       // [2 * npairs][2][128][2048]
    int8_t* nlx;                        // [2 * npairs][2][128][128]
    uint64_t wait_ns;                   // limit of each wait of the exchange (the drain at exit keeps its own)
    uint32_t* out_spins;                // [nchains][64] (zeroed)
    unsigned long long* out_sum_sh;
    unsigned long long* out_sum_bs;
    unsigned long long* out_flips;
    int32_t* out_trace;
    int32_t* out_h;
    int* err;
    long long* prof;
};

__global__ void __launch_bounds__(kResThreads, 1)
    tensor_res_kernel(const __grid_constant__ CUtensorMap mapD, const __grid_constant__ CUtensorMap mapNL,
                      const __grid_constant__ CUtensorMap mapJ, const __grid_constant__ ResParams P) {
    constexpr int R = 8, NPAD = 2048;
    constexpr uint32_t TILE = kM * kKChunk;                 // 16 KB D / n_lin tile
    constexpr uint32_t JCHUNK = kResYS * kKChunk;           // 8 KB of resident J per K chunk
    constexpr uint32_t IDESC_H = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(kResYS >> 3) << 17) | (uint32_t(kM >> 4) << 24);
    constexpr uint32_t IDESC_NL = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(16 >> 3) << 17) | (uint32_t(kM >> 4) << 24);

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* jres = smem;                                   // 16 x 8 KB
    uint8_t* ones = smem + 16 * JCHUNK;                     // 2 KB: row 0 = 128 x int8(1), rows 1..15 = 0
    uint8_t* stages = ones + 2048;                          // kResStages x 16 KB (1024-aligned)
    uint64_t* bars = reinterpret_cast<uint64_t*>(stages + kResStages * TILE);
    // bars: full[5], empty[5], hready[2], jbar, init, fields read[2], drain
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kResStages + 7);
    uint32_t* s_issued = tmem_slot + 1;                     // [kResStages] copies issued into each stage (drain)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cs = int(blockIdx.x % kResSlices);
    const int gp0 = int(blockIdx.x / kResSlices), gstride = int(gridDim.x / kResSlices);
    const int n = P.n, S = P.S;
    int* err = P.err;
    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + kResStages);
    const uint32_t bar_h0 = smem_u32(bars + 2 * kResStages), bar_j = smem_u32(bars + 2 * kResStages + 2);
    const uint32_t bar_init = smem_u32(bars + 2 * kResStages + 3);   // decision warps: fields of a new pair set
    // decision warps: group g's fields for step m have been read, so its step-m tiles may now be accumulated (other
    // slices can publish step m before this CTA has read the fields it decides step m from)
    const uint32_t bar_rd0 = smem_u32(bars + 2 * kResStages + 4);
    const uint32_t bar_fin = smem_u32(bars + 2 * kResStages + 6);    // MMA thread: drain before TMEM is freed

    if (tid == 0) {
        for (int s = 0; s < kResStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_h0, 1);
        mbar_init(bar_h0 + 8, 1);
        mbar_init(bar_rd0, 1);
        mbar_init(bar_rd0 + 8, 1);
        mbar_init(bar_j, 1);
        mbar_init(bar_init, 1);
        mbar_init(bar_fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < kResStages) s_issued[tid] = 0u;
    for (int i = tid; i < 2048; i += blockDim.x) ones[i] = i < 128 ? 1 : 0;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == kResMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(256)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // resident J slice: rows cs*64 .. +64 of J_perm, 16 chunks of 128 columns
    if (warp == kDW && lane == 0) {
        mbar_arrive_expect_tx(bar_j, 16 * JCHUNK);
        for (int kc = 0; kc < 16; ++kc) tma_load_2d(smem_u32(jres + kc * JCHUNK), &mapJ, kc * kKChunk, cs * kResYS, bar_j);
    }

    // decision-thread geometry: replica r (TMEM lane), column quarter qq: RNG lanes 8cs + 2qq + j, columns qq*16 ..
    const int r = (warp & 3) * 32 + lane, qq = warp >> 2;
    const uint32_t tl = uint32_t((warp & 3) * 32) << 16;
    uint32_t hph[2] = {0u, 0u};            // decision side: completed "h ready" phases per group
    uint32_t q = 0;                        // running chunk index (producers, MMA)
    bool jready = false;
    uint32_t iph = 0u;                     // MMA thread: completed "fields set" phases
    uint32_t rph[2] = {0u, 0u};            // MMA thread: completed "fields read" phases per group
    uint32_t q_ok = 0;                     // MMA thread: chunks 0 .. q_ok - 1 were waited for and consumed
    const bool prof = P.prof != nullptr;
    long long pr[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const long long t_loop0 = clock64();

    for (int pw = gp0; pw < P.npairs; pw += gstride) {
        const int G[2] = {2 * pw, 2 * pw + 1};
        if (warp < kDW) {
            // ---------------- decision warps ----------------
            Xoshiro rng[2][2];
            uint32_t sw[2], dw[2], nlacc_prev[2] = {0u, 0u};
            int32_t nlin_prev[2] = {0, 0};
            long long flips[2] = {0, 0};
            const int chain[2] = {G[0] * kM + r, G[1] * kM + r};
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                sw[g] = 0u;
                dw[g] = 0u;
                uint32_t db[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    rng_seed(rng[g][j], P.seed, P.trial_offset + uint32_t(chain[g]), uint32_t(8 * cs + 2 * qq + j));
#pragma unroll
                    for (int k = 0; k < R; ++k) {
                        const int col = j * R + k, i = k * 256 + 8 * cs + 2 * qq + j;
                        const uint32_t rv = rng_next(rng[g][j]);
                        const bool valid = i < n;
                        const uint32_t up = valid ? (rv >> 31) : 1u;
                        sw[g] |= up << col;
                        if (valid && !up) dw[g] |= 1u << col;
                        db[col >> 2] |= (valid ? (up ? 0x01u : 0xFFu) : 0u) << (8 * (col & 3));
                    }
                }
                int8_t* drow = P.dbuf + ((size_t(G[g]) * 2 + 1) * kM + r) * NPAD + cs * kResYS + qq * 16;
                *reinterpret_cast<uint4*>(drow) = make_uint4(db[0], db[1], db[2], db[3]);
                P.nlx[((size_t(G[g]) * 2 + 1) * kM + r) * 128 + cs * 4 + qq] = 0;
                // fields := bias, n_lin accumulator := 0
                uint32_t v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    v[e] = P.bias_perm ? uint32_t(P.bias_perm[cs * kResYS + qq * 16 + e]) : 0u;
                tmem_st16(tmem + tl + uint32_t(g * kResYS + qq * 16), v);
                if (qq == 0) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] = 0u;
                    tmem_st16(tmem + tl + uint32_t(128 + g * 16), v);
                }
            }
            tmem_wait_st();
            writer_fence();
            tc_fence_before();
            asm volatile("bar.sync 1, %0;" ::"r"(kDW * 32) : "memory");
            if (tid == 0) {
                // the MMA thread may accumulate into these fields only after they are set: tiles of other slices
                // can land before this CTA leaves its previous pair
                mbar_arrive(bar_init);
                flag_publish(P.flags + G[0] * kResSlices + cs, 1u);
                flag_publish(P.flags + G[1] * kResSlices + cs, 1u);
            }
            for (int m = 0; m <= S; ++m) {
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    long long t0 = prof ? clock64() : 0;
                    if (!err_set(err)) mbar_wait_for(bar_h0 + 8 * g, hph[g] & 1u, err, kErrHready, P.wait_ns);
                    ++hph[g];
                    tc_fence_after();
                    if (prof) { const long long t1 = clock64(); pr[0] += t1 - t0; t0 = t1; }
                    uint32_t hv[16], nv;
                    tmem_ld16(tmem + tl + uint32_t(g * kResYS + qq * 16), hv);
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];"
                                 : "=r"(nv)
                                 : "r"(tmem + tl + uint32_t(128 + g * 16)));
                    tmem_wait_ld();
                    const int32_t nlin = int32_t(nv - nlacc_prev[g]);   // n_lin of step m - 1 (0 before step 0)
                    nlacc_prev[g] = nv;
                    const bool writer = chain[g] < P.nchains;
                    if (m >= 1 && writer && cs == 0 && qq == 0 && P.out_trace) P.out_trace[size_t(chain[g]) * S + (m - 1)] = nlin;
                    nlin_prev[g] = nlin;
                    if (m == S) {
                        // final fields: outputs
                        long long sh = 0, bs = 0;
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            const int j = e / R, k = e % R, i = k * 256 + 8 * cs + 2 * qq + j;
                            if (i >= n) continue;
                            const bool up = (sw[g] >> e) & 1u;
                            const int32_t h = int32_t(hv[e]);
                            sh += up ? h : -h;
                            if (P.bias_perm) {
                                const int32_t b = P.bias_perm[cs * kResYS + qq * 16 + e];
                                bs += up ? b : -b;
                            }
                            if (writer) {
                                if (up) atomicOr(P.out_spins + size_t(chain[g]) * 64 + (i >> 5), 1u << (i & 31));
                                if (P.out_h) P.out_h[size_t(chain[g]) * n + i] = h;
                            }
                        }
                        if (writer) {
                            atomicAdd(P.out_sum_sh + chain[g], static_cast<unsigned long long>(sh));
                            atomicAdd(P.out_sum_bs + chain[g], static_cast<unsigned long long>(bs));
                            atomicAdd(P.out_flips + chain[g], static_cast<unsigned long long>(flips[g]));
                        }
                        continue;
                    }
                    const int t = m;
                    const int32_t fourT = __ldg(P.fourT + t), twoT = fourT >> 1, qv = __ldg(P.q + t);
                    const int32_t corr = step_corr(nlin_prev[g], __ldg(P.kcorr + t), __ldg(P.kconst + t));
                    const uint32_t lw = uint32_t(2 * twoT - 1);
                    const int32_t hcl = P.hclamp;
                    uint32_t db[4] = {0u, 0u, 0u, 0u};
                    uint32_t nsw = sw[g], ndw = 0u;
                    int nl = 0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const int j = e / R, k = e % R, i = k * 256 + 8 * cs + 2 * qq + j;
                        const uint32_t u = rng_next(rng[g][j]);
                        const bool valid = i < n;
                        const bool up = (sw[g] >> e) & 1u, dif = (dw[g] >> e) & 1u;
                        const int32_t h = int32_t(hv[e]);
                        int32_t hs = up ? h : -h;
                        if (hcl > 0) hs = max(-hcl, min(hs, hcl));
                        const int32_t x = qv + (dif ? corr : -corr);
                        const int32_t zt = hs * 65536 + x;
                        const int32_t thr = threshold16(u, fourT);
                        const bool fl = valid && (zt - thr < 0);
                        nl += (valid && (uint32_t(zt + twoT - 1) < lw)) ? 1 : 0;
                        if (fl) {
                            nsw ^= 1u << e;
                            ndw |= 1u << e;
                            db[e >> 2] |= (up ? 0xFEu : 0x02u) << (8 * (e & 3));
                            ++flips[g];
                        }
                    }
                    sw[g] = nsw;
                    dw[g] = ndw;
                    const int par = m & 1;
                    int8_t* drow = P.dbuf + ((size_t(G[g]) * 2 + par) * kM + r) * NPAD + cs * kResYS + qq * 16;
                    *reinterpret_cast<uint4*>(drow) = make_uint4(db[0], db[1], db[2], db[3]);
                    P.nlx[((size_t(G[g]) * 2 + par) * kM + r) * 128 + cs * 4 + qq] = int8_t(nl);
                    writer_fence();
                    tc_fence_before();
                    if (prof) { const long long t1 = clock64(); pr[1] += t1 - t0; t0 = t1; }
                    asm volatile("bar.sync 1, %0;" ::"r"(kDW * 32) : "memory");
                    if (tid == 0) {
                        mbar_arrive(bar_rd0 + 8 * g);
                        flag_publish(P.flags + G[g] * kResSlices + cs, uint32_t(m + 2));
                    }
                    if (prof) pr[2] += clock64() - t0;
                }
            }
            tc_fence_before();
        } else if (warp < kDW + kResPW) {
            // ---------------- producer warps (all lanes poll the 32 slice flags at once; lane 0 issues) ----------
            const int pwid = warp - kDW;
            uint32_t ready = 0u;                   // slices known to have published (m, g)
            for (int m = -1; m < S; ++m) {
                const int par = m & 1;
                for (int g = 0; g < 2; ++g) {
                    const int ay = (G[g] * 2 + par) * kM;
                    const uint32_t* fl = P.flags + G[g] * kResSlices;
                    const uint32_t target = uint32_t(m + 2);
                    ready = 0u;
                    for (int c = 0; c < kResChunks; ++c, ++q) {
                        if (int(q % kResPW) != pwid) continue;
                        // every branch below is warp-uniform: lane 0 decides and broadcasts
                        if (__shfl_sync(0xffffffffu, err_set(err) ? 1 : 0, 0)) continue;
                        const int s = int(q % kResStages);
                        const uint32_t u = q / kResStages;
                        const long long w0 = prof ? clock64() : 0;
                        if (u >= 1) {
                            const int w = lane == 0 ? (mbar_wait_for(bar_empty + 8 * s, (u - 1) & 1u, err, kErrEmpty, P.wait_ns) ? 1 : 0) : 1;
                            if (!__shfl_sync(0xffffffffu, w, 0)) continue;
                        }
                        const uint32_t need = c < 16 ? (3u << (2 * c)) : 0xffffffffu;
                        bool ok = (ready & need) == need;
                        if (!ok) {
                            const uint64_t t0 = globaltimer();
                            for (uint32_t k = 1;; ++k) {
                                uint32_t v;
                                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(fl + lane) : "memory");
                                ready = __ballot_sync(0xffffffffu, v >= target);
                                if ((ready & need) == need) { ok = true; break; }
                                if ((k & 63u) == 0 && __shfl_sync(0xffffffffu, globaltimer() - t0 > P.wait_ns, 0)) {
                                    if (lane == 0) atomicCAS(err, 0, kErrFlag);
                                    break;
                                }
                            }
                        }
                        if (prof) pr[7] += clock64() - w0;
                        if (!ok) continue;
                        if (lane == 0) {
                            asm volatile("fence.proxy.async.global;" ::: "memory");
                            const uint32_t dst = smem_u32(stages + size_t(s) * TILE);
                            mbar_arrive_expect_tx(bar_full + 8 * s, TILE);
                            if (c < 16) tma_load_2d(dst, &mapD, c * kKChunk, ay, bar_full + 8 * s);
                            else tma_load_2d(dst, &mapNL, 0, ay, bar_full + 8 * s);
                            atomicAdd(s_issued + s, 1u);
                        }
                        __syncwarp();
                    }
                }
            }
        } else if (warp == kResMmaWarp) {
            // ---------------- MMA thread ----------------
            if (lane == 0) {
                // jready only once the J copy is seen landed: after a wait that gave up, the drain at exit waits
                // for it (a copy must not land in shared memory the CTA has released)
                if (!jready && !err_set(err)) jready = mbar_wait_for(bar_j, 0u, err, kErrJ, P.wait_ns);
                if (!err_set(err)) mbar_wait_for(bar_init, iph & 1u, err, kErrInit, P.wait_ns);
                ++iph;
                tc_fence_after();
                for (int m = -1; m < S; ++m) {
                    for (int g = 0; g < 2; ++g) {
                        const long long t0 = prof ? clock64() : 0;
                        if (m >= 0) {
                            if (!err_set(err)) mbar_wait_for(bar_rd0 + 8 * g, rph[g] & 1u, err, kErrRead, P.wait_ns);
                            ++rph[g];
                            tc_fence_after();
                        }
                        for (int c = 0; c < kResChunks; ++c, ++q) {
                            const int s = int(q % kResStages);
                            const uint32_t u = q / kResStages;
                            const long long w0 = prof ? clock64() : 0;
                            const bool ok = !err_set(err) && mbar_wait_for(bar_full + 8 * s, u & 1u, err, kErrFull, P.wait_ns);
                            if (ok) q_ok = q + 1;
                            if (prof) pr[5] += clock64() - w0;
                            tc_fence_after();
                            const long long i0 = prof ? clock64() : 0;
                            if (ok) {
                                const uint32_t a0 = smem_u32(stages + size_t(s) * TILE);
                                if (c < 16) {
                                    const uint32_t b0 = smem_u32(jres + c * JCHUNK);
#pragma unroll
                                    for (int kk = 0; kk < kKChunk / 32; ++kk)
                                        mma_i8(tmem + uint32_t(g * kResYS), sw128_desc(a0 + 32 * kk), sw128_desc(b0 + 32 * kk),
                                               IDESC_H, 1u);
                                } else {
                                    const uint32_t b0 = smem_u32(ones);
#pragma unroll
                                    for (int kk = 0; kk < kKChunk / 32; ++kk)
                                        mma_i8(tmem + uint32_t(128 + g * 16), sw128_desc(a0 + 32 * kk),
                                               sw128_desc(b0 + 32 * kk), IDESC_NL, 1u);
                                }
                            }
                            const long long i1 = prof ? clock64() : 0;
                            mma_commit(bar_empty + 8 * s);
                            if (prof) { const long long i2 = clock64(); pr[9] += i1 - i0; pr[10] += i2 - i1; }
                        }
                        mma_commit(bar_h0 + 8 * g);
                        if (prof) pr[6] += clock64() - t0;
                    }
                }
            } else {
                q += uint32_t(S + 1) * 2 * kResChunks;
            }
            __syncwarp();
        }
    }
    // every warp has left the loop, so no copy or MMA is issued after this barrier: the MMA thread waits (fixed
    // bound) for the copies still in flight -- after a wait that gave up, some were issued but never consumed -- and
    // for every MMA it issued, before the CTA releases shared memory and TMEM
    __syncthreads();
    if (warp == kResMmaWarp && lane == 0) {
        if (!jready) mbar_wait_for(bar_j, 0u, nullptr, 0, kWaitNs);
        for (int s = 0; s < kResStages; ++s) {
            // uses of stage s consumed (chunks q < q_ok with q mod stages = s), then the issued ones not consumed
            uint32_t u = q_ok > uint32_t(s) ? (q_ok - uint32_t(s) + kResStages - 1) / kResStages : 0u;
            for (uint32_t k = 0; u < s_issued[s] && k < 64; ++k, ++u) mbar_wait_for(bar_full + 8 * s, u & 1u, nullptr, 0, kWaitNs);
        }
        mma_commit(bar_fin);
        mbar_wait_for(bar_fin, 0u, nullptr, 0, kWaitNs);
    }
    if (prof) {
        long long* dst = P.prof + size_t(blockIdx.x) * kProfSlots;
        if (warp == 0 && lane == 0) {
            dst[0] = pr[0]; dst[1] = pr[1]; dst[2] = pr[2];
        }
        if (warp == kResMmaWarp && lane == 0) {
            dst[5] = pr[5]; dst[6] = pr[6]; dst[8] = clock64() - t_loop0; dst[9] = pr[9]; dst[10] = pr[10];
        }
        if (warp == kDW && lane == 0) dst[7] = pr[7];
    }
    __syncthreads();
    if (warp == kResMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------ host side
// 2-D uint8 tensor [rows][cols] (cols contiguous), box = box_rows x 128 bytes, 128-byte swizzle.
bool make_map(CUtensorMap* map, void* base, uint64_t cols, uint64_t rows, uint32_t box_rows) {
    return make_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, base, cols, rows, uint32_t(kKChunk), box_rows);
}

template <int R>
size_t smem_bytes_t() {
    constexpr size_t NC = 16 * R;
    return 1024 + kStages * (size_t(kM) * kKChunk + NC * kKChunk) + (2 * kStages + 1) * 8 + 16 + kM * 4;
}

template <int R>
int launch_t(const TensorParams& P, int groups, const CUtensorMap& A, const CUtensorMap& B, cudaStream_t st,
             std::string* why) {
    auto fn = tensor_kernel<R>;
    const size_t smem = smem_bytes_t<R>();
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) {
        if (why) *why = std::string("kernel attributes: ") + cudaGetErrorString(e);
        return -2;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kC;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(kC * groups);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    e = cudaLaunchKernelEx(&cfg, fn, A, B, P);
    if (e != cudaSuccess) {
        if (why) *why = std::string("launch: ") + cudaGetErrorString(e);
        return -2;
    }
    return 0;
}

template <int R>
int max_clusters_t(int* out) {
    auto fn = tensor_kernel<R>;
    const size_t smem = smem_bytes_t<R>();
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kC;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(kC);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(out, fn, &cfg);
    return int(e);
}

size_t res_smem_bytes() {
    return 1024 + 16 * size_t(kResYS) * kKChunk + 2048 + size_t(kResStages) * kM * kKChunk + (2 * kResStages + 7) * 8 + 16 +
           4 * kResStages;
}

// Concurrent pair slots of the resident kernel (32 co-resident CTAs each).
int res_pair_slots(int npairs, int* out) {
    auto fn = tensor_res_kernel;
    const size_t smem = res_smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    int per_sm = 0, dev = 0, sms = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kResThreads, smem);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return int(e);
    *out = std::max(0, std::min(npairs, (per_sm * sms) / kResSlices));
    return 0;
}

}  // namespace

int tensor_geometry(int n, int nchains, TensorGeometry* g) {
    const int np = std::max(2048, ((n + 255) / 256) * 256);
    const int R = np / 256;
    if (stream_supported(n)) {
        g->cluster = 1;
        g->ctas = 128;
        g->max_active_clusters = 128;
        return 0;
    }
    if (R == 8) {
        const int npairs = ((nchains + kM - 1) / kM + 1) / 2;
        int slots = 0;
        const int rc = res_pair_slots(npairs, &slots);
        g->cluster = 1;
        g->ctas = kResSlices * slots;
        g->max_active_clusters = g->ctas;
        return rc;
    }
    g->cluster = kC;
    g->ctas = kC * ((nchains + kM - 1) / kM);
    if (R == 12) return max_clusters_t<12>(&g->max_active_clusters);
    if (R == 16) return max_clusters_t<16>(&g->max_active_clusters);
    return int(cudaErrorInvalidValue);
}

bool tensor_supported(int n, int K, int nchains) {
    (void)K;
    const int np = std::max(2048, ((n + 255) / 256) * 256);
    const int R = np / 256;
    return nchains >= 1 && (R == 8 || R == 12 || R == 16 || stream_supported(n));
}

int tensor_build_instance(const int8_t* J, int n, TensorInstance* out, std::string* why) {
    const int np = std::max(2048, ((n + 255) / 256) * 256);
    const int R = np / 256, nc = 16 * R;
    if (!(R == 8 || R == 12 || R == 16)) {
        if (why) *why = "tensor engine supports NP in {2048, 3072, 4096} and (8192, 16384]";
        return -1;
    }
    std::vector<int> p(np);
    for (int i = 0; i < np; ++i) {
        const int l = i % 256, k = i / 256, cc = l / 16, jl = l % 16;
        p[i] = cc * nc + jl * R + k;
    }
    const int npp = np;
    std::vector<int8_t> Jp(size_t(npp) * npp, 0);
    for (int x = 0; x < n; ++x) {
        for (int y = 0; y < n; ++y) {
            const int8_t v = J[size_t(x) * n + y];
            Jp[size_t(p[y]) * npp + p[x]] = v;   // row = y (N), col = x (K)
        }
    }
    out->n = n;
    out->np = np;
    out->npp = npp;
    out->perm.assign(p.begin(), p.end());
    cudaError_t e = cudaMalloc(&out->d_J, Jp.size());
    if (e == cudaSuccess) e = cudaMemcpy(out->d_J, Jp.data(), Jp.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        if (why) *why = std::string("upload J: ") + cudaGetErrorString(e);
        return -2;
    }
    out->bytes = Jp.size();
    return 0;
}

namespace {

// Permuted bias on the device (built once per instance from the caller's device bias) and its max |b|.
int ensure_bias_perm(TensorInstance* ti, const int32_t* bias, cudaStream_t st, std::string* why) {
    if (!bias || ti->d_bias_perm) return 0;
    if (capturing(st)) return setup_code(cudaErrorStreamCaptureUnsupported);
    std::vector<int32_t> b(ti->n), bp(ti->npp, 0);
    cudaError_t e = cudaMemcpy(b.data(), bias, size_t(ti->n) * 4, cudaMemcpyDeviceToHost);
    for (int i = 0; i < ti->n && e == cudaSuccess; ++i) bp[ti->perm[i]] = b[i];
    if (e == cudaSuccess) e = cudaMalloc(&ti->d_bias_perm, size_t(ti->npp) * 4);
    if (e == cudaSuccess) e = cudaMemcpy(ti->d_bias_perm, bp.data(), size_t(ti->npp) * 4, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        if (why) *why = std::string("bias: ") + cudaGetErrorString(e);
        if (ti->d_bias_perm) cudaFree(ti->d_bias_perm);
        ti->d_bias_perm = nullptr;
        return setup_code(e);
    }
    return 0;
}

int res_run(TensorInstance* ti, const TensorRun& r, cudaStream_t st, std::string* why) {
    const int npairs = ((r.nchains + kM - 1) / kM + 1) / 2;
    const int ngroups = 2 * npairs;
    int slots = 0;
    int rc = res_pair_slots(npairs, &slots);
    if (rc || slots < 1) {
        if (why) *why = "the resident tensor kernel cannot be co-resident on this device";
        return -2;
    }
    const size_t fbytes = size_t(ngroups) * kResSlices * 4;
    const size_t dbytes = size_t(ngroups) * 2 * kM * 2048;
    const size_t nbytes = size_t(ngroups) * 2 * kM * 128;
    const size_t need = 256 + fbytes + dbytes + nbytes + 256;
    ti->last_err = nullptr;
    cudaError_t e = ti->ws.ensure(need, st);
    if (e != cudaSuccess) {
        if (why) *why = std::string("workspace: ") + cudaGetErrorString(e);
        return setup_code(e);
    }
    uint8_t* base = ti->ws.p;
    int* err = reinterpret_cast<int*>(base);
    uint32_t* flags = reinterpret_cast<uint32_t*>(base + 256);
    int8_t* dbuf = reinterpret_cast<int8_t*>(base + 256 + ((fbytes + 255) / 256) * 256);
    int8_t* nlx = dbuf + dbytes;
    CUtensorMap mapD, mapNL, mapJ;
    if (!make_map(&mapD, dbuf, 2048, uint64_t(ngroups) * 2 * kM, kM) ||
        !make_map(&mapNL, nlx, 128, uint64_t(ngroups) * 2 * kM, kM) || !make_map(&mapJ, ti->d_J, 2048, 2048, kResYS)) {
        if (why) *why = "cuTensorMapEncodeTiled failed";
        return -2;
    }
    e = cudaMemsetAsync(r.out_spins, 0, size_t(r.nchains) * 64 * 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_sum_sh, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_sum_bs, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_flips, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(base, 0, 256 + fbytes, st);     // error word + flags
    if (e != cudaSuccess) {
        if (why) *why = std::string("memset: ") + cudaGetErrorString(e);
        return -2;
    }
    ResParams P{};
    P.n = ti->n;
    P.S = r.tab.S;
    P.npairs = npairs;
    P.fourT = r.tab.fourT;
    P.q = r.tab.q;
    P.kcorr = r.tab.kcorr;
    P.kconst = r.tab.kconst;
    P.hclamp = r.hclamp;
    P.bias_perm = r.bias ? ti->d_bias_perm : nullptr;
    P.seed = r.seed;
    P.trial_offset = r.trial_offset;
    P.nchains = r.nchains;
    P.flags = flags;
    P.dbuf = dbuf;
    P.nlx = nlx;
    P.out_spins = r.out_spins;
    P.out_sum_sh = reinterpret_cast<unsigned long long*>(r.out_sum_sh);
    P.out_sum_bs = reinterpret_cast<unsigned long long*>(r.out_sum_bs);
    P.out_flips = reinterpret_cast<unsigned long long*>(r.out_flips);
    P.out_trace = r.out_trace;
    P.out_h = r.out_h;
    P.err = err;
    P.prof = r.prof;
    P.wait_ns = r.wait_ns;
    auto fn = tensor_res_kernel;
    const size_t smem = res_smem_bytes();
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(kResSlices * slots);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, fn, mapD, mapNL, mapJ, P);
    if (e != cudaSuccess) {
        if (why) *why = std::string("launch: ") + cudaGetErrorString(e);
        return -2;
    }
    ti->last_err = err;
    ti->last_ctas = kResSlices * slots;
    ti->last_cluster = 1;
    return 0;
}

}  // namespace

int tensor_wave_chains(int n, int* out) {
    const int R = std::max(2048, ((n + 255) / 256) * 256) / 256;
    constexpr int kMany = 1 << 20;   // more groups than any device holds: the query returns the device's limit
    int slots = 0, rc = 0;
    *out = 0;
    if (stream_supported(n)) {
        *out = stream_wave_chains();
        return 0;
    }
    if (R == 8) {
        rc = res_pair_slots(kMany, &slots);        // two groups per 32-CTA pair slot
        *out = 2 * slots * kM;
    } else if (R == 12 || R == 16) {
        rc = R == 12 ? max_clusters_t<12>(&slots) : max_clusters_t<16>(&slots);   // one group per cluster
        *out = slots * kM;
    } else {
        rc = int(cudaErrorInvalidValue);
    }
    return rc;
}

int tensor_run(TensorInstance* ti, const TensorRun& r, cudaStream_t st, std::string* why) {
    const int np = ti->np, R = np / 256;
    int rc0 = ensure_bias_perm(ti, r.bias, st, why);
    if (rc0) return rc0;
    if (ti->stream) return stream_run(ti, r, r.bias ? ti->d_bias_perm : nullptr, st, why);
    if (R == 8) return res_run(ti, r, st, why);
    const int groups = (r.nchains + kM - 1) / kM;
    // workspace: exchange buffers, permuted bias, error word
    const size_t dbytes = size_t(groups) * 2 * kM * np;
    const size_t nlbytes = size_t(groups) * 2 * kC * kM * 4;
    ti->last_err = nullptr;
    cudaError_t e = ti->ws.ensure(dbytes + nlbytes + 256, st);
    if (e != cudaSuccess) {
        if (why) *why = std::string("workspace: ") + cudaGetErrorString(e);
        return setup_code(e);
    }
    int8_t* dbuf = reinterpret_cast<int8_t*>(ti->ws.p);
    int32_t* nlbuf = reinterpret_cast<int32_t*>(ti->ws.p + dbytes);
    int* err = reinterpret_cast<int*>(ti->ws.p + dbytes + nlbytes);
    CUtensorMap mapA, mapB;
    if (!make_map(&mapA, dbuf, uint64_t(np), uint64_t(groups) * 2 * kM, kM) ||
        !make_map(&mapB, ti->d_J, uint64_t(np), uint64_t(np), uint32_t(16 * R))) {
        if (why) *why = "cuTensorMapEncodeTiled failed";
        return -2;
    }
    const int words = np / 32;
    e = cudaMemsetAsync(r.out_spins, 0, size_t(r.nchains) * words * 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_sum_sh, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_sum_bs, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_flips, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, 4, st);
    if (e != cudaSuccess) {
        if (why) *why = std::string("memset: ") + cudaGetErrorString(e);
        return -2;
    }
    TensorParams P{};
    P.n = ti->n;
    P.np = np;
    P.R = R;
    P.nc = 16 * R;
    P.S = r.tab.S;
    P.fourT = r.tab.fourT;
    P.q = r.tab.q;
    P.kcorr = r.tab.kcorr;
    P.kconst = r.tab.kconst;
    P.hclamp = r.hclamp;
    P.bias_perm = r.bias ? ti->d_bias_perm : nullptr;
    P.seed = r.seed;
    P.trial_offset = r.trial_offset;
    P.nchains = r.nchains;
    P.dbuf = dbuf;
    P.nlbuf = nlbuf;
    P.out_spins = r.out_spins;
    P.out_sum_sh = reinterpret_cast<unsigned long long*>(r.out_sum_sh);
    P.out_sum_bs = reinterpret_cast<unsigned long long*>(r.out_sum_bs);
    P.out_flips = reinterpret_cast<unsigned long long*>(r.out_flips);
    P.out_trace = r.out_trace;
    P.out_h = r.out_h;
    P.err = err;
    P.prof = r.prof;
    int rc = -1;
    if (R == 12) rc = launch_t<12>(P, groups, mapA, mapB, st, why);   // NP = 2048 runs the resident kernel above
    else if (R == 16) rc = launch_t<16>(P, groups, mapA, mapB, st, why);
    if (rc) return rc;
    ti->last_err = err;
    ti->last_ctas = kC * groups;
    ti->last_cluster = kC;
    return 0;
}

int tensor_check_error(const int* err, cudaStream_t st, std::string* why) {
    if (!err) return 0;
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, err, 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        if (why) *why = std::string("error word: ") + cudaGetErrorString(e);
        return -2;
    }
    if (h) {
        if (why) *why = "a bounded device wait expired (code " + std::to_string(h) + ")";
        return -3;
    }
    return 0;
}

void tensor_free_instance(TensorInstance* ti) {
    if (!ti) return;
    if (ti->d_J) cudaFree(ti->d_J);
    if (ti->d_bias_perm) cudaFree(ti->d_bias_perm);
    ti->d_J = nullptr;
    ti->d_bias_perm = nullptr;
    ti->ws.free();
    ti->last_err = nullptr;
}

}  // namespace anc
