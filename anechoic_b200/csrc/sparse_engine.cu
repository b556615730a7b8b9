// Bit-exact SCA annealing of sparse instances (CSR rows): the plain engine's path for K = 0 (see anc_plain.cuh for the job
// and queue structures and the reference lines), in four forms. A step is a chain of dependent phases, so what bounds a
// launch depends on how many anneals share an SM (B200, us per step, R = 2000 spins of mean degree 20, phi 0.25):
//
// kSparseOne, one CTA of 512 threads per SM (plain_kernel, plain_engine.cu): up to one anneal per SM and NP <= 4096. 4.0 for 148.
// kSparseWide and kSparseHalf (sparse_wide_kernel): one CTA of 1024 threads or two of 512. 8 warps own the RNG lanes and make the
//   next step's draws while the others decide the current step's slots, which then need not follow the lanes' rounds.
//   20000-spin torus: 13.8 for up to 148 anneals (16.1 on the CTA of 512 threads); 296 anneals of R: 5.8 (8.0 in two waves).
// kSparseNarrow (sparse_kernel): several anneals per SM, 256 threads each, one per RNG lane, at most 64 registers and 6.25 bytes
//   of shared memory per slot. Every warp keeps its own flip list, so a step takes two CTA barriers. 600 anneals of R: 14.2
//   (19.7 in waves of one per SM); bound by issue slots (72 % busy), most of them in applying edges.
// kSparseGroups (sparse_group_kernel): eight replicas of an instance per CTA with pulled, packed updates (below): 2368 anneals of
//   R: 23.2 (63.3 in waves of one per SM, 43 in the narrow form); it needs unit weights and rows of at most kGroupDegree edges.
// sparse_form picks one by the anneals per SM, the size and the row length.
#include <algorithm>

#include "anc_plain.cuh"

namespace anc {
namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr int kNarrow = 256;
constexpr int kMaxChunks = 4;              // 32-round words of a thread's bits: NP <= 32768

// log2 of the lanes per row: the power of two at or above mean degree (in fetched words) / SE, at most 32.
template <int SE>
__device__ __forceinline__ int lanes_log2(int words, int n) {
    const int deg = (words + SE * n - 1) / (SE * max(n, 1));
    int lg = 0;
    while (lg < 5 && (1 << lg) < deg) ++lg;
    return lg;
}

// One word of edges: (y << 8) | uint8(J), or with E16 two edges y | [J = -1] << 15 (y >= kEdgePad: no edge).
template <bool E16>
__device__ __forceinline__ void apply_word(uint32_t v, int32_t m, int32_t* h) {
    if (E16) {
        const uint32_t lo = v & 0xffffu, hi = v >> 16;
        if (~lo & kEdgePad) atomicAdd(&h[lo & 0x7fffu], (lo >> 15) ? -m : m);
        if (~hi & kEdgePad) atomicAdd(&h[hi & 0x7fffu], (hi >> 15) ? -m : m);
    } else {
        atomicAdd(&h[v >> 8], m * int32_t(int8_t(v & 0xffu)));
    }
}

// Field update by one warp: h_y += m J_xy over the rows x of its nf list entries (slot | [new spin -1] << 15), m = mult
// with the new spin's sign. Groups of 2^lg lanes take SB rows each: first the bounds of all, then SE words per lane of
// each, and only then the atomics, so a warp keeps many fetches in flight.
template <int SB, int SE, bool E16>
__device__ __forceinline__ void row_pass(const int32_t* __restrict__ row_ptr, const uint32_t* __restrict__ adj,
                                         const uint16_t* list, int nf, int lg, int32_t* h, int mult, int lane) {
    const int G = 1 << lg, sub = lane & (G - 1), NG = 32 >> lg;
    for (int f0 = lane >> lg; f0 < nf; f0 += NG * SB) {
        int k0[SB], k1[SB];
        int32_t m[SB];
        uint32_t a[SB][SE];
#pragma unroll
        for (int b = 0; b < SB; ++b) {
            const int f = f0 + b * NG;
            k0[b] = 0;
            k1[b] = 0;
            m[b] = 0;
            if (f < nf) {
                const uint32_t e = list[f];
                const int x = int(e & 0x7fffu);
                m[b] = (e >> 15) ? -mult : mult;
                k0[b] = __ldg(row_ptr + x) + sub;
                k1[b] = __ldg(row_ptr + x + 1);
            }
        }
#pragma unroll
        for (int b = 0; b < SB; ++b)
#pragma unroll
            for (int e = 0; e < SE; ++e) a[b][e] = k0[b] + e * G < k1[b] ? __ldg(adj + k0[b] + e * G) : 0u;
#pragma unroll
        for (int b = 0; b < SB; ++b) {
#pragma unroll
            for (int e = 0; e < SE; ++e)
                if (k0[b] + e * G < k1[b]) apply_word<E16>(a[b][e], m[b], h);
            for (int k = k0[b] + SE * G; k < k1[b]; k += G) apply_word<E16>(__ldg(adj + k), m[b], h);
        }
    }
}

template <int SB, int SE>
__device__ __forceinline__ void rows(const PlainJob& job, const uint16_t* list, int nf, int lg, int32_t* h, int mult,
                                     int lane) {
    if (job.csr16) row_pass<SB, SE, true>(job.row_ptr, job.adj, list, nf, lg, h, mult, lane);
    else row_pass<SB, SE, false>(job.row_ptr, job.adj, list, nf, lg, h, mult, lane);
}

__device__ __forceinline__ int64_t warp_sum64(int64_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// The next work item of the launch's queue, or nitems when it is empty; called by every thread.
__device__ __forceinline__ int next_item(const PlainLaunch& L, int* s_item) {
    __syncthreads();
    if (threadIdx.x == 0) *s_item = atomicAdd(L.next_item, 1);
    __syncthreads();
    return *s_item;
}

template <int SB, int SE>
__global__ void __launch_bounds__(kNarrow, 4) sparse_kernel(const __grid_constant__ PlainLaunch L) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ int s_item, s_lin[8];
    __shared__ long long s_red[3][8];
    int32_t* h = reinterpret_cast<int32_t*>(smem_raw);                       // [np_max]
    uint32_t* Sb = reinterpret_cast<uint32_t*>(h + L.np_max);                // [chunks][256] spin bits (1 = up) by round
    const int chunks_max = (L.np_max / kLanes + 31) / 32;
    uint32_t* Db = Sb + chunks_max * kLanes;                                 // [chunks][256] flipped in the last step
    uint16_t* lists = reinterpret_cast<uint16_t*>(Db + chunks_max * kLanes); // [8][np_max / 8]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (int item = next_item(L, &s_item); item < L.nitems; item = next_item(L, &s_item)) {
        const int2 it = L.items ? L.items[item] : make_int2(0, item);
        const PlainJob& job = L.items ? L.jobs[it.x] : L.job0;
        const int n = job.n, np = job.np, R = np / kLanes, S = job.tab.S, c = it.y;
        const int32_t hclamp = job.hclamp;
        const int32_t* __restrict__ bias = job.bias;
        int32_t* trace_out = (job.trace && job.out_trace) ? job.out_trace + size_t(c) * S : nullptr;
        uint16_t* list = lists + warp * (np / 8);
        const int lg = lanes_log2<SE>(__ldg(job.row_ptr + n), n);

        for (int i = tid; i < np; i += kNarrow) h[i] = (i < n && bias) ? bias[i] : 0;
        // initial spins (draw >> 31; padding +1), s_prev = +1 everywhere, initial flips = all active slots
        Xoshiro rng;
        rng_seed(rng, job.seed, job.trial_offset + uint32_t(c), uint32_t(tid));
        int cnt = 0;
        for (int k0 = 0; k0 < R; k0 += 32) {
            uint32_t s = 0u, d = 0u;
            const int ke = min(32, R - k0);
            for (int k = 0; k < ke; ++k) {
                const uint32_t r = rng_next(rng);
                const int i = (k0 + k) * kLanes + tid;
                const bool valid = i < n;
                const uint32_t up = valid ? (r >> 31) : 1u;
                s |= up << k;
                d |= (valid && !up ? 1u : 0u) << k;
                const uint32_t b = __ballot_sync(FULL, valid);
                if (valid) list[cnt + __popc(b & lanemask_lt())] = uint16_t(i | ((up ^ 1u) << 15));
                cnt += __popc(b);
            }
            Sb[(k0 >> 5) * kLanes + tid] = s;
            Db[(k0 >> 5) * kLanes + tid] = d;
        }
        __syncthreads();
        rows<SB, SE>(job, list, cnt, lg, h, 1, lane);
        __syncthreads();

        int32_t nlin_prev = 0;
        long long flips = 0;
        for (int t = 0; t < S; ++t) {
            const int32_t fourT = __ldg(job.tab.fourT + t), twoT = fourT >> 1, qv = __ldg(job.tab.q + t);
            const int32_t corr = step_corr(nlin_prev, __ldg(job.tab.kcorr + t), __ldg(job.tab.kconst + t));
            const int32_t xs = qv - corr, twocorr = 2 * corr, c1 = twoT - 1;
            const uint32_t lw = uint32_t(2 * twoT - 1);
            int nl = 0;
            cnt = 0;
            for (int k0 = 0; k0 < R; k0 += 32) {
                uint32_t* sp = Sb + (k0 >> 5) * kLanes + tid;
                uint32_t* dp = Db + (k0 >> 5) * kLanes + tid;
                const uint32_t s = *sp, d = *dp;
                uint32_t f = 0u;
                const int ke = min(32, R - k0);
#pragma unroll 2
                for (int k = 0; k < ke; ++k) {
                    const uint32_t u = rng_next(rng);
                    const int i = (k0 + k) * kLanes + tid;
                    const int32_t hv = h[i];
                    const uint32_t up = (s >> k) & 1u;
                    int32_t hs = up ? hv : -hv;
                    if (hclamp > 0) hs = max(-hclamp, min(hs, hclamp));
                    int32_t zt = hs * 65536 + xs;                       // q - (s == s_prev ? corr : -corr)
                    if ((d >> k) & 1u) zt += twocorr;
                    const int32_t thr = __mulhi(int32_t((u & 0xffff0000u) ^ 0x80000000u), fourT);
                    const bool valid = i < n;
                    const bool fl = valid && zt < thr;
                    nl += (valid && uint32_t(zt + c1) < lw) ? 1 : 0;
                    const uint32_t fb = __ballot_sync(FULL, fl);
                    if (fl) {
                        list[cnt + __popc(fb & lanemask_lt())] = uint16_t(uint32_t(i) | (up << 15));
                        f |= 1u << k;
                    }
                    cnt += __popc(fb);
                }
                *sp = s ^ f;
                *dp = f;
            }
            nl = __reduce_add_sync(FULL, nl);
            if (lane == 0) s_lin[warp] = nl;
            flips += cnt;
            __syncthreads();
            nlin_prev = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w) nlin_prev += s_lin[w];
            if (tid == 0 && trace_out) trace_out[t] = nlin_prev;
            rows<SB, SE>(job, list, cnt, lg, h, 2, lane);
            __syncthreads();
        }
        // outputs
        long long sh = 0, bs = 0;
        for (int k = 0; k < R; ++k) {
            const int i = k * kLanes + tid;
            const bool valid = i < n, up = (Sb[(k >> 5) * kLanes + tid] >> (k & 31)) & 1u;
            if (valid) {
                const int32_t hv = h[i];
                sh += up ? hv : -hv;
                if (bias) bs += up ? bias[i] : -bias[i];
                if (job.out_h) job.out_h[size_t(c) * n + i] = hv;
            }
            const uint32_t w = __ballot_sync(FULL, valid && up);
            if (lane == 0) job.out_spins[size_t(c) * job.nw + k * 8 + warp] = w;
        }
        sh = warp_sum64(sh);
        bs = warp_sum64(bs);
        if (lane == 0) {
            s_red[0][warp] = sh;
            s_red[1][warp] = bs;
            s_red[2][warp] = flips;
        }
        __syncthreads();
        if (tid == 0) {
            long long a = 0, b = 0, f = 0;
            for (int w = 0; w < 8; ++w) { a += s_red[0][w]; b += s_red[1][w]; f += s_red[2][w]; }
            job.out_sum_sh[c] = a;
            job.out_sum_bs[c] = b;
            job.out_flips[c] = f;
        }
    }
}

// TW threads: warps 0 .. 7 own the RNG lanes, the ND others the slots.
template <int TW, int SB, int SE>
__global__ void __launch_bounds__(TW, 1024 / TW) sparse_wide_kernel(const __grid_constant__ PlainLaunch L) {
    constexpr int NW = TW / 32, ND = NW - 8, LPR = ND / 8;      // LPR lists per RNG warp
    static_assert(ND >= 8 && ND % 8 == 0, "each RNG warp helps LPR deciding warps with their rows");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ int s_item, s_lin[ND], s_cnt[ND];
    __shared__ long long s_red[3][NW];
    const int cap = (L.np_max / 32 + ND - 1) / ND * 32;
    int32_t* h = reinterpret_cast<int32_t*>(smem_raw);                            // [np_max]
    uint32_t* Sw = reinterpret_cast<uint32_t*>(h + L.np_max);                     // [np_max / 32] spins (1 = up)
    uint32_t* Dw = Sw + L.np_max / 32;                                            // [np_max / 32] flipped in the last step
    uint16_t* draws = reinterpret_cast<uint16_t*>(Dw + L.np_max / 32);            // [2][np_max] top 16 bits of a step's draws
    uint16_t* lists = draws + 2 * L.np_max;                                       // [ND][cap]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool drawer = warp < 8;
    const int w0 = warp - 8;                                                      // deciding warp: words w0, w0 + ND, ...

    for (int item = next_item(L, &s_item); item < L.nitems; item = next_item(L, &s_item)) {
        const int2 it = L.items ? L.items[item] : make_int2(0, item);
        const PlainJob& job = L.items ? L.jobs[it.x] : L.job0;
        const int n = job.n, np = job.np, R = np / kLanes, nw = np / 32, S = job.tab.S, c = it.y;
        const int32_t hclamp = job.hclamp;
        const int32_t* __restrict__ bias = job.bias;
        int32_t* trace_out = (job.trace && job.out_trace) ? job.out_trace + size_t(c) * S : nullptr;
        const int lg = lanes_log2<SE>(__ldg(job.row_ptr + n), n);
        Xoshiro rng;
        auto draw_step = [&](uint16_t* to) {
#pragma unroll 4
            for (int k = 0; k < R; ++k) to[k * kLanes + tid] = uint16_t(rng_next(rng) >> 16);
        };
        // a deciding warp does the first 3/4 of its rows (half with ND = 8), its RNG warp the rest
        auto update = [&](int mult) {
            if (drawer) {
                for (int j = 0; j < LPR; ++j) {
                    const int w = warp * LPR + j, nf = s_cnt[w], own = nf - nf / (LPR + 1);
                    rows<SB, SE>(job, lists + w * cap + own, nf - own, lg, h, mult, lane);
                }
            } else {
                const int nf = s_cnt[w0];
                rows<SB, SE>(job, lists + w0 * cap, nf - nf / (LPR + 1), lg, h, mult, lane);
            }
        };
        for (int i = tid; i < np; i += TW) h[i] = (i < n && bias) ? bias[i] : 0;
        if (drawer) {
            rng_seed(rng, job.seed, job.trial_offset + uint32_t(c), uint32_t(tid));
            draw_step(draws);
        }
        __syncthreads();
        long long flips = 0;
        if (drawer) {
            draw_step(draws + np);
        } else {
            // initial spins (draw >> 31; padding +1), s_prev = +1 everywhere, initial flips = all active slots
            uint16_t* list = lists + w0 * cap;
            int cnt = 0;
            for (int wi = w0; wi < nw; wi += ND) {
                const int i = 32 * wi + lane;
                const bool valid = i < n;
                const uint32_t up = valid ? uint32_t(draws[i]) >> 15 : 1u;
                const uint32_t sb = __ballot_sync(FULL, up != 0), vb = __ballot_sync(FULL, valid);
                if (lane == 0) {
                    Sw[wi] = sb;
                    Dw[wi] = vb & ~sb;
                }
                if (valid) list[cnt + __popc(vb & lanemask_lt())] = uint16_t(uint32_t(i) | ((up ^ 1u) << 15));
                cnt += __popc(vb);
            }
            if (lane == 0) s_cnt[w0] = cnt;
        }
        __syncthreads();
        update(1);
        __syncthreads();

        int32_t nlin_prev = 0;
        for (int t = 0; t < S; ++t) {
            if (drawer) {
                if (t + 1 < S) draw_step(draws + (t & 1) * np);        // step t + 1's draws; step t reads the other half
            } else {
                const uint16_t* dr = draws + ((t + 1) & 1) * np;
                const int32_t fourT = __ldg(job.tab.fourT + t), twoT = fourT >> 1, qv = __ldg(job.tab.q + t);
                const int32_t corr = step_corr(nlin_prev, __ldg(job.tab.kcorr + t), __ldg(job.tab.kconst + t));
                const int32_t xs = qv - corr, twocorr = 2 * corr, c1 = twoT - 1;
                const uint32_t lw = uint32_t(2 * twoT - 1);
                uint16_t* list = lists + w0 * cap;
                int cnt = 0, nl = 0;
#pragma unroll 4
                for (int wi = w0; wi < nw; wi += ND) {
                    const int i = 32 * wi + lane;
                    const uint32_t Sword = Sw[wi], Dword = Dw[wi];
                    const int32_t hv = h[i];
                    const int32_t thr = __mulhi(int32_t((uint32_t(dr[i]) << 16) ^ 0x80000000u), fourT);
                    const uint32_t up = (Sword >> lane) & 1u;
                    int32_t hs = up ? hv : -hv;
                    if (hclamp > 0) hs = max(-hclamp, min(hs, hclamp));
                    int32_t zt = hs * 65536 + xs;
                    if ((Dword >> lane) & 1u) zt += twocorr;
                    const bool valid = i < n;
                    const bool fl = valid && zt < thr;
                    nl += (valid && uint32_t(zt + c1) < lw) ? 1 : 0;
                    const uint32_t fb = __ballot_sync(FULL, fl);
                    if (lane == 0) {
                        Sw[wi] = Sword ^ fb;
                        Dw[wi] = fb;
                    }
                    if (fl) list[cnt + __popc(fb & lanemask_lt())] = uint16_t(uint32_t(i) | (up << 15));
                    cnt += __popc(fb);
                }
                nl = __reduce_add_sync(FULL, nl);
                if (lane == 0) {
                    s_lin[w0] = nl;
                    s_cnt[w0] = cnt;
                }
                flips += cnt;
            }
            __syncthreads();
            nlin_prev = __reduce_add_sync(FULL, lane < ND ? s_lin[lane] : 0);
            if (tid == 0 && trace_out) trace_out[t] = nlin_prev;
            update(2);
            __syncthreads();
        }
        // outputs
        long long sh = 0, bs = 0;
        for (int wi = warp; wi < nw; wi += NW) {
            const int i = 32 * wi + lane;
            const bool valid = i < n, up = (Sw[wi] >> lane) & 1u;
            if (valid) {
                const int32_t hv = h[i];
                sh += up ? hv : -hv;
                if (bias) bs += up ? bias[i] : -bias[i];
                if (job.out_h) job.out_h[size_t(c) * n + i] = hv;
            }
            const uint32_t w = __ballot_sync(FULL, valid && up);
            if (lane == 0) job.out_spins[size_t(c) * job.nw + wi] = w;
        }
        sh = warp_sum64(sh);
        bs = warp_sum64(bs);
        if (lane == 0) {
            s_red[0][warp] = sh;
            s_red[1][warp] = bs;
            s_red[2][warp] = flips;
        }
        __syncthreads();
        if (tid == 0) {
            long long a = 0, b = 0, f = 0;
            for (int w = 0; w < NW; ++w) { a += s_red[0][w]; b += s_red[1][w]; f += s_red[2][w]; }
            job.out_sum_sh[c] = a;
            job.out_sum_bs[c] = b;
            job.out_flips[c] = f;
        }
    }
}

// Eight replicas of an instance per CTA of 512 threads, four per thread: thread (RNG lane l, quad q) decides the lane's slots
// for replicas 4q .. 4q + 3. The updates are pulled: each step a slot sums what its neighbours did in the last one, so there
// are no atomics and one CTA barrier per step (a step reads one half of `moves` and writes the other). A slot's moves of
// four replicas are the bytes of one word (1 + s'_x for a flip to s'_x, else 1). With P the sum of the words of a row's +
// edges and N of its - edges, every byte of P - N + 2 (minus edges) is sum_x J_xy s'_x over the flips plus the row's edge
// count, in 0 .. 240 for rows of up to 120 edges, so one 32-bit sum holds the four bytes whatever borrows it had on the way.
// The kernel is bound by issue slots (ncu: IPC 2.7 of 4), so what a word of two edges costs counts: the rows are stored in
// slices of 32 with the same number of words for all (padding edges name one of 32 words that hold 0), so a warp's loop has
// no per-lane conditions and its loads are coalesced, and an edge is a byte offset into `moves`.
// The fields, 4 h + 2 [flipped last step] + [s = +1], are in global memory: each thread touches its own slots only, a
// round ahead of their use and past L1, which keeps the rows.
constexpr int kQuads = kGroupReplicas / 4, kGroupThreads = 256 * kQuads;

// 32-bit shared-memory accesses by address (through the generic pointer the compiler rebuilt the base at every access)
__device__ __forceinline__ int32_t lds32(uint32_t addr) {
    int32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v)); }

template <int WE, bool CLAMP>
__global__ void __launch_bounds__(kGroupThreads, 4 / kQuads) sparse_group_kernel(const __grid_constant__ PlainLaunch L) {
    constexpr int Q = kQuads, TPB = kGroupThreads, NR = kGroupReplicas;
    static_assert(Q == 2, "edges are offsets of 8 bytes a slot");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ int s_item;
    __shared__ uint32_t s_cnt[3][NR];          // a step's counts per replica, each below 2^16: n_lin | flips << 16
    __shared__ unsigned long long s_red[2][NR];
    __shared__ long long s_fl[NR];             // flips so far; thread r alone uses replica r's
    const uint32_t half = uint32_t(L.np_max + 32) * 4 * Q;                   // bytes of a half of moves
    const uint32_t base = uint32_t(__cvta_generic_to_shared(smem_raw));
    int4* h = reinterpret_cast<int4*>(L.group_h) + size_t(blockIdx.x) * L.np_max * Q + threadIdx.x;
    const int tid = threadIdx.x, lane = tid & 31;
    const int l = tid / Q, q = tid % Q;
    const uint32_t quad_lanes = 0x55555555u << q;                            // the warp's lanes of this quad

    for (int item = next_item(L, &s_item); item < L.nitems; item = next_item(L, &s_item)) {
        const int2 it = L.items ? L.items[item] : make_int2(0, NR * item);
        const PlainJob& job = L.items ? L.jobs[it.x] : L.job0;
        const int n = job.n, np = job.np, R = np / kLanes, RA = (n + kLanes - 1) / kLanes, S = job.tab.S, c0 = it.y + 4 * q;
        const int32_t hclamp = job.hclamp > 0 ? job.hclamp : 0x7fffffff;     // 0: the job's fields need no clamp
        const int32_t* __restrict__ bias = job.bias;
        const uint32_t* __restrict__ row_c = job.row_counts;
        const uint2* __restrict__ slice_t = job.slice_info + (l >> 5);       // slice 8 k + l / 32
        const uint32_t* __restrict__ words = job.slices + (l & 31);
        const bool tracer = job.trace && job.out_trace && tid < NR && it.y + tid < job.ntrials;

        // initial spins (draw >> 31), s_prev = +1: the first step's moves are s0 itself, with factor 1
        Xoshiro rng[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) rng_seed(rng[r], job.seed, job.trial_offset + uint32_t(c0 + r), uint32_t(l));
        for (int k = 0; k < R; ++k) {
            const int y = k * kLanes + l;
            const bool valid = y < n;
            const int b4 = (valid && bias) ? bias[y] * 4 : 0;
            uint32_t w = 0u;
            int hv[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint32_t u = rng_next(rng[r]);
                const uint32_t up = valid ? (u >> 31) : 1u;
                w |= (2u * up) << (8 * r);
                hv[r] = b4 + int(up ? 1u : 2u);
            }
            reinterpret_cast<uint32_t*>(smem_raw)[k * TPB + tid] = w;
            __stcg(h + k * TPB, make_int4(hv[0], hv[1], hv[2], hv[3]));
        }
        if (tid < 32 * Q) {                       // the words that padding edges name
            reinterpret_cast<uint32_t*>(smem_raw)[np * Q + tid] = 0u;
            reinterpret_cast<uint32_t*>(smem_raw + half)[np * Q + tid] = 0u;
        }
        if (tid < 3 * NR) (&s_cnt[0][0])[tid] = 0u;
        if (tid < NR) s_fl[tid] = 0;
        if (tid < 2 * NR) (&s_red[0][0])[tid] = 0ull;
        __syncthreads();

        // signed sum of the row's words of this quad in the half at byte offset cur, bytes offset by the row's edges
        auto row_sum = [&](uint32_t cur, uint2 sl, uint32_t rc) {
            const uint32_t* a = words + sl.x;
            const uint32_t at = base + cur + uint32_t(4 * q);
            auto part = [&](int cnt) {
                int32_t p = 0;
                auto add = [&](uint32_t word) { p += lds32(at + (word & 0xffffu)) + lds32(at + (word >> 16)); };
                for (; cnt >= WE; cnt -= WE, a += WE * 32) {
                    uint32_t v[WE];
#pragma unroll
                    for (int j = 0; j < WE; ++j) v[j] = __ldg(a + j * 32);
#pragma unroll
                    for (int j = 0; j < WE; ++j) add(v[j]);
                }
                if (WE > 1)
                    for (; cnt > 0; --cnt, a += 32) add(__ldg(a));
                return p;
            };
            const int32_t plus = part(int(sl.y & 0xffffu)), minus = part(int(sl.y >> 16));
            return uint32_t(plus - minus) + (rc >> 8) * 0x02020202u;
        };
        for (int t = 0; t < S; ++t) {
            const uint32_t cur = (t & 1) ? half : 0u;
            const uint32_t nxt = base + (half - cur) + uint32_t(4 * tid);
            const int32_t mult4 = t == 0 ? 4 : 8;                           // 4 x the update's factor (1, then 2)
            const int32_t fourT = __ldg(job.tab.fourT + t), qv = __ldg(job.tab.q + t), c1 = (fourT >> 1) - 1;
            const uint32_t lw = uint32_t(2 * (fourT >> 1) - 1);
            int32_t corr[4];
            {
                const int64_t kcorr = __ldg(job.tab.kcorr + t);
                const int32_t kconst = __ldg(job.tab.kconst + t);
#pragma unroll
                for (int r = 0; r < 4; ++r) corr[r] = step_corr(t ? int(s_cnt[(t + 2) % 3][4 * q + r] & 0xffffu) : 0, kcorr, kconst);
            }
            uint32_t nl = 0u, nf = 0u;                                      // a byte per replica: RA <= 31
            uint2 sn = __ldg(slice_t);
            uint32_t rn = l < n ? __ldg(row_c + l) : 0u;
#pragma unroll 1
            for (int k = 0; k < RA; ++k) {
                const int y = k * kLanes + l;
                const bool valid = y < n;
                const uint2 sl = sn;
                const uint32_t rc = rn;
                const int4 old = __ldcg(h + k * TPB);
                if (k + 1 < RA) {
                    sn = __ldg(slice_t + 8 * (k + 1));
                    rn = y + kLanes < n ? __ldg(row_c + y + kLanes) : 0u;
                }
                const uint32_t sum = row_sum(cur, sl, rc);
                const int32_t less = mult4 * int32_t(rc & 0xffu);
                int hv[4] = {old.x - less, old.y - less, old.z - less, old.w - less};
                uint32_t w = 0x01010101u;
                const int32_t vm = valid ? -1 : 0;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    // branch-free: flipped = -1 / 0 from the sign of z - r, which the range plan keeps inside int32
                    const int32_t g = hv[r] + mult4 * int32_t((sum >> (8 * r)) & 0xffu);       // 4 h + the state bits
                    const int32_t s1 = 2 * (g & 1) - 1;                                         // s
                    int32_t zt = (g & 2) ? qv + corr[r] : qv - corr[r];
                    if (CLAMP) zt += max(-hclamp, min((g >> 2) * s1, hclamp)) * 65536;
                    else zt += (g & ~3) * (s1 * 16384);
                    const uint32_t u = rng_next(rng[r]);
                    const int32_t thr = __mulhi(int32_t((u & 0xffff0000u) ^ 0x80000000u), fourT);
                    const int32_t flipped = ((zt - thr) >> 31) & vm;
                    nf -= uint32_t(flipped) << (8 * r);
                    nl += (valid & (uint32_t(zt + c1) < lw)) ? 1u << (8 * r) : 0u;
                    w += uint32_t(flipped * s1) << (8 * r);                                     // byte 1 - s for a flip
                    hv[r] = (g & ~2) ^ (flipped & 3);
                }
                sts32(nxt + uint32_t(4 * TPB) * uint32_t(k), w);
                __stcg(h + k * TPB, make_int4(hv[0], hv[1], hv[2], hv[3]));
            }
            for (int k = RA; k < R; ++k)                // rounds of padding slots only draw
#pragma unroll
                for (int r = 0; r < 4; ++r) rng_next(rng[r]);
            // per-replica counts of the warp: 16 lanes x 31 rounds fit 16 bits
            const uint32_t n02 = __reduce_add_sync(quad_lanes, nl & 0x00ff00ffu), n13 = __reduce_add_sync(quad_lanes, (nl >> 8) & 0x00ff00ffu);
            const uint32_t f02 = __reduce_add_sync(quad_lanes, nf & 0x00ff00ffu), f13 = __reduce_add_sync(quad_lanes, (nf >> 8) & 0x00ff00ffu);
            if (lane < Q) {
                uint32_t* sc4 = &s_cnt[t % 3][4 * q];
                atomicAdd(sc4, (n02 & 0xffffu) | f02 << 16);
                atomicAdd(sc4 + 1, (n13 & 0xffffu) | f13 << 16);
                atomicAdd(sc4 + 2, n02 >> 16 | (f02 & 0xffff0000u));
                atomicAdd(sc4 + 3, n13 >> 16 | (f13 & 0xffff0000u));
            }
            if (tid < NR) s_cnt[(t + 1) % 3][tid] = 0u;     // last read before the previous barrier
            __syncthreads();
            if (tid < NR) {
                const uint32_t sc = s_cnt[t % 3][tid];
                if (tracer) job.out_trace[size_t(it.y + tid) * S + t] = int32_t(sc & 0xffffu);
                s_fl[tid] += sc >> 16;
            }
        }
        // the last step's moves into the fields, and the outputs
        const uint32_t cur = (S & 1) ? half : 0u;
        long long sh[4] = {0, 0, 0, 0}, bs[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int k = 0; k < R; ++k) {
            const int y = k * kLanes + l;
            const bool valid = y < n;
            uint32_t sum = 0u, rc = 0u;
            if (k < RA) {                                   // uniform: a slice exists for every active round
                rc = valid ? __ldg(row_c + y) : 0u;
                sum = row_sum(cur, __ldg(slice_t + 8 * k), rc);
            }
            const int4 old = __ldcg(h + k * TPB);
            const int hv[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int32_t hf = (hv[r] + 8 * (int32_t((sum >> (8 * r)) & 0xffu) - int32_t(rc & 0xffu))) >> 2;
                const bool up = hv[r] & 1, writer = c0 + r < job.ntrials;
                if (valid) {
                    sh[r] += up ? hf : -hf;
                    if (bias) bs[r] += up ? bias[y] : -bias[y];
                    if (job.out_h && writer) job.out_h[size_t(c0 + r) * n + y] = hf;
                }
                // bits 2 j + q of the ballot are this quad's lanes j = 0 .. 15 of the warp
                uint32_t x = (__ballot_sync(FULL, valid && up) >> q) & 0x55555555u;
                x = (x | (x >> 1)) & 0x33333333u;
                x = (x | (x >> 2)) & 0x0f0f0f0fu;
                x = (x | (x >> 4)) & 0x00ff00ffu;
                x = (x | (x >> 8)) & 0xffffu;
                if (lane < Q && writer)
                    reinterpret_cast<uint16_t*>(job.out_spins + size_t(c0 + r) * job.nw + k * 8)[tid >> 5] = uint16_t(x);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            atomicAdd(&s_red[0][4 * q + r], static_cast<unsigned long long>(sh[r]));
            if (bias) atomicAdd(&s_red[1][4 * q + r], static_cast<unsigned long long>(bs[r]));
        }
        __syncthreads();
        if (tid < NR && it.y + tid < job.ntrials) {
            job.out_sum_sh[it.y + tid] = int64_t(s_red[0][tid]);
            job.out_sum_bs[it.y + tid] = int64_t(s_red[1][tid]);
            job.out_flips[it.y + tid] = s_fl[tid];
        }
    }
}

// ------------------------------------------------------------------------------------------------ host side
using SparseFn = void (*)(const PlainLaunch);

SparseFn narrow_fn(int variant) {
    switch (variant) {
        case 1: return sparse_kernel<1, 4>;
        case 2: return sparse_kernel<2, 4>;
        case 3: return sparse_kernel<1, 16>;
        default: return sparse_kernel<1, 8>;
    }
}
template <int TW>
SparseFn wide_fn(int variant) {
    switch (variant) {
        case 1: return sparse_wide_kernel<TW, 1, 4>;
        case 2: return sparse_wide_kernel<TW, 2, 4>;
        case 3: return sparse_wide_kernel<TW, 1, 16>;
        default: return sparse_wide_kernel<TW, 1, 8>;
    }
}

template <bool CLAMP>
SparseFn group_fn(int variant) {
    switch (variant) {
        case 1: return sparse_group_kernel<2, CLAMP>;
        case 2: return sparse_group_kernel<3, CLAMP>;
        case 3: return sparse_group_kernel<6, CLAMP>;
        default: return sparse_group_kernel<4, CLAMP>;
    }
}

size_t narrow_smem(int np) { return size_t(np) * 6 + size_t((np / kLanes + 31) / 32) * kLanes * 8; }
size_t wide_smem(int np, int tw) {
    const int nd = tw / 32 - 8;
    return size_t(np) * 8 + size_t(np / 32) * 8 + size_t(nd) * ((np / 32 + nd - 1) / nd * 32) * 2;
}

constexpr size_t kSmemLimit = 224 * 1024;
bool wide_fits(int np) { return wide_smem(np, 1024) <= kSmemLimit; }
bool half_fits(int np) { return 2 * (wide_smem(np, 512) + 2048) <= kSmemLimit; }
size_t group_smem(int np) { return size_t(np + 32) * 2 * kGroupReplicas; }
int group_per_sm(int np) { return int(std::min<size_t>(1024 / kGroupThreads, kSmemLimit / (group_smem(np) + 1024))); }
int group_ctas(int np, int nitems, int sms) { return std::min(nitems, group_per_sm(np) * sms); }

}  // namespace

int sparse_max_blocks_per_sm(int np_max, int* out) {
    *out = 0;
    int least = 1 << 30;
    for (int v = 0; v < kSparseVariants; ++v) {
        SparseFn fn = narrow_fn(v);
        cudaError_t e = allow_max_smem(fn);
        int b = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, kNarrow, narrow_smem(np_max));
        if (e != cudaSuccess) return int(e);
        least = b < least ? b : least;
    }
    *out = least;
    return 0;
}

size_t sparse_group_scratch(int np_max, int nitems, int sms) {
    return size_t(np_max) * kGroupReplicas * group_ctas(np_max, nitems, sms);
}

// Where groups are the quickest form: from about five or six anneals per SM with long rows, where every CTA has few groups' worth
// of gathers to hide behind each other, else from eight. us per step, groups / narrow form: degree 20, n = 2000: 21.8 / 18.4 for
// 900 anneals, 21.9 / 26.3 for 1184, 41 / 44 for 2400; degree 32, n = 2000: 23 / 23 for 740 and 23 / 26 for 900; degree 48,
// n = 4000: 54 / 51 for 740, 55 / 64 for 1184; degree 4: 14.6 / 10.2 for 1200 at n = 2000. Above NP = 7072 an SM holds one group
// CTA, so a launch of several waves pays only if the last is nearly full: n = 7900, degree 20: 66 / 81 for 1184 anneals,
// 129 / 109 for 1600. A batch counts all its anneals and passes a degree of at least 8: mixed with others the short rows gain
// too (51 instances: 41 ms, against 46 with the short ones in the narrow form).
bool sparse_groups(int np, double degree, int64_t anneals, int sms) {
    if (np > kGroupNp || degree < 8.0 || anneals < (degree >= 48.0 ? 6 : degree >= 32.0 ? 5 : 8) * int64_t(sms)) return false;
    const int64_t groups = (anneals + kGroupReplicas - 1) / kGroupReplicas, waves = (groups + sms - 1) / sms;
    return waves == 1 || group_per_sm(np) > 1 || 10 * groups >= 8 * sms * waves;
}

// The other forms, us per step, one / wide / half / narrow (B200, phi 0.25; - where it does not fit):
//   one anneal per SM: the wide form gains above NP = 4096, n = 5500 .. 20000: 14 .. 41 / 11 .. 33 at degree 4;
//   two: half where two fit (NP <= 10880), n = 2000, degree 20: 8.7 / 8.7 / 6.2 / 9, else wide in two waves: n = 12000,
//     degree 20: 42 / 34 / - / 45;
//   three: narrow, n = 10000, degree 20: 54 / 44 / 44 / 42, except that long rows of 32-bit edges make three of its CTAs slower
//     than two halves while few SMs have three: n = 800, 80 edges, 310 anneals: 15.4 / 16 / 14.6 / 18;
//   more: narrow where four CTAs fit (NP <= 8448) and rows are short, n = 7900, degree 20, 592 anneals: 58 / 50 / 42 / 40;
//     with long rows its warps wait for one another's atomics: degree 80, 740 anneals: 134 / 112 / 106 / 138. Three per SM
//     fill their waves less: n = 10000, degree 20, 592 anneals: 72 / 59 / 53 / 74; n = 12000, degree 32: 109 / 88 / - / 126 and
//     degree 4: 46 / 42 / - / 43, 1184 anneals 92 / 84 / - / 71. Two per SM never gain on wide: n = 16000, 1184 anneals:
//     129 / 108 / - / 114 at degree 4, 410 / 334 / - / 495 at degree 80.
SparseForm sparse_form(int np, double degree, double words, int anneals, bool slices, int per_sm, int sms) {
    if (slices && sparse_groups(np, degree, anneals, sms)) return kSparseGroups;
    const bool wide = wide_fits(np), half = half_fits(np);
    if (wide && np > 4096 && (anneals <= sms || per_sm < 3)) return kSparseWide;
    if (anneals <= sms || per_sm < 2) return kSparseOne;
    if (anneals <= 2 * sms) return half ? kSparseHalf : wide ? kSparseWide : kSparseOne;
    if (anneals <= 3 * sms) return half && words >= 64.0 && 2 * anneals <= 5 * sms ? kSparseHalf : kSparseNarrow;
    if (per_sm < 4 && half) return degree >= 16.0 ? kSparseHalf : kSparseNarrow;
    if (per_sm < 4 && wide) return degree >= (anneals <= 5 * sms ? 12.0 : 24.0) ? kSparseWide : kSparseNarrow;
    return np > 4096 && half && degree >= 48.0 ? kSparseHalf : kSparseNarrow;
}

int sparse_wave(SparseForm form, int per_sm, int sms) {
    switch (form) {
        case kSparseHalf: return 2 * sms;
        case kSparseNarrow: return per_sm * sms;
        case kSparseGroups: return kGroupReplicas * sms;      // of a CTA per SM
        default: return sms;
    }
}

// A batch's instances of one class: those of some size alone on their SMs, few anneals one by one (kBatchAlone), many in the
// narrow form where at least three fit (above).
SparseForm sparse_batch_form(int np_max, int np_min, int nitems, int per_sm, int sms) {
    const bool mixed = np_min <= 4096;        // some of the sizes gain from the smaller CTA
    if (wide_fits(np_max) && np_max > 4096 && !mixed && (nitems <= sms || per_sm < 3)) return kSparseWide;
    return nitems <= kBatchAlone * sms || per_sm < 3 ? kSparseOne : kSparseNarrow;
}

int sparse_launch(const PlainLaunch& L, int per_sm, int sms, cudaStream_t st) {
    if (L.np_max / kLanes > 32 * kMaxChunks) return int(cudaErrorInvalidValue);
    const int v = L.sparse_variant;
    SparseFn fn = nullptr;
    int grid = L.nitems, threads = 0;
    size_t smem = 0;
    switch (L.form) {
        case kSparseGroups:
            fn = L.clamp ? group_fn<true>(v) : group_fn<false>(v);
            threads = kGroupThreads;
            smem = group_smem(L.np_max);
            grid = group_ctas(L.np_max, L.nitems, sms);
            break;
        case kSparseWide:
            fn = wide_fn<1024>(v);
            threads = 1024;
            smem = wide_smem(L.np_max, threads);
            grid = std::min(grid, sms);
            break;
        case kSparseHalf:
            fn = wide_fn<512>(v);
            threads = 512;
            smem = wide_smem(L.np_max, threads);
            grid = std::min(grid, 2 * sms);
            break;
        case kSparseNarrow:
            fn = narrow_fn(v);
            threads = kNarrow;
            smem = narrow_smem(L.np_max);
            grid = std::min(grid, per_sm * sms);
            break;
        default:      // plain_engine.cu
            return plain_launch(L, 0, 12, std::min(grid, sms), plain_smem_bytes(L.np_max, L.np_max / 32, 0, 12), st);
    }
    const cudaError_t e = allow_max_smem(fn);
    if (e != cudaSuccess) return int(e);
    fn<<<grid, threads, smem, st>>>(L);
    return int(cudaGetLastError());
}

}  // namespace anc
