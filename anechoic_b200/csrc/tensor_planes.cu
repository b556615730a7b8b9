// Batched engine for replicas sharing a dense J with J held on chip as one or two packed e2m1 planes: NP = 2048 ..
// 6144 in any multiple of 256, couplings up to 4 bits. At NP = 2048 with |J| <= 1 it is what the API calls the fp4 kernel.
//
// Planes. Every |J| in {0, 1, 2, 3, 4, 6} is one e2m1 value; 5 = 4 + 1 and 7 = 6 + 1 take a second plane with entries
// in {0, +-1}. The field update is J dS = J_0 dS + J_1 dS: the same dS tile multiplied by each plane's slice into the
// same f32 accumulator (kind::mxf4, unit block scales). Products and partial sums are integers below 2^18 (at these sizes
// max_y sum_x |J_xy| + max |b| < 2^16, planes_supported), so f32 accumulation is exact in any order.
//
// Layout. RP = rounds padded to a multiple of 4 (columns k >= R of a lane are never decided and have zero couplings);
// slot i = k*256 + l sits at permuted column p = l*RP + k, so a lane's slots are contiguous. CTA cs of a replica group
// owns lanes 2 LT cs .. +2 LT - 1: decision thread (replica, half hf) owns LT of them, LT*RP <= 64 columns. dS rows are
// 128*RP bytes = RP tiles of 128 bytes (256 columns); a CTA's J slice (N = 2 CH rows per plane, CH = LT*RP padded to 8)
// stays in shared memory for the whole launch. A group takes 128 / LT CTAs, so the grid holds 148 LT / 128 groups.
//
// Per step (the golden model's step, sca_ref_bias.hpp:44-68): decide from the f32 fields in
// TMEM; publish dS nibbles and an n_lin byte per thread through L2; make the next step's draws; fetch the group's dS tile
// by tile (cp.async, an NS-deep ring, the own tile first) as the tiles' publications appear in the poller warp's shared
// mirror; 4 MMAs per tile and plane. Each tile has one counter, which every CTA owning columns of it increments with
// release semantics: a poller lane watches one word per tile (one word per CTA took up to four acquire
// loads in a row per lane: 15.0 instead of 18.3 us a step at n = 5000). Rows of replicas beyond the batch are neither decided
// nor fetched (what the MMA reads there stays finite: e2m1 has no infinity or NaN).
//
// Bounds. A step is a chain of latencies, not of bytes or operations: decide, publish through L2, see the counters, fetch,
// multiply tile after tile, read the fields. What shortened it (n = 5000, +-1, 128 anneals, us per step on a B200; n = 2000,
// 4-bit, 256 anneals behind the slash):
//   plain engine / int8 kernel before                                                                      61.0 / 23.1
//   this kernel with one flag per CTA and the decision warps waiting for their copies                       18.3 / 8.3
//   one counter per tile                                                                                    15.0 / 7.5
//   copies that arrive on the stage's barrier themselves, one stage per pair of warps                       14.4 / 7.2
//   a converged MMA warp with an elected lane (20 instead of 80 cycles to issue an MMA)                     13.4 / 6.5
//   n_lin as coalesced reductions into 8 sums per replica, wider dS stores                                   9.1 / 5.9
//   two MMA warps, each with its own accumulator (the decision adds the two)                                 7.4 / 5.2
//   fewer lanes per thread where the groups fit                                                              7.4 / 4.6
// n = 2000, +-1, 1024 anneals: 8.7 us a step with the fp4 kernel before (one MMA thread, decision warps waiting for their
// copies), 6.15 here.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "anc_f4.cuh"
#include "anc_ptx.cuh"
#include "anc_tensor.cuh"

namespace anc {
namespace {

using namespace ptx;

constexpr int kM = 128;                    // replicas per group (MMA M, TMEM lanes)
constexpr int kDW = 8;                     // decision warps
constexpr int kMmaWarps = 2;               // MMA warps, each with its own accumulator
constexpr int kMmaWarp = kDW, kPollWarp = kDW + kMmaWarps;
constexpr int kThreads = (kDW + kMmaWarps + 1) * 32;
constexpr uint32_t kTile = 128 * 128;      // dS tile: 128 replicas x 256 e2m1 columns
constexpr uint32_t kSfCol = 400;           // TMEM columns 384 .. 511 hold scale factors 0x7F (1.0)
constexpr uint32_t kAccCol = 128;          // MMA warp a accumulates at column 128 a
constexpr uint32_t kTmemCols = 512;
constexpr int NS = 4;                      // stages of the dS ring
constexpr int kNlCopies = 8;               // n_lin sums per replica and step, so that few CTAs add to one word
constexpr int kFlagStride = 8;             // words between tile counters (a 32-byte sector each)
constexpr int kErrFull = 1, kErrEmpty = 2, kErrHready = 3, kErrFlag = 4, kErrJ = 5;

struct PlanesParams {
    int n, S, R, ngroups;
    const int32_t* fourT;
    const int32_t* q;
    const int64_t* kcorr;
    const int32_t* kconst;
    int32_t hclamp;
    const int32_t* bias_perm;           // [256 RP] or null
    uint64_t seed;
    uint32_t trial_offset;
    int nchains;
    uint32_t* flags;                    // [ngroups][RP tiles], kFlagStride apart: publications counted (zeroed)
    uint8_t* dbuf;                      // [ngroups][2][128][128 RP] packed e2m1
    int32_t* nls;                       // [ngroups][3][kNlCopies][128] n_lin sums of steps m mod 3 (zeroed)
    uint64_t wait_ns;
    uint32_t* out_spins;                // [nchains][words] (zeroed)
    int words;
    unsigned long long* out_sum_sh;
    unsigned long long* out_sum_bs;
    unsigned long long* out_flips;
    int32_t* out_trace;
    int32_t* out_h;
    int* err;
    long long* prof;                    // [CTAs][kTensorProfSlots] clock64 totals of thread 0 and the first MMA warp, or null
};

template <int RP_, int LT_, int W_>
struct Geo {
    static constexpr int RP = RP_, LT = LT_, W = W_;
    static constexpr int CC = LT * RP;                   // columns of a decision thread
    static constexpr int CH = (CC + 7) / 8 * 8;          // its TMEM columns
    static constexpr int N = 2 * CH;                     // MMA N
    static constexpr int C = 2 * CC;                     // columns of a CTA
    static constexpr int NSL = 128 / LT;                 // CTAs per group
    static constexpr int ROWB = 128 * RP;                // bytes of a dS row
    static constexpr uint32_t JT = uint32_t(N) * 128;    // bytes of a J tile (one plane)
    static constexpr uint32_t JBYTES = uint32_t(W) * RP * JT;
    static_assert(CC <= 64 && N % 16 == 0 && RP % 4 == 0 && 128 % LT == 0, "geometry");
};

constexpr int kBars = 2 * NS + 3;          // full[NS], empty[NS], fields ready, J loaded, drain

// 8 / 16 / 32 TMEM columns from taddr (a multiple of the count) into v[0 ..)
__device__ __forceinline__ void tld8(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tst8(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tld16(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
}

// Fields of columns c0 .. c0 + NC - 1 of a thread: the sums of the MMA warps' accumulators (integers, so exact), loads in
// flight together.
template <int NC>
__device__ __forceinline__ void load_fields(uint32_t taddr, uint32_t (&v)[NC]) {
    uint32_t w[NC];
#pragma unroll
    for (int a = 0; a < kMmaWarps; ++a) {
        if constexpr (NC % 16 == 0) {
#pragma unroll
            for (int c = 0; c < NC; c += 16) tld16(taddr + uint32_t(a) * kAccCol + uint32_t(c), (a ? w : v) + c);
        } else {
#pragma unroll
            for (int c = 0; c < NC; c += 8) tld8(taddr + uint32_t(a) * kAccCol + uint32_t(c), (a ? w : v) + c);
        }
    }
    tmem_wait_ld();
    if constexpr (kMmaWarps == 2) {
#pragma unroll
        for (int c = 0; c < NC; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + __uint_as_float(w[c]));
    }
}

// A step's draws of the thread's LT lanes, every lane's stream in round order, kept as the top 16 bits with the top
// bit flipped (u16 - 32768): column col = j*RP + k in the high half of pk[col / 2] for even k, in the low half for odd.
// Rounds k <= RP - 4 exist for every R this RP serves.
template <class G>
__device__ __forceinline__ void draw(Xoshiro (&rng)[G::LT], uint32_t (&pk)[G::CC / 2], int R) {
#pragma unroll
    for (int k = 0; k < G::RP; ++k) {
        if (k <= G::RP - 4 || k < R) {
#pragma unroll
            for (int j = 0; j < G::LT; ++j) {
                const uint32_t u = rng_next(rng[j]);
                uint32_t& w = pk[(j * G::RP + k) / 2];
                if (k & 1) w |= (u >> 16) ^ 0x8000u;
                else w = (u & 0xffff0000u) ^ 0x80000000u;
            }
        }
    }
}

// Decisions of the thread's columns 32 E .. of at most 32: flip mask fm and mask lm of the linear band -2T < z < 2T.
//   r = floor((u16 - 32768) * 4T / 65536) = mulhi((u16 - 32768) << 16, 4T);
//   s*h: the field in f32 with its sign flipped for s = -1 (bit 31 of ~sw), clamped when the range plan asks;
//   z = s*h*65536 + q -/+ corr through the exact conversion 1.5*2^23 + x (|x| < 2^22): the low 16 bits of that encoding are
//   x, so encoding << 16 = x * 65536 modulo 2^32.
template <class G, int E, bool CLAMP>
__device__ __forceinline__ void decide(uint32_t taddr, const uint32_t (&pk)[G::CC / 2], uint32_t sw, uint32_t dw,
                                       int32_t xs, int32_t twocorr, int32_t fourT, int32_t c1, uint32_t lw, float hclf,
                                       uint32_t& fm, uint32_t& lm) {
    constexpr int NC = G::CH - 32 * E < 32 ? G::CH - 32 * E : 32, ND = G::CC - 32 * E < 32 ? G::CC - 32 * E : 32;
    uint32_t hv[NC];
    load_fields<NC>(taddr + uint32_t(32 * E), hv);
    fm = lm = 0u;
#pragma unroll
    for (int b = 0; b < ND; ++b) {
        const uint32_t w = pk[(32 * E + b) / 2];
        const uint32_t a16 = (b & 1) ? (w << 16) : (w & 0xffff0000u);
        const int32_t thr = __mulhi(int32_t(a16), fourT);
        float hsf = __uint_as_float(hv[b] ^ ((~sw << (31 - b)) & 0x80000000u));
        if (CLAMP) hsf = fminf(fmaxf(hsf, -hclf), hclf);
        const int32_t zb = __float_as_int(hsf + 12582912.0f);
        int32_t zt = (zb << 16) + xs;
        if ((dw >> b) & 1u) zt += twocorr;
        if (zt < thr) fm |= 1u << b;
        if (uint32_t(zt + c1) < lw) lm |= 1u << b;
    }
}

// A thread's dS nibbles (LT*RP/2 bytes) to its place in the row, in the widest words its alignment allows: a warp's lanes
// write 32 different rows, so every store instruction costs 32 sectors.
template <int CC>
__device__ __forceinline__ void store_nibbles(uint8_t* dst, int hf, const uint32_t (&w)[8]) {
    constexpr int B = CC / 2;
    if constexpr (B % 16 == 0) {
#pragma unroll
        for (int i = 0; i < B / 16; ++i)
            reinterpret_cast<uint4*>(dst)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    } else if constexpr (B % 8 == 0) {
#pragma unroll
        for (int i = 0; i < B / 8; ++i) reinterpret_cast<uint2*>(dst)[i] = make_uint2(w[2 * i], w[2 * i + 1]);
    } else if constexpr (B % 4 == 0) {
#pragma unroll
        for (int i = 0; i < B / 4; ++i) reinterpret_cast<uint32_t*>(dst)[i] = w[i];
    } else {
        // 10 bytes: half 0 starts on a 4-byte boundary, half 1 two bytes behind one
        static_assert(B == 10, "LT * RP = 20");
        if (hf == 0) {
            reinterpret_cast<uint32_t*>(dst)[0] = w[0];
            reinterpret_cast<uint32_t*>(dst)[1] = w[1];
            reinterpret_cast<uint16_t*>(dst)[4] = uint16_t(w[2]);
        } else {
            reinterpret_cast<uint16_t*>(dst)[0] = uint16_t(w[0]);
            reinterpret_cast<uint32_t*>(dst + 2)[0] = __funnelshift_r(w[0], w[1], 16);
            reinterpret_cast<uint32_t*>(dst + 2)[1] = __funnelshift_r(w[1], w[2], 16);
        }
    }
}

// After the CTA barrier behind the step's stores: one more publication of each tile that holds columns of this CTA (one
// or two tiles; one thread each).
template <class G>
__device__ __forceinline__ void publish(const PlanesParams& P, int g, int cs, int tid) {
    const int first = cs * G::C / 256, last = (cs * G::C + G::C - 1) / 256;
    if ((tid & 31) == 0 && tid / 32 <= last - first)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.flags + (size_t(g) * G::RP + first + tid / 32) * kFlagStride)
                     : "memory");
}

// Fetch one step's dS (step m, parity m & 1) into the ring, tile t of the step into stage t mod NS (RP is a multiple of
// NS, so a stage keeps its tiles' order over the steps): warps s and s + 4 copy every tile of stage s, in alternating
// blocks of four rows (those of the batch's replicas), each tile as soon as its stage is free and its counter shows every
// publication. The copies are asynchronous and their completion arrives on the stage's barrier by itself (one arrival
// per lane), so a warp never waits for a copy. A stage's warps wait for each of its phases in turn: a warp that skipped
// phases could take the parity of one two back for the one it waits for. Returns the replica's n_lin when want_nlin.
// ok, once false, stops copies and arrivals.
template <class G>
__device__ __forceinline__ int32_t exchange(const PlanesParams& P, int g, int m, uint32_t stages_u32, uint32_t bar_full,
                                            uint32_t bar_empty, uint32_t q, int tid, int r, int rows, bool want_nlin,
                                            const uint32_t* s_tile, uint32_t tbase, int rot, bool& ok) {
    const int lane = tid & 31;
    int* err = P.err;
    const int par = m & 1;
    const uint32_t target = tbase + uint32_t(m + 2);
    // wait (bounded) until this lane's word of the poller's mirror reaches the target (cta scope; the poller acquired
    // the counter at gpu scope)
    auto wait_tile = [&](int tk) {
        const uint32_t fa = smem_u32(s_tile + tk);
        uint32_t v;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(fa) : "memory");
        bool seen = v >= target;
        if (!seen) {
            const uint64_t t0 = globaltimer();
            for (uint32_t k = 1; !seen; ++k) {
                asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(fa) : "memory");
                seen = v >= target;
                if (!seen && ((k & 255u) == 0 || P.wait_ns == 0) && globaltimer() - t0 >= P.wait_ns) {
                    atomicCAS(err, 0, kErrFlag);
                    break;
                }
            }
        }
        return __all_sync(0xffffffffu, seen);
    };
    static_assert(kDW == 2 * NS && G::RP % NS == 0, "two warps per stage");
    const int st = (tid >> 5) & 3, half = tid >> 7;
    const int row0 = 4 * half + (lane >> 3), ch = lane & 7;      // rows row0 + 8 i
    const uint8_t* src = P.dbuf + (size_t(g * 2 + par) * kM + row0) * G::ROWB + ch * 16;
    const uint32_t dst = stages_u32 + uint32_t(st) * kTile + uint32_t(row0 * 128 + ((ch ^ row0) << 4));   // 128-byte swizzle
    const int nc = (rows + 7) / 8;
#pragma unroll 1
    for (int t = st; t < G::RP; t += NS) {
        const uint32_t u = (q + uint32_t(t)) / NS;
        const int tk = t + rot < G::RP ? t + rot : t + rot - G::RP;
        if (ok && u >= 1)
            ok = __all_sync(0xffffffffu, mbar_wait_for(bar_empty + 8 * st, (u - 1) & 1u, err, kErrEmpty, P.wait_ns));
        if (ok) ok = wait_tile(tk);
        if (ok) {
            const uint8_t* sp = src + tk * 128;
#pragma unroll 8
            for (int c = 0; c < nc; ++c) cp_async16(dst + uint32_t(c * 1024), sp + size_t(c) * 8 * G::ROWB);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_full + 8 * st) : "memory");
        }
    }
    int32_t nl = 0;
    if (ok && want_nlin) {
        ok = wait_tile(lane < G::RP ? lane : 0);      // every tile of the step, so every CTA's n_lin byte
        __syncwarp();
        if (ok) {
            const int32_t* np = P.nls + (size_t(g) * 3 + uint32_t(m) % 3u) * kNlCopies * kM + r;
            int32_t v[kNlCopies];
#pragma unroll
            for (int i = 0; i < kNlCopies; ++i) v[i] = __ldcg(np + i * kM);
#pragma unroll
            for (int i = 0; i < kNlCopies; ++i) nl += v[i];
        }
    }
    return nl;
}

template <class G>
__global__ void __launch_bounds__(kThreads, 1)
    tensor_planes_kernel(const __grid_constant__ CUtensorMap mapJ, const __grid_constant__ PlanesParams P) {
    constexpr int RP = G::RP, LT = G::LT, CC = G::CC, CH = G::CH;
    constexpr uint32_t IDESC = (1u << 7) | (1u << 10) | (uint32_t(G::N >> 3) << 17) | (1u << 23) | (uint32_t(kM >> 4) << 24);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* jres = smem;                                   // [W][RP] tiles of N x 128 bytes
    uint8_t* stages = smem + G::JBYTES;                     // NS x 16 KB
    uint64_t* bars = reinterpret_cast<uint64_t*>(stages + NS * kTile);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
    __shared__ uint32_t s_tile[RP];                         // mirror of the tile counters: gi * (S + 2) + steps published

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cs = int(blockIdx.x % G::NSL);
    const int gs0 = int(blockIdx.x / G::NSL), gstride = int(gridDim.x / G::NSL);
    const int n = P.n, S = P.S, R = P.R;
    int* err = P.err;
    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + NS);
    const uint32_t bar_h = smem_u32(bars + 2 * NS), bar_j = smem_u32(bars + 2 * NS + 1);
    const uint32_t bar_fin = smem_u32(bars + 2 * NS + 2);

    if (tid < RP) s_tile[tid] = 0u;
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(bar_full + 8 * s, 64);    // the lanes of the two warps that copy the tile
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_h, kMmaWarps);
        mbar_init(bar_j, 1);
        mbar_init(bar_fin, kMmaWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp == kMmaWarp && lane == 0) {
        // J rows of half hf start at permuted column (2 cs + hf) CC; CH - CC rows of the next lanes pad the tile (their
        // accumulator columns are never read), rows past the last plane arrive as zeros
        mbar_arrive_expect_tx(bar_j, G::JBYTES);
        for (int w = 0; w < G::W; ++w)
            for (int t = 0; t < RP; ++t)
                for (int hf = 0; hf < 2; ++hf)
                    tma_load_2d(smem_u32(jres + (w * RP + t) * G::JT + hf * CH * 128), &mapJ, t * 128,
                                w * 256 * RP + (2 * cs + hf) * CC, bar_j);
    }
    const uint32_t tl = uint32_t((warp & 3) * 32) << 16;
    if (warp < 4) {
        uint32_t v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0x7F7F7F7Fu;
        for (int c0 = 384; c0 < 512; c0 += 16) tmem_st16(tmem + tl + uint32_t(c0), v);
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const int r = (warp & 3) * 32 + lane, hf = warp >> 2;
    uint32_t hph = 0u, q = 0;
    bool jready = false;
    const bool prof = P.prof != nullptr;
    long long pc[5] = {0, 0, 0, 0, 0}, pt = 0;     // phase totals (slots of kTensorProfSlots), the last mark
    const long long loop0 = clock64();
    auto mark = [&](int i) {
        if (prof) {
            const long long now = clock64();
            if (i >= 0) pc[i] += now - pt;
            pt = now;
        }
    };

    for (int g = gs0, gi = 0; g < P.ngroups; g += gstride, ++gi) {
        const uint32_t tbase = uint32_t(gi) * uint32_t(S + 2);
        if (warp < kDW) {
            // ---------------- decision warps ----------------
            const int chain = g * kM + r, rows = min(kM, P.nchains - g * kM);
            const bool writer = chain < P.nchains;
            const bool active = (warp & 3) * 32 < rows;      // warp-uniform: some replica of the batch
            const int l0 = (2 * cs + hf) * LT;               // first RNG lane of this thread
            const uint32_t tf = tmem + tl + uint32_t(hf * CH);
            const int rot = cs * G::C / 256;                 // the tile holding the own slice comes first
            uint8_t* const drow = P.dbuf + (size_t(g) * 2 * kM + r) * G::ROWB + (2 * cs + hf) * (CC / 2);
            uint32_t sw[2] = {0u, 0u}, dw[2] = {0u, 0u}, vmask[2] = {0u, 0u};
            long long flips = 0;
            Xoshiro rng[LT];
            uint32_t pk[CC / 2];
#pragma unroll
            for (int i = 0; i < CC / 2; ++i) pk[i] = 0u;
            if (active) {
                uint32_t db[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
                for (int j = 0; j < LT; ++j)
                    rng_seed(rng[j], P.seed, P.trial_offset + uint32_t(chain), uint32_t(l0 + j));
#pragma unroll
                for (int k = 0; k < RP; ++k) {
                    if (k <= RP - 4 || k < R) {
#pragma unroll
                        for (int j = 0; j < LT; ++j) {
                            const int col = j * RP + k, i = k * 256 + l0 + j;
                            const uint32_t rv = rng_next(rng[j]);
                            const bool valid = i < n;
                            const uint32_t up = valid ? (rv >> 31) : 1u;
                            sw[col >> 5] |= up << (col & 31);
                            if (valid) vmask[col >> 5] |= 1u << (col & 31);
                            if (valid && !up) dw[col >> 5] |= 1u << (col & 31);
                            db[col >> 3] |= (valid ? (up ? 0x2u : 0xAu) : 0u) << (4 * (col & 7));   // e2m1 +1 / -1
                        }
                    }
                }
                store_nibbles<CC>(drow + size_t(kM) * G::ROWB, hf, db);     // the state D = s0 (parity 1)
#pragma unroll 1
                for (int c = 0; c < CH; c += 8) {
                    uint32_t v[8];
#pragma unroll
                    for (int x = 0; x < 8; ++x)
                        v[x] = __float_as_uint(P.bias_perm && c + x < CC ? float(P.bias_perm[(2 * cs + hf) * CC + c + x]) : 0.f);
                    tst8(tf + uint32_t(c), v);
#pragma unroll
                    for (int x = 0; x < 8; ++x) v[x] = 0u;
                    for (int a = 1; a < kMmaWarps; ++a) tst8(tf + uint32_t(a) * kAccCol + uint32_t(c), v);
                }
                tmem_wait_st();
            }
            tc_fence_before();
            asm volatile("bar.sync 1, %0;" ::"r"(kDW * 32) : "memory");
            publish<G>(P, g, cs, tid);
            const bool eok = !err_set(err);
            if (active) draw<G>(rng, pk, R);
            bool ok = __all_sync(0xffffffffu, eok);
            int32_t nlin_next = exchange<G>(P, g, -1, smem_u32(stages), bar_full, bar_empty, q, tid, r, rows, false,
                                                   s_tile, tbase, rot, ok);
            q += RP;
            const float hclf = float(P.hclamp);
            for (int m = 0; m <= S; ++m) {
                const int t = m < S ? m : S - 1;
                const int32_t fourT = __ldg(P.fourT + t), qv = __ldg(P.q + t), kconst = __ldg(P.kconst + t);
                const int64_t kcorr = __ldg(P.kcorr + t);
                mark(-1);
                if (ok) ok = __all_sync(0xffffffffu, mbar_wait_for(bar_h, hph & 1u, err, kErrHready, P.wait_ns));
                ++hph;
                tc_fence_after();
                mark(0);
                const int32_t nlin_prev = nlin_next;
                if (m >= 1 && writer && cs == 0 && hf == 0 && P.out_trace) P.out_trace[size_t(chain) * S + (m - 1)] = nlin_prev;
                if (m == S) {
                    if (active) {
                        long long sh = 0, bs = 0;
#pragma unroll 1
                        for (int c = 0; c < CC; c += 8) {
                            uint32_t hc[8];
                            tld8(tf + uint32_t(c), hc);
                            tmem_wait_ld();
                            for (int a = 1; a < kMmaWarps; ++a) {
                                uint32_t h2[8];
                                tld8(tf + uint32_t(a) * kAccCol + uint32_t(c), h2);
                                tmem_wait_ld();
#pragma unroll
                                for (int x = 0; x < 8; ++x) hc[x] = __float_as_uint(__uint_as_float(hc[x]) + __uint_as_float(h2[x]));
                            }
#pragma unroll
                            for (int x = 0; x < 8; ++x) {
                                const int col = c + x, j = col / RP, k = col - j * RP, i = k * 256 + l0 + j;
                                if (col >= CC || k >= R || i >= n) continue;
                                const bool up = ((col < 32 ? sw[0] : sw[1]) >> (col & 31)) & 1u;
                                const int32_t h = __float2int_rn(__uint_as_float(hc[x]));
                                sh += up ? h : -h;
                                if (P.bias_perm) {
                                    const int32_t b = P.bias_perm[(2 * cs + hf) * CC + col];
                                    bs += up ? b : -b;
                                }
                                if (writer) {
                                    if (up) atomicOr(P.out_spins + size_t(chain) * P.words + (i >> 5), 1u << (i & 31));
                                    if (P.out_h) P.out_h[size_t(chain) * n + i] = h;
                                }
                            }
                        }
                        if (writer) {
                            atomicAdd(P.out_sum_sh + chain, static_cast<unsigned long long>(sh));
                            atomicAdd(P.out_sum_bs + chain, static_cast<unsigned long long>(bs));
                            atomicAdd(P.out_flips + chain, static_cast<unsigned long long>(flips));
                        }
                    }
                    continue;
                }
                const int par = m & 1;
                if (active) {
                    const int32_t twoT = fourT >> 1;
                    const int32_t corr = step_corr(nlin_prev, kcorr, kconst);
                    const uint32_t lw = uint32_t(2 * twoT - 1);
                    const int32_t xs = qv - corr, c1 = twoT - 1, twocorr = 2 * corr;
                    uint32_t fm[2] = {0u, 0u}, lm[2] = {0u, 0u}, dq[8];
                    if (P.hclamp > 0) {
                        decide<G, 0, true>(tf, pk, sw[0], dw[0], xs, twocorr, fourT, c1, lw, hclf, fm[0], lm[0]);
                        if constexpr (CC > 32) decide<G, 1, true>(tf, pk, sw[1], dw[1], xs, twocorr, fourT, c1, lw, hclf, fm[1], lm[1]);
                    } else {
                        decide<G, 0, false>(tf, pk, sw[0], dw[0], xs, twocorr, fourT, c1, lw, hclf, fm[0], lm[0]);
                        if constexpr (CC > 32) decide<G, 1, false>(tf, pk, sw[1], dw[1], xs, twocorr, fourT, c1, lw, hclf, fm[1], lm[1]);
                    }
                    int nl = 0;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        fm[e] &= vmask[e];
                        nl += __popc(lm[e] & vmask[e]);
                        flips += __popc(fm[e]);
                        const uint4 d4 = f4_dnibbles(fm[e], fm[e] & sw[e]);
                        dq[4 * e] = d4.x; dq[4 * e + 1] = d4.y; dq[4 * e + 2] = d4.z; dq[4 * e + 3] = d4.w;
                        sw[e] ^= fm[e];
                        dw[e] = fm[e];
                    }
                    store_nibbles<CC>(drow + size_t(par) * kM * G::ROWB, hf, dq);
                    atomicAdd(P.nls + ((size_t(g) * 3 + uint32_t(m) % 3u) * kNlCopies + cs % kNlCopies) * kM + r, nl);
                }
                tc_fence_before();
                mark(1);
                asm volatile("bar.sync 1, %0;" ::"r"(kDW * 32) : "memory");
                publish<G>(P, g, cs, tid);
                mark(2);
                const bool eok2 = !err_set(err);
                if (active && m + 1 < S) draw<G>(rng, pk, R);
                ok = ok && __all_sync(0xffffffffu, eok2);
                mark(3);
                nlin_next = exchange<G>(P, g, m, smem_u32(stages), bar_full, bar_empty, q, tid, r, rows, active,
                                               s_tile, tbase, rot, ok);
                q += RP;
                mark(4);
                // every CTA of the group has published step m, so none reads step m - 1's sums any more; they become
                // step m + 2's, whose writers wait for this CTA's publication of step m + 1
                if (cs < kNlCopies && hf == 0)
                    P.nls[((size_t(g) * 3 + uint32_t(m + 2) % 3u) * kNlCopies + cs) * kM + r] = 0;
            }
            tc_fence_before();
        } else if (warp < kPollWarp) {
            // ---------------- MMA warps: converged, one elected lane issues; warp a takes tiles t = a mod kMmaWarps ------
            const uint32_t a = uint32_t(warp - kMmaWarp);
            if (!jready) {
                bool jok = true;
                if (lane == 0) jok = !err_set(err) && mbar_wait_for(bar_j, 0u, err, kErrJ, P.wait_ns);
                jready = __all_sync(0xffffffffu, jok);
            }
            const uint32_t utmem = __shfl_sync(0xffffffffu, tmem, 0);
            const uint32_t acc = utmem + __shfl_sync(0xffffffffu, a, 0) * kAccCol, sf = utmem + kSfCol;
            const uint64_t a0 = sw128_desc(smem_u32(stages)), b0 = sw128_desc(smem_u32(jres));
            const int tk0 = cs * G::C / 256 + int(a);
            const bool lead = elect_one();
            bool mok = jready;
#pragma unroll 1
            for (int m = -1; m < S; ++m) {
                mok = mok && __all_sync(0xffffffffu, !err_set(err));
                int tk = tk0 < RP ? tk0 : tk0 - RP;
                const long long c0 = prof ? clock64() : 0;
#pragma unroll 1
                for (int t0 = 0; t0 < RP; t0 += NS, q += NS) {
#pragma unroll
                    for (int s0 = 0; s0 < NS; s0 += kMmaWarps) {
                        const uint32_t s = uint32_t(s0) + a;
                        mark(-1);
                        if (mok) mok = __all_sync(0xffffffffu, mbar_wait_for(bar_full + 8 * s, (q / NS) & 1u, err, kErrFull, P.wait_ns));
                        mark(0);
                        tc_fence_after();
                        if (lead) {
                            if (mok) {
                                // the copies wrote shared memory through the generic proxy
                                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                                const uint64_t ad = a0 + uint64_t(s * (kTile >> 4)), bd = b0 + uint64_t(uint32_t(tk) * (G::JT >> 4));
#pragma unroll
                                for (int w = 0; w < G::W; ++w)
#pragma unroll
                                    for (int kk = 0; kk < 4; ++kk)
                                        mma_mxf4(acc, ad + uint64_t(2 * kk), bd + uint64_t(w * RP * (G::JT >> 4) + 2 * kk), IDESC, sf,
                                                 sf + 48u);
                            }
                            mma_commit(bar_empty + 8 * s);
                        }
                        __syncwarp();
                        tk += kMmaWarps;
                        if (tk >= RP) tk -= RP;
                    }
                }
                if (lead) mma_commit(bar_h);
                __syncwarp();
                if (prof) pc[1] += clock64() - c0;
            }
        } else if (warp == kPollWarp) {
            // ---------------- poller: lane t mirrors the counter of tile t ----------------
            static_assert(RP <= 32, "one lane per tile");
            const int tl0 = lane < RP ? lane : 0;
            const uint32_t* fl = P.flags + (size_t(g) * RP + tl0) * kFlagStride;
            const uint32_t cnt = uint32_t((256 * tl0 + 255) / G::C - 256 * tl0 / G::C + 1);    // CTAs of the tile
            bool pok = !err_set(err);
            for (uint32_t target = 1; pok && target <= uint32_t(S + 1); ++target) {
                const uint64_t t0 = globaltimer();
                bool seen = lane >= RP;
                for (uint32_t k = 1;; ++k) {
                    if (!seen) {
                        uint32_t v;
                        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(fl) : "memory");
                        if (v >= cnt * target) {
                            asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(s_tile + lane)),
                                         "r"(tbase + target)
                                         : "memory");
                            seen = true;
                        }
                    }
                    if (__all_sync(0xffffffffu, seen)) break;
                    if ((k & 63u) == 0) {
                        const bool late = lane == 0 && globaltimer() - t0 > P.wait_ns;
                        if (late) atomicCAS(err, 0, kErrFlag);
                        if (__shfl_sync(0xffffffffu, (late || (lane == 0 && err_set(err))) ? 1 : 0, 0)) {
                            pok = false;
                            break;
                        }
                    }
                }
            }
        }
    }
    if (warp >= kMmaWarp && warp < kPollWarp && elect_one()) {
        // drain: every MMA issued has completed (and the J copy has landed) before TMEM and shared memory go away
        if (!jready) mbar_wait_for(bar_j, 0u, nullptr, 0, kWaitNs);
        mma_commit(bar_fin);
        mbar_wait_for(bar_fin, 0u, nullptr, 0, kWaitNs);
    }
    if (prof && lane == 0 && (warp == 0 || warp == kMmaWarp)) {
        long long* dst = P.prof + size_t(blockIdx.x) * kTensorProfSlots;
        if (warp == 0) {
            for (int i = 0; i < 5; ++i) dst[i] = pc[i];
        } else {
            dst[5] = pc[0];
            dst[6] = pc[1];
            dst[8] = clock64() - loop0;
        }
    }
    cp_async_wait_all();  // no copy may land in shared memory the CTA has released
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// The plain engine's bit planes ([K][np][nwj] words, bit y of row x: K = 1 [J_xy = +1]; K >= 2 plane 0 [J_xy < 0], plane b
// bit b - 1 of |J_xy|) -> W e2m1 planes [W][256 RP][128 RP] of permuted rows and columns, two columns per byte (the even one
// in the low nibble). One block per permuted row y, which reads bit row y (J is symmetric).
__global__ void planes_pack_kernel(const uint32_t* __restrict__ bits, int K, int np, int nwj, int n, int R, int RP, int W,
                                   uint8_t* __restrict__ out) {
    const int py = blockIdx.x, ly = py / RP, ky = py - ly * RP, y = ky * 256 + ly;
    const size_t plane = size_t(256 * RP) * (128 * RP), bplane = size_t(np) * nwj;
    const uint32_t* row = bits + size_t(y) * nwj;
    for (int b = threadIdx.x; b < 128 * RP; b += blockDim.x) {
        uint32_t c0 = 0u, c1 = 0u;
        for (int h = 0; h < 2; ++h) {
            const int px = 2 * b + h, lx = px / RP, kx = px - lx * RP, x = kx * 256 + lx;
            if (ky >= R || kx >= R || y >= n || x >= n || x == y) continue;
            const uint32_t b0 = (row[x >> 5] >> (x & 31)) & 1u;
            uint32_t a = 1u, neg = b0;
            if (K == 1) {
                neg = b0 ^ 1u;
            } else {
                a = 0u;
                for (int p = 1; p < K; ++p) a |= ((row[bplane * p + (x >> 5)] >> (x & 31)) & 1u) << (p - 1);
            }
            // e2m1 codes: 1.0 = 2, 2.0 = 4, 3.0 = 5, 4.0 = 6, 6.0 = 7; 5 = 4 + 1 and 7 = 6 + 1
            const uint32_t mag = (0x77665420u >> (4 * a)) & 0xFu, sgn = neg << 3;
            c0 |= (a ? mag | sgn : 0u) << (4 * h);
            c1 |= ((a == 5 || a == 7) ? 2u | sgn : 0u) << (4 * h);
        }
        out[size_t(py) * (128 * RP) + b] = uint8_t(c0);
        if (W > 1) out[plane + size_t(py) * (128 * RP) + b] = uint8_t(c1);
    }
}

// ------------------------------------------------------------------------------------------------ host side
using PlanesKernel = void (*)(const CUtensorMap, const PlanesParams);
struct Config {
    int rp, w, lt, ch;
    uint32_t jbytes;
    double us;
    PlanesKernel fn;
};

template <int RP, int LT, int W>
Config config(double us) {
    using G = Geo<RP, LT, W>;
    return {RP, W, LT, G::CH, G::JBYTES, us, tensor_planes_kernel<G>};
}

// The compiled geometries: the lanes per thread LT with which the J slice (256 LT RP^2 W bytes) leaves room for the dS
// ring. A larger LT runs more replica groups at once on the device's SMs (LT in 128 CTAs' worth), a smaller one has shorter
// decisions and smaller slices per CTA; us is the measured step (B200, |J| as the planes hold it, 1 .. 128 LT anneals).
constexpr int kConfigs = 13;
const Config* planes_configs() {
    static const Config cfg[kConfigs] = {
        config<8, 8, 1>(6.2),  config<8, 4, 1>(4.6),  config<8, 2, 1>(4.2),  config<8, 4, 2>(5.2),  config<8, 2, 2>(4.8),
        config<12, 4, 1>(6.8), config<12, 2, 1>(5.9), config<12, 2, 2>(6.5), config<16, 2, 1>(6.3), config<16, 1, 1>(5.7),
        config<16, 1, 2>(6.5), config<20, 1, 1>(7.4), config<24, 1, 1>(8.2)};
    return cfg;
}

// Replica groups a device of `sms` SMs runs at once (one CTA per SM).
int group_slots(const Config& c, int sms) { return sms / (128 / c.lt); }

// The geometry for ngroups replica groups: the fewest waves, then the smallest LT (the quicker step). Measured at
// n = 2000, +-1, 1 .. 4 groups: LT = 4 4.6 us a step, LT = 8 6.2; at 8 groups LT = 4 takes two waves, 9.2 against 6.2.
const Config* planes_config(int R, int W, int ngroups, int sms) {
    const int rp = (R + 3) / 4 * 4;
    const Config *cfg = planes_configs(), *best = nullptr;
    int best_waves = 0;
    for (int i = 0; i < kConfigs; ++i) {
        const Config& c = cfg[i];
        if (c.rp != rp || c.w != W || group_slots(c, sms) < 1) continue;
        const int waves = (ngroups + group_slots(c, sms) - 1) / group_slots(c, sms);
        if (!best || waves < best_waves || (waves == best_waves && c.lt < best->lt)) {
            best = &c;
            best_waves = waves;
        }
    }
    return best;
}

size_t planes_smem(const Config& c) {
    return 1024 + size_t(c.jbytes) + size_t(NS) * kTile + size_t(kBars) * 8 + 16;
}

int rounds_of(int n) { return std::max(2048, ((n + 255) / 256) * 256) / 256; }

int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return sms;
}

// Geometry of a launch: variant 0 by rule, 1 .. 3 force LT = 8, 4 or 2 (NP = 2048, one plane).
const Config* launch_config(int R, int W, int ngroups, int sms, int variant) {
    if (variant == 0) return planes_config(R, W, ngroups, sms);
    const Config* cfg = planes_configs();
    for (int i = 0; i < kConfigs; ++i)
        if (cfg[i].rp == (R + 3) / 4 * 4 && cfg[i].w == W && cfg[i].lt == 16 >> variant && group_slots(cfg[i], sms) > 0) return &cfg[i];
    return nullptr;
}

int planes_of(int maxabs) { return maxabs <= 4 ? 1 : 2; }

}  // namespace

// One plane holds |J| <= 4; two hold |J| <= 7. The sizes keep every field below 2^16, and so every f32 partial sum an exact
// integer, whatever the instance: with the largest accepted bias, 6144 * 4 + 32767 = 57343 and 4096 * 7 + 32767 = 61439.
bool planes_supported(int n, int maxabs) {
    return maxabs <= 7 && planes_config(rounds_of(n), planes_of(maxabs), 1, 128) != nullptr;
}

double planes_step_us(int n, int maxabs, int nchains, int sms) {
    const int ngroups = (nchains + kM - 1) / kM;
    const Config* c = planes_config(rounds_of(n), planes_of(maxabs), ngroups, sms);
    return c ? double((ngroups + group_slots(*c, sms) - 1) / group_slots(*c, sms)) * c->us : -1.0;
}

int planes_wave_chains(int n, int maxabs) {
    const int sms = sm_count();
    const Config* c = planes_config(rounds_of(n), planes_of(maxabs), 1 << 20, sms);     // many groups: the largest LT
    return c ? group_slots(*c, sms) * kM : 0;
}

int planes_max_ctas() { return sm_count(); }

int planes_build(const uint32_t* bits, int K, int nwj, int n, const int32_t* bias, int maxabs, PlanesInstance* out,
                 cudaStream_t st, std::string* why) {
    const int R = rounds_of(n), W = planes_of(maxabs);
    const int RP = (R + 3) / 4 * 4;
    const size_t bytes = size_t(W) * (256 * RP) * (128 * RP);
    cudaError_t e = cudaMalloc(&out->d_J, bytes);
    if (e == cudaSuccess) {
        planes_pack_kernel<<<256 * RP, 256, 0, st>>>(bits, K, 256 * R, nwj, n, R, RP, W, out->d_J);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && bias) {
        std::vector<int32_t> bp(size_t(256) * RP, 0);
        for (int i = 0; i < n; ++i) bp[size_t(i & 255) * RP + (i >> 8)] = bias[i];
        e = cudaMalloc(&out->d_bias, bp.size() * 4);
        if (e == cudaSuccess) e = cudaMemcpy(out->d_bias, bp.data(), bp.size() * 4, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);     // other streams may run this instance next
    if (e != cudaSuccess) {
        if (why) *why = std::string("J planes: ") + cudaGetErrorString(e);
        planes_free(out);
        return setup_code(e);
    }
    out->n = n;
    out->R = R;
    out->W = W;
    return 0;
}

int planes_run(PlanesInstance* pi, const TensorRun& r, cudaStream_t st, std::string* why) {
    const int ngroups = (r.nchains + kM - 1) / kM, words = pi->R * 8, sms = sm_count();
    const Config* pc = launch_config(pi->R, pi->W, ngroups, sms, r.variant);
    if (!pc) {
        if (why) *why = "the planes kernel cannot be co-resident on this device";
        return -2;
    }
    const Config& c = *pc;
    const int nsl = 128 / c.lt, slots = std::min(ngroups, group_slots(c, sms));
    cudaError_t e = cudaFuncSetAttribute(c.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(planes_smem(c)));
    if (e != cudaSuccess) {
        if (why) *why = std::string("kernel attributes: ") + cudaGetErrorString(e);
        return -2;
    }
    const size_t fbytes = (size_t(ngroups) * c.rp * kFlagStride * 4 + 255) / 256 * 256;
    const size_t dbytes = size_t(ngroups) * 2 * kM * (128 * c.rp);
    const size_t nbytes = size_t(ngroups) * 3 * kNlCopies * kM * 4;
    const size_t need = 256 + fbytes + nbytes + dbytes;
    pi->last_err = nullptr;
    e = pi->ws.ensure(need, st);
    if (e != cudaSuccess) {
        if (why) *why = std::string("workspace: ") + cudaGetErrorString(e);
        return setup_code(e);
    }
    uint8_t* base = pi->ws.p;
    CUtensorMap mapJ;
    if (!make_map_2d(&mapJ, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, pi->d_J, uint64_t(128) * c.rp, uint64_t(256) * c.rp * c.w,
                     128, uint32_t(c.ch))) {
        if (why) *why = "cuTensorMapEncodeTiled failed";
        return -2;
    }
    e = cudaMemsetAsync(r.out_spins, 0, size_t(r.nchains) * words * 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_sum_sh, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_sum_bs, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.out_flips, 0, size_t(r.nchains) * 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(base, 0, 256 + fbytes + nbytes, st);     // error word, counters, n_lin sums
    if (e != cudaSuccess) {
        if (why) *why = std::string("memset: ") + cudaGetErrorString(e);
        return -2;
    }
    PlanesParams P{};
    P.n = pi->n;
    P.S = r.tab.S;
    P.R = pi->R;
    P.ngroups = ngroups;
    P.fourT = r.tab.fourT;
    P.q = r.tab.q;
    P.kcorr = r.tab.kcorr;
    P.kconst = r.tab.kconst;
    P.hclamp = r.hclamp;
    P.bias_perm = r.bias ? pi->d_bias : nullptr;
    P.seed = r.seed;
    P.trial_offset = r.trial_offset;
    P.nchains = r.nchains;
    P.flags = reinterpret_cast<uint32_t*>(base + 256);
    P.nls = reinterpret_cast<int32_t*>(base + 256 + fbytes);
    P.dbuf = base + 256 + fbytes + nbytes;
    P.wait_ns = r.wait_ns;
    P.out_spins = r.out_spins;
    P.words = words;
    P.out_sum_sh = reinterpret_cast<unsigned long long*>(r.out_sum_sh);
    P.out_sum_bs = reinterpret_cast<unsigned long long*>(r.out_sum_bs);
    P.out_flips = reinterpret_cast<unsigned long long*>(r.out_flips);
    P.out_trace = r.out_trace;
    P.out_h = r.out_h;
    P.err = reinterpret_cast<int*>(base);
    P.prof = r.prof;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(nsl * slots);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = planes_smem(c);
    cfg.stream = st;
    e = cudaLaunchKernelEx(&cfg, c.fn, mapJ, P);
    if (e != cudaSuccess) {
        if (why) *why = std::string("launch: ") + cudaGetErrorString(e);
        return -2;
    }
    pi->last_err = P.err;
    pi->last_ctas = nsl * slots;
    return 0;
}

void planes_free(PlanesInstance* pi) {
    if (pi->d_J) cudaFree(pi->d_J);
    if (pi->d_bias) cudaFree(pi->d_bias);
    pi->ws.free();
    *pi = PlanesInstance{};
}

}  // namespace anc
