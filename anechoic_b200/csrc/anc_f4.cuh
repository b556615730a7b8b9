// Device helpers of the e2m1 tensor kernels (tensor_engine.cu, tensor_planes.cu): flag publication, asynchronous copies
// and the packing of dS.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace anc {

// Release store alone: the writes of the CTA's other threads are ordered before it by the preceding bar.sync, and
// release is cumulative over them.
__device__ __forceinline__ void flag_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// dS nibbles of 8 columns: flipped down->up = +2 (0x4), up->down = -2 (0xC); word w holds columns 8w .. 8w+7.
__device__ __forceinline__ uint4 f4_dnibbles(uint32_t fm, uint32_t fdn) {
    uint32_t db[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        uint32_t a8 = (fm >> (8 * w)) & 0xFFu, b8 = (fdn >> (8 * w)) & 0xFFu;
        a8 = (a8 | (a8 << 12)) & 0x000F000Fu; a8 = (a8 | (a8 << 6)) & 0x03030303u; a8 = (a8 | (a8 << 3)) & 0x11111111u;
        b8 = (b8 | (b8 << 12)) & 0x000F000Fu; b8 = (b8 | (b8 << 6)) & 0x03030303u; b8 = (b8 | (b8 << 3)) & 0x11111111u;
        db[w] = (a8 << 2) | (b8 << 3);
    }
    return make_uint4(db[0], db[1], db[2], db[3]);
}

// 16-byte global -> shared copy through L2 only (cp.async.cg), and its commit-group bookkeeping.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most n of this thread's commit groups are pending (n folds to a constant once the caller's loop is
// unrolled; larger n waits for all).
__device__ __forceinline__ void cp_async_wait(int n) {
    switch (n) {
        case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    }
}

}  // namespace anc
