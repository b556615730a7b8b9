// Device helpers of the e2m1 tensor kernel (tensor_planes.cu): the packing of dS and asynchronous copies.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace anc {

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

// 16-byte global -> shared copy through L2 only (cp.async.cg), and the wait for all of this thread's copies.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace anc
