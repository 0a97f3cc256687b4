// Finished rows of the fp16 / d_head 128 kernels: into the caller's buffer, or, head-sharded, into every rank's full-width one.
#pragma once
#include "ca_kernels.h"
#include "ca_ptx.cuh"

namespace ca {

// fp16 output row of a pair: to `out`, or into every rank's full-width buffer
__device__ __forceinline__ void store_row(const MergeParams& p, int pair, int lane, const float4& acc, float inv) {
    const __half2 h01 = __floats2half2_rn(acc.x * inv, acc.y * inv);
    const __half2 h23 = __floats2half2_rn(acc.z * inv, acc.w * inv);
    uint2 packed;
    packed.x = *reinterpret_cast<const uint32_t*>(&h01);
    packed.y = *reinterpret_cast<const uint32_t*>(&h23);
    if (p.n_peers == 0) {
        *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.out) + (size_t)pair * FAST_D + 4 * lane) = packed;
    } else {
        // head-sharded: the row goes into every rank's full-width output
        const int row = pair / p.n_heads;
        const int head = pair - row * p.n_heads;
        const size_t off = ((size_t)row * p.total_heads + p.head_offset + head) * FAST_D + 4 * lane;
        if (p.mc_out) {
            // one store to the multicast address: the switch replicates it into every rank's buffer
            asm volatile("multimem.st.weak.global.v2.f16x2 [%0], {%1, %2};" ::"l"(reinterpret_cast<__half*>(p.mc_out) + off),
                         "r"(packed.x), "r"(packed.y)
                         : "memory");
        } else {
            // plain stores to peer memory over NVLink
#pragma unroll
            for (int i = 0; i < MERGE_MAX_PEERS; i++)
                if (i < p.n_peers) *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.peer_out[i]) + off) = packed;
        }
    }
}

// The same for a lane that owns eight consecutive output elements (granule g of the row)
__device__ __forceinline__ void store_row8(const MergeParams& p, int row, int head, int g, const float (&o)[8], float inv) {
    uint4 packed;
    packed.x = ptx::pack_half2(o[0] * inv, o[1] * inv);
    packed.y = ptx::pack_half2(o[2] * inv, o[3] * inv);
    packed.z = ptx::pack_half2(o[4] * inv, o[5] * inv);
    packed.w = ptx::pack_half2(o[6] * inv, o[7] * inv);
    if (p.n_peers == 0) {
        *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.out) + ((size_t)row * p.n_heads + head) * FAST_D + 8 * g) = packed;
    } else {
        const size_t off = ((size_t)row * p.total_heads + p.head_offset + head) * FAST_D + 8 * g;
        if (p.mc_out) {
            asm volatile("multimem.st.weak.global.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(reinterpret_cast<__half*>(p.mc_out) + off),
                         "r"(packed.x), "r"(packed.y), "r"(packed.z), "r"(packed.w)
                         : "memory");
        } else {
#pragma unroll
            for (int i = 0; i < MERGE_MAX_PEERS; i++)
                if (i < p.n_peers) *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.peer_out[i]) + off) = packed;
        }
    }
}

}  // namespace ca
