// Decode attention of small steps in ONE launch: fp16 caches with rows of whole 16-byte granules and d_head <= 128, and bf16 caches of
// grouped heads (1, 2, 4 or 8 query heads to a key/value head) of 64 or 128 elements.
//
// A unit is a key/value head and a block of up to 8 columns: consecutive rows, each with the query heads of the group; its work is the list
// of chunks that any of the rows sees, each with the set of columns that see it, so a shared chunk is read once for the block.  The list is cut into steps of 16
// tokens, dealt in consecutive ranges to the warps of a CLUSTER of 1 to 8 CTAs per unit (cut by the host, ca_plan.h).  A
// warp takes K and V from global memory straight into registers, as the operands of mma.sync:
//   S^T = K Q^T          lane (g, c) = (lane / 4, lane % 4) holds granules 4 j + c of tokens g and g + 8: their four registers are
//                        the A operands of two MMAs (the contraction's order is free as long as q follows it)
//   O^T += V^T P^T       lane (g, c) holds granules 8 i + g of tokens 2 c, 2 c + 1, 2 c + 8, 2 c + 9; byte permutes of two tokens'
//                        registers give the A operands.  P goes from the one layout to the other by movmatrix, as the sum of two
//                        numbers of the cache's type (22 bits of the fp32 weight in fp16, 16 in bf16)
// The 8 columns of both products are those of the block.  When the set of columns changes along a warp's range, what it has
// is combined into the warp's own area of shared memory, for the rows that saw it only: what the other columns hold is
// dropped, so a row's infinities never meet another row.  Areas are combined per CTA, and the CTAs' results through
// distributed shared memory: no partial results in global memory, no second launch.
// Infinite values of an fp16 cache: a weight's hi part times infinity is the result, its lo part times infinity is NaN or the other
// infinity.  A row with an element that is not finite in any CTA is computed once more, with fp32 weights in fp32 products (redo): what
// is not a number then is none.  The rows' marks travel with what the CTAs tell each other anyway.
// Bound: latency (launch, work list, tokens, meeting), and the bytes in flight: 8 KiB a warp, K of the next step requested
// as soon as K of this one is used, V likewise; 12 warps of an SM have 96 KiB under way.  A step is 16 MMAs (8 cycles each of a
// scheduler's time, 20 until the result is there) and one trip to memory; maxima are exchanged between lanes only when a score
// exceeds the reference in use by 2^8, as in the other kernels.
// Measured (B200, steps back to back, partial results and merge or any-geometry kernel -> here): 32 heads of 128, one row of 1500
// tokens 12.3 -> 8.9 us; 8 heads, 4 rows of 300 tokens 9.6 -> 7.5; 12 heads of 64, 16 rows of 500 shared and up to 333 own tokens
// 12.8 -> 8.8 (8.8, 7.5 and 8.7 without the second look at infinite values).  Errors against 64 bits are the
// rounding of the result alone (2.1e-4 of its norm; weights of 11 bits: 2.8e-4).
// Tried and slower: a ring of three steps per warp in shared memory, filled by cp.async (8 warps on an SM instead of 12, a third more
// instructions): one row of 1500 tokens 9.3 -> 10.5 us.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "ca_kernels.h"
#include "ca_launch.cuh"
#include "ca_plan.h"
#include "ca_ptx.cuh"
#include "ca_types.cuh"

namespace ca {
namespace {
using namespace ptx;

constexpr int D_WARPS = DIRECT_WARPS, D_ROWS = DIRECT_ROWS, D_STEP = DIRECT_STEP;

__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
    uint32_t t;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(t) : "r"(v));
    return t;
}
template <typename T> __device__ __forceinline__ void mma_16bit(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (std::is_same_v<T, __half>)
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float2 half2_of(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
template <typename T> __device__ __forceinline__ uint32_t pack_pair(float a, float b) {
    if constexpr (std::is_same_v<T, __half>) return pack_half2(a, b);
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// weights as hi + lo pairs (column, column + 1)
template <typename T> __device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
    hi = pack_pair<T>(a, b);
    if constexpr (std::is_same_v<T, __half>) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
        lo = pack_pair<T>(a - f.x, b - f.y);
    } else {
        lo = pack_pair<T>(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
    }
}

// A row's reference follows its maximum in steps of at least 2^STEP, 2^SHIFT below it: weights are at most 2^(STEP + SHIFT).  As fp16
// numbers they reach up to that end of the range, so that what their hi and lo parts leave out, 2^-25 at most, is 2^-36 of the
// largest weight, less than an fp32 sum leaves out.  (Without the shift it was 2^-25: 4000 tokens of 2^-26 beside one of 1 were no tokens.)
// Errors against 64 bits, 60 shapes (heads of 32 to 128, 1 to 16 rows, 4 to 4000 own and up to 500 shared tokens, scores spread by 0.1 to
// 16): 1.00001 times those of the any-geometry kernel's fp32 weights in the mean, 1.0004 at most.  12 heads of 64, 16 rows of 500 shared and
// up to 333 own tokens: 8.69 us without shift and with steps of 2^8, 8.78 so.
template <typename T> struct Reference {
    static constexpr float STEP = 8.f, SHIFT = 0.f;
};
template <> struct Reference<__half> {
    static constexpr float STEP = 4.f, SHIFT = 11.f;
};

// Shared memory of a CTA: O of each warp's rows, then their maxima and sums.
template <int VG> struct DirectSmem {
    static constexpr int DV = VG * 64, PITCH = DV + 4;             // floats of a row
    static __host__ __device__ constexpr int stats(int rows) { return D_WARPS * rows * PITCH * 4; }
    static __host__ __device__ constexpr int again(int rows) { return stats(rows) + D_WARPS * rows * 8 + D_WARPS * 4; }  // [2] rows, [2][D_ROWS]
    static __host__ __device__ constexpr int bytes(int rows) { return again(rows) + (2 + 2 * D_ROWS) * 4; }
};

// fp16 elements d .. d + 7 of column n, where its row goes
template <bool PEERS> __device__ __forceinline__ void store_half8(const DirectParams& p, int row, int head, int d, const uint4& packed) {
    if (!PEERS) {
        *reinterpret_cast<uint4*>(static_cast<__half*>(p.out) + ((size_t)row * p.n_heads + head) * p.d + d) = packed;
    } else {  // head-sharded: into every rank's full-width output, by the switch or by plain stores over NVLink
        const size_t to = ((size_t)row * p.total_heads + p.head_offset + head) * p.d + d;
        if (p.mc_out) {
            asm volatile("multimem.st.weak.global.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(static_cast<__half*>(p.mc_out) + to), "r"(packed.x),
                         "r"(packed.y), "r"(packed.z), "r"(packed.w)
                         : "memory");
        } else {
            for (int k = 0; k < p.n_peers; k++) *reinterpret_cast<uint4*>(static_cast<__half*>(p.peer_out[k]) + to) = packed;
        }
    }
}

// Rows of an fp16 block once more over all of their tokens, row by row, a half-warp per token, a lane per granule.  A function of its own: as
// a part of the kernel it cost every step time, by what the compiler made of the rest (32 heads, 1 row of 1500 tokens 8.8 without it, 9.1 as a
// part, 8.9 so; 4 rows of 256 shared and 200 own 9.4, 9.8, 9.5; 12 heads of 64, 16 rows of 500 and 333 8.7, 8.8, 8.8).
template <int VG, bool PANELS, bool PEERS> __device__ __noinline__ void redo(const DirectParams& p, uint8_t* smem, int rows_again) {
    using Smem = DirectSmem<VG>;
    constexpr int DV = Smem::DV, PITCH = Smem::PITCH;
    float* const area = reinterpret_cast<float*>(smem);
    const float* const again_m = reinterpret_cast<const float*>(smem + Smem::again(p.block_rows)) + 2;
    const float* const again_inv = again_m + D_ROWS;
    const int unit = blockIdx.x / p.cluster, block = unit / p.n_heads, head = unit - block * p.n_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, C = p.chunk_size;
    const int2 rows = __ldg(p.blocks + block);
    const int row_begin = rows.x, n_rows = rows.y;
    int e_begin = 0, e_end = -1;  // the block's entries
    for (int w = 0; w < p.cluster * D_WARPS; w++) {
        const int4 of = __ldg(p.ranges + (size_t)block * (p.cluster * D_WARPS) + w);
        if (of.x > of.z) continue;
        if (e_end < 0) e_begin = of.x;
        e_end = of.z;
    }
    const int G = lane & 15;
    for (int n = 0; n < n_rows; n++) {
        if (!((rows_again >> n) & 1)) continue;
        const float mm = again_m[n], ref = mm == -INFINITY ? 0.f : mm;
        uint4 qn = make_uint4(0u, 0u, 0u, 0u);
        if (G < p.gpr) qn = __ldg(reinterpret_cast<const uint4*>(p.q) + ((size_t)(row_begin + n) * p.n_heads + head) * p.gpr + G);
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] = 0.f;
        for (int e = e_begin; e <= e_end; e++) {
            const int4 of = __ldg(p.entries + e);
            if (!((of.z >> n) & 1) || of.x < 0 || of.x >= p.max_chunks) continue;
            const int tokens = min(C, of.y + (of.w ? p.delta_tokens : 0));
            const uint8_t* const base = p.pool + ((size_t)of.x * p.n_heads + head) * (size_t)p.pair_bytes;
            for (int t0 = 0; t0 < tokens; t0 += 2 * D_WARPS) {
                const int t = t0 + 2 * warp + (lane >> 4);
                const bool on = t < tokens && G < p.gpr;
                const size_t at = PANELS ? (size_t)((((G >> 3) * C + t) * 8 + ((G & 7) ^ (t & 7))) * 16) : (size_t)((t * p.gpr + G) * 16);
                float x = 0.f;
                uint4 vn = make_uint4(0u, 0u, 0u, 0u);
                if (on) {
                    const uint4 kn = __ldg(reinterpret_cast<const uint4*>(base + at));
                    vn = __ldg(reinterpret_cast<const uint4*>(base + p.v_offset + at));
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 a = half2_of((&qn.x)[k]), b = half2_of((&kn.x)[k]);
                        x = fmaf(a.x, b.x, x);
                        x = fmaf(a.y, b.y, x);
                    }
                }
#pragma unroll
                for (int off = 8; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
                if (on) {
                    const float w = exp2f(x * p.scale_log2 - ref);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 b = half2_of((&vn.x)[k]);
                        acc[2 * k] = fmaf(w, b.x, acc[2 * k]);
                        acc[2 * k + 1] = fmaf(w, b.y, acc[2 * k + 1]);
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 16);
        if (lane < 16 && 8 * lane < DV) {
            float4* const dst = reinterpret_cast<float4*>(area + warp * PITCH + 8 * lane);
            dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
            dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        }
        __syncthreads();
        if (threadIdx.x < DV / 8 && 8 * (int)threadIdx.x < p.d) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                v[k] = 0.f;
#pragma unroll
                for (int w = 0; w < D_WARPS; w++) v[k] += area[w * PITCH + 8 * threadIdx.x + k];
            }
            const float inv = again_inv[n];
            store_half8<PEERS>(p, row_begin + n, head, 8 * (int)threadIdx.x,
                               make_uint4(pack_half2(v[0] * inv, v[1] * inv), pack_half2(v[2] * inv, v[3] * inv), pack_half2(v[4] * inv, v[5] * inv), pack_half2(v[6] * inv, v[7] * inv)));
        }
        __syncthreads();
    }
}

// KQ: groups of 4 granules of a K row; VG: groups of 8 granules of a V row; PANELS: the pool's swizzled layout (ca_layout.h).
// LO: 0 weights as one fp16 number; 1 hi and lo in two products; 2 blocks of up to 4 rows, columns 4 .. 7 repeat the rows and take
// the lo parts, so that one product does both.
// T bf16: grouped heads, with the sink and the values' turn of their layers.
template <typename T, int KQ, int VG, bool PANELS, int LO, bool PEERS>
__global__ void __launch_bounds__(D_WARPS * 32, VG == 2 ? 3 : 4) attn_direct_kernel(const __grid_constant__ DirectParams p) {
    using Smem = DirectSmem<VG>;
    constexpr int DV = Smem::DV, PITCH = Smem::PITCH;
    extern __shared__ __align__(16) uint8_t smem[];
    float* const area = reinterpret_cast<float*>(smem);                                // [warps][block_rows][PITCH]
    float* const area_m = reinterpret_cast<float*>(smem + Smem::stats(p.block_rows));  // [warps][block_rows]
    float* const area_l = area_m + D_WARPS * p.block_rows;
    int* const area_have = reinterpret_cast<int*>(area_l + D_WARPS * p.block_rows);    // [warps]: rows of which the warp saw a token
    // rows with an element that is not finite, in this CTA and among those that it stores; a row's reference and its factor
    constexpr bool REDO = LO != 0 && std::is_same_v<T, __half>;
    int* const again = reinterpret_cast<int*>(smem + Smem::again(p.block_rows));
    float* const again_m = reinterpret_cast<float*>(again + 2);
    float* const again_inv = again_m + D_ROWS;
    if (REDO && threadIdx.x < 2) again[threadIdx.x] = 0;

    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int unit = blockIdx.x / p.cluster, rank = blockIdx.x - unit * p.cluster;
    const int block = unit / p.n_heads, head = unit - block * p.n_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int4 range = __ldg(p.ranges + (size_t)block * (p.cluster * D_WARPS) + rank * D_WARPS + warp);  // entry, step | entry, step (end)
    const int2 rows = __ldg(p.blocks + block);
    constexpr bool GROUPED = std::is_same_v<T, __nv_bfloat16>;
    const int row_begin = rows.x, n_rows = GROUPED ? rows.y * p.group : rows.y;  // from here on a row is a column: a row's query head
    const int C = p.chunk_size;
    // (row, query head) of column n, numbered as in q and out
    auto pair_of = [&](int n) {
        if (!GROUPED) return (size_t)(row_begin + n) * p.n_heads + head;
        return ((size_t)(row_begin + n / p.group) * p.n_heads + head) * p.group + n % p.group;
    };

    // byte offsets of this lane's granules inside a tile, from token t0 on (a multiple of 16)
    const int row_bytes = PANELS ? 128 : p.gpr * 16;
    int k_off[KQ], v_off[VG][2];
#pragma unroll
    for (int j = 0; j < KQ; j++) {
        const int G = 4 * j + c;
        k_off[j] = PANELS ? (((G >> 3) * C + g) * 8 + ((G & 7) ^ g)) * 16 : (g * p.gpr + G) * 16;
    }
#pragma unroll
    for (int i = 0; i < VG; i++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int t = 2 * c + u;
            v_off[i][u] = PANELS ? ((i * C + t) * 8 + (g ^ t)) * 16 : (t * p.gpr + 8 * i + g) * 16;
        }

    int entry = range.x;
    int4 ahead = make_int4(0, 0, 0, 0);  // entry `entry`, requested before it is needed
    if (entry <= range.z) ahead = __ldg(p.entries + entry);
    const uint8_t* tile = p.pool;  // from the step's first token on
    int left = 0, mask = 0;        // tokens of the entry from there on that are this warp's; rows that see them
    int skip = range.y * D_STEP;   // tokens of the first entry that are other warps'
    // on to the next step with tokens; left <= 0: there is none
    auto advance = [&]() {
        left -= D_STEP;
        tile += D_STEP * row_bytes;
        while (left <= 0 && entry <= range.z) {
            const int4 e = ahead;  // chunk, tokens, rows, tail
            if (entry < range.z) ahead = __ldg(p.entries + entry + 1);
            int n = min(C, e.y + (e.w ? p.delta_tokens : 0));
            // a range may end inside its last entry; one that goes to the entry's end takes the tokens appended since, too
            if (entry == range.z) n = min(n, range.w * D_STEP);
            if (e.x < 0 || e.x >= p.max_chunks) {
                if (lane == 0) atomicCAS(p.status, STATUS_OK, STATUS_BAD_WORK_LIST);
                n = 0;
            }
            left = n - skip;
            mask = e.z;
            if (left > 0) tile = p.pool + ((size_t)e.x * p.n_heads + head) * (size_t)p.pair_bytes + (size_t)skip * row_bytes;
            skip = 0;
            entry++;
        }
    };
    uint4 kr[KQ][2], vr[VG][4];
    auto load_k = [&]() {
#pragma unroll
        for (int j = 0; j < KQ; j++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
                kr[j][u] = make_uint4(0u, 0u, 0u, 0u);
                if (g + 8 * u < left && (PANELS || 4 * j + c < p.gpr)) kr[j][u] = __ldg(reinterpret_cast<const uint4*>(tile + k_off[j] + 8 * u * row_bytes));
            }
    };
    auto load_v = [&]() {
#pragma unroll
        for (int i = 0; i < VG; i++)
#pragma unroll
            for (int u = 0; u < 4; u++) {
                vr[i][u] = make_uint4(0u, 0u, 0u, 0u);
                if (2 * c + (u & 1) + 8 * (u >> 1) < left && (PANELS || 8 * i + g < p.gpr))
                    vr[i][u] = __ldg(reinterpret_cast<const uint4*>(tile + p.v_offset + v_off[i][u & 1] + 8 * (u >> 1) * row_bytes));
            }
    };
    advance();
    if (left > 0) {
        load_k();
        load_v();
    }
    // q as the B operands: column g is row g of the block
    uint4 q[KQ];
#pragma unroll
    for (int j = 0; j < KQ; j++) {
        const int G = 4 * j + c, r = LO == 2 ? g & 3 : g;
        q[j] = make_uint4(0u, 0u, 0u, 0u);
        if (r < n_rows && G < p.gpr) q[j] = __ldg(reinterpret_cast<const uint4*>(p.q) + pair_of(r) * p.gpr + G);
    }

    float o[VG * 4][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < VG * 4; j++)
#pragma unroll
        for (int k = 0; k < 4; k++) o[j][k] = 0.f;
    int have = 0;
    while (left > 0) {
        const int n_here = left, rows_here = mask;
        float s2[2][4];
#pragma unroll
        for (int k = 0; k < 4; k++) s2[0][k] = s2[1][k] = 0.f;
#pragma unroll
        for (int j = 0; j < KQ; j++) {
            mma_16bit<T>(s2[0], kr[j][0].x, kr[j][1].x, kr[j][0].y, kr[j][1].y, q[j].x, q[j].y);
            mma_16bit<T>(s2[1], kr[j][0].z, kr[j][1].z, kr[j][0].w, kr[j][1].w, q[j].z, q[j].w);
        }
        advance();
        if (left > 0) load_k();
        float s[4];  // token g: columns 2 c, 2 c + 1; token g + 8: the same
#pragma unroll
        for (int k = 0; k < 4; k++) s[k] = g + 8 * (k >> 1) < n_here ? (s2[0][k] + s2[1][k]) * p.scale_log2 : -INFINITY;
        constexpr float STEP = Reference<T>::STEP, SHIFT = Reference<T>::SHIFT;
        if (__any_sync(0xffffffffu, fmaxf(s[0], s[2]) > m[0] + (STEP + SHIFT) || fmaxf(s[1], s[3]) > m[1] + (STEP + SHIFT))) {
            float alpha[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float mx = fmaxf(s[h], s[2 + h]);
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float mn = fmaxf(m[h], mx - SHIFT);
                alpha[h] = fast_exp2(m[h] - (mn == -INFINITY ? 0.f : mn));
                m[h] = mn;
                l[h] *= alpha[h];
            }
#pragma unroll
            for (int j = 0; j < VG * 4; j++)
#pragma unroll
                for (int k = 0; k < 4; k++) o[j][k] *= alpha[k & 1];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float ref = m[h] == -INFINITY ? 0.f : m[h];  // only scores of -inf: weights of zero
            s[h] = fast_exp2(s[h] - ref);
            s[2 + h] = fast_exp2(s[2 + h] - ref);
            l[h] += s[h] + s[2 + h];  // this lane's tokens
        }
        uint32_t hi0, lo0, hi1, lo1;
        split_pair<T>(s[0], s[1], hi0, lo0);
        split_pair<T>(s[2], s[3], hi1, lo1);
        if (LO == 2 && c >= 2) {
            hi0 = lo0;
            hi1 = lo1;
        }
        hi0 = transpose_8x8(hi0);
        hi1 = transpose_8x8(hi1);
        if (LO == 1) {
            lo0 = transpose_8x8(lo0);
            lo1 = transpose_8x8(lo1);
        }
#pragma unroll
        for (int i = 0; i < VG; i++)
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const uint32_t t0 = (&vr[i][0].x)[r], t1 = (&vr[i][1].x)[r], t8 = (&vr[i][2].x)[r], t9 = (&vr[i][3].x)[r];
                const uint32_t a0 = __byte_perm(t0, t1, 0x5410), a1 = __byte_perm(t0, t1, 0x7632);
                const uint32_t a2 = __byte_perm(t8, t9, 0x5410), a3 = __byte_perm(t8, t9, 0x7632);
                mma_16bit<T>(o[i * 4 + r], a0, a1, a2, a3, hi0, hi1);
                if (LO == 1) mma_16bit<T>(o[i * 4 + r], a0, a1, a2, a3, lo0, lo1);
            }
        if (left > 0) load_v();
        if (left <= 0 || mask != rows_here) {
            // ---- what was gathered belongs to the rows of `rows_here`: into the warp's area
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float sum = l[h];
                sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                sum += __shfl_xor_sync(0xffffffffu, sum, 8);
                sum += __shfl_xor_sync(0xffffffffu, sum, 16);
                if (LO == 2) {
#pragma unroll
                    for (int j = 0; j < VG * 4; j++)
#pragma unroll
                        for (int k = h; k < 4; k += 2) o[j][k] += __shfl_xor_sync(0xffffffffu, o[j][k], 2);
                }
                const int n = 2 * c + h, slot = warp * p.block_rows + n;
                const bool mine = (rows_here >> n) & 1, more = mine && ((have >> n) & 1);
                float keep = 0.f, scale = 1.f, mn = m[h];
                if (more) {
                    const float m0 = area_m[slot];
                    mn = fmaxf(m0, m[h]);
                    const float ref = mn == -INFINITY ? 0.f : mn;
                    keep = fast_exp2(m0 - ref);
                    scale = fast_exp2(m[h] - ref);
                    sum = sum * scale + area_l[slot] * keep;
                }
                if (mine) {
#pragma unroll
                    for (int i = 0; i < VG; i++)
#pragma unroll
                        for (int half = 0; half < 2; half++) {
                            float4* dst = reinterpret_cast<float4*>(area + slot * PITCH + 64 * i + 8 * g + 4 * half);
                            float4 v = make_float4(o[4 * i + 2 * half][h], o[4 * i + 2 * half][2 + h], o[4 * i + 2 * half + 1][h], o[4 * i + 2 * half + 1][2 + h]);
                            if (more) {
                                const float4 w = *dst;
                                v.x = v.x * scale + w.x * keep;
                                v.y = v.y * scale + w.y * keep;
                                v.z = v.z * scale + w.z * keep;
                                v.w = v.w * scale + w.w * keep;
                            }
                            *dst = v;
                        }
                }
                __syncwarp();
                if (mine && g == 0) {
                    area_m[slot] = mn;
                    area_l[slot] = sum;
                }
                m[h] = -INFINITY;
                l[h] = 0.f;
            }
            __syncwarp();
            have |= rows_here;
#pragma unroll
            for (int j = 0; j < VG * 4; j++)
#pragma unroll
                for (int k = 0; k < 4; k++) o[j][k] = 0.f;
        }
    }
    if (lane == 0) area_have[warp] = have;
    __syncthreads();

    // ---- the warps of the CTA, into the place of warp 0
    int has[D_WARPS], any = 0;
#pragma unroll
    for (int w = 0; w < D_WARPS; w++) {
        has[w] = area_have[w];
        any |= has[w];
    }
    auto weights = [&](int n, float (&a)[D_WARPS], float& mm, float& ll) {  // of the warps' results for row n
        mm = -INFINITY;
        ll = 0.f;
#pragma unroll
        for (int w = 0; w < D_WARPS; w++)
            if ((has[w] >> n) & 1) mm = fmaxf(mm, area_m[w * p.block_rows + n]);
        const float ref = mm == -INFINITY ? 0.f : mm;
#pragma unroll
        for (int w = 0; w < D_WARPS; w++) {
            a[w] = 0.f;
            if ((has[w] >> n) & 1) {
                a[w] = fast_exp2(area_m[w * p.block_rows + n] - ref);
                ll = fmaf(a[w], area_l[w * p.block_rows + n], ll);
            }
        }
    };
    for (int i = threadIdx.x; i < n_rows * (DV / 4); i += D_WARPS * 32) {
        const int n = i / (DV / 4), d = 4 * (i - n * (DV / 4));
        float a[D_WARPS], mm, ll;
        weights(n, a, mm, ll);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < D_WARPS; w++)
            if ((has[w] >> n) & 1) {
                const float4 v = *reinterpret_cast<const float4*>(area + (w * p.block_rows + n) * PITCH + d);
                acc.x = fmaf(a[w], v.x, acc.x);
                acc.y = fmaf(a[w], v.y, acc.y);
                acc.z = fmaf(a[w], v.z, acc.z);
                acc.w = fmaf(a[w], v.w, acc.w);
            }
        *reinterpret_cast<float4*>(area + n * PITCH + d) = acc;
        if (REDO && ((acc.x + acc.y) + (acc.z + acc.w)) * 0.f != 0.f) atomicOr(again, 1 << n);  // infinity and NaN times zero are NaN
    }
    float m_here = -INFINITY, l_here = 0.f;
    if (threadIdx.x < n_rows) {
        float a[D_WARPS];
        weights(threadIdx.x, a, m_here, l_here);
    }
    __syncthreads();
    if (threadIdx.x < n_rows) {
        area_m[threadIdx.x] = m_here;
        area_l[threadIdx.x] = l_here;
    }
    if (threadIdx.x == 0) area_have[0] = REDO ? any | again[0] << D_ROWS : any;
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (p.cluster > 1) cl.sync();
    else __syncthreads();
    // ---- the CTAs of the unit: the rows are dealt to them; as many lanes side by side as CTAs hold eight elements of a row, each of
    // another CTA's result, so that all are on their way at once
    const int r = threadIdx.x & (p.cluster - 1), mine = (n_rows - rank + p.cluster - 1) / p.cluster;
    const float* from = p.cluster > 1 ? cl.map_shared_rank(area, r) : area;
    const float* from_m = from + (area_m - area);
    const uint32_t group = ((1u << p.cluster) - 1) << (lane - r);  // the lanes of a row's other elements may have left the loop
    for (int i = threadIdx.x / p.cluster; i < mine * (DV / 8); i += D_WARPS * 32 / p.cluster) {
        const int n = rank + (i / (DV / 8)) * p.cluster, d = 8 * (i % (DV / 8));
        const float4 v0 = *reinterpret_cast<const float4*>(from + n * PITCH + d), v1 = *reinterpret_cast<const float4*>(from + n * PITCH + d + 4);
        const float m_r = from_m[n];
        float sum = from_m[D_WARPS * p.block_rows + n], mm = m_r, v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        int seen = reinterpret_cast<const int*>(from_m)[2 * D_WARPS * p.block_rows];
        if (p.cluster > 1) {
#pragma unroll
            for (int off = 1; off < DIRECT_MAX_CLUSTER; off <<= 1)
                if (off < p.cluster) mm = fmaxf(mm, __shfl_xor_sync(group, mm, off));
            const float a = fast_exp2(m_r - (mm == -INFINITY ? 0.f : mm));
            sum *= a;
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] *= a;
#pragma unroll
            for (int off = 1; off < DIRECT_MAX_CLUSTER; off <<= 1) {
                if (off >= p.cluster) break;
                sum += __shfl_xor_sync(group, sum, off);
                seen |= __shfl_xor_sync(group, seen, off);
#pragma unroll
                for (int k = 0; k < 8; k++) v[k] += __shfl_xor_sync(group, v[k], off);
            }
        }
        // a row with no token yields zeros; one whose scores are all -inf has no softmax (zeros where the work lists of items say so)
        float inv;
        if (GROUPED && p.sink) {  // one more entry of score zero
            const float top = fmaxf(mm, 0.f), keep = fast_exp2(mm - top);
            inv = keep / (sum * keep + fast_exp2(-top));
        } else {
            inv = mm == -INFINITY ? (((seen >> n) & 1) && !p.zero_if_none ? nanf("") : 0.f) : 1.f / sum;
        }
        if (r > 0 || d >= p.d) continue;
        if (REDO && ((seen >> (D_ROWS + n)) & 1)) {
            if (d == 0) {
                atomicOr(again + 1, 1 << n);
                again_m[n] = mm;
                again_inv[n] = inv;
            }
            continue;
        }
        if (GROUPED && p.value_freq) {  // values were cached turned by their position: back by the row's
            const float pos = (float)__ldg(p.positions + row_begin + n / p.group);
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                float sn, cs;
                fast_sincos(pos * __ldg(p.value_freq + (d + k) / 2), &sn, &cs);
                const float x = v[k] * cs + v[k + 1] * sn;
                v[k + 1] = v[k + 1] * cs - v[k] * sn;
                v[k] = x;
            }
        }
        const uint4 packed = make_uint4(pack_pair<T>(v[0] * inv, v[1] * inv), pack_pair<T>(v[2] * inv, v[3] * inv), pack_pair<T>(v[4] * inv, v[5] * inv),
                                        pack_pair<T>(v[6] * inv, v[7] * inv));
        if (GROUPED)
            *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + pair_of(n) * p.d + d) = packed;
        else
            store_half8<PEERS>(p, row_begin + n, head, d, packed);
    }
    if (p.cluster > 1) cl.sync();  // the other CTAs' shared memory is read until here
    if (!REDO) return;
    int rows_again;
    if (p.cluster == 1) {
        rows_again = area_have[0] >> D_ROWS;
        if (rows_again == 0) return;
        __syncthreads();
    } else {
        rows_again = again[1];
        if (rows_again == 0) return;
    }
    if constexpr (REDO) redo<VG, PANELS, PEERS>(p, smem, rows_again);
}

template <typename T, int KQ, int VG, bool PANELS, int LO, bool PEERS = false> cudaError_t launch(const DirectParams& p, cudaStream_t stream) {
    auto* const kernel = attn_direct_kernel<T, KQ, VG, PANELS, LO, PEERS>;
    return launch_kernel(kernel, dim3((unsigned)((int64_t)p.n_blocks * p.n_heads * p.cluster)), D_WARPS * 32, DirectSmem<VG>::bytes(p.block_rows), p.cluster,
                         (p.dependent & DEPENDENT_ATTENTION) != 0, stream, p);
}

}  // namespace

bool attn_direct_serves(const Geometry& g) {
    return g.esize == 2 && g.epg == 8 && g.d_head == g.d_value && g.d_head <= 128 && g.chunk_size >= D_STEP;
}
bool attn_direct_serves_grouped(const Geometry& g, const ca_head_shape& shape, int group) {
    return attn_direct_serves(g) && g.swz != 0 && shape.d_key == g.d_head && shape.d_value == g.d_head && group <= D_ROWS && (group & (group - 1)) == 0;
}

template <int KQ, int VG, bool PANELS> static cudaError_t launch_rows(const DirectParams& p, cudaStream_t stream) {
    if constexpr (PANELS) {
        if (p.group > 0)
            return p.n_peers > 0 ? cudaErrorInvalidValue
                                 : (p.block_rows <= 4 ? launch<__nv_bfloat16, KQ, VG, PANELS, 2>(p, stream) : launch<__nv_bfloat16, KQ, VG, PANELS, 1>(p, stream));
    }
    if constexpr (PANELS && VG == 2) {  // the geometry of the item lists
        if (p.n_peers > 0) return p.block_rows <= 4 ? launch<__half, KQ, VG, PANELS, 2, true>(p, stream) : launch<__half, KQ, VG, PANELS, 0, true>(p, stream);
        if (p.block_rows > 4 && p.one_weight) return launch<__half, KQ, VG, PANELS, 0>(p, stream);
    }
    if (p.n_peers > 0 || p.group > 0) return cudaErrorInvalidValue;
    return p.block_rows <= 4 ? launch<__half, KQ, VG, PANELS, 2>(p, stream) : launch<__half, KQ, VG, PANELS, 1>(p, stream);
}

cudaError_t launch_attn_direct(const DirectParams& p, bool panels, cudaStream_t stream) {
    if (p.n_blocks <= 0) return cudaSuccess;
    if (panels) return p.gpr == 8 ? launch_rows<2, 1, true>(p, stream) : launch_rows<4, 2, true>(p, stream);
    if (p.gpr <= 4) return launch_rows<1, 1, false>(p, stream);
    if (p.gpr <= 8) return launch_rows<2, 1, false>(p, stream);
    if (p.gpr <= 12) return launch_rows<3, 2, false>(p, stream);
    return launch_rows<4, 2, false>(p, stream);
}

}  // namespace ca
