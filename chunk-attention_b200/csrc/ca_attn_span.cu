// Causal attention of portions of prompts over the chunk pool on the Blackwell tensor path: tcgen05.mma (bf16) with
// accumulators in tensor memory, K/V chunks staged verbatim by 1-D TMA bulk copies.  For caches of 64-token chunks and
// head sizes of 64 or 128 elements, whose pool tiles are the tensor cores' own 128-byte-swizzled operand layout; other
// geometries take the mma.sync kernel (ca_attn_rows.cu).
//
// A piece of work is a (block of up to 128 query rows, key/value head).  The rows are the query heads of a group for consecutive
// tokens of one span (row r: head r % group of token r / group), and walk the span's chunks from position 0 to the last
// row's own position; only the tiles that reach past the first row's position are masked.
//   S = Q K^T      M = 128 rows, N = 64 tokens; A = the queries, one TMA tensor copy per panel; B = a K tile; D in TMEM, two
//                  buffers, so that S of tile j + 1 is computed under the softmax of tile j
//   softmax        one thread per row (= TMEM lane), fp32, log2 units; the accumulator is rescaled only when a row's
//                  maximum has grown by more than 8.  The weights go back over S as bf16 hi + lo parts (SPLIT): their sum
//                  has 16 bits of the fp32 weight
//   O += P V       A = P from TMEM, B = the V tile (MN-major panels)
// and finishes its rows: sink, normalisation, the turn back of rotated values, bf16 store through shared memory.
// Warp roles: 0-3 softmax and epilogue, 4 TMA producer over a ring of four tile slots, 5 TMEM and the MMA issue, 6 the next
// piece of work.  Two CTAs share an SM, so one's softmax runs under the other's MMAs.
//
// Why a CTA stays for several pieces: with one CTA per piece, 8 prompts of 1024 tokens (2048 pieces of 8.5 tiles on average, 32 heads on 8
// of 128) took 140 us, of which 70 were the CTAs' starts and ends (list, positions, chunk numbers, K and Q one after the
// other, then the epilogue, with nothing under them).  Now a CTA takes over pieces that have not been launched yet (cluster
// launch control: the hardware's own queue, so the balance is that of single pieces), a warp reads the next one's description
// while the present one runs, its first tiles, queries and S are fetched and computed under the epilogue, and every ring and
// phase simply goes on: 118.7 us, 64 prompts of 128 tokens 82 -> 55.5.  One long prompt (8192 tokens) is bound by the tensor pipe, 73 % busy
// with three products a tile, and stays at 575 to 590 us.
//
// Every wait is bounded: on expiry a status code is recorded, every role falls through to the common exit, and the TMEM
// columns are freed there.
#include <cuda.h>

#include <atomic>

#include "ca_kernels.h"
#include "ca_ptx.cuh"
#include "ca_softmax.cuh"
#include "ca_tensor_map.h"
#include "ca_types.cuh"

namespace ca {
namespace {
using namespace ptx;

constexpr int A_ROWS = 128, A_TOK = 64, A_SLOTS = 4, A_THREADS = 256;
constexpr int A_SOFTMAX_REGS = 200, A_OTHER_REGS = 56;  // per thread; the block is launched with 2 x 128 (checked at the launch)
constexpr int A_TMEM_COLS = 256, A_COL_S = 128;
constexpr int A_NUM_BARS = 2 * A_SLOTS + 13;
constexpr float A_NEG_BIG = -1.0e30f, A_RESCALE_STEP = 8.f;

// tcgen05.mma.kind::f16 instruction descriptor with bf16 operands (formats 1 in both operand fields)
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool b_mn_major) { return umma_idesc_f16(m, n, false, b_mn_major) | (1u << 7) | (1u << 10); }

__device__ __forceinline__ void report(int* status, int code) { atomicCAS(status, STATUS_OK, code); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// A piece of work as the roles read it; n_tiles = 0: there is none left
struct alignas(16) Work {
    int token0, n_rows, n_tiles;
    int tail;   // tokens of the last tile
    int open;   // tokens every row of the block sees
    int kvh;
    int withheld;  // failure-path tests: the producer stops here
    const int32_t* list;
};

template <int DK, int DV> struct Sizes {
    static constexpr int Q_BYTES = A_ROWS * DK * 2, Q_PANEL = A_ROWS * 128;
    static constexpr int K_BYTES = A_TOK * DK * 2, V_BYTES = A_TOK * DV * 2;
    static constexpr int SLOT = K_BYTES > V_BYTES ? K_BYTES : V_BYTES;
    static constexpr int OUT_PITCH = 64 + 16;  // 32 columns of a row at a time
    static constexpr int OUT = Q_BYTES + A_SLOTS * SLOT;
    static constexpr int WORK = OUT + A_ROWS * OUT_PITCH, CLC = WORK + 2 * (int)sizeof(Work), BARS = CLC + 16;
    static constexpr int SMEM = BARS + A_NUM_BARS * 8 + 8;
};

template <int DK, int DV, bool SPLIT>
__global__ void __launch_bounds__(A_THREADS, 2) span_attn_kernel(const SpanAttnParams p, const __grid_constant__ CUtensorMap q_map) {
    using Z = Sizes<DK, DV>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const uint32_t ring = sbase + Z::Q_BYTES;
    const uint32_t full_bar = sbase + Z::BARS;
    const uint32_t empty_bar = full_bar + 8 * A_SLOTS;
    const uint32_t s_full = empty_bar + 8 * A_SLOTS;  // [2]
    const uint32_t p_full = s_full + 16;              // [2]
    const uint32_t work_full = p_full + 16;           // [2]
    const uint32_t work_empty = work_full + 16;       // [2]
    const uint32_t o_done = work_empty + 16;
    const uint32_t o_free = o_done + 8;
    const uint32_t q_full = o_free + 8;
    const uint32_t q_empty = q_full + 8;
    const uint32_t clc_bar = q_empty + 8;
    Work* const work = reinterpret_cast<Work*>(smem + Z::WORK);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Z::BARS + A_NUM_BARS * 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.n_kv_heads, group = p.group, H = G * group;

    if (threadIdx.x == 0) {
        for (int i = 0; i < A_SLOTS; i++) {
            mbar_init(full_bar + 8 * i, 1);
            mbar_init(empty_bar + 8 * i, 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(s_full + 8 * b, 1);
            mbar_init(p_full + 8 * b, 4 * 32);
            mbar_init(work_full + 8 * b, 1);
            mbar_init(work_empty + 8 * b, 4 * 32 + 2);
        }
        mbar_init(o_done, 1);
        mbar_init(o_free, 4 * 32);
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        mbar_init(clc_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {  // the warp that allocates is the warp that frees
        tmem_alloc(smem_u32(tmem_slot), A_TMEM_COLS);
        tmem_relinquish_alloc_permit();
    }
    tc_fence_before_thread_sync();
    __syncthreads();
    tc_fence_after_thread_sync();
    const uint32_t tmem_base = *tmem_slot;
    // a wait of a single thread: false, with the code recorded, when the limit ran out
    auto wait = [&](uint32_t bar, int parity, int code) {
        if (mbar_wait_bounded(bar, parity, p.wait_limit)) return true;
        report(p.status, code);
        return false;
    };

    if (warp >= 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(A_OTHER_REGS));
        if (warp == 6 && lane == 0) {
            // ---- the next piece of work, asked for when the piece before the present one is finished
            int item = blockIdx.x;
            for (int n = 0;; n++) {
                if (n > 0) {
                    if (!wait(work_empty + 8 * (n & 1), ((n >> 1) & 1) ^ 1, STATUS_EMPTY_WAIT_TIMEOUT)) break;
                    mbar_arrive_expect_tx(clc_bar, 16);
                    clc_try_cancel(sbase + Z::CLC, clc_bar);
                    if (!wait(clc_bar, (n - 1) & 1, STATUS_FULL_WAIT_TIMEOUT)) {
                        wait(clc_bar, (n - 1) & 1, STATUS_DRAIN_TIMEOUT);  // the answer is still on its way into this CTA's memory
                        break;
                    }
                    item = clc_block(sbase + Z::CLC);
                    fence_proxy_async();  // read before the next answer is written
                }
                Work w{};
                if (item >= 0) {
                    const int4 blk = __ldg(reinterpret_cast<const int4*>(p.blocks) + item / G);
                    const int n_ctx = __ldg(p.positions + blk.z - 1) + 1;
                    w.token0 = blk.y;
                    w.n_rows = (blk.z - blk.y) * group;
                    w.n_tiles = (n_ctx + A_TOK - 1) / A_TOK;
                    w.tail = n_ctx - (w.n_tiles - 1) * A_TOK;
                    w.open = __ldg(p.positions + blk.y) + 1;
                    w.kvh = item % G;
                    w.withheld = item == p.withhold_item;
                    w.list = p.path_chunks + __ldg(p.path_off + blk.x);
                }
                work[n & 1] = w;
                mbar_arrive(work_full + 8 * (n & 1));
                if (item < 0) break;
            }
        } else if (warp == 4 && lane == 0) {
            // ---- producer: slot i & 3 takes K of tile i / 2 (even i) or its V (odd i), i counted over all pieces
            int issued = 0, q_issued = 0, n = 0;
            for (bool live = true; live; n++) {
                if (!wait(work_full + 8 * (n & 1), (n >> 1) & 1, STATUS_FULL_WAIT_TIMEOUT)) break;
                const Work w = work[n & 1];
                mbar_arrive(work_empty + 8 * (n & 1));
                if (w.n_tiles == 0) break;
                int chunk = __ldg(w.list);
                for (int j = 0; j < w.n_tiles && live; j++) {
                    const int next = j + 1 < w.n_tiles ? __ldg(w.list + j + 1) : 0;  // on its way while slots are waited for
                    if (chunk < 0 || chunk >= p.max_chunks) {
                        report(p.status, STATUS_BAD_WORK_LIST);  // keep the pipeline moving on a chunk that exists
                        chunk = 0;
                    }
                    const uint8_t* src = static_cast<const uint8_t*>(p.pool) + ((size_t)chunk * G + w.kvh) * (size_t)(Z::K_BYTES + Z::V_BYTES);
                    const uint32_t lines = j + 1 < w.n_tiles ? A_TOK : w.tail;
                    for (int side = 0; side < 2; side++) {
                        const int slot = issued & (A_SLOTS - 1);
                        if (!wait(empty_bar + 8 * slot, ((issued / A_SLOTS) & 1) ^ 1, STATUS_EMPTY_WAIT_TIMEOUT)) {
                            live = false;
                            break;
                        }
                        const uint32_t dst = ring + slot * Z::SLOT, bar = full_bar + 8 * slot;
                        const int panels = side ? DV / 64 : DK / 64;
                        const uint8_t* from = src + side * Z::K_BYTES;
                        mbar_arrive_expect_tx(bar, panels * lines * 128);
                        if (lines == A_TOK) {
                            bulk_copy_g2s(dst, from, panels * A_TOK * 128, bar);
                        } else {
                            for (int pn = 0; pn < panels; pn++) bulk_copy_g2s(dst + pn * (A_TOK * 128), from + pn * (A_TOK * 128), lines * 128, bar);
                        }
                        issued++;
                        if (j == 0 && side == 0) {
                            // the queries follow the first K tile.  Rows past the block are other tokens' or zeros: nobody reads theirs
                            if (w.withheld || !wait(q_empty, (n & 1) ^ 1, STATUS_EMPTY_WAIT_TIMEOUT)) {
                                live = false;
                                break;
                            }
                            mbar_arrive_expect_tx(q_full, (DK / 64) * p.block_tokens * group * 128);
#pragma unroll
                            for (int pn = 0; pn < DK / 64; pn++) tma_load_3d(sbase + pn * Z::Q_PANEL, &q_map, 64 * pn, w.kvh * group, w.token0, q_full);
                            q_issued++;
                        }
                    }
                    chunk = next;
                }
            }
            for (int f = issued > A_SLOTS ? issued - A_SLOTS : 0; f < issued; f++)
                if (!wait(full_bar + 8 * (f & (A_SLOTS - 1)), (f / A_SLOTS) & 1, STATUS_DRAIN_TIMEOUT)) break;
            if (q_issued > 0) wait(q_full, (q_issued - 1) & 1, STATUS_DRAIN_TIMEOUT);  // pieces begun may be one more
        } else if (warp == 5 && elect_one()) {
            // ---- MMA issuer: one thread; t counts tiles over all pieces
            constexpr uint32_t DESC_HI = umma_desc_sw128_hi(1024);
            constexpr uint32_t IDESC_QK = idesc_bf16(A_ROWS, A_TOK, false), IDESC_PV = idesc_bf16(A_ROWS, DV, true);
            const uint32_t q_lo = umma_desc_sw128_lo(sbase, 16);
            auto issue_qk = [&](int t) {
                const int i = 2 * t, slot = i & (A_SLOTS - 1);
                if (!wait(full_bar + 8 * slot, (i / A_SLOTS) & 1, STATUS_FULL_WAIT_TIMEOUT)) return false;
                tc_fence_after_thread_sync();
                const uint32_t d = tmem_base + A_COL_S + (t & 1) * A_TOK;
                const uint32_t b_lo = umma_desc_sw128_lo(ring + slot * Z::SLOT, 16);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ks++) {
                    const uint64_t a = umma_desc_pack(q_lo + (((ks >> 2) * Z::Q_PANEL + (ks & 3) * 32) >> 4), DESC_HI);
                    const uint64_t b = umma_desc_pack(b_lo + (((ks >> 2) * (A_TOK * 128) + (ks & 3) * 32) >> 4), DESC_HI);
                    umma_ss_f16(d, a, b, IDESC_QK, ks > 0 ? 1u : 0u);
                }
                umma_commit(s_full + 8 * (t & 1));
                umma_commit(empty_bar + 8 * slot);
                return true;
            };
            int t = 0;
            bool live = true;
            for (int n = 0; live; n++) {
                if (!wait(work_full + 8 * (n & 1), (n >> 1) & 1, STATUS_FULL_WAIT_TIMEOUT)) break;
                const int n_tiles = work[n & 1].n_tiles;
                mbar_arrive(work_empty + 8 * (n & 1));
                if (n_tiles == 0) break;
                live = wait(q_full, n & 1, STATUS_FULL_WAIT_TIMEOUT) && issue_qk(t);
                if (live && n_tiles == 1) umma_commit(q_empty);
                for (int j = 0; j < n_tiles && live; j++, t++) {
                    if (j + 1 < n_tiles) {
                        if (!(live = issue_qk(t + 1))) break;
                        if (j + 2 == n_tiles) umma_commit(q_empty);
                    }
                    const int i = 2 * t + 1, slot = i & (A_SLOTS - 1);
                    live = wait(p_full + 8 * (t & 1), (t >> 1) & 1, STATUS_FULL_WAIT_TIMEOUT) &&
                           wait(full_bar + 8 * slot, (i / A_SLOTS) & 1, STATUS_FULL_WAIT_TIMEOUT) &&
                           (j > 0 || wait(o_free, (n & 1) ^ 1, STATUS_FULL_WAIT_TIMEOUT));  // the piece before has read its O
                    if (!live) break;
                    tc_fence_after_thread_sync();
                    const uint32_t a_tmem = tmem_base + A_COL_S + (t & 1) * A_TOK;  // hi parts, then lo parts, two bf16 per column
                    const uint32_t v_lo = umma_desc_sw128_lo(ring + slot * Z::SLOT, A_TOK * 128);
#pragma unroll
                    for (int part = 0; part < (SPLIT ? 2 : 1); part++)
#pragma unroll
                        for (int kk = 0; kk < 4; kk++) {
                            const uint64_t b = umma_desc_pack(v_lo + ((kk * 2048) >> 4), DESC_HI);
                            umma_ts_f16(tmem_base, a_tmem + part * 32 + kk * 8, b, IDESC_PV, (j > 0 || kk > 0 || part > 0) ? 1u : 0u);
                        }
                    umma_commit(empty_bar + 8 * slot);
                    umma_commit(o_done);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(A_SOFTMAX_REGS));
        // ---- softmax: thread r owns query row r = TMEM lane r
        const int r = threadIdx.x;
        // a negative scale: the largest score is then that of the negated product
        const uint32_t flip = p.scale_log2 < 0.f ? 0x80000000u : 0u;
        const float scale = fabsf(p.scale_log2);
        const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
        uint8_t* const stage = smem + Z::OUT + warp * 32 * Z::OUT_PITCH;
        auto wait_all = [&](uint32_t bar, int parity) {  // by a whole warp
            const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, p.wait_limit));
            if (!ok && lane == 0) report(p.status, STATUS_FULL_WAIT_TIMEOUT);
            return ok;
        };
        int t = 0;
        bool live = true;
        for (int n = 0; live; n++) {
            if (!wait_all(work_full + 8 * (n & 1), (n >> 1) & 1)) break;
            const Work w = work[n & 1];
            if (w.n_tiles == 0) break;
            const bool active = r < w.n_rows;
            const int my_token = w.token0 + (active ? r / group : 0);
            const int limit = active ? __ldg(p.positions + my_token) + 1 : 0;
            float m_used = A_NEG_BIG, l = 0.f;
            for (int j = 0; j < w.n_tiles; j++, t++) {
                const int b = t & 1;
                if (!(live = wait_all(s_full + 8 * b, (t >> 1) & 1))) break;
                tc_fence_after_thread_sync();
                uint32_t s0[32], s1[32];
                tmem_ld32(lane_addr + A_COL_S + b * A_TOK, s0);
                tmem_ld32(lane_addr + A_COL_S + b * A_TOK + 32, s1);
                tmem_wait_ld();
                if (flip) {
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        s0[i] ^= flip;
                        s1[i] ^= flip;
                    }
                }
                if ((j + 1) * A_TOK > w.open) {
                    const int seen = limit - j * A_TOK;
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        if (i >= seen) s0[i] = 0xff800000u;
                        if (32 + i >= seen) s1[i] = 0xff800000u;
                    }
                }
                float alpha = 1.f;
                bool rescale = false;
                {
                    const float mx = fmaxf(tile_max(s0, s1) * scale, A_NEG_BIG);
                    if (j == 0) {
                        m_used = mx;
                    } else if (mx > m_used + A_RESCALE_STEP) {
                        alpha = fast_exp2(m_used - mx);
                        m_used = mx;
                        l *= alpha;
                        rescale = true;
                    }
                }
                l += tile_weights(s0, s1, scale, m_used);
                uint32_t pk[32];
                if (SPLIT) {
                    uint32_t lo[32];
                    split_weights(s0, pk, lo);
                    split_weights(s1, pk + 16, lo + 16);
                    tmem_st32(lane_addr + A_COL_S + b * A_TOK, pk);
                    tmem_st32(lane_addr + A_COL_S + b * A_TOK + 32, lo);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        pk[i] = pack_bf16(__uint_as_float(s0[2 * i]), __uint_as_float(s0[2 * i + 1]));
                        pk[16 + i] = pack_bf16(__uint_as_float(s1[2 * i]), __uint_as_float(s1[2 * i + 1]));
                    }
                    tmem_st32(lane_addr + A_COL_S + b * A_TOK, pk);
                }
                // O += P V of tile t - 1 is complete (every thread follows o_done phase by phase)
                if (j > 0 && !(live = wait_all(o_done, (t - 1) & 1))) break;
                if (__any_sync(0xffffffffu, rescale)) {
                    tc_fence_after_thread_sync();
#pragma unroll 1
                    for (int c = 0; c < DV / 32; c++) {
                        uint32_t o[32];
                        tmem_ld32(lane_addr + c * 32, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st32(lane_addr + c * 32, o);
                    }
                }
                if (j + 1 == w.n_tiles && w.tail < A_TOK) {
                    // Only the stored tokens of the last tile are copied.  The rows of V behind them meet weights of zero, so they
                    // only have to be finite; the slot's earlier tile may be another sequence's.  Its MMA, of tile t - 2, is complete.
                    const uint32_t v_slot = ring + ((2 * t + 1) & (A_SLOTS - 1)) * Z::SLOT;
                    const int grans = (A_TOK - w.tail) * 8;
                    for (int i = r; i < (DV / 64) * grans; i += 4 * 32)
                        sts128_zero(v_slot + (i / grans) * (A_TOK * 128) + w.tail * 128 + (i % grans) * 16);
                    fence_proxy_async();
                }
                tmem_wait_st();
                tc_fence_before_thread_sync();
                mbar_arrive(p_full + 8 * b);
            }
            if (!live || !(live = wait_all(o_done, (t - 1) & 1))) break;
            tc_fence_after_thread_sync();
            // ---- epilogue: the sink has score 0; rows leave as bf16, 32 columns at a time through the warp's own shared memory
            float inv;
            {
                float total = l;
                float M = m_used;
                if (p.sink) {
                    M = fmaxf(m_used, 0.f);
                    total = l * fast_exp2(m_used - M) + fast_exp2(-M);
                }
                inv = total > 0.f ? fast_exp2(m_used - M) / total : 0.f;
            }
            const float pos = (float)(limit - 1);
            const int rows_here = min(32, w.n_rows - warp * 32);
            __nv_bfloat16* to[4];  // four lanes to a row
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int row = warp * 32 + 8 * k + (lane >> 2), token = w.token0 + row / group, head = w.kvh * group + row % group;
                to[k] = static_cast<__nv_bfloat16*>(p.out) + ((size_t)token * H + head) * DV + 8 * (lane & 3);
            }
            // A loop, not unrolled: this code runs once a piece, and straight through it the warps waited for instructions
#pragma unroll 1
            for (int c = 0; c < DV / 32; c++) {
                uint32_t o[32];
                tmem_ld32(lane_addr + c * 32, o);
                tmem_wait_ld();
                if (c == DV / 32 - 1) {  // the accumulator may be overwritten
                    tc_fence_before_thread_sync();
                    mbar_arrive(o_free);
                }
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float a = __uint_as_float(o[2 * i]) * inv, bb = __uint_as_float(o[2 * i + 1]) * inv;
                    if (p.value_freq) {
                        float sn, cs;
                        fast_sincos(pos * __ldg(p.value_freq + c * 16 + i), &sn, &cs);
                        const float u = a * cs + bb * sn;
                        bb = bb * cs - a * sn;
                        a = u;
                    }
                    o[i] = pack_bf16(a, bb);
                }
                __syncwarp();  // the 32 columns before have been read
#pragma unroll
                for (int i = 0; i < 4; i++)
                    *reinterpret_cast<uint4*>(stage + lane * Z::OUT_PITCH + 16 * i) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int rr = 8 * k + (lane >> 2);
                    const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * Z::OUT_PITCH + 16 * (lane & 3));
                    if (rr < rows_here) *reinterpret_cast<uint4*>(to[k] + 32 * c) = v;
                }
            }
            mbar_arrive(work_empty + 8 * (n & 1));
        }
    }
    // ---- common exit: nobody touches TMEM after this barrier, then the allocating warp frees it
    tc_fence_before_thread_sync();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after_thread_sync();
        tmem_dealloc(tmem_base, A_TMEM_COLS);
    }
}

// Queries as [tokens][heads][d] in boxes of one panel of a group's heads for a block's tokens: the rows of a block in their order
bool make_query_map(CUtensorMap* m, const SpanAttnParams& p, int d) {
    const TensorMapEncode encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t heads = (cuuint64_t)p.n_kv_heads * p.group;
    const cuuint64_t dims[3] = {(cuuint64_t)d, heads, (cuuint64_t)p.n_tokens}, strides[2] = {(cuuint64_t)d * 2, heads * d * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)p.group, (cuuint32_t)p.block_tokens}, step[3] = {1, 1, 1};
    return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p.q), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int DK, int DV>
cudaError_t launch(const SpanAttnParams& p, cudaStream_t stream) {
    auto* k = p.split_weights ? span_attn_kernel<DK, DV, true> : span_attn_kernel<DK, DV, false>;
    constexpr int smem = Sizes<DK, DV>::SMEM;
    static_assert(2 * (smem + 1024) <= 233472, "two CTAs do not fit in one SM's shared memory");
    CUtensorMap queries;
    if (!make_query_map(&queries, p, DK)) return cudaErrorInvalidValue;
    // With fewer registers the warps would wait for them for good.  What the compiler gave the kernel does not change: asking on every
    // launch made a call on a short prompt wait 1.1 us longer for its host part (40 tokens: 9.6 us a call, 8.5 so).
    static std::atomic<bool> enough[2];
    cudaError_t e = cudaSuccess;
    if (!enough[p.split_weights ? 1 : 0]) {
        cudaFuncAttributes have;
        e = cudaFuncGetAttributes(&have, k);
        if (e == cudaSuccess && 2 * have.numRegs < A_SOFTMAX_REGS + A_OTHER_REGS) e = cudaErrorInvalidConfiguration;
        if (e == cudaSuccess) enough[p.split_weights ? 1 : 0] = true;
    }
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    k<<<p.n_blocks * p.n_kv_heads, A_THREADS, smem, stream>>>(p, queries);
    return cudaGetLastError();
}

}  // namespace

bool span_attn_serves(const Geometry& g, int d_value, int block_query_rows) {
    return g.esize == 2 && g.chunk_size == A_TOK && (g.d_head == 64 || g.d_head == 128) && (g.d_value == 64 || g.d_value == 128) &&
           g.d_value == d_value && block_query_rows <= A_ROWS;
}

cudaError_t launch_span_attn(const SpanAttnParams& p, int d_key, int d_value, cudaStream_t stream) {
    if (d_key == 128) return d_value == 128 ? launch<128, 128>(p, stream) : launch<128, 64>(p, stream);
    return d_value == 128 ? launch<64, 128>(p, stream) : launch<64, 64>(p, stream);
}

}  // namespace ca
