// Sequence-first-only attention for any geometry (fp16 or fp32, d_head <= 256, any chunk
// size), fp32 arithmetic with accurate expf.  It serves the geometries the tensor-core/TMA kernels
// do not (the reference's CPU tests use fp32 with d_head 4..128 and chunk sizes 2..1024,
// tests/test_chunk_attn_cpu.py:24-385), `partition = 2` requests (the reference's
// sequence-first-only mode, cpp/chunk_attn/kernel_cpu_mkl.cpp:122-242), and is the in-library
// cross-check of the fast path.
//
// attn_split_kernel (rows of whole 16-byte granules): a CLUSTER of 1 to 8 CTAs of 4 warps per (row, head).  The row's
// root-to-leaf path is cut into blocks of 4 to 32 tokens that all warps of the cluster take in turn.  LPT (8, or 4 for
// narrow heads) neighbouring lanes share a token: each holds granules sub, sub + LPT, ... of its K and V row, so a warp
// load covers whole 128-byte lines of 32 / LPT tokens, and all K and V loads of a block are in flight together.  Every
// group of LPT lanes keeps its own running (max, sum, O); groups, warps and CTAs are combined once at the end, the CTAs
// through distributed shared memory.
// Bound: latency.  A block is a chain of one memory access and a handful of shuffles and exponentials, about 1.3 us from
// cold memory, so what counts is how few blocks a warp walks in a row.  Measured (B200, kernel alone, one CTA per row with a
// lane per token -> this kernel): 4 x 288 tokens, 8 fp32 heads of 64: 32.4 -> 5.5 us; 16 x 833, 12 fp16 heads of 64:
// 73.5 -> 11.7 us.
// attn_elem_kernel (rows that are not whole granules, odd d_head): one CTA per (row, head), a warp per 32 tokens, lane j
// computes the score of token j element by element.
//
// A row is one query token: the last token of a sequence (decode), or token t of a batch of portions
// (prefill), which then sees the positions up to its own.  Grouped heads, values of another width
// than the keys, a unit term in the softmax denominator and values that were cached rotated
// (the output row is turned back) are parameters of the walk.
#include <cooperative_groups.h>

#include "ca_kernels.h"
#include "ca_launch.cuh"
#include "ca_types.cuh"

namespace ca {
namespace {

constexpr int GEN_WARPS = 4;
constexpr int GEN_MAX_D = 256;
// CTAs up to which a row's cluster grows.  Measured at 1, 2 and 4 times this (16 x 500 + 256 tokens, 8 fp32 heads of 64):
// 9.5 / 14.2 / 14.2 us, 16 x 833 fp16: 11.7 / 12.3 / 14.9: more CTAs of a cluster only wait for each other.
constexpr int64_t GEN_SPLIT_CTAS = B200_SMS * 4;

// A finished row leaves: value(e) is element e of it.  Values that were cached turned by their own position are turned
// back by the row's.
template <typename T, typename F> __device__ __forceinline__ void store_row(const GenericParams& p, int pair, int row, F value) {
    const int width = p.out_width;  // stored elements of a value row, without padding
    T* out = reinterpret_cast<T*>(p.out) + (size_t)pair * width;
    if (!p.value_freq) {
        for (int e = threadIdx.x; e < width; e += blockDim.x) out[e] = from_f32<T>(value(e));
        return;
    }
    const float pos = (float)p.positions[row];
    for (int i = threadIdx.x; 2 * i < width; i += blockDim.x) {
        const float a = value(2 * i), b = 2 * i + 1 < width ? value(2 * i + 1) : 0.f;
        float sn, cs;
        sincosf(pos * p.value_freq[i], &sn, &cs);
        out[2 * i] = from_f32<T>(a * cs + b * sn);
        if (2 * i + 1 < width) out[2 * i + 1] = from_f32<T>(b * cs - a * sn);
    }
}

// A lane owns elements lane + 32 i of the output row.
template <typename T>
__global__ void __launch_bounds__(GEN_WARPS * 32) attn_elem_kernel(const GenericParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr int OWN = GEN_MAX_D / 32;  // output elements a lane may own
    __shared__ float q_s[GEN_MAX_D];
    __shared__ float part[GEN_WARPS][GEN_MAX_D + 2];

    const int pair = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_q_heads = p.geo.n_heads * p.group;
    const int row = pair / n_q_heads;
    const int qh = pair - row * n_q_heads;
    const int h = qh / p.group;  // key/value head
    const int d = p.geo.d_head, dv = p.geo.d_value;
    const Geometry v_side = tile_side(p.geo, 1);
    const int s = p.row_entry ? p.row_entry[row] : row;  // whose path the row walks
    const int limit = p.row_entry ? p.positions[row] + 1 : 0x7fffffff;  // tokens of it the row sees
    const T* pool = reinterpret_cast<const T*>(p.pool);
    {
        const T* q = reinterpret_cast<const T*>(p.q) + (size_t)pair * d;
        for (int e = threadIdx.x; e < d; e += blockDim.x) q_s[e] = to_f32(q[e]) * p.scale;
    }
    __syncthreads();

    float o[OWN];
#pragma unroll
    for (int i = 0; i < OWN; i++) o[i] = 0.f;
    float m = -INFINITY, l = 0.f;

    const int pb = p.path_off[s], pe = p.path_off[s + 1];
    int turn = 0;  // blocks are dealt to the warps round-robin
    int first = 0; // position of the chunk's first token
    for (int pi = pb; pi < pe && first < limit; pi++) {
        int nt = p.path_tokens ? p.path_tokens[pi] : p.geo.chunk_size;
        if (pi == pe - 1 && p.path_tokens) nt = min(nt + p.delta_tokens, p.geo.chunk_size);  // the row's tail
        const int before = first;
        first += nt;
        nt = min(nt, limit - before);
        const T* kt = pool + tile_base_elems(p.geo, p.path_chunks[pi], h, 0);
        const T* vt = kt + p.geo.tile_elems;
        for (int t0 = 0; t0 < nt; t0 += 32, turn++) {
            if ((turn & (GEN_WARPS - 1)) != warp) continue;
            const int nv = min(32, nt - t0);
            const int t = t0 + lane;
            // ---- scores: lane j <-> token t0 + j
            float sc = -INFINITY;
            if (lane < nv) {
                float acc = 0.f;
                for (int e = 0; e < d; e++) acc = fmaf(q_s[e], to_f32(kt[tile_elem_offset(p.geo, t, e)]), acc);
                sc = acc;
            }
            // ---- online softmax over the block
            const float mn = fmaxf(m, warp_max(sc));
            const float alpha = expf(m - mn);  // exp(-inf) = 0 before the first token
            const float pj = lane < nv ? expf(sc - mn) : 0.f;
            l = l * alpha + warp_sum(pj);
            m = mn;
#pragma unroll
            for (int i = 0; i < OWN; i++) o[i] *= alpha;
            // ---- O += P V: every lane walks the block's tokens over the elements it owns
            for (int j = 0; j < nv; j++) {
                const float pw = __shfl_sync(0xffffffffu, pj, j);
                const int tj = t0 + j;
#pragma unroll
                for (int i = 0; i < OWN; i++) {
                    const int e = lane + 32 * i;
                    if (e < dv) o[i] = fmaf(pw, to_f32(vt[tile_elem_offset(v_side, tj, e)]), o[i]);
                }
            }
        }
    }

    // ---- combine the warps
    if (lane == 0) {
        part[warp][GEN_MAX_D] = m;
        part[warp][GEN_MAX_D + 1] = l;
    }
#pragma unroll
    for (int i = 0; i < OWN; i++) {
        const int e = lane + 32 * i;
        if (e < dv) part[warp][e] = o[i];
    }
    __syncthreads();
    float mm = p.sink ? 0.f : -INFINITY;  // the sink is a score of 0 without a value
#pragma unroll
    for (int w = 0; w < GEN_WARPS; w++) mm = fmaxf(mm, part[w][GEN_MAX_D]);
    float wgt[GEN_WARPS];
    float ll = p.sink ? expf(-mm) : 0.f;
#pragma unroll
    for (int w = 0; w < GEN_WARPS; w++) {
        // a warp that saw no token has max -inf and sum 0: it contributes nothing
        wgt[w] = part[w][GEN_MAX_D + 1] > 0.f ? expf(part[w][GEN_MAX_D] - mm) : 0.f;
        ll = fmaf(wgt[w], part[w][GEN_MAX_D + 1], ll);
    }
    const float inv = ll > 0.f ? 1.f / ll : 0.f;  // a row with no token yields zeros
    store_row<T>(p, pair, row, [&](int e) {
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < GEN_WARPS; w++) acc = fmaf(wgt[w], part[w][e], acc);
        return acc * inv;
    });
}

// ---- rows of whole granules ---------------------------------------------------------------------------------------------
// LPT lanes per token, GPL granules per lane (of a K row and of a V row), U tokens per lane and block.
template <typename T, int LPT, int GPL, int U>
__global__ void __launch_bounds__(GEN_WARPS * 32) attn_split_kernel(const GenericParams p, const int cluster) {
    constexpr int EPG = Granule<T>::N, TPG = 32 / LPT, BLOCK = TPG * U, SPAN = LPT * GPL * EPG;
    __shared__ float part[GEN_WARPS][SPAN];
    __shared__ float part_m[GEN_WARPS], part_l[GEN_WARPS];
    __shared__ int part_seen[GEN_WARPS];
    __shared__ float comb[SPAN + 3];  // this CTA's O, max, sum, and whether it saw a token

    // launched as a programmatic dependent: nothing in global memory is touched before the kernel ahead is complete
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int pair = blockIdx.x / cluster, rank = blockIdx.x - pair * cluster;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane % LPT, grp = lane / LPT;
    const int n_q_heads = p.geo.n_heads * p.group;
    const int row = pair / n_q_heads;
    const int h = (pair - row * n_q_heads) / p.group;  // key/value head
    const int C = p.geo.chunk_size, gpr = p.geo.gpr, v_gpr = p.geo.v_gpr;
    const int s = p.row_entry ? p.row_entry[row] : row;  // whose path the row walks
    const T* pool = reinterpret_cast<const T*>(p.pool);

    float q[GPL][EPG];
#pragma unroll
    for (int i = 0; i < GPL; i++) {
        const int g = sub + LPT * i;
        const T* src = reinterpret_cast<const T*>(p.q) + (size_t)pair * p.geo.d_head + g * EPG;
#pragma unroll
        for (int k = 0; k < EPG; k++) q[i][k] = g < gpr ? to_f32(src[k]) * p.scale : 0.f;
    }

    const int pb = p.path_off[s], pe = p.path_off[s + 1];
    const int blocks_per_chunk = (C + BLOCK - 1) / BLOCK;
    // with path_tokens (decode) a row sees what its chunks hold, else the positions up to its own
    int limit = 0x7fffffff, n_chunks = pe - pb;
    if (p.row_entry) {
        limit = p.positions[row] + 1;
        if (!p.path_tokens) n_chunks = min(n_chunks, (limit + C - 1) / C);
    }
    const int n_blocks = n_chunks * blocks_per_chunk;

    float m = -INFINITY, l = 0.f, o[GPL][EPG];
    bool seen = false;
#pragma unroll
    for (int i = 0; i < GPL; i++)
#pragma unroll
        for (int k = 0; k < EPG; k++) o[i][k] = 0.f;

    for (int b = rank * GEN_WARPS + warp; b < n_blocks; b += cluster * GEN_WARPS) {
        const int ci = b / blocks_per_chunk, t0 = (b - ci * blocks_per_chunk) * BLOCK, pi = pb + ci;
        int nt = C;
        if (p.path_tokens) {
            nt = p.path_tokens[pi];
            if (pi == pe - 1) nt = min(nt + p.delta_tokens, C);  // the row's tail
        } else {
            nt = min(C, limit - ci * C);
        }
        if (t0 >= nt) continue;
        const T* kt = pool + tile_base_elems(p.geo, p.path_chunks[pi], h, 0);
        const T* vt = kt + p.geo.tile_elems;
        Pack<T, EPG> kr[U][GPL], vr[U][GPL];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int t = t0 + u * TPG + grp;
#pragma unroll
            for (int i = 0; i < GPL; i++) {
                const int g = sub + LPT * i;
                const int kg = p.geo.swz ? ((g >> 3) * C + t) * 8 + ((g & 7) ^ (t & 7)) : t * gpr + g;
                const int vg = p.geo.v_swz ? ((g >> 3) * C + t) * 8 + ((g & 7) ^ (t & 7)) : t * v_gpr + g;
                uint4 z = make_uint4(0, 0, 0, 0), w = z;
                if (t < nt && g < gpr) z = __ldg(reinterpret_cast<const uint4*>(kt) + kg);
                if (t < nt && g < v_gpr) w = __ldg(reinterpret_cast<const uint4*>(vt) + vg);
                kr[u][i] = *reinterpret_cast<Pack<T, EPG>*>(&z);
                vr[u][i] = *reinterpret_cast<Pack<T, EPG>*>(&w);
            }
        }
        float sc[U], mn = m;
#pragma unroll
        for (int u = 0; u < U; u++) {
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < GPL; i++)
#pragma unroll
                for (int k = 0; k < EPG; k++) acc = fmaf(q[i][k], to_f32(kr[u][i].v[k]), acc);
#pragma unroll
            for (int off = 1; off < LPT; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
            const bool on = t0 + u * TPG + grp < nt;
            seen |= on;
            sc[u] = on ? acc : -INFINITY;
            mn = fmaxf(mn, sc[u]);
        }
        const float ref = mn == -INFINITY ? 0.f : mn;  // nothing seen yet, or only scores of -inf: weights of zero
        const float alpha = expf(m - ref);
        m = mn;
        l *= alpha;
#pragma unroll
        for (int u = 0; u < U; u++) {
            sc[u] = expf(sc[u] - ref);
            l += sc[u];
        }
#pragma unroll
        for (int i = 0; i < GPL; i++)
#pragma unroll
            for (int k = 0; k < EPG; k++) {
                float acc = o[i][k] * alpha;
#pragma unroll
                for (int u = 0; u < U; u++) acc = fmaf(sc[u], to_f32(vr[u][i].v[k]), acc);
                o[i][k] = acc;
            }
    }

    // ---- the groups of a warp, then the warps, then the CTAs
#pragma unroll
    for (int off = LPT; off < 32; off <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, off), l2 = __shfl_xor_sync(0xffffffffu, l, off);
        const float mn = fmaxf(m, m2), ref = mn == -INFINITY ? 0.f : mn;
        const float a = expf(m - ref), a2 = expf(m2 - ref);
        m = mn;
        l = l * a + l2 * a2;
#pragma unroll
        for (int i = 0; i < GPL; i++)
#pragma unroll
            for (int k = 0; k < EPG; k++) o[i][k] = o[i][k] * a + __shfl_xor_sync(0xffffffffu, o[i][k], off) * a2;
    }
    seen = __any_sync(0xffffffffu, seen);
    if (grp == 0)
#pragma unroll
        for (int i = 0; i < GPL; i++)
#pragma unroll
            for (int k = 0; k < EPG; k++) part[warp][(sub + LPT * i) * EPG + k] = o[i][k];
    if (lane == 0) {
        part_m[warp] = m;
        part_l[warp] = l;
        part_seen[warp] = seen;
    }
    __syncthreads();
    float mm = -INFINITY, ll = 0.f, wgt[GEN_WARPS];
    int any = 0;
#pragma unroll
    for (int w = 0; w < GEN_WARPS; w++) mm = fmaxf(mm, part_m[w]);
    const float mref = mm == -INFINITY ? 0.f : mm;
#pragma unroll
    for (int w = 0; w < GEN_WARPS; w++) {
        wgt[w] = expf(part_m[w] - mref);
        ll = fmaf(wgt[w], part_l[w], ll);
        any |= part_seen[w];
    }
    for (int e = threadIdx.x; e < SPAN; e += GEN_WARPS * 32) {
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < GEN_WARPS; w++) acc = fmaf(wgt[w], part[w][e], acc);
        comb[e] = acc;
    }
    if (threadIdx.x == 0) {
        comb[SPAN] = mm;
        comb[SPAN + 1] = ll;
        comb[SPAN + 2] = any ? 1.f : 0.f;
    }
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (cluster > 1) cl.sync();
    else __syncthreads();
    if (rank == 0) {
        float big = p.sink ? 0.f : -INFINITY, sum, w[8], some = 0.f;  // the sink is a score of 0 without a value
        const float* from[8];
#pragma unroll
        for (int r = 0; r < 8; r++)
            if (r < cluster) {
                from[r] = cluster > 1 ? cl.map_shared_rank(comb, r) : comb;
                w[r] = from[r][SPAN];
                big = fmaxf(big, w[r]);
                some += from[r][SPAN + 2];
            }
        const float ref = big == -INFINITY ? 0.f : big;
        sum = p.sink ? expf(-ref) : 0.f;
#pragma unroll
        for (int r = 0; r < 8; r++)
            if (r < cluster) {
                w[r] = expf(w[r] - ref);
                sum = fmaf(w[r], from[r][SPAN + 1], sum);
            }
        // a row with no token yields zeros; one whose scores are all -inf has no softmax
        const float inv = big == -INFINITY ? (some > 0.f ? nanf("") : 0.f) : (sum > 0.f ? 1.f / sum : sum);
        store_row<T>(p, pair, row, [&](int e) {
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < 8; r++)
                if (r < cluster) acc = fmaf(w[r], from[r][e], acc);
            return acc * inv;
        });
    }
    if (cluster > 1) cl.sync();  // the other CTAs' shared memory is read until here
}

// Dependent launches: 4 x 288 tokens, 8 fp32 heads of 64, steps back to back: 7.2 -> 5.8 us.
template <typename T, int LPT, int GPL, int U> cudaError_t launch_split(const GenericParams& p, unsigned pairs, cudaStream_t stream) {
    // as many CTAs per row as still run beside each other and have a block of tokens for each of their warps
    int cluster = 1;
    while (cluster < 8 && (int64_t)pairs * cluster * 2 <= GEN_SPLIT_CTAS && (p.max_tokens == 0 || cluster * GEN_WARPS * (32 / LPT * U) < p.max_tokens)) cluster *= 2;
    return launch_kernel(attn_split_kernel<T, LPT, GPL, U>, dim3(pairs * cluster), GEN_WARPS * 32, 0, cluster, (p.dependent & DEPENDENT_ATTENTION) != 0, stream, p, cluster);
}

template <typename T> cudaError_t launch_generic(const GenericParams& p, unsigned pairs, cudaStream_t stream) {
    // 16-byte granule reads need the pool base aligned (rows and tiles then are, too)
    if (p.geo.epg == 1 || reinterpret_cast<uintptr_t>(p.pool) % 16 != 0)
        return launch_kernel(attn_elem_kernel<T>, dim3(pairs), GEN_WARPS * 32, 0, 1, (p.dependent & DEPENDENT_ATTENTION) != 0, stream, p);
    const int g = p.geo.gpr > p.geo.v_gpr ? p.geo.gpr : p.geo.v_gpr;
    if (g <= 4) return launch_split<T, 4, 1, 4>(p, pairs, stream);
    if (g <= 8) return launch_split<T, 8, 1, 4>(p, pairs, stream);
    if (g <= 16) return launch_split<T, 8, 2, 4>(p, pairs, stream);
    if constexpr (sizeof(T) == 4)
        if (g > 32) return launch_split<T, 8, 8, 1>(p, pairs, stream);
    return launch_split<T, 8, 4, 2>(p, pairs, stream);
}

}  // namespace

cudaError_t launch_attn_seq_generic(const GenericParams& p, int dtype, cudaStream_t stream) {
    const int64_t pairs = (int64_t)p.n_rows * p.geo.n_heads * p.group;
    if (pairs <= 0) return cudaSuccess;
    if (p.geo.d_head > GEN_MAX_D || p.geo.d_value > GEN_MAX_D || pairs > 0x7fffffff) return cudaErrorInvalidValue;
    if (dtype == 2) return cudaErrorInvalidValue;  // bf16 caches have a head shape and run on the tensor-core kernels
    if (dtype == 0) return launch_generic<__half>(p, (unsigned)pairs, stream);
    return launch_generic<float>(p, (unsigned)pairs, stream);
}

}  // namespace ca
