// From the projections of a batch of tokens to attention operands, in one kernel: per-head RMS norm of q and k,
// rotation of q and k (interleaved pairs, a leading part of each head), rotation of v by its position, and the
// store - q to a dense buffer, k and v straight into the token's row of the chunk pool.  A decode step writes row
// s of the batch into the next free row of sequence s's tail chunk; a portion of a prompt names the pool row of
// every token, and tokens whose chunk an earlier sequence already filled are not written.
//
// A token's angles go to shared memory once; then a group of lanes takes a head at a time, in 16-byte granules (heads whose
// size or alignment does not allow that: a warp per head, one rotation pair per lane and step).  All arithmetic in fp32, one
// rounding at the store.  Heads are padded with zeros to whole 16-byte granules in the pool and in q, so that the attention
// kernels read granules for every head size.
#include <algorithm>

#include "ca_kernels.h"
#include "ca_types.cuh"

namespace ca {
namespace {

constexpr int QKV_WARPS = 4;
constexpr int QKV_MAX_D = 256;
constexpr int QKV_STEPS = QKV_MAX_D / 64;  // pairs a lane owns

template <typename T>
__global__ void __launch_bounds__(QKV_WARPS * 32) store_qkv_kernel(const QkvParams p) {
    __shared__ float2 turn_k[QKV_MAX_D / 2], turn_v[QKV_MAX_D / 2];  // (cos, sin) of every pair
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float pos = (float)p.positions[t];
    const int kp = p.key_freq ? p.rot_dims / 2 : 0, vp = p.value_freq ? p.d_value / 2 : 0;
    for (int i = threadIdx.x; i < kp + vp; i += blockDim.x) {
        float sn, cs;
        sincos_for<T>(pos * (i < kp ? p.key_freq[i] : p.value_freq[i - kp]), &sn, &cs);
        (i < kp ? turn_k[i] : turn_v[i - kp]) = make_float2(cs, sn);
    }
    int chunk, slot;
    if (p.tok_slot) {
        const int s = p.tok_slot[t];
        chunk = s < 0 ? -1 : s / p.geo.chunk_size;
        slot = s - chunk * p.geo.chunk_size;
    } else {
        chunk = p.tail_chunk[t];
        slot = p.tail_tokens[t] + p.delta_tokens;
        if (slot >= p.geo.chunk_size) chunk = -1;  // rejected on the host; never write past the tile
    }
    __syncthreads();
    const int G = p.geo.n_heads, H = G * p.group;
    const T* row = reinterpret_cast<const T*>(p.qkv) + (size_t)t * p.row_stride;
    T* pool = reinterpret_cast<T*>(p.pool);
    const Geometry v_side = tile_side(p.geo, 1);
    for (int u = warp; u < H + 2 * G; u += QKV_WARPS) {
        const int kind = u < H ? 0 : (u < H + G ? 1 : 2);  // q, k, v
        const int h = kind == 0 ? u : (kind == 1 ? u - H : u - H - G);
        if (kind > 0 && chunk < 0) continue;
        const int d = kind == 2 ? p.d_value : p.d_key;
        const int padded = kind == 2 ? p.geo.d_value : p.geo.d_head;
        const T* src = row + (kind == 2 ? (H + G) * p.d_key + h * p.d_value : u * p.d_key);
        float a[QKV_STEPS], b[QKV_STEPS];
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < QKV_STEPS; j++) {
            const int e = 2 * (lane + 32 * j);
            a[j] = e < d ? to_f32(src[e]) : 0.f;
            b[j] = e + 1 < d ? to_f32(src[e + 1]) : 0.f;
            ss = fmaf(a[j], a[j], fmaf(b[j], b[j], ss));
        }
        const float* w = kind == 0 ? p.q_norm : (kind == 1 ? p.k_norm : nullptr);
        if (w) {
            const float inv = 1.f / sqrtf(warp_sum(ss) / d + p.eps);
#pragma unroll
            for (int j = 0; j < QKV_STEPS; j++) {
                const int e = 2 * (lane + 32 * j);
                if (e < d) a[j] = a[j] * inv * w[e];
                if (e + 1 < d) b[j] = b[j] * inv * w[e + 1];
            }
        }
        const int pairs = kind == 2 ? vp : kp;
        const float2* turn = kind == 2 ? turn_v : turn_k;
        T* dst;
        Geometry side = p.geo;
        if (kind == 0) {
            dst = reinterpret_cast<T*>(p.q_out) + ((size_t)t * H + h) * padded;
        } else {
            if (kind == 2) side = v_side;
            dst = pool + tile_base_elems(p.geo, chunk, h, kind - 1);
        }
#pragma unroll
        for (int j = 0; j < QKV_STEPS; j++) {
            const int i = lane + 32 * j, e = 2 * i;
            if (e >= padded) break;
            if (i < pairs) {
                const float2 cs = turn[i];
                const float x = a[j], y = b[j];
                a[j] = x * cs.x - y * cs.y;
                b[j] = y * cs.x + x * cs.y;
            }
            // a pair never straddles two granules, and padded rows have an even number of elements
            const int64_t off = kind == 0 ? e : tile_elem_offset(side, slot, e);
            Pack<T, 2> o;
            o.v[0] = from_f32<T>(a[j]);
            o.v[1] = from_f32<T>(b[j]);
            *reinterpret_cast<Pack<T, 2>*>(dst + off) = o;
        }
    }
}

// Heads of whole granules, at most LANES * GP of them: a group of LANES lanes takes a head at a time, lane g its granules g, g + LANES, ...
//
// A prompt is bound by HBM (every element read and written once), but one CTA per token with a granule per lane was bound by its
// instructions (per granule a division, a square root, a reduction, two addresses and the weights) and by one dependent load after the
// other: 8192 tokens of 32 + 8 + 8 heads of 128 took 77.6 us.  So a lane takes GP granules of a head, a CTA walks tokens with the next
// pass's granules requested before the present ones are turned, a thread keeps its frequencies for all tokens, squares and weights go in
// pairs of fp32: the same tokens take 46.3 us (4.3 TB/s where a copy reaches 6.5).  Mean, root and reciprocal are the correctly rounded
// ones for every type: the hardware's approximate ones take 45.1 us, but some 16-bit results then round the other way.  A grid of 6 CTAs
// an SM: up to 888 tokens are one to a CTA.
constexpr int QKV_VEC_THREADS = 128, QKV_VEC_CTAS = 6;

__device__ __forceinline__ void widen(uint32_t v, float& lo, float& hi, __nv_bfloat16) {
    lo = __uint_as_float(v << 16);
    hi = __uint_as_float(v & 0xffff0000u);
}
__device__ __forceinline__ void widen(uint32_t v, float& lo, float& hi, __half) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
    lo = f.x;
    hi = f.y;
}
__device__ __forceinline__ uint32_t narrow(float lo, float hi, __nv_bfloat16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t narrow(float lo, float hi, __half) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <typename T, int LANES, int GP>
__global__ void __launch_bounds__(QKV_VEC_THREADS, QKV_VEC_CTAS) store_qkv_vec_kernel(const QkvParams p) {
    constexpr int EPG = 16 / sizeof(T), PPG = EPG / 2, PER_PASS = QKV_VEC_THREADS / LANES;
    __shared__ __align__(16) float2 turns[2][QKV_MAX_D];  // (cos, sin) of every pair of keys, then of values; of a token and the next
    const int tid = threadIdx.x, g = tid & (LANES - 1), first = tid / LANES;
    const int kp = p.key_freq ? p.rot_dims / 2 : 0, vp = p.value_freq ? p.d_value / 2 : 0, np = kp + vp;
    const int G = p.geo.n_heads, H = G * p.group, units = H + 2 * G;
    const int k_room = (kp + 1) & ~1;  // values' angles start at a 16-byte boundary
    const int k_left = p.d_key - g * EPG, v_left = p.d_value - g * EPG;  // granule j of this lane exists when j * LANES * EPG is below
    // what a later granule of a lane adds to the pool offset of its first one (LANES is a multiple of the 8 granules of a panel's line)
    const int k_step = LANES * (p.geo.swz ? p.geo.chunk_size : 1) * 16, v_step = LANES * (p.geo.v_swz ? p.geo.chunk_size : 1) * 16;
    const uint32_t head_bytes = (uint32_t)(p.geo.tile_elems + p.geo.v_tile_elems) * sizeof(T);
    const int v_from = (H + G) * p.d_key;
    const Geometry v_side = tile_side(p.geo, 1);

    uint4 next[GP];
    auto request = [&](int t, int u) {
        const T* src = reinterpret_cast<const T*>(p.qkv) + (size_t)t * p.row_stride + g * EPG + (u < H + G ? u * p.d_key : v_from + (u - H - G) * p.d_value);
        const int left = u < units ? (u < H + G ? k_left : v_left) : 0;
#pragma unroll
        for (int j = 0; j < GP; j++) {
            next[j] = make_uint4(0u, 0u, 0u, 0u);
            if (j * LANES * EPG < left) next[j] = *reinterpret_cast<const uint4*>(src + j * LANES * EPG);
        }
    };
    auto place_of = [&](int t, int& a, int& b) {  // what names the token's pool row
        a = p.tok_slot ? p.tok_slot[t] : p.tail_chunk[t];
        b = p.tok_slot ? 0 : p.tail_tokens[t];
    };
    int t = blockIdx.x, place_a, place_b, buf = 0;
    if (t >= p.n_tokens) return;
    request(t, first);
    float pos = (float)p.positions[t];
    place_of(t, place_a, place_b);
    float freq[2];  // at most 256 pairs
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int n = tid + i * QKV_VEC_THREADS;
        freq[i] = n < np ? (n < kp ? p.key_freq[n] : p.value_freq[n - kp]) : 0.f;
    }
    for (; t < p.n_tokens; t += gridDim.x, buf ^= 1) {
        const int t2 = t + gridDim.x;
        float2* const turn = turns[buf];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int n = tid + i * QKV_VEC_THREADS;
            if (n < np) {
                float sn, cs;
                sincos_for<T>(pos * freq[i], &sn, &cs);
                turn[n < kp ? n : n - kp + k_room] = make_float2(cs, sn);
            }
        }
        int chunk = place_a, slot = place_b + p.delta_tokens;
        if (p.tok_slot) {
            chunk = place_a < 0 ? -1 : place_a / p.geo.chunk_size;
            slot = place_a - chunk * p.geo.chunk_size;
        } else if (slot >= p.geo.chunk_size) {
            chunk = -1;  // rejected on the host; never write past the tile
        }
        if (t2 < p.n_tokens) {
            pos = (float)p.positions[t2];
            place_of(t2, place_a, place_b);
        }
        uint8_t* const at = static_cast<uint8_t*>(p.pool) + (size_t)max(chunk, 0) * p.geo.chunk_elems * sizeof(T);
        uint8_t* const k_at = at + tile_granule_index(p.geo, slot, g) * 16;
        uint8_t* const v_at = at + (p.geo.tile_elems * sizeof(T) + tile_granule_index(v_side, slot, g) * 16);
        uint8_t* const q_at = static_cast<uint8_t*>(p.q_out) + ((size_t)t * H * p.geo.d_head + g * EPG) * sizeof(T);
        __syncthreads();  // one a token: the other buffer is written only when every warp is past this token's angles
        for (int u0 = 0; u0 < units; u0 += PER_PASS) {
            const int u = u0 + first;
            uint4 in[GP];
#pragma unroll
            for (int j = 0; j < GP; j++) in[j] = next[j];
            if (u0 + PER_PASS < units) request(t, u + PER_PASS);
            else if (t2 < p.n_tokens) request(t2, first);
            if ((tid & ~31) / LANES + u0 >= units) continue;  // a warp without a head
            uint64_t x[GP][PPG];
            uint64_t s2 = 0;  // a pair of zeros
#pragma unroll
            for (int j = 0; j < GP; j++) {
                const uint32_t w32[4] = {in[j].x, in[j].y, in[j].z, in[j].w};
#pragma unroll
                for (int i = 0; i < PPG; i++) {
                    float lo, hi;
                    if constexpr (sizeof(T) == 4) {
                        lo = __uint_as_float(w32[2 * i]);
                        hi = __uint_as_float(w32[2 * i + 1]);
                    } else {
                        widen(w32[i], lo, hi, T());
                    }
                    x[j][i] = pair_f32(lo, hi);
                    s2 = fma_f32x2(x[j][i], x[j][i], s2);
                }
            }
            const float* w = u < H ? p.q_norm : (u < H + G ? p.k_norm : nullptr);
            uint64_t inv2 = 0;
            if (p.q_norm || p.k_norm) {
                float ss, ss_hi;
                unpair_f32(s2, ss, ss_hi);
                ss += ss_hi;
#pragma unroll
                for (int off = LANES >> 1; off >= 1; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
                const float inv = 1.f / sqrtf(ss / (float)p.d_key + p.eps);
                inv2 = pair_f32(inv, inv);
            }
            if (u >= units || (u >= H && chunk < 0)) continue;
            const bool value = u >= H + G;
            const int left = value ? v_left : k_left, pairs = (value ? vp : kp) - g * PPG;
            const float2* turn_of = turn + (value ? k_room : 0) + g * PPG;
            uint8_t* dst = u < H ? q_at + (size_t)((uint32_t)u * (uint32_t)(p.geo.d_head * sizeof(T)))
                                 : (value ? v_at + (uint64_t)(uint32_t)(u - H - G) * head_bytes : k_at + (uint64_t)(uint32_t)(u - H) * head_bytes);
            const int step = u < H ? LANES * 16 : (value ? v_step : k_step);
#pragma unroll
            for (int j = 0; j < GP; j++) {
                if (j * LANES * EPG >= left) break;
                if (w) {
#pragma unroll
                    for (int i = 0; i < PPG; i += 2) {
                        const float4 ww = *reinterpret_cast<const float4*>(w + (g + j * LANES) * EPG + 2 * i);
                        x[j][i] = mul_f32x2(x[j][i], mul_f32x2(inv2, pair_f32(ww.x, ww.y)));
                        x[j][i + 1] = mul_f32x2(x[j][i + 1], mul_f32x2(inv2, pair_f32(ww.z, ww.w)));
                    }
                }
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < PPG; i++) {
                    float a, b;
                    unpair_f32(x[j][i], a, b);
                    if (j * LANES * PPG + i < pairs) {
                        const float2 cs = turn_of[j * LANES * PPG + i];
                        const float c = a;
                        a = a * cs.x - b * cs.y;
                        b = b * cs.x + c * cs.y;
                    }
                    if constexpr (sizeof(T) == 4) {
                        o[2 * i] = __float_as_uint(a);
                        o[2 * i + 1] = __float_as_uint(b);
                    } else {
                        o[i] = narrow(a, b, T());
                    }
                }
                *reinterpret_cast<uint4*>(dst + j * step) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
}

template <typename T, int LANES, int GP>
void run_store_qkv_vec(const QkvParams& p, cudaStream_t stream) {
    store_qkv_vec_kernel<T, LANES, GP><<<std::min(p.n_tokens, QKV_VEC_CTAS * B200_SMS), QKV_VEC_THREADS, 0, stream>>>(p);
}
template <typename T>
void run_store_qkv(const QkvParams& p, cudaStream_t stream) {
    constexpr int EPG = 16 / sizeof(T);
    auto aligned = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
    const int granules = std::max(p.d_key, p.d_value) / EPG;
    if (p.d_key % EPG == 0 && p.d_value % EPG == 0 && p.row_stride % EPG == 0 && aligned(p.qkv) && aligned(p.q_norm) && aligned(p.k_norm) &&
        granules <= 32) {
        if (granules <= 8) run_store_qkv_vec<T, 8, 1>(p, stream);
        else if (granules <= 16) run_store_qkv_vec<T, 8, 2>(p, stream);
        else run_store_qkv_vec<T, 16, 2>(p, stream);
    } else {
        store_qkv_kernel<T><<<p.n_tokens, QKV_WARPS * 32, 0, stream>>>(p);
    }
}

}  // namespace

cudaError_t launch_store_qkv(const QkvParams& p, int dtype, cudaStream_t stream) {
    if (p.n_tokens <= 0) return cudaSuccess;
    if (p.geo.d_head > QKV_MAX_D || p.geo.d_value > QKV_MAX_D || p.geo.epg < 2) return cudaErrorInvalidValue;
    if (dtype == 2) run_store_qkv<__nv_bfloat16>(p, stream);
    else if (dtype == 1) run_store_qkv<float>(p, stream);
    else run_store_qkv<__half>(p, stream);
    return cudaGetLastError();
}

}  // namespace ca
