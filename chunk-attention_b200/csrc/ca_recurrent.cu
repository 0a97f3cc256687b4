// Recurrent sequence mixers over batches of spans (consecutive tokens of several sequences, each with a state slot):
// causal depthwise convolution + SiLU, the selective scan of Mamba, and linear attention with a per-head decay.
// States are fp32, live in [slots][...] arrays of the caller, and are read at a span's start (taken as zero at position
// 0, so a slot needs no clearing before it is used again) and written at its end.
//
// The work of a step is listed as PIECES of at most `work_len` tokens of one span (ca_spans).  A step whose spans are
// all single pieces runs a recurrence in one launch; otherwise the scan takes three: local end state of every piece
// from zero, a sweep over the pieces of each sequence that turns them into initial states, and the outputs.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "../../include/chunk_attn_b200.h"
#include "ca_kernels.h"
#include "ca_types.cuh"

namespace ca {
namespace {

int fail(const char* msg, int code = CA_ERR_INVALID) {
    set_last_error(msg);
    return code;
}
int done() {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CA_OK : fail(cudaGetErrorString(e), CA_ERR_CUDA);
}
constexpr float LOG2E = 1.4426950408889634f;

// ---- convolution ------------------------------------------------------------------------------------------------
// A thread owns V channels and one piece.  KMAX - 1 previous inputs sit in registers, oldest first; a filter with
// fewer taps is right-aligned.  The thread of a span's first piece reads the state and, having read it, puts the
// span's last inputs back.
template <typename T, int V, int KMAX>
__global__ void __launch_bounds__(128) conv_silu_kernel(T* __restrict__ out, const T* __restrict__ x, int64_t x_stride,
                                                        const float* __restrict__ taps, const float* __restrict__ bias,
                                                        float* __restrict__ state, const ca_spans sp, int channels, int K) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (c >= channels) return;
    const int4 wk = reinterpret_cast<const int4*>(sp.work)[blockIdx.y];
    const int e = wk.x, t0 = wk.y, t1 = wk.z, first = sp.cu[e], last = sp.cu[e + 1];
    float tap[KMAX][V], hist[KMAX][V], b[V];
#pragma unroll
    for (int j = 0; j < KMAX; j++)
#pragma unroll
        for (int v = 0; v < V; v++) tap[j][v] = j >= KMAX - K ? taps[(size_t)(c + v) * K + j - (KMAX - K)] : 0.f;
#pragma unroll
    for (int v = 0; v < V; v++) b[v] = bias[c + v];
    float* st = state + (size_t)sp.slot[e] * (K - 1) * channels + c;
    const bool live = sp.start[e] > 0;
    // input at offset i from the span's first token, reaching back into the state
    auto input = [&](int i, float (&o)[V]) {
        if (i >= 0) {
            const Pack<T, V> a = *reinterpret_cast<const Pack<T, V>*>(x + (size_t)(first + i) * x_stride + c);
#pragma unroll
            for (int v = 0; v < V; v++) o[v] = to_f32(a.v[v]);
        } else {
#pragma unroll
            for (int v = 0; v < V; v++) o[v] = live ? st[(size_t)(i + K - 1) * channels + v] : 0.f;
        }
    };
    const int off = t0 - first;
#pragma unroll
    for (int j = 0; j < KMAX - 1; j++) {
        if (j >= KMAX - K) {
            input(off - (KMAX - 1) + j, hist[j]);
        } else {
#pragma unroll
            for (int v = 0; v < V; v++) hist[j][v] = 0.f;
        }
    }
    if (off == 0) {
        const int n = last - first;
        float keep[KMAX][V];
#pragma unroll
        for (int j = 0; j < KMAX - 1; j++)
            if (j >= KMAX - K) input(n - (KMAX - 1) + j, keep[j]);
#pragma unroll
        for (int j = 0; j < KMAX - 1; j++)
            if (j >= KMAX - K)
#pragma unroll
                for (int v = 0; v < V; v++) st[(size_t)(j - (KMAX - K)) * channels + v] = keep[j][v];
    }
    constexpr int GROUP = 4;  // tokens requested together
    for (int tg = t0; tg < t1; tg += GROUP) {
        Pack<T, V> in[GROUP];
#pragma unroll
        for (int k = 0; k < GROUP; k++) in[k] = *reinterpret_cast<const Pack<T, V>*>(x + (size_t)min(tg + k, t1 - 1) * x_stride + c);
#pragma unroll
        for (int k = 0; k < GROUP; k++) {
            if (tg + k < t1) {
                Pack<T, V> o;
#pragma unroll
                for (int v = 0; v < V; v++) {
                    const float xv = to_f32(in[k].v[v]);
                    float acc = fmaf(xv, tap[KMAX - 1][v], b[v]);
#pragma unroll
                    for (int j = 0; j < KMAX - 1; j++) acc = fmaf(hist[j][v], tap[j][v], acc);
#pragma unroll
                    for (int j = 0; j < KMAX - 2; j++) hist[j][v] = hist[j + 1][v];
                    if (KMAX > 1) hist[KMAX > 1 ? KMAX - 2 : 0][v] = xv;
                    o.v[v] = from_f32<T>(silu_for<T>(acc));
                }
                *reinterpret_cast<Pack<T, V>*>(out + (size_t)(tg + k) * channels + c) = o;
            }
        }
    }
}

// ---- selective scan ---------------------------------------------------------------------------------------------
struct ScanParams {
    void* y;                 // [T, C]
    const void* x;           // [T, C]
    const void* z;           // gate, row stride z_stride
    int64_t z_stride;
    const float* dt;         // [T, C] before bias and softplus
    const float* dt_bias;    // [C]
    const float* A;          // [C, N] (negative)
    const float* bc;         // row t: B at bc + t * bc_stride, C behind it
    int64_t bc_stride;
    const float* D;          // [C]
    float* state;            // [slots, C, N]
    float* piece_state;      // [pieces, C, N]
    float* piece_dt;         // [pieces, C]: sum of dt over the piece
    int C, N;
    int run;                 // pieces a CTA takes (0: whole spans)
    bool bc_vec;             // rows of bc can be read 16 bytes at a time
    bool x_vec;              // and those of x, z and dt
    ca_spans sp;
};
constexpr int SCAN_THREADS = 128;
// Tokens that are staged at a time (two buffers): of fp32 rows fewer, for as many CTAs on an SM
template <typename T> constexpr int scan_tokens() { return sizeof(T) == 4 ? 16 : 32; }
// CTAs of an SM with NS states per lane, by registers
constexpr int scan_blocks(int ns) { return ns >= 16 ? 4 : ns >= 8 ? 4 : 6; }


// What a stage holds: B and C, zero past N, and the rows of a CTA's channels
template <typename T, int L, int NS> struct ScanStage {
    static constexpr int TOKENS = scan_tokens<T>();
    static constexpr int CHANNELS = SCAN_THREADS / L;
    static constexpr int DT = TOKENS * 2 * L * NS * 4, X = DT + TOKENS * CHANNELS * 4, GATE = X + TOKENS * CHANNELS * (int)sizeof(T);
    static constexpr int BYTES = GATE + TOKENS * CHANNELS * (int)sizeof(T);
};
// n rows of ROW bytes, of which `valid` exist, 16 bytes at a time by all threads of the CTA
template <int ROW> __device__ __forceinline__ void scan_copy(uint8_t* to, const uint8_t* from, size_t stride, int n, int valid) {
    static_assert(ROW % 16 == 0, "16-byte parts");
    constexpr int PARTS = ROW / 16;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(to);
    for (int i = threadIdx.x; i < n * PARTS; i += SCAN_THREADS) {
        const int row = i / PARTS, b = i % PARTS * 16;
        if (b < valid) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + row * ROW + b), "l"(from + row * stride + b) : "memory");
    }
}

// a state's rate in powers of two, finite where A is not NaN: a step of no length must leave the state as it is
__device__ __forceinline__ float scan_rate(float A) {
    const float a = A * LOG2E;
    return isinf(a) ? copysignf(3.402823466e38f, a) : a;
}

// L lanes share a channel, NS states each, in quads: lane ln has states 4 (ln + L i) .. + 3, so that the lanes' reads of B and C meet
// different banks.  Of a group of tokens, lane i of a channel evaluates the step size and, at the end, the output of tokens i, i + L, ...;
// dt and dt x travel by shuffles, the lanes' parts of the outputs by halving exchanges of the whole group.
// PHASE 0: whole spans, in turn where a CTA has several: state in, outputs, state out.  1: end state of the run from zero, and
// sum of dt.  2: outputs from the run's initial state.
template <typename T, int L, int NS, int PHASE>
__global__ void __launch_bounds__(SCAN_THREADS, scan_blocks(NS)) scan_kernel(const ScanParams p) {
    extern __shared__ __align__(16) uint8_t scan_s[];  // two stages
    using Z = ScanStage<T, L, NS>;
    constexpr int GROUP = L <= 8 ? 8 : L;  // tokens of one exchange
    constexpr int NP = L * NS, OWN = GROUP / L, CB = Z::CHANNELS, TOKENS = Z::TOKENS;
    static_assert(TOKENS % GROUP == 0, "groups of the staged tokens");
    const int c0 = blockIdx.x * CB, ch = threadIdx.x / L, c = c0 + ch;
    const int ln = threadIdx.x & (L - 1), base = (threadIdx.x & 31) & ~(L - 1), N = p.N;
    const bool on = c < p.C;
    const int cc = on ? c : p.C - 1;
    // Copies of B and C: 16 bytes each where rows allow it.  Thread i takes parts i, i + SCAN_THREADS, ... of the rows laid end to end
    const int width = p.bc_vec ? 4 : 1, parts = 2 * N / width;
    const int row0 = threadIdx.x / parts, part0 = threadIdx.x % parts, row_step = SCAN_THREADS / parts, part_step = SCAN_THREADS % parts;
    auto stage = [&](int tb, int t1, int buf) {  // the next tokens, asynchronously; B and C are zero for what a group has behind the last
        uint8_t* to = scan_s + buf * Z::BYTES;
        const int nt = min(TOKENS, t1 - tb), rows = (nt + GROUP - 1) / GROUP * GROUP;
        for (int row = row0, part = part0; row < rows;) {
            const int r = part * width;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(to + (row * 2 * NP + (r < N ? r : r - N + NP)) * 4);
            const float* src = p.bc + (size_t)(tb + min(row, nt - 1)) * p.bc_stride + r;
            if (p.bc_vec)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(row < nt ? 16 : 0) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(row < nt ? 4 : 0) : "memory");
            row += row_step;
            part += part_step;
            if (part >= parts) {
                part -= parts;
                row++;
            }
        }
        if (p.x_vec) {
            scan_copy<4 * CB>(to + Z::DT, reinterpret_cast<const uint8_t*>(p.dt + (size_t)tb * p.C + c0), (size_t)p.C * 4, nt, (p.C - c0) * 4);
            constexpr int ROW = CB * (int)sizeof(T);
            const int valid = (p.C - c0) * (int)sizeof(T);
            scan_copy<ROW>(to + Z::X, reinterpret_cast<const uint8_t*>(static_cast<const T*>(p.x) + (size_t)tb * p.C + c0), (size_t)p.C * sizeof(T), nt, valid);
            if (PHASE != 1)
                scan_copy<ROW>(to + Z::GATE, reinterpret_cast<const uint8_t*>(static_cast<const T*>(p.z) + (size_t)tb * p.z_stride + c0), (size_t)p.z_stride * sizeof(T), nt, valid);
        } else {
            for (int i = threadIdx.x; i < nt * CB; i += SCAN_THREADS) {
                const int t = tb + i / CB, k = c0 + i % CB;
                if (k >= p.C) continue;
                reinterpret_cast<float*>(to + Z::DT)[i] = p.dt[(size_t)t * p.C + k];
                reinterpret_cast<T*>(to + Z::X)[i] = static_cast<const T*>(p.x)[(size_t)t * p.C + k];
                if (PHASE != 1) reinterpret_cast<T*>(to + Z::GATE)[i] = static_cast<const T*>(p.z)[(size_t)t * p.z_stride + k];
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int unit = blockIdx.y;
    if (PHASE == 0 && gridDim.y == p.sp.n_entries && p.sp.n_entries <= SCAN_THREADS) {  // the longest spans first
        __shared__ int ranked;
        const int E = p.sp.n_entries, e = threadIdx.x;
        if (e < E) {
            const int len = p.sp.cu[e + 1] - p.sp.cu[e];
            int rank = 0;
            for (int k = 0; k < E; k++) {
                const int other = p.sp.cu[k + 1] - p.sp.cu[k];
                rank += other > len || (other == len && k < e);
            }
            if (rank == unit) ranked = e;
        }
        __syncthreads();
        unit = ranked;
    }
    int e = unit, t0, t1;
    if (PHASE == 0) {
        t0 = p.sp.cu[e];
        t1 = p.sp.cu[e + 1];
    } else {
        const int4 wk = reinterpret_cast<const int4*>(p.sp.work)[unit];
        if (wk.w % p.run) return;  // a run starts at every run-th piece
        e = wk.x;
        t0 = wk.y;
        t1 = min(p.sp.cu[e + 1], t0 + p.run * p.sp.work_len);
    }
    int buf = 0;
    stage(t0, t1, 0);
    uint64_t A2[NS / 2];  // pairs of states
    auto rate = [&](int n) { return n < N ? scan_rate(p.A[(size_t)cc * N + n]) : 0.f; };
#pragma unroll
    for (int i = 0; i < NS; i += 2) {
        const int n = 4 * (ln + L * (i / 4)) + i % 4;
        A2[i / 2] = pair_f32(rate(n), rate(n + 1));
    }
    const float bias = p.dt_bias[cc], D = PHASE == 1 ? 0.f : p.D[cc];
    T* Y = static_cast<T*>(p.y) + cc;
    if (N < NP)  // the padding past N is never copied into
        for (int i = threadIdx.x; i < TOKENS * 2 * NP; i += SCAN_THREADS)
            if (i % NP >= N) reinterpret_cast<float*>(scan_s)[i] = reinterpret_cast<float*>(scan_s + Z::BYTES)[i] = 0.f;
    const bool vec = N % 4 == 0;
    float sum_dt = 0.f;
    for (bool first = true;;) {
        const int after = unit + gridDim.y;  // this CTA's next span
        const bool more = PHASE == 0 && after < p.sp.n_entries;
        const int a0 = more ? p.sp.cu[after] : 0, a1 = more ? p.sp.cu[after + 1] : 0;
        float S[NS];
        float* slot = p.state + ((size_t)p.sp.slot[e] * p.C + cc) * N;
        float* piece = PHASE == 0 ? nullptr : p.piece_state + ((size_t)unit * p.C + cc) * N;
        const float* from = PHASE == 0 ? slot : piece;
#pragma unroll
        for (int i = 0; i < NS; i++) S[i] = 0.f;
        if (PHASE == 2 || (PHASE == 0 && p.sp.start[e] > 0)) {
#pragma unroll
            for (int i = 0; i < NS; i += 4) {
                const int n = 4 * (ln + L * (i / 4));
                if (vec) {
                    if (n < N) {
                        const float4 v = *reinterpret_cast<const float4*>(from + n);
                        S[i] = v.x; S[i + 1] = v.y; S[i + 2] = v.z; S[i + 3] = v.w;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (n + j < N) S[i + j] = from[n + j];
                }
            }
        }
        uint64_t S2[NS / 2];
#pragma unroll
        for (int i = 0; i < NS; i += 2) S2[i / 2] = pair_f32(S[i], S[i + 1]);
        if (t0 == t1 && more) stage(a0, a1, buf);  // a span without tokens: nothing below requests the next one's
        for (int tb = t0; tb < t1; tb += TOKENS, buf ^= 1, first = false) {
            const int nt = min(TOKENS, t1 - tb);
            if (!first) __syncthreads();  // the other buffer is free
            const bool same = tb + TOKENS < t1;
            if (same || more) {
                stage(same ? tb + TOKENS : a0, same ? t1 : a1, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            const uint8_t* now = scan_s + buf * Z::BYTES;
            for (int g = 0; g < nt; g += GROUP) {
                float xs[OWN], ds[OWN], us[OWN], ys[GROUP];
                const int t = tb + g + ln, at = (g + ln) * CB + ch;  // this lane's tokens: t + k * L
                T* const y_row = Y + (size_t)(tb + g) * p.C;
                auto inputs = [&](int k) {
                    const bool valid = t + k * L < t1;
                    xs[k] = valid ? to_f32(reinterpret_cast<const T*>(now + Z::X)[at + k * L * CB]) : 0.f;
                    const float raw = reinterpret_cast<const float*>(now + Z::DT)[at + k * L * CB] + bias;
                    ds[k] = softplus_f(valid ? raw : -1e30f);  // a step of no length, exactly 0, leaves the state as it is
                    us[k] = ds[k] * xs[k];
                    if (PHASE == 1) sum_dt += ds[k];
                };
                constexpr int HALF = (OWN + 1) / 2;  // the tokens of a lane in the first half of a group
                const bool both = OWN == 1 || nt - g > HALF * L;
#pragma unroll
                for (int k = 0; k < HALF; k++) inputs(k);
                if (both) {
#pragma unroll
                    for (int k = HALF; k < OWN; k++) inputs(k);
                } else {
#pragma unroll
                    for (int k = HALF; k < OWN; k++) xs[k] = ds[k] = us[k] = 0.f;
                }
                const float* rows = reinterpret_cast<const float*>(now) + g * 2 * NP + 4 * ln;
                auto token = [&](int k) {
                    float dt = ds[k / L], u = us[k / L];
                    if (L > 1) {
                        dt = __shfl_sync(0xffffffffu, dt, base + k % L);
                        u = __shfl_sync(0xffffffffu, u, base + k % L);
                    }
                    const uint64_t dt2 = pair_f32(dt, dt), u2 = pair_f32(u, u);
                    uint64_t y2;
#pragma unroll
                    for (int i = 0; i < NS; i += 4) {
                        const float* B = rows + k * 2 * NP + L * i;
                        const ulonglong2 b4 = *reinterpret_cast<const ulonglong2*>(B), c4 = *reinterpret_cast<const ulonglong2*>(B + NP);
                        const uint64_t bb[2] = {b4.x, b4.y}, cc2[2] = {c4.x, c4.y};
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            uint64_t& s2 = S2[i / 2 + j];
                            float lo, hi;
                            unpair_f32(mul_f32x2(dt2, A2[i / 2 + j]), lo, hi);
                            s2 = fma_f32x2(pair_f32(exp2_approx(lo), exp2_approx(hi)), s2, mul_f32x2(u2, bb[j]));
                            if (PHASE != 1) y2 = i + j == 0 ? mul_f32x2(s2, cc2[j]) : fma_f32x2(s2, cc2[j], y2);
                        }
                    }
                    if (PHASE != 1) {
                        float y, y_hi;
                        unpair_f32(y2, y, y_hi);
                        ys[k] = y + y_hi;
                    }
                };
                // four at a time: short spans end there, and four are enough to cover one another's latencies
#pragma unroll
                for (int q = 0; q < GROUP; q += 4) {
                    if (q == 0 || nt - g > q) {
#pragma unroll
                        for (int k = q; k < q + 4; k++) token(k);
                    } else if (PHASE != 1) {
#pragma unroll
                        for (int k = q; k < q + 4; k++) ys[k] = 0.f;
                    }
                }
                if (PHASE != 1) {
                    // the lanes' parts: a lane gives up half of the tokens it still has, for the other half of its partner's
#pragma unroll
                    for (int off = L / 2; off >= 1; off >>= 1) {
                        const bool upper = ln & off;
#pragma unroll
                        for (int k = 0; k < GROUP; k++)
                            if (k % L < off) {
                                const float got = __shfl_xor_sync(0xffffffffu, upper ? ys[k] : ys[k + off], off);
                                ys[k] = (upper ? ys[k + off] : ys[k]) + got;
                            }
                    }
                    // the gates of all tokens at once: behind a branch each, they waited for one another
                    auto outputs = [&](auto first_k, auto end_k) {
                        constexpr int from = decltype(first_k)::value, to = decltype(end_k)::value;
                        float o[to - from + 1];
#pragma unroll
                        for (int k = from; k < to; k++)
                            o[k - from] = fmaf(D, xs[k], ys[k * L]) * silu_for<T>(to_f32(reinterpret_cast<const T*>(now + Z::GATE)[at + k * L * CB]));
#pragma unroll
                        for (int k = from; k < to; k++)
                            if (on && t + k * L < t1) y_row[(ln + k * L) * p.C] = from_f32<T>(o[k - from]);
                    };
                    outputs(std::integral_constant<int, 0>(), std::integral_constant<int, HALF>());
                    if (both) outputs(std::integral_constant<int, HALF>(), std::integral_constant<int, OWN>());
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NS; i += 2) unpair_f32(S2[i / 2], S[i], S[i + 1]);
        if (PHASE == 1) {
#pragma unroll
            for (int off = L / 2; off >= 1; off >>= 1) sum_dt += __shfl_xor_sync(0xffffffffu, sum_dt, off);
        }
        if (PHASE != 2 && on) {
            float* dst = PHASE == 0 ? slot : piece;
#pragma unroll
            for (int i = 0; i < NS; i += 4) {
                const int n = 4 * (ln + L * (i / 4));
                if (vec) {
                    if (n < N) *reinterpret_cast<float4*>(dst + n) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (n + j < N) dst[n + j] = S[i + j];
                }
            }
            if (PHASE == 1 && ln == 0) p.piece_dt[(size_t)unit * p.C + c] = sum_dt;
        }
        if (!more) break;
        unit = e = after;
        t0 = a0;
        t1 = a1;
    }
}

// Short spans: eight states a lane, inputs straight to registers, so that eight CTAs share an SM and one's beginning and end hide under the
// others' tokens.  Of a group of eight tokens, lane i of a channel reads the inputs of tokens i, i + L, ... and evaluates their step size
// and, at the end, their output; dt and dt x travel by shuffles, B and C through shared memory.
constexpr int SHORT_TOKENS = 32;  // whose B and C are staged at a time (two buffers)
template <typename T, int L>
__global__ void __launch_bounds__(SCAN_THREADS, L == 1 ? 6 : 8) scan_short_kernel(const ScanParams p) {
    constexpr int NS = 8, GROUP = 8, NP = L * NS, OWN = GROUP / L, BUF = SHORT_TOKENS * 2 * NP;
    __shared__ __align__(16) float bc_s[2 * BUF];  // 2 x [SHORT_TOKENS][B: L * NS | C: L * NS], zero past N
    const int c = blockIdx.x * (SCAN_THREADS / L) + threadIdx.x / L;
    const int ln = threadIdx.x & (L - 1), base = (threadIdx.x & 31) & ~(L - 1), n0 = ln * NS, N = p.N;
    const bool on = c < p.C, vec = N % 4 == 0;
    const int cc = on ? c : p.C - 1;
    uint64_t A2[NS / 2];  // pairs of states
#pragma unroll
    for (int i = 0; i < NS; i += 2) {
        const float* a = p.A + (size_t)cc * N + n0 + i;
        A2[i / 2] = pair_f32(n0 + i < N ? scan_rate(a[0]) : 0.f, n0 + i + 1 < N ? scan_rate(a[1]) : 0.f);
    }
    const float bias = p.dt_bias[cc], D = p.D[cc];
    const T* X = static_cast<const T*>(p.x) + cc;
    const T* Z = static_cast<const T*>(p.z) + cc;
    T* Y = static_cast<T*>(p.y) + cc;
    const float* DT = p.dt + cc;
    if (N < NP)  // the padding past N is never copied into
        for (int i = threadIdx.x; i < 2 * BUF; i += SCAN_THREADS)
            if (i % NP >= N) bc_s[i] = 0.f;
    const int e = blockIdx.y, t0 = p.sp.cu[e], t1 = p.sp.cu[e + 1];
    float S[NS];
    float* slot = p.state + ((size_t)p.sp.slot[e] * p.C + cc) * N + n0;
#pragma unroll
    for (int i = 0; i < NS; i++) S[i] = 0.f;
    if (p.sp.start[e] > 0) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < NS; i += 4)
                if (n0 + i < N) {
                    const float4 v = *reinterpret_cast<const float4*>(slot + i);
                    S[i] = v.x; S[i + 1] = v.y; S[i + 2] = v.z; S[i + 3] = v.w;
                }
        } else {
#pragma unroll
            for (int i = 0; i < NS; i++)
                if (n0 + i < N) S[i] = slot[i];
        }
    }
    uint64_t S2[NS / 2];
#pragma unroll
    for (int i = 0; i < NS; i += 2) S2[i / 2] = pair_f32(S[i], S[i + 1]);
    auto stage = [&](int tb, int buf) {  // B and C of the next tokens, asynchronously
        const int nt = min(SHORT_TOKENS, t1 - tb);
        for (int i = threadIdx.x; i < nt * 2 * N; i += SCAN_THREADS) {
            const int tt = i / (2 * N), r = i - tt * 2 * N;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(bc_s + buf * BUF + tt * 2 * NP + (r < N ? r : r - N + NP));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(p.bc + (size_t)(tb + tt) * p.bc_stride + r) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float nd[OWN];
    T nx[OWN], nz[OWN];  // as they come: a conversion here would wait for the loads
    auto request = [&](int t) {  // this lane's tokens of the group that starts at t
#pragma unroll
        for (int k = 0; k < OWN; k++) {
            const int tk = ln + k * L;
            nd[k] = 0.f;
            nx[k] = nz[k] = from_f32<T>(0.f);
            if (t + tk < t1) {
                nx[k] = X[(size_t)(t + tk) * p.C];
                nd[k] = DT[(size_t)(t + tk) * p.C];
                nz[k] = Z[(size_t)(t + tk) * p.z_stride];
            }
        }
    };
    stage(t0, 0);
    request(t0);
    int buf = 0;
    for (int tb = t0; tb < t1; tb += SHORT_TOKENS, buf ^= 1) {
        const int nt = min(SHORT_TOKENS, t1 - tb);
        if (tb > t0) __syncthreads();  // the other buffer is free
        if (tb + SHORT_TOKENS < t1) {
            stage(tb + SHORT_TOKENS, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        for (int g = 0; g < nt; g += GROUP) {
            float xs[OWN], ds[OWN], us[OWN], ys[OWN], zs[OWN];
#pragma unroll
            for (int k = 0; k < OWN; k++) {
                xs[k] = to_f32(nx[k]);
                zs[k] = to_f32(nz[k]);
                ds[k] = softplus_f(nd[k] + bias);
                us[k] = ds[k] * xs[k];
                ys[k] = 0.f;
            }
            if (tb + g + GROUP < t1) request(tb + g + GROUP);
            auto token = [&](int k) {
                float dt = ds[k / L], u = us[k / L];
                if (L > 1) {
                    dt = __shfl_sync(0xffffffffu, dt, base + k % L);
                    u = __shfl_sync(0xffffffffu, u, base + k % L);
                }
                const float* B = bc_s + buf * BUF + (g + k) * 2 * NP + n0;
                const uint64_t dt2 = pair_f32(dt, dt), u2 = pair_f32(u, u);
                uint64_t y2 = 0;
#pragma unroll
                for (int i = 0; i < NS; i += 4) {
                    const ulonglong2 b4 = *reinterpret_cast<const ulonglong2*>(B + i), c4 = *reinterpret_cast<const ulonglong2*>(B + NP + i);
                    const uint64_t bb[2] = {b4.x, b4.y}, cc2[2] = {c4.x, c4.y};
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        uint64_t& s2 = S2[i / 2 + j];
                        float lo, hi;
                        unpair_f32(mul_f32x2(dt2, A2[i / 2 + j]), lo, hi);
                        s2 = fma_f32x2(pair_f32(exp2_approx(lo), exp2_approx(hi)), s2, mul_f32x2(u2, bb[j]));
                        y2 = fma_f32x2(s2, cc2[j], y2);
                    }
                }
                float y, y_hi;
                unpair_f32(y2, y, y_hi);
                y += y_hi;
#pragma unroll
                for (int off = L >> 1; off >= 1; off >>= 1) y += __shfl_xor_sync(0xffffffffu, y, off);
                if (k % L == ln) ys[k / L] = y;
            };
            if (nt - g >= GROUP) {
#pragma unroll
                for (int k = 0; k < GROUP; k++) token(k);
            } else {
#pragma unroll
                for (int k = 0; k < GROUP; k++)
                    if (g + k < nt) token(k);
            }
#pragma unroll
            for (int k = 0; k < OWN; k++) {
                const int tk = ln + k * L;
                if (on && g + tk < nt) Y[(size_t)(tb + g + tk) * p.C] = from_f32<T>(fmaf(D, xs[k], ys[k]) * silu_for<T>(zs[k]));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NS; i += 2) unpair_f32(S2[i / 2], S[i], S[i + 1]);
    if (!on) return;
    if (vec) {
#pragma unroll
        for (int i = 0; i < NS; i += 4)
            if (n0 + i < N) *reinterpret_cast<float4*>(slot + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < NS; i++)
            if (n0 + i < N) slot[i] = S[i];
    }
}

// One token per span: four states per lane straight from and to memory, a few spans in turn per CTA so that A is read
// once for them, everything of the next span requested before this one is worked on.
template <typename T, int L, bool VEC>
__global__ void __launch_bounds__(SCAN_THREADS) scan_step_kernel(const ScanParams p) {
    const int c = blockIdx.x * (SCAN_THREADS / L) + threadIdx.x / L;
    const int ln = threadIdx.x & (L - 1), N = p.N;
    const bool on = c < p.C;
    const int cc = on ? c : p.C - 1;
    constexpr int NS = 4;
    const int n0 = ln * NS;
    float A2[NS];
#pragma unroll
    for (int i = 0; i < NS; i++) A2[i] = n0 + i < N ? p.A[(size_t)cc * N + n0 + i] * LOG2E : 0.f;
    const float bias = p.dt_bias[cc], D = p.D[cc];
    struct Inputs {  // of one span, as they come
        float S[NS], B[NS], C[NS], dt;
        T x, z;
    } in;
    auto request = [&](int e) {
#pragma unroll
        for (int i = 0; i < NS; i++) in.S[i] = in.B[i] = in.C[i] = 0.f;
        if (e >= p.sp.n_entries) return;
        const size_t t = p.sp.cu[e];
        in.x = static_cast<const T*>(p.x)[t * p.C + cc];
        in.z = static_cast<const T*>(p.z)[t * p.z_stride + cc];
        in.dt = p.dt[t * p.C + cc];
        const float* B = p.bc + t * p.bc_stride + n0;
#pragma unroll
        for (int i = 0; i < NS; i++)
            if (n0 + i < N) {
                in.B[i] = __ldg(B + i);
                in.C[i] = __ldg(B + N + i);
            }
        if (p.sp.start[e] == 0) return;
        const float* s = p.state + ((size_t)p.sp.slot[e] * p.C + cc) * N + n0;
        if (VEC) {
            if (n0 < N) {
                const float4 v = *reinterpret_cast<const float4*>(s);
                in.S[0] = v.x; in.S[1] = v.y; in.S[2] = v.z; in.S[3] = v.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < NS; i++)
                if (n0 + i < N) in.S[i] = s[i];
        }
    };
    request(blockIdx.y);
    for (int e = blockIdx.y; e < p.sp.n_entries; e += gridDim.y) {
        Inputs now = in;
        request(e + gridDim.y);
        const float x = to_f32(now.x), dt = softplus_f(now.dt + bias), u = dt * x;
        float y = 0.f;
#pragma unroll
        for (int i = 0; i < NS; i++) {
            now.S[i] = fmaf(exp2_approx(dt * A2[i]), now.S[i], u * now.B[i]);
            y = fmaf(now.S[i], now.C[i], y);
        }
#pragma unroll
        for (int off = L >> 1; off >= 1; off >>= 1) y += __shfl_xor_sync(0xffffffffu, y, off);
        float* s = p.state + ((size_t)p.sp.slot[e] * p.C + cc) * N + n0;
        if (on) {
            if (VEC) {
                if (n0 < N) *reinterpret_cast<float4*>(s) = make_float4(now.S[0], now.S[1], now.S[2], now.S[3]);
            } else {
#pragma unroll
                for (int i = 0; i < NS; i++)
                    if (n0 + i < N) s[i] = now.S[i];
            }
            if (ln == 0) static_cast<T*>(p.y)[(size_t)p.sp.cu[e] * p.C + c] = from_f32<T>(fmaf(D, x, y) * silu_for<T>(to_f32(now.z)));
        }
    }
}

// per (span, channel, state): end states of the runs -> initial states, and the span's end state to its slot
__global__ void scan_sweep_kernel(const ScanParams p) {
    const int e = blockIdx.y;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, CN = (int64_t)p.C * p.N;
    if (i >= CN) return;
    const int c = (int)(i / p.N);
    const float A2 = p.A[i] * LOG2E;
    float* slot = p.state + (size_t)p.sp.slot[e] * CN + i;
    float S = p.sp.start[e] > 0 ? *slot : 0.f;
    for (int w = p.sp.work_off[e]; w < p.sp.work_off[e + 1]; w += p.run) {
        float* piece = p.piece_state + (size_t)w * CN + i;
        const float local = *piece;
        *piece = S;
        S = fmaf(exp2_approx(A2 * p.piece_dt[(size_t)w * p.C + c]), S, local);
    }
    *slot = S;
}

// Lanes per channel with per_lane states each
int scan_lanes(int n_states, int per_lane) {
    int lanes = 1;
    while (lanes < 32 && lanes * per_lane < n_states) lanes *= 2;
    return lanes;
}
// instances of the scan: the others are slower at every size, or their lanes have no states
constexpr bool scan_instance(int lanes, int per_lane) { return per_lane == 4 ? lanes <= 4 : per_lane == 8 ? lanes <= 16 : lanes >= 4 && lanes <= 16; }
struct ScanShape {
    int per_lane;  // states
    int run;       // pieces of a CTA, 0: whole spans
};
// States per lane and, where whole spans leave the GPU idle, the length of runs, by estimates of the time: a token costs a warp alone
// `alone` ns, and each warp of an SM's quarter `busy` ns where many share it (8 tokens a group, bf16).  Runs are two passes and a sweep.
// 8192 channels of 16 states, 4 | 8 | 16 states a lane: 64 spans of 128 tokens 478 | 398 | 387 us, 8 of 596 to 1000 361 | 306 | 355,
// one of 4096 356 | 363 | 617 (in runs 440), one of 2048 channels 280 | 363 | 613 (in runs 134).  4096 channels, 8 spans: 64 states
// 694 | 567 | 526, 128 states - | 1192 | 978.
ScanShape scan_shape(const ca_spans& sp, int channels, int n_states) {
    constexpr double SWEEP_NS = 8000.0;
    const int pieces = (sp.max_tokens + sp.work_len - 1) / sp.work_len;
    ScanShape best{n_states > 128 ? 16 : 8, 0};
    double best_t = 0;
    for (int ns = 4; ns <= 16; ns *= 2) {
        const int L = scan_lanes(n_states, ns);
        if (!scan_instance(L, ns) || L * ns < n_states || (ns > 4 && L == 1 && n_states <= ns / 2)) continue;
        const double alone = ns == 4 ? (L == 1 ? 116 : L == 2 ? 85 : 70) : ns == 8 ? (L == 1 ? 130 : 88) : 150;
        const double busy = ns == 4 ? (L == 1 ? 46 : L == 2 ? 38 : 34) : ns == 8 ? (L == 1 ? 62 : 56) : 104;
        const int64_t blocks = ((int64_t)channels * L + SCAN_THREADS - 1) / SCAN_THREADS;
        // CTAs of equal lengths on every SM; a few more on some of them are a longer time
        auto pass = [&](double tokens_each, double ctas, double longest) {
            const double per_sm = ctas / B200_SMS, uneven = per_sm > scan_blocks(ns) ? per_sm + 0.3 : std::ceil(per_sm);
            const double chain = longest * alone, work = tokens_each * uneven * busy;
            return std::max(chain, work) + 0.26 * std::min(chain, work);
        };
        for (int run = 0; run < pieces; run = run == 0 ? 1 : run + std::max(1, run / 4)) {
            double t;
            if (run == 0) {
                t = pass((double)sp.n_tokens / sp.n_entries, (double)blocks * sp.n_entries, sp.max_tokens);
            } else {
                const double runs = (double)sp.n_work / run + 0.5 * sp.n_entries * (run - 1) / run;
                t = SWEEP_NS + 2.0 * pass((double)sp.n_tokens / runs, blocks * runs, (double)run * sp.work_len);
            }
            if (best_t == 0 || t < best_t) {
                best_t = t;
                best = ScanShape{ns, run};
            }
        }
    }
    return best;
}

// Whether whole spans go to the kernel of short ones.  Staged inputs, and lanes with fewer or more states, cost a CTA its beginning and the SM
// the CTAs that would hide it.  Spans of equal length, this kernel | the other one, us: 8192 channels of 16 states, fp32, 200 spans of 3 tokens
// 103 | 124, 64 of 33 144 | 164, of 64 248 | 272, of 96 365 | 388, 16 of 128 134 | 133, 8 of 33 25 | 25, of 64 40 | 39; bf16, 200 of 3 99 | 121, 64 of
// 33 134 | 144, of 64 228 | 233, of 96 334 | 331; 2048 channels, fp32, 16 of 3 6 | 6, of 40 19 | 17, 64 of 33 42 | 44; bf16, 64 of 40 44 | 42.
// 8192 channels of 8 states, bf16, 64 of 5 28 | 32, of 12 49 | 39; fp32, of 5 29 | 32, of 8 39 | 34; 24 states, fp32, 64 of 5 72 | 90, of 17 148 | 174, of
// 64 444 | 472, bf16, of 17 150 | 156, of 20 165 | 155; 32 states, 64 of 5 79 | 93, of 8 95 | 95.  4096 of 64 states: 64 of 33 249 | 155, 200 of 3 283 | 156.
bool scan_short(const ca_spans& sp, int channels, int n_states, bool bits16) {
    if (n_states <= 4 || n_states > 32 || sp.max_tokens > 128 || sp.n_entries > 65535) return false;  // a span is a row of the grid
    const int per_block = SCAN_THREADS / scan_lanes(n_states, 8);
    const double ctas = (double)((channels + per_block - 1) / per_block) * sp.n_entries, mean = (double)sp.n_tokens / sp.n_entries;
    if (n_states <= 8) return bits16 && mean <= 6;
    if (n_states > 24) return mean <= 6;
    if (mean <= 9) return true;
    if (n_states > 16) return ctas >= 1024 && mean <= (bits16 ? 18 : 64);
    return bits16 ? ctas >= 4096 && mean <= 56 : (ctas >= 1024 && mean <= 36) || (ctas >= 2048 && mean <= 100);
}

// CTAs of the kernel with staged inputs that share the spans.  One each, or, of short spans, several: a CTA's beginning costs as much as about 7
// tokens (200 spans of 3 tokens, 8192 channels of 16 states: 133 us with one each, 90 so; 64 of 20: 107 and 81), and the next span's rows arrive
// under the present one.
int scan_rows(const ca_spans& sp, int blocks, int resident) {
    constexpr int SHORT = 40, BEGIN = 7;
    const int E = sp.n_entries;
    if (sp.max_tokens > SHORT) return E;
    auto time = [&](int rows) {  // a few CTAs behind the last full wave take most of another one
        const double waves = (double)blocks * rows / resident, full = std::floor(waves), each = (E + rows - 1) / rows;
        return (waves <= 1.0 ? 1.0 : full + (waves > full ? std::max(waves - full, 0.7) : 0.0)) * (each * sp.n_tokens / E + BEGIN);
    };
    int best = E;
    for (int rows = std::min(E, 4 * resident / blocks + 1); rows >= 1; rows--)
        if (time(rows) < time(best)) best = rows;
    return best;
}

template <typename T, int L, int NS>
void launch_scan(const ScanParams& p, cudaStream_t stream) {
    constexpr int per_block = SCAN_THREADS / L;
    const int blocks = (p.C + per_block - 1) / per_block;
    constexpr int smem = 2 * ScanStage<T, L, NS>::BYTES;
    static_assert(smem <= 227 * 1024 - 1024, "two stages");
    if (smem > 40 * 1024) {
        cudaFuncSetAttribute(scan_kernel<T, L, NS, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(scan_kernel<T, L, NS, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(scan_kernel<T, L, NS, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    }
    if (p.run == 0) {
        const int rows = scan_rows(p.sp, blocks, B200_SMS * std::min(scan_blocks(NS), 227 * 1024 / (smem + 1024)));
        scan_kernel<T, L, NS, 0><<<dim3(blocks, rows), SCAN_THREADS, smem, stream>>>(p);
    } else {
        scan_kernel<T, L, NS, 1><<<dim3(blocks, p.sp.n_work), SCAN_THREADS, smem, stream>>>(p);
        scan_sweep_kernel<<<dim3((unsigned)(((int64_t)p.C * p.N + 255) / 256), p.sp.n_entries), 256, 0, stream>>>(p);
        scan_kernel<T, L, NS, 2><<<dim3(blocks, p.sp.n_work), SCAN_THREADS, smem, stream>>>(p);
    }
}
template <typename T, int L>
void launch_scan_step(const ScanParams& p, cudaStream_t stream) {
    constexpr int per_block = SCAN_THREADS / L;
    const int blocks = (p.C + per_block - 1) / per_block;
    const dim3 grid(blocks, std::min(p.sp.n_entries, std::max(1, B200_SMS * 64 / blocks)));
    if (p.N % 4 == 0) scan_step_kernel<T, L, true><<<grid, SCAN_THREADS, 0, stream>>>(p);
    else scan_step_kernel<T, L, false><<<grid, SCAN_THREADS, 0, stream>>>(p);
}
// f(integral_constant L)
template <typename F> void by_lanes(int lanes, F&& f) {
    switch (lanes) {
        case 1: f(std::integral_constant<int, 1>()); break;
        case 2: f(std::integral_constant<int, 2>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        case 16: f(std::integral_constant<int, 16>()); break;
        default: f(std::integral_constant<int, 32>());
    }
}

// ---- linear attention with decay --------------------------------------------------------------------------------
struct DecayParams {
    void* out;               // [T, H * dv]
    const void* qkv;         // row t: q heads | k heads | v heads, before SiLU
    int64_t row_stride;
    const float* decay;      // [H]
    float* state;            // [slots, H, dk, dv]
    float* scratch;          // [pieces, H, dk, dv] or null
    int H, dk, dv;
    ca_spans sp;
};

// One token per span: CTA per (span, head).  Threads span the columns of the state (VEC wide) and split its rows.
constexpr int DECAY_STEP_THREADS = 256;
template <typename T, int V>
__global__ void __launch_bounds__(DECAY_STEP_THREADS) decay_step_kernel(const DecayParams p) {
    extern __shared__ float sm[];
    float* q = sm;                       // [dk]
    float* k = q + p.dk;                 // [dk]
    float* red = k + p.dk;               // [row groups][dv]
    const int e = blockIdx.y, h = blockIdx.x, t = p.sp.cu[e];
    const T* row = static_cast<const T*>(p.qkv) + (size_t)t * p.row_stride;
    const int Hk = p.H * p.dk;
    for (int i = threadIdx.x; i < p.dk; i += blockDim.x) {
        q[i] = silu_f(to_f32(row[h * p.dk + i]));
        k[i] = silu_f(to_f32(row[Hk + h * p.dk + i]));
    }
    __syncthreads();
    const int cols = p.dv / V, groups = max(1, DECAY_STEP_THREADS / cols);
    const float d = p.decay[h];
    const bool live = p.sp.start[e] > 0;
    float* S = p.state + ((size_t)p.sp.slot[e] * p.H + h) * p.dk * p.dv;
    // a group of `cols` threads takes every groups-th row; wider values than threads loop over the columns
    for (int base = 0; base < cols; base += DECAY_STEP_THREADS) {
        const int cg = cols <= DECAY_STEP_THREADS ? threadIdx.x % cols : base + threadIdx.x;
        const int rg = cols <= DECAY_STEP_THREADS ? threadIdx.x / cols : 0;
        if (rg < groups && cg < cols) {
            float v[V], acc[V];
#pragma unroll
            for (int i = 0; i < V; i++) {
                v[i] = silu_f(to_f32(row[2 * Hk + h * p.dv + cg * V + i]));
                acc[i] = 0.f;
            }
            constexpr int AHEAD = 8;  // rows requested together
            for (int r0 = rg; r0 < p.dk; r0 += AHEAD * groups) {
                Pack<float, V> s[AHEAD];
#pragma unroll
                for (int x = 0; x < AHEAD; x++) {
                    const int r = r0 + x * groups;
                    if (live && r < p.dk) {
                        s[x] = *reinterpret_cast<const Pack<float, V>*>(S + (size_t)r * p.dv + cg * V);
                    } else {
#pragma unroll
                        for (int i = 0; i < V; i++) s[x].v[i] = 0.f;
                    }
                }
#pragma unroll
                for (int x = 0; x < AHEAD; x++) {
                    const int r = r0 + x * groups;
                    if (r >= p.dk) break;
#pragma unroll
                    for (int i = 0; i < V; i++) {
                        s[x].v[i] = fmaf(k[r], v[i], d * s[x].v[i]);
                        acc[i] = fmaf(q[r], s[x].v[i], acc[i]);
                    }
                    *reinterpret_cast<Pack<float, V>*>(S + (size_t)r * p.dv + cg * V) = s[x];
                }
            }
#pragma unroll
            for (int i = 0; i < V; i++) red[rg * p.dv + cg * V + i] = acc[i];
        }
    }
    __syncthreads();
    T* out = static_cast<T*>(p.out) + ((size_t)t * p.H + h) * p.dv;
    for (int i = threadIdx.x; i < p.dv; i += blockDim.x) {
        float s = 0.f;
        for (int r = 0; r < min(groups, p.dk); r++) s += red[r * p.dv + i];
        out[i] = from_f32<T>(s);
    }
}

// Whole spans, fp32 on CUDA cores: CTA per (span, head, 32 columns of the values), blocks of 32 tokens in turn.
constexpr int DS_TOK = 32, DS_COL = 32, DS_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(DS_THREADS) decay_span_kernel(const DecayParams p) {
    extern __shared__ float sm[];
    const int dk = p.dk, pitch = dk + 1;
    float* q = sm;                              // [32][dk + 1]
    float* k = q + DS_TOK * pitch;              // [32][dk + 1]
    float* S = k + DS_TOK * pitch;              // [dk][33]
    float* v = S + dk * (DS_COL + 1);           // [32][33]
    float* P = v + DS_TOK * (DS_COL + 1);       // [32][33]
    float* pw = P + DS_TOK * (DS_COL + 1);      // decay^0 .. decay^32
    const int h = blockIdx.x, c0 = blockIdx.y * DS_COL, e = blockIdx.z;
    const int n_cols = min(DS_COL, p.dv - c0), Hk = p.H * dk;
    const float d = p.decay[h];
    for (int i = threadIdx.x; i <= DS_TOK; i += DS_THREADS) pw[i] = powf(d, (float)i);
    float* St = p.state + ((size_t)p.sp.slot[e] * p.H + h) * dk * p.dv;
    const bool live = p.sp.start[e] > 0;
    for (int i = threadIdx.x; i < dk * DS_COL; i += DS_THREADS) {
        const int r = i / DS_COL, c = i % DS_COL;
        S[r * (DS_COL + 1) + c] = live && c < n_cols ? St[(size_t)r * p.dv + c0 + c] : 0.f;
    }
    const int t_end = p.sp.cu[e + 1];
    for (int t0 = p.sp.cu[e]; t0 < t_end; t0 += DS_TOK) {
        const int n = min(DS_TOK, t_end - t0);
        __syncthreads();
        for (int i = threadIdx.x; i < DS_TOK * dk; i += DS_THREADS) {
            const int r = i / dk, c = i % dk;
            const T* row = static_cast<const T*>(p.qkv) + (size_t)(t0 + min(r, n - 1)) * p.row_stride;
            q[r * pitch + c] = r < n ? silu_f(to_f32(row[h * dk + c])) : 0.f;
            k[r * pitch + c] = r < n ? silu_f(to_f32(row[Hk + h * dk + c])) : 0.f;
        }
        for (int i = threadIdx.x; i < DS_TOK * DS_COL; i += DS_THREADS) {
            const int r = i / DS_COL, c = i % DS_COL;
            const T* row = static_cast<const T*>(p.qkv) + (size_t)(t0 + min(r, n - 1)) * p.row_stride;
            v[r * (DS_COL + 1) + c] = r < n && c < n_cols ? silu_f(to_f32(row[2 * Hk + h * p.dv + c0 + c])) : 0.f;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < DS_TOK * DS_TOK; i += DS_THREADS) {
            const int r = i / DS_TOK, j = i % DS_TOK;
            float acc = 0.f;
            if (j <= r) {
                for (int x = 0; x < dk; x++) acc = fmaf(q[r * pitch + x], k[j * pitch + x], acc);
                acc *= pw[r - j];
            }
            P[r * (DS_COL + 1) + j] = acc;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < DS_TOK * DS_COL; i += DS_THREADS) {
            const int r = i / DS_COL, c = i % DS_COL;
            if (r >= n || c >= n_cols) continue;
            float far = 0.f, near = 0.f;
            for (int x = 0; x < dk; x++) far = fmaf(q[r * pitch + x], S[x * (DS_COL + 1) + c], far);
            for (int j = 0; j <= r; j++) near = fmaf(P[r * (DS_COL + 1) + j], v[j * (DS_COL + 1) + c], near);
            static_cast<T*>(p.out)[((size_t)(t0 + r) * p.H + h) * p.dv + c0 + c] = from_f32<T>(fmaf(pw[r + 1], far, near));
        }
        __syncthreads();
        for (int i = threadIdx.x; i < dk * DS_COL; i += DS_THREADS) {
            const int r = i / DS_COL, c = i % DS_COL;
            float acc = pw[n] * S[r * (DS_COL + 1) + c];
            for (int j = 0; j < n; j++) acc = fmaf(pw[n - 1 - j] * k[j * pitch + r], v[j * (DS_COL + 1) + c], acc);
            S[r * (DS_COL + 1) + c] = acc;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < dk * DS_COL; i += DS_THREADS) {
        const int r = i / DS_COL, c = i % DS_COL;
        if (c < n_cols) St[(size_t)r * p.dv + c0 + c] = S[r * (DS_COL + 1) + c];
    }
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

template <typename T>
int conv_silu(void* out, const void* x, int64_t x_stride, const float* taps, const float* bias, float* state, const ca_spans& sp,
              int channels, int K, cudaStream_t stream) {
    auto packs = [&](int v) { return channels % v == 0 && x_stride % v == 0 && reinterpret_cast<uintptr_t>(x) % (v * sizeof(T)) == 0; };
    const int v = packs(4) && K <= 4 ? 4 : (packs(2) ? 2 : 1);
    const int per = 128 * v;
    const dim3 grid((channels + per - 1) / per, sp.n_work);
    T* o = static_cast<T*>(out);
    const T* in = static_cast<const T*>(x);
#define CA_CONV(V, KM) conv_silu_kernel<T, V, KM><<<grid, 128, 0, stream>>>(o, in, x_stride, taps, bias, state, sp, channels, K)
    if (v == 4) {
        CA_CONV(4, 4);
    } else if (v == 2) {
        if (K <= 4) CA_CONV(2, 4); else CA_CONV(2, 16);
    } else {
        if (K <= 4) CA_CONV(1, 4); else CA_CONV(1, 16);
    }
#undef CA_CONV
    return done();
}

template <typename T>
int selective_scan(const ScanParams& p, int per_lane, cudaStream_t stream) {
    if (p.sp.max_tokens == 1 && p.N <= 128)
        by_lanes(scan_lanes(p.N, 4), [&](auto l) { launch_scan_step<T, decltype(l)::value>(p, stream); });
    else if (p.run == 0 && scan_short(p.sp, p.C, p.N, sizeof(T) == 2))
        by_lanes(scan_lanes(p.N, 8), [&](auto l) {
            constexpr int L = decltype(l)::value;
            if constexpr (L <= 4) scan_short_kernel<T, L><<<dim3((p.C * L + SCAN_THREADS - 1) / SCAN_THREADS, p.sp.n_entries), SCAN_THREADS, 0, stream>>>(p);
        });
    else
        by_lanes(scan_lanes(p.N, per_lane), [&](auto l) {
            constexpr int L = decltype(l)::value;
            if constexpr (scan_instance(L, 4))
                if (per_lane == 4) launch_scan<T, L, 4>(p, stream);
            if constexpr (scan_instance(L, 8))
                if (per_lane == 8) launch_scan<T, L, 8>(p, stream);
            if constexpr (scan_instance(L, 16))
                if (per_lane == 16) launch_scan<T, L, 16>(p, stream);
        });
    return done();
}

// Pieces per CTA of the tensor-core kernels (one CTA per SM; an even number, for blocks of 128 tokens): the run length that needs the fewest block times, counting two
// passes for runs and one for whole spans (0).
int decay_run(const ca_spans& sp, int heads) {
    const int longest = (sp.max_tokens + sp.work_len - 1) / sp.work_len;
    if (longest <= 1) return 0;
    auto waves = [](int64_t ctas) { return (double)((ctas + B200_SMS - 1) / B200_SMS); };
    double best = waves((int64_t)sp.n_entries * heads) * longest;
    int best_run = 0;
    for (int run = 2; run < longest; run += 2) {
        const int64_t runs = (sp.n_work + (int64_t)(run - 1) * sp.n_entries) / run;  // at most
        // in times of a piece: a run's two passes with their start, and the sweep over the runs
        const double cost = waves(runs * heads) * (run + 1.0) * 1.75 + 2.0 + 0.2 * runs;
        if (cost < best) {
            best = cost;
            best_run = run;
        }
    }
    return best_run;
}

template <typename T>
int decay_attention(const DecayParams& p, cudaStream_t stream) {
    if (p.sp.max_tokens == 1) {
        const bool v4 = p.dv % 4 == 0;
        const int cols = p.dv / (v4 ? 4 : 1), groups = cols >= DECAY_STEP_THREADS ? 1 : DECAY_STEP_THREADS / cols;
        const size_t smem = (size_t)(2 * p.dk + groups * p.dv) * sizeof(float);
        const dim3 grid(p.H, p.sp.n_entries);
        if (v4) decay_step_kernel<T, 4><<<grid, DECAY_STEP_THREADS, smem, stream>>>(p);
        else decay_step_kernel<T, 1><<<grid, DECAY_STEP_THREADS, smem, stream>>>(p);
        return done();
    }
    if (std::is_same<T, __nv_bfloat16>::value && decay_mma_serves(p.dk, p.dv, p.row_stride, p.qkv, p.sp.work_len)) {
        DecayMmaParams m{p.out, p.qkv, p.row_stride, p.decay, p.state, p.scratch, p.H, p.dk, p.dv, decay_run(p.sp, p.H), p.sp};
        if (m.run > 0 && !p.scratch) return fail("decay_attention: this batch needs scratch");
        // short portions leave most of a 128-token block empty
        const bool tc = decay_tc_serves(p.dk, p.dv) && p.sp.max_tokens > 32;
        const cudaError_t e = tc ? launch_decay_tc(m, stream) : launch_decay_mma(m, stream);
        return e == cudaSuccess ? CA_OK : fail(cudaGetErrorString(e), CA_ERR_CUDA);
    }
    const size_t smem = (size_t)(2 * DS_TOK * (p.dk + 1) + p.dk * (DS_COL + 1) + 2 * DS_TOK * (DS_COL + 1) + DS_TOK + 1) * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(decay_span_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(cudaGetErrorString(e), CA_ERR_CUDA);
    const dim3 grid(p.H, (p.dv + DS_COL - 1) / DS_COL, p.sp.n_entries);
    decay_span_kernel<T><<<grid, DS_THREADS, smem, stream>>>(p);
    return done();
}

bool spans_ok(const ca_spans* sp) {
    return sp && sp->n_entries > 0 && sp->n_tokens >= sp->n_entries && sp->n_work >= sp->n_entries && sp->cu && sp->start &&
           sp->slot && sp->work && sp->work_off && aligned16(sp->work);
}

}  // namespace
}  // namespace ca

using namespace ca;

extern "C" {

int ca_conv_silu(void* out, const void* x, int64_t x_stride, const float* taps, const float* bias, float* state, const ca_spans* sp,
                 int channels, int n_taps, int dtype, ca_stream stream) {
    if (!spans_ok(sp)) return fail("conv_silu: bad spans");
    if (channels <= 0 || n_taps < 1 || n_taps > 16 || n_taps > sp->work_len) return fail("conv_silu: 1 to 16 taps, no more than a piece has tokens");
    if (!out || !x || !taps || !bias || !state) return fail("conv_silu: null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == CA_DTYPE_BF16) return conv_silu<__nv_bfloat16>(out, x, x_stride, taps, bias, state, *sp, channels, n_taps, s);
    if (dtype == CA_DTYPE_F32) return conv_silu<float>(out, x, x_stride, taps, bias, state, *sp, channels, n_taps, s);
    return fail("conv_silu: unknown element type");
}

int64_t ca_scan_scratch_floats(const ca_spans* sp, int channels, int n_states) {
    if (!sp || channels <= 0 || n_states <= 0 || scan_shape(*sp, channels, n_states).run == 0) return 0;
    return (int64_t)sp->n_work * channels * ((int64_t)n_states + 1);
}

int ca_selective_scan(void* y, const void* x, const void* z, int64_t z_stride, const float* dt, const float* dt_bias, const float* A,
                      const float* bc, int64_t bc_stride, const float* D, float* state, float* scratch, const ca_spans* sp,
                      int channels, int n_states, int dtype, ca_stream stream) {
    if (!spans_ok(sp)) return fail("selective_scan: bad spans");
    if (channels <= 0 || n_states < 1 || n_states > 256) return fail("selective_scan: 1 to 256 states per channel");
    if (!y || !x || !z || !dt || !dt_bias || !A || !bc || !D || !state) return fail("selective_scan: null pointer");
    ScanParams p;
    const ScanShape shape = scan_shape(*sp, channels, n_states);
    const size_t es = dtype == CA_DTYPE_F32 ? 4 : 2;
    p.run = shape.run;
    p.x_vec = channels * es % 16 == 0 && z_stride * es % 16 == 0 && aligned16(x) && aligned16(z) && aligned16(dt);
    p.bc_vec = n_states % 4 == 0 && bc_stride % 4 == 0 && aligned16(bc);
    if (p.run > 0 && !scratch) return fail("selective_scan: this batch needs scratch");
    p.y = y; p.x = x; p.z = z; p.z_stride = z_stride; p.dt = dt; p.dt_bias = dt_bias; p.A = A; p.bc = bc; p.bc_stride = bc_stride;
    p.D = D; p.state = state; p.piece_state = scratch;
    p.piece_dt = scratch ? scratch + (size_t)sp->n_work * channels * n_states : nullptr;
    p.C = channels; p.N = n_states; p.sp = *sp;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == CA_DTYPE_BF16) return selective_scan<__nv_bfloat16>(p, shape.per_lane, s);
    if (dtype == CA_DTYPE_F32) return selective_scan<float>(p, shape.per_lane, s);
    return fail("selective_scan: unknown element type");
}

int ca_block_status(int32_t* status, ca_stream stream) {
    if (!status) return fail("block_status: null pointer");
    const cudaError_t e = read_decay_status(status, static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? CA_OK : fail(cudaGetErrorString(e), CA_ERR_CUDA);
}

int64_t ca_decay_scratch_floats(const ca_spans* sp, int n_heads, int d_key, int d_value, int dtype) {
    if (!sp || dtype != CA_DTYPE_BF16 || sp->max_tokens <= 1 || n_heads <= 0 || decay_run(*sp, n_heads) == 0) return 0;
    return (int64_t)sp->n_work * n_heads * d_key * d_value;
}

int ca_decay_attention(void* out, const void* qkv, int64_t row_stride, const float* decay, float* state, float* scratch, const ca_spans* sp,
                       int n_heads, int d_key, int d_value, int dtype, ca_stream stream) {
    if (!spans_ok(sp)) return fail("decay_attention: bad spans");
    if (n_heads <= 0 || d_key <= 0 || d_key > 256 || d_value <= 0 || d_value > 1024) return fail("decay_attention: head sizes out of range");
    if (!out || !qkv || !decay || !state) return fail("decay_attention: null pointer");
    DecayParams p;
    p.out = out; p.qkv = qkv; p.row_stride = row_stride; p.decay = decay; p.state = state; p.scratch = scratch;
    p.H = n_heads; p.dk = d_key; p.dv = d_value; p.sp = *sp;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == CA_DTYPE_BF16) return decay_attention<__nv_bfloat16>(p, s);
    if (dtype == CA_DTYPE_F32) return decay_attention<float>(p, s);
    return fail("decay_attention: unknown element type");
}

}  // extern "C"
