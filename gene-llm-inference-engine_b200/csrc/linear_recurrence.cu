// Mixers that carry a state of fixed size per request instead of keys and values: the recurrence
//
//     S_t = a_t S_(t-1) + b_t k_t v_t^T        (S: dk x dv per head, 32-bit, in the request's state slot)
//     o_t = S_t^T q_t + D v_t
//
// with its families of decay: a constant a per head and b = 1 (linear attention with decay);
// a_t = exp(-exp(A_log) dt_t), b_t = dt_t with dt_t = softplus(raw_t + bias) per head and token (state-space
// duality); and a factor of its own for every row of S, S_t = diag(alpha_t) S_(t-1) + k_t v_t^T with
// alpha_t = sigmoid(z_t)^(1/tau) per head, key channel and token (gated linear attention). Around it: the short causal convolution over a request's tokens whose last inputs are state too (with or without a bias
// and SiLU), and the unit-RMS norm over groups of channels with a gate before (SiLU) or after (sigmoid or SiLU) the norm.
//
// A step's rows are segments (one per request: seg_start, seg_len, state_slots as the step's descriptor holds
// them on the device). Tokens of a segment are taken in order, one after the other, by the same threads with the
// same arithmetic however the request was cut into steps and whatever else is in the batch; decays, step sizes,
// gates, norms and the state are 32-bit.
#include "common.cuh"
#include "device_limit.h"

namespace gi {

// Two 32-bit multiply-adds (products) in one instruction, each rounded like fmaf's (a product's).
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long mul_pair(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long make_pair(float a, float b) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 split_pair(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ float silu_f(float z) { return z * (1.0f / (1.0f + expf(-z))); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ---------------------------------------------------------------------------------- causal convolution
// out[t, c] = act(bias[c] + sum_j w[c, j] * u(t - (taps-1) + j, c)), act SiLU or nothing, bias optional; u before the segment's first row is the
// request's conv state [taps-1, C] (oldest first; zeros for a new request), u before the sequence is zero.
__global__ void __launch_bounds__(256)
causal_conv_kernel(const float* __restrict__ in, int ld, int in_off, const float* __restrict__ weight,
                   const float* __restrict__ bias, const float* __restrict__ state, long long slot_stride,
                   const int* __restrict__ row_req, const int* __restrict__ seg_start,
                   const int* __restrict__ state_slots, float* __restrict__ out, int C, int taps, int T, int act) {
    pdl_prologue();
    const int c = blockIdx.x * 256 + threadIdx.x;
    const int t = blockIdx.y;
    if (c >= C) return;
    const int r = row_req[t];
    const int rel = t - seg_start[r];
    const float* st = state + static_cast<long long>(state_slots[r]) * slot_stride;
    float acc = bias ? bias[c] : 0.f;
    for (int j = 0; j < taps; ++j) {
        const int back = taps - 1 - j;                 // how many tokens before t
        float u;
        if (back <= rel) u = in[static_cast<size_t>(t - back) * ld + in_off + c];
        else u = st[static_cast<size_t>(taps - 1 + rel - back) * C + c];
        acc = fmaf(weight[static_cast<size_t>(c) * taps + j], u, acc);
    }
    out[static_cast<size_t>(t) * C + c] = act ? silu_f(acc) : acc;
}

// The state after the step: the last taps-1 inputs of each segment (older ones from the old state).
__global__ void __launch_bounds__(256)
conv_state_update_kernel(const float* __restrict__ in, int ld, int in_off, float* __restrict__ state, long long slot_stride,
                         const int* __restrict__ seg_start, const int* __restrict__ seg_len,
                         const int* __restrict__ state_slots, int C, int taps) {
    pdl_prologue();
    const int c = blockIdx.x * 256 + threadIdx.x;
    const int r = blockIdx.y;
    if (c >= C) return;
    const int n = seg_len[r], s0 = seg_start[r];
    float* st = state + static_cast<long long>(state_slots[r]) * slot_stride;
    const int keep = taps - 1;
    float vals[16];
    for (int j = 0; j < keep; ++j) {
        const int rel = n - keep + j;                 // index among the segment's rows; negative: old state
        vals[j] = rel >= 0 ? in[static_cast<size_t>(s0 + rel) * ld + in_off + c] : st[static_cast<size_t>(keep + rel) * C + c];
    }
    for (int j = 0; j < keep; ++j) st[static_cast<size_t>(j) * C + c] = vals[j];
}

// The same for channels in whole fours whose rows are 16-byte aligned and 2 to 4 taps; the arithmetic of an output is the one
// above. A thread has four channels.
__device__ __forceinline__ void conv_tap(float4& acc, const float (&w)[16], int taps, int j, const float4& u) {
    acc.x = fmaf(w[j], u.x, acc.x); acc.y = fmaf(w[taps + j], u.y, acc.y);
    acc.z = fmaf(w[2 * taps + j], u.z, acc.z); acc.w = fmaf(w[3 * taps + j], u.w, acc.w);
}
template <int TAPS>
__device__ __forceinline__ void conv_weights(float (&w)[16], float4& first, const float* weight, const float* bias, int c) {
#pragma unroll
    for (int j = 0; j < TAPS; ++j)          // 4 TAPS values in a row
        *reinterpret_cast<float4*>(&w[4 * j]) = __ldg(reinterpret_cast<const float4*>(weight + static_cast<size_t>(c) * TAPS) + j);
    first = bias ? __ldg(reinterpret_cast<const float4*>(bias + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void conv_store(float* out, float4 v, int act) {
    if (act) { v.x = silu_f(v.x); v.y = silu_f(v.y); v.z = silu_f(v.z); v.w = silu_f(v.w); }
    *reinterpret_cast<float4*>(out) = v;
}

// Long segments: RUN consecutive rows a thread, every row asked for once and all at once (a value at a time and once per tap,
// 2,048 rows of 3,072 channels took 37 us; the bytes need 8).
template <int TAPS, int RUN>
__global__ void __launch_bounds__(128)
causal_conv_run_kernel(const float* __restrict__ in, int ld, int in_off, const float* __restrict__ weight,
                       const float* __restrict__ bias, const float* __restrict__ state, long long slot_stride,
                       const int* __restrict__ row_req, const int* __restrict__ seg_start,
                       const int* __restrict__ state_slots, float* __restrict__ out, int C, int T, int act) {
    pdl_launch_dependents();
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4, t0 = blockIdx.y * RUN;
    if (c >= C) return;
    float w[16];
    float4 first;
    conv_weights<TAPS>(w, first, weight, bias, c);      // the weights belong to no earlier kernel
    pdl_wait();
    float4 u[RUN + TAPS - 1];                           // rows t0 - (TAPS - 1) .. t0 + RUN - 1
#pragma unroll
    for (int k = 0; k < RUN + TAPS - 1; ++k) {
        const int t = t0 - (TAPS - 1) + k;
        u[k] = (t >= 0 && t < T) ? *reinterpret_cast<const float4*>(in + static_cast<size_t>(t) * ld + in_off + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < RUN; ++k) {
        const int t = t0 + k;
        if (t >= T) break;
        const int r = row_req[t], rel = t - seg_start[r];
        float4 acc = first;
        if (rel >= TAPS - 1) {
#pragma unroll
            for (int j = 0; j < TAPS; ++j) conv_tap(acc, w, TAPS, j, u[k + j]);
        } else {
            const float* st = state + static_cast<long long>(state_slots[r]) * slot_stride + c;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) {
                const int back = TAPS - 1 - j;
                conv_tap(acc, w, TAPS, j, back <= rel ? u[k + j] : *reinterpret_cast<const float4*>(st + static_cast<size_t>(TAPS - 1 + rel - back) * C));
            }
        }
        conv_store(out + static_cast<size_t>(t) * C + c, acc, act);
    }
}

// Segments of a token each (decoding): a thread walks through a whole segment and leaves the state behind it (one launch
// less, and the state is read once).
template <int TAPS>
__global__ void __launch_bounds__(128)
causal_conv_walk_kernel(const float* __restrict__ in, int ld, int in_off, const float* __restrict__ weight,
                        const float* __restrict__ bias, float* __restrict__ state, long long slot_stride,
                        const int* __restrict__ seg_start, const int* __restrict__ seg_len,
                        const int* __restrict__ state_slots, float* __restrict__ out, int C, int act) {
    pdl_launch_dependents();
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4, r = blockIdx.y;
    if (c >= C) return;
    float w[16];
    float4 first;
    conv_weights<TAPS>(w, first, weight, bias, c);
    pdl_wait();
    const int n = seg_len[r], s0 = seg_start[r];
    if (n <= 0) return;
    float* st = state + static_cast<long long>(state_slots[r]) * slot_stride + c;
    float4 u[TAPS];
#pragma unroll
    for (int j = 0; j < TAPS - 1; ++j) u[j] = *reinterpret_cast<const float4*>(st + static_cast<size_t>(j) * C);
    for (int t = s0; t < s0 + n; ++t) {
        u[TAPS - 1] = *reinterpret_cast<const float4*>(in + static_cast<size_t>(t) * ld + in_off + c);
        float4 acc = first;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) conv_tap(acc, w, TAPS, j, u[j]);
        conv_store(out + static_cast<size_t>(t) * C + c, acc, act);
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) u[j] = u[j + 1];
    }
#pragma unroll
    for (int j = 0; j < TAPS - 1; ++j) *reinterpret_cast<float4*>(st + static_cast<size_t>(j) * C) = u[j];
}

// ---------------------------------------------------------------------------------- the recurrence
// A block owns 32 columns (or more) of one head's state of one request, each thread a few rows x 4 columns of it in registers, as pairs of
// neighbouring columns: two multiply-adds an instruction, the factors of a row staged twice so that they are read as pairs (1,153
// tokens of 16 heads of 128 x 128: 100 -> 93 us, 2,048 tokens of 32 heads of 128 x 64: 137 -> 121, a token with a decay per row 10.3 -> 6.6).
// Tokens are staged a chunk at a time in shared memory (activated, with their a and b).
//
// Long segments are cut into parts of part_len tokens that run side by side (kParts): every part starts from a zero
// state and leaves its own end state U_p and, per token, the product A_t of the decays since the part's start
// (scan kernel); the parts' true start states follow from S_(p+1) = A_end(p) S_p + U_p, S_0 the request's state
// (link kernel, a short loop per state element); and every token gets what the start state adds to it,
// o_t += A_t S_p^T q_t (apply kernel, a small matrix product per part). Steps whose segments all fit one part run
// the scan kernel alone, straight on the state slot.
constexpr int kScanChunk = 8;

struct ScanArgs {
    const float* q; const float* k; const float* v;      // rows of ld_q / ld_k / ld_v floats, at these column offsets
    int ld_q, ld_k, ld_v, q_off, k_off, v_off;
    int H, group;                                         // head h reads q/k head h / group
    int dk, dv;
    int act;                                              // 1: SiLU on q, k and v when they are read
    const float* decay;                                   // [H] constant decays, or null for the dt form
    const float* dt_raw; int ld_dt, dt_off;               // [T, ld_dt] at dt_off + h
    const float* dt_bias; const float* a_log; const float* skip;      // [H] each; skip may be null
    const float* gate_raw; int ld_gate, gate_off;         // [T, ld_gate] at gate_off + h * dk + i: z of the per-row decay, or null
    const float* gate_bias; float inv_tau;                // [H * dk] added to z (may be null); alpha = sigmoid(z)^inv_tau
    float q_scale;                                        // a constant on the queries
    float* state; long long slot_stride; long long state_off;          // per slot: [H, dk, dv] at state_off
    const int* seg_start; const int* seg_len; const int* state_slots;
    float* out;                                           // [T, H * dv]
    int part_len, max_parts;                              // kParts: tokens per part, parts per request in the grid
    float* ws_state;                                      // [parts of the step, H, dk, dv]
    float* ws_decay;                                      // [T, H]; with per-row decays [T, H, dk]
};

// sigmoid(z)^(1/tau) = exp(-softplus(-z) / tau)
__device__ __forceinline__ float row_decay(float z, float inv_tau) { return expf(-softplus_f(-z) * inv_tau); }

// Where request r's parts start among the step's parts: the parts of the requests before it.
__device__ __forceinline__ int parts_before(const ScanArgs& p, int r) {
    int base = 0;
    for (int i = 0; i < r; ++i) base += (p.seg_len[i] + p.part_len - 1) / p.part_len;
    return base;
}

// (Left alone the compiler takes the kernel past 128 registers a thread, with a decay per row to 168, and a launch of a
// few heads' blocks then needs a second, nearly empty round over the SMs: it is held to 512 threads an SM. Five blocks of 128
// instead of four, which 96 registers allow without spills: 115 instead of 100 us at 640 blocks.)
//
// kCG: groups of four columns of a block. What a block does besides walking, activations and decays of each staged token, it does for all its
// columns at once: parts of a long segment take 256 threads' worth of columns (1,153 tokens of 16 heads of 128 x 128 in 32
// columns a block 93 us, in 64 86; a decay per row, 2,048 tokens of 16 heads of 64 x 128, 135 and in 128 columns 81), single
// tokens the narrow blocks that give every SM one.
template <int kDk, int kRT, int kCG, bool kParts, bool kRowDecay>
struct ScanShared {
    static constexpr int kGroups = kDk / kRT, kCols = 4 * kCG;
    static constexpr int kChunk = kDk > 128 && (kRowDecay || !kParts) ? kScanChunk / 2 : kScanChunk;      // tokens staged at a time
    float2 q[kChunk][kDk], k[kChunk][kDk];                // twice each: the factors of a pair of columns
    float v[kChunk][kCols];
    float o[kChunk][kGroups][kCols];
    float2 av[kRowDecay ? kChunk : 1][kRowDecay ? kDk : 2];           // per-row decays of the staged tokens
    float a[kChunk], b[kChunk];
};
template <int kDk, int kRT, int kCG, bool kParts, bool kRowDecay>
__global__ void __launch_bounds__(kDk / kRT * kCG, (kRowDecay || kDk <= 128) ? 512 / (kDk / kRT * kCG) : 1)
linear_scan_kernel(const ScanArgs p) {
    pdl_prologue();
    // A thread owns kRT rows x 4 columns of the state in registers (thread = row group x column group; a block covers
    // all kDk padded rows and 4 kCG columns): per token it reads kRT k and q values and 4 v values from shared memory
    // for 4 kRT state elements. A token's output is the sum over the row groups, added up in their order once per
    // chunk of tokens.
    constexpr int kGroups = kDk / kRT;                    // row groups
    constexpr int kThreads = kGroups * kCG, kCols = 4 * kCG;
    using Shared = ScanShared<kDk, kRT, kCG, kParts, kRowDecay>;
    constexpr int kChunk = Shared::kChunk;
    constexpr int kPerThread = kChunk * kDk / kThreads;   // q (and k) values a thread stages per chunk
    constexpr int kVPerThread = kChunk * kCols / kThreads;
    extern __shared__ __align__(16) unsigned char scan_smem[];
    Shared& shared = *reinterpret_cast<Shared*>(scan_smem);
    auto &s_q = shared.q, &s_k = shared.k;
    auto &s_av = shared.av;
    auto &s_v = shared.v;
    auto &s_o = shared.o;
    auto &s_a = shared.a, &s_b = shared.b;
    const int tile = blockIdx.x, h = blockIdx.y;
    const int r = kParts ? blockIdx.z / p.max_parts : blockIdx.z;
    const int part_idx = kParts ? blockIdx.z % p.max_parts : 0;
    const int g = h / p.group;
    const int cg = threadIdx.x % kCG, rg = threadIdx.x / kCG;
    const int j0 = tile * kCols + cg * 4;             // first of this thread's columns
    int n = p.seg_len[r], s0 = p.seg_start[r];
    float* S;
    if (kParts) {
        if (part_idx * p.part_len >= n) return;
        s0 += part_idx * p.part_len;
        n = min(p.part_len, n - part_idx * p.part_len);
        S = p.ws_state + (static_cast<size_t>(parts_before(p, r) + part_idx) * p.H + h) * p.dk * p.dv;
    } else {
        S = p.state + static_cast<long long>(p.state_slots[r]) * p.slot_stride + p.state_off +
            static_cast<long long>(h) * p.dk * p.dv;
    }
    unsigned long long s[kRT][2];                          // pairs of neighbouring columns
#pragma unroll
    for (int i = 0; i < kRT; ++i) {
        const int row = rg * kRT + i;
        float v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c)
            v[c] = (!kParts && row < p.dk && j0 + c < p.dv) ? S[static_cast<size_t>(row) * p.dv + j0 + c] : 0.f;
        s[i][0] = make_pair(v[0], v[1]); s[i][1] = make_pair(v[2], v[3]);
    }
    const float skip = p.skip ? p.skip[h] : 0.f;
    const float a_const = p.decay ? p.decay[h] : 0.f;
    const bool stepped = !kRowDecay && !p.decay;         // a and b from the step size
    const float neg_rate = stepped ? -expf(p.a_log[h]) : 0.f;
    const float bias = stepped ? p.dt_bias[h] : 0.f;
    float cum = 1.f;                                      // thread 0: product of the decays since the part's start
    constexpr int kCumPerThread = (kDk + kThreads - 1) / kThreads;
    float cumv[kCumPerThread];                            // per-row decays: the products of rows threadIdx.x + u * kThreads
#pragma unroll
    for (int u = 0; u < kCumPerThread; ++u) cumv[u] = 1.f;
    // the loads of a chunk are requested while the chunk before it is worked on
    float qv[kPerThread], kv[kPerThread], zv[kRowDecay ? kPerThread : 1], vv[kVPerThread], dt_raw = 0.f;
    auto request = [&](int c0) {
        const int m = min(kChunk, n - c0);
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            const int e = threadIdx.x + u * kThreads;
            const int tt = e / kDk, i = e % kDk;
            const size_t t = static_cast<size_t>(s0 + c0 + tt);
            const bool in = tt < m && i < p.dk;
            qv[u] = in ? p.q[t * p.ld_q + p.q_off + g * p.dk + i] : 0.f;
            kv[u] = in ? p.k[t * p.ld_k + p.k_off + g * p.dk + i] : 0.f;
            if (kRowDecay)
                zv[u] = in ? p.gate_raw[t * p.ld_gate + p.gate_off + h * p.dk + i] + (p.gate_bias ? p.gate_bias[h * p.dk + i] : 0.f) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kVPerThread; ++u) {
            const int e = threadIdx.x + u * kThreads;
            const int tt = e / kCols, jj = tile * kCols + e % kCols;
            vv[u] = (tt < m && jj < p.dv) ? p.v[static_cast<size_t>(s0 + c0 + tt) * p.ld_v + p.v_off + h * p.dv + jj] : 0.f;
        }
        if (!kRowDecay && !p.decay && threadIdx.x < m)
            dt_raw = p.dt_raw[static_cast<size_t>(s0 + c0 + threadIdx.x) * p.ld_dt + p.dt_off + h];
    };
    request(0);
    for (int c0 = 0; c0 < n; c0 += kChunk) {
        const int m = min(kChunk, n - c0);
        __syncthreads();                                  // the chunk before is done with the staging buffers
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            const int e = threadIdx.x + u * kThreads;
            if (!kParts && e / kDk >= m) break;           // (64 single tokens, 16 heads of 128 x 128: 31.1 -> 27.4 us)
            const float q = (p.act ? silu_f(qv[u]) : qv[u]) * p.q_scale, k = p.act ? silu_f(kv[u]) : kv[u];
            s_q[e / kDk][e % kDk] = make_float2(q, q);
            s_k[e / kDk][e % kDk] = make_float2(k, k);
            if (kRowDecay) {
                const float a = (e / kDk < m && e % kDk < p.dk) ? row_decay(zv[u], p.inv_tau) : 1.f;
                s_av[e / kDk][e % kDk] = make_float2(a, a);
            }
        }
#pragma unroll
        for (int u = 0; u < kVPerThread; ++u) {
            const int e = threadIdx.x + u * kThreads;
            s_v[e / kCols][e % kCols] = p.act ? silu_f(vv[u]) : vv[u];
        }
        if (threadIdx.x < m) {
            if (kRowDecay) {
                s_a[threadIdx.x] = 1.f;
                s_b[threadIdx.x] = 1.f;
            } else if (p.decay) {
                s_a[threadIdx.x] = a_const;
                s_b[threadIdx.x] = 1.f;
            } else {
                const float dt = softplus_f(dt_raw + bias);
                s_a[threadIdx.x] = expf(neg_rate * dt);
                s_b[threadIdx.x] = dt;
            }
        }
        __syncthreads();
        if (c0 + kChunk < n) request(c0 + kChunk);
        if (kParts && !kRowDecay && tile == 0 && threadIdx.x == 0) {
            for (int tt = 0; tt < m; ++tt) {
                cum *= s_a[tt];
                p.ws_decay[static_cast<size_t>(s0 + c0 + tt) * p.H + h] = cum;
            }
        }
        if (kParts && kRowDecay && tile == 0) {
#pragma unroll
            for (int u = 0; u < kCumPerThread; ++u) {
                const int i = threadIdx.x + u * kThreads;
                if (i < p.dk) {
                    for (int tt = 0; tt < m; ++tt) {
                        cumv[u] *= s_av[tt][i].x;
                        p.ws_decay[(static_cast<size_t>(s0 + c0 + tt) * p.H + h) * p.dk + i] = cumv[u];
                    }
                }
            }
        }
        for (int tt = 0; tt < m; ++tt) {
            const float a = s_a[tt], b = s_b[tt];
            const ulonglong2 v4 = *reinterpret_cast<const ulonglong2*>(&s_v[tt][cg * 4]);
            const unsigned long long bb = make_pair(b, b), aa = make_pair(a, a);
            const unsigned long long bv[2] = {mul_pair(bb, v4.x), mul_pair(bb, v4.y)};
            unsigned long long o[2] = {0ull, 0ull};
            const ulonglong2* k2 = reinterpret_cast<const ulonglong2*>(&s_k[tt][rg * kRT]);
            const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(&s_q[tt][rg * kRT]);
            const ulonglong2* a2 = reinterpret_cast<const ulonglong2*>(&s_av[kRowDecay ? tt : 0][kRowDecay ? rg * kRT : 0]);
#pragma unroll
            for (int i2 = 0; i2 < kRT / 2; ++i2) {
                const ulonglong2 kk = k2[i2], qq = q2[i2];
                const unsigned long long kr[2] = {kk.x, kk.y}, qr[2] = {qq.x, qq.y};
                unsigned long long ar[2] = {aa, aa};
                if (kRowDecay) { const ulonglong2 av = a2[i2]; ar[0] = av.x; ar[1] = av.y; }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        unsigned long long& x = s[2 * i2 + u][c];
                        x = fma_pair(ar[u], x, mul_pair(kr[u], bv[c]));
                        o[c] = fma_pair(x, qr[u], o[c]);
                    }
                }
            }
            *reinterpret_cast<ulonglong2*>(&s_o[tt][rg][cg * 4]) = make_ulonglong2(o[0], o[1]);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < m * kCols; e += kThreads) {
            const int tt = e / kCols, c = e % kCols;
            const int jj = tile * kCols + c;
            float o = 0.f;
#pragma unroll
            for (int w = 0; w < kGroups; ++w) o += s_o[tt][w][c];
            if (jj < p.dv)
                p.out[static_cast<size_t>(s0 + c0 + tt) * p.H * p.dv + h * p.dv + jj] = fmaf(skip, s_v[tt][c], o);
        }
    }
#pragma unroll
    for (int i = 0; i < kRT; ++i) {
        const int row = rg * kRT + i;
        const float2 lo = split_pair(s[i][0]), hi = split_pair(s[i][1]);
        const float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (row < p.dk && j0 + c < p.dv) S[static_cast<size_t>(row) * p.dv + j0 + c] = v[c];
    }
}

// The parts' start states: one thread per element of a request's state walks over the request's parts.
__global__ void __launch_bounds__(256)
scan_link_kernel(const ScanArgs p) {
    pdl_prologue();
    const int r = blockIdx.y;
    const size_t per_head = static_cast<size_t>(p.dk) * p.dv;
    const size_t e = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
    if (e >= per_head * p.H) return;
    const int h = static_cast<int>(e / per_head);
    const int n = p.seg_len[r], s0 = p.seg_start[r];
    const int parts = (n + p.part_len - 1) / p.part_len;
    float* slot = p.state + static_cast<long long>(p.state_slots[r]) * p.slot_stride + p.state_off;
    float* ws = p.ws_state + static_cast<size_t>(parts_before(p, r)) * p.H * per_head;
    float S = slot[e];
    constexpr int kBatch = 8;                             // parts whose loads are in flight together
    for (int q0 = 0; q0 < parts; q0 += kBatch) {
        float U[kBatch], A[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int q = q0 + u;
            const bool in = q < parts;
            const int last = s0 + min((q + 1) * p.part_len, n) - 1;
            U[u] = in ? ws[static_cast<size_t>(q) * p.H * per_head + e] : 0.f;
            A[u] = !in ? 1.f : p.gate_raw ? p.ws_decay[(static_cast<size_t>(last) * p.H + h) * p.dk + (e % per_head) / p.dv]
                                          : p.ws_decay[static_cast<size_t>(last) * p.H + h];
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if (q0 + u < parts) {
                ws[static_cast<size_t>(q0 + u) * p.H * per_head + e] = S;      // the state this part starts from
                S = fmaf(A[u], S, U[u]);
            }
        }
    }
    slot[e] = S;
}

// o_t += A_t S_p^T q_t for 64 tokens of a part, one head and kDv columns (64 or 128): a small matrix product whose tiles lie in
// registers. The queries (by channel) in shared memory, the start state's rows staged 16 at a time; a thread has 8 tokens x
// kDv / 16 columns, a warp 16 tokens. (16 tokens x 32 columns a block, four sums a thread, read shared memory twice for
// every four multiply-adds: 72 us at twelve parts of 16 heads of 128 x 128, of which the multiply-adds need 11.)
constexpr int kApplyRows = 64, kApplyStep = 16;

template <int kDk, int kDv>
__global__ void __launch_bounds__(128)
scan_apply_kernel(const ScanArgs p, int blocks_per_part) {            // grid (column blocks x token blocks of a part, H, requests x parts)
    pdl_prologue();
    constexpr int kT = kApplyRows + 4, kX = kDv + 4, kTN = kDv / 16, kPer = kApplyStep * kDv / 128;
    extern __shared__ __align__(16) float apply_smem[];
    float* s_q = apply_smem;                           // [kDk][kT]
    float* s_x = s_q + kDk * kT;                       // [kApplyStep][kX]
    const int h = blockIdx.y, g = h / p.group;
    const int r = blockIdx.z / p.max_parts, part_idx = blockIdx.z % p.max_parts, t0 = blockIdx.x % blocks_per_part * kApplyRows;
    int n = p.seg_len[r], s0 = p.seg_start[r];
    if (part_idx * p.part_len >= n) return;
    s0 += part_idx * p.part_len;
    n = min(p.part_len, n - part_idx * p.part_len);
    if (t0 >= n) return;
    s0 += t0;
    const int tid = threadIdx.x, rows = min(kApplyRows, n - t0), c0 = blockIdx.x / blocks_per_part * kDv;
    const int tm = tid / 16 * 8, tn = tid % 16 * 4;    // this thread's tokens tm .. tm + 7; columns tn .. tn + 3 (and 64 further on)
    const bool works = tid / 32 * 16 < rows;
    const float* S = p.ws_state + (static_cast<size_t>(parts_before(p, r) + part_idx) * p.H + h) * p.dk * p.dv;
    float xv[kPer];
    auto request = [&](int i0) {                       // asked for while the rows before them are worked on
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int e = tid + u * 128, i = i0 + e / kDv, j = c0 + e % kDv;
            xv[u] = (i < p.dk && j < p.dv) ? S[static_cast<size_t>(i) * p.dv + j] : 0.f;
        }
    };
    request(0);
    // the queries, 16 loads of a thread in flight
    constexpr int kBatch = kApplyRows * kDk / 128 < 16 ? kApplyRows * kDk / 128 : 16;
    for (int e0 = tid; e0 < kApplyRows * kDk; e0 += 128 * kBatch) {
        float qv[kBatch], cv[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + u * 128, t = e / kDk, i = e % kDk;
            const bool in = t < rows && i < p.dk;
            qv[u] = in ? p.q[static_cast<size_t>(s0 + t) * p.ld_q + p.q_off + g * p.dk + i] : 0.f;
            // per-row decays: the product since the part's start scales the query's own channel
            cv[u] = (in && p.gate_raw) ? p.ws_decay[(static_cast<size_t>(s0 + t) * p.H + h) * p.dk + i] : 1.f;
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int e = e0 + u * 128;
            s_q[e % kDk * kT + e / kDk] = (p.act ? silu_f(qv[u]) : qv[u]) * p.q_scale * cv[u];
        }
    }
    unsigned long long acc[8][kTN / 2];                // pairs of neighbouring columns
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int j = 0; j < kTN / 2; ++j) acc[m][j] = 0ull;
    for (int i0 = 0; i0 < p.dk; i0 += kApplyStep) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; ++u) { const int e = tid + u * 128; s_x[e / kDv * kX + e % kDv] = xv[u]; }
        __syncthreads();
        if (i0 + kApplyStep < p.dk) request(i0 + kApplyStep);
        if (!works) continue;
#pragma unroll
        for (int i = 0; i < kApplyStep; ++i) {
            float l[8];
            unsigned long long x[kTN / 2];
            *reinterpret_cast<float4*>(&l[0]) = *reinterpret_cast<const float4*>(s_q + (i0 + i) * kT + tm);
            *reinterpret_cast<float4*>(&l[4]) = *reinterpret_cast<const float4*>(s_q + (i0 + i) * kT + tm + 4);
#pragma unroll
            for (int j = 0; j < kTN; j += 4) {
                const ulonglong2 four = *reinterpret_cast<const ulonglong2*>(s_x + i * kX + tn + j * 16);
                x[j / 2] = four.x; x[j / 2 + 1] = four.y;
            }
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const unsigned long long lm = make_pair(l[m], l[m]);
#pragma unroll
                for (int j = 0; j < kTN / 2; ++j) acc[m][j] = fma_pair(lm, x[j], acc[m][j]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        if (tm + m >= rows) continue;
        const size_t t = static_cast<size_t>(s0 + tm + m);
        const float f = p.gate_raw ? 1.f : p.ws_decay[t * p.H + h];
        float* o = p.out + t * p.H * p.dv + h * p.dv;
#pragma unroll
        for (int j = 0; j < kTN; ++j) {
            const int col = c0 + tn + (j & 3) + (j & 4) * 16;
            const float2 two = split_pair(acc[m][j / 2]);
            if (col < p.dv) o[col] = fmaf(f, j & 1 ? two.y : two.x, o[col]);
        }
    }
}

// ---------------------------------------------------------------------------------- gated group norm
// One block per (token, group). mode 0: out = w * unit_rms(y) * sigmoid(gate); mode 1: out = w * unit_rms(y * silu(gate));
// mode 2: out = w * unit_rms(y) * silu(gate).
// Groups of at most 4096 channels in 16-byte pieces (kVec) are read once and kept in registers between the sum
// and the scaling; the sum's order (a fixed strided assignment, a fixed xor tree, the warps in index order) is
// the same in both forms.
template <typename TOut, bool kVec>
__global__ void __launch_bounds__(256)
gated_group_norm_kernel(const float* __restrict__ y, const float* __restrict__ gate, int ld_gate, int gate_off,
                        const float* __restrict__ weight, TOut* __restrict__ out, int W, int groups, float eps,
                        int mode, float out_scale) {
    pdl_prologue();
    __shared__ float warp_part[8];
    const int t = blockIdx.x, grp = blockIdx.y;
    const int n = W / groups;
    const float* yr = y + static_cast<size_t>(t) * W + grp * n;
    const float* gr = gate + static_cast<size_t>(t) * ld_gate + gate_off + grp * n;
    TOut* o = out + static_cast<size_t>(t) * W + grp * n;
    const float* w = weight + grp * n;
    float ss = 0.f;
    float4 kept[4], gk[4];
    if (kVec) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = threadIdx.x + k * 256;
            kept[k] = gk[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < n / 4) {
                kept[k] = reinterpret_cast<const float4*>(yr)[i];
                gk[k] = reinterpret_cast<const float4*>(gr)[i];
                if (mode == 1) {
                    kept[k].x *= silu_f(gk[k].x); kept[k].y *= silu_f(gk[k].y);
                    kept[k].z *= silu_f(gk[k].z); kept[k].w *= silu_f(gk[k].w);
                }
            }
            ss = fmaf(kept[k].x, kept[k].x, ss); ss = fmaf(kept[k].y, kept[k].y, ss);
            ss = fmaf(kept[k].z, kept[k].z, ss); ss = fmaf(kept[k].w, kept[k].w, ss);
        }
    } else {
        for (int d = threadIdx.x; d < n; d += 256) {
            const float v = mode == 1 ? yr[d] * silu_f(gr[d]) : yr[d];
            ss = fmaf(v, v, ss);
        }
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) total += warp_part[k];
    const float scale = 1.0f / sqrtf(total / static_cast<float>(n) + eps);
    if (kVec) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = threadIdx.x + k * 256;
            if (i >= n / 4) continue;
            const float4 ww = reinterpret_cast<const float4*>(w)[i];
            float r[4] = {ww.x * (scale * kept[k].x), ww.y * (scale * kept[k].y), ww.z * (scale * kept[k].z), ww.w * (scale * kept[k].w)};
            if (mode == 0) {
                r[0] *= 1.0f / (1.0f + expf(-gk[k].x)); r[1] *= 1.0f / (1.0f + expf(-gk[k].y));
                r[2] *= 1.0f / (1.0f + expf(-gk[k].z)); r[3] *= 1.0f / (1.0f + expf(-gk[k].w));
            } else if (mode == 2) {
                r[0] *= silu_f(gk[k].x); r[1] *= silu_f(gk[k].y); r[2] *= silu_f(gk[k].z); r[3] *= silu_f(gk[k].w);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) o[4 * i + c] = from_float<TOut>(r[c] * out_scale);
        }
    } else {
        for (int d = threadIdx.x; d < n; d += 256) {
            float v;
            if (mode == 1) v = w[d] * (scale * (yr[d] * silu_f(gr[d])));
            else if (mode == 2) v = w[d] * (scale * yr[d]) * silu_f(gr[d]);
            else v = w[d] * (scale * yr[d]) * (1.0f / (1.0f + expf(-gr[d])));
            o[d] = from_float<TOut>(v * out_scale);
        }
    }
}

// The same for groups of at most 512 channels in 16-byte pieces: a warp per (token, group), eight groups a block, no
// block barrier; a lane keeps its up to four pieces in registers. The sum's order: a lane's chain over its pieces, then
// the fixed xor tree.
template <typename TOut>
__global__ void __launch_bounds__(256)
gated_group_norm_warp_kernel(const float* __restrict__ y, const float* __restrict__ gate, int ld_gate, int gate_off,
                             const float* __restrict__ weight, TOut* __restrict__ out, int W, int groups, float eps,
                             int mode, float out_scale, long long total_groups) {
    pdl_prologue();
    const long long item = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (item >= total_groups) return;
    const int lane = threadIdx.x & 31;
    const long long t = item / groups;
    const int grp = static_cast<int>(item % groups);
    const int n = W / groups;
    const float4* yr = reinterpret_cast<const float4*>(y + static_cast<size_t>(t) * W + grp * n);
    const float4* gr = reinterpret_cast<const float4*>(gate + static_cast<size_t>(t) * ld_gate + gate_off + grp * n);
    const float4* w = reinterpret_cast<const float4*>(weight + grp * n);
    TOut* o = out + static_cast<size_t>(t) * W + grp * n;
    float4 kept[4], gk[4];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = lane + k * 32;
        kept[k] = gk[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n / 4) {
            kept[k] = yr[i];
            gk[k] = gr[i];
            if (mode == 1) {
                kept[k].x *= silu_f(gk[k].x); kept[k].y *= silu_f(gk[k].y);
                kept[k].z *= silu_f(gk[k].z); kept[k].w *= silu_f(gk[k].w);
            }
        }
        ss = fmaf(kept[k].x, kept[k].x, ss); ss = fmaf(kept[k].y, kept[k].y, ss);
        ss = fmaf(kept[k].z, kept[k].z, ss); ss = fmaf(kept[k].w, kept[k].w, ss);
    }
    ss = warp_sum(ss);
    const float scale = 1.0f / sqrtf(ss / static_cast<float>(n) + eps);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = lane + k * 32;
        if (i >= n / 4) continue;
        const float4 ww = w[i];
        float r[4] = {ww.x * (scale * kept[k].x), ww.y * (scale * kept[k].y), ww.z * (scale * kept[k].z), ww.w * (scale * kept[k].w)};
        if (mode == 0) {
            r[0] *= 1.0f / (1.0f + expf(-gk[k].x)); r[1] *= 1.0f / (1.0f + expf(-gk[k].y));
            r[2] *= 1.0f / (1.0f + expf(-gk[k].z)); r[3] *= 1.0f / (1.0f + expf(-gk[k].w));
        } else if (mode == 2) {
            r[0] *= silu_f(gk[k].x); r[1] *= silu_f(gk[k].y); r[2] *= silu_f(gk[k].z); r[3] *= silu_f(gk[k].w);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) o[4 * i + c] = from_float<TOut>(r[c] * out_scale);
    }
}

}  // namespace gi

using namespace gi;

static int gi_causal_conv_impl(const float* in, int ld, int in_off, const float* weight, const float* bias, float* state,
                               long long slot_stride, long long state_off, const int* row_req, const int* seg_start,
                               const int* seg_len, const int* state_slots, float* out, int C, int taps, int T, int R,
                               int act, void* stream) {
    if (T == 0) return 0;
    GI_REQUIRE(T > 0 && R > 0 && C > 0, "causal_conv: sizes must be positive");
    GI_REQUIRE(taps >= 1 && taps <= 17, "causal_conv: %d taps are not supported (1 to 17)", taps);
    GI_REQUIRE(T <= 65535 && R <= 65535, "causal_conv: %d rows in one step exceed the grid limit 65535", T);
    GI_REQUIRE(in_off >= 0 && in_off + C <= ld, "causal_conv: the channels lie outside the input row of %d", ld);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned cb = (C + 255) / 256, cb4 = (C / 4 + 127) / 128;
    auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    const bool fours = C % 4 == 0 && ld % 4 == 0 && in_off % 4 == 0 && slot_stride % 4 == 0 && state_off % 4 == 0 && taps >= 2 && taps <= 4 &&
                       aligned(in) && aligned(weight) && aligned(bias) && aligned(state) && aligned(out);
    if (fours && T == R) {
        auto walk = [&](auto kernel) {
            launch_kernel(kernel, dim3(cb4, R), dim3(128), 0, st, in, ld, in_off, weight, bias, state + state_off, slot_stride, seg_start, seg_len, state_slots,
                          out, C, act);
        };
        if (taps == 2) walk(causal_conv_walk_kernel<2>);
        else if (taps == 3) walk(causal_conv_walk_kernel<3>);
        else walk(causal_conv_walk_kernel<4>);
        return check_launch("causal_conv");
    }
    if (fours) {
        // runs of eight rows once they fill the SMs (four blocks of 128 threads each), else of two
        const bool longer = static_cast<long long>(cb4) * ((T + 7) / 8) >= 148 * 4;
        auto run = [&](auto kernel, int rows) {
            launch_kernel(kernel, dim3(cb4, (T + rows - 1) / rows), dim3(128), 0, st, in, ld, in_off, weight, bias, static_cast<const float*>(state + state_off),
                          slot_stride, row_req, seg_start, state_slots, out, C, T, act);
        };
        if (taps == 2) { if (longer) run(causal_conv_run_kernel<2, 8>, 8); else run(causal_conv_run_kernel<2, 2>, 2); }
        else if (taps == 3) { if (longer) run(causal_conv_run_kernel<3, 8>, 8); else run(causal_conv_run_kernel<3, 2>, 2); }
        else { if (longer) run(causal_conv_run_kernel<4, 8>, 8); else run(causal_conv_run_kernel<4, 2>, 2); }
    } else launch_kernel((causal_conv_kernel), dim3(cb, T), dim3(256), 0, st, in, ld, in_off, weight, bias,
                  static_cast<const float*>(state + state_off), slot_stride, row_req, seg_start, state_slots, out, C, taps, T, act);
    if (taps > 1)
        launch_kernel((conv_state_update_kernel), dim3(cb, R), dim3(256), 0, st, in, ld, in_off, state + state_off, slot_stride,
                      seg_start, seg_len, state_slots, C, taps);
    return check_launch("causal_conv");
}

template <int kDk, int kDv>
static int launch_apply(const ScanArgs& a, int R, cudaStream_t st) {
    constexpr int smem = (kDk * (kApplyRows + 4) + kApplyStep * (kDv + 4)) * 4;
    static SharedLimit limit;
    const cudaError_t ready = limit.allow(reinterpret_cast<const void*>(scan_apply_kernel<kDk, kDv>), smem);
    if (ready != cudaSuccess) { set_error("linear_scan: %s", cudaGetErrorString(ready)); return 1; }
    const int blocks = (a.part_len + kApplyRows - 1) / kApplyRows;
    launch_kernel((scan_apply_kernel<kDk, kDv>), dim3((a.dv + kDv - 1) / kDv * blocks, a.H, R * a.max_parts), dim3(128), smem, st, a, blocks);
    return check_launch("linear_scan");
}

template <int kDk, int kRT, int kCG, bool kParts, bool kRowDecay>
static int launch_scan_as(const ScanArgs& a, int blocks, cudaStream_t st) {
    constexpr int kSmem = static_cast<int>(sizeof(ScanShared<kDk, kRT, kCG, kParts, kRowDecay>));
    if constexpr (kSmem > 48 * 1024) {
        static SharedLimit limit;
        const cudaError_t ready = limit.allow(reinterpret_cast<const void*>(linear_scan_kernel<kDk, kRT, kCG, kParts, kRowDecay>), kSmem);
        if (ready != cudaSuccess) { set_error("linear_scan: %s", cudaGetErrorString(ready)); return 1; }
    }
    launch_kernel((linear_scan_kernel<kDk, kRT, kCG, kParts, kRowDecay>), dim3((a.dv + 4 * kCG - 1) / (4 * kCG), a.H, blocks), dim3(kDk / kRT * kCG), kSmem, st, a);
    return check_launch("linear_scan");
}

template <int kDk, int kRT>
static int launch_scan(const ScanArgs& a, int R, cudaStream_t st) {
    const bool rows = a.gate_raw != nullptr;
    if (a.part_len == 0) return rows ? launch_scan_as<kDk, kRT, 8, false, true>(a, R, st) : launch_scan_as<kDk, kRT, 8, false, false>(a, R, st);
    // parts: blocks of 256 threads where the values are that wide (other state sizes: as narrow as single tokens)
    constexpr int kWide = kDk == 128 ? 16 : kDk == 64 ? 32 : 8, kHalf = kWide > 16 ? 16 : kWide;
    const int blocks = R * a.max_parts;
    int rc;
    if (kWide > kHalf && a.dv > 64) rc = rows ? launch_scan_as<kDk, kRT, kWide, true, true>(a, blocks, st) : launch_scan_as<kDk, kRT, kWide, true, false>(a, blocks, st);
    else if (kHalf > 8 && a.dv > 32) rc = rows ? launch_scan_as<kDk, kRT, kHalf, true, true>(a, blocks, st) : launch_scan_as<kDk, kRT, kHalf, true, false>(a, blocks, st);
    else rc = rows ? launch_scan_as<kDk, kRT, 8, true, true>(a, blocks, st) : launch_scan_as<kDk, kRT, 8, true, false>(a, blocks, st);
    if (rc != 0) return rc;
    const size_t elements = static_cast<size_t>(a.H) * a.dk * a.dv;
    launch_kernel((scan_link_kernel), dim3(static_cast<unsigned>((elements + 255) / 256), R), dim3(256), 0, st, a);
    return a.dv <= 64 ? launch_apply<kDk, 64>(a, R, st) : launch_apply<kDk, 128>(a, R, st);
}

// part_len 0: every segment is walked from the request's state by one block per head and column tile. Otherwise
// segments are cut into parts of part_len tokens (at most max_parts per request) that run side by side; ws_state
// holds [parts of the step, H, dk, dv] floats and ws_decay [T, H].
static int gi_linear_scan_impl(const float* q, int ld_q, int q_off, const float* k, int ld_k, int k_off, const float* v,
                               int ld_v, int v_off, int H, int group, int dk, int dv, int act, const float* decay,
                               const float* dt_raw, int ld_dt, int dt_off, const float* dt_bias, const float* a_log,
                               const float* skip, const float* gate_raw, int ld_gate, int gate_off, const float* gate_bias,
                               float inv_tau, float q_scale, float* state, long long slot_stride, long long state_off,
                               const int* seg_start, const int* seg_len, const int* state_slots, float* out, int R,
                               int part_len, int max_parts, float* ws_state, float* ws_decay, void* stream) {
    if (R == 0) return 0;
    GI_REQUIRE(R > 0 && H > 0 && dk > 0 && dv > 0 && group > 0, "linear_scan: sizes must be positive");
    GI_REQUIRE(H % group == 0, "linear_scan: %d heads are not a multiple of the group size %d", H, group);
    GI_REQUIRE(dk <= 256, "linear_scan: %d state rows per head exceed 256", dk);
    GI_REQUIRE(decay != nullptr || gate_raw != nullptr || (dt_raw != nullptr && dt_bias != nullptr && a_log != nullptr),
               "linear_scan: neither constant decays nor step sizes nor per-row decays are given");
    GI_REQUIRE(gate_raw == nullptr || (group == 1 && gate_off >= 0 && gate_off + H * dk <= ld_gate),
               "linear_scan: per-row decays need a key head per head and their columns inside a row of %d", ld_gate);
    GI_REQUIRE(part_len == 0 || (part_len > 0 && max_parts > 0 && ws_state != nullptr && ws_decay != nullptr),
               "linear_scan: parts need their length, their number and both workspaces");
    GI_REQUIRE(static_cast<long long>(R) * (part_len ? max_parts : 1) <= 65535 && H <= 65535, "linear_scan: the grid limit 65535 is exceeded");
    ScanArgs a{q, k, v, ld_q, ld_k, ld_v, q_off, k_off, v_off, H, group, dk, dv, act, decay, dt_raw, ld_dt, dt_off, dt_bias,
               a_log, skip, gate_raw, ld_gate, gate_off, gate_bias, inv_tau, q_scale, state, slot_stride, state_off, seg_start, seg_len, state_slots, out, part_len, max_parts, ws_state,
               ws_decay};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // (padded state rows, rows per thread)
    if (dk <= 16) return launch_scan<16, 4>(a, R, st);
    if (dk <= 32) return launch_scan<32, 4>(a, R, st);
    if (dk <= 64) return launch_scan<64, 8>(a, R, st);
    if (dk <= 128) return launch_scan<128, 8>(a, R, st);
    return launch_scan<256, 16>(a, R, st);
}

static int gi_gated_group_norm_impl(const float* y, const float* gate, int ld_gate, int gate_off, const float* weight, void* out,
                                    int out_dtype, int T, int W, int groups, float eps, int mode, float out_scale, void* stream) {
    if (T == 0) return 0;
    GI_REQUIRE(T > 0 && W > 0 && groups > 0 && W % groups == 0, "gated_group_norm: %d channels do not split into %d groups", W, groups);
    GI_REQUIRE(T <= 2147483647 && groups <= 65535, "gated_group_norm: the grid limit is exceeded");
    GI_REQUIRE(mode >= 0 && mode <= 2, "gated_group_norm: unknown mode %d", mode);
    GI_REQUIRE(gate_off >= 0 && gate_off + W <= ld_gate, "gated_group_norm: the gate lies outside its row of %d", ld_gate);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int n = W / groups;
    const bool vec = n % 4 == 0 && n <= 4096 && W % 4 == 0 && ld_gate % 4 == 0 && gate_off % 4 == 0 &&
                     reinterpret_cast<uintptr_t>(y) % 16 == 0 && reinterpret_cast<uintptr_t>(gate) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(weight) % 16 == 0;
    if (vec && n <= 512 && groups > 1 && (out_dtype == kBF16 || out_dtype == kF32)) {
        // small groups: a warp per group
        const long long total = static_cast<long long>(T) * groups;
        const unsigned blocks = static_cast<unsigned>((total + 7) / 8);
        if (out_dtype == kBF16) launch_kernel((gated_group_norm_warp_kernel<__nv_bfloat16>), dim3(blocks), dim3(256), 0, st, y, gate, ld_gate, gate_off, weight, static_cast<__nv_bfloat16*>(out), W, groups, eps, mode, out_scale, total);
        else launch_kernel((gated_group_norm_warp_kernel<float>), dim3(blocks), dim3(256), 0, st, y, gate, ld_gate, gate_off, weight, static_cast<float*>(out), W, groups, eps, mode, out_scale, total);
        return check_launch("gated_group_norm");
    }
    if (out_dtype == kBF16) {
        if (vec) launch_kernel((gated_group_norm_kernel<__nv_bfloat16, true>), dim3(T, groups), dim3(256), 0, st, y, gate, ld_gate, gate_off, weight, static_cast<__nv_bfloat16*>(out), W, groups, eps, mode, out_scale);
        else launch_kernel((gated_group_norm_kernel<__nv_bfloat16, false>), dim3(T, groups), dim3(256), 0, st, y, gate, ld_gate, gate_off, weight, static_cast<__nv_bfloat16*>(out), W, groups, eps, mode, out_scale);
    } else if (out_dtype == kF32) {
        if (vec) launch_kernel((gated_group_norm_kernel<float, true>), dim3(T, groups), dim3(256), 0, st, y, gate, ld_gate, gate_off, weight, static_cast<float*>(out), W, groups, eps, mode, out_scale);
        else launch_kernel((gated_group_norm_kernel<float, false>), dim3(T, groups), dim3(256), 0, st, y, gate, ld_gate, gate_off, weight, static_cast<float*>(out), W, groups, eps, mode, out_scale);
    }
    else
        GI_REQUIRE(false, "gated_group_norm: unsupported output dtype code %d", out_dtype);
    return check_launch("gated_group_norm");
}

extern "C" int gi_causal_conv(const float* in, int ld, int in_off, const float* weight, const float* bias, float* state, long long slot_stride, long long state_off, const int* row_req, const int* seg_start, const int* seg_len, const int* state_slots, float* out, int C, int taps, int T, int R, int act, void* stream) {
    return gi::dispatch(gi_causal_conv_impl, in, ld, in_off, weight, bias, state, slot_stride, state_off, row_req, seg_start, seg_len, state_slots, out, C, taps, T, R, act, stream);
}

extern "C" int gi_linear_scan(const float* q, int ld_q, int q_off, const float* k, int ld_k, int k_off, const float* v, int ld_v, int v_off, int H, int group, int dk, int dv, int act, const float* decay, const float* dt_raw, int ld_dt, int dt_off, const float* dt_bias, const float* a_log, const float* skip, const float* gate_raw, int ld_gate, int gate_off, const float* gate_bias, float inv_tau, float q_scale, float* state, long long slot_stride, long long state_off, const int* seg_start, const int* seg_len, const int* state_slots, float* out, int R, int part_len, int max_parts, float* ws_state, float* ws_decay, void* stream) {
    return gi::dispatch(gi_linear_scan_impl, q, ld_q, q_off, k, ld_k, k_off, v, ld_v, v_off, H, group, dk, dv, act, decay, dt_raw, ld_dt, dt_off, dt_bias, a_log, skip, gate_raw, ld_gate, gate_off, gate_bias, inv_tau, q_scale, state, slot_stride, state_off, seg_start, seg_len, state_slots, out, R, part_len, max_parts, ws_state, ws_decay, stream);
}

extern "C" int gi_gated_group_norm(const float* y, const float* gate, int ld_gate, int gate_off, const float* weight, void* out, int out_dtype, int T, int W, int groups, float eps, int mode, float out_scale, void* stream) {
    return gi::dispatch(gi_gated_group_norm_impl, y, gate, ld_gate, gate_off, weight, out, out_dtype, T, W, groups, eps, mode, out_scale, stream);
}
