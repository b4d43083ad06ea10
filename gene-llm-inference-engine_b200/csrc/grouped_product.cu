// Matrix products whose weight matrix depends on the row: one matrix per head, or one per expert.
//
//   grouped_product   out[row, g-th slice] (=) W[g] a[row, g-th slice]  for tiles of 16 rows that share a group g
//     heads    every row (token) runs through every group (head) h: a's columns a_off + h * a_gs .. + K,
//              W[h] = w + h * w_gs [N, K], out's columns o_off + h * o_gs .. + N; optionally ``tail`` more
//              columns behind a head's K inputs are rotated by the row's position and copied behind its N outputs
//              (queries of an attention over a shared latent: the plain part goes through the head's key matrix,
//              the rotated part stays; pairs of neighbours or of the two halves); optionally every output is multiplied by
//              the sigmoid of a gate value of its own, or of one of its head's (32-bit, in a row of the token: the heads'
//              outputs of a gated attention)
//     experts  rows are (token, choice) pairs sorted by expert: tile i belongs to expert tile_group[i], its rows are
//              sorted_rows[16 i ..] (-1: none); the input row is pair / a_div, the output row the pair;
//              gated: out = act(W_gate a) * (W_up a) with W[g] = [gate rows; up rows]; else optionally out = act(W a)
//   route             per token: z = W_r x in 32-bit, s = sigmoid(z) or softmax(z) over all experts, the ``top`` experts by
//                     s + correction; weights s, or s / (sum of the chosen s + 1e-20), times a constant; optionally also
//                     sigmoid(w_g x), one number per token (the gate of an expert that every token uses)
//   route_align       buckets the pairs by expert into tiles of 16 rows (padding with -1), one block; for many rows
//                     into tiles of 128, the token tiles of the tensor-core product that takes a matrix per tile
//   gather_rows       a[r] = x[sorted_rows[r] / top] (zeros for padding): the rows in the tiles' order, optionally times
//                     the pair's weight (where it scales what the expert reads)
//   route_combine     y[t] += sum_k weight[t, k] * part[row of pair t * top + k] in the order of k (weights of 1 where they
//                     scaled the experts' inputs), optionally plus gate[t] * more[t] (the gated expert of every token)
//
// bfloat16 weights in aligned rows run on the tensor cores (grouped_mma_kernel for few rows, decoding, where the weights stream once;
// head_mma_kernel for the heads' matrices), 32-bit inputs with all their bits. The true 32-bit path, a few pairs of 32-bit inputs and
// what is not aligned run on the CUDA cores with 32-bit fused multiply-adds, in three forms: tiles of 16 x 64 outputs, tiles of 64 x 64
// (many rows through the heads' matrices) and the few-row form further down. In the tiled forms an output element is one chain of
// multiply-adds in the order of k over its own row, whichever tile the row landed in; in the few-row form it is the sum of
// a warp's lanes' chains by a fixed tree. (Many rows through the experts' matrices in bfloat16: gi_gemm_tc_grouped.)
#include <cooperative_groups.h>

#include "common.cuh"
#include "device_limit.h"

namespace gi {

constexpr int kGpTM = 16, kGpTN = 64, kGpTK = 32;

struct GroupedArgs {
    const void* a; long long lda; int a_off; int a_gs; int a_div;
    const void* w; long long w_gs; int ldw; long long up_off;     // W[g] = w + g * w_gs, rows of ldw; the up rows start at up_off
    void* out; int out_is_f32; long long ldo; int o_off; int o_gs;
    int N, K, rows, groups;                                       // experts form: the pairs and the experts
    const int* tile_group; const int* sorted_rows; const int* n_tiles;   // experts form (else null)
    int w_constant;                                               // no kernel that may still be running writes w: it may be read before the wait
    int act; float act_limit;                                     // gated: a GateAct code and its limit
    int out_act;                                                  // not gated: a PlainAct code
    // rotated tail (heads form)
    int tail; const float* freq; float amplitude; int tail_interleaved; const int* positions;
    // output gate (heads form): out *= sigmoid(gate[row, gate_off + h * gate_hs + n * gate_ns]), 32-bit (else null): a value
    // per output (strides N, 1) or per head (1, 0)
    const float* gate; long long ldg; int gate_off, gate_hs, gate_ns;
    // experts form: what the products of a pair are multiplied with before the activation (the pair's weight when it scales
    // what its expert reads), 32-bit by pair (else null)
    const float* scales;
};

__device__ __forceinline__ float gp_gate_value(const GroupedArgs& p, int r, int g, int n) {
    return p.gate[static_cast<size_t>(r) * p.ldg + p.gate_off + static_cast<size_t>(g) * p.gate_hs + static_cast<size_t>(n) * p.gate_ns];
}

// Pair pr of the rotated tail of row r, head g.
template <typename TA>
__device__ __forceinline__ void gp_rotate_pair(const GroupedArgs& p, const TA* tail_in, int r, int g, int pr) {
    float sn, cs;
    sincosf(static_cast<float>(p.positions[r]) * p.freq[pr], &sn, &cs);
    sn *= p.amplitude; cs *= p.amplitude;
    const int iu = p.tail_interleaved ? 2 * pr : pr, iv = p.tail_interleaved ? 2 * pr + 1 : pr + p.tail / 2;
    const float u = to_float(tail_in[iu]), v = to_float(tail_in[iv]);
    const size_t o = static_cast<size_t>(r) * p.ldo + p.o_off + static_cast<size_t>(g) * p.o_gs + p.N;
    const float ru = u * cs - v * sn, rv = v * cs + u * sn;
    if (p.out_is_f32) { static_cast<float*>(p.out)[o + iu] = ru; static_cast<float*>(p.out)[o + iv] = rv; }
    else { static_cast<__nv_bfloat16*>(p.out)[o + iu] = __float2bfloat16_rn(ru); static_cast<__nv_bfloat16*>(p.out)[o + iv] = __float2bfloat16_rn(rv); }
}

// The element-wise sigmoid gate of the heads form, on output n of head g of row r.
__device__ __forceinline__ float gp_gated(const GroupedArgs& p, float v, int r, int g, int n) {
    if (p.gate == nullptr) return v;
    return v * sigmoid_f(gp_gate_value(p, r, g, n));
}

template <typename TA, typename TW, bool GATED>
__global__ void __launch_bounds__(128)
grouped_product_kernel(const GroupedArgs p) {
    pdl_prologue();
    constexpr int U = GATED ? 1 : 0;
    __shared__ float s_a[kGpTK][kGpTM + 1];
    __shared__ __align__(16) float s_w[U + 1][kGpTK][kGpTN + 4];
    __shared__ int s_row[kGpTM];

    const int tid = threadIdx.x;
    int g, row0 = 0;
    if (p.tile_group) {
        if (static_cast<int>(blockIdx.x) >= *p.n_tiles) return;
        g = p.tile_group[blockIdx.x];
        if (tid < kGpTM) s_row[tid] = p.sorted_rows[blockIdx.x * kGpTM + tid];
    } else {
        g = blockIdx.x % p.groups;
        row0 = (blockIdx.x / p.groups) * kGpTM;
        if (tid < kGpTM) s_row[tid] = row0 + tid < p.rows ? row0 + tid : -1;
    }
    __syncthreads();
    const int n0 = blockIdx.y * kGpTN;
    const TA* A = static_cast<const TA*>(p.a);
    const TW* W = static_cast<const TW*>(p.w) + static_cast<size_t>(g) * p.w_gs;

    // rotated tail: only the blocks of the first tile of outputs do it
    if (p.tail > 0 && blockIdx.y == 0) {
        for (int i = tid; i < kGpTM * (p.tail / 2); i += 128) {
            const int m = i / (p.tail / 2), pr = i % (p.tail / 2);
            const int r = s_row[m];
            if (r < 0) continue;
            gp_rotate_pair(p, A + static_cast<size_t>(r) * p.lda + p.a_off + static_cast<size_t>(g) * p.a_gs + p.K, r, g, pr);
        }
    }

    const int tm = (tid >> 4) * 2, tn = (tid & 15) * 4;
    float acc[2][4] = {}, acc_up[U + 1][4] = {};
    for (int k0 = 0; k0 < p.K; k0 += kGpTK) {
        // rows of a: 16 x 32 values
        for (int i = tid; i < kGpTM * kGpTK; i += 128) {
            const int m = i / kGpTK, k = i % kGpTK;
            const int r = s_row[m];
            float v = 0.f;
            if (r >= 0 && k0 + k < p.K)
                v = to_float(A[static_cast<size_t>(r / p.a_div) * p.lda + p.a_off + static_cast<size_t>(g) * p.a_gs + k0 + k]);
            s_a[k][m] = v;
        }
        // rows of W: 64 x 32 values (and the up rows)
        for (int i = tid; i < kGpTN * kGpTK; i += 128) {
            const int n = i / kGpTK, k = i % kGpTK;
            const bool in = n0 + n < p.N && k0 + k < p.K;
            const size_t off = static_cast<size_t>(n0 + n) * p.ldw + k0 + k;
            s_w[0][k][n] = in ? to_float(W[off]) : 0.f;
            if (GATED) s_w[U][k][n] = in ? to_float(W[p.up_off + off]) : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < kGpTK; ++k) {
            const float a0 = s_a[k][tm], a1 = s_a[k][tm + 1];
            const float4 w4 = *reinterpret_cast<const float4*>(&s_w[0][k][tn]);
            acc[0][0] = fmaf(a0, w4.x, acc[0][0]); acc[0][1] = fmaf(a0, w4.y, acc[0][1]);
            acc[0][2] = fmaf(a0, w4.z, acc[0][2]); acc[0][3] = fmaf(a0, w4.w, acc[0][3]);
            acc[1][0] = fmaf(a1, w4.x, acc[1][0]); acc[1][1] = fmaf(a1, w4.y, acc[1][1]);
            acc[1][2] = fmaf(a1, w4.z, acc[1][2]); acc[1][3] = fmaf(a1, w4.w, acc[1][3]);
            if (GATED) {
                const float4 u4 = *reinterpret_cast<const float4*>(&s_w[U][k][tn]);
                acc_up[0][0] = fmaf(a0, u4.x, acc_up[0][0]); acc_up[0][1] = fmaf(a0, u4.y, acc_up[0][1]);
                acc_up[0][2] = fmaf(a0, u4.z, acc_up[0][2]); acc_up[0][3] = fmaf(a0, u4.w, acc_up[0][3]);
                acc_up[U][0] = fmaf(a1, u4.x, acc_up[U][0]); acc_up[U][1] = fmaf(a1, u4.y, acc_up[U][1]);
                acc_up[U][2] = fmaf(a1, u4.z, acc_up[U][2]); acc_up[U][3] = fmaf(a1, u4.w, acc_up[U][3]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = s_row[tm + i];
        if (r < 0) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tn + j;
            if (n >= p.N) continue;
            const float sc = p.scales ? p.scales[r] : 1.f;
            float v = sc * acc[i][j];
            if (GATED) v = gated_value(v, sc * acc_up[U * i][j], p.act, p.act_limit);
            else v = plain_value(v, p.out_act);
            v = gp_gated(p, v, r, g, n);
            const size_t o = static_cast<size_t>(r) * p.ldo + p.o_off + static_cast<size_t>(g) * p.o_gs + n;
            if (p.out_is_f32) static_cast<float*>(p.out)[o] = v;
            else static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v);
        }
    }
}

// The same products for few rows (decoding), with 32-bit weights or, very few rows (few_on_cuda_cores), bfloat16 ones: the weights are
// what takes the time. A warp streams four or eight output rows of a group's matrix (gated: and their up rows) through a ring in shared memory, 512 bytes of each a step, by asynchronous copies
// of 16 bytes; every lane copies exactly the pieces that it multiplies itself, so the ring needs no barrier, and 48 KB or more
// are in flight per block whatever the warps are doing. Each step's pieces are multiplied with up to eight rows of the tile, read
// through the cache; more rows stream the weights again, from L2. An output element is the sum of its lanes' partial sums (lane l takes
// the pieces l, l + 32, ...), added by a fixed xor tree: it depends on its own row only.
constexpr int kGrWarps = 4;
constexpr int kGrFew = 8;             // rows of a tile that are multiplied with a piece of the weights while it is in registers

template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// The few-row forms: group and rows of tile x; lane i gets the i-th of its rows. Returns how many there are. HALVES: tile x is half of a
// tile, its first eight rows or the others.
template <bool HALVES = false>
__device__ __forceinline__ int gm_tile(const GroupedArgs& p, int x, int lane, int& g, int& row) {
    int r = -1, half = 0;
    if (HALVES) { half = x & 1; x >>= 1; }
    if (p.tile_group) {
        g = p.tile_group[x];
        if (lane < kGpTM) r = p.sorted_rows[x * kGpTM + lane];
    } else {
        g = x % p.groups;
        if (lane < kGpTM) r = x / p.groups * kGpTM + lane;
        if (r >= p.rows) r = -1;
    }
    const unsigned some = __ballot_sync(0xffffffffu, r >= 0);       // the empty places left out
    row = r;
    if (some & (some + 1)) row = __shfl_sync(0xffffffffu, r, __fns(some, 0, lane + 1) & 31);
    if (HALVES) {
        if (half) row = __shfl_sync(0xffffffffu, row, (lane + 8) & 31);
        return max(0, min(8, __popc(some) - 8 * half));
    }
    return __popc(some);
}

// Four neighbouring weights of a lane's piece in shared memory, as 32-bit values.
__device__ __forceinline__ float4 piece4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 piece4(const __nv_bfloat16* p) { return load4<__nv_bfloat16>(p); }

// The few-row form's units of work, taken by the grid's warps in turn: (tile, four or eight output rows), and for a tile of more than
// kGrFew rows a second pass over the same weights. A warp's ring runs on from unit to unit.
// ROWS: output rows of a unit, 4 or, not gated, 8.
template <typename TA, typename TW, bool GATED, int ROWS>
struct RowsStream {
    static constexpr int kPiece = 16 / sizeof(TW);       // values per step of a lane: the weights' 16 bytes
    static constexpr int kW = GATED ? 2 * ROWS : ROWS;   // rows of weights that it streams (gated: and the up rows)
    static constexpr int kBlocks = ROWS == 8 ? 2 : 3;    // blocks an SM: 8 rows need more than the 168 registers of three
    static constexpr int kSmem = (ROWS == 8 ? 96 : 64) * 1024;
    static constexpr int kStages = kSmem / (kGrWarps * kW * 512);

    const GroupedArgs& p;
    uint4* ring;                 // this lane's place in the warp's first stage
    int lane, units, per_tile, stride, pieces, steps;
    // the step that is requested next
    int unit, pass, passes, step, issued = 0;
    const TW* wrow;              // the unit's first row of weights; `last`: the last that there is
    int last;

    __device__ __forceinline__ void seek() {
        for (; unit < units; unit += stride) {
            int g, row;
            passes = (gm_tile(p, unit / per_tile, lane, g, row) + kGrFew - 1) / kGrFew;
            if (passes == 0) continue;
            const TW* W = static_cast<const TW*>(p.w) + static_cast<size_t>(g) * p.w_gs;
            const int n_first = unit % per_tile * ROWS;
            wrow = W + static_cast<size_t>(n_first) * p.ldw;
            last = p.N - 1 - n_first;
            pass = step = 0;
            return;
        }
    }
    __device__ __forceinline__ void request() {
        if (unit < units) {
            const int c = step * 32 + lane;
            if (c < pieces) {
                const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(ring + (issued % kStages) * (kW * 32)));
#pragma unroll
                for (int r = 0; r < kW; ++r) {
                    const TW* src = wrow + static_cast<long long>(min(r % ROWS, last)) * p.ldw + (r >= ROWS ? p.up_off : 0) + c * kPiece;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + r * 512), "l"(src) : "memory");
                }
            }
            if (++step == steps) {
                step = 0;
                if (++pass == passes) { unit += stride; seek(); }
            }
        }
        ++issued;
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
};

// MR rows of a tile (m_here of them are real, the last is repeated) against the output rows from n_first on. ``row``:
// lane i has the tile's i-th row; ``done``: steps of the warp's ring taken so far. With 8 output rows up to two rows' inputs are
// asked for a step ahead.
template <int MR, typename TA, typename TW, bool GATED, int ROWS>
__device__ __forceinline__ void grouped_rows_unit(RowsStream<TA, TW, GATED, ROWS>& q, int g, int row, int n_first, int m0, int m_here, int& done) {
    const GroupedArgs& p = q.p;
    using Stream = RowsStream<TA, TW, GATED, ROWS>;
    constexpr int kW = Stream::kW, kStages = Stream::kStages, kPiece = Stream::kPiece;
    constexpr bool kAhead = ROWS == 8 && MR <= 2;
    const TA* A = static_cast<const TA*>(p.a) + p.a_off + static_cast<size_t>(g) * p.a_gs;
    const TA* arow[MR];
#pragma unroll
    for (int i = 0; i < MR; ++i) arow[i] = A + static_cast<size_t>(__shfl_sync(0xffffffffu, row, m0 + min(i, m_here - 1)) / p.a_div) * p.lda;
    // the output gate's values of the unit's outputs, (row of weights, row of the tile) by lane, asked for before the weights arrive
    constexpr int kGates = ROWS * kGrFew / 32;
    float gate_z[kGates];
    if (p.gate != nullptr) {
#pragma unroll
        for (int u = 0; u < kGates; ++u) {
            const int gr = (q.lane + 32 * u) / kGrFew, gi_ = q.lane % kGrFew;
            const int gate_row = __shfl_sync(0xffffffffu, row, m0 + min(gi_, m_here - 1));
            gate_z[u] = (gi_ < m_here && n_first + gr < p.N) ? gp_gate_value(p, gate_row, g, n_first + gr) : 0.f;
        }
    }
    float acc[kW][MR];
#pragma unroll
    for (int r = 0; r < kW; ++r)
#pragma unroll
        for (int i = 0; i < MR; ++i) acc[r][i] = 0.f;
    float4 av[MR][kAhead ? kPiece / 4 : 1], next[kAhead ? MR : 1][kPiece / 4];
    auto fetch = [&](float4 (&dst)[kPiece / 4], const TA* src, int at) {
#pragma unroll
        for (int h = 0; h < kPiece / 4; ++h) dst[h] = load4<TA>(src + at * kPiece + 4 * h);
    };
    if constexpr (kAhead) {
        if (q.lane < q.pieces)
#pragma unroll
            for (int i = 0; i < MR; ++i) fetch(av[i], arow[i], q.lane);
    }
    for (int step = 0; step < q.steps; ++step, ++done) {
        const int c = step * 32 + q.lane;
        if constexpr (kAhead) {
            if (c + 32 < q.pieces)
#pragma unroll
                for (int i = 0; i < MR; ++i) fetch(next[i], arow[i], c + 32);
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        if (c < q.pieces) {
            const uint4* stage = q.ring + (done % kStages) * (kW * 32);
#pragma unroll
            for (int h = 0; h < kPiece / 4; ++h) {
                if constexpr (!kAhead) {
#pragma unroll
                    for (int i = 0; i < MR; ++i) av[i][0] = load4<TA>(arow[i] + c * kPiece + 4 * h);
                }
#pragma unroll
                for (int r = 0; r < kW; ++r) {
                    const float4 w = piece4(reinterpret_cast<const TW*>(stage + r * 32) + 4 * h);
#pragma unroll
                    for (int i = 0; i < MR; ++i) {
                        const float4 x = av[i][kAhead ? h : 0];
                        acc[r][i] = fmaf(x.x, w.x, acc[r][i]); acc[r][i] = fmaf(x.y, w.y, acc[r][i]);
                        acc[r][i] = fmaf(x.z, w.z, acc[r][i]); acc[r][i] = fmaf(x.w, w.w, acc[r][i]);
                    }
                }
            }
        }
        if constexpr (kAhead) {
#pragma unroll
            for (int i = 0; i < MR; ++i)
#pragma unroll
                for (int h = 0; h < kPiece / 4; ++h) av[i][h] = next[i][h];
        }
        q.request();                                  // into the stage read a step ago, by this lane alone
    }
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        if (i >= m_here) break;
        const int out_row = __shfl_sync(0xffffffffu, row, m0 + i);
        const float sc = p.scales ? p.scales[out_row] : 1.f;
        float mine = 0.f;                             // lane r ends up with output row r
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            float v = sc * warp_sum(acc[r][i]);
            if (GATED) v = gated_value(v, sc * warp_sum(acc[GATED ? r + ROWS : 0][i]), p.act, p.act_limit);
            else v = plain_value(v, p.out_act);
            if (p.gate != nullptr) v *= 1.0f / (1.0f + expf(-__shfl_sync(0xffffffffu, gate_z[r * kGrFew / 32], (r * kGrFew + i) % 32)));
            if (q.lane == r) mine = v;
        }
        if (q.lane < ROWS && n_first + q.lane < p.N) {
            const size_t o = static_cast<size_t>(out_row) * p.ldo + p.o_off + static_cast<size_t>(g) * p.o_gs + n_first + q.lane;
            if (p.out_is_f32) static_cast<float*>(p.out)[o] = mine;
            else static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(mine);
        }
    }
}

// tiles: how many there are (experts form: at most; the number is read on the device)
template <typename TA, typename TW, bool GATED, int ROWS>
__global__ void __launch_bounds__(kGrWarps * 32, (RowsStream<TA, TW, GATED, ROWS>::kBlocks))
grouped_rows_kernel(const GroupedArgs p, int tiles) {
    extern __shared__ uint4 s_ring[];
    pdl_prologue();
    using Stream = RowsStream<TA, TW, GATED, ROWS>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Stream q{p};
    q.ring = s_ring + warp * (Stream::kStages * Stream::kW * 32) + lane;
    q.lane = lane;
    q.per_tile = (p.N + ROWS - 1) / ROWS;
    q.units = (p.tile_group ? *p.n_tiles : tiles) * q.per_tile;
    q.stride = gridDim.x * kGrWarps;
    q.pieces = p.K / Stream::kPiece;
    q.steps = (q.pieces + 31) / 32;
    const int first = blockIdx.x * kGrWarps + warp;
    q.unit = first;
    q.seek();
    for (int i = 0; i < Stream::kStages - 1; ++i) q.request();
    int done = 0, x = -1, g = 0, row = -1, m_count = 0;
    for (int unit = first; unit < q.units; unit += q.stride) {
        if (unit / q.per_tile != x) { x = unit / q.per_tile; m_count = gm_tile(p, x, lane, g, row); }
        const int n_first = unit % q.per_tile * ROWS;
        for (int m0 = 0; m0 < m_count; m0 += kGrFew) {
            const int m_here = min(kGrFew, m_count - m0);
            if (m_here == 1) grouped_rows_unit<1>(q, g, row, n_first, m0, m_here, done);
            else if (m_here == 2) grouped_rows_unit<2>(q, g, row, n_first, m0, m_here, done);
            else if (m_here <= 4) grouped_rows_unit<4>(q, g, row, n_first, m0, m_here, done);
            else grouped_rows_unit<8>(q, g, row, n_first, m0, m_here, done);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The few-row form of bfloat16 weights, on the tensor cores (mma.sync m16n8k16: tcgen05 would want the rows of 64 or 128 outputs in one
// tile, too coarse to share a few experts' matrices evenly among 148 SMs, and multiplies a few tokens no faster than memory brings
// the weights). A unit is MT x 16 rows of weights (gated: eight gate rows and the eight up rows of the same outputs) over all of K,
// the work of a block; its eight warps share K in blocks of 64 values, dealt in turn, each with a ring of cp.async pieces of its own
// that runs on from unit to unit. The ring's lane mapping is the fragments': a lane's 16 bytes are eight neighbouring k of one row, its
// share of two products whose k are taken in an order of their own (the same for weights and inputs), so nothing is rearranged and no
// lane reads what another one copied. Inputs are asked for a step ahead, in registers. Per unit the warps' sums meet once in shared
// memory, where they are added in pairs.
// bfloat16 inputs are multiplied as they are, up to sixteen rows of a tile with a piece of the weights; a 32-bit input is cut into three
// bfloat16 values whose sum it is (24 bits of mantissa in three times eight; a part below 2^-126 may count as zero), so its products are
// exact as well. The cutting costs more instructions than the products, so its units are of 32 rows, and of eight rows of a tile
// (a tile with more is two, whose weights meet in L2). The tensor cores cut the sums that they carry on, so each
// product of sixteen k starts from zero and is added by the CUDA cores, rounded (the second and third parts' sums are carried on: a
// cut there is 2^-8 of one in the first). An output element depends on its own row only, not on the row's place in a tile.
// Measured, sixteen pairs of eight experts, on the CUDA cores -> here: gated 2 x 4,096 outputs of 2,048 bfloat16 inputs 62.6 -> 48.6 us
// when they spread evenly (41.6 of bytes), 90 -> 46 in a token's step; 2,048 outputs of 4,096 32-bit inputs there 54 -> 30. Errors against 64 bits:
// 1.25e-7 of the outputs' size (1.29e-7 before) and 0.87e-7 (2.1e-7 before).
constexpr int kGmWarps = 8, kGmSub = 2;                      // sub-blocks of 32 k per step of a warp's ring
constexpr int kGmBlocks = 2;                                 // an SM
template <typename TA> struct GmShape;
template <> struct GmShape<__nv_bfloat16> { static constexpr int MT = 1, NT = 2, kStages = 6; };
template <> struct GmShape<float> { static constexpr int MT = 2, NT = 1, kStages = 3; };
template <typename TA> struct GmSizes {                      // bytes
    static constexpr int kStage = kGmSub * GmShape<TA>::MT * 1024, kRing = kGmWarps * GmShape<TA>::kStages * kStage;
    static constexpr int kSums = 2 * kGmWarps * 2 * 32 * 16;             // MT x NT fragments of a warp, twice
};

__device__ __forceinline__ void gm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Two products of sixteen k, added up and into a sum of the CUDA cores.
__device__ __forceinline__ void gm_mma_add(float (&c)[4], const uint4& w0, const uint4& w1, const uint32_t (&x)[4]) {
    float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
    gm_mma(d, w0.x, w1.x, w0.y, w1.y, x[0], x[1]);
    gm_mma(e, w0.z, w1.z, w0.w, w1.w, x[2], x[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += d[i] + e[i];
}

// Two 32-bit sums or differences in one instruction.
__device__ __forceinline__ unsigned long long gm_pair(float a, float b) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 gm_split(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ unsigned long long gm_plus(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long gm_minus(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(gm_pair(-1.f, -1.f)), "l"(a));
    return d;
}

// Eight neighbouring values of an input row as they are read (GmInput) and as they are multiplied (GmParts): what they add to the
// sums with eight values of weight rows w0 and w1. An input's second and third parts may be zero, and zero times an infinite weight is
// none, where the input times the weight is infinite: then the first parts' sums alone, which are infinite or none too, are the answer (the parts
// have the input's sign, so what the others add could not change it; of an input below 2^-126 there may be no first part either).
template <typename TA> struct GmParts;
template <typename TA> struct GmInput;
template <> struct GmParts<__nv_bfloat16> {
    uint4 v;
    __device__ __forceinline__ void multiply(float (&c)[4], float (&)[4], const uint4& w0, const uint4& w1) const {
        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
        gm_mma_add(c, w0, w1, x);
    }
};
template <> struct GmInput<__nv_bfloat16> {
    uint4 v;
    __device__ __forceinline__ void zero() { v = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ GmParts<__nv_bfloat16> parts() const { return {v}; }
};
template <> struct GmParts<float> {
    uint32_t top[4], mid[4], low[4];
    __device__ __forceinline__ void multiply(float (&c)[4], float (&rest)[4], const uint4& w0, const uint4& w1) const {
        gm_mma(rest, w0.x, w1.x, w0.y, w1.y, low[0], low[1]);
        gm_mma(rest, w0.z, w1.z, w0.w, w1.w, low[2], low[3]);
        gm_mma(rest, w0.x, w1.x, w0.y, w1.y, mid[0], mid[1]);
        gm_mma(rest, w0.z, w1.z, w0.w, w1.w, mid[2], mid[3]);
        gm_mma_add(c, w0, w1, top);
    }
};
template <> struct GmInput<float> {
    float4 a, b;
    __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load(const float* p) {
        a = *reinterpret_cast<const float4*>(p);
        b = *(reinterpret_cast<const float4*>(p) + 1);
    }
    __device__ __forceinline__ GmParts<float> parts() const {
        const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float top[8], mid[8], low[8];
        auto cut = [](float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); };
        unsigned long long sum = 0ull;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {               // cut, not rounded: each difference is exact
            top[i] = cut(x[i]); top[i + 1] = cut(x[i + 1]);
            const unsigned long long rest = gm_minus(gm_pair(x[i], x[i + 1]), gm_pair(top[i], top[i + 1]));
            const float2 r = gm_split(rest);
            mid[i] = cut(r.x); mid[i + 1] = cut(r.y);
            const unsigned long long last = gm_minus(rest, gm_pair(mid[i], mid[i + 1]));
            const float2 l = gm_split(last);
            low[i] = l.x; low[i + 1] = l.y;
            sum = gm_plus(sum, last);
        }
        const float2 sums = gm_split(sum);
        const float any = sums.x + sums.y;
        if (any != any) {                              // an infinity or none: it alone, its differences are none
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if ((__float_as_uint(x[i]) & 0x7f800000u) == 0x7f800000u) {
                    top[i] = x[i] != x[i] ? __uint_as_float(0x7fc00000u) : x[i];
                    mid[i] = low[i] = 0.f;
                }
        }
        GmParts<float> p;
#pragma unroll
        for (int i = 0; i < 4; ++i) {                  // the upper halves of two values
            p.top[i] = __byte_perm(__float_as_uint(top[2 * i]), __float_as_uint(top[2 * i + 1]), 0x7632);
            p.mid[i] = __byte_perm(__float_as_uint(mid[2 * i]), __float_as_uint(mid[2 * i + 1]), 0x7632);
            p.low[i] = __byte_perm(__float_as_uint(low[2 * i]), __float_as_uint(low[2 * i + 1]), 0x7632);
        }
        return p;
    }
};

// Where a walk through a block's units stands: tile, unit within it, and the tile's group and rows.
template <bool HALVES>
struct GmWalk {
    int x, n, g = 0, row = -1, count = 0;            // x: tile, n: unit of the tile (its outputs start at n * kOut)
    int known = -1;
    // To the first unit from (x, n) on, in strides, whose tile has rows; false: there is none.
    __device__ __forceinline__ bool seek(const GroupedArgs& p, int tiles, int per_tile, int stride, int lane) {
        for (;; n += stride) {
            while (n >= per_tile) { n -= per_tile; ++x; }
            if (x >= tiles) return false;
            if (known != x) { known = x; count = gm_tile<HALVES>(p, x, lane, g, row); }
            if (count > 0) return true;
        }
    }
};

template <typename TA, bool GATED>
__global__ void __launch_bounds__(kGmWarps * 32, kGmBlocks)
grouped_mma_kernel(const GroupedArgs p, int tiles_given) {
    extern __shared__ uint4 s_ring[];
    pdl_prologue();
    constexpr int MT = GmShape<TA>::MT, NT = GmShape<TA>::NT, kStages = GmShape<TA>::kStages, kStage = GmSizes<TA>::kStage;
    constexpr bool kHalves = NT == 1;
    constexpr int kOut = GATED ? 8 * MT : 16 * MT;                  // outputs of a unit
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gr = lane >> 2, kq = (lane & 3) * 8;
    uint4* ring = s_ring + warp * (kStages * kStage / 16) + lane;
    float4* sums = reinterpret_cast<float4*>(s_ring + GmSizes<TA>::kRing / 16);
    const int per_tile = (p.N + kOut - 1) / kOut, stride = gridDim.x;
    const int tiles = (p.tile_group ? *p.n_tiles : tiles_given) * (kHalves ? 2 : 1);
    constexpr int kStepK = kGmSub * 32;
    const int steps = (p.K + kGmWarps * kStepK - 1) / (kGmWarps * kStepK);      // step i of warp w: k from (i * kGmWarps + w) * kStepK on

    // what is requested next: weights. Row gr + 8 r of the unit (r < 2 MT); gated: the up rows are the odd r
    GmWalk<kHalves> rq{static_cast<int>(blockIdx.x) / per_tile, static_cast<int>(blockIdx.x) % per_tile};
    int rq_k = 0;                                                   // of the unit's K, without this warp's and lane's own offset
    const __nv_bfloat16* rq_w[2 * MT];
    bool rq_on = false;
    const int k_mine = warp * kStepK + kq;
    auto seek = [&]() {
        rq_on = rq.seek(p, tiles, per_tile, stride, lane);
        if (!rq_on) return;
        const int n_first = rq.n * kOut, last = p.N - 1 - n_first;
        const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(p.w) + static_cast<size_t>(rq.g) * p.w_gs + static_cast<size_t>(n_first) * p.ldw;
#pragma unroll
        for (int r = 0; r < 2 * MT; ++r)
            rq_w[r] = w + static_cast<long long>(min(gr + 8 * (GATED ? r / 2 : r), last)) * p.ldw + (GATED && (r & 1) ? p.up_off : 0);
        rq_k = 0;
    };
    const unsigned ring_at = static_cast<unsigned>(__cvta_generic_to_shared(ring));
    unsigned rq_at = 0;
    auto request = [&]() {
        if (rq_on) {
#pragma unroll
            for (int j = 0; j < kGmSub; ++j) {
                const int k = rq_k + k_mine + j * 32;
                const int bytes = k < p.K ? 16 : 0, off = k < p.K ? k : 0;      // 0: zeros, nothing is read (K is a multiple of 8)
#pragma unroll
                for (int r = 0; r < 2 * MT; ++r)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring_at + rq_at + (j * 2 * MT + r) * 512), "l"(rq_w[r] + off), "r"(bytes) : "memory");
            }
            rq_k += kGmWarps * kStepK;
            if (rq_k >= p.K) { rq.n += stride; seek(); }
        }
        rq_at = rq_at + kStage == kStages * kStage ? 0 : rq_at + kStage;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // ... and inputs: rows gr (and gr + 8) of the tile of the unit that `in_at` walks to
    GmWalk<kHalves> in_at = rq;
    int in_k = 0;
    bool in_on = false;
    const TA* in_a[NT];
    GmInput<TA> in[NT][kGmSub];
    auto in_seek = [&]() {
        const int before = in_at.known;
        in_on = in_at.seek(p, tiles, per_tile, stride, lane);
        in_k = 0;
        if (!in_on || before == in_at.known) return;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int r = __shfl_sync(0xffffffffu, in_at.row, gr + 8 * t);
            in_a[t] = static_cast<const TA*>(p.a) + static_cast<size_t>(gr + 8 * t < in_at.count ? r / p.a_div : 0) * p.lda + p.a_off + static_cast<size_t>(in_at.g) * p.a_gs;
        }
    };
    auto fetch = [&]() {
        if (!in_on) return;
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int j = 0; j < kGmSub; ++j) {
                const int k = in_k + k_mine + j * 32;
                if (gr + 8 * t < in_at.count && k < p.K) in[t][j].load(in_a[t] + k);
                else in[t][j].zero();
            }
        in_k += kGmWarps * kStepK;
        if (in_k >= p.K) { in_at.n += stride; in_seek(); }
    };

    seek();
    for (int i = 0; i < kStages - 1; ++i) request();
    in_seek();
    fetch();
    GmWalk<kHalves> at{static_cast<int>(blockIdx.x) / per_tile, static_cast<int>(blockIdx.x) % per_tile};
    unsigned got = 0;
    for (int turn = 0; at.seek(p, tiles, per_tile, stride, lane); at.n += stride, ++turn) {
        float acc[kGmSub][MT][NT][4], rest[MT][NT][4];              // (a sum for each sub-block: chains half as long)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[0][m][t][i] = acc[1][m][t][i] = rest[m][t][i] = 0.f;
        for (int step = 0; step < steps; ++step) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            const uint4* stage = ring + got / 16;
            got = got + kStage == kStages * kStage ? 0 : got + kStage;
#pragma unroll
            for (int j = 0; j < kGmSub; ++j)
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    if (t > 0 && at.count <= 8) break;
                    const GmParts<TA> x = in[t][j].parts();
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const uint4 w0 = stage[(j * 2 * MT + 2 * m) * 32], w1 = stage[(j * 2 * MT + 2 * m + 1) * 32];
                        x.multiply(acc[j][m][t], rest[m][t], w0, w1);
                    }
                }
            fetch();
            request();                                              // into the stage read a step ago, by this lane alone
        }
        float4* mine = sums + (turn & 1) * (kGmWarps * 2 * 32) + lane;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < NT; ++t)
                if (8 * t < at.count) {
                    float v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        v[i] = acc[0][m][t][i] + (acc[1][m][t][i] + rest[m][t][i]);
                        if (sizeof(TA) == 4 && v[i] != v[i]) v[i] = acc[0][m][t][i] + acc[1][m][t][i];      // (GmParts: a part that is zero and an infinite weight)
                    }
                    mine[(warp * 2 + m * NT + t) * 32] = make_float4(v[0], v[1], v[2], v[3]);
                }
        __syncthreads();         // (this half is written again two units on, behind the next barrier, which every reader of it meets later)
        // warps 0 .. 3, warp w: fragment w / 2 (of rows of weights, or of the tile's rows), of the tile's rows 2 (lane % 4) + w % 2 of eight
        const int f = warp >> 1, t = NT == 2 ? f : 0, m_rows = NT == 2 ? 0 : f * (GATED ? 8 : 16), m = 8 * t + (lane & 3) * 2 + (warp & 1);
        if (warp < 4 && 8 * t < at.count) {
            const int out_row = __shfl_sync(0xffffffffu, at.row, m);
            if (m < at.count) {
                float u0[kGmWarps], u1[kGmWarps];
#pragma unroll
                for (int w = 0; w < kGmWarps; ++w) {
                    const float4 part = mine[(w * 2 + f) * 32];
                    u0[w] = warp & 1 ? part.y : part.x;
                    u1[w] = warp & 1 ? part.w : part.z;
                }
                float v0 = ((u0[0] + u0[1]) + (u0[2] + u0[3])) + ((u0[4] + u0[5]) + (u0[6] + u0[7]));
                float v1 = ((u1[0] + u1[1]) + (u1[2] + u1[3])) + ((u1[4] + u1[5]) + (u1[6] + u1[7]));
                const int n_first = at.n * kOut + m_rows;
                if (p.scales) { const float sc = p.scales[out_row]; v0 *= sc; v1 *= sc; }
                auto store = [&](int n, float value) {
                    if (n >= p.N) return;
                    value = gp_gated(p, value, out_row, at.g, n);
                    const size_t o = static_cast<size_t>(out_row) * p.ldo + p.o_off + static_cast<size_t>(at.g) * p.o_gs + n;
                    if (p.out_is_f32) static_cast<float*>(p.out)[o] = value;
                    else static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(value);
                };
                if (GATED) {
                    store(n_first + gr, gated_value(v0, v1, p.act, p.act_limit));
                } else {
                    store(n_first + gr, plain_value(v0, p.out_act));
                    store(n_first + gr + 8, plain_value(v1, p.out_act));
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The heads form of bfloat16 weights: every row count with a rotated tail, and without one where the rows are more than the few-row form
// takes. A warp has MT x 16 outputs of NT x 8 rows, its operands straight from memory in the fragments' layout (as in the few-row
// form), a step of 32 k ahead, the first weights asked for before the wait where they are constant. kFew: the block's four
// warps lie along the outputs (few rows: the weights are what is read), else along the rows. A sum goes through K in the same
// order with the same products in either shape: a token's result is the same to the bit whatever else is in the step. Measured, 16 heads,
// on the CUDA cores -> here: 512 to 64, 1,273 rows 91 -> 34 us; 64 to 512 with a tail, 8 rows 14.6 -> 2.7, 1,273 rows 51 -> 43; 128 to 1,024
// 28 -> 4.7 and 173 -> 110.
template <typename TA, int MT, int NT, bool kFew>
__global__ void __launch_bounds__(128)
head_mma_kernel(const GroupedArgs p) {
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gr = lane >> 2, kq = (lane & 3) * 8, g = blockIdx.x;
    const int n0 = (kFew ? blockIdx.y * 4 + warp : blockIdx.y) * (16 * MT);
    const int row0 = (kFew ? blockIdx.z : blockIdx.z * 4 + warp) * (8 * NT), rows = min(8 * NT, p.rows - row0);
    if (rows <= 0) return;
    const TA* A = static_cast<const TA*>(p.a) + static_cast<size_t>(row0) * p.lda + p.a_off + static_cast<size_t>(g) * p.a_gs;
    const __nv_bfloat16* W = static_cast<const __nv_bfloat16*>(p.w) + static_cast<size_t>(g) * p.w_gs;
    uint4 w[MT][2], w_next[MT][2];
    GmInput<TA> in[NT], in_next[NT];
    auto weights = [&](uint4 (&dst)[MT][2], int k0) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                dst[i][half] = k0 + kq < p.K ? *reinterpret_cast<const uint4*>(W + static_cast<size_t>(min(n0 + 16 * i + 8 * half + gr, p.N - 1)) * p.ldw + k0 + kq)
                                             : make_uint4(0, 0, 0, 0);
    };
    auto inputs = [&](GmInput<TA> (&dst)[NT], int k0) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            if (8 * t + gr < rows && k0 + kq < p.K) dst[t].load(A + static_cast<size_t>(8 * t + gr) * p.lda + k0 + kq);
            else dst[t].zero();
        }
    };
    if (!p.w_constant) pdl_wait();
    if (n0 < p.N) weights(w, 0);
    pdl_wait();
    if (p.tail > 0 && blockIdx.y == 0) {                // the rotated tail, by the blocks of the first outputs
        const int first = kFew ? threadIdx.x : lane, step = kFew ? 128 : 32, half = p.tail / 2;
        for (int i = first; i < rows * half; i += step)
            gp_rotate_pair(p, A + static_cast<size_t>(i / half) * p.lda + p.K, row0 + i / half, g, i % half);
    }
    if (n0 >= p.N) return;
    float acc[MT][NT][4], rest[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][t][e] = rest[i][t][e] = 0.f;
    inputs(in, 0);
    for (int k0 = 0; k0 < p.K; k0 += 32) {
        if (k0 + 32 < p.K) { weights(w_next, k0 + 32); inputs(in_next, k0 + 32); }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const GmParts<TA> x = in[t].parts();
#pragma unroll
            for (int i = 0; i < MT; ++i) x.multiply(acc[i][t], rest[i][t], w[i][0], w[i][1]);
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) { w[i][0] = w_next[i][0]; w[i][1] = w_next[i][1]; }
#pragma unroll
        for (int t = 0; t < NT; ++t) in[t] = in_next[t];
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int m = 8 * t + (lane & 3) * 2 + (e & 1), n = n0 + 16 * i + 8 * (e >> 1) + gr;
                if (m >= rows || n >= p.N) continue;
                float v = acc[i][t][e] + rest[i][t][e];
                if (sizeof(TA) == 4 && v != v) v = acc[i][t][e];                 // (GmParts: a part that is zero and an infinite weight)
                v = gp_gated(p, v, row0 + m, g, n);
                const size_t o = static_cast<size_t>(row0 + m) * p.ldo + p.o_off + static_cast<size_t>(g) * p.o_gs + n;
                if (p.out_is_f32) static_cast<float*>(p.out)[o] = v;
                else static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v);
            }
}

// The heads form of 32-bit weights with a rotated tail for up to four rows: short inputs and many outputs, where a tile's rounds through shared
// memory and its sixteen rows cost more than its multiply-adds, and the few-row form spends its time on its sums. A thread has one
// output of every row, its weights in registers (asked for before the wait where they are constant). The sum is one
// chain in the order of k, as in the tiles of 16 and of 64: a token's result is the same to the bit whatever else is in the step.
constexpr int kGcRows = 4, kGcCols = 64, kGcK = 64;

__global__ void __launch_bounds__(kGcCols)
head_product_few_kernel(const GroupedArgs p) {
    pdl_launch_dependents();
    constexpr int kPiece = 4, kPieces = kGcK / kPiece;
    __shared__ __align__(16) float s_a[kGcK][kGcRows];
    const int tid = threadIdx.x, g = blockIdx.x, n = blockIdx.y * kGcCols + tid;
    const float* A = static_cast<const float*>(p.a) + p.a_off + static_cast<size_t>(g) * p.a_gs;
    const float* wrow = static_cast<const float*>(p.w) + static_cast<size_t>(g) * p.w_gs + static_cast<size_t>(min(n, p.N - 1)) * p.ldw;
    uint4 wv[kPieces];
    auto request = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int k = k0 + i * kPiece;                 // (K is a multiple of a piece)
            wv[i] = k < p.K ? *reinterpret_cast<const uint4*>(wrow + k) : make_uint4(0, 0, 0, 0);
        }
    };
    if (!p.w_constant) pdl_wait();
    request(0);
    pdl_wait();
    if (blockIdx.y == 0)
        for (int i = tid; i < p.rows * (p.tail / 2); i += kGcCols) {
            const int r = i / (p.tail / 2);
            gp_rotate_pair(p, A + static_cast<size_t>(r) * p.lda + p.K, r, g, i % (p.tail / 2));
        }
    float acc[kGcRows] = {};
    for (int k0 = 0; k0 < p.K; k0 += kGcK) {
        __syncthreads();
        for (int i = tid; i < kGcK * kGcRows; i += kGcCols) {
            const int m = i / kGcK, k = i % kGcK;
            s_a[k][m] = m < p.rows && k0 + k < p.K ? to_float(A[static_cast<size_t>(m) * p.lda + k0 + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const float w[kPiece] = {__uint_as_float(wv[i].x), __uint_as_float(wv[i].y), __uint_as_float(wv[i].z), __uint_as_float(wv[i].w)};
#pragma unroll
            for (int j = 0; j < kPiece; ++j) {
                const float4 a = *reinterpret_cast<const float4*>(s_a[i * kPiece + j]);
                acc[0] = fmaf(a.x, w[j], acc[0]); acc[1] = fmaf(a.y, w[j], acc[1]);
                acc[2] = fmaf(a.z, w[j], acc[2]); acc[3] = fmaf(a.w, w[j], acc[3]);
            }
        }
        if (k0 + kGcK < p.K) request(k0 + kGcK);
    }
    if (n >= p.N) return;
#pragma unroll
    for (int r = 0; r < kGcRows; ++r) {
        if (r >= p.rows) break;
        const float v = gp_gated(p, acc[r], r, g, n);
        const size_t o = static_cast<size_t>(r) * p.ldo + p.o_off + static_cast<size_t>(g) * p.o_gs + n;
        if (p.out_is_f32) static_cast<float*>(p.out)[o] = v;
        else static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v);
    }
}

// The heads form for many rows (prompt portions): tiles of 64 rows x 64 outputs, a thread 4 x 4 of them, so that two
// 16-byte reads of shared memory feed sixteen multiply-adds. Inputs 32-bit or bfloat16, weights likewise; rows of four
// values must be aligned (the caller checks). An output element is one chain of multiply-adds in the order of k.
constexpr int kG64 = 64, kG64K = 16;

template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
head_product64_kernel(const GroupedArgs p) {
    pdl_prologue();
    __shared__ __align__(16) float s_a[kG64K][kG64 + 4];
    __shared__ __align__(16) float s_w[kG64K][kG64 + 4];
    const int tid = threadIdx.x;
    const int g = blockIdx.x % p.groups;
    const int row0 = (blockIdx.x / p.groups) * kG64;
    const int n0 = blockIdx.y * kG64;
    const TA* A = static_cast<const TA*>(p.a) + p.a_off + static_cast<size_t>(g) * p.a_gs;
    const TW* W = static_cast<const TW*>(p.w) + static_cast<size_t>(g) * p.w_gs;

    if (p.tail > 0 && blockIdx.y == 0) {            // the rotated tail, by the blocks of the first tile of outputs
        for (int i = tid; i < kG64 * (p.tail / 2); i += 256) {
            const int m = i / (p.tail / 2), pr = i % (p.tail / 2);
            const int r = row0 + m;
            if (r >= p.rows) continue;
            gp_rotate_pair(p, A + static_cast<size_t>(r) * p.lda + p.K, r, g, pr);
        }
    }

    const int lr = tid >> 2, lk = (tid & 3) * 4;             // what this thread brings in: row (or output) lr, values lk..lk+3
    const int ty = (tid >> 4) * 4, tx = (tid & 15) * 4;      // its 4 x 4 outputs
    float acc[4][4] = {};
    for (int k0 = 0; k0 < p.K; k0 += kG64K) {
        float4 av = make_float4(0.f, 0.f, 0.f, 0.f), wv = av;
        if (row0 + lr < p.rows && k0 + lk < p.K) av = load4<TA>(A + static_cast<size_t>(row0 + lr) * p.lda + k0 + lk);
        if (n0 + lr < p.N && k0 + lk < p.K) wv = load4<TW>(W + static_cast<size_t>(n0 + lr) * p.ldw + k0 + lk);
        __syncthreads();                                      // the tile before is done with
        s_a[lk][lr] = av.x; s_a[lk + 1][lr] = av.y; s_a[lk + 2][lr] = av.z; s_a[lk + 3][lr] = av.w;
        s_w[lk][lr] = wv.x; s_w[lk + 1][lr] = wv.y; s_w[lk + 2][lr] = wv.z; s_w[lk + 3][lr] = wv.w;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kG64K; ++k) {
            const float4 a4 = *reinterpret_cast<const float4*>(&s_a[k][ty]);
            const float4 w4 = *reinterpret_cast<const float4*>(&s_w[k][tx]);
            const float ar[4] = {a4.x, a4.y, a4.z, a4.w}, wr[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], wr[j], acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty + i;
        if (r >= p.rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + j;
            if (n >= p.N) continue;
            const size_t o = static_cast<size_t>(r) * p.ldo + p.o_off + static_cast<size_t>(g) * p.o_gs + n;
            const float v = gp_gated(p, acc[i][j], r, g, n);
            if (p.out_is_f32) static_cast<float*>(p.out)[o] = v;
            else static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v);
        }
    }
}

// ------------------------------------------------------------------------------------------------ routing
constexpr int kRouteMaxExperts = 1024;

// Where the pairs go: tiles of tile_rows rows per expert, in the order of the experts.
struct RouteAlign {
    int* ids; int n_pairs, E;                      // (the fused router writes the ids through this pointer too)
    int* sorted_rows; int* tile_group; int* n_tiles; int max_tiles, tile_rows; int* pair_row;
};
// One block: counts per expert, then tiles per expert in expert order. `empty`: the places hold -1 already.
__device__ __forceinline__ void route_align_block(const RouteAlign& p, int* s_count, int* s_start, bool empty) {
    const int tid = threadIdx.x, threads = blockDim.x;
    for (int e = tid; e < p.E; e += threads) s_count[e] = 0;
    if (!empty) for (int i = tid; i < p.max_tiles * p.tile_rows; i += threads) p.sorted_rows[i] = -1;
    __syncthreads();
    for (int i = tid; i < p.n_pairs; i += threads) atomicAdd(&s_count[p.ids[i]], 1);
    __syncthreads();
    if (tid == 0) {
        int tiles = 0;
        for (int e = 0; e < p.E; ++e) {
            s_start[e] = tiles * p.tile_rows;
            const int n = (s_count[e] + p.tile_rows - 1) / p.tile_rows;
            for (int i = 0; i < n; ++i) p.tile_group[tiles + i] = e;
            tiles += n;
        }
        *p.n_tiles = tiles;
    }
    __syncthreads();
    // a pair takes the next free row of its expert (which row does not matter: an output element is computed from
    // its own row alone, in the same order of operations in every row of a tile)
    for (int i = tid; i < p.n_pairs; i += threads) {
        const int row = atomicAdd(&s_start[p.ids[i]], 1);
        p.sorted_rows[row] = i;
        if (p.pair_row) p.pair_row[i] = row;
    }
}
__global__ void __launch_bounds__(1024)
route_align_kernel(const RouteAlign p) {
    pdl_prologue();
    __shared__ int s_count[kRouteMaxExperts], s_start[kRouteMaxExperts];
    route_align_block(p, s_count, s_start, false);
}

// A warp per expert (and one for the gate). A step of few tokens waits for the router's weights, 8 KB a row of 2,048: with few
// tokens there are as many warps as rows, and a warp's first 1,024 weights are asked for before the wait for the kernel ahead
// (they belong to no earlier kernel). With eight loads in flight and a ninth row in a second round two tokens took 17 us.
// FUSED (up to eight tokens): the tokens' blocks are one cluster, whose first block also buckets the pairs once all are there (a
// launch less on the way from the router to the experts' weights). BATCH: weights a lane has in flight; with many
// tokens 8, whose blocks hide one another's waits (1,273 tokens: 15.5 us; with 32 22 us; four tokens a block, sharing what is read: 24 us).
template <typename TX, bool FUSED, int BATCH>
__global__ void __launch_bounds__(BATCH > 8 ? 1024 : 256)
route_kernel(const TX* __restrict__ x, int D, const float* __restrict__ w, const float* __restrict__ correction, int E, int top,
             int softmax, int renormalise, float factor, float* __restrict__ weights,
             const float* __restrict__ gate_w, float* __restrict__ gate_out, int T, const RouteAlign align) {
    pdl_launch_dependents();
    extern __shared__ float s_x[];                 // [D], then the scores and the choice scores [E]
    float* s_score = s_x + D;
    float* s_choice = s_score + E;
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x / 32;
    const int n_rows = E + (gate_w ? 1 : 0);
    float v[BATCH];
    auto request = [&](int e, int d0) {
        const float* row = (e < E ? w + static_cast<size_t>(e) * D : gate_w) + d0 + lane;
        if (d0 + 32 * BATCH <= D) {
#pragma unroll
            for (int i = 0; i < BATCH; ++i) v[i] = row[32 * i];
        } else {
#pragma unroll
            for (int i = 0; i < BATCH; ++i) v[i] = d0 + lane + 32 * i < D ? row[32 * i] : 0.f;
        }
    };
    if (warp < n_rows) request(warp, 0);
    pdl_wait();
    if (FUSED) {
        if (t == 0)                                    // the places of the pairs, while the weights are on their way
            for (int i = threadIdx.x; i < align.max_tiles * align.tile_rows; i += blockDim.x) align.sorted_rows[i] = -1;
        if (t >= T) {                                  // a cluster has a power of two of blocks
            cooperative_groups::this_cluster().sync();
            return;
        }
    }
    for (int d = threadIdx.x; d < D; d += blockDim.x) s_x[d] = to_float(x[static_cast<size_t>(t) * D + d]);
    __syncthreads();
    for (int e = warp; e < n_rows; e += warps) {
        float z = 0.f;
        for (int d0 = 0; d0 < D; d0 += 32 * BATCH) {
            if (e != warp || d0 > 0) request(e, d0);
            if (d0 + 32 * BATCH <= D) {
#pragma unroll
                for (int i = 0; i < BATCH; ++i) z = fmaf(v[i], s_x[d0 + lane + 32 * i], z);
            } else {
#pragma unroll
                for (int i = 0; i < BATCH; ++i)
                    if (d0 + lane + 32 * i < D) z = fmaf(v[i], s_x[d0 + lane + 32 * i], z);
            }
        }
        z = warp_sum(z);
        if (lane != 0) continue;
        if (e == E) {
            gate_out[t] = sigmoid_f(z);
        } else {
            const float s = softmax ? z : 1.0f / (1.0f + expf(-z));
            s_score[e] = s;
            s_choice[e] = s + (correction ? correction[e] : 0.f);
        }
    }
    __syncthreads();
    if (warp == 0) {
        if (softmax) {
            float m = -INFINITY;
            for (int e = lane; e < E; e += 32) m = fmaxf(m, s_score[e]);
            m = warp_max(m);
            float sum = 0.f;
            for (int e = lane; e < E; e += 32) sum += expf(s_score[e] - m);
            const float inv = 1.0f / warp_sum(sum);
            for (int e = lane; e < E; e += 32) {
                const float s = expf(s_score[e] - m) * inv;
                s_score[e] = s;
                s_choice[e] = s + (correction ? correction[e] : 0.f);
            }
            __syncwarp();
        }
        float chosen = 0.f;
        // the ``top`` largest choice scores, the lowest index among equals; a chosen expert leaves the contest
        for (int k = 0; k < top; ++k) {
            float best = -INFINITY;
            int best_e = 0x7fffffff;
            for (int e = lane; e < E; e += 32) {
                const float c = s_choice[e];
                if (c > best) { best = c; best_e = e; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
                if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
            }
            if (best_e >= E) best_e = 0;                 // no comparable score (a row of NaN): any expert, but a real one
            chosen += s_score[best_e];
            if (lane == 0) {
                align.ids[static_cast<size_t>(t) * top + k] = best_e;
                weights[static_cast<size_t>(t) * top + k] = s_score[best_e] * factor;
                s_choice[best_e] = -INFINITY;
            }
            __syncwarp();
        }
        if (renormalise) {
            const float inv = 1.0f / (chosen + 1e-20f);
            for (int k = lane; k < top; k += 32) weights[static_cast<size_t>(t) * top + k] *= inv;
        }
    }
    if (FUSED) {
        cooperative_groups::this_cluster().sync();     // every token's experts are in memory
        if (t == 0) route_align_block(align, reinterpret_cast<int*>(s_score), reinterpret_cast<int*>(s_choice), true);
    }
}

// Experts fixed per token id: ids[t, :] = table[token of row t, :], every weight 1 / top. A token given as -(k + 1) is read
// from place k of the feedback buffer (the id a sampling kernel left on the device), as the embedding kernel reads it.
__global__ void __launch_bounds__(256)
route_table_kernel(const int* __restrict__ tokens, const int* __restrict__ feedback, const int* __restrict__ table, int vocab, int E,
                   int top, int* __restrict__ ids, float* __restrict__ weights, int n_pairs) {
    pdl_prologue();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n_pairs) return;
    int tok = tokens[i / top];
    if (tok < 0) tok = feedback ? feedback[-tok - 1] : 0;
    tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
    int e = table[static_cast<size_t>(tok) * top + i % top];
    e = e < 0 ? 0 : (e >= E ? E - 1 : e);                  // the table is checked when the model is built
    ids[i] = e;
    weights[i] = 1.0f / static_cast<float>(top);
}

template <typename T>
__global__ void __launch_bounds__(256)
gather_rows_kernel(const T* __restrict__ x, int D, int a_div, const int* __restrict__ sorted_rows, const int* __restrict__ n_tiles,
                   int tile_rows, const float* __restrict__ scales, T* __restrict__ out) {
    pdl_prologue();
    const int r = blockIdx.x;
    if (r >= *n_tiles * tile_rows) return;
    const int pair = sorted_rows[r];
    T* dst = out + static_cast<size_t>(r) * D;
    if (pair < 0) {
        for (int d = threadIdx.x; d < D; d += 256) dst[d] = from_float<T>(0.f);
        return;
    }
    const T* src = x + static_cast<size_t>(pair / a_div) * D;
    if (scales) {
        const float sc = scales[pair];
        if (D % 8 == 0 && sizeof(T) == 2) {
            for (int d = threadIdx.x; d < D / 8; d += 256) {
                uint4 raw = reinterpret_cast<const uint4*>(src)[d];
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(h[i]);
                    h[i] = __floats2bfloat162_rn(sc * f.x, sc * f.y);
                }
                reinterpret_cast<uint4*>(dst)[d] = raw;
            }
        } else {
            for (int d = threadIdx.x; d < D; d += 256) dst[d] = from_float<T>(sc * to_float(src[d]));
        }
        return;
    }
    if (D % 8 == 0 && sizeof(T) == 2) {
        for (int d = threadIdx.x; d < D / 8; d += 256) reinterpret_cast<uint4*>(dst)[d] = reinterpret_cast<const uint4*>(src)[d];
    } else {
        for (int d = threadIdx.x; d < D; d += 256) dst[d] = src[d];
    }
}

__global__ void __launch_bounds__(256)
route_combine_kernel(const float* __restrict__ part, const float* __restrict__ weights, const int* __restrict__ pair_row,
                     const float* __restrict__ more, const float* __restrict__ more_gate, float* __restrict__ y, int D, int top, size_t total) {
    pdl_prologue();
    const size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
    if (i >= total) return;
    const size_t t = i / D;
    const int d = static_cast<int>(i % D);
    float v = y[i];
    for (int k = 0; k < top; ++k) {
        const size_t row = pair_row ? static_cast<size_t>(pair_row[t * top + k]) : t * top + k;
        v = fmaf(weights ? weights[t * top + k] : 1.f, part[row * D + d], v);
    }
    if (more) v = fmaf(more_gate[t], more[i], v);
    y[i] = v;
}

// The same, four values a thread in 16-byte pieces (D a multiple of 4, pointers aligned; a value at a time: 17 us for 1,273 tokens
// of two experts, whose bytes need 7).
__global__ void __launch_bounds__(256)
route_combine4_kernel(const float4* __restrict__ part, const float* __restrict__ weights, const int* __restrict__ pair_row,
                      const float4* __restrict__ more, const float* __restrict__ more_gate, float4* __restrict__ y, int D4, int top, size_t total4) {
    pdl_prologue();
    const size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
    if (i >= total4) return;
    const int t = static_cast<int>(i / D4), d = static_cast<int>(i % D4);
    float4 v = y[i];
    auto add = [&](float f, const float4& x) { v.x = fmaf(f, x.x, v.x); v.y = fmaf(f, x.y, v.y); v.z = fmaf(f, x.z, v.z); v.w = fmaf(f, x.w, v.w); };
#pragma unroll 2
    for (int k = 0; k < top; ++k) {
        const size_t pair = static_cast<size_t>(t) * top + k, row = pair_row ? static_cast<size_t>(pair_row[pair]) : pair;
        add(weights ? weights[pair] : 1.f, part[row * D4 + d]);
    }
    if (more) add(more_gate[t], more[i]);
    y[i] = v;
}

// Whether every 16-byte load of the few-row form is aligned: pieces of the weights' rows and of the inputs' rows.
static bool rows_form_fits(const GroupedArgs& p, int a_dtype, int w_dtype) {
    const int piece = w_dtype == kBF16 ? 8 : 4;
    const size_t a_size = a_dtype == kBF16 ? 2 : 4;
    if (a_dtype == kBF16 && w_dtype == kF32) return false;
    if (p.K % piece || p.ldw % piece || p.w_gs % piece || p.up_off % piece) return false;
    if (reinterpret_cast<uintptr_t>(p.w) % 16 || reinterpret_cast<uintptr_t>(p.a) % 16) return false;
    const int a_piece = static_cast<int>(16 / a_size);
    return p.lda % a_piece == 0 && p.a_off % a_piece == 0 && p.a_gs % a_piece == 0;
}

template <typename TA, typename TW, bool GATED, int ROWS>
static int launch_grouped_rows_as(const GroupedArgs& p, unsigned tiles, cudaStream_t st) {
    using Stream = RowsStream<TA, TW, GATED, ROWS>;
    static SharedLimit limit;
    const cudaError_t ready = limit.allow(reinterpret_cast<const void*>(grouped_rows_kernel<TA, TW, GATED, ROWS>), Stream::kSmem);
    if (ready != cudaSuccess) { set_error("grouped_product (rows): %s", cudaGetErrorString(ready)); return 1; }
    const int sms = sm_count();
    const long long blocks = (static_cast<long long>(tiles) * ((p.N + ROWS - 1) / ROWS) + kGrWarps - 1) / kGrWarps;
    GI_REQUIRE(blocks * kGrWarps <= 2147483647LL - 3 * 1024 * kGrWarps, "grouped_product: too many tiles");
    launch_kernel((grouped_rows_kernel<TA, TW, GATED, ROWS>), dim3(static_cast<unsigned>(std::min<long long>(blocks, Stream::kBlocks * sms))), dim3(kGrWarps * 32),
                  Stream::kSmem, st, p, static_cast<int>(tiles));
    return check_launch("grouped_product (rows)");
}
template <typename TA, bool GATED>
static int launch_grouped_mma(const GroupedArgs& p, unsigned tiles, cudaStream_t st) {
    constexpr int kSmem = GmSizes<TA>::kRing + GmSizes<TA>::kSums, kOut = (GATED ? 8 : 16) * GmShape<TA>::MT;
    static SharedLimit limit;
    const cudaError_t ready = limit.allow(reinterpret_cast<const void*>(grouped_mma_kernel<TA, GATED>), kSmem);
    if (ready != cudaSuccess) { set_error("grouped_product (few rows): %s", cudaGetErrorString(ready)); return 1; }
    const int sms = sm_count();
    const long long units = static_cast<long long>(tiles) * (2 / GmShape<TA>::NT) * ((p.N + kOut - 1) / kOut);
    GI_REQUIRE(units <= 2147483647LL - 4 * 1024, "grouped_product: too many tiles");
    launch_kernel((grouped_mma_kernel<TA, GATED>), dim3(static_cast<unsigned>(std::min<long long>(units, kGmBlocks * sms))), dim3(kGmWarps * 32), kSmem, st, p, static_cast<int>(tiles));
    return check_launch("grouped_product (few rows)");
}
// Where few rows of bfloat16 weights are multiplied on the CUDA cores: the time there goes with the rows of the fullest tile, on the tensor
// cores with the tiles and the outputs (a tile's first row costs as much as eight), more with 32-bit inputs, which are cut into parts.
static bool few_on_cuda_cores(const GroupedArgs& p, bool a_is_f32) {
    // Heads: us on the CUDA cores / on the tensor cores, 32-bit inputs, 128 of 128 x 512: one row 9.7 / 28.2, eight 20.5 / 28.7, twelve
    // 29.9 / 28.8; bfloat16 inputs one 9.5 / 17.8, four 13.1 / 17.8. Of few heads a row or two are faster alone (16 of 64 x 512: 3.8 / 5.6), but
    // not in a token's step (11.2 / 7.6, code and inputs cold).
    if (!p.tile_group) return p.groups >= 64 && p.rows <= (a_is_f32 ? 10 : 5);
    // Experts: p.rows pairs of p.groups experts. Most have a tile of their own while they are fewer than the experts, or two an expert of
    // up to four or of very many. Weights from memory, 32-bit inputs: six pairs of eight experts, 2,048 outputs of 4,096 inputs 32.3 / 32.3,
    // 4,608 of 2,048 29.2 / 40.6; eight 33.8 / 41.5 on eight of them and 19.6 / 16.0 on two (in a token's step 32.5 / 31.4); 16 of 32, 768 of 2,048
    // 18.2 / 23.4, 32 22.8 / 28.1, 64 39.9 / 30.7; 128 of 64, 512 of 1,024 26.9 / 27.1; 2, 2, 2, 2 of four 18.5 / 26.6, 3, 3 of two 18.7 / 15.3, four of one 18.5 / 13.8.
    // bfloat16 inputs, which need no cutting, only where K is short, so that a unit's work is little beside its beginning and end: 16 of
    // 64, gated, 2 x 1,024 of 512 15.6 / 20.1, 32 of 128, 256 of 512 6.8 / 8.1; of 2,048 inputs 12 of 32 21.8 / 19.9.
    const int experts = p.groups;
    if (a_is_f32) return experts <= 4 || experts >= 64 ? p.rows <= 2 * experts : experts >= 16 ? p.rows <= experts : 4 * p.rows <= 3 * experts;
    return p.rows >= 6 && p.rows <= experts && p.K <= 1024;
}
template <bool GATED>
static int launch_grouped_rows(const GroupedArgs& p, int a_dtype, int w_dtype, unsigned tiles, cudaStream_t st) {
    if (w_dtype == kF32) return launch_grouped_rows_as<float, float, GATED, 4>(p, tiles, st);
    const bool f32 = a_dtype == kF32;
    if (few_on_cuda_cores(p, f32)) {
        // eight rows a unit for 32-bit inputs, as many bytes as four rows of weights for every two; heads' matrices and gated
        // ones are too small, or need too many registers, for that
        if constexpr (!GATED)
            if (f32 && p.tile_group) return launch_grouped_rows_as<float, __nv_bfloat16, false, 8>(p, tiles, st);
        return f32 ? launch_grouped_rows_as<float, __nv_bfloat16, GATED, 4>(p, tiles, st) : launch_grouped_rows_as<__nv_bfloat16, __nv_bfloat16, GATED, 4>(p, tiles, st);
    }
    return f32 ? launch_grouped_mma<float, GATED>(p, tiles, st) : launch_grouped_mma<__nv_bfloat16, GATED>(p, tiles, st);
}

template <bool GATED>
static int launch_grouped(const GroupedArgs& p, int a_dtype, int w_dtype, dim3 grid, cudaStream_t st) {
    if (a_dtype == kF32 && w_dtype == kF32) launch_kernel((grouped_product_kernel<float, float, GATED>), grid, dim3(128), 0, st, p);
    else if (a_dtype == kF32 && w_dtype == kBF16) launch_kernel((grouped_product_kernel<float, __nv_bfloat16, GATED>), grid, dim3(128), 0, st, p);
    else if (a_dtype == kBF16 && w_dtype == kBF16) launch_kernel((grouped_product_kernel<__nv_bfloat16, __nv_bfloat16, GATED>), grid, dim3(128), 0, st, p);
    else { set_error("grouped_product: inputs of dtype code %d with weights of %d are not built", a_dtype, w_dtype); return 2; }
    return check_launch("grouped_product");
}

// bfloat16 weights in pieces that rows_form_fits has looked at. Up to 8 rows a block has 64 outputs, with more 64 rows and 64 outputs.
template <typename TA>
static int launch_head_mma(const GroupedArgs& p, cudaStream_t st) {
    const unsigned heads = static_cast<unsigned>(p.groups), blocks_n = static_cast<unsigned>((p.N + 63) / 64);
    GI_REQUIRE(blocks_n <= 65535, "head_product: too many tiles");
    if (p.rows <= 8) launch_kernel((head_mma_kernel<TA, 1, 1, true>), dim3(heads, blocks_n), dim3(128), 0, st, p);
    else if (p.rows <= 32) launch_kernel((head_mma_kernel<TA, 1, 2, true>), dim3(heads, blocks_n, (p.rows + 15) / 16), dim3(128), 0, st, p);
    else launch_kernel((head_mma_kernel<TA, 4, 2, false>), dim3(heads, blocks_n, (p.rows + 63) / 64), dim3(128), 0, st, p);
    return check_launch("head_product (tensor cores)");
}

}  // namespace gi

using namespace gi;

extern "C" int gi_grouped_tile_rows() { return kGpTM; }

static int gi_head_product_impl(const void* a, int a_dtype, long long lda, int a_off, int a_gs, const void* w, int w_dtype,
                                long long w_gs, void* out, int out_dtype, long long ldo, int o_off, int o_gs, int rows, int heads,
                                int N, int K, int tail, const float* freq, float amplitude, int tail_interleaved, const int* positions, const float* gate,
                                long long ldg, int gate_off, int gate_per_head, int w_constant, void* stream) {
    if (rows == 0) return 0;
    GI_REQUIRE(rows > 0 && heads > 0 && N > 0 && K > 0, "head_product: sizes must be positive");
    GI_REQUIRE(gate == nullptr || (gate_off >= 0 && gate_off + static_cast<long long>(heads) * (gate_per_head ? 1 : N) <= ldg), "head_product: the gate's columns lie outside its rows");
    GI_REQUIRE(tail >= 0 && tail % 2 == 0 && (tail == 0 || (freq && positions)), "head_product: a rotated tail needs an even size, frequencies and positions");
    GI_REQUIRE(out_dtype == kF32 || out_dtype == kBF16, "head_product: unsupported output dtype");
    GroupedArgs p = {};
    p.a = a; p.lda = lda; p.a_off = a_off; p.a_gs = a_gs; p.a_div = 1;
    p.w = w; p.w_gs = w_gs; p.ldw = K; p.up_off = 0; p.w_constant = w_constant;
    p.out = out; p.out_is_f32 = out_dtype == kF32; p.ldo = ldo; p.o_off = o_off; p.o_gs = o_gs;
    p.N = N; p.K = K; p.rows = rows; p.groups = heads;
    p.tail = tail; p.freq = freq; p.amplitude = amplitude; p.tail_interleaved = tail_interleaved; p.positions = positions;
    p.gate = gate; p.ldg = ldg; p.gate_off = gate_off; p.gate_hs = gate_per_head ? 1 : N; p.gate_ns = gate_per_head ? 0 : 1;
    const long long tiles = static_cast<long long>((rows + kGpTM - 1) / kGpTM) * heads;
    GI_REQUIRE(tiles <= 2147483647LL, "head_product: too many tiles");
    dim3 grid(static_cast<unsigned>(tiles), (N + kGpTN - 1) / kGpTN);
    // few tokens without a tail: the heads' matrices are what is read, their K shared by a block's warps; else bfloat16 weights on the
    // tensor cores at every row count. (With a tail every row count has the same sums to the bit, whatever form it runs.)
    if (rows_form_fits(p, a_dtype, w_dtype)) {
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        if (tail == 0 && rows <= 2 * kGpTM) return launch_grouped_rows<false>(p, a_dtype, w_dtype, static_cast<unsigned>(tiles), st);
        if (w_dtype == kBF16 && rows <= 65535 * 64)                   // (blocks of rows along the grid's third axis; more: below)
            return a_dtype == kF32 ? launch_head_mma<float>(p, st) : launch_head_mma<__nv_bfloat16>(p, st);
        if (tail > 0 && rows <= kGcRows) {
            launch_kernel(head_product_few_kernel, dim3(heads, (N + kGcCols - 1) / kGcCols), dim3(kGcCols), 0, st, p);
            return check_launch("head_product (few rows)");
        }
    }
    // many tokens: tiles of 64 x 64 where every group of four values is aligned (K in whole fours: no ragged piece)
    if (rows >= 2 * kG64 && K % 4 == 0 && lda % 4 == 0 && a_off % 4 == 0 && a_gs % 4 == 0 && w_gs % 4 == 0 &&
        reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0 && !(a_dtype == kBF16 && w_dtype == kF32)) {
        const long long tiles64 = static_cast<long long>((rows + kG64 - 1) / kG64) * heads;
        GI_REQUIRE(tiles64 <= 2147483647LL, "head_product: too many tiles");
        dim3 grid64(static_cast<unsigned>(tiles64), (N + kG64 - 1) / kG64);
        cudaStream_t st64 = static_cast<cudaStream_t>(stream);
        if (a_dtype == kF32 && w_dtype == kF32) launch_kernel((head_product64_kernel<float, float>), grid64, dim3(256), 0, st64, p);
        else if (a_dtype == kF32) launch_kernel((head_product64_kernel<float, __nv_bfloat16>), grid64, dim3(256), 0, st64, p);
        else launch_kernel((head_product64_kernel<__nv_bfloat16, __nv_bfloat16>), grid64, dim3(256), 0, st64, p);
        return check_launch("head_product (tiles of 64)");
    }
    return launch_grouped<false>(p, a_dtype, w_dtype, grid, static_cast<cudaStream_t>(stream));
}

static int gi_expert_product_impl(const void* a, int a_dtype, long long lda, int a_div, const void* w, int w_dtype, long long w_gs,
                                  int ldw, long long up_off, int gated, int act, float act_limit, const float* scales, void* out, int out_dtype, long long ldo,
                                  int N, int K, const int* tile_group, const int* sorted_rows, const int* n_tiles, int max_tiles,
                                  int pairs, int experts, void* stream) {
    if (max_tiles == 0) return 0;
    GI_REQUIRE(max_tiles > 0 && N > 0 && K > 0 && a_div > 0, "expert_product: sizes must be positive");
    GI_REQUIRE(tile_group && sorted_rows && n_tiles, "expert_product: the sorted rows are missing");
    GI_REQUIRE(act >= 0 && act < (gated ? static_cast<int>(kActCount) : static_cast<int>(kPlainCount)), "expert_product: unknown activation code %d", act);
    GroupedArgs p = {};
    p.a = a; p.lda = lda; p.a_div = a_div;
    p.w = w; p.w_gs = w_gs; p.ldw = ldw; p.up_off = up_off;
    p.out = out; p.out_is_f32 = out_dtype == kF32; p.ldo = ldo;
    p.N = N; p.K = K; p.groups = experts; p.rows = pairs;
    p.tile_group = tile_group; p.sorted_rows = sorted_rows; p.n_tiles = n_tiles; p.act = gated ? act : 0; p.act_limit = act_limit;
    p.out_act = gated ? kPlainNone : act;
    p.scales = scales;
    dim3 grid(max_tiles, (N + kGpTN - 1) / kGpTN);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows_form_fits(p, a_dtype, w_dtype))
        return gated ? launch_grouped_rows<true>(p, a_dtype, w_dtype, max_tiles, st) : launch_grouped_rows<false>(p, a_dtype, w_dtype, max_tiles, st);
    return gated ? launch_grouped<true>(p, a_dtype, w_dtype, grid, st) : launch_grouped<false>(p, a_dtype, w_dtype, grid, st);
}

static int gi_route_impl(const void* x, int x_dtype, int T, int D, const float* w, const float* correction, int E, int top,
                         int softmax, int renormalise, float factor, int* ids, float* weights, int* sorted_rows, int* tile_group, int* n_tiles, int max_tiles, int tile_rows,
                         int* pair_row, const float* gate_w, float* gate_out, void* stream) {
    if (T == 0) return 0;
    GI_REQUIRE((gate_w == nullptr) == (gate_out == nullptr), "route: a gate needs its row and a place for its values");
    GI_REQUIRE(T > 0 && D > 0 && E > 0 && top > 0 && top <= E, "route: sizes must be positive and top at most the experts");
    GI_REQUIRE(E <= kRouteMaxExperts, "route: %d experts exceed %d", E, kRouteMaxExperts);
    GI_REQUIRE(static_cast<size_t>(D) * 4 <= 160 * 1024, "route: a row of %d values does not fit shared memory", D);
    const long long pairs = static_cast<long long>(T) * top;
    GI_REQUIRE(tile_rows > 0, "route: tiles must have rows");
    GI_REQUIRE(max_tiles >= (pairs + tile_rows - 1) / tile_rows + std::min<long long>(E, pairs) - 1, "route: room for %d tiles is too little", max_tiles);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rows = E + (gate_w ? 1 : 0);
    const int threads = T <= 64 ? std::min(1024, 32 * std::max(8, rows)) : 256;
    const RouteAlign align{ids, static_cast<int>(pairs), E, sorted_rows, tile_group, n_tiles, max_tiles, tile_rows, pair_row};
    // a cluster of up to eight blocks is portable; the places are few there (tiles of 128 rows belong to many tokens)
    const bool fused = T <= 8 && tile_rows == kGpTM;
    const size_t per_token = (static_cast<size_t>(D) + 2 * static_cast<size_t>(E)) * 4;
    const bool many = T > 64;
    auto launch = [&](auto kernel, auto* values) {
        const size_t smem = per_token;
        if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        int blocks = T;
        if (fused) for (blocks = 1; blocks < T; blocks *= 2) {}
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = g_pdl_enabled ? 1 : 0;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = fused ? blocks : 1;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = fused ? 2 : 1;
        counted(cudaLaunchKernelEx(&cfg, kernel, values, D, w, correction, E, top, softmax, renormalise, factor, weights, gate_w, gate_out, T, align));
    };
    if (x_dtype == kF32) {
        const float* values = static_cast<const float*>(x);
        if (fused) launch(route_kernel<float, true, 32>, values);
        else if (many) launch(route_kernel<float, false, 8>, values);
        else launch(route_kernel<float, false, 32>, values);
    } else if (x_dtype == kBF16) {
        const __nv_bfloat16* values = static_cast<const __nv_bfloat16*>(x);
        if (fused) launch(route_kernel<__nv_bfloat16, true, 32>, values);
        else if (many) launch(route_kernel<__nv_bfloat16, false, 8>, values);
        else launch(route_kernel<__nv_bfloat16, false, 32>, values);
    } else {
        GI_REQUIRE(false, "route: unsupported dtype code %d", x_dtype);
    }
    if (check_launch("route")) return 1;
    if (fused) return 0;
    launch_kernel(route_align_kernel, dim3(1), dim3(1024), 0, st, align);
    return check_launch("route_align");
}

static int gi_route_table_impl(const int* tokens, const int* feedback, const int* table, int vocab, int T, int E, int top, int* ids,
                               float* weights, int* sorted_rows, int* tile_group, int* n_tiles, int max_tiles, int tile_rows,
                               int* pair_row, void* stream) {
    if (T == 0) return 0;
    GI_REQUIRE(T > 0 && vocab > 0 && E > 0 && top > 0 && top <= E, "route_table: sizes must be positive and top at most the experts");
    GI_REQUIRE(E <= kRouteMaxExperts, "route_table: %d experts exceed %d", E, kRouteMaxExperts);
    const long long pairs = static_cast<long long>(T) * top;
    GI_REQUIRE(tile_rows > 0 && pairs <= 2147483647LL, "route_table: tiles must have rows");
    GI_REQUIRE(max_tiles >= (pairs + tile_rows - 1) / tile_rows + std::min<long long>(E, pairs) - 1, "route_table: room for %d tiles is too little", max_tiles);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    launch_kernel(route_table_kernel, dim3(static_cast<unsigned>((pairs + 255) / 256)), dim3(256), 0, st, tokens, feedback, table, vocab, E, top,
                  ids, weights, static_cast<int>(pairs));
    if (check_launch("route_table")) return 1;
    launch_kernel(route_align_kernel, dim3(1), dim3(1024), 0, st, RouteAlign{ids, static_cast<int>(pairs), E, sorted_rows, tile_group, n_tiles, max_tiles, tile_rows, pair_row});
    return check_launch("route_align");
}

static int gi_gather_rows_impl(const void* x, int dtype, int D, int a_div, const int* sorted_rows, const int* n_tiles, int tile_rows,
                               int max_rows, const float* scales, void* out, void* stream) {
    if (max_rows == 0) return 0;
    GI_REQUIRE(max_rows > 0 && D > 0 && a_div > 0 && tile_rows > 0, "gather_rows: sizes must be positive");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == kBF16)
        launch_kernel((gather_rows_kernel<__nv_bfloat16>), dim3(max_rows), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(x), D, a_div,
                      sorted_rows, n_tiles, tile_rows, scales, static_cast<__nv_bfloat16*>(out));
    else if (dtype == kF32)
        launch_kernel((gather_rows_kernel<float>), dim3(max_rows), dim3(256), 0, st, static_cast<const float*>(x), D, a_div, sorted_rows,
                      n_tiles, tile_rows, scales, static_cast<float*>(out));
    else
        GI_REQUIRE(false, "gather_rows: unsupported dtype code %d", dtype);
    return check_launch("gather_rows");
}

static int gi_route_combine_impl(const float* part, const float* weights, const int* pair_row, const float* more, const float* more_gate, float* y, int T, int D, int top, void* stream) {
    if (T == 0) return 0;
    GI_REQUIRE(T > 0 && D > 0 && top > 0, "route_combine: sizes must be positive");
    GI_REQUIRE((more == nullptr) == (more_gate == nullptr), "route_combine: a gated part needs its gate");
    const size_t total = static_cast<size_t>(T) * D;
    auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    if (D % 4 == 0 && aligned(part) && aligned(more) && aligned(y)) {
        launch_kernel(route_combine4_kernel, dim3(static_cast<unsigned>((total / 4 + 255) / 256)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                      reinterpret_cast<const float4*>(part), weights, pair_row, reinterpret_cast<const float4*>(more), more_gate, reinterpret_cast<float4*>(y), D / 4, top, total / 4);
        return check_launch("route_combine");
    }
    launch_kernel(route_combine_kernel, dim3(static_cast<unsigned>((total + 255) / 256)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                  part, weights, pair_row, more, more_gate, y, D, top, total);
    return check_launch("route_combine");
}

extern "C" int gi_head_product(const void* a, int a_dtype, long long lda, int a_off, int a_gs, const void* w, int w_dtype,
                               long long w_gs, void* out, int out_dtype, long long ldo, int o_off, int o_gs, int rows, int heads,
                               int N, int K, int tail, const float* freq, float amplitude, int tail_interleaved, const int* positions, const float* gate,
                               long long ldg, int gate_off, int gate_per_head, int w_constant, void* stream) {
    return gi::dispatch(gi_head_product_impl, a, a_dtype, lda, a_off, a_gs, w, w_dtype, w_gs, out, out_dtype, ldo, o_off, o_gs, rows,
                        heads, N, K, tail, freq, amplitude, tail_interleaved, positions, gate, ldg, gate_off, gate_per_head, w_constant, stream);
}

extern "C" int gi_expert_product(const void* a, int a_dtype, long long lda, int a_div, const void* w, int w_dtype, long long w_gs,
                                 int ldw, long long up_off, int gated, int act, float act_limit, const float* scales, void* out, int out_dtype, long long ldo, int N, int K,
                                 const int* tile_group, const int* sorted_rows, const int* n_tiles, int max_tiles, int pairs, int experts, void* stream) {
    return gi::dispatch(gi_expert_product_impl, a, a_dtype, lda, a_div, w, w_dtype, w_gs, ldw, up_off, gated, act, act_limit, scales, out, out_dtype, ldo,
                        N, K, tile_group, sorted_rows, n_tiles, max_tiles, pairs, experts, stream);
}

extern "C" int gi_route(const void* x, int x_dtype, int T, int D, const float* w, const float* correction, int E, int top,
                        int softmax, int renormalise, float factor, int* ids, float* weights, int* sorted_rows, int* tile_group, int* n_tiles, int max_tiles, int tile_rows, int* pair_row,
                        const float* gate_w, float* gate_out, void* stream) {
    return gi::dispatch(gi_route_impl, x, x_dtype, T, D, w, correction, E, top, softmax, renormalise, factor, ids, weights, sorted_rows, tile_group, n_tiles,
                        max_tiles, tile_rows, pair_row, gate_w, gate_out, stream);
}

extern "C" int gi_route_table(const int* tokens, const int* feedback, const int* table, int vocab, int T, int E, int top, int* ids,
                              float* weights, int* sorted_rows, int* tile_group, int* n_tiles, int max_tiles, int tile_rows,
                              int* pair_row, void* stream) {
    return gi::dispatch(gi_route_table_impl, tokens, feedback, table, vocab, T, E, top, ids, weights, sorted_rows, tile_group, n_tiles,
                        max_tiles, tile_rows, pair_row, stream);
}

extern "C" int gi_gather_rows(const void* x, int dtype, int D, int a_div, const int* sorted_rows, const int* n_tiles, int tile_rows,
                              int max_rows, const float* scales, void* out, void* stream) {
    return gi::dispatch(gi_gather_rows_impl, x, dtype, D, a_div, sorted_rows, n_tiles, tile_rows, max_rows, scales, out, stream);
}

extern "C" int gi_route_combine(const float* part, const float* weights, const int* pair_row, const float* more, const float* more_gate, float* y, int T, int D, int top, void* stream) {
    return gi::dispatch(gi_route_combine_impl, part, weights, pair_row, more, more_gate, y, T, D, top, stream);
}
