// Matrix product of the true 32-bit path: C[M,N] (+)= A[M,K] * W[N,K]^T, all 32-bit, on the CUDA cores.
//
// Bounds: with few rows the weights' bytes (every weight is used M times), with many the fused multiply-adds
// (128 a clock and SM) and, as close, the reads of shared memory: a warp's 16-byte read takes four clocks whether its lanes read
// one place or 32, so a thread's tile of TM x TN outputs costs (TM + TN) reads for every 4 TM TN multiply-adds, and the
// four quarters of an SM share the port (which is why a thread's tile is not smaller). The plain kernel (gemm_simt.cu) came
// near neither: loads of single values, none in flight while it multiplied, and 32 blocks at N = 2048. Here
//   - operands pass through shared memory in a ring of tiles of BK values, copied asynchronously in pieces of
//     16 bytes (cp.async), as they lie in memory: rows along k, padded by 4 values so that the 16-byte reads of eight rows
//     fall into different banks;
//   - a thread keeps of each output two sums, over even and over odd k: a pair of neighbouring k is then one packed
//     multiply-add of two register pairs as they were read (no transposing, no duplicating; half the instructions);
//   - a thread has 8 x 8 outputs for many rows (8 x 4 in twice the warps: 3 % slower; 16 x 8 single sums, which read less: 40 %
//     slower, two warps a scheduler of 255 registers); with up to 2, 4, 6, 8, 16 or 32 rows blocks of that height (few rows would
//     multiply zeros in a tall one), up to 16 rows of a single warp, so that N = 2048 still gives every SM a block or two;
//   - where the blocks along N alone leave SMs idle, K is cut into up to 8 chunks, one per CTA of a cluster, whose sums are
//     added in the order of the chunks through distributed shared memory: no workspace and no second launch.
// An output is (over chunks s) sum of (even_s + odd_s); chunks depend on N and K only. So a row's result does not depend
// on M, on the block's height or on where the row sits in the batch (how tokens are cut into steps), and its chains are
// half as long or shorter than one chain over all of K.
// Measured on prompts of 268 rows and steps of 6 (four layers of the 1B sizes, 32-bit): all products of a prompt step 9.9 ms
// before, 4.3 ms now; of a token step 6.5 before, 0.52 now (the head of 128,256 rows 1,180 us before, 207 now); logits off from
// 64 bits by 4.4e-6 before, 1.6e-6 now; the pass with its five sampled steps 59.5 to 8.5 ms (the sampling kernel among it).
#include <cooperative_groups.h>

#include "device_limit.h"
#include "gemm_f32.cuh"

namespace gi {
namespace {

constexpr int kMaxChunks = 8, kChunkStep = 32;          // a chunk's length is a multiple of kChunkStep

__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ void copy16(float* smem, const float* global, bool valid) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    const int bytes = valid ? 16 : 0;                 // 0: the 16 bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(global), "r"(bytes) : "memory");
}

template <int BM_, int BN_, int TM_, int TN_, int BK_, int STAGES_, int BLOCKS_>
struct F32Tile {
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, BK = BK_, kStages = STAGES_, kBlocks = BLOCKS_;      // kBlocks: an SM
    static constexpr int kRowsT = BM / TM, kColsT = BN / TN, kThreads = kRowsT * kColsT;      // threads along m and n
    static constexpr int kLaneM = kRowsT < 4 ? kRowsT : 4, kLaneN = 32 / kLaneM;
    static constexpr int kPad = BK + 4;
    static constexpr int kStage = (BM + BN) * kPad;                   // floats of a stage
    static constexpr size_t kSmem = sizeof(float) * kStage * kStages;
    static constexpr int kPieces = BK / 4, kCopyRows = kThreads / kPieces;                    // rows that one round of copies covers
    static_assert(BM * BN <= kStage * kStages, "the block's sums reuse the ring");
    static_assert(kRowsT % kLaneM == 0 && kColsT % kLaneN == 0 && BN % kCopyRows == 0 && kChunkStep % BK == 0, "");
};
using Tile2 = F32Tile<2, 64, 2, 2, 32, 5, 4>;
using Tile4 = F32Tile<4, 64, 4, 2, 32, 5, 4>;
using Tile6 = F32Tile<6, 64, 6, 2, 32, 5, 4>;
using Tile8 = F32Tile<8, 64, 8, 2, 32, 5, 4>;
using Tile16 = F32Tile<16, 64, 8, 4, 32, 4, 4>;
using Tile32 = F32Tile<32, 128, 8, 4, 32, 3, 3>;
using Tile40 = F32Tile<40, 128, 5, 8, 32, 4, 2>;
using Tile48 = F32Tile<48, 128, 6, 8, 32, 4, 2>;
using Tile56 = F32Tile<56, 128, 7, 8, 32, 4, 2>;
using Tile64 = F32Tile<64, 128, 8, 8, 32, 4, 2>;

// grid (chunks, blocks of rows, blocks of columns), clusters of `chunks` along x. kc: length of a chunk.
template <typename T>
__global__ void __launch_bounds__(T::kThreads, T::kBlocks)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                int lda, int ldw, int ldc, int kc, int accumulate, int w_constant) {
    constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, kStages = T::kStages, kPad = T::kPad;
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int kWarpsM = T::kRowsT / T::kLaneM;
    const int tm = (warp % kWarpsM) * T::kLaneM + lane / T::kLaneN;
    const int tn = (warp / kWarpsM) * T::kLaneN + lane % T::kLaneN;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.z * BN;
    const int chunk = blockIdx.x, k_begin = chunk * kc, k_end = min(K, k_begin + kc);
    const int tiles = k_end > k_begin ? (k_end - k_begin + T::BK - 1) / T::BK : 0;

    // thread t copies piece t % kPieces of rows t / kPieces, + kCopyRows, ... of either operand
    const int cr = t / T::kPieces, ck = (t % T::kPieces) * 4;
    auto load_a = [&](int tile) {
        float* s = smem + (tile % kStages) * T::kStage + ck;
        const int k = k_begin + tile * T::BK + ck;
#pragma unroll
        for (int r = 0; r < (BM + T::kCopyRows - 1) / T::kCopyRows; ++r) {
            const int row = cr + r * T::kCopyRows;
            if (BM % T::kCopyRows == 0 || row < BM) {
                const bool ok = k < k_end && m0 + row < M;
                copy16(s + row * kPad, ok ? A + static_cast<size_t>(m0 + row) * lda + k : A, ok);
            }
        }
    };
    auto load_w = [&](int tile) {
        float* s = smem + (tile % kStages) * T::kStage + ck;
        const int k = k_begin + tile * T::BK + ck;
#pragma unroll
        for (int r = 0; r < BN / T::kCopyRows; ++r) {
            const int row = cr + r * T::kCopyRows;
            const bool ok = k < k_end && n0 + row < N;
            copy16(s + (BM + row) * kPad, ok ? W + static_cast<size_t>(n0 + row) * ldw + k : W, ok);
        }
    };
    auto commit = []() { asm volatile("cp.async.commit_group;" ::: "memory"); };

    unsigned long long acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    // w_constant: the weights of the first tiles are asked for before the wait for the kernel ahead, as no kernel that may still be running
    // writes them (six rows in a token's step: N = 16,384, K = 2,048 33.2 -> 28.9 us, N = 3,072 8.4 -> 7.5)
    if (!w_constant) pdl_wait();
    for (int i = 0; i < kStages - 1; ++i)
        if (i < tiles) load_w(i);
    pdl_wait();
    for (int i = 0; i < kStages - 1; ++i) {
        if (i < tiles) load_a(i);
        commit();
    }
    for (int tile = 0; tile < tiles; ++tile) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();                              // the tile is there for all, and all are done with the one before it
        if (tile + kStages - 1 < tiles) { load_a(tile + kStages - 1); load_w(tile + kStages - 1); }
        commit();
        const float* sa = smem + (tile % kStages) * T::kStage + tm * kPad;
        const float* sw = smem + (tile % kStages) * T::kStage + (BM + tn) * kPad;
#pragma unroll
        for (int k = 0; k < T::BK; k += 4) {
            ulonglong2 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(sa + i * T::kRowsT * kPad + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(sw + j * T::kColsT * kPad + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fma_pair(a[i].y, w.y, fma_pair(a[i].x, w.x, acc[i][j]));
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the chunk's sums [BM, BN] in the ring's place
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const float even = __uint_as_float(static_cast<unsigned>(acc[i][j])), odd = __uint_as_float(static_cast<unsigned>(acc[i][j] >> 32));
            smem[(tm + i * T::kRowsT) * BN + tn + j * T::kColsT] = even + odd;
        }
    const int chunks = gridDim.x;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    if (chunks > 1) cluster.sync();
    else __syncthreads();
    // CTA `chunk` finishes every chunks-th row of the block: the chunks' sums in their order
    for (int row = chunk; row < BM && m0 + row < M; row += chunks) {
#pragma unroll
        for (int col = t; col < BN; col += T::kThreads) {
            float v = smem[row * BN + col];
            if (chunks > 1) {
                float part[kMaxChunks];
#pragma unroll
                for (int s = 0; s < kMaxChunks; ++s)
                    if (s < chunks) part[s] = *cluster.map_shared_rank(smem + row * BN + col, s);
                v = part[0];
#pragma unroll
                for (int s = 1; s < kMaxChunks; ++s)
                    if (s < chunks) v += part[s];
            }
            if (n0 + col < N) {
                float* c = C + static_cast<size_t>(m0 + row) * ldc + n0 + col;
                *c = accumulate ? *c + v : v;
            }
        }
    }
    if (chunks > 1) cluster.sync();                   // a CTA's sums stay until all have read them
}

template <typename T>
int launch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int chunks, int kc,
           int accumulate, int w_constant, cudaStream_t st) {
    static SharedLimit limit;
    const cudaError_t ready = limit.allow(reinterpret_cast<const void*>(gemm_f32_kernel<T>), static_cast<int>(T::kSmem));
    if (ready != cudaSuccess) { set_error("gemm: %s", cudaGetErrorString(ready)); return 1; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(chunks, (M + T::BM - 1) / T::BM, (N + T::BN - 1) / T::BN);
    cfg.blockDim = dim3(T::kThreads);
    cfg.dynamicSmemBytes = T::kSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = g_pdl_enabled ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = chunks;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    counted(cudaLaunchKernelEx(&cfg, gemm_f32_kernel<T>, A, W, C, M, N, K, lda, ldw, ldc, kc, accumulate, w_constant));
    return check_launch("gemm_f32");
}

}  // namespace

// Rows of 16-byte pieces (copy16), blocks within the grid's limits.
bool gemm_f32_takes(const float* A, const float* W, int M, int N, int K, int lda, int ldw) {
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && aligned(A) && aligned(W) && (M + 63) / 64 <= 65535 && (N + 63) / 64 <= 65535;
}

int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate, int w_constant, cudaStream_t st) {
    // Chunks of K until the blocks along N fill the 148 SMs, none shorter than 256: by N and K alone (see above).
    int chunks = 1;
    while (chunks < kMaxChunks && (N + 127) / 128 * chunks < 148 && K / (2 * chunks) >= 256) chunks *= 2;
    const int kc = ((K + chunks - 1) / chunks + kChunkStep - 1) / kChunkStep * kChunkStep;
    if (M <= 2) return launch<Tile2>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (M <= 4) return launch<Tile4>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (M <= 6) return launch<Tile6>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (M <= 8) return launch<Tile8>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (M <= 16) return launch<Tile16>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (M <= 32) return launch<Tile32>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    // More rows: blocks of 8 x 5 .. 8 rows, the height whose rounds over the SMs (two blocks each) are the least work: a block that is
    // half outside the matrix, or a last round that is nearly empty, costs as much as a full one. A block's time goes with its
    // rows and a row's worth of the rest; a last round of a block an SM takes 0.7 of one of two; clusters of four and eight leave
    // places that no further one fits; and another height has to promise 4 %, as the promise is that rough. Of 551 products of 33 to 2,048
    // rows (100 to 128,256 outputs of 36 to 14,336 inputs) the height taken is 1.2 % slower than the best (blocks of 64: 20 %), and two
    // are more than 3 % slower than blocks of 64 (by 5 at most). (268 rows, blocks of 64 -> the height taken: 16,384 outputs of
    // 2,048 inputs 495 -> 455 us in blocks of 56; 2,048 of 2,048 and 8,192 together 189 -> 171 each and 3,072 of 2,048 122 -> 112 in blocks of 48.)
    int best = 8;
    long long least = -1;
    const int at_once = 2 * sm_count() - (chunks > 2 ? 12 : 0);
    for (int tm = 8; tm >= 5; --tm) {
        const int rows = (M + 8 * tm - 1) / (8 * tm);
        if (rows > 65535) break;                           // the grid's limit
        const long long blocks = static_cast<long long>(chunks) * ((N + 127) / 128) * rows;
        const long long left = blocks % at_once;
        const long long cost = (blocks / at_once * 10 + (left == 0 ? 0 : 2 * left <= at_once ? 7 : 10)) * (tm + 1);
        if (least < 0 || (best == 8 ? cost * 100 < least * 96 : cost < least)) { least = cost; best = tm; }
    }
    if (best == 5) return launch<Tile40>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (best == 6) return launch<Tile48>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    if (best == 7) return launch<Tile56>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
    return launch<Tile64>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, w_constant, st);
}

}  // namespace gi
