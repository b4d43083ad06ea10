// Matrix product of the true 32-bit path: C[M,N] (+)= A[M,K] * W[N,K]^T, all 32-bit, on the CUDA cores.
//
// Bounds: with few rows the weights' bytes (every weight is used M times), with many the fused multiply-adds
// (128 a clock and SM). The plain kernel (gemm_simt.cu) came near neither: loads of single values, none in flight while it
// multiplied, and 32 blocks at N = 2048. Here
//   - operands pass through shared memory in a ring of kStages tiles of kBK values, copied asynchronously in pieces of
//     16 bytes (cp.async), as they lie in memory: rows along k, padded to 36 values so that the 16-byte reads of eight rows
//     fall into different banks;
//   - a thread keeps 8 x (BM / 8) outputs, and of each output two sums, over even and over odd k: a pair of neighbouring k
//     is then one packed multiply-add of two register pairs as they were read (no transposing, no duplicating);
//   - blocks of 64, 32, 16 or 8 rows by M (few rows would multiply zeros in a tall block);
//   - where the blocks along N alone leave SMs idle, K is cut into up to 8 chunks, one per CTA of a cluster, whose sums are
//     added in the order of the chunks through distributed shared memory: no workspace and no second launch.
// An output is (over chunks s) sum of (even_s + odd_s); chunks depend on N and K only. So a row's result does not depend
// on M, on the block's height or on where the row sits in the batch (how tokens are cut into steps), and its chains are
// half as long or shorter than one chain over all of K.
// Measured on prompts of 268 rows and steps of 6 (four layers of the 1B sizes, 32-bit): all products of a prompt step 10.0 ms
// before, 3.3 ms now; logits off from 64 bits by 4.4e-6 before, 1.6e-6 now; the sampled pass 59.5 to 16.3 ms.
#include <cooperative_groups.h>

#include "gemm_f32.cuh"

namespace gi {
namespace {

constexpr int kBN = 128, kBK = 32, kPad = 36, kThreads = 128, kStages = 4, kMaxChunks = 8;

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

template <int BM>
struct F32Tile {
    static constexpr int kTN = BM / 8;                                // outputs a thread has along n; along m: 8
    static constexpr int kRowsT = BM / 8, kColsT = kThreads / kRowsT; // threads along m and n
    static constexpr int kLaneM = kRowsT < 4 ? kRowsT : 4, kLaneN = 32 / kLaneM;
    static constexpr int kStage = (BM + kBN) * kPad;                  // floats of a stage
    static constexpr size_t kSmem = sizeof(float) * kStage * kStages;
    static_assert(BM * kBN <= kStage * kStages, "the block's sums reuse the ring");
};

// grid (chunks, blocks of rows, blocks of columns), clusters of `chunks` along x. kc: length of a chunk, a multiple of kBK.
template <int BM>
__global__ void __launch_bounds__(kThreads, 2)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                int lda, int ldw, int ldc, int kc, int accumulate) {
    using T = F32Tile<BM>;
    extern __shared__ __align__(16) float smem[];
    pdl_prologue();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int kWarpsM = T::kRowsT / T::kLaneM;
    const int tm = (warp % kWarpsM) * T::kLaneM + lane / T::kLaneN;
    const int tn = (warp / kWarpsM) * T::kLaneN + lane % T::kLaneN;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.z * kBN;
    const int chunk = blockIdx.x, k_begin = chunk * kc, k_end = min(K, k_begin + kc);
    const int tiles = k_end > k_begin ? (k_end - k_begin + kBK - 1) / kBK : 0;

    // thread t copies piece t % 8 of rows t / 8, t / 8 + 16, ... of either operand
    const int cr = t / 8, ck = (t % 8) * 4;
    auto load = [&](int tile) {
        if (tile < tiles) {
            float* s = smem + (tile % kStages) * T::kStage;
            const int k = k_begin + tile * kBK + ck;
            const bool in_k = k < k_end;
#pragma unroll
            for (int r = 0; r < (BM + 15) / 16; ++r) {
                const int row = cr + r * 16;
                if (BM >= 16 || row < BM) {
                    const bool ok = in_k && m0 + row < M;
                    copy16(s + row * kPad + ck, ok ? A + static_cast<size_t>(m0 + row) * lda + k : A, ok);
                }
            }
#pragma unroll
            for (int r = 0; r < kBN / 16; ++r) {
                const int row = cr + r * 16;
                const bool ok = in_k && n0 + row < N;
                copy16(s + (BM + row) * kPad + ck, ok ? W + static_cast<size_t>(n0 + row) * ldw + k : W, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    unsigned long long acc[8][T::kTN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < T::kTN; ++j) acc[i][j] = 0ull;

    for (int i = 0; i < kStages - 1; ++i) load(i);
    for (int tile = 0; tile < tiles; ++tile) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();                              // the tile is there for all, and all are done with the one before it
        load(tile + kStages - 1);
        const float* sa = smem + (tile % kStages) * T::kStage + tm * kPad;
        const float* sw = smem + (tile % kStages) * T::kStage + (BM + tn) * kPad;
#pragma unroll
        for (int k = 0; k < kBK; k += 4) {
            ulonglong2 a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(sa + i * T::kRowsT * kPad + k);
#pragma unroll
            for (int j = 0; j < T::kTN; ++j) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(sw + j * T::kColsT * kPad + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fma_pair(a[i].y, w.y, fma_pair(a[i].x, w.x, acc[i][j]));
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the chunk's sums [BM, kBN] in the ring's place
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < T::kTN; ++j) {
            const float even = __uint_as_float(static_cast<unsigned>(acc[i][j])), odd = __uint_as_float(static_cast<unsigned>(acc[i][j] >> 32));
            smem[(tm + i * T::kRowsT) * kBN + tn + j * T::kColsT] = even + odd;
        }
    const int chunks = gridDim.x;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    if (chunks > 1) cluster.sync();
    else __syncthreads();
    // CTA `chunk` finishes every chunks-th row of the block: the chunks' sums in their order
    const int n = n0 + t;
    for (int row = chunk; row < BM && m0 + row < M; row += chunks) {
        float v = 0.f;
        if (chunks > 1) {
            float part[kMaxChunks];
#pragma unroll
            for (int s = 0; s < kMaxChunks; ++s)
                if (s < chunks) part[s] = *cluster.map_shared_rank(smem + row * kBN + t, s);
            v = part[0];
#pragma unroll
            for (int s = 1; s < kMaxChunks; ++s)
                if (s < chunks) v += part[s];
        } else {
            v = smem[row * kBN + t];
        }
        if (n < N) {
            float* c = C + static_cast<size_t>(m0 + row) * ldc + n;
            *c = accumulate ? *c + v : v;
        }
    }
    if (chunks > 1) cluster.sync();                   // a CTA's sums stay until all have read them
}

template <int BM>
int launch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int chunks, int kc,
           int accumulate, cudaStream_t st) {
    static const cudaError_t ready = cudaFuncSetAttribute(gemm_f32_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          static_cast<int>(F32Tile<BM>::kSmem));
    if (ready != cudaSuccess) { set_error("gemm: %s", cudaGetErrorString(ready)); return 1; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(chunks, (M + BM - 1) / BM, (N + kBN - 1) / kBN);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = F32Tile<BM>::kSmem;
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
    cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BM>, A, W, C, M, N, K, lda, ldw, ldc, kc, accumulate);
    return check_launch("gemm_f32");
}

}  // namespace

// Rows of 16-byte pieces (copy16), blocks within the grid's limits.
bool gemm_f32_takes(const float* A, const float* W, int M, int N, int K, int lda, int ldw) {
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && aligned(A) && aligned(W) && (M + 63) / 64 <= 65535 && (N + kBN - 1) / kBN <= 65535;
}

int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate, cudaStream_t st) {
    // Chunks of K until the blocks along N fill the 148 SMs, none shorter than 256: by N and K alone (see above).
    int chunks = 1;
    while (chunks < kMaxChunks && (N + kBN - 1) / kBN * chunks < 148 && K / (2 * chunks) >= 256) chunks *= 2;
    const int kc = ((K + chunks - 1) / chunks + kBK - 1) / kBK * kBK;
    if (M <= 8) return launch<8>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, st);
    if (M <= 16) return launch<16>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, st);
    if (M <= 32) return launch<32>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, st);
    return launch<64>(A, W, C, M, N, K, lda, ldw, ldc, chunks, kc, accumulate, st);
}

}  // namespace gi
