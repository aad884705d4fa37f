// C[M, N] = A[M, K] * W[N, K]^T in true 32-bit: FMA on the CUDA cores, no tensor cores, no TF32.
//
// This is the matrix product of the 32-bit path (the reference leaves the TF32 switch to PyTorch's
// global flags, utils/attention.py:119-124; here the 32-bit path cannot use reduced precision at
// all).  Each output element is one thread's running sum over k = 0 .. K-1 in ascending order, so a
// row's result does not depend on how many other rows the call has: the 32-bit path gives
// bit-identical activations however a prompt is cut.
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;  // 256 threads, 4x4 outputs each
}

__global__ void __launch_bounds__(256) gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w,
                                                       float* __restrict__ c, int m_total, int n_total, int k_total,
                                                       int lda, int ldw, int ldc) {
    pdl_trigger();   // let the next kernel start launching
    pdl_wait();      // everything before this kernel in the stream is complete and visible
    __shared__ float a_tile[BK][BM + 4];
    __shared__ float w_tile[BK][BN + 4];
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int thread = threadIdx.x;
    const int row_group = thread / 16, col_group = thread % 16;  // outputs (row_group*4.., col_group*4..)
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

    const int load_k = thread % BK, load_row = thread / BK;  // 16 rows per pass, 4 passes
    for (int k0 = 0; k0 < k_total; k0 += BK) {
#pragma unroll
        for (int pass = 0; pass < BM / 16; ++pass) {
            const int row = load_row + pass * 16;
            const int k = k0 + load_k;
            const int gm = m0 + row, gn = n0 + row;
            a_tile[load_k][row] = (gm < m_total && k < k_total) ? a[(size_t)gm * lda + k] : 0.0f;
            w_tile[load_k][row] = (gn < n_total && k < k_total) ? w[(size_t)gn * ldw + k] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a_values[TM], w_values[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a_values[i] = a_tile[k][row_group * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w_values[j] = w_tile[k][col_group * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a_values[i], w_values[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + row_group * TM + i;
        if (gm >= m_total) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + col_group * TN + j;
            if (gn < n_total) c[(size_t)gm * ldc + gn] = acc[i][j];
        }
    }
}

// The same product for few rows (M <= 32), where a launch is the latency of its loads and not arithmetic: a block owns 32
// columns, the columns are a warp's lanes and the rows are dealt to four warps, ROWS each.  W goes through shared memory in
// pieces of 128 along K, three of them in flight; where the caller says that W is a weight, which the kernel in front does not
// write, the first three are asked for before that kernel has ended.  Every output is still one thread's running sum over
// ascending k, so the results are those of the kernel above bit for bit.  Few rows / tiles of 64 x 64, us: W [4096, 4096] 28 / 354 at 1
// row, 39 / 338 at 8, 46 / 346 at 16, 79 / 349 at 32; [1024, 4096] 27 / 322, 37 / 341, 45 / 348, 77 / 354; [24576, 4096] 129 / 656, 136 / 658,
// 195 / 659, 333 / 663; [4096, 12288] 81 / 1069, 113 / 1021, 136 / 1039, 232 / 1066; [1024, 1024] 7 / 80, 10 / 85, 12 / 86, 20 / 88.
namespace {
constexpr int kColumns = 32, kPiece = 128, kPitch = kPiece + 4, kDeep = 3, kFewThreads = 128, kFewRows = 32;

__device__ __forceinline__ void copy16(float* to, const float* from, bool present) {
    const int bytes = present ? 16 : 0;      // 0: the 16 bytes are filled with zeros and nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }
}  // namespace

template <int ROWS>
__global__ void __launch_bounds__(kFewThreads) gemm_f32_few_rows_kernel(const float* __restrict__ a, const float* __restrict__ w,
                                                                        float* __restrict__ c, int m_total, int n_total, int k_total,
                                                                        int lda, int ldw, int ldc, int w_settled) {
    pdl_trigger();   // let the next kernel start launching
    if (!w_settled) pdl_wait();
    extern __shared__ __align__(16) float stages[];      // [kDeep]{ W [kColumns][kPitch], rows [4 ROWS][kPitch] }
    constexpr int kStage = (kColumns + 4 * ROWS) * kPitch, kVectors = kPiece / 4;
    const int n0 = blockIdx.x * kColumns;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pieces = (k_total + kPiece - 1) / kPiece;

    auto load_w = [&](int piece) {
        float* to = stages + piece % kDeep * kStage;
        const int k = piece * kPiece + lane * 4;
#pragma unroll
        for (int column = warp; column < kColumns; column += kFewThreads / kVectors) {
            const bool present = n0 + column < n_total && k < k_total;
            copy16(to + column * kPitch + lane * 4, present ? w + (size_t)(n0 + column) * ldw + k : w, present);
        }
    };
    auto load_rows = [&](int piece) {
        float* to = stages + piece % kDeep * kStage + kColumns * kPitch;
        const int k = piece * kPiece + lane * 4;
#pragma unroll
        for (int row = warp; row < 4 * ROWS; row += kFewThreads / kVectors) {
            const bool present = row < m_total && k < k_total;
            copy16(to + row * kPitch + lane * 4, present ? a + (size_t)row * lda + k : a, present);
        }
    };

    for (int piece = 0; piece < kDeep && piece < pieces; ++piece) load_w(piece);
    pdl_wait();      // everything before this kernel in the stream is complete and visible
#pragma unroll
    for (int piece = 0; piece < kDeep; ++piece) {
        if (piece < pieces) load_rows(piece);
        copy_commit();
    }
    float sums[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) sums[r] = 0.0f;
    for (int piece = 0; piece < pieces; ++piece) {
        copy_wait<kDeep - 1>();
        __syncthreads();
        const float* column = stages + piece % kDeep * kStage + lane * kPitch;
        const float* rows = stages + piece % kDeep * kStage + (kColumns + warp * ROWS) * kPitch;
#pragma unroll 8
        for (int k = 0; k < kPiece; k += 4) {      // past the end of K both factors are zero
            const float4 right = *reinterpret_cast<const float4*>(column + k);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const float4 left = *reinterpret_cast<const float4*>(rows + r * kPitch + k);
                sums[r] = fmaf(left.w, right.w, fmaf(left.z, right.z, fmaf(left.y, right.y, fmaf(left.x, right.x, sums[r]))));
            }
        }
        __syncthreads();
        if (piece + kDeep < pieces) {
            load_w(piece + kDeep);
            load_rows(piece + kDeep);
        }
        copy_commit();
    }
    if (n0 + lane < n_total) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
            if (warp * ROWS + r < m_total) c[(size_t)(warp * ROWS + r) * ldc + n0 + lane] = sums[r];
    }
}

template <int ROWS>
static int few_rows_launch(const float* a, const float* w, float* c, int m, int n, int k, int lda, int ldw, int ldc, int w_settled, cudaStream_t stream) {
    const size_t shared = (size_t)kDeep * (kColumns + 4 * ROWS) * kPitch * sizeof(float);
    if (int status = llm_raise_shared_limit(reinterpret_cast<const void*>(gemm_f32_few_rows_kernel<ROWS>), shared, "gemm_f32")) return status;
    llm_launch(gemm_f32_few_rows_kernel<ROWS>, dim3((unsigned)((n + kColumns - 1) / kColumns)), kFewThreads, shared, stream, a, w, c, m, n, k,
               lda, ldw, ldc, w_settled);
    return llm_check_launch("gemm_f32");
}

// w_settled: the caller vouches that no kernel which may still be running writes w (it is a model's weight).
LLM_EXPORT int llm_gemm_f32(const float* a, const float* w, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                            int w_settled, cudaStream_t stream) {
    if (m == 0 || n == 0) return LLM_OK;
    // few rows whose 16-byte pieces are aligned and whole; any other product runs in tiles of 64 x 64
    if (m <= kFewRows && k > 0 && k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && aligned16(a) && aligned16(w)) {
        if (m <= 4) return few_rows_launch<1>(a, w, c, m, n, k, lda, ldw, ldc, w_settled, stream);
        if (m <= 8) return few_rows_launch<2>(a, w, c, m, n, k, lda, ldw, ldc, w_settled, stream);
        if (m <= 16) return few_rows_launch<4>(a, w, c, m, n, k, lda, ldw, ldc, w_settled, stream);
        return few_rows_launch<8>(a, w, c, m, n, k, lda, ldw, ldc, w_settled, stream);
    }
    const int blocks_m = (m + BM - 1) / BM;
    if ((n + BN - 1) / BN > 65535) {
        llm_set_error("gemm_f32: at most %d output columns per launch, got %d", 65535 * BN, n);
        return LLM_REFUSED;
    }
    dim3 grid(blocks_m, (n + BN - 1) / BN);
    llm_launch(gemm_f32_kernel, grid, 256, 0, stream, a, w, c, m, n, k, lda, ldw, ldc);
    return llm_check_launch("gemm_f32");
}
