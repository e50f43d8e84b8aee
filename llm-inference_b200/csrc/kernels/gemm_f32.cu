// True 32-bit matrix product for the float32 path:  C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]); matrices that `b200_gemm_f32_split_takes`
// names go to the kernel in gemm_f32_split.cu instead.
//
// Plain FMA on CUDA cores: no tensor cores, no TF32, no split accumulation. Each output
// element is one chain of FMAs over k = 0..K-1 in order, so a row's result does not depend on
// how many other rows are in the call, nor on the tile that computed it. Linear layers are x * W^T with W stored
// [out_features, in_features] (python/instinct/backends/base.py:83-101).
//
// What bounds it: an SM issues 128 FMAs a cycle and takes 32 numbers a cycle out of shared memory, however many lanes want the
// same one, so a thread should do up to four FMAs per number it reads: 8 x 4 outputs a thread (12 numbers for 32 FMAs). Both operands
// keep their rows in shared memory (k runs along them), so tiles arrive by cp.async, three stages deep, and a thread reads four
// k of a row at once; its rows and columns are spread over the tile so that neighbouring lanes read rows 4 banks apart.
#include "common.cuh"

namespace {

constexpr int BK = 32, kLd = BK + 4, kStages = 3;

template <int kBytes>
__device__ __forceinline__ void stage_copy(float* smem, const float* gmem, bool valid) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? kBytes : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(kBytes), "r"(bytes) : "memory");
}

// Rows row0 .. row0 + ROWS of src [rows][ld], k0 .. k0 + BK, zeros outside; W numbers a copy.
template <int ROWS, int THREADS, int W>
__device__ __forceinline__ void stage_tile(float* dst, const float* src, int rows, int64_t ld, int K, int row0, int k0) {
  constexpr int kPerRow = BK / W;
#pragma unroll 4
  for (int idx = threadIdx.x; idx < ROWS * kPerRow; idx += THREADS) {
    const int r = idx / kPerRow, k = idx % kPerRow * W;
    const bool valid = row0 + r < rows && k0 + k < K;
    stage_copy<4 * W>(dst + r * kLd + k, valid ? src + (row0 + r) * ld + k0 + k : src, valid);
  }
}

template <int BM, int BN>
constexpr size_t tile_smem() {
  return sizeof(float) * kStages * (BM + BN) * kLd;
}

template <int BM, int BN, int TM, int TN, int W>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ Wt, const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K,
                int lda, int ldw, int ldc, int64_t batch_a, int64_t batch_w, int64_t batch_c) {
  extern __shared__ __align__(16) float gemm_smem[];
  constexpr int kRowThreads = BM / TM, kColThreads = BN / TN, kThreads = kRowThreads * kColThreads, kStage = (BM + BN) * kLd;
  // One product per blockIdx.z: the operands of product b start b strides further on.
  A += blockIdx.z * batch_a;
  Wt += blockIdx.z * batch_w;
  C += blockIdx.z * batch_c;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tc = threadIdx.x % kColThreads, tr = threadIdx.x / kColThreads;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  const int steps = (K + BK - 1) / BK;
  auto fetch = [&](int step) {
    if (step < steps) {
      float* stage = gemm_smem + step % kStages * kStage;
      stage_tile<BM, kThreads, W>(stage, A, M, lda, K, m0, step * BK);
      stage_tile<BN, kThreads, W>(stage + BM * kLd, Wt, N, ldw, K, n0, step * BK);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) fetch(s);
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    fetch(step + kStages - 1);  // into the stage that everybody has left
    const float* as = gemm_smem + step % kStages * kStage + tr * kLd;
    const float* ws = gemm_smem + step % kStages * kStage + BM * kLd + tc * kLd;
#pragma unroll 2
    for (int k = 0; k < BK; k += 4) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * kRowThreads * kLd + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * kColThreads * kLd + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + tr + i * kRowThreads;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tc + j * kColThreads;
      if (n < N) C[static_cast<int64_t>(m) * ldc + n] = acc[i][j] + (bias ? bias[n] : 0.f);
    }
  }
}

struct Product {
  const float* A;
  const float* W;
  const float* bias;
  float* C;
  int M, N, K, lda, ldw, ldc, batch;
  int64_t stride_a, stride_w, stride_c;
};

template <int BM, int BN, int TM, int TN>
int launch_tiles(const Product& p, bool wide, cudaStream_t stream) {
  constexpr size_t smem = tile_smem<BM, BN>();
  static OncePerDevice raised;
  if (!raised([] {
        return cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess &&
               cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess;
      }))
    return b200_fail("gemm_f32: cannot size shared memory");
  const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, p.batch);
  B200_REQUIRE(grid.y <= 65535, "gemm_f32: too many rows (%d)", p.M);
  auto kernel = wide ? gemm_f32_kernel<BM, BN, TM, TN, 4> : gemm_f32_kernel<BM, BN, TM, TN, 1>;
  kernel<<<grid, (BM / TM) * (BN / TN), smem, stream>>>(p.A, p.W, p.bias, p.C, p.M, p.N, p.K, p.lda, p.ldw, p.ldc, p.stride_a, p.stride_w, p.stride_c);
  return b200_check_launch("gemm_f32");
}

// Tiles of 64 x 64 outputs, 8 x 4 a thread, where there are enough of them for every SM; tiles of 16 x 32, 2 x 4 a thread, for few rows and
// wherever they come to at most three an SM: each tile walks all of K, so a product of few tiles takes the time of one tile's walk, which
// is the shorter the fewer outputs it has. Measured on a B200 (N x K, rows; us; in brackets the other tile), at sizes that the
// tensor cores do not take:
//   64 x 1,536:     1 row 38 (64 x 64: 63), 500 rows 39 (65), 2,048 rows 43 (65)
//   2,048 x 1,537:  1 row 60 (90), 33 rows 63 (90), 100 rows 90 (16 x 32: 83), 500 rows 138 (16 x 32: 224), 2,048 rows 436 (828)
//   17,920 x 128:   16 rows 6.7 (64 x 64: 10.7), 33 rows 11.1 (16 x 32: 14.3), 500 rows 64 (112), 2,048 rows 236 (435)
//   4,096 x 64:     1 row 3.1 (64 x 64: 4.3), 33 rows 3.9 (4.6), 100 rows 5.0 (16 x 32: 5.6), 500 rows 10.6 (16), 2,048 rows 31 (55)
//   12 heads, 512 x 128 each: 16 rows 5.1 (64 x 64: 7.4), 33 rows 7.5 (16 x 32: 6.6), 100 rows 11 (11.5), 2,048 rows 83 (152)
// Tiles of 128 x 128 and 64 x 128 with 8 x 8 a thread were slower throughout (2,735 and 2,709 us for 2,048 rows of 17,920 x 1,536).
int launch_product(const Product& p, cudaStream_t stream) {
  const bool wide = p.K % 4 == 0 && p.lda % 4 == 0 && p.ldw % 4 == 0 && p.stride_a % 4 == 0 && p.stride_w % 4 == 0 &&
                    reinterpret_cast<uintptr_t>(p.A) % 16 == 0 && reinterpret_cast<uintptr_t>(p.W) % 16 == 0;
  const int64_t small_tiles = static_cast<int64_t>((p.M + 15) / 16) * ((p.N + 31) / 32) * p.batch;
  if (p.M <= 16 || small_tiles <= 3 * b200_sm_count_host()) return launch_tiles<16, 32, 2, 4>(p, wide, stream);
  return launch_tiles<64, 64, 8, 4>(p, wide, stream);
}

}  // namespace

B200_API int b200_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M,
                           int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32: bad sizes %d x %d x %d", M, N, K);
  B200_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: leading dimensions too small");
  return launch_product({A, W, bias, C, M, N, K, lda, ldw, ldc, 1, 0, 0, 0}, stream);
}

// `batch` products of the same shape in one launch: C_b = A_b * W_b^T, each operand's b-th
// matrix `stride_*` elements after the first (a head's slice of a wider row, for instance).
B200_API int b200_gemm_f32_batched(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                                   int batch, int64_t stride_a, int64_t stride_w, int64_t stride_c, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  B200_REQUIRE(M > 0 && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm_f32_batched: bad sizes %d x %d x %d x %d", batch, M,
               N, K);
  B200_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32_batched: leading dimensions too small");
  return launch_product({A, W, nullptr, C, M, N, K, lda, ldw, ldc, batch, stride_a, stride_w, stride_c}, stream);
}
