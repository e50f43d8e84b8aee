// True 32-bit matrix product on the fifth-generation tensor cores:  C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]), 32-bit operands and result.
//
// A number is the sum of three bfloat16 ones to its last bit: the nearest, the nearest to what is left, and the rest (8 + 8 + 8 bits). Of the nine
// products of two such sums the six largest are taken; the others come to at most 2^-24 of the whole. Products of 8-bit numbers are exact in 32
// bits. `tcgen05.mma` drops bits below the last when it adds, so its chains are short: over 64 numbers the twenty small products first, the
// four large ones last, into an accumulator of their own, which is then added to 32-bit registers with ordinary rounding. Against 64
// bits results are nearer than those of the FMA kernel (gemm_f32.cu), whose chains are K long: figures at `b200_gemm_f32_split_takes`.
//
// A block computes 128 rows of W by TOKENS rows of A (D[row of W][token]: W is the MMA's 128-row side). Eight warps fetch 32-bit rows, 64
// numbers a stage, take them apart and store the parts K-major with 128-byte swizzle; one elected thread issues the 24 products of a
// stage; four warps add up the accumulators, two of which take turns in TMEM. An output's sums are the same whatever the tile, so a row's result
// does not depend on how many rows are in the call. Outputs that are not finite are made again as one chain of FMAs (`chain`).
//
// What bounds it: what an SM takes out of L2, 48 KB a stage at 128 x 64 and 64 KB at 128 x 128. Of 32 us for 500 rows by 2,048 x 1,536, a form
// that only fetches takes 25, the products and the taking apart the rest. Tried: two stages ahead in registers instead of one, no change; numbers by
// cp.async and W's parts in TMEM, 36 us (17,920 rows of W, 2,048 of A: 858 against 716).
// Every wait is bounded; a block that gives up sets the timeout bit, frees its TMEM and leaves.
#include "common.cuh"
#include "split_mma.cuh"

namespace {

constexpr int kRows = 128;      // rows of W a block: MMA M
constexpr int kBlockK = 64;     // numbers a stage: 128 bytes of a part, one swizzle row
constexpr int kMmaK = 16;
constexpr int kParts = 3;
constexpr int kFetchWarps = 8;  // warps 0-7 fetch, 8 issues (9-11 only give their registers away), 12-15 add up
constexpr int kAddWarp = 12;
constexpr int kFetchThreads = kFetchWarps * 32;
constexpr int kThreads = 512;
// Registers a thread of the three kinds of warps, out of 512 x 128 at launch.
constexpr int kFetchRegisters = 120, kIssueRegisters = 56, kAddRegisters = 208;
static_assert(2 * kFetchRegisters + kIssueRegisters + kAddRegisters <= 4 * 128, "more registers than the block was launched with");
constexpr long long kWaitCycles = 4000000000LL;  // about two seconds
constexpr int ERRBIT_TIMEOUT = 8;

__host__ __device__ constexpr int split_stages(int tokens) { return tokens <= 64 ? 3 : 2; }
__host__ __device__ constexpr uint32_t part_bytes(int rows) { return static_cast<uint32_t>(rows) * kBlockK * 2; }
__host__ __device__ constexpr uint32_t stage_bytes(int tokens) { return kParts * part_bytes(kRows + tokens); }
constexpr size_t split_smem(int tokens) { return static_cast<size_t>(split_stages(tokens)) * stage_bytes(tokens) + 1024; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory"); }
// Bounded wait for the phase with the given parity to complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_addr(bar);
  const long long start = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - start > kWaitCycles) return false;
  }
}
// Shared-memory matrix descriptor of a K-major tile with 128-byte rows and 128-byte swizzle: groups of 8 rows are 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t addr) {
  uint64_t desc = 0;
  desc |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
  desc |= static_cast<uint64_t>(1) << 16;
  desc |= static_cast<uint64_t>(1024 >> 4) << 32;
  desc |= static_cast<uint64_t>(1) << 46;  // descriptor version (sm_100)
  desc |= static_cast<uint64_t>(2) << 61;  // SWIZZLE_128B
  return desc;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate ? 1u : 0u)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_load_16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Operands are taken times 2^16, sums times 2^-32. Without that the third parts of numbers below 2^-110 fall under bfloat16's smallest one
// (relative error 1.5e-5 at 2^-118); with it every 32-bit number below 2^112 is its parts exactly, and what is larger, or a sum above 2^96, is made by `chain`.
constexpr float kOperandScale = 65536.f, kSumScale = 1.f / (65536.f * 65536.f);
__device__ __forceinline__ uint64_t pair(float lo, float hi) { return static_cast<uint64_t>(__float_as_uint(hi)) << 32 | __float_as_uint(lo); }
// Eight neighbouring numbers of a row, in parts, to piece `piece` of the row in the three tiles of parts.
__device__ __forceinline__ void store_parts(unsigned char* tile, uint32_t bytes, int row, int piece, float4 a, float4 b) {
  unsigned char* to = tile + row * 128 + ((piece ^ (row & 7)) << 4);
  // Two numbers an instruction, as a register pair.
  uint64_t v[4] = {pair(a.x, a.y), pair(a.z, a.w), pair(b.x, b.y), pair(b.z, b.w)};
#pragma unroll
  for (int i = 0; i < 4; ++i) asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v[i]) : "l"(v[i]), "l"(pair(kOperandScale, kOperandScale)));
#pragma unroll
  for (int p = 0; p < kParts; ++p) {
    uint32_t word[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      word[i] = pack_bf16(__uint_as_float(static_cast<uint32_t>(v[i])), __uint_as_float(static_cast<uint32_t>(v[i] >> 32)));
      if (p + 1 < kParts) asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v[i]) : "l"(v[i]), "l"(pair(__uint_as_float(word[i] << 16), __uint_as_float(word[i] & 0xffff0000u))));
    }
    *reinterpret_cast<uint4*>(to + p * bytes) = make_uint4(word[0], word[1], word[2], word[3]);
  }
}

struct SplitProduct {
  const float* A;
  const float* W;
  const float* bias;
  float* C;
  int M, N, K, lda, ldw, ldc;
  int* err;
};

__device__ __forceinline__ bool any_nan(float4 v) { return isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w); }
// An output as the FMA kernel makes it, where the sum of the products of parts is not finite: an infinite operand (whose parts are NaN), or a sum
// that passes the range on its way, may be the reason, and the output is infinite, or finite after all. Where a row has a NaN it stays NaN.
__device__ __noinline__ float chain(const SplitProduct& p, int m, int n) {
  const float* a = p.A + static_cast<int64_t>(m) * p.lda;
  const float* w = p.W + static_cast<int64_t>(n) * p.ldw;
  float sum = 0.f;
  for (int k = 0; k < p.K; k += 4) {
    const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
    sum = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, sum))));
  }
  return sum;
}

template <int TOKENS>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_split_kernel(const __grid_constant__ SplitProduct p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  constexpr int kStages = split_stages(TOKENS);
  constexpr uint32_t kColumns = 2 * TOKENS < 32 ? 32 : 2 * TOKENS;  // of TMEM: two accumulators; a power of two
  constexpr int kWItems = kRows * 8 / kFetchThreads, kAItems = TOKENS * 8 >= kFetchThreads ? TOKENS * 8 / kFetchThreads : 1;
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages], sum_full[2], sum_empty[2];
  __shared__ uint32_t tmem_base_shared;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kRows, m0 = blockIdx.y * TOKENS;
  const int steps = (p.K + kBlockK - 1) / kBlockK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&full_bar[s], kFetchWarps), mbar_init(&empty_bar[s], 1);
    for (int b = 0; b < 2; ++b) mbar_init(&sum_full[b], 1), mbar_init(&sum_empty[b], 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kFetchWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_shared)), "r"(kColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_shared;
  wait_for_predecessor();
  let_successor_start();

  if (warp < kFetchWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFetchRegisters));
    // ---- fetch: eight lanes a row, eight numbers a lane; a stage's numbers are on the way while the one before is taken apart ----
    const int piece = threadIdx.x & 7, row0 = threadIdx.x >> 3;  // rows row0, row0 + 32, ..
    const bool takes_a = TOKENS * 8 >= kFetchThreads || row0 < TOKENS;
    float4 w[kWItems][2], a[kAItems][2];
    const float* w_at = p.W + static_cast<int64_t>(n0 + row0) * p.ldw + piece * 8;  // of the stage that is fetched next
    const float* a_at = p.A + static_cast<int64_t>(m0 + row0) * p.lda + piece * 8;
    const int64_t w_step = 32LL * p.ldw, a_step = 32LL * p.lda;
    const int w_rows = p.N - n0 - row0, a_rows = takes_a ? p.M - m0 - row0 : 0;  // row 32 i is one if above 32 i
    int left = p.K - piece * 8;
    auto fetch = [&](float4 (&to)[2], const float* from, bool valid) {
#pragma unroll
      for (int h = 0; h < 2; ++h) to[h] = valid && left > 4 * h ? *reinterpret_cast<const float4*>(from + 4 * h) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto fetch_w = [&](int i) { fetch(w[i], w_at + i * w_step, w_rows > 32 * i); };
    auto fetch_a = [&](int i) { fetch(a[i], a_at + i * a_step, a_rows > 32 * i); };
    auto go_on = [&] { w_at += kBlockK, a_at += kBlockK, left -= kBlockK; };
    auto fetch_all = [&] {
#pragma unroll
      for (int i = 0; i < kWItems; ++i) fetch_w(i);
#pragma unroll
      for (int i = 0; i < kAItems; ++i) fetch_a(i);
    };
    fetch_all(), go_on();
    for (int step = 0; step < steps; ++step) {
      const int s = step % kStages;
      if (step >= kStages && !mbar_wait(&empty_bar[s], (step / kStages - 1) & 1)) {
        if (lane == 0) atomicOr(p.err, ERRBIT_TIMEOUT);
        break;
      }
      unsigned char* stage = tiles + static_cast<size_t>(s) * stage_bytes(TOKENS);
      // The next stage's numbers are asked for as soon as registers are free (none past K); behind all stores in blocks of sixteen tokens, since a launch may
      // have few of those and each then waits for its own stores behind the loads (1 row, 128 x 8,960: 105 us, early 115). Larger tiles are taken
      // where there are blocks for most SMs (early and behind: 500 rows, 17,920 x 1,536 172 and 182 us, 100 rows, 1,536 x 8,960 127 and 130).
      constexpr bool kEarly = TOKENS >= 32;
#pragma unroll
      for (int i = 0; i < kWItems; ++i) {
        store_parts(stage, part_bytes(kRows), row0 + 32 * i, piece, w[i][0], w[i][1]);
        if (kEarly) fetch_w(i);
      }
#pragma unroll
      for (int i = 0; i < kAItems; ++i) {
        if (takes_a) store_parts(stage + kParts * part_bytes(kRows), part_bytes(TOKENS), row0 + 32 * i, piece, a[i][0], a[i][1]);
        if (kEarly) fetch_a(i);
      }
      if (kEarly) go_on();
      else if (step + 1 < steps) fetch_all(), go_on();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[s]);
    }
  } else if (warp < kAddWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegisters));
    if (warp == kFetchWarps) {
      // ---- issue: the whole warp walks the loop, one elected lane issues ----
      uint32_t chosen;
      asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(chosen));
      const bool leader = chosen != 0;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(TOKENS >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24);
      const uint64_t w_first = umma_smem_desc(smem_addr(tiles)), a_first = umma_smem_desc(smem_addr(tiles) + kParts * part_bytes(kRows));
      for (int step = 0; step < steps; ++step) {
        const int s = step % kStages, b = step & 1;
        if (!mbar_wait(&full_bar[s], (step / kStages) & 1) || (step >= 2 && !mbar_wait(&sum_empty[b], (step / 2 - 1) & 1))) {
          if (leader) atomicOr(p.err, ERRBIT_TIMEOUT);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader) {
          constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
          const uint64_t stage_units = static_cast<uint64_t>(s) * (stage_bytes(TOKENS) >> 4);
#pragma unroll
          for (int x = 0; x < 6; ++x)
#pragma unroll
            for (int k = 0; k < kBlockK / kMmaK; ++k) {
              const uint64_t at = stage_units + static_cast<uint64_t>(k * (kMmaK * 2 >> 4));
              umma_bf16(tmem_base + b * TOKENS, w_first + at + order[x][0] * (part_bytes(kRows) >> 4), a_first + at + order[x][1] * (part_bytes(TOKENS) >> 4), idesc,
                        x > 0 || k > 0);
            }
          umma_commit(&empty_bar[s]);
          umma_commit(&sum_full[b]);
        }
        __syncwarp();
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kAddRegisters));
    // ---- add up: TMEM lanes 32 * quarter .. + 31 are rows of W, columns are tokens ----
    const int quarter = warp & 3;  // a warp reads the lanes of its place among four
    const int n = n0 + quarter * 32 + lane;
    float sum[TOKENS];
#pragma unroll
    for (int i = 0; i < TOKENS; ++i) sum[i] = 0.f;
    bool have = true;
    for (int step = 0; step < steps; ++step) {
      const int b = step & 1;
      if (!mbar_wait(&sum_full[b], (step / 2) & 1)) {
        if (lane == 0) atomicOr(p.err, ERRBIT_TIMEOUT);
        have = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < TOKENS; c += 16) {
        float part[16];
        tmem_load_16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + b * TOKENS + c, part);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[c + i] += part[i];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&sum_empty[b]);
    }
    uint32_t odd[(TOKENS + 31) / 32] = {};  // tokens whose sum is not finite
    const float more = p.bias != nullptr && n < p.N ? p.bias[n] : 0.f;
    if (have && n < p.N) {
#pragma unroll
      for (int i = 0; i < TOKENS; ++i) {
        if (m0 + i >= p.M) break;
        if (!isfinite(sum[i])) odd[i / 32] |= 1u << (i % 32);
        p.C[static_cast<int64_t>(m0 + i) * p.ldc + n] = fmaf(sum[i], kSumScale, more);
      }
    }
    __syncwarp();
    bool looked = false, spoilt = false;  // at the lane's row of W; that has a NaN
#pragma unroll
    for (int word = 0; word < (TOKENS + 31) / 32; ++word)
      for (uint32_t any = __reduce_or_sync(0xffffffffu, odd[word]); any != 0; any &= any - 1) {
        const int bit = __ffs(any) - 1, m = m0 + word * 32 + bit;
        bool nan = false;
        for (int k = lane * 4; k < p.K; k += 128) nan |= any_nan(*reinterpret_cast<const float4*>(p.A + static_cast<int64_t>(m) * p.lda + k));
        if (__any_sync(0xffffffffu, nan) || !(odd[word] >> bit & 1)) continue;  // NaN it stays
        if (!looked) {
          looked = true;
          for (int k = 0; k < p.K; k += 4) spoilt |= any_nan(*reinterpret_cast<const float4*>(p.W + static_cast<int64_t>(n) * p.ldw + k));
        }
        if (!spoilt) p.C[static_cast<int64_t>(m) * p.ldc + n] = chain(p, m, n) + more;
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kFetchWarps) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kColumns) : "memory");
}

template <int TOKENS>
int launch_tokens(const SplitProduct& p, cudaStream_t stream) {
  static OncePerDevice raised;
  if (!raised([] { return cudaFuncSetAttribute(gemm_f32_split_kernel<TOKENS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(split_smem(TOKENS))) == cudaSuccess; }))
    return b200_fail("gemm_f32_split: cannot size shared memory");
  const dim3 grid((p.N + kRows - 1) / kRows, (p.M + TOKENS - 1) / TOKENS);
  B200_REQUIRE(grid.y <= 65535, "gemm_f32_split: too many rows (%d)", p.M);
  launch_kernel(gemm_f32_split_kernel<TOKENS>, grid, dim3(kThreads), split_smem(TOKENS), stream, p);
  return b200_check_launch("gemm_f32_split");
}

}  // namespace

// Whether this kernel takes a product, by its matrix alone, so that all calls with one matrix sum alike. Measured on a B200 (N x K, rows; us;
// FMA kernel and this one; error against 64 bits): 2,048 x 1,536: 1 row 41 and 22, 100 rows 68 and 24, 500 rows 108 and 34, 2,048 rows 313 and 85 (7.0e-7 and
// 1.2e-7); 17,920 x 1,536: 16 rows 60 and 33, 500 rows 701 and 179, 2,048 rows 2,634 and 716; 1,536 x 8,960: 1 row 220 and 110, 500 rows 601
// and 178 (1.7e-6 and 2.3e-7). Level, at what a launch takes, for 128 x 256 up to 500 rows (2,048 rows 15 and 11); 4,096 x 64 at
// 2,048 rows 34 and 35.
B200_API int b200_gemm_f32_split_takes(int N, int K) { return N >= 128 && K >= 256 && K % 4 == 0 ? 1 : 0; }

// `tokens`: 16, 32, 64 or 128 rows of A a block; 0: by the sizes.
B200_API int b200_gemm_f32_split(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int tokens, int* err,
                                 cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  B200_REQUIRE(M > 0 && N > 0 && K > 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0, "gemm_f32_split: bad sizes %d x %d x %d", M, N, K);
  B200_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32_split: leading dimensions too small");
  B200_REQUIRE(reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(W) % 16 == 0, "gemm_f32_split: operands must be 16-byte aligned");
  const SplitProduct p = {A, W, bias, C, M, N, K, lda, ldw, ldc, err};
  if (tokens == 0) {
    // The tile that is done first: as many waves of blocks as the SMs need, a wave as long as one tile takes (2,048 x 1,536).
    constexpr int tiles[4] = {16, 32, 64, 128}, times[4] = {23, 26, 33, 41};
    int64_t best = 0;
    for (int i = 0; i < 4; ++i) {
      const int64_t blocks = static_cast<int64_t>((N + kRows - 1) / kRows) * ((M + tiles[i] - 1) / tiles[i]), sms = b200_sm_count_host();
      const int64_t time = (blocks + sms - 1) / sms * times[i];
      if (i == 0 || time < best) best = time, tokens = tiles[i];
    }
  }
  if (tokens == 16) return launch_tokens<16>(p, stream);
  if (tokens == 32) return launch_tokens<32>(p, stream);
  if (tokens == 64) return launch_tokens<64>(p, stream);
  B200_REQUIRE(tokens == 128, "gemm_f32_split: tiles of 16, 32, 64 or 128 rows");
  return launch_tokens<128>(p, stream);
}
