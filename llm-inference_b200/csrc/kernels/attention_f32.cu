// Attention of prompt portions over the paged cache in 32 bits: the tiled form of the plain kernel (attention_plain.cu).
//
// One block takes 32 rows of one kv head, a row being a (token, query head) pair of a request, token by token with the query heads
// that share the kv head side by side, and walks the request's keys 64 at a time: scores as a 32 x 64 product, the running softmax,
// then the weighted sum of values as a 32 x head_dim product, everything 32-bit FMAs. Keys and values come by cp.async, the values
// while the scores are formed and the next keys while the values are summed. A row's result does not depend on what else is in the
// call beyond the order in which its keys' tiles begin. Windows and a sink (a start value of maximum and sum) are taken; other
// shapes of scores, kept first keys and single tokens run the plain kernel.
//
// What bounds it: operands out of shared memory, 2 (scores) and 2.7 (values) FMAs per number. The plain kernel reads every key row
// once per (token, head) and forms one score a thread. Measured on a B200 (500 tokens, 12 heads of 128 on 2 kv heads, one request):
// 325 -> 88 us; 2,048 tokens 4,545 -> 501 us, behind 4,000 others 22.2 -> 2.4 ms.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int kRows = 32, kKeys = 64, kThreads = 128;
constexpr int kLdP = kKeys + 4;

__device__ __forceinline__ void stage_copy(float* smem, const float* gmem, bool valid) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}

struct PortionParams {
  const float* q;
  const float* keys;
  const float* values;
  const int* block_table;
  const int* seq_q_start;
  const int* seq_q_len;
  const int* seq_kv_len;
  const float* sink;  // [q_heads] or null
  float* out;
  int* err;
  int first_seq, max_pages, num_pages, q_heads, kv_heads, head_dim, page_size, window;
  float scale;
};

constexpr size_t portion_smem(int dim) {
  return sizeof(float) * (kRows * (dim + 4) + 2 * kKeys * (dim + 4) + kRows * kLdP + kRows) + 2 * kKeys * sizeof(int64_t);
}

template <int DIM>
__global__ void __launch_bounds__(kThreads)
portion_attention_f32_kernel(const PortionParams p) {
  extern __shared__ __align__(16) float attention_smem[];
  constexpr int kLd = DIM + 4;
  constexpr int kColGroups = DIM / 4, kRowGroups = kThreads / kColGroups, kOwnRows = kRows / kRowGroups;  // of the values' product
  float* qs = attention_smem;         // [kRows][kLd]
  float* ks = qs + kRows * kLd;       // [kKeys][kLd]
  float* vs = ks + kKeys * kLd;       // [kKeys][kLd]
  float* ps = vs + kKeys * kLd;       // [kRows][kLdP]
  float* alphas = ps + kRows * kLdP;  // [kRows]: factor of the running output; at the end 1 / sum
  int64_t* offsets = reinterpret_cast<int64_t*>(alphas + kRows);  // [2][kKeys]: rows of two tiles, -1: not to be read
  const int seq = p.first_seq + blockIdx.z, kvh = blockIdx.y;
  const int group = p.q_heads / p.kv_heads;
  const int len = p.seq_q_len[seq], start = p.seq_q_start[seq], begin = p.seq_kv_len[seq] - len;  // begin: position of the first new token
  const int row_blocks = (len * group + kRows - 1) / kRows;
  const int block = row_blocks - 1 - static_cast<int>(blockIdx.x);  // the rows with most keys first
  if (block < 0) return;
  const int row0 = block * kRows, rows = min(kRows, len * group - row0);
  const int tid = threadIdx.x;
  const int* table = p.block_table + static_cast<int64_t>(seq) * p.max_pages;
  const int last_pos = begin + (row0 + rows - 1) / group, first_pos = begin + row0 / group;
  const int lo = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
  const int tiles = (last_pos - lo) / kKeys + 1;
  auto look_up = [&](int tile) {  // where the tile's rows are
    if (tid < kKeys) {
      const int j = lo + tile * kKeys + tid;
      int64_t offset = -1;
      if (tile < tiles && j <= last_pos) {
        const int logical = j / p.page_size;
        const int page = logical < p.max_pages ? table[logical] : -1;
        if (page < 0 || page >= p.num_pages) atomicOr(p.err, ERRBIT_BAD_PAGE);
        else offset = kv_row_offset(page, kvh, j % p.page_size, p.kv_heads, p.page_size, p.head_dim);
      }
      offsets[(tile & 1) * kKeys + tid] = offset;
    }
  };
  auto fetch = [&](float* to, const float* arena, int tile) {
    for (int idx = tid; idx < kKeys * (DIM / 4); idx += kThreads) {
      const int r = idx / (DIM / 4), c = idx % (DIM / 4) * 4;
      const int64_t offset = offsets[(tile & 1) * kKeys + r];
      const bool valid = offset >= 0 && c < p.head_dim;
      stage_copy(to + r * kLd + c, valid ? arena + offset + c : arena, valid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int idx = tid; idx < kRows * (DIM / 4); idx += kThreads) {
    const int r = idx / (DIM / 4), c = idx % (DIM / 4) * 4;
    const int item = row0 + r, token = item / group, head = kvh * group + item % group;
    const bool valid = r < rows && c < p.head_dim;
    stage_copy(qs + r * kLd + c, valid ? p.q + (static_cast<int64_t>(start + token) * p.q_heads + head) * p.head_dim + c : p.q, valid);
  }
  look_up(0);
  __syncthreads();
  fetch(ks, p.keys, 0);  // its group holds the queries too
  const int tc = tid & 15, tr = tid >> 4;                  // scores: rows tr, tr + 8, .., keys tc, tc + 16, ..
  const int cg = tid % kColGroups, rg = tid / kColGroups;  // values: rows rg, rg + kRowGroups, .., dims 4 cg .. + 3
  float top[4], sum[4];
  int pos[4], from[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int item = row0 + tr + 8 * i;
    pos[i] = tr + 8 * i < rows ? begin + item / group : -1;
    from[i] = p.window > 0 ? pos[i] - p.window + 1 : 0;
    const float* sink = p.sink ? p.sink + kvh * group + item % group : nullptr;
    top[i] = sink ? *sink : -INFINITY;
    sum[i] = sink ? 1.f : 0.f;
  }
  float acc[kOwnRows][4];
#pragma unroll
  for (int i = 0; i < kOwnRows; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  for (int tile = 0; tile < tiles; ++tile) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the keys are there; nobody reads the values any more
    fetch(vs, p.values, tile);
    look_up(tile + 1);
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll 4
    for (int c = 0; c < DIM; c += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        a[x] = *reinterpret_cast<const float4*>(qs + (tr + 8 * x) * kLd + c);
        b[x] = *reinterpret_cast<const float4*>(ks + (tc + 16 * x) * kLd + c);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
    }
    const int64_t* tile_rows = offsets + (tile & 1) * kKeys;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float best = -INFINITY;
      bool seen[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = lo + tile * kKeys + tc + 16 * j;
        seen[j] = key <= pos[i] && key >= from[i] && tile_rows[tc + 16 * j] >= 0;
        s[i][j] = seen[j] ? s[i][j] * p.scale : -INFINITY;
        best = fmaxf(best, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
      const float new_top = fmaxf(top[i], best);
      const float alpha = top[i] > -INFINITY ? expf(top[i] - new_top) : 0.f;
      float part = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float weight = seen[j] && new_top > -INFINITY ? expf(s[i][j] - new_top) : 0.f;
        ps[(tr + 8 * i) * kLdP + tc + 16 * j] = seen[j] ? weight : -0.f;  // a minus sign marks what the row does not see
        part += weight;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      sum[i] = sum[i] * alpha + part;
      top[i] = new_top;
      if (tc == 0) alphas[tr + 8 * i] = alpha;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // weights and values are there, the next tile's rows looked up, the keys read
    if (tile + 1 < tiles) fetch(ks, p.keys, tile + 1);
#pragma unroll
    for (int i = 0; i < kOwnRows; ++i) {
      const float alpha = alphas[rg + kRowGroups * i];
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[i][x] *= alpha;
    }
    // Where some row does not see some key, such a key's value stays out even if it is not finite.
    const bool whole = lo + (tile + 1) * kKeys - 1 <= first_pos && (p.window == 0 || lo + tile * kKeys >= last_pos - p.window + 1);
    auto add_values = [&](auto masked) {
#pragma unroll 4
      for (int j = 0; j < kKeys; j += 4) {
        float4 v[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) v[x] = *reinterpret_cast<const float4*>(vs + (j + x) * kLd + cg * 4);
#pragma unroll
        for (int i = 0; i < kOwnRows; ++i) {
          const float4 weight = *reinterpret_cast<const float4*>(ps + (rg + kRowGroups * i) * kLdP + j);
          const float w[4] = {weight.x, weight.y, weight.z, weight.w};
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if (decltype(masked)::value && __float_as_int(w[x]) < 0) continue;
            acc[i][0] = fmaf(w[x], v[x].x, acc[i][0]), acc[i][1] = fmaf(w[x], v[x].y, acc[i][1]);
            acc[i][2] = fmaf(w[x], v[x].z, acc[i][2]), acc[i][3] = fmaf(w[x], v[x].w, acc[i][3]);
          }
        }
      }
    };
    if (whole) add_values(std::false_type{});
    else add_values(std::true_type{});
  }
  __syncthreads();
  if (tc == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) alphas[tr + 8 * i] = sum[i] > 0.f ? 1.f / sum[i] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kOwnRows; ++i) {
    const int r = rg + kRowGroups * i;
    if (r >= rows || cg * 4 >= p.head_dim) continue;
    const int item = row0 + r, token = item / group, head = kvh * group + item % group;
    const float inv = alphas[r];
    *reinterpret_cast<float4*>(p.out + (static_cast<int64_t>(start + token) * p.q_heads + head) * p.head_dim + cg * 4) =
        make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
  }
}

}  // namespace

// Sizes the tiled form takes.
B200_API int b200_portion_attention_f32_supported(int q_heads, int kv_heads, int head_dim) {
  return kv_heads > 0 && kv_heads <= 65535 && q_heads > 0 && q_heads % kv_heads == 0 && head_dim > 0 && head_dim % 4 == 0 && head_dim <= 128;
}

// Attention of the requests first_seq .. first_seq + num_seqs of the step (float32 queries, keys, values and outputs).
B200_API int b200_portion_attention_f32(const float* q, const float* k_arena, const float* v_arena, const int* block_table, int max_pages, int num_pages,
                                        const int* seq_q_start, const int* seq_q_len, const int* seq_kv_len, int first_seq, int num_seqs, int max_q_len,
                                        const float* sink, float* out, int q_heads, int kv_heads, int head_dim, int page_size, int window, float scale, int* err,
                                        cudaStream_t stream) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  B200_REQUIRE(b200_portion_attention_f32_supported(q_heads, kv_heads, head_dim), "portion_attention_f32: shape not taken");
  B200_REQUIRE(page_size > 0 && max_pages > 0 && window >= 0 && num_seqs <= 65535, "portion_attention_f32: bad geometry");
  const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  B200_REQUIRE(aligned(q) && aligned(k_arena) && aligned(v_arena) && aligned(out), "portion_attention_f32: operands must be aligned to 16 bytes");
  const PortionParams p{q, k_arena, v_arena, block_table, seq_q_start, seq_q_len, seq_kv_len, sink, out, err,
                        first_seq, max_pages, num_pages, q_heads, kv_heads, head_dim, page_size, window, scale};
  const bool narrow = head_dim <= 64;
  auto kernel = narrow ? portion_attention_f32_kernel<64> : portion_attention_f32_kernel<128>;
  static OncePerDevice raised;
  const auto raise = [] {
    return cudaFuncSetAttribute(portion_attention_f32_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(portion_smem(64))) == cudaSuccess &&
           cudaFuncSetAttribute(portion_attention_f32_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(portion_smem(128))) == cudaSuccess;
  };
  B200_REQUIRE(raised(raise), "portion_attention_f32: cannot size shared memory");
  const int64_t rows = static_cast<int64_t>(max_q_len) * (q_heads / kv_heads);
  const dim3 grid(static_cast<unsigned>((rows + kRows - 1) / kRows), kv_heads, num_seqs);
  kernel<<<grid, kThreads, portion_smem(narrow ? 64 : 128), stream>>>(p);
  return b200_check_launch("portion_attention_f32");
}
