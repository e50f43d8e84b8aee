// Attention of prompt portions over the paged cache in 32 bits: the tiled form of the plain kernel (attention_plain.cu).
//
// One block takes 32 rows of one kv head, a row being a (token, query head) pair of a request, token by token with the query heads
// that share the kv head side by side, and walks the request's keys 64 at a time. A warp has sixteen of the rows and sixteen of every 64 keys: scores,
// running softmax and weighted sum of values are its own until the end, when the four parts of the keys meet. Both products are tensor-core
// products of 32-bit numbers taken apart into three bfloat16 ones (split_mma.cuh); eight warps more take the next tile's keys and values
// apart, into shared memory as the lanes want them, while this one's are multiplied; where a block has few keys, each warp fetches its own (`few_keys`). Windows and a sink (a start value of
// maximum and sum) are taken; other shapes of scores, kept first keys and single tokens run the plain kernel.
//
// What bounds it: the tensor core's 1,536 products a tile (3,300 cycles of an SM) and, in turn with them, the taking apart. The plain kernel reads
// every key row once per (token, head) and forms one score a thread; FMAs over tiles in shared memory read 2 (scores) and 2.7 (values) FMAs'
// worth a number. Measured on a B200 (500 tokens, 12 heads of 128 on 2 kv heads, one request): plain 325, FMAs 76, now 46 us; 2,048
// tokens 487 and 415 us, behind 4,000 others 2.4 and 2.0 ms; 8 tokens behind 1,000 others 116 and 79. Error against 64 bits (500 tokens,
// 2-norm) 6.7e-7 and 2.3e-7.
#include "common.cuh"
#include "split_mma.cuh"

namespace {

constexpr int kRows = 32, kKeys = 64;
constexpr int kKeyParts = kKeys / 16;                 // warps that share sixteen rows
constexpr int kWarps = kRows / 16 * kKeyParts;        // that multiply
constexpr int kApart = 2 * kKeyParts;                 // behind them: that take apart, half the numbers of sixteen keys each
constexpr int kOwnThreads = kWarps * 32, kThreads = kOwnThreads + kApart * 32;
constexpr int kChunk = 2;                             // blocks of 16 x 16 numbers on the way in a warp's registers
// Registers a thread of either kind, out of 512 x 128 at launch.
constexpr int kOwnRegisters = 168, kApartRegisters = 88;
static_assert(kThreads == 512 && kOwnRegisters + kApartRegisters <= 2 * 128, "more registers than the block was launched with");

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

// Parts of 16 x 16 numbers, a uint4 a part and lane.
constexpr int kBlock = 3 * 32;
constexpr size_t portion_smem(int dim, bool direct) {
  return direct ? sizeof(float) * kWarps * 16 * (dim + 4) : sizeof(uint4) * (kRows / 16 + 2 * 2 * kKeyParts) * (dim / 16) * kBlock;
}

// Two tiles take turns: barrier `id` is met by the warps that multiply and those that take apart, of which one side only arrives.
__device__ __forceinline__ void meet(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kThreads) : "memory"); }
__device__ __forceinline__ void arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kThreads) : "memory"); }
__device__ __forceinline__ void meet_own() { asm volatile("bar.sync 5, %0;" ::"n"(kOwnThreads) : "memory"); }
constexpr int kFull = 1, kEmpty = 3;  // + tile % 2

__device__ __forceinline__ float4 finite_part(float4 v) {
  return make_float4(isfinite(v.x) ? v.x : 0.f, isfinite(v.y) ? v.y : 0.f, isfinite(v.z) ? v.z : 0.f, isfinite(v.w) ? v.w : 0.f);
}
__device__ __forceinline__ void store_block(uint4* to, const SplitB& first, const SplitB& second) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < 3; ++p) to[p * 32 + lane] = make_uint4(first.lo.part[p], first.hi.part[p], second.lo.part[p], second.hi.part[p]);
}
__device__ __forceinline__ void load_block(const uint4* from, SplitB* to) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint4 word = from[p * 32 + lane];
    to[0].lo.part[p] = word.x, to[0].hi.part[p] = word.y, to[1].lo.part[p] = word.z, to[1].hi.part[p] = word.w;
  }
}

// One row by one warp, of the numbers themselves, a lane a key and then four of the row's numbers: where a product of parts is not finite, an
// infinite operand (whose parts are NaN) or a number next to the largest may be the reason, and the row may be finite, or infinite. A NaN in its scores
// leaves the row as it is, NaN.
__device__ __noinline__ void attend_row(const PortionParams& p, int seq, int kvh, int token, int head, int pos) {
  const int lane = threadIdx.x & 31, from = p.window > 0 ? max(0, pos - p.window + 1) : 0;
  const float* own = p.q + (static_cast<int64_t>(token) * p.q_heads + head) * p.head_dim;
  const int* table = p.block_table + static_cast<int64_t>(seq) * p.max_pages;
  float top = p.sink != nullptr ? p.sink[head] : -INFINITY, sum = p.sink != nullptr ? 1.f : 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  bool nan = false;
  for (int c = lane; c < p.head_dim; c += 32) nan |= isnan(own[c]);
  if (__any_sync(0xffffffffu, nan)) return;
  for (int key0 = from; key0 <= pos; key0 += 32) {
    const int key = key0 + lane, logical = key / p.page_size;
    const int page = key <= pos && logical < p.max_pages ? table[logical] : -1;
    const int64_t offset = page >= 0 && page < p.num_pages ? kv_row_offset(page, kvh, key % p.page_size, p.kv_heads, p.page_size, p.head_dim) : -1;
    float score = -INFINITY;
    if (offset >= 0) {
      score = 0.f;
      for (int c = 0; c < p.head_dim; ++c) score = fmaf(own[c], p.keys[offset + c], score);
      score *= p.scale;
    }
    if (__any_sync(0xffffffffu, isnan(score))) return;
    float best = score;
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    const float new_top = fmaxf(top, best), alpha = top > -INFINITY ? expf(top - new_top) : 0.f;
    const float weight = score != -INFINITY ? expf(score - new_top) : 0.f;
    float more = weight;
    for (int o = 16; o > 0; o >>= 1) more += __shfl_xor_sync(0xffffffffu, more, o);
    sum = fmaf(sum, alpha, more);
    top = new_top;
    acc = make_float4(acc.x * alpha, acc.y * alpha, acc.z * alpha, acc.w * alpha);
    for (int j = 0; j < 32; ++j) {
      const int64_t at = __shfl_sync(0xffffffffu, offset, j);
      const float w = __shfl_sync(0xffffffffu, weight, j);
      if (at < 0 || lane * 4 >= p.head_dim) continue;
      const float4 v = *reinterpret_cast<const float4*>(p.values + at + lane * 4);
      acc = make_float4(fmaf(w, v.x, acc.x), fmaf(w, v.y, acc.y), fmaf(w, v.z, acc.z), fmaf(w, v.w, acc.w));
    }
  }
  const float inv = sum > 0.f ? 1.f / sum : 0.f;
  if (lane * 4 < p.head_dim)
    *reinterpret_cast<float4*>(p.out + (static_cast<int64_t>(token) * p.q_heads + head) * p.head_dim + lane * 4) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
}

template <int DIM, bool DIRECT>  // DIRECT: no warps that take apart, each fetches what it multiplies by
__global__ void __launch_bounds__(DIRECT ? kOwnThreads : kThreads, DIRECT ? 2 : 1)
portion_attention_f32_kernel(const __grid_constant__ PortionParams p) {
  extern __shared__ __align__(16) uint4 attention_smem[];
  constexpr int kSteps = DIM / 16;                        // sixteens of a head's numbers
  constexpr int kTile = kKeyParts * kSteps * kBlock;      // of keys, or of values
  constexpr int kLdO = DIM + 4;
  uint4* qs = attention_smem;                             // [kRows / 16][kSteps][kBlock]
  uint4* ks = qs + kRows / 16 * kSteps * kBlock;          // [2][kKeyParts][kSteps][kBlock]: tiles of eight keys
  uint4* vs = ks + 2 * kTile;                             // [2][kKeyParts][kSteps][kBlock]: tiles of eight of a value's numbers
  __shared__ int64_t offsets[2][kKeys];                   // rows of two tiles, -1: not to be read
  __shared__ int spoilt[2][kApart];                       // values that are not finite
  __shared__ float tops[kWarps][16], totals[kWarps][16];
  const int seq = p.first_seq + blockIdx.z, kvh = blockIdx.y;
  const int group = p.q_heads / p.kv_heads;
  const int len = p.seq_q_len[seq], start = p.seq_q_start[seq], begin = p.seq_kv_len[seq] - len;  // begin: position of the first new token
  const int row_blocks = (len * group + kRows - 1) / kRows;
  const int block = row_blocks - 1 - static_cast<int>(blockIdx.x);  // the rows with most keys first
  if (block < 0) return;
  const int row0 = block * kRows, rows = min(kRows, len * group - row0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int* table = p.block_table + static_cast<int64_t>(seq) * p.max_pages;
  const int last_pos = begin + (row0 + rows - 1) / group, first_pos = begin + row0 / group;
  const int lo = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
  const int tiles = (last_pos - lo) / kKeys + 1;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto query = [&](int r, int c) {
    const int item = row0 + r, token = item / group, head = kvh * group + item % group;
    return r < rows && c < p.head_dim ? *reinterpret_cast<const float4*>(p.q + (static_cast<int64_t>(start + token) * p.q_heads + head) * p.head_dim + c) : zero;
  };
  for (int item = warp; item < kRows / 16 * kSteps; item += (DIRECT ? kOwnThreads : kThreads) / 32) {
    const int r = item / kSteps * 16 + g, c = item % kSteps * 16 + 4 * q;
    const SplitA a = split_rows(query(r, c), query(r + 8, c));
#pragma unroll
    for (int x = 0; x < 3; ++x) qs[(item * 3 + x) * 32 + lane] = make_uint4(a.part[x][0], a.part[x][1], a.part[x][2], a.part[x][3]);
  }
  __syncthreads();
  if (!DIRECT && warp >= kWarps) {
    // ---- take apart: half the numbers of sixteen keys a warp, chunk after chunk ----
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kApartRegisters));
    constexpr int kChunks = kSteps / 2 / kChunk;
    const int part = (warp - kWarps) / 2, half = (warp - kWarps) % 2, step0 = half * (kSteps / 2);
    float4 k_next[kChunk][2], v_next[kChunk][2];
    int64_t own = -1;  // of key lane % 16: where its row is
    auto look_up = [&](int tile) {
      const int j = lo + tile * kKeys + part * 16 + (lane & 15);
      own = -1;
      if (tile < tiles && j <= last_pos) {
        const int logical = j / p.page_size;
        const int page = logical < p.max_pages ? table[logical] : -1;
        if (page < 0 || page >= p.num_pages) atomicOr(p.err, ERRBIT_BAD_PAGE);
        else own = kv_row_offset(page, kvh, j % p.page_size, p.kv_heads, p.page_size, p.head_dim);
      }
    };
    int64_t key_at[2], value_at[4];
    auto spread = [&] {
#pragma unroll
      for (int t = 0; t < 2; ++t) key_at[t] = __shfl_sync(0xffffffffu, own, in_sixteen(t, g));
#pragma unroll
      for (int x = 0; x < 4; ++x) value_at[x] = __shfl_sync(0xffffffffu, own, 4 * q + x);
    };
    auto fetch = [&](int step, int i) {
      const int c0 = (step0 + step + i) * 16;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int c = c0 + 4 * q, cv = c0 + 8 * t + g;
        k_next[i][t] = key_at[t] >= 0 && c < p.head_dim ? *reinterpret_cast<const float4*>(p.keys + key_at[t] + c) : zero;
        const bool in = cv < p.head_dim;
        v_next[i][t] = make_float4(in && value_at[0] >= 0 ? p.values[value_at[0] + cv] : 0.f, in && value_at[1] >= 0 ? p.values[value_at[1] + cv] : 0.f,
                                   in && value_at[2] >= 0 ? p.values[value_at[2] + cv] : 0.f, in && value_at[3] >= 0 ? p.values[value_at[3] + cv] : 0.f);
      }
    };
    look_up(0), spread();
#pragma unroll
    for (int i = 0; i < kChunk; ++i) fetch(0, i);
    for (int tile = 0; tile < tiles; ++tile) {
      const int b = tile & 1;
      if (tile >= 2) meet(kEmpty + b);
      if (half == 0 && lane < 16) offsets[b][part * 16 + lane] = own;
      bool finite = true;
#pragma unroll 1
      for (int chunk = 0; chunk < kChunks; ++chunk) {
        if (chunk + 1 == kChunks) look_up(tile + 1), spread();
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
          const int at = b * kTile + (part * kSteps + step0 + chunk * kChunk + i) * kBlock;
          store_block(ks + at, SplitB(k_next[i][0]), SplitB(k_next[i][1]));
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            float4& v = v_next[i][t];
            if (all_finite(v)) continue;
            finite = false, v = finite_part(v);  // zeros for now
          }
          store_block(vs + at, SplitB(v_next[i][0]), SplitB(v_next[i][1]));
          fetch(chunk + 1 < kChunks ? (chunk + 1) * kChunk : 0, i);  // the next chunk's, of the next tile behind a tile's last (past the last one: zeros)
        }
      }
      const bool any = __any_sync(0xffffffffu, !finite);
      if (lane == 0) spoilt[b][warp - kWarps] = any;
      arrive(kFull + b);
    }
    return;
  }
  if constexpr (!DIRECT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kOwnRegisters));
  const int own_rows = warp / kKeyParts * 16, own_keys = warp % kKeyParts;
  int pos[2], from[2];
  float top[2], sum[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = own_rows + g + 8 * h, item = row0 + r;
    pos[h] = r < rows ? begin + item / group : -1;
    from[h] = p.window > 0 ? pos[h] - p.window + 1 : 0;
    const float* sink = p.sink && own_keys == 0 ? p.sink + kvh * group + item % group : nullptr;
    top[h] = sink ? *sink : -INFINITY;
    sum[h] = sink && q == 0 ? 1.f : 0.f;  // a lane's share
  }
  float acc[2 * kSteps][4];
#pragma unroll
  for (int i = 0; i < 2 * kSteps; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  for (int tile = 0; tile < tiles; ++tile) {
    const int b = tile & 1;
    int64_t row = -1;  // DIRECT: of key lane % 16: where its row is
    if constexpr (DIRECT) {
      const int part0 = lo + tile * kKeys + own_keys * 16, j = part0 + (lane & 15);
      if (part0 > last_pos) break;  // the last tile's last keys
      if (j <= last_pos) {
        const int logical = j / p.page_size;
        const int page = logical < p.max_pages ? table[logical] : -1;
        if (page < 0 || page >= p.num_pages) atomicOr(p.err, ERRBIT_BAD_PAGE);
        else row = kv_row_offset(page, kvh, j % p.page_size, p.kv_heads, p.page_size, p.head_dim);
      }
    } else {
      meet(kFull + b);
    }
    // Scores of sixteen rows and sixteen keys, of which the lane has keys 4 q .. + 3.
    float score[2][4] = {};
    {
      constexpr int kTogether = 2;
      const float* at[2];
      float4 next[2 * kTogether];
      const auto fetch_keys = [&](int s) {
#pragma unroll
        for (int n = 0; n < 2 * kTogether; ++n) {
          const int c = (s + n / 2) * 16 + 4 * q;
          next[n] = at[n % 2] != nullptr && c < p.head_dim ? *reinterpret_cast<const float4*>(at[n % 2] + c) : zero;
        }
      };
      if constexpr (DIRECT) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int64_t key_at = __shfl_sync(0xffffffffu, row, in_sixteen(t, g));
          at[t] = key_at >= 0 ? p.keys + key_at : nullptr;
        }
        fetch_keys(0);
      }
#pragma unroll 1
      for (int s = 0; s < kSteps; s += kTogether) {
        float sums[2 * kTogether][4];
        SplitA own[kTogether];
        SplitB right[2 * kTogether];
#pragma unroll
        for (int x = 0; x < kTogether; ++x) {
#pragma unroll
          for (int y = 0; y < 3; ++y) {
            const uint4 word = qs[((own_rows / 16 * kSteps + s + x) * 3 + y) * 32 + lane];
            own[x].part[y][0] = word.x, own[x].part[y][1] = word.y, own[x].part[y][2] = word.z, own[x].part[y][3] = word.w;
          }
          if constexpr (!DIRECT) load_block(ks + b * kTile + (own_keys * kSteps + s + x) * kBlock, right + 2 * x);
        }
        if constexpr (DIRECT) {
#pragma unroll
          for (int n = 0; n < 2 * kTogether; ++n) right[n] = SplitB(next[n]);
          if (s + kTogether < kSteps) fetch_keys(s + kTogether);
        }
#pragma unroll
        for (int n = 0; n < 2 * kTogether; ++n) mma_split(sums[n], own[n / 2], right[n]);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int i = 0; i < 4; ++i) score[t][i] += sums[t][i] + sums[2 + t][i];
      }
    }
    const int key0 = lo + tile * kKeys + own_keys * 16 + 4 * q;
    const auto own_offset = [&](int i) { return DIRECT ? __shfl_sync(0xffffffffu, row, 4 * q + i) : offsets[b][own_keys * 16 + 4 * q + i]; };
    float weight[2][4], alpha[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float best = -INFINITY;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int key = key0 + i;
        const bool seen = own_offset(i) >= 0 && key <= pos[h] && key >= from[h];
        weight[h][i] = seen ? score[i >> 1][2 * h + (i & 1)] * p.scale : -INFINITY;
        best = fmaxf(best, weight[h][i]);
      }
      best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 1));
      best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 2));
      const float new_top = fmaxf(top[h], best);
      alpha[h] = top[h] > -INFINITY ? expf(top[h] - new_top) : 0.f;
      float more = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        weight[h][i] = weight[h][i] != -INFINITY ? expf(weight[h][i] - new_top) : 0.f;  // a score that is NaN stays, also where no other is seen
        more += weight[h][i];
      }
      sum[h] = fmaf(sum[h], alpha[h], more);
      top[h] = new_top;
    }
    const SplitA left = split_rows(make_float4(weight[0][0], weight[0][1], weight[0][2], weight[0][3]), make_float4(weight[1][0], weight[1][1], weight[1][2], weight[1][3]));
    float4 v[4];
    const float* value_at[4];
    if constexpr (DIRECT) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t at = own_offset(i);
        value_at[i] = at >= 0 ? p.values + at + g : nullptr;
      }
    }
    const auto fetch_values = [&](int s) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int c = s * 16 + 8 * n;
        const bool in = c + g < p.head_dim;
        v[n] = make_float4(in && value_at[0] ? value_at[0][c] : 0.f, in && value_at[1] ? value_at[1][c] : 0.f, in && value_at[2] ? value_at[2][c] : 0.f,
                           in && value_at[3] ? value_at[3][c] : 0.f);
      }
    };
    bool finite = true;
    if constexpr (DIRECT) fetch_values(0);
#pragma unroll
    for (int s = 0; s < kSteps; s += 2) {
      SplitB right[4];
      if constexpr (DIRECT) {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          if (!all_finite(v[n])) finite = false, v[n] = finite_part(v[n]);
          right[n] = SplitB(v[n]);
        }
        if (s + 2 < kSteps) fetch_values(s + 2);
      } else {
        load_block(vs + b * kTile + (own_keys * kSteps + s) * kBlock, right);
        load_block(vs + b * kTile + (own_keys * kSteps + s + 1) * kBlock, right + 2);
      }
      float sums[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) mma_split(sums[n], left, right[n]);
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[2 * s + n][i] = fmaf(acc[2 * s + n][i], alpha[i >> 1], sums[n][i]);
    }
    if (DIRECT ? __any_sync(0xffffffffu, !finite) : spoilt[b][2 * own_keys] | spoilt[b][2 * own_keys + 1]) {  // what is not finite reaches the rows that see its key, and no others
      for (int j = 0; j < 16; ++j) {
        const int key = lo + tile * kKeys + own_keys * 16 + j;
        const int64_t offset = DIRECT ? __shfl_sync(0xffffffffu, row, j) : offsets[b][own_keys * 16 + j];
        if (offset < 0) continue;
#pragma unroll
        for (int x = 0; x < 2 * kSteps; ++x)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int c = x * 8 + 2 * q + (i & 1), h = i >> 1;
            if (c < p.head_dim && key <= pos[h] && key >= from[h] && !isfinite(p.values[offset + c])) acc[x][i] += p.values[offset + c];
          }
      }
    }
    if (!DIRECT && tile + 2 < tiles) arrive(kEmpty + b);
  }
  // The four parts of the keys meet.
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
    sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
    if (q == 0) tops[warp][g + 8 * h] = top[h], totals[warp][g + 8 * h] = sum[h];
  }
  meet_own();  // the parts have been read too
  float* os = reinterpret_cast<float*>(DIRECT ? qs : ks);  // [kWarps][16][kLdO]
  static_assert(sizeof(float) * kWarps * 16 * kLdO <= sizeof(uint4) * 4 * kTile, "the warps' sums do not fit where keys and values were");
#pragma unroll
  for (int x = 0; x < 2 * kSteps; ++x)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float2*>(os + (warp * 16 + g + 8 * h) * kLdO + x * 8 + 2 * q) = make_float2(acc[x][2 * h], acc[x][2 * h + 1]);
  meet_own();
  static_assert(32 % (DIM / 4) == 0, "a row's numbers are those of one warp");
  uint32_t odd = 0;  // rows to be made again
  for (int idx = tid; idx < rows * (DIM / 4); idx += kOwnThreads) {
    const int r = idx / (DIM / 4), c = idx % (DIM / 4) * 4;
    if (c >= p.head_dim) continue;
    const int first = r / 16 * kKeyParts;
    float whole_top = -INFINITY, total = 0.f;
#pragma unroll
    for (int w = 0; w < kKeyParts; ++w) whole_top = fmaxf(whole_top, tops[first + w][r % 16]);
    float4 o = zero;
#pragma unroll
    for (int w = 0; w < kKeyParts; ++w) {
      const float t = tops[first + w][r % 16], factor = t > -INFINITY ? expf(t - whole_top) : 0.f;
      const float4 v = *reinterpret_cast<const float4*>(os + ((first + w) * 16 + r % 16) * kLdO + c);
      total = fmaf(totals[first + w][r % 16], factor, total);
      o.x = fmaf(v.x, factor, o.x), o.y = fmaf(v.y, factor, o.y), o.z = fmaf(v.z, factor, o.z), o.w = fmaf(v.w, factor, o.w);
    }
    const float inv = total > 0.f ? 1.f / total : 0.f;
    const int item = row0 + r, token = item / group, head = kvh * group + item % group;
    o = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    // NaN beside a finite sum of weights comes from values and stands.
    if (!isfinite(total) || isinf(o.x) || isinf(o.y) || isinf(o.z) || isinf(o.w)) odd |= 1u << r;
    *reinterpret_cast<float4*>(p.out + (static_cast<int64_t>(start + token) * p.q_heads + head) * p.head_dim + c) = o;
  }
  odd = __reduce_or_sync(0xffffffffu, odd);
  for (; odd != 0; odd &= odd - 1) {
    const int item = row0 + __ffs(odd) - 1;
    __syncwarp();
    attend_row(p, seq, kvh, start + item / group, kvh * group + item % group, begin + item / group);
  }
}

}  // namespace

// Sizes the tiled form takes.
B200_API int b200_portion_attention_f32_supported(int q_heads, int kv_heads, int head_dim) {
  return kv_heads > 0 && kv_heads <= 65535 && q_heads > 0 && q_heads % kv_heads == 0 && head_dim > 0 && head_dim % 4 == 0 && head_dim <= 128;
}

// Whether a block's keys are too few for warps that take apart: one block has an SM to itself then, and what it does alone (its look at its
// request, its queries, its first keys, the join of the parts) is most of it. Without them a warp fetches and takes apart what it multiplies by, which is
// twice that work, but two blocks share an SM. Both give the same bits. Measured on a B200, with and without, heads of 128 (12 on 2): 192 blocks
// of one tile of keys 21 and 16 us, 768 57 and 44, 192 of two 21 and 23, 256 36 and 34, 512 of three 66 and 63, 256 of six 63 and 65; heads of 64
// (8): 128 of one 9.2 and 8.6, 512 25 and 16, 256 of three 15 and 12, 128 15 and 17, 512 of five 30 and 27, 1,024 of nine 92 and 90.
static bool few_keys(bool narrow, int tokens, int max_kv_len, int group, int kv_heads, int num_seqs, int window) {
  const int64_t blocks = (static_cast<int64_t>(tokens) * group + static_cast<int64_t>(num_seqs) * (kRows / 2)) / kRows * kv_heads, sms = b200_sm_count_host();
  const int64_t keys = window > 0 && max_kv_len > window + kRows / group ? window + kRows / group : max_kv_len, tiles = (keys + kKeys - 1) / kKeys;
  if (narrow) return tiles <= (blocks > 6 * sms ? 9 : (blocks > 2 * sms ? 6 : (blocks > sms ? 3 : 1)));
  return tiles <= (blocks > 4 * sms ? 4 : (blocks > sms ? 2 : 0));
}

// Attention of the requests first_seq .. first_seq + num_seqs of the step (float32 queries, keys, values and outputs), which have `tokens` new tokens, at
// most max_q_len each and max_kv_len with those before. `form`: 1 without warps that take apart, 2 with them; 0: by the sizes.
B200_API int b200_portion_attention_f32(const float* q, const float* k_arena, const float* v_arena, const int* block_table, int max_pages, int num_pages,
                                        const int* seq_q_start, const int* seq_q_len, const int* seq_kv_len, int first_seq, int num_seqs, int max_q_len,
                                        const float* sink, float* out, int q_heads, int kv_heads, int head_dim, int page_size, int window, float scale, int tokens, int max_kv_len,
                                        int form, int* err, cudaStream_t stream) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  B200_REQUIRE(b200_portion_attention_f32_supported(q_heads, kv_heads, head_dim), "portion_attention_f32: shape not taken");
  B200_REQUIRE(page_size > 0 && max_pages > 0 && window >= 0 && num_seqs <= 65535, "portion_attention_f32: bad geometry");
  const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  B200_REQUIRE(aligned(q) && aligned(k_arena) && aligned(v_arena) && aligned(out), "portion_attention_f32: operands must be aligned to 16 bytes");
  const PortionParams p{q, k_arena, v_arena, block_table, seq_q_start, seq_q_len, seq_kv_len, sink, out, err,
                        first_seq, max_pages, num_pages, q_heads, kv_heads, head_dim, page_size, window, scale};
  const bool narrow = head_dim <= 64, direct = form == 0 ? few_keys(narrow, tokens, max_kv_len, q_heads / kv_heads, kv_heads, num_seqs, window) : form == 1;
  auto kernel = direct ? (narrow ? portion_attention_f32_kernel<64, true> : portion_attention_f32_kernel<128, true>)
                       : (narrow ? portion_attention_f32_kernel<64, false> : portion_attention_f32_kernel<128, false>);
  static OncePerDevice raised;
  const auto raise = [] {
    const auto raise_one = [](auto form_of, size_t bytes) { return cudaFuncSetAttribute(form_of, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) == cudaSuccess; };
    return raise_one(portion_attention_f32_kernel<64, false>, portion_smem(64, false)) && raise_one(portion_attention_f32_kernel<128, false>, portion_smem(128, false)) &&
           raise_one(portion_attention_f32_kernel<64, true>, portion_smem(64, true)) && raise_one(portion_attention_f32_kernel<128, true>, portion_smem(128, true));
  };
  B200_REQUIRE(raised(raise), "portion_attention_f32: cannot size shared memory");
  const int64_t rows = static_cast<int64_t>(max_q_len) * (q_heads / kv_heads);
  const dim3 grid(static_cast<unsigned>((rows + kRows - 1) / kRows), kv_heads, num_seqs);
  kernel<<<grid, direct ? kOwnThreads : kThreads, portion_smem(narrow ? 64 : 128, direct), stream>>>(p);
  return b200_check_launch("portion_attention_f32");
}
