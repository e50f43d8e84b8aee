// Recurrent matrix states over prompt portions, 32 tokens at a time: the delta rule (one decay per head, or one per head and key
// channel), the generalized delta rule, the rule with a decay per channel and a bonus for the current token, and the matrix memory's
// (one decay and one weight per head and token, a normaliser beside the state).
//
// Token by token a portion costs tokens x the latency of one step, however few columns a head's state has. Over a chunk of tokens
// the rule S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q is a handful of small matrix products (the chunkwise form of
// delta rules: Yang, Kautz and Hatamizadeh, "Gated Delta Networks: Improving Mamba2 with Delta Rule"; with a decay per key channel
// every product over channels carries the decays between its two tokens). With S the state in front of the chunk, G_ij the product
// of the decays of tokens j + 1 .. i (per channel), e_i the product up to token i:
//   u_i = beta_i (v_i - S^T (e_i k_i) - sum_{j < i} (k_i . G_ij k_j) u_j),   o_i = S^T (e_i q_i) + sum_{j <= i} (q_i . G_ij k_j) u_j,
//   S <- e_last S + sum_j (G_last,j k_j) u_j^T.
// With L_ij = beta_i k_i . G_ij k_j (j < i): U = W + Y S, W = (I + L)^-1 diag(beta) V, Y = -(I + L)^-1 diag(beta) (e K).
// The generalized rule S <- w S + b (u^T S) + k v^T (b = -a u), o = S^T r, has the same form in X_i = u_i^T S_{i-1}: with
// N_ij = u_i . G_{i-1,j} b_j and M_ij = u_i . G_{i-1,j} k_j (j < i), X = W + Y S, W = (I - N)^-1 M V, Y = (I - N)^-1 (e_{i-1} u_i), and what
// the values alone add to S and to o is known in front of the walk. Without the removal (S <- w S + k v^T, o = S^T r read before the
// update) nothing is left of a walk but sums of whole chunks.
// Kernels:
//   chunk_prepare, linear_chunk_prepare   all chunks side by side: pairs of tokens, W, Y, scaled rows, the values' own sums;
//   chunk_walk       a head's chunks one after another, a tile of 16 columns of S per block: U = W + Y S, S <- e S + (G_last K)^T U;
//   chunk_scan       the same without U: S <- e S + the chunk's own sum, element by element;
//   chunk_out        all chunks side by side again: O = (e Q) S + A U, from the states left at each chunk's start.
// Only what the next chunk waits for is in the walk. All numbers stay 32-bit: products are FMAs where a token meets its group of eight, and
// elsewhere tensor-core products of numbers taken apart into three bfloat16 ones (`mma_split`). Against 64 bits, outputs and states are nearer than
// with FMAs throughout (2,048 tokens, 2-norm: a decay per channel 1.74e-7 and 1.41e-7, before 1.92e-7 and 1.61e-7; generalized rule 1.62e-7
// and 1.43e-7, before 1.96e-7 and 1.68e-7; without a removal 2.01e-7 and 1.91e-7, before 2.22e-7 and 2.05e-7). Decays enter as products (or
// sums of their logarithms) from token j on, never as quotients of products from the chunk's start, so strong decays in front of a pair
// cost it no digits.
//
// Measured on a B200 (one request of 2,048 tokens, all three kernels; FMAs throughout, now): heads of 128 x 128, a decay per channel, 12 of them
// 230 -> 148 us (prepare 60 -> 41, walk 135 -> 80, out 35 -> 22), 28 of them 430 -> 273; one decay per head 228 -> 149; 24 heads of 64 x 64 under the
// generalized rule 229 -> 145 us (prepare 97 -> 64, walk 91 -> 55, out 35 -> 21), without a removal 87 -> 68.
#include <type_traits>

#include "common.cuh"
#include "split_mma.cuh"

namespace {

constexpr int C = 32;            // tokens per chunk
constexpr int kColumns = 16;     // columns of the state per block of the walk
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxRows = 256;    // key channels per head

__host__ __device__ constexpr int padded_rows(int dk) { return dk <= 64 ? 64 : (dk <= 128 ? 128 : 256); }
__host__ __device__ constexpr int padded_columns(int dv) { return (dv + kColumns - 1) / kColumns * kColumns; }
// A chunk's place among all chunks of the step: different for all (request, chunk), below tokens / C + requests + 1.
__device__ __forceinline__ int64_t chunk_place(int start, int seq, int chunk) { return static_cast<int64_t>(start / C) + seq + chunk; }

enum Rule { kDelta = 0, kGeneralDelta = 1, kLinear = 2, kMemory = 3 };

template <int kBytes>
__device__ __forceinline__ void stage_copy(float* smem, const void* gmem, bool valid = true) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? kBytes : 0;
  if (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(kBytes), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit_copies() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void wait_copies() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// n rows `from` [..][ld] of `width` numbers to dst [C][ROWS + 4]; rows past n and columns from `width` on become zeros. W numbers a copy.
template <int ROWS, int W>
__device__ __forceinline__ void stage_rows(float* dst, const float* from, int n, int64_t ld, int width) {
  constexpr int kPerRow = ROWS / W, kAtOnce = kThreads / kPerRow;  // rows
  const int r0 = threadIdx.x / kPerRow, c = threadIdx.x % kPerRow * W;
  const float* at = from + r0 * ld + c;
  float* to = dst + r0 * (ROWS + 4) + c;
#pragma unroll
  for (int i = 0; i < C / kAtOnce; ++i) {
    const bool valid = r0 + i * kAtOnce < n && c < width;
    stage_copy<4 * W>(to + i * kAtOnce * (ROWS + 4), valid ? at + i * kAtOnce * ld : from, valid);
  }
}

__device__ __forceinline__ float from_pair(float give, float keep, int with) { return keep + __shfl_xor_sync(0xffffffffu, give, with); }

// What the preparing kernels hand on, and the walk's result, by (chunk's place, head): rows of `padded_rows(dk)` and `padded_columns(dv)`
// numbers, whole chunks of C tokens (those past a request's end are zeros in y, kd and x). Each array runs along what its reader multiplies
// over, four neighbouring numbers for the lane that wants them; y, kd and s lie as the lanes of a warp want them side by side (`y_place`,
// `kd_place`, `s_place`).
struct Scratch {
  int head0, heads;  // the heads that a pass takes: all, or as many as the scratch holds
  float* y;   // [chunks][heads][rows x C]
  float* kd;  // [chunks][heads][rows x C]: G_last,j k_j
  float* qt;  // [chunks][heads][C][rows]: e_i q_i
  float* x;   // [chunks][heads][columns][C]: W, then U
  float* a;   // [chunks][heads][C][C]: what reads out U
  float* av;  // [chunks][heads][C][C]: what reads out V
  float* e;   // [chunks][heads][rows]: e_last
  float* n;   // [chunks][heads][rows]: the matrix memory's normaliser, likewise
  float* s;   // [chunks][heads][columns x rows]: what the values alone add, then the state in front of each chunk
};

// Rows of sixteen are a warp's of the walk. y: by (sixteen rows, sixteen tokens, tile) the lanes' four rows of a token each.
__device__ __forceinline__ int y_place(int token, int row) {
  const int g = (token & 12) / 2 + (token & 1), tile = token / 16 * 2 + (token >> 1 & 1);
  return row / 16 * (16 * C) + tile * 128 + g * 16 + (row & 15);
}
// kd: by (sixteen rows, tile, sixteen tokens) the lanes' four tokens of a row each.
__device__ __forceinline__ int kd_place(int token, int row) {
  const int g = (row & 12) / 2 + (row & 1), tile = row >> 1 & 1;
  return row / 16 * (16 * C) + (tile * 2 + token / 16) * 128 + g * 16 + (token & 15);
}
// s: by (sixteen columns, sixteen rows, eight of the columns) the lanes' four rows of a column each.
__device__ __forceinline__ int s_place(int col, int row, int rows) {
  return col / 16 * (16 * rows) + row / 16 * 256 + (col >> 3 & 1) * 128 + (col & 7) * 16 + (row & 15);
}

// --- what does not depend on the state -------------------------------------------------------------------------------------------
//
// One block per (chunk, head, request). Pairs of tokens: the chunk's rows form four groups of eight. Between groups every decay product splits
// at the group's border, G_ij = (product up to i inside i's group) (whole groups between) (product from j + 1 to the end of j's group),
// three factors without a quotient, so those pairs are plain products of scaled rows: tiles of eight rows of two left operands by eight
// of the right one on the tensor cores. Inside a group, where G_ij is a run of products for each j, a warp has a group and a left operand, a lane two
// channels at a time of all its tokens in registers; the lanes' sums meet by shuffles. With one decay per head pairs are products of the raw
// rows and G_ij stands beside them, so all pairs are tiles.
// Columns of [e K | V]: (I + L) X = R in halves of sixteen tokens, X1 = T11 R1, X2 = T22 (R2 - L21 X1), with the two halves' inverses made
// by a warp, a lane per column; transposed (X^T = R^T T^T, sixteen columns a warp at a time), every result is the next product's operand in
// the lanes that hold it.
// What bounds it: instructions (some 20,000 of a warp for a chunk of a head of 128 x 128) and the barriers between its seven phases, three blocks
// an SM. With operands of pairs out of shared memory for every FMA, a thread per column of the triangular system and sums of the warps
// through shared memory, two blocks an SM waited for shared memory most of the time: 2,048 tokens of 12 heads of 128 x 128, a decay per channel 60 ->
// 41 us, one per head 56 -> 39; 24 heads of 64 x 64, the generalized rule 97 -> 64, the rule without a removal 54 -> 37. (A first form of this one
// with two blocks an SM: 50, 47, 87 and 47; with three: 43, 39, 77 and 39.)
constexpr int kGroup = 8, kGroups = C / kGroup;
constexpr int kBetween = 6;             // pairs of different groups
constexpr int kTiles = kBetween + kGroups;  // and of a group with itself
constexpr int kLdT = 20;                // numbers from row to row of an inverse

// left_i . G_ij right_j for i, j of one group (j < i; DIAGONAL: j <= i) into `to` [C][C + 1], by one warp. BEFORE: the left row meets the decays
// of tokens j + 1 .. i - 1 only.
template <int ROWS, bool BEFORE, bool DIAGONAL>
__device__ __forceinline__ void pairs_in_group(const float* left, const float* right, const float* decays, int group, float* to) {
  constexpr int ld = ROWS + 4, kPairs = DIAGONAL ? 36 : 28;
  const int lane = threadIdx.x & 31;
  float acc[36] = {};
#pragma unroll 1
  for (int x = 0; x < ROWS / 64; ++x) {
    const int at = group * kGroup * ld + x * 64 + lane * 2;
    float2 l[kGroup], g[kGroup], r[kGroup];
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      l[i] = *reinterpret_cast<const float2*>(left + at + i * ld);
      g[i] = *reinterpret_cast<const float2*>(decays + at + i * ld);
      r[i] = *reinterpret_cast<const float2*>(right + at + i * ld);
    }
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      float2 p = r[j];
#pragma unroll
      for (int i = DIAGONAL ? j : j + 1; i < kGroup; ++i) {
        const int pair = DIAGONAL ? i * (i + 1) / 2 + j : i * (i - 1) / 2 + j;
        if (!BEFORE && i > j) p.x *= g[i].x, p.y *= g[i].y;
        acc[pair] = fmaf(l[i].x, p.x, fmaf(l[i].y, p.y, acc[pair]));
        if (BEFORE) p.x *= g[i].x, p.y *= g[i].y;
      }
    }
  }
  // Every lane ends with one of the first 32 sums, and with one of the last four.
#pragma unroll
  for (int w = 16; w > 0; w /= 2)
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const bool high = lane & w;
      acc[k] = from_pair(high ? acc[k] : acc[k + w], high ? acc[k + w] : acc[k], w);
    }
  if (DIAGONAL) {
#pragma unroll
    for (int w = 2; w > 0; w /= 2)
#pragma unroll
      for (int k = 32; k < 32 + w; ++k) {
        const bool high = lane & w;
        acc[k] = from_pair(high ? acc[k] : acc[k + w], high ? acc[k + w] : acc[k], w);
      }
#pragma unroll
    for (int w = 4; w < 32; w *= 2) acc[32] = from_pair(acc[32], acc[32], w);
  }
  auto store = [&](int pair, float sum) {
    int i = 0;
#pragma unroll
    for (int row = 1; row < kGroup; ++row) i += pair >= row * (row + 1) / 2 ? 1 : 0;
    const int j = pair - i * (i + 1) / 2;
    to[(group * kGroup + i + (DIAGONAL ? 0 : 1)) * (C + 1) + group * kGroup + j] = sum;
  };
  if (lane < kPairs) store(lane, acc[0]);
  if (DIAGONAL && lane < 4) store(32 + lane, acc[32]);
}

// Tile `tile` of the pairs: rows of group gi of both left operands by rows of group gj <= gi of RIGHTS right ones into `to` [left][right] [C][C + 1], by
// one warp. DECAYS: gj < gi, rows carry their decays inside their own groups, `whole` holds the groups' decays multiplied.
template <int ROWS, int LEFTS, int RIGHTS, bool DECAYS>
__device__ __forceinline__ void pair_tile(const float* left0, const float* left1, const float* const (&right)[RIGHTS], const float* whole, int tile,
                                          float* const (&to)[LEFTS][RIGHTS]) {
  constexpr int ld = ROWS + 4, kTogether = 4 / RIGHTS;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  int gi = 0;  // tiles (1, 0), (2, 0), (2, 1), .., or with (i, i) too
#pragma unroll
  for (int row = 1; row < kGroups; ++row) gi += tile >= row * (row + 1) / 2 ? 1 : 0;
  const int gj = tile - gi * (gi + 1) / 2;
  if (DECAYS) ++gi;
  const int at_left = (gi * kGroup + g) * ld + 4 * q, at_right = (gj * kGroup + g) * ld + 4 * q;
  float acc[RIGHTS][4] = {};
#pragma unroll 1
  for (int step = 0; step < ROWS / 16; step += kTogether) {
    float part[kTogether][RIGHTS][4];
#pragma unroll
    for (int x = 0; x < kTogether; ++x) {
      const int c = (step + x) * 16;
      const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
      const SplitA a = split_rows(*reinterpret_cast<const float4*>(left0 + at_left + c), LEFTS == 2 ? *reinterpret_cast<const float4*>(left1 + at_left + c) : none);
      float4 r[RIGHTS];
#pragma unroll
      for (int y = 0; y < RIGHTS; ++y) r[y] = *reinterpret_cast<const float4*>(right[y] + at_right + c);
      if (DECAYS) {
        for (int between = gj + 1; between < gi; ++between) {
          const float4 w = *reinterpret_cast<const float4*>(whole + between * ROWS + c + 4 * q);
#pragma unroll
          for (int y = 0; y < RIGHTS; ++y) r[y].x *= w.x, r[y].y *= w.y, r[y].z *= w.z, r[y].w *= w.w;
        }
      }
#pragma unroll
      for (int y = 0; y < RIGHTS; ++y) mma_split(part[x][y], a, SplitB(r[y]));
    }
#pragma unroll
    for (int y = 0; y < RIGHTS; ++y)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (kTogether == 4) acc[y][i] += (part[0][y][i] + part[1][y][i]) + (part[kTogether / 2][y][i] + part[kTogether - 1][y][i]);
        else acc[y][i] += part[0][y][i] + part[kTogether - 1][y][i];
      }
  }
  const int at = (gi * kGroup + g) * (C + 1) + gj * kGroup + 2 * q;
#pragma unroll
  for (int y = 0; y < RIGHTS; ++y) {
    to[0][y][at] = acc[y][0], to[0][y][at + 1] = acc[y][1];
    if (LEFTS == 2) to[LEFTS - 1][y][at] = acc[y][2], to[LEFTS - 1][y][at + 1] = acc[y][3];
  }
}

// (I + l)^-1 of both halves of sixteen tokens on the diagonal of l [C][C], to `inverse` [C][kLdT], by one warp: a lane per column.
__device__ __forceinline__ void invert_halves(const float* l, float* inverse) {
  const int lane = threadIdx.x & 31, half = lane & 16, column = lane & 15;
  float x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float sum0 = i == column ? 1.f : 0.f, sum1 = 0.f;
#pragma unroll
    for (int j = 0; j < i; j += 4) {
      const float4 row = *reinterpret_cast<const float4*>(l + (half + i) * C + half + j);
      sum0 = fmaf(-row.x, x[j], sum0);
      if (j + 1 < i) sum1 = fmaf(-row.y, x[j + 1], sum1);
      if (j + 2 < i) sum0 = fmaf(-row.z, x[j + 2], sum0);
      if (j + 3 < i) sum1 = fmaf(-row.w, x[j + 3], sum1);
    }
    x[i] = sum0 + sum1;
    inverse[(half + i) * kLdT + column] = i >= column ? x[i] : 0.f;
  }
}

// Sixteen columns of numbers by token, of which a lane has columns g and g + 8, tokens 4 q .. + 3 of both halves: [half][column].
struct Columns {
  float4 v[2][2];
};
__device__ __forceinline__ SplitA split_columns(const float4 (&v)[2]) { return split_rows(v[0], v[1]); }
// The same of a triangle that all columns meet: its operands in parts, [tile][part][lane], made once.
constexpr int kTriangle = 2 * 3 * 32;  // uint2 of sixteen rows by sixteen tokens
__device__ __forceinline__ void pack_triangle(uint2* to, const float* m, int ld) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const SplitB b(*reinterpret_cast<const float4*>(m + in_sixteen(t, g) * ld + 4 * q));
#pragma unroll
    for (int p = 0; p < 3; ++p) to[(t * 3 + p) * 32 + lane] = make_uint2(b.lo.part[p], b.hi.part[p]);
  }
}
__device__ __forceinline__ void times_triangle(float4 (&to)[2], const SplitA& a, const uint2* m) {
  const int lane = threadIdx.x & 31;
  float part[2][4];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    SplitB b;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint2 word = m[(t * 3 + p) * 32 + lane];
      b.lo.part[p] = word.x, b.hi.part[p] = word.y;
    }
    mma_split(part[t], a, b);
  }
  to[0] = make_float4(part[0][0], part[0][1], part[1][0], part[1][1]);
  to[1] = make_float4(part[0][2], part[0][3], part[1][2], part[1][3]);
}
// a (sixteen columns by sixteen tokens) times the transposed sixteen rows of m, `ld` numbers apart.
__device__ __forceinline__ void times_rows(float4 (&to)[2], const SplitA& a, const float* m, int ld) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  float part[2][4];
#pragma unroll
  for (int t = 0; t < 2; ++t) mma_split(part[t], a, SplitB(*reinterpret_cast<const float4*>(m + in_sixteen(t, g) * ld + 4 * q)));
  to[0] = make_float4(part[0][0], part[0][1], part[1][0], part[1][1]);
  to[1] = make_float4(part[0][2], part[0][3], part[1][2], part[1][3]);
}
__device__ __forceinline__ float4 minus(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
__device__ __forceinline__ float4 plus(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// What is not finite must not reach the tokens in front of it by way of a zero in a triangle: it goes into the products as a zero, and the
// tokens from it on are NaN behind them. Lowers `first` to the first such token of the lane's two columns in half h.
__device__ __forceinline__ void take_out(float4 (&r)[2], int h, int2& first) {
  if (!__any_sync(0xffffffffu, !all_finite(r[0]) || !all_finite(r[1]))) return;
  const int q = threadIdx.x & 3;
  int found[2] = {C, C};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float* v[4] = {&r[c].x, &r[c].y, &r[c].z, &r[c].w};
#pragma unroll
    for (int i = 3; i >= 0; --i)
      if (!isfinite(*v[i])) *v[i] = 0.f, found[c] = h * 16 + 4 * q + i;
    found[c] = min(found[c], __shfl_xor_sync(0xffffffffu, found[c], 1));
    found[c] = min(found[c], __shfl_xor_sync(0xffffffffu, found[c], 2));
  }
  first.x = min(first.x, found[0]), first.y = min(first.y, found[1]);
}
// The lane's numbers of tokens from `from` on become NaN, those from n on zeros.
__device__ __forceinline__ void put_back(Columns& x, int2 from, int n) {
  if (n == C && !__any_sync(0xffffffffu, min(from.x, from.y) < C)) return;
  const int q = threadIdx.x & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float* v[4] = {&x.v[h][c].x, &x.v[h][c].y, &x.v[h][c].z, &x.v[h][c].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int token = h * 16 + 4 * q + i;
        if (token >= (c == 0 ? from.x : from.y)) *v[i] = NAN;
        if (token >= n) *v[i] = 0.f;
      }
    }
}
// (I + l) x = r in place; `triangles`: T11, L21 and T22; `spoilt`: the first token of either column that is not to be read any more; zeros
// from token n on.
__device__ __forceinline__ void solve_columns(Columns& r, const uint2* triangles, int2 spoilt, int n) {
  float4 product[2];
  take_out(r.v[0], 0, spoilt);
  times_triangle(r.v[0], split_columns(r.v[0]), triangles);
  times_triangle(product, split_columns(r.v[0]), triangles + kTriangle);
  r.v[1][0] = minus(r.v[1][0], product[0]), r.v[1][1] = minus(r.v[1][1], product[1]);
  take_out(r.v[1], 1, spoilt);
  times_triangle(r.v[1], split_columns(r.v[1]), triangles + 2 * kTriangle);
  put_back(r, spoilt, n);
}
// To `y` (rows row0 .. + 15 of the state) or to `x` (columns from `to` on).
__device__ __forceinline__ void store_y(float* y, int row0, const Columns& r) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  float* to = y + y_place(4 * q, row0) + g;  // tokens 4 q + i: i / 2 is the tile, i % 2 the next lane's
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float v[4] = {r.v[h][c].x, r.v[h][c].y, r.v[h][c].z, r.v[h][c].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) to[h * 256 + i / 2 * 128 + i % 2 * 16 + 8 * c] = v[i];
    }
}
__device__ __forceinline__ void store_x(float* x, const Columns& r) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < 2; ++c) *reinterpret_cast<float4*>(x + (g + 8 * c) * C + h * 16 + 4 * q) = r.v[h][c];
}
// Columns c0 .. + 15 of the chunk's values: rows v + token * ld, zeros past n tokens and dv columns.
__device__ __forceinline__ Columns load_values(const float* v, int64_t ld, int c0, int dv, int n) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const float* base = v + 4 * q * ld + c0 + g;
  Columns r;
  if (n == C && c0 + 16 <= dv) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) (&r.v[h][c].x)[i] = base[(h * 16 + i) * ld + 8 * c];
    return r;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int token = h * 16 + 4 * q, column = c0 + g + 8 * c;
      const float* at = base + h * 16 * ld + 8 * c;
      r.v[h][c] = make_float4(column < dv && token < n ? at[0] : 0.f, column < dv && token + 1 < n ? at[ld] : 0.f,
                              column < dv && token + 2 < n ? at[2 * ld] : 0.f, column < dv && token + 3 < n ? at[3 * ld] : 0.f);
    }
  return r;
}

size_t prepare_smem(int rows) { return sizeof(float) * (3 * C * (rows + 4) + 2 * kGroups * rows + C * C + 3 * C + 2 * C * (C + 1)); }

template <int ROWS, int W, bool PER_HEAD>
__global__ void __launch_bounds__(kThreads, ROWS <= 128 ? 3 : 1)
chunk_prepare_kernel(const float* q, const float* k, const float* v, const float* beta, const float* decay, const int* __restrict__ seq_q_start,
                     const int* __restrict__ seq_q_len, int heads, int kv_heads, int dk, int dv, Scratch to) {
  extern __shared__ __align__(16) float chunk_smem[];
  let_successor_start();
  const int seq = blockIdx.z, own_head = blockIdx.y, head = to.head0 + own_head, chunk = blockIdx.x;
  const int n = min(C, seq_q_len[seq] - chunk * C);
  if (n <= 0) return;
  const int start = seq_q_start[seq], kvh = head / (heads / kv_heads);
  const int64_t first = static_cast<int64_t>(start) + chunk * C, place = chunk_place(start, seq, chunk) * to.heads + own_head;
  constexpr int rows = ROWS, ld = ROWS + 4;
  const int columns = padded_columns(dv);
  float* ks = chunk_smem;                     // [C][ld]: keys, then times the decays of their group up to their own token
  float* qs = ks + C * ld;                    // [C][ld]: queries, then likewise
  float* gs = qs + C * ld;                    // [C][ld]: decays, then keys times the decays from the next token to their group's end
  float* whole = gs + C * ld;                 // [groups][rows]: each group's decays multiplied
  float* front = whole + kGroups * rows;      // [groups][rows]: the decays in front of each group multiplied
  float* ls = front + kGroups * rows;         // [C][C]
  float* bs = ls + C * C;                     // [C]: beta
  float* es = bs + C;                         // [C]: PER_HEAD: e_i
  float* fs = es + C;                         // [C]: PER_HEAD: G_last,j
  float* kk = fs + C;                         // [C][C + 1]: k_i . G_ij k_j
  float* qk = kk + C * (C + 1);               // [C][C + 1]: q_i . G_ij k_j
  uint2* triangles = reinterpret_cast<uint2*>(kk);  // [3][kTriangle], behind the pairs
  float* inverse = kk + 6 * kTriangle;              // [C][kLdT]
  static_assert(6 * kTriangle + C * kLdT <= 2 * C * (C + 1), "the triangles do not fit where the pairs were");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  wait_for_predecessor();
  const int64_t qk_ld = static_cast<int64_t>(kv_heads) * dk, qk_at = first * qk_ld + static_cast<int64_t>(kvh) * dk;
  stage_rows<ROWS, W>(ks, k + qk_at, n, qk_ld, dk);
  stage_rows<ROWS, W>(qs, q + qk_at, n, qk_ld, dk);
  if (!PER_HEAD) stage_rows<ROWS, W>(gs, decay + (first * heads + head) * dk, n, static_cast<int64_t>(heads) * dk, dk);
  if (tid < C) bs[tid] = tid < n ? beta[(first + tid) * heads + head] : 0.f;
  commit_copies();
  wait_copies<0>();
  __syncthreads();
  if (PER_HEAD) {
    for (int tile = warp; tile < kTiles; tile += kWarps) pair_tile<ROWS, 2, 1, false>(ks, qs, {ks}, nullptr, tile, {{kk}, {qk}});
  } else {
    if (warp < kGroups) pairs_in_group<ROWS, false, false>(ks, ks, gs, warp, kk);
    else pairs_in_group<ROWS, false, true>(qs, ks, gs, warp - kGroups, qk);
    __syncthreads();
    for (int item = tid; item < kGroups * rows; item += kThreads) {  // a thread per (group, channel)
      const int c = item % rows, at = item / rows * kGroup * ld + c;
      float key[kGroup], g[kGroup];
      float run = 1.f;
#pragma unroll
      for (int r = 0; r < kGroup; ++r) {
        key[r] = ks[at + r * ld];
        g[r] = item / rows * kGroup + r < n ? gs[at + r * ld] : 1.f;
        run *= g[r];
        ks[at + r * ld] = key[r] * run;
        qs[at + r * ld] *= run;
      }
      whole[item] = run;
      run = 1.f;
#pragma unroll
      for (int r = kGroup - 1; r >= 0; --r) {
        gs[at + r * ld] = key[r] * run;
        run *= g[r];
      }
    }
    __syncthreads();
    if (warp < kBetween) pair_tile<ROWS, 2, 1, true>(ks, qs, {gs}, whole, warp, {{kk}, {qk}});
  }
  __syncthreads();
  float* a = to.a + place * C * C + lane;
  if (!PER_HEAD) {
#pragma unroll
    for (int i = warp; i < C; i += kWarps) {
      ls[i * C + lane] = lane < i ? bs[i] * kk[i * (C + 1) + lane] : 0.f;
      a[i * C] = lane <= i ? qk[i * (C + 1) + lane] : 0.f;
    }
  } else {
    float own = 0.f, d = 0.f, prefix = 0.f, e = 0.f;
    own = lane < n ? decay[(first + lane) * heads + head] : 0.f;
    for (int i = 0; i < C; ++i) {
      {  // D_ij of column j = lane, the sum of the logarithms from token j + 1 on, grows with i from zero at i = j
        const float gi = __shfl_sync(0xffffffffu, own, i);
        d = i > lane ? d + gi : 0.f;
        prefix += gi;
        if (i == lane) e = prefix;
      }
      if ((i & 7) == warp) {
        const float between = expf(d);
        ls[i * C + lane] = lane < i ? bs[i] * between * kk[i * (C + 1) + lane] : 0.f;
        a[i * C] = lane <= i ? between * qk[i * (C + 1) + lane] : 0.f;
      }
    }
    if (warp == 0) es[lane] = expf(e), fs[lane] = expf(d);  // d is now D_last,j: tokens past n added nothing
  }
  __syncthreads();
  if (warp == 0) {
    invert_halves(ls, inverse);
    __syncwarp();
    pack_triangle(triangles, inverse, kLdT), pack_triangle(triangles + 2 * kTriangle, inverse + 16 * kLdT, kLdT);
  } else if (warp == 1) {
    pack_triangle(triangles + kTriangle, ls + 16 * C, C);
  }
  // Scaled rows: a thread per (half of the chunk, channel). The warp that inverts is the last to come.
  for (int item = kThreads - 1 - tid; item < 2 * rows; item += kThreads) {
    const int column = item % rows, half = item / rows;
    float* qt = to.qt + (place * C + half * 16) * rows + column;
    float* kd = to.kd + place * rows * C + kd_place(half * 16, column);
    float before[2], after[2];  // whole groups in front of and behind the half's two
    if (!PER_HEAD) {
      before[0] = 1.f, after[1] = 1.f;
      for (int g = 0; g < 2 * half; ++g) before[0] *= whole[g * rows + column];
      before[1] = before[0] * whole[2 * half * rows + column];
      for (int g = 2 * half + 2; g < kGroups; ++g) after[1] *= whole[g * rows + column];
      after[0] = after[1] * whole[(2 * half + 1) * rows + column];
      front[2 * half * rows + column] = before[0], front[(2 * half + 1) * rows + column] = before[1];
      if (half == 1) to.e[place * rows + column] = before[1] * whole[3 * rows + column];
    } else if (half == 1) {
      to.e[place * rows + column] = es[n - 1];
    }
#pragma unroll
    for (int i0 = 0; i0 < 16; i0 += 4) {
      float decayed[4];
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int i = half * 16 + i0 + y;
        qt[(i0 + y) * rows] = (PER_HEAD ? es[i] : before[i0 / kGroup]) * qs[i * ld + column];
        decayed[y] = i < n ? (PER_HEAD ? fs[i] * ks[i * ld + column] : after[i0 / kGroup] * gs[i * ld + column]) : 0.f;
      }
      *reinterpret_cast<float4*>(kd + kd_place(i0, 0)) = make_float4(decayed[0], decayed[1], decayed[2], decayed[3]);
    }
  }
  __syncthreads();
  for (int tile = warp; tile < (rows + columns) / 16; tile += kWarps) {  // sixteen columns of [-beta e K | beta V]
    const int g = lane >> 2, q4 = 4 * (lane & 3);
    Columns r;
    if (tile < rows / 16) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int column = tile * 16 + g + 8 * c, token = h * 16 + q4;
          const float4 b = *reinterpret_cast<const float4*>(bs + token), e = PER_HEAD ? *reinterpret_cast<const float4*>(es + token) : b;
          const float before = PER_HEAD ? 1.f : front[token / kGroup * rows + column];
          const float* key = ks + token * ld + column;
          r.v[h][c] = make_float4(-b.x * ((PER_HEAD ? e.x : before) * key[0]), -b.y * ((PER_HEAD ? e.y : before) * key[ld]),
                                  -b.z * ((PER_HEAD ? e.z : before) * key[2 * ld]), -b.w * ((PER_HEAD ? e.w : before) * key[3 * ld]));
        }
    } else {
      r = load_values(v + (first * heads + head) * dv, static_cast<int64_t>(heads) * dv, (tile - rows / 16) * 16, dv, n);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 b = *reinterpret_cast<const float4*>(bs + h * 16 + q4);
#pragma unroll
        for (int c = 0; c < 2; ++c) r.v[h][c].x *= b.x, r.v[h][c].y *= b.y, r.v[h][c].z *= b.z, r.v[h][c].w *= b.w;
      }
    }
    solve_columns(r, triangles, make_int2(C, C), n);
    if (tile < rows / 16) store_y(to.y + place * rows * C, tile * 16, r);
    else store_x(to.x + (place * columns + tile * 16 - rows) * C, r);
  }
}

// --- the same for rules in which the values enter as they are ---------------------------------------------------------------------------
//
// GENERAL: S <- w S + b (u^T S) + k v^T, o = S^T r, with b = -au. kLinear: S <- w S + k v^T, o = S^T r + bonus v read before the update.
// MEMORY: S <- keep S + put k v^T and n <- keep n + put k with two numbers per head and token, o = S^T r and n . r after the update, r
// times `scale`: pairs are products of the raw rows, times the keeps between them.
// One block per (chunk, head, request); the sums of the values (G_last K)^T V go where the chunk's state will be.
constexpr int kMaxLinearRows = 128;

size_t linear_prepare_smem(int rows, int rule) {
  const bool general = rule == kGeneralDelta;
  return sizeof(float) * ((general ? 5 : (rule == kMemory ? 2 : 3)) * C * (rows + 4) + 2 * C + kGroups * rows + (general ? 4 : 1) * C * (C + 1) +
                          (general ? 2 * C * C : 0));
}

struct LinearRule {
  const float* r;
  const float* k;
  const float* v;
  const float* w;
  const float* au;     // GENERAL
  const float* u;      // GENERAL
  const float* bonus;  // kLinear: [tokens][heads]
  const float* put;    // MEMORY: [tokens][heads], as is w (the keeps)
  float scale;         // MEMORY
  int64_t ld;          // numbers from token to token of r, k, w, au and u (a head's numbers start at head * dk)
  int64_t v_ld;        // of v (at head * dv)
};

template <int ROWS, int W, int RULE>
__global__ void __launch_bounds__(kThreads, ROWS <= 64 ? 3 : 2)
linear_chunk_prepare_kernel(LinearRule in, const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int heads, int dk, int dv, Scratch to) {
  extern __shared__ __align__(16) float chunk_smem[];
  let_successor_start();
  const int seq = blockIdx.z, own_head = blockIdx.y, head = to.head0 + own_head, chunk = blockIdx.x;
  const int n = min(C, seq_q_len[seq] - chunk * C);
  if (n <= 0) return;
  const int start = seq_q_start[seq];
  const int64_t first = static_cast<int64_t>(start) + chunk * C, place = chunk_place(start, seq, chunk) * to.heads + own_head;
  constexpr int rows = ROWS, ld = ROWS + 4;
  const int columns = padded_columns(dv);
  constexpr bool GENERAL = RULE == kGeneralDelta, MEMORY = RULE == kMemory;
  float* ls = chunk_smem;                                // GENERAL: [C][C]: -N
  float* ms = ls + (GENERAL ? C * C : 0);                // GENERAL: [C][C]: M
  float* rs = ms + (GENERAL ? C * C : 0);                // [C][ld]: r, then times the decays of its group in front of (GENERAL: up to) its token
  float* ks = rs + C * ld;                               // [C][ld]: k, then times the decays from the next token to its group's, then the chunk's end
  float* gs = ks + C * ld;                               // [C][ld]
  float* us = gs + (MEMORY ? 0 : C * ld);                // GENERAL: [C][ld]: u, then times the decays of its group in front of its token
  float* bb = us + (GENERAL ? C * ld : 0);               // GENERAL: [C][ld]: -au, then as k
  float* whole = bb + (GENERAL ? C * ld : 0);            // [groups][rows]
  float* es = whole + kGroups * rows;                    // MEMORY: [C]: the keeps up to a token, multiplied
  float* fs = es + C;                                    // MEMORY: [C]: the keeps behind a token times its put
  float* rk = fs + C;                                    // [C][C + 1]: r_i . G k_j
  float* uk = rk + C * (C + 1);
  float* rb = uk + C * (C + 1);
  float* ub = rb + C * (C + 1);
  uint2* triangles = reinterpret_cast<uint2*>(rk);       // GENERAL: [3][kTriangle], behind the pairs
  float* inverse = rk + 6 * kTriangle;                   // GENERAL: [C][kLdT], likewise
  float* front = gs;                                     // GENERAL: [groups][rows]: the decays in front of each group, behind the decays themselves
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int64_t at_in = first * in.ld + static_cast<int64_t>(head) * dk;
  const float* values = in.v + first * in.v_ld + static_cast<int64_t>(head) * dv;
  wait_for_predecessor();
  stage_rows<ROWS, W>(rs, in.r + at_in, n, in.ld, dk);
  stage_rows<ROWS, W>(ks, in.k + at_in, n, in.ld, dk);
  if (!MEMORY) stage_rows<ROWS, W>(gs, in.w + at_in, n, in.ld, dk);
  if (GENERAL) {
    stage_rows<ROWS, W>(us, in.u + at_in, n, in.ld, dk);
    stage_rows<ROWS, W>(bb, in.au + at_in, n, in.ld, dk);
  }
  commit_copies();
  wait_copies<0>();
  __syncthreads();
  if (MEMORY) {
    for (int tile = warp; tile < kTiles; tile += kWarps) pair_tile<ROWS, 1, 1, false>(rs, nullptr, {ks}, nullptr, tile, {{rk}});
    __syncthreads();
    // Column j = lane: the keeps of tokens j + 1 .. i multiplied, from one at i = j on.
    const int64_t at = (first + lane) * heads + head;
    const float keep = lane < n ? in.w[at] : 1.f, put = lane < n ? in.put[at] : 0.f;
    float d = 1.f, prefix = 1.f, e = 1.f;
    for (int i = 0; i < C; ++i) {
      const float own = __shfl_sync(0xffffffffu, keep, i);
      d = i > lane ? d * own : 1.f;
      prefix *= own;
      if (i == lane) e = prefix;
      if ((i & 7) == warp) to.av[(place * C + i) * C + lane] = lane <= i ? d * put * rk[i * (C + 1) + lane] * in.scale : 0.f;
    }
    if (warp == 0) es[lane] = e, fs[lane] = d * put;
    __syncthreads();
    for (int c = tid; c < rows; c += kThreads) {
      float* qt = to.qt + place * C * rows + c;
      float sum = 0.f;
#pragma unroll 8
      for (int i = 0; i < C; ++i) {
        const float key = fs[i] * ks[i * ld + c];
        ks[i * ld + c] = key;
        sum += key;
        qt[i * rows] = es[i] * in.scale * rs[i * ld + c];
      }
      to.n[place * rows + c] = sum;
      to.e[place * rows + c] = es[n - 1];
    }
    __syncthreads();
  } else {
    if (warp < kGroups) {
      // One after the other through the same code: an SM holds about half of this kernel's.
#pragma unroll 1
      for (int right = 0; right < (GENERAL ? 2 : 1); ++right)
        pairs_in_group<ROWS, true, false>(GENERAL ? us : rs, right == 0 ? ks : bb, gs, warp, GENERAL ? (right == 0 ? uk : ub) : rk);
    } else if (GENERAL) {
#pragma unroll 1
      for (int right = 0; right < 2; ++right) pairs_in_group<ROWS, false, true>(rs, right == 0 ? ks : bb, gs, warp - kGroups, right == 0 ? rk : rb);
    }
    __syncthreads();
    for (int item = tid; item < kGroups * rows; item += kThreads) {  // a thread per (group, channel)
      const int c = item % rows, at = item / rows * kGroup * ld + c;
      float decays[kGroup];
      float run = 1.f;
#pragma unroll
      for (int r = 0; r < kGroup; ++r) {
        decays[r] = item / rows * kGroup + r < n ? gs[at + r * ld] : 1.f;
        if (GENERAL) us[at + r * ld] *= run;
        else rs[at + r * ld] *= run;
        run *= decays[r];
        if (GENERAL) rs[at + r * ld] *= run;
      }
      whole[item] = run;
      run = 1.f;
#pragma unroll
      for (int r = kGroup - 1; r >= 0; --r) {
        ks[at + r * ld] *= run;
        if (GENERAL) bb[at + r * ld] *= run;
        run *= decays[r];
      }
    }
    __syncthreads();
    if (warp < kBetween) {
      if constexpr (GENERAL) pair_tile<ROWS, 2, 2, true>(us, rs, {ks, bb}, whole, warp, {{uk, ub}, {rk, rb}});
      else pair_tile<ROWS, 1, 1, true>(rs, nullptr, {ks}, whole, warp, {{rk}});
    }
    __syncthreads();
    for (int i = warp; i < C; i += kWarps) {
      const int at = i * (C + 1) + lane;
      const int64_t row = (place * C + i) * C + lane;
      if (GENERAL) {  // au came in with its own sign: b = -au
        ls[i * C + lane] = lane < i ? ub[at] : 0.f;
        ms[i * C + lane] = lane < i ? uk[at] : 0.f;
        to.a[row] = lane <= i ? -rb[at] : 0.f;
        to.av[row] = lane <= i ? rk[at] : 0.f;
      } else {
        to.av[row] = lane < i ? rk[at] : (lane == i && i < n ? in.bonus[(first + i) * heads + head] : 0.f);
      }
    }
    // Scaled rows: r times all decays in front of (or up to) its token, k and b times all decays behind theirs; a thread per (group, channel).
    for (int item = tid; item < kGroups * rows; item += kThreads) {
      const int c = item % rows, group = item / rows;
      float before = 1.f, after = 1.f;
#pragma unroll
      for (int x = 0; x < kGroups - 1; ++x) {
        before *= x < group ? whole[x * rows + c] : 1.f;
        after *= x + 1 > group ? whole[(x + 1) * rows + c] : 1.f;
      }
      float* qt = to.qt + (place * C + group * kGroup) * rows + c;
#pragma unroll
      for (int r = 0; r < kGroup; ++r) {
        const int at = (group * kGroup + r) * ld + c;
        qt[r * rows] = before * rs[at];
        ks[at] *= after;
      }
      if (GENERAL) {
        front[item] = before;
        float decayed[kGroup];
#pragma unroll
        for (int r = 0; r < kGroup; ++r) decayed[r] = group * kGroup + r < n ? -after * bb[(group * kGroup + r) * ld + c] : 0.f;
        float* kd = to.kd + place * rows * C + kd_place(group * kGroup, c);
        *reinterpret_cast<float4*>(kd) = make_float4(decayed[0], decayed[1], decayed[2], decayed[3]);
        *reinterpret_cast<float4*>(kd + 4) = make_float4(decayed[4], decayed[5], decayed[6], decayed[7]);
      }
      if (group == kGroups - 1) to.e[place * rows + c] = before * whole[item];
    }
    __syncthreads();
    if (GENERAL) {
      if (warp == 0) {
        invert_halves(ls, inverse);
        __syncwarp();
        pack_triangle(triangles, inverse, kLdT), pack_triangle(triangles + 2 * kTriangle, inverse + 16 * kLdT, kLdT);
      } else if (warp == 1) {
        pack_triangle(triangles + kTriangle, ls + 16 * C, C);
      }
      __syncthreads();
      for (int tile = warp; tile < (rows + columns) / 16; tile += kWarps) {  // sixteen columns of [e U | M V]
        Columns r;
        int2 spoilt = make_int2(C, C);
        if (tile < rows / 16) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int column = tile * 16 + g + 8 * c, token = h * 16 + 4 * q;
              const float before = front[token / kGroup * rows + column];
              const float* at = us + token * ld + column;
              r.v[h][c] = make_float4(before * at[0], before * at[ld], before * at[2 * ld], before * at[3 * ld]);
            }
        } else {
          r = load_values(values, in.v_ld, (tile - rows / 16) * 16, dv, n);
          take_out(r.v[0], 0, spoilt), take_out(r.v[1], 1, spoilt);
          const SplitA v0 = split_columns(r.v[0]), v1 = split_columns(r.v[1]);
          float4 more[2];
          times_rows(r.v[0], v0, ms, C);
          times_rows(r.v[1], v0, ms + 16 * C, C);
          times_rows(more, v1, ms + 16 * C + 16, C);
          r.v[1][0] = plus(r.v[1][0], more[0]), r.v[1][1] = plus(r.v[1][1], more[1]);
        }
        solve_columns(r, triangles, spoilt, n);
        if (tile < rows / 16) store_y(to.y + place * rows * C, tile * 16, r);
        else store_x(to.x + (place * columns + tile * 16 - rows) * C, r);
      }
    }
  }
  // (G_last K)^T V, transposed: sixteen columns by 32 rows a warp at a time.
  for (int item = warp; item < columns / 16 * (rows / 32); item += kWarps) {
    const int col0 = item / (rows / 32) * 16, row0 = item % (rows / 32) * 32;
    const Columns r = load_values(values, in.v_ld, col0, dv, n);
    const SplitA left[2] = {split_columns(r.v[0]), split_columns(r.v[1])};
#pragma unroll
    for (int block = 0; block < 2; ++block) {
      float part[2][2][4];  // [tile][half of the tokens]
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float* at = ks + (h * 16 + 4 * q) * ld + row0 + block * 16 + in_sixteen(t, g);
          mma_split(part[t][h], left[h], SplitB(make_float4(at[0], at[ld], at[2 * ld], at[3 * ld])));
        }
      float* s = to.s + place * columns * rows + s_place(col0, row0 + block * 16, rows) + lane * 4;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        *reinterpret_cast<float4*>(s + c * 128) = make_float4(part[0][0][2 * c] + part[0][1][2 * c], part[0][0][2 * c + 1] + part[0][1][2 * c + 1],
                                                              part[1][0][2 * c] + part[1][1][2 * c], part[1][0][2 * c + 1] + part[1][1][2 * c + 1]);
    }
  }
}

// Four neighbouring rows of a column of a head's state a thread, from chunk to chunk: eight chunks' sums are asked for at a time. A warp
// has eight columns of sixteen rows, so that the state, whose rows run the other way, is read and written in whole sectors too.
constexpr int kScanThreads = 64;  // small blocks: 24 heads of 64 x 64 are 384 of them, one for every warp scheduler of the chip
__global__ void __launch_bounds__(kScanThreads, 1)
chunk_scan_kernel(const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, const int* __restrict__ seq_slot, int heads, int dk, int dv, Scratch from,
                  float* state, float* normaliser) {
  let_successor_start();
  const int seq = blockIdx.z, own_head = blockIdx.y, head = from.head0 + own_head;
  const int start = seq_q_start[seq], len = seq_q_len[seq], chunks = (len + C - 1) / C;
  const int rows = padded_rows(dk), columns = padded_columns(dv);
  const int idx = blockIdx.x * kScanThreads + threadIdx.x;
  if (idx * 4 >= rows * columns) {  // the blocks behind the state's: a number of the normaliser a thread
    const int c = idx - (rows * columns / 4 + kScanThreads - 1) / kScanThreads * kScanThreads;
    if (normaliser == nullptr || c < 0 || c >= rows) return;
    wait_for_predecessor();
    float* own = normaliser + (static_cast<int64_t>(seq_slot[seq]) * heads + head) * dk + c;
    float n = c < dk ? *own : 0.f;
    const int64_t step = static_cast<int64_t>(from.heads) * rows, at = (chunk_place(start, seq, 0) * from.heads + own_head) * rows + c;
    for (int chunk = 0; chunk < chunks; ++chunk) {
      const float add = from.n[at + chunk * step];
      from.n[at + chunk * step] = n;
      n = fmaf(from.e[at + chunk * step], n, add);
    }
    if (c < dk && chunks > 0) *own = n;
    return;
  }
  const int tile = idx / 32, lane = threadIdx.x & 31;  // `s_place` from thread to thread
  const int row = tile / 2 % (rows / 16) * 16 + (lane & 3) * 4, col = tile / 2 / (rows / 16) * 16 + (tile & 1) * 8 + lane / 4;
  float* base = state + (static_cast<int64_t>(seq_slot[seq]) * heads + head) * dk * dv + static_cast<int64_t>(row) * dv + col;
  float s[4];
  wait_for_predecessor();
#pragma unroll
  for (int x = 0; x < 4; ++x) s[x] = row + x < dk && col < dv ? base[static_cast<int64_t>(x) * dv] : 0.f;
  const int64_t place = chunk_place(start, seq, 0) * from.heads + own_head;
  const float* e = from.e + place * rows + row;
  float* sums = from.s + place * columns * rows + idx * 4;
  const int64_t step_e = static_cast<int64_t>(from.heads) * rows, step = step_e * columns;
  constexpr int kAhead = 8;
  for (int chunk = 0; chunk < chunks; chunk += kAhead) {
    float4 add[kAhead], keep[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (chunk + i < chunks) add[i] = *reinterpret_cast<const float4*>(sums + (chunk + i) * step), keep[i] = *reinterpret_cast<const float4*>(e + (chunk + i) * step_e);
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (chunk + i < chunks) {
        *reinterpret_cast<float4*>(sums + (chunk + i) * step) = make_float4(s[0], s[1], s[2], s[3]);
        s[0] = fmaf(keep[i].x, s[0], add[i].x), s[1] = fmaf(keep[i].y, s[1], add[i].y);
        s[2] = fmaf(keep[i].z, s[2], add[i].z), s[3] = fmaf(keep[i].w, s[3], add[i].w);
      }
  }
  if (chunks > 0) {
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (row + x < dk && col < dv) base[static_cast<int64_t>(x) * dv] = s[x];
  }
}

// --- the walk ------------------------------------------------------------------------------------------------------------------------
//
// One block per (16 columns of the state, head, request), a warp per 16 rows, which it keeps in registers, transposed, as the tensor core
// leaves them (D: 16 columns x 2 times 8 rows): D's layout is A's, so the state goes into the next chunk's first product without leaving
// its lanes. That product, U^T = W^T + S^T Y^T, is summed over the warps through shared memory, each warp adding up its share of the sums; S^T <-
// e S^T + U^T Kd then wants nothing of the other warps. A lane's share of the operands comes by its own asynchronous copies, one or two chunks ahead,
// so that nobody waits for anybody's (loads into registers a chunk ahead did: 101 us where this takes 80, a third of it spent
// waiting for memory; copies that also go into L1 112).
// What bounds it: the chain product, sum over warps, product, in turn and once a chunk: 2,400 cycles, of which the tensor core works 830 (heads
// of 128 x 128). Tried: operands in parts in memory, made where they are prepared, half as many bytes again: 76 us, but 5 us more there;
// taking them apart while the warps wait for one another: 95 us.
constexpr int kSumPairs = 8;  // pairs of U^T's numbers that a lane holds: (half of the chunk, pair of four tokens, column g or g + 8)
// Three stages where two blocks then still fit an SM: with what the values add, up to 64 rows (128 rows in three stages had an SM to themselves: generalized
// rule, 28 heads of 128 x 128, all three kernels, 2,048 tokens 410 us, in two stages 372; 8 requests of 300 tokens 470 and 430).
__host__ __device__ constexpr int walk_stages(int rows, bool add) { return rows <= (add ? 64 : 128) ? 3 : 2; }
__host__ __device__ constexpr int own_pairs(int rows) { return rows < 16 * kSumPairs ? 16 * kSumPairs / rows : 1; }  // that a warp adds up
// Bytes of a stage: per lane four pieces of y, four of kd, two of what the values add and its pairs of W; and e.
__host__ __device__ constexpr int walk_stage(int rows, bool add) { return 2 * rows * (16 * (add ? 10 : 8) + 8 * own_pairs(rows)) + 4 * rows; }
constexpr size_t walk_smem(int rows, bool add) { return walk_stages(rows, add) * walk_stage(rows, add); }
static_assert(2 * (walk_smem(128, false) + 5 * 1024) <= 228 * 1024 && 2 * (walk_smem(128, true) + 5 * 1024) <= 228 * 1024, "two blocks of 128 rows do not fit an SM");

template <int ROWS, bool ADD>  // ADD: what the values alone add to S stands where the chunk's state goes
__global__ void __launch_bounds__(2 * ROWS, ROWS <= 128 ? 2 : 1)
chunk_walk_kernel(const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, const int* __restrict__ seq_slot, int heads, int dk, int dv,
                  Scratch from, float* state) {
  extern __shared__ __align__(16) float chunk_smem[];
  constexpr int kParts = ROWS / 16, kOwn = own_pairs(ROWS), kLanes = 2 * ROWS, kStages = walk_stages(ROWS, ADD);
  constexpr int kPairsAt = (ADD ? 10 : 8) * kLanes * 4, kDecaysAt = kPairsAt + kOwn * kLanes * 2;  // in a stage
  __shared__ uint4 us[2][3][32];  // U^T in parts, as the lanes of every warp want it
  let_successor_start();
  const int col0 = blockIdx.x * kColumns, own_head = blockIdx.y, head = from.head0 + own_head, seq = blockIdx.z;
  const int start = seq_q_start[seq], len = seq_q_len[seq];
  const int columns = padded_columns(dv), chunks = (len + C - 1) / C;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int row0 = warp * 16 + 4 * q;  // the four rows that the lane keeps, of columns g and g + 8
  const bool adds_up = kParts <= kSumPairs || warp < kSumPairs;
  const int64_t place = chunk_place(start, seq, 0) * from.heads + own_head;
  const float* y = from.y + place * ROWS * C + warp * 16 * C + lane * 4;
  const float* kd = from.kd + place * ROWS * C + warp * 16 * C + lane * 4;
  const float* e = from.e + place * ROWS + row0;
  float* s_out = from.s + place * columns * ROWS + col0 * ROWS + warp * 256 + lane * 4;
  int64_t x_at[kOwn];
#pragma unroll
  for (int o = 0; o < kOwn; ++o) {
    const int pair = warp + o * kParts;
    x_at[o] = (place * columns + col0 + g + 8 * (pair & 1)) * C + 16 * (pair >> 2) + 4 * q + (pair & 2);
  }
  const int64_t step = from.heads, step_y = step * C * ROWS, step_s = step * columns * ROWS, step_x = step * columns * C;
  auto stage_of = [&](int chunk) { return chunk_smem + chunk % kStages * (walk_stage(ROWS, ADD) / 4); };
  auto fetch = [&](int chunk) {
    if (chunk < chunks) {
      float* stage = stage_of(chunk) + tid * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        stage_copy<16>(stage + i * kLanes * 4, y + chunk * step_y + i * 128, true);
        stage_copy<16>(stage + (4 + i) * kLanes * 4, kd + chunk * step_y + i * 128, true);
      }
      if (ADD) {
        stage_copy<16>(stage + 8 * kLanes * 4, s_out + chunk * step_s, true);
        stage_copy<16>(stage + 9 * kLanes * 4, s_out + chunk * step_s + 128, true);
      }
      if (lane < 4) stage_copy<16>(stage_of(chunk) + kDecaysAt + row0, e + chunk * step * ROWS, true);
#pragma unroll
      for (int o = 0; o < kOwn; ++o)
        if (adds_up) stage_copy<8>(stage_of(chunk) + kPairsAt + (o * kLanes + tid) * 2, from.x + x_at[o] + chunk * step_x, true);
    }
    commit_copies();
  };
  auto staged = [&](int chunk, int piece) { return *reinterpret_cast<const float4*>(stage_of(chunk) + (piece * kLanes + tid) * 4); };
  float* s_base = state + (static_cast<int64_t>(seq_slot[seq]) * heads + head) * dk * dv + col0;
  auto in_state = [&](int t, int i) -> float* {  // where s[t][i] comes from and goes to
    const int row = row0 + 2 * t + (i & 1), col = g + 8 * (i >> 1);
    return row < dk && col0 + col < dv ? s_base + static_cast<int64_t>(row) * dv + col : nullptr;
  };
  float s[2][4];  // rows row0 + 2 t, + 1 of column g, the same of column g + 8
  wait_for_predecessor();
  if (chunks == 0) return;
#pragma unroll
  for (int chunk = 0; chunk < kStages - 1; ++chunk) fetch(chunk);
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* at = in_state(t, i);
      s[t][i] = at != nullptr ? *at : 0.f;
    }
  for (int chunk = 0; chunk < chunks; ++chunk) {
    __syncwarp();  // four lanes copy the warp's decays
    fetch(chunk + kStages - 1);
    wait_copies<kStages - 1>();
    float* own_sums = stage_of(chunk) + warp * 128 + lane * 2;  // a warp's sums go where its share of Y was
    {
      SplitA left;
#pragma unroll
      for (int t = 0; t < 2; ++t) left.set(2 * t, split_pair(s[t][0], s[t][1])), left.set(2 * t + 1, split_pair(s[t][2], s[t][3]));
      float acc[4][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) mma_split(acc[t], left, SplitB(staged(chunk, t)));
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) *reinterpret_cast<float2*>(own_sums + t * kLanes * 4 + h * 64) = make_float2(acc[t][2 * h], acc[t][2 * h + 1]);
    }
    // The state in front of the chunk, for `chunk_out`.
    *reinterpret_cast<float4*>(s_out + chunk * step_s) = make_float4(s[0][0], s[0][1], s[1][0], s[1][1]);
    *reinterpret_cast<float4*>(s_out + chunk * step_s + 128) = make_float4(s[0][2], s[0][3], s[1][2], s[1][3]);
    __syncthreads();
    if (adds_up) {
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int pair = warp + o * kParts;
        float2 part[kParts];
#pragma unroll
        for (int w = 0; w < kParts; ++w) part[w] = *reinterpret_cast<const float2*>(stage_of(chunk) + (pair >> 1) * kLanes * 4 + w * 128 + (pair & 1) * 64 + lane * 2);
        const float2 w = *reinterpret_cast<const float2*>(stage_of(chunk) + kPairsAt + (o * kLanes + tid) * 2);
#pragma unroll
        for (int half = kParts / 2; half > 0; half /= 2)
#pragma unroll
          for (int i = 0; i < half; ++i) part[i].x += part[i + half].x, part[i].y += part[i + half].y;
        const float2 u = make_float2(part[0].x + w.x, part[0].y + w.y);
        const Split parts = split_pair(u.x, u.y);
#pragma unroll
        for (int p = 0; p < 3; ++p) reinterpret_cast<uint32_t*>(&us[pair >> 2][p][lane])[pair & 3] = parts.part[p];
        *reinterpret_cast<float2*>(from.x + x_at[o] + chunk * step_x) = u;
      }
    }
    __syncthreads();
    float sum[2][2][4];  // apart from the state, which is rounded once a chunk
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      SplitA left;
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const uint4 word = us[h][p][lane];
        left.part[p][0] = word.x, left.part[p][1] = word.y, left.part[p][2] = word.z, left.part[p][3] = word.w;
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) mma_split(sum[t][h], left, SplitB(staged(chunk, 4 + 2 * t + h)));
    }
    const float4 ef = *reinterpret_cast<const float4*>(stage_of(chunk) + kDecaysAt + row0);
    const float decays[4] = {ef.x, ef.y, ef.z, ef.w};
    float values[2][4] = {};
    if (ADD) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 add = staged(chunk, 8 + h);
        values[h][0] = add.x, values[h][1] = add.y, values[h][2] = add.z, values[h][3] = add.w;
      }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float more = sum[t][0][i] + sum[t][1][i];
        if (ADD) more += values[i >> 1][2 * t + (i & 1)];
        s[t][i] = fmaf(decays[2 * t + (i & 1)], s[t][i], more);
      }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* at = in_state(t, i);
      if (at != nullptr) *at = s[t][i];
    }
}

// --- outputs ---------------------------------------------------------------------------------------------------------------------------
//
// One block per (chunk, head, request and COLS columns), 32 columns a warp: O = Qt S (+ A U) (+ Av V) as one product over rows + 32 (+ 32)
// numbers, 16 at a time, each lane's share of the operands straight from memory one step ahead (by asynchronous copies three steps ahead: 4 us
// slower). Pairs of tokens form a triangle: a token
// leaves out those behind it. What is not finite there times a pair's zero would not be zero, so it goes into the product as a zero, and the
// tokens that it does reach are set to NaN behind it.
template <int COLS, bool WITH_U, bool WITH_V>
__global__ void __launch_bounds__(COLS, 384 / COLS)
chunk_out_kernel(const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int heads, int dv, int rows, int tiles, Scratch from, const float* v,
                 int64_t v_ld, float* out, float* den) {
  let_successor_start();
  const int seq = blockIdx.z / tiles, own_head = blockIdx.y, head = from.head0 + own_head, chunk = blockIdx.x;
  const int start = seq_q_start[seq], n = min(C, seq_q_len[seq] - chunk * C);
  if (n <= 0) return;
  const int64_t first = static_cast<int64_t>(start) + chunk * C, place = chunk_place(start, seq, chunk) * from.heads + own_head;
  const int columns = padded_columns(dv);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int col0 = blockIdx.z % tiles * COLS + warp * 32;  // columns col0 + 8 t + g in B, col0 + 8 t + 2 q, + 1 in D
  const int state_steps = rows / 16;
  constexpr int kPairSteps = (WITH_U ? 2 : 0) + (WITH_V ? 2 : 0);
  wait_for_predecessor();
  if (den != nullptr && blockIdx.z % tiles == 0) {  // the normaliser read out as the state is: n . (e q) + the chunk's own pairs
    constexpr int kWarpTokens = C / (COLS / 32), kMost = kMaxLinearRows / 32;
    float n0[kMost], sum[kWarpTokens];
#pragma unroll
    for (int x = 0; x < kMost; ++x) n0[x] = x * 32 < rows ? from.n[place * rows + x * 32 + lane] : 0.f;
#pragma unroll
    for (int i = 0; i < kWarpTokens; ++i) {  // all tokens' numbers on the way at once: one after the other they took 9 us
      const int r = warp * kWarpTokens + i;
      sum[i] = from.av[(place * C + r) * C + lane];
#pragma unroll
      for (int x = 0; x < kMost; ++x)
        if (x * 32 < rows) sum[i] = fmaf(from.qt[(place * C + r) * rows + x * 32 + lane], n0[x], sum[i]);
    }
#pragma unroll
    for (int i = 0; i < kWarpTokens; ++i) {
      const float whole = warp_sum(sum[i]);
      if (lane == 0 && warp * kWarpTokens + i < n) den[(first + warp * kWarpTokens + i) * heads + head] = whole;
    }
  }
  if (col0 >= columns) return;
  float4 left[4], right[4];
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* qt = from.qt + place * C * rows + g * rows + 4 * q;
  const float* states = from.s + place * columns * rows + s_place(col0, 0, rows) + lane * 4;  // 8 t + g columns on, 16 rows 256 numbers on
  auto fetch_state = [&](int step) {
#pragma unroll
    for (int r = 0; r < 4; ++r) left[r] = *reinterpret_cast<const float4*>(qt + 8 * r * rows + step * 16);
#pragma unroll
    for (int t = 0; t < 4; ++t)
      right[t] = col0 + 8 * t < columns ? *reinterpret_cast<const float4*>(states + t / 2 * 16 * rows + t % 2 * 128 + step * 256) : zero;
  };
  auto fetch_pairs = [&](bool is_u, int half) {  // sixteen of the chunk's tokens
    const float* pairs = (is_u ? from.a : from.av) + place * C * C + half * 16;
#pragma unroll
    for (int r = 0; r < 4; ++r) left[r] = *reinterpret_cast<const float4*>(pairs + (8 * r + g) * C + 4 * q);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int col = col0 + 8 * t + g, token = half * 16 + 4 * q;
      if (is_u) {
        right[t] = col < columns ? *reinterpret_cast<const float4*>(from.x + (place * columns + col) * C + token) : zero;
      } else {
        const float* at = v + (first + token) * v_ld + static_cast<int64_t>(head) * dv + col;
        const bool valid = col < dv;
        right[t] = make_float4(valid && token < n ? at[0] : 0.f, valid && token + 1 < n ? at[v_ld] : 0.f, valid && token + 2 < n ? at[2 * v_ld] : 0.f,
                               valid && token + 3 < n ? at[3 * v_ld] : 0.f);
      }
    }
  };
  float acc[2][4][4];  // tokens 16 m + g (+ 8) of columns 2 q, + 1 of tile t
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[m][t][0] = acc[m][t][1] = acc[m][t][2] = acc[m][t][3] = 0.f;
  auto multiply = [&](int from_m, auto fetch_next) {  // tokens in front of 16 from_m are left out
    const SplitA a[2] = {split_rows(left[0], left[1]), split_rows(left[2], left[3])};
    const SplitB b[4] = {SplitB(right[0]), SplitB(right[1]), SplitB(right[2]), SplitB(right[3])};
    fetch_next();
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      if (m < from_m || 16 * m >= n) continue;
      float sum[4][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) mma_split(sum[t], a[m], b[t]);
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][t][i] += sum[t][i];
    }
  };
  fetch_state(0);
  for (int step = 0; step < state_steps; ++step)
    multiply(0, [&] {
      if (step + 1 < state_steps) fetch_state(step + 1);
      else fetch_pairs(WITH_U, 0);
    });
  int spoilt[4] = {C, C, C, C};  // the first token of a column whose U or V is not finite
  bool any_spoilt = false;
#pragma unroll 1
  for (int pairs = 0; pairs < kPairSteps; ++pairs) {
    const int half = pairs & 1;
    bool found = false;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (all_finite(right[t])) continue;
      float* numbers[4] = {&right[t].x, &right[t].y, &right[t].z, &right[t].w};
#pragma unroll
      for (int i = 3; i >= 0; --i)
        if (!isfinite(*numbers[i])) *numbers[i] = 0.f, spoilt[t] = min(spoilt[t], half * 16 + 4 * q + i), found = true;
    }
    any_spoilt |= __any_sync(0xffffffffu, found);
    multiply(half, [&] {
      if (pairs + 1 < kPairSteps) fetch_pairs(WITH_U && pairs + 1 < 2, (pairs + 1) & 1);
    });
  }
  if (any_spoilt) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      int token = spoilt[t];  // of column g: the least of its four lanes
      token = min(token, __shfl_xor_sync(0xffffffffu, token, 1));
      token = min(token, __shfl_xor_sync(0xffffffffu, token, 2));
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int from_token = __shfl_sync(0xffffffffu, token, (2 * q + c) * 4);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          if (16 * m + g >= from_token) acc[m][t][c] = NAN;
          if (16 * m + g + 8 >= from_token) acc[m][t][2 + c] = NAN;
        }
      }
    }
  }
  const bool wide = dv % 2 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int token = 16 * m + 8 * r + g;
      if (token >= n) continue;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int col = col0 + 8 * t + 2 * q;
        float* to = out + ((first + token) * heads + head) * dv + col;
        if (wide) {
          if (col < dv) *reinterpret_cast<float2*>(to) = make_float2(acc[m][t][2 * r], acc[m][t][2 * r + 1]);
        } else {
          if (col < dv) to[0] = acc[m][t][2 * r];
          if (col + 1 < dv) to[1] = acc[m][t][2 * r + 1];
        }
      }
    }
}

// --- host ------------------------------------------------------------------------------------------------------------------------------

struct Sizes {
  int tokens, seqs, max_q_len, heads, dk, dv;
};

int64_t aligned_floats(int64_t n) { return (n + 3) / 4 * 4; }

// The scratch's arrays for so many heads one after another in `base` (null pointers with a null base); returns the numbers they need.
int64_t lay_out(int rule, const Sizes& z, int heads, float* base, Scratch* to) {
  const int64_t rows = padded_rows(z.dk), columns = padded_columns(z.dv);
  const int64_t chunks = (static_cast<int64_t>(z.tokens) / C + z.seqs + 1) * heads, per_head = chunks * C;
  const int64_t with_u = rule == kDelta || rule == kGeneralDelta ? 1 : 0, with_v = rule != kDelta ? 1 : 0, with_n = rule == kMemory ? 1 : 0;
  const int64_t sizes[9] = {with_u * per_head * rows, with_u * per_head * rows, per_head * rows, with_u * per_head * columns,
                            with_u * per_head * C, with_v * per_head * C, chunks * rows, with_n * chunks * rows, chunks * rows * columns};
  float** arrays[9] = {&to->y, &to->kd, &to->qt, &to->x, &to->a, &to->av, &to->e, &to->n, &to->s};
  to->head0 = 0, to->heads = heads;
  int64_t at = 0;
  for (int i = 0; i < 9; ++i) {
    *arrays[i] = base == nullptr ? nullptr : base + at;
    at += aligned_floats(sizes[i]);
  }
  return at;
}

template <typename Kernel>
bool raise_smem(Kernel kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) == cudaSuccess;
}

template <int ROWS>
bool raise_prepares() {
  const size_t delta = prepare_smem(ROWS);
  bool ok = raise_smem(chunk_prepare_kernel<ROWS, 1, false>, delta) && raise_smem(chunk_prepare_kernel<ROWS, 4, false>, delta) &&
            raise_smem(chunk_prepare_kernel<ROWS, 1, true>, delta) && raise_smem(chunk_prepare_kernel<ROWS, 4, true>, delta) &&
            raise_smem(chunk_walk_kernel<ROWS, false>, walk_smem(ROWS, false));
  if constexpr (ROWS <= kMaxLinearRows) {
    const size_t general = linear_prepare_smem(ROWS, kGeneralDelta), linear = linear_prepare_smem(ROWS, kLinear), memory = linear_prepare_smem(ROWS, kMemory);
    ok = ok && raise_smem(linear_chunk_prepare_kernel<ROWS, 1, kLinear>, linear) && raise_smem(linear_chunk_prepare_kernel<ROWS, 4, kLinear>, linear) &&
         raise_smem(linear_chunk_prepare_kernel<ROWS, 1, kGeneralDelta>, general) && raise_smem(linear_chunk_prepare_kernel<ROWS, 4, kGeneralDelta>, general) &&
         raise_smem(linear_chunk_prepare_kernel<ROWS, 1, kMemory>, memory) && raise_smem(linear_chunk_prepare_kernel<ROWS, 4, kMemory>, memory) &&
         raise_smem(chunk_walk_kernel<ROWS, true>, walk_smem(ROWS, true));
  }
  return ok;
}

bool raise_all() {
  static OncePerDevice raised;
  return raised([] { return raise_prepares<64>() && raise_prepares<128>() && raise_prepares<256>(); });
}

template <int ROWS>
auto delta_prepare_form(bool wide, bool per_head) {
  return per_head ? (wide ? chunk_prepare_kernel<ROWS, 4, true> : chunk_prepare_kernel<ROWS, 1, true>)
                  : (wide ? chunk_prepare_kernel<ROWS, 4, false> : chunk_prepare_kernel<ROWS, 1, false>);
}

template <int ROWS>
auto linear_prepare_form(bool wide, int rule) {
  return rule == kGeneralDelta ? (wide ? linear_chunk_prepare_kernel<ROWS, 4, kGeneralDelta> : linear_chunk_prepare_kernel<ROWS, 1, kGeneralDelta>)
         : rule == kMemory     ? (wide ? linear_chunk_prepare_kernel<ROWS, 4, kMemory> : linear_chunk_prepare_kernel<ROWS, 1, kMemory>)
                               : (wide ? linear_chunk_prepare_kernel<ROWS, 4, kLinear> : linear_chunk_prepare_kernel<ROWS, 1, kLinear>);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Heads know nothing of one another, so a scratch that does not hold all of them takes them in as few equal parts as fit, one after the
// other through the same scratch. Each part costs another walk of the same length with fewer blocks: 2,048 tokens of 28 heads of 128 x 128
// with one decay per head take 273 us in one part, 320 in two, 395 in three, 487 in four (token by token 815), 24 heads of 64 x 64 under the
// generalized rule 145, 205, 271 and 328 (450). Three hold steps of 55,000 tokens of 28 heads; `ops.py` has why they end there.
template <typename Pass>
int part_by_part(const char* name, int rule, const Sizes& z, float* base, int64_t floats, Pass pass) {
  Scratch scratch;
  int heads = z.heads;
  for (int parts = 2; heads > 1 && lay_out(rule, z, heads, nullptr, &scratch) > floats; ++parts) heads = (z.heads + parts - 1) / parts;
  B200_REQUIRE(aligned16(base) && lay_out(rule, z, heads, base, &scratch) <= floats, "%s: scratch too small or not aligned to 16 bytes", name);
  B200_REQUIRE(z.seqs <= 65535 && static_cast<int64_t>(z.seqs) * ((padded_columns(z.dv) + 127) / 128) <= 65535, "%s: too many requests", name);
  B200_REQUIRE(raise_all(), "%s: cannot size shared memory", name);
  for (int head = 0; head < z.heads; head += heads) {
    scratch.head0 = head, scratch.heads = min(heads, z.heads - head);
    if (int status = pass(scratch)) return status;
  }
  return 0;
}

struct Requests {
  const int* q_start;
  const int* q_len;
  const int* slot;
};

int launch_walk(const Sizes& z, const Requests& req, bool add, const Scratch& scratch, float* state, cudaStream_t stream) {
  const int rows = padded_rows(z.dk);
  auto walk = add ? (rows == 64 ? chunk_walk_kernel<64, true> : chunk_walk_kernel<128, true>)
                  : (rows == 64 ? chunk_walk_kernel<64, false> : (rows == 128 ? chunk_walk_kernel<128, false> : chunk_walk_kernel<256, false>));
  // The ordinary way, not early: the few long-lived blocks should spread over all SMs, not over those the kernel in front leaves first.
  launch_kernel_as(true, walk, dim3(padded_columns(z.dv) / kColumns, scratch.heads, z.seqs), dim3(2 * rows), walk_smem(rows, add), stream, req.q_start, req.q_len, req.slot,
                   z.heads, z.dk, z.dv, scratch, state);
  return b200_check_launch("chunk_walk");
}

template <bool WITH_U, bool WITH_V>
int launch_out(const Sizes& z, const Requests& req, const Scratch& scratch, const float* v, int64_t v_ld, float* out, float* den, cudaStream_t stream) {
  const int columns = padded_columns(z.dv), cols = columns <= 64 ? 64 : 128, tiles = (columns + cols - 1) / cols;
  launch_kernel(cols == 64 ? chunk_out_kernel<64, WITH_U, WITH_V> : chunk_out_kernel<128, WITH_U, WITH_V>, dim3((z.max_q_len + C - 1) / C, scratch.heads, z.seqs * tiles),
                dim3(cols), 0, stream, req.q_start, req.q_len, z.heads, z.dv, padded_rows(z.dk), tiles, scratch, v, v_ld, out, den);
  return b200_check_launch("chunk_out");
}

int launch_linear_prepare(const Sizes& z, const Requests& req, int rule, bool wide, const LinearRule& in, const Scratch& scratch, cudaStream_t stream) {
  const int rows = padded_rows(z.dk);
  launch_kernel(rows == 64 ? linear_prepare_form<64>(wide, rule) : linear_prepare_form<128>(wide, rule), dim3((z.max_q_len + C - 1) / C, scratch.heads, z.seqs),
                dim3(kThreads), linear_prepare_smem(rows, rule), stream, in, req.q_start, req.q_len, z.heads, z.dk, z.dv, scratch);
  return b200_check_launch("linear_chunk_prepare");
}

int launch_scan(const Sizes& z, const Requests& req, const Scratch& scratch, float* state, float* normaliser, cudaStream_t stream) {
  const int rows = padded_rows(z.dk), blocks = (rows * padded_columns(z.dv) / 4 + kScanThreads - 1) / kScanThreads;
  launch_kernel(chunk_scan_kernel, dim3(blocks + (normaliser != nullptr ? (rows + kScanThreads - 1) / kScanThreads : 0), scratch.heads, z.seqs), dim3(kScanThreads), 0, stream, req.q_start,
                req.q_len, req.slot, z.heads, z.dk, z.dv, scratch, state, normaliser);
  return b200_check_launch("chunk_scan");
}

}  // namespace

// Sizes the chunked form takes (`rule`: 0 the delta rule, 1 the generalized one, 2 the one without a removal, 3 the matrix memory); the
// caller walks token by token otherwise.
static bool sizes_taken(int rule, int heads, int kv_heads, int dk, int dv) {
  return heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0 && dk > 0 && dk <= (rule == kDelta ? kMaxRows : kMaxLinearRows) && dv > 0 &&
         dv <= 65536;
}

// Numbers of scratch (32-bit, aligned to 16 bytes) that a call needs to take all heads at once; 0: sizes the chunked form does not take. A
// call takes any scratch that holds at least one head.
B200_API int64_t b200_state_chunks_scratch(int rule, int tokens, int seqs, int heads, int kv_heads, int dk, int dv) {
  if (!sizes_taken(rule, heads, kv_heads, dk, dv)) return 0;
  Scratch scratch;
  return lay_out(rule, {tokens, seqs, 0, heads, dk, dv}, heads, nullptr, &scratch);
}

// The delta rule over every request's new tokens; operands as `delta_prepare` leaves them. per_head = 0: `decay` [tokens][heads][dk]
// holds factors; per_head = 1: [tokens][heads] logarithms.
B200_API int b200_delta_chunks(const float* q, const float* k, const float* v, const float* beta, const float* decay, int per_head, const int* seq_q_start,
                               const int* seq_q_len, const int* seq_slot, int tokens, int seqs, int max_q_len, int heads, int kv_heads, int dk, int dv,
                               float* scratch, int64_t scratch_floats, float* state, float* out, cudaStream_t stream) {
  if (seqs == 0 || tokens == 0) return 0;
  B200_REQUIRE(tokens > 0 && seqs > 0 && max_q_len > 0 && sizes_taken(kDelta, heads, kv_heads, dk, dv), "delta_chunks: shape not taken");
  const Sizes z = {tokens, seqs, max_q_len, heads, dk, dv};
  const Requests req = {seq_q_start, seq_q_len, seq_slot};
  const bool wide = dk % 4 == 0 && aligned16(q) && aligned16(k) && (per_head || aligned16(decay));
  const int rows = padded_rows(dk);
  auto prepare = rows == 64 ? delta_prepare_form<64>(wide, per_head) : (rows == 128 ? delta_prepare_form<128>(wide, per_head) : delta_prepare_form<256>(wide, per_head));
  return part_by_part("delta_chunks", kDelta, z, scratch, scratch_floats, [&](const Scratch& parts) -> int {
    launch_kernel(prepare, dim3((max_q_len + C - 1) / C, parts.heads, seqs), dim3(kThreads), prepare_smem(rows), stream, q, k, v, beta, decay, seq_q_start,
                  seq_q_len, heads, kv_heads, dk, dv, parts);
    if (int status = b200_check_launch("chunk_prepare")) return status;
    if (int status = launch_walk(z, req, false, parts, state, stream)) return status;
    return launch_out<true, false>(z, req, parts, v, static_cast<int64_t>(heads) * dv, out, nullptr, stream);
  });
}

// The rules in which the values enter as they are. With `u` the generalized delta rule S <- w S - au (u^T S) + k v^T, o = S^T r; with
// `bonus` [tokens][heads] instead S <- w S + k v^T, o = (S in front of the token)^T r + bonus v. Operands [tokens][heads * dk], v
// [tokens][heads * dv].
B200_API int b200_linear_chunks(const float* r, const float* k, const float* v, const float* w, const float* au, const float* u, const float* bonus,
                                const int* seq_q_start, const int* seq_q_len, const int* seq_slot, int tokens, int seqs, int max_q_len, int heads, int dk, int dv,
                                float* scratch, int64_t scratch_floats, float* state, float* out, cudaStream_t stream) {
  if (seqs == 0 || tokens == 0) return 0;
  const int rule = u != nullptr ? kGeneralDelta : kLinear;
  B200_REQUIRE((u != nullptr) == (au != nullptr) && (u != nullptr) != (bonus != nullptr), "linear_chunks: either u and au or a bonus");
  B200_REQUIRE(tokens > 0 && seqs > 0 && max_q_len > 0 && sizes_taken(rule, heads, heads, dk, dv), "linear_chunks: shape not taken");
  const Sizes z = {tokens, seqs, max_q_len, heads, dk, dv};
  const Requests req = {seq_q_start, seq_q_len, seq_slot};
  const bool wide = dk % 4 == 0 && dv % 4 == 0 && aligned16(r) && aligned16(k) && aligned16(v) && aligned16(w) && aligned16(au) && aligned16(u);
  const LinearRule in{r, k, v, w, au, u, bonus, nullptr, 1.f, static_cast<int64_t>(heads) * dk, static_cast<int64_t>(heads) * dv};
  return part_by_part("linear_chunks", rule, z, scratch, scratch_floats, [&](const Scratch& parts) -> int {
    if (int status = launch_linear_prepare(z, req, rule, wide, in, parts, stream)) return status;
    if (rule == kGeneralDelta) {
      if (int status = launch_walk(z, req, true, parts, state, stream)) return status;
      return launch_out<true, true>(z, req, parts, v, in.v_ld, out, nullptr, stream);
    }
    if (int status = launch_scan(z, req, parts, state, nullptr, stream)) return status;
    return launch_out<false, true>(z, req, parts, v, in.v_ld, out, nullptr, stream);
  });
}

// The matrix memory: S <- keep S + put k v^T, n <- keep n + put k, num = scale S^T q, den = scale n . q after the update. q, k, v: rows ld numbers apart, a
// head's numbers side by side; keep, put, den [tokens][heads]; num [tokens][heads][dv]. Called by b200_mlstm.
extern "C" int b200_memory_chunks(const float* q, const float* k, const float* v, int64_t ld, const float* keep, const float* put, float scale, const int* seq_q_start,
                                  const int* seq_q_len, const int* seq_slot, int tokens, int seqs, int max_q_len, int heads, int dk, int dv, float* scratch,
                                  int64_t scratch_floats, float* S, float* n, float* num, float* den, cudaStream_t stream) {
  B200_REQUIRE(tokens > 0 && seqs > 0 && max_q_len > 0 && sizes_taken(kMemory, heads, heads, dk, dv), "memory_chunks: shape not taken");
  const Sizes z = {tokens, seqs, max_q_len, heads, dk, dv};
  const Requests req = {seq_q_start, seq_q_len, seq_slot};
  const bool wide = dk % 4 == 0 && dv % 4 == 0 && ld % 4 == 0 && aligned16(q) && aligned16(k) && aligned16(v);
  const LinearRule in{q, k, v, keep, nullptr, nullptr, nullptr, put, scale, ld, ld};
  return part_by_part("memory_chunks", kMemory, z, scratch, scratch_floats, [&](const Scratch& parts) -> int {
    if (int status = launch_linear_prepare(z, req, kMemory, wide, in, parts, stream)) return status;
    if (int status = launch_scan(z, req, parts, S, n, stream)) return status;
    return launch_out<false, true>(z, req, parts, v, ld, num, den, stream);
  });
}
