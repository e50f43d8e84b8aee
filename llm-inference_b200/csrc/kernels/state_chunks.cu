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
// Only what the next chunk waits for is in the walk. Everything is 32-bit FMAs (no reduced-precision tensor-core mode): state,
// decays and gates stay what they are token by token, up to the order of sums. Decays enter as products (or sums of their logarithms)
// from token j on, never as quotients of products from the chunk's start, so strong decays in front of a pair cost it no digits.
//
// What bounds it: the walk, a chain of chunks in which a block does 2 x 32 x dk x 16 FMAs per chunk (1,024 cycles of an SM's FMA pipe
// at dk = 128) and takes about twice as many cycles' worth of operands out of shared memory, between two block-wide barriers.
// Measured on a B200 (one request of 2,048 tokens, heads of 128 x 128; all three kernels): a decay per channel, 12 heads: 731 us token
// by token -> 252 us (prepare 60, walk 130, out 60), 28 heads: 941 -> 449; one decay per head (before: outputs and triangular products
// inside the walk): 305 -> 252 and 525 -> 450. 24 heads of 64 x 64: the generalized rule 473 -> 244 us (prepare 100, walk 90, out 35), the
// rule without a removal 564 -> 101 us (prepare 51, scan 16, out 27).
#include <type_traits>

#include "common.cuh"

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
__device__ __forceinline__ void stage_copy(float* smem, const float* gmem, bool valid) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? kBytes : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(kBytes), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit_copies() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void wait_copies() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// Rows `first .. first + n` of src [tokens][ld] from column `at` on, `width` numbers each, to dst [C][dst_ld], a warp per row; rows
// past n and columns from `width` to `padded` become zeros. W numbers a copy.
template <int W>
__device__ __forceinline__ void stage_rows(float* dst, int dst_ld, const float* src, int64_t first, int n, int64_t ld, int64_t at, int width, int padded) {
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < C; r += kWarps) {
    const float* from = src + (r < n ? (first + r) * ld + at : 0);
    for (int c = lane * W; c < padded; c += 32 * W) {
      const bool valid = r < n && c < width;
      stage_copy<4 * W>(dst + r * dst_ld + c, valid ? from + c : src, valid);
    }
  }
}

// Two 32-bit numbers in one register pair, multiplied and added as such (two FMAs an instruction).
using pair_t = unsigned long long;
__device__ __forceinline__ pair_t fma_pair(pair_t a, pair_t b, pair_t c) {
  pair_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ pair_t mul_pair(pair_t a, pair_t b) {
  pair_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float sum_pair(pair_t a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}
struct quad_t {  // four neighbouring numbers
  pair_t lo, hi;
};
__device__ __forceinline__ quad_t load_quad(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}

// What `chunk_prepare` hands on, and the walk's result. Rows of `padded_rows(dk)` and `padded_columns(dv)` numbers, so all copies
// are whole 16-byte steps whatever the sizes.
struct Scratch {
  int head0, heads;  // the heads that a pass takes: all, or as many as the scratch holds
  float* y;   // [tokens][heads][rows]
  float* kd;  // [tokens][heads][rows]: G_last,j k_j
  float* qt;  // [tokens][heads][rows]: e_i q_i
  float* x;   // [tokens][heads][columns]: W, then U
  float* a;   // [tokens][heads][C]: what reads out U
  float* av;  // [tokens][heads][C]: what reads out V
  float* e;   // [chunks][heads][rows]: e_last
  float* n;   // [chunks][heads][rows]: the matrix memory's normaliser, likewise
  float* s;   // [chunks][heads][rows][columns]: what the values alone add, then the state in front of each chunk
};

// Solves (I + l) x = rhs in place, row after row: x_i = rhs_i - sum_{j < i} l[i][j] x_j.
__device__ __forceinline__ void substitute(const float* l, float (&x)[C]) {
#pragma unroll
  for (int i = 1; i < C; ++i) {
    float sum0 = x[i], sum1 = 0.f;
#pragma unroll
    for (int j = 0; j < i; j += 4) {
      const float4 row = *reinterpret_cast<const float4*>(l + i * C + j);
      sum0 = fmaf(-row.x, x[j], sum0);
      if (j + 1 < i) sum1 = fmaf(-row.y, x[j + 1], sum1);
      if (j + 2 < i) sum0 = fmaf(-row.z, x[j + 2], sum0);
      if (j + 3 < i) sum1 = fmaf(-row.w, x[j + 3], sum1);
    }
    x[i] = sum0 + sum1;
  }
}

// --- what does not depend on the state -------------------------------------------------------------------------------------------
//
// One block per (chunk, head, request). Pairs of tokens: the chunk's rows form four groups of eight. Inside a group a lane has a token
// j and carries p = G_ij k_j from row to row. Between groups every decay product splits at the group's border, G_ij = (product up
// to i inside i's group) (whole groups between) (product from j + 1 to the end of j's group), three factors without a quotient, so
// those pairs are plain products of scaled rows. A warp has an eighth of the channels; the warps' sums meet in shared memory.
// PER_HEAD: one decay per head, given as its logarithm; pairs are products of the raw rows and G_ij = exp of the sum of logarithms.
// Columns: a thread per column of [e K | V] solves the triangular system by substitution.
constexpr int kGroup = 8, kGroups = C / kGroup;
constexpr int kBetween = 6;  // pairs of groups
__host__ __device__ constexpr int inside_sums(int lefts) { return kGroup * lefts * 32; }  // numbers that a warp hands on
__host__ __device__ constexpr int between_sums(int lefts) { return kBetween * 2 * lefts * 32; }

// left_i . G_ij right_j for i, j in one group, over the warp's eighth of the channels: lane j, rows i = 8 (j / 8) + r. BEFORE: the first left
// row meets the decays of tokens j + 1 .. i - 1 only. Without DECAYS: left_i . right_j.
template <int ROWS, int LEFTS, bool DECAYS, bool BEFORE>
__device__ __forceinline__ void pairs_inside(const float* left0, const float* left1, const float* right, const float* decays, float* sums) {
  constexpr int ld = ROWS + 4, slice = ROWS / kWarps;
  const int c0 = threadIdx.x / 32 * slice;
  const int lane = threadIdx.x & 31, own = lane & 7, group = (lane & ~7) * ld;
  pair_t acc[kGroup][LEFTS];
#pragma unroll
  for (int r = 0; r < kGroup; ++r)
#pragma unroll
    for (int x = 0; x < LEFTS; ++x) acc[r][x] = 0;
#pragma unroll 2
  for (int c = c0; c < c0 + slice; c += 4) {
    const quad_t mine = load_quad(right + lane * ld + c);
    quad_t p = mine;
    if (DECAYS) p = {0, 0};
#pragma unroll
    for (int r = 0; r < kGroup; ++r) {
      const int at = group + r * ld + c;
      const quad_t a = load_quad(left0 + at);
      if (BEFORE) acc[r][0] = fma_pair(a.hi, p.hi, fma_pair(a.lo, p.lo, acc[r][0]));
      if (DECAYS) {
        const quad_t g = load_quad(decays + at);
        p.lo = r == own ? mine.lo : mul_pair(p.lo, g.lo);
        p.hi = r == own ? mine.hi : mul_pair(p.hi, g.hi);
      }
      if (!BEFORE) acc[r][0] = fma_pair(a.hi, p.hi, fma_pair(a.lo, p.lo, acc[r][0]));
      if (LEFTS == 2) {
        const quad_t b = load_quad(left1 + at);
        acc[r][LEFTS - 1] = fma_pair(b.hi, p.hi, fma_pair(b.lo, p.lo, acc[r][LEFTS - 1]));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kGroup; ++r)
#pragma unroll
    for (int x = 0; x < LEFTS; ++x) sums[(r * LEFTS + x) * 32 + lane] = sum_pair(acc[r][x]);
}

// The same for j in a group b before i's group g, from rows that carry their decays inside their own groups: lane = token 8 b + lane % 8,
// rows 8 g + 2 (lane / 8) and the next one; `whole` holds the groups' decays multiplied.
template <int ROWS, int LEFTS, bool DECAYS>
__device__ __forceinline__ void pairs_between(const float* left0, const float* left1, const float* ends, const float* whole, float* sums) {
  constexpr int rows = ROWS, ld = ROWS + 4, slice = ROWS / kWarps;
  const int c0 = threadIdx.x / 32 * slice;
  const int lane = threadIdx.x & 31, at0 = (lane >> 3) * 2 * ld;
  const float* right = ends + (lane & 7) * ld;
  pair_t acc[kBetween][2][LEFTS];
#pragma unroll
  for (int x = 0; x < kBetween; ++x)
#pragma unroll
    for (int y = 0; y < LEFTS; ++y) acc[x][0][y] = acc[x][1][y] = 0;
  for (int c = c0; c < c0 + slice; c += 4) {
    quad_t p[kGroups - 1];
#pragma unroll
    for (int b = 0; b < kGroups - 1; ++b) p[b] = load_quad(right + b * kGroup * ld + c);
    int x = 0;
#pragma unroll
    for (int g = 1; g < kGroups; ++g) {
      if (DECAYS && g > 1) {  // the groups that are now whole ones between
        const quad_t between = load_quad(whole + (g - 1) * rows + c);
#pragma unroll
        for (int b = 0; b < g - 1; ++b) p[b].lo = mul_pair(p[b].lo, between.lo), p[b].hi = mul_pair(p[b].hi, between.hi);
      }
      quad_t left[2][LEFTS];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int at = at0 + (g * kGroup + r) * ld + c;
        left[r][0] = load_quad(left0 + at);
        if (LEFTS == 2) left[r][LEFTS - 1] = load_quad(left1 + at);
      }
#pragma unroll
      for (int b = 0; b < g; ++b, ++x)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int y = 0; y < LEFTS; ++y) acc[x][r][y] = fma_pair(left[r][y].hi, p[b].hi, fma_pair(left[r][y].lo, p[b].lo, acc[x][r][y]));
    }
  }
#pragma unroll
  for (int x = 0; x < kBetween; ++x)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int y = 0; y < LEFTS; ++y) sums[((x * 2 + r) * LEFTS + y) * 32 + lane] = sum_pair(acc[x][r][y]);
}

// The warps' sums of either kind, `stride` numbers from warp to warp, added up into the [C][C + 1] matrices of the left rows.
template <int LEFTS, bool INSIDE>
__device__ __forceinline__ void add_up(const float* sums, int stride, float* to0, float* to1) {
  for (int idx = threadIdx.x; idx < (INSIDE ? inside_sums(LEFTS) : between_sums(LEFTS)); idx += kThreads) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += sums[w * stride + idx];
    const int l = idx % 32, y = idx / 32 % LEFTS, o = idx / 32 / LEFTS;
    int i, j;
    if (INSIDE) {
      i = (l & ~7) + o, j = l;
    } else {
      const int x = o / 2, g = x == 0 ? 1 : (x < 3 ? 2 : 3), b = x - (g == 1 ? 0 : (g == 2 ? 1 : 3));
      i = g * kGroup + (l >> 3) * 2 + (o & 1), j = b * kGroup + (l & 7);
    }
    (y == 0 ? to0 : to1)[i * (C + 1) + j] = sum;
  }
}

constexpr int kWarpSums = inside_sums(2) + between_sums(2);
size_t prepare_smem(int rows) {
  return sizeof(float) * (3 * C * (rows + 4) + kGroups * rows + kWarps * kWarpSums + 2 * C * (C + 1) + C * C + 3 * C);
}

template <int ROWS, int W, bool PER_HEAD>
__global__ void __launch_bounds__(kThreads, 2)
chunk_prepare_kernel(const float* q, const float* k, const float* v, const float* beta, const float* decay, const int* __restrict__ seq_q_start,
                     const int* __restrict__ seq_q_len, int heads, int kv_heads, int dk, int dv, Scratch to) {
  extern __shared__ __align__(16) float chunk_smem[];
  let_successor_start();
  const int seq = blockIdx.z, own_head = blockIdx.y, head = to.head0 + own_head, chunk = blockIdx.x;
  const int n = min(C, seq_q_len[seq] - chunk * C);
  if (n <= 0) return;
  const int start = seq_q_start[seq], kvh = head / (heads / kv_heads);
  const int64_t first = static_cast<int64_t>(start) + chunk * C;
  constexpr int rows = ROWS, ld = ROWS + 4;
  const int columns = padded_columns(dv);
  float* ks = chunk_smem;                     // [C][ld]: keys, then times the decays of their group up to their own token
  float* qs = ks + C * ld;                    // [C][ld]: queries, then likewise
  float* gs = qs + C * ld;                    // [C][ld]: decays, then keys times the decays from the next token to their group's end
  float* whole = gs + C * ld;                 // [groups][rows]: each group's decays multiplied
  float* ls = whole + kGroups * rows;         // [C][C]
  float* sums = ls + C * C;                   // [warps][kWarpSums]
  float* kk = sums + kWarps * kWarpSums;      // [C][C + 1]: k_i . G_ij k_j
  float* qk = kk + C * (C + 1);               // [C][C + 1]: q_i . G_ij k_j
  float* bs = qk + C * (C + 1);               // [C]: beta
  float* es = bs + C;                         // [C]: PER_HEAD: e_i
  float* fs = es + C;                         // [C]: PER_HEAD: G_last,j
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  wait_for_predecessor();
  stage_rows<W>(ks, ld, k, first, n, static_cast<int64_t>(kv_heads) * dk, static_cast<int64_t>(kvh) * dk, dk, rows);
  stage_rows<W>(qs, ld, q, first, n, static_cast<int64_t>(kv_heads) * dk, static_cast<int64_t>(kvh) * dk, dk, rows);
  if (!PER_HEAD) stage_rows<W>(gs, ld, decay, first, n, static_cast<int64_t>(heads) * dk, static_cast<int64_t>(head) * dk, dk, rows);
  if (tid < C) bs[tid] = tid < n ? beta[(first + tid) * heads + head] : 0.f;
  commit_copies();
  wait_copies<0>();
  __syncthreads();
  float* mine = sums + warp * kWarpSums;
  pairs_inside<ROWS, 2, !PER_HEAD, false>(ks, qs, ks, gs, mine);
  if (!PER_HEAD) {
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
  }
  pairs_between<ROWS, 2, !PER_HEAD>(ks, qs, PER_HEAD ? ks : gs, whole, mine + inside_sums(2));
  __syncthreads();
  add_up<2, true>(sums, kWarpSums, kk, qk);
  add_up<2, false>(sums + inside_sums(2), kWarpSums, kk, qk);
  __syncthreads();
  {
    float own = 0.f, d = 0.f, prefix = 0.f, e = 0.f;
    if (PER_HEAD) own = lane < n ? decay[(first + lane) * heads + head] : 0.f;
    float* a = to.a + (first * to.heads + own_head) * C + lane;
    for (int i = 0; i < C; ++i) {
      if (PER_HEAD) {  // D_ij of column j = lane, the sum of the logarithms from token j + 1 on, grows with i from zero at i = j
        const float gi = __shfl_sync(0xffffffffu, own, i);
        d = i > lane ? d + gi : 0.f;
        prefix += gi;
        if (i == lane) e = prefix;
      }
      if ((i & 7) == warp) {
        const float between = PER_HEAD ? expf(d) : 1.f;
        ls[i * C + lane] = lane < i ? bs[i] * between * kk[i * (C + 1) + lane] : 0.f;
        if (i < n) a[static_cast<int64_t>(i) * to.heads * C] = lane <= i ? between * qk[i * (C + 1) + lane] : 0.f;
      }
    }
    if (PER_HEAD && warp == 0) es[lane] = expf(e), fs[lane] = expf(d);  // d is now D_last,j: tokens past n added nothing
  }
  __syncthreads();
  for (int column = tid; column < rows + columns; column += kThreads) {
    float x[C];
    float* to_x;
    const int64_t stride = static_cast<int64_t>(to.heads) * (column < rows ? rows : columns);
    if (column < rows) {
      const int64_t at = (first * to.heads + own_head) * rows + column;
      float* qt = to.qt + at;
      float* kd = to.kd + at;
      to_x = to.y + at;
      float before[kGroups], after[kGroups];  // whole groups in front of and behind a token's own
      if (!PER_HEAD) {
        before[0] = after[kGroups - 1] = 1.f;
#pragma unroll
        for (int g = 1; g < kGroups; ++g) before[g] = before[g - 1] * whole[(g - 1) * rows + column];
#pragma unroll
        for (int g = kGroups - 2; g >= 0; --g) after[g] = after[g + 1] * whole[(g + 1) * rows + column];
      }
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const float key = ks[i * ld + column], e = PER_HEAD ? es[i] : before[i / kGroup];
        if (i < n) {
          *qt = e * qs[i * ld + column];
          *kd = PER_HEAD ? fs[i] * key : after[i / kGroup] * gs[i * ld + column];
        }
        qt += stride, kd += stride;
        x[i] = -bs[i] * e * key;
      }
      to.e[(chunk_place(start, seq, chunk) * to.heads + own_head) * rows + column] =
          PER_HEAD ? es[n - 1] : before[kGroups - 1] * whole[(kGroups - 1) * rows + column];
    } else {
      const int c = column - rows;
      const float* value = v + (first * heads + head) * dv + c;
      to_x = to.x + (first * to.heads + own_head) * columns + c;
#pragma unroll
      for (int i = 0; i < C; ++i) x[i] = i < n && c < dv ? value[static_cast<int64_t>(i) * heads * dv] : 0.f;
#pragma unroll
      for (int i = 0; i < C; ++i) x[i] *= bs[i];
    }
    substitute(ls, x);
#pragma unroll
    for (int i = 0; i < C; ++i) {
      if (i < n) *to_x = x[i];
      to_x += stride;
    }
  }
}

// --- the same for rules in which the values enter as they are ---------------------------------------------------------------------------
//
// GENERAL: S <- w S + b (u^T S) + k v^T, o = S^T r, with b = -au. kLinear: S <- w S + k v^T, o = S^T r + bonus v read before the update.
// MEMORY: S <- keep S + put k v^T and n <- keep n + put k with two numbers per head and token, o = S^T r and n . r after the update, r
// times `scale`: pairs are products of the raw rows, times the keeps between them.
// One block per (chunk, head, request); the sums of the values (G_last K)^T V go where the chunk's state will be.
constexpr int kValueTile = 64;
constexpr int kLdV = kValueTile + 4;
constexpr int kMaxLinearRows = 128;

__host__ __device__ constexpr int linear_warp_sums(bool general) { return general ? 2 * inside_sums(2) : between_sums(1); }
size_t linear_prepare_smem(int rows, int rule) {
  const bool general = rule == kGeneralDelta;
  return sizeof(float) * ((general ? 5 : (rule == kMemory ? 2 : 3)) * C * (rows + 4) + 3 * C + C * kLdV + kGroups * rows + kWarps * linear_warp_sums(general) + (general ? 4 : 1) * C * (C + 1) +
                          (general ? 2 : 0) * C * C);
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
__global__ void __launch_bounds__(kThreads, 2)
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
  constexpr int kSums = linear_warp_sums(GENERAL);
  float* ls = chunk_smem;                                // GENERAL: [C][C]: -N
  float* ms = ls + (GENERAL ? C * C : 0);                // GENERAL: [C][C]: M
  float* rs = ms + (GENERAL ? C * C : 0);                // [C][ld]: r, then times the decays of its group in front of (GENERAL: up to) its token
  float* ks = rs + C * ld;                               // [C][ld]: k, then times the decays from the next token to its group's end
  float* gs = ks + C * ld;                               // [C][ld]
  float* us = gs + (MEMORY ? 0 : C * ld);                // GENERAL: [C][ld]: u, then times the decays of its group in front of its token
  float* bb = us + (GENERAL ? C * ld : 0);               // GENERAL: [C][ld]: -au, then as k
  float* vs = bb + (GENERAL ? C * ld : 0);               // [C][kLdV]: a tile of the values
  float* whole = vs + C * kLdV;                          // [groups][rows]
  float* sums = whole + kGroups * rows;                  // [warps][kSums]
  float* rk = sums + kWarps * kSums;                     // [C][C + 1]: r_i . G k_j
  float* uk = rk + C * (C + 1);
  float* rb = uk + C * (C + 1);
  float* ub = rb + C * (C + 1);
  float* es = MEMORY ? uk : ub + (GENERAL ? C * (C + 1) : 0);  // MEMORY: [C]: the keeps up to a token, multiplied
  float* fs = es + C;                                           // MEMORY: [C]: the keeps behind a token times its put
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t ld_in = in.ld, at_in = static_cast<int64_t>(head) * dk;
  auto stage_values = [&](int col0) {
    for (int r = warp; r < C; r += kWarps)
      for (int c = lane * W; c < kValueTile; c += 32 * W) {
        const bool valid = r < n && col0 + c < dv;
        stage_copy<4 * W>(vs + r * kLdV + c, valid ? in.v + (first + r) * in.v_ld + static_cast<int64_t>(head) * dv + col0 + c : in.v, valid);
      }
  };
  wait_for_predecessor();
  stage_rows<W>(rs, ld, in.r, first, n, ld_in, at_in, dk, rows);
  stage_rows<W>(ks, ld, in.k, first, n, ld_in, at_in, dk, rows);
  if (!MEMORY) stage_rows<W>(gs, ld, in.w, first, n, ld_in, at_in, dk, rows);
  if (GENERAL) {
    stage_rows<W>(us, ld, in.u, first, n, ld_in, at_in, dk, rows);
    stage_rows<W>(bb, ld, in.au, first, n, ld_in, at_in, dk, rows);
  }
  stage_values(0);
  commit_copies();
  wait_copies<0>();
  __syncthreads();
  float* mine = sums + warp * kSums;
  if (GENERAL) {
    pairs_inside<ROWS, 2, true, true>(us, rs, ks, gs, mine);
    pairs_inside<ROWS, 2, true, true>(us, rs, bb, gs, mine + inside_sums(2));
  } else {
    pairs_inside<ROWS, 1, !MEMORY, !MEMORY>(rs, nullptr, ks, gs, mine);
  }
  __syncthreads();
  if (GENERAL) {
    add_up<2, true>(sums, kSums, uk, rk);
    add_up<2, true>(sums + inside_sums(2), kSums, ub, rb);
  } else {
    add_up<1, true>(sums, kSums, rk, nullptr);
  }
  for (int item = tid; !MEMORY && item < kGroups * rows; item += kThreads) {  // a thread per (group, channel)
    const int c = item % rows, at = item / rows * kGroup * ld + c;
    float g[kGroup];
    float run = 1.f;
#pragma unroll
    for (int r = 0; r < kGroup; ++r) {
      g[r] = item / rows * kGroup + r < n ? gs[at + r * ld] : 1.f;
      if (GENERAL) us[at + r * ld] *= run;
      else rs[at + r * ld] *= run;
      run *= g[r];
      if (GENERAL) rs[at + r * ld] *= run;
    }
    whole[item] = run;
    run = 1.f;
#pragma unroll
    for (int r = kGroup - 1; r >= 0; --r) {
      ks[at + r * ld] *= run;
      if (GENERAL) bb[at + r * ld] *= run;
      run *= g[r];
    }
  }
  __syncthreads();
  if (GENERAL) {
    pairs_between<ROWS, 2, true>(us, rs, ks, whole, mine);
    __syncthreads();
    add_up<2, false>(sums, kSums, uk, rk);
    __syncthreads();
    pairs_between<ROWS, 2, true>(us, rs, bb, whole, mine);
    __syncthreads();
    add_up<2, false>(sums, kSums, ub, rb);
  } else {
    pairs_between<ROWS, 1, !MEMORY>(rs, nullptr, ks, whole, mine);
    __syncthreads();
    add_up<1, false>(sums, kSums, rk, nullptr);
  }
  __syncthreads();
  if constexpr (MEMORY) {
    // Column j = lane: the keeps of tokens j + 1 .. i multiplied, from one at i = j on.
    const int64_t at = (first + lane) * heads + head;
    const float keep = lane < n ? in.w[at] : 1.f, put = lane < n ? in.put[at] : 0.f;
    float d = 1.f, prefix = 1.f, e = 1.f;
    for (int i = 0; i < C; ++i) {
      const float own = __shfl_sync(0xffffffffu, keep, i);
      d = i > lane ? d * own : 1.f;
      prefix *= own;
      if (i == lane) e = prefix;
      if ((i & 7) == warp && i < n) to.av[((first + i) * to.heads + own_head) * C + lane] = lane <= i ? d * put * rk[i * (C + 1) + lane] * in.scale : 0.f;
    }
    if (warp == 0) es[lane] = e, fs[lane] = d * put;
    __syncthreads();
    for (int c = tid; c < rows; c += kThreads) {
      float* qt = to.qt + (first * to.heads + own_head) * rows + c;
      float sum = 0.f;
#pragma unroll 8
      for (int i = 0; i < C; ++i) {
        const float key = fs[i] * ks[i * ld + c];
        ks[i * ld + c] = key;
        sum += key;
        if (i < n) *qt = es[i] * in.scale * rs[i * ld + c];
        qt += static_cast<int64_t>(to.heads) * rows;
      }
      to.n[place * rows + c] = sum;
      to.e[place * rows + c] = es[n - 1];
#pragma unroll
      for (int g = 0; g < kGroups; ++g) whole[g * rows + c] = 1.f;
    }
    __syncthreads();
  }
  for (int i = warp; !MEMORY && i < C; i += kWarps) {
    const int at = i * (C + 1) + lane;
    const int64_t row = ((first + i) * to.heads + own_head) * C + lane;
    if (GENERAL) {  // au came in with its own sign: b = -au
      ls[i * C + lane] = lane < i ? ub[at] : 0.f;
      ms[i * C + lane] = lane < i ? uk[at] : 0.f;
      if (i < n) {
        to.a[row] = lane <= i ? -rb[at] : 0.f;
        to.av[row] = lane <= i ? rk[at] : 0.f;
      }
    } else if (i < n) {
      to.av[row] = lane < i ? rk[at] : (lane == i ? in.bonus[(first + i) * heads + head] : 0.f);
    }
  }
  // Scaled rows: r times all decays in front of (or up to) its token, b times all decays behind its token; a thread per (group, channel).
  for (int item = tid; !MEMORY && item < kGroups * rows; item += kThreads) {
    const int c = item % rows, group = item / rows;
    float before = 1.f, after = 1.f;
#pragma unroll
    for (int g = 0; g < kGroups - 1; ++g) {
      before *= g < group ? whole[g * rows + c] : 1.f;
      after *= g + 1 > group ? whole[(g + 1) * rows + c] : 1.f;
    }
    const int64_t at = ((first + group * kGroup) * to.heads + own_head) * rows + c, step = static_cast<int64_t>(to.heads) * rows;
    float* qt = to.qt + at;
    float* kd = to.kd + at;
#pragma unroll
    for (int r = 0; r < kGroup; ++r) {
      const int from = (group * kGroup + r) * ld + c;
      if (group * kGroup + r < n) {
        *qt = before * rs[from];
        if (GENERAL) *kd = -after * bb[from];
      }
      qt += step, kd += step;
    }
  }
  for (int c = tid; !MEMORY && c < rows; c += kThreads) to.e[place * rows + c] = whole[c] * whole[rows + c] * whole[2 * rows + c] * whole[3 * rows + c];
  if (GENERAL) __syncthreads();
  for (int col0 = 0; col0 < columns; col0 += kValueTile) {
    if (col0 > 0) {
      __syncthreads();
      stage_values(col0);
      commit_copies();
      wait_copies<0>();
      __syncthreads();
    }
    if (GENERAL && tid < kValueTile + (col0 == 0 ? rows : 0)) {  // a thread per column of [M V | e U]
      float x[C];
      float* to_x;
      int64_t stride;
      const int c = tid;
      if (tid < kValueTile) {
        float value[C];
#pragma unroll
        for (int i = 0; i < C; ++i) value[i] = vs[i * kLdV + c];
#pragma unroll
        for (int i = 0; i < C; ++i) {
          float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
          for (int j = 0; j < i; j += 4) {
            const float4 row = *reinterpret_cast<const float4*>(ms + i * C + j);
            sum0 = fmaf(row.x, value[j], sum0);
            if (j + 1 < i) sum1 = fmaf(row.y, value[j + 1], sum1);
            if (j + 2 < i) sum0 = fmaf(row.z, value[j + 2], sum0);
            if (j + 3 < i) sum1 = fmaf(row.w, value[j + 3], sum1);
          }
          x[i] = sum0 + sum1;
        }
        stride = static_cast<int64_t>(to.heads) * columns;
        to_x = to.x + (first * to.heads + own_head) * columns + col0 + c;
      } else {
        const int channel = c - kValueTile;
        float before = 1.f;
#pragma unroll
        for (int i = 0; i < C; ++i) {
          if (i > 0 && i % kGroup == 0) before *= whole[(i / kGroup - 1) * rows + channel];
          x[i] = before * us[i * ld + channel];
        }
        stride = static_cast<int64_t>(to.heads) * rows;
        to_x = to.y + (first * to.heads + own_head) * rows + channel;
      }
      substitute(ls, x);
      if (tid >= kValueTile || col0 + c < columns) {
#pragma unroll
        for (int i = 0; i < C; ++i) {
          if (i < n) *to_x = x[i];
          to_x += stride;
        }
      }
    }
    // (G_last K)^T V over the tile: four rows by four columns a thread, group after group of tokens.
    const int rt = (tid & 15) * 4, ct = (tid >> 4) * 4;
    for (int row = rt; row < rows; row += 64) {
      float acc[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const float4 scale = *reinterpret_cast<const float4*>(whole + g * rows + row);
        const float f[4] = {scale.x, scale.y, scale.z, scale.w};
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] *= f[r], acc[r][1] *= f[r], acc[r][2] *= f[r], acc[r][3] *= f[r];
#pragma unroll
        for (int j = g * kGroup; j < (g + 1) * kGroup; ++j) {
          const float4 key = *reinterpret_cast<const float4*>(ks + j * ld + row), value = *reinterpret_cast<const float4*>(vs + j * kLdV + ct);
          const float a[4] = {key.x, key.y, key.z, key.w};
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            acc[r][0] = fmaf(a[r], value.x, acc[r][0]), acc[r][1] = fmaf(a[r], value.y, acc[r][1]);
            acc[r][2] = fmaf(a[r], value.z, acc[r][2]), acc[r][3] = fmaf(a[r], value.w, acc[r][3]);
          }
        }
      }
      if (col0 + ct < columns) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          *reinterpret_cast<float4*>(to.s + (place * rows + row + r) * columns + col0 + ct) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      }
    }
  }
}

// Four neighbouring numbers of a head's state a thread, from chunk to chunk: eight chunks' sums are asked for at a time.
__global__ void __launch_bounds__(kThreads)
chunk_scan_kernel(const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, const int* __restrict__ seq_slot, int heads, int dk, int dv, Scratch from,
                  float* state, float* normaliser) {
  let_successor_start();
  const int seq = blockIdx.z, own_head = blockIdx.y, head = from.head0 + own_head;
  const int start = seq_q_start[seq], len = seq_q_len[seq], chunks = (len + C - 1) / C;
  const int rows = padded_rows(dk), columns = padded_columns(dv);
  const int item = (blockIdx.x * kThreads + threadIdx.x) * 4;
  if (item >= rows * columns) {  // the blocks behind the state's: a number of the normaliser a thread
    const int c = blockIdx.x * kThreads + threadIdx.x - (rows * columns / 4 + kThreads - 1) / kThreads * kThreads;
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
  const int row = item / columns, col = item % columns;
  float* base = state + (static_cast<int64_t>(seq_slot[seq]) * heads + head) * dk * dv + static_cast<int64_t>(row) * dv + col;
  float s[4];
  wait_for_predecessor();
#pragma unroll
  for (int x = 0; x < 4; ++x) s[x] = row < dk && col + x < dv ? base[x] : 0.f;
  const int64_t place = chunk_place(start, seq, 0) * from.heads + own_head;
  const float* e = from.e + place * rows + row;
  float* sums = from.s + place * rows * columns + item;
  const int64_t step_e = static_cast<int64_t>(from.heads) * rows, step = step_e * columns;
  constexpr int kAhead = 8;
  for (int chunk = 0; chunk < chunks; chunk += kAhead) {
    float4 add[kAhead];
    float keep[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (chunk + i < chunks) add[i] = *reinterpret_cast<const float4*>(sums + (chunk + i) * step), keep[i] = e[(chunk + i) * step_e];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (chunk + i < chunks) {
        *reinterpret_cast<float4*>(sums + (chunk + i) * step) = make_float4(s[0], s[1], s[2], s[3]);
        s[0] = fmaf(keep[i], s[0], add[i].x), s[1] = fmaf(keep[i], s[1], add[i].y);
        s[2] = fmaf(keep[i], s[2], add[i].z), s[3] = fmaf(keep[i], s[3], add[i].w);
      }
  }
  if (chunks > 0) {
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (row < dk && col + x < dv) base[x] = s[x];
  }
}

// --- the walk ------------------------------------------------------------------------------------------------------------------------
//
// One block per (16 columns of the state, head, request). U = W + Y S: a warp has four tokens, its lanes four groups of columns times
// eight parts of the rows, whose sums meet by shuffles. S <- e S + Kd^T U: a warp has an eighth of the rows, a lane four rows by four
// columns over every kSplit-th token; after the shuffles it keeps its kPer rows of S in registers, with a transposed copy in shared
// memory for the next chunk's first product.
__host__ __device__ constexpr int walk_stage(int rows) { return 2 * C * (rows + 4) + C * kColumns + rows; }
__host__ __device__ constexpr int walk_tile(int rows) { return kColumns * (rows + 8); }
constexpr int kMaxRowX = 24;
constexpr size_t walk_smem(int rows) { return sizeof(float) * (2 * walk_stage(rows) + walk_tile(rows) + C * kMaxRowX); }

__device__ __forceinline__ float from_pair(float give, float keep, int with) { return keep + __shfl_xor_sync(0xffffffffu, give, with); }

template <int ROWS, bool ADD>  // ADD: what the values alone add to S stands where the chunk's state goes
__global__ void __launch_bounds__(kThreads, ROWS <= 128 ? 2 : 1)
chunk_walk_kernel(const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, const int* __restrict__ seq_slot, int heads, int dk, int dv,
                  Scratch from, float* state) {
  extern __shared__ __align__(16) float chunk_smem[];
  constexpr int kSplit = kThreads / ROWS;         // lanes that share a tile of S: 4, 2 or 1
  constexpr int kPer = 4 / kSplit;                // rows of S that a lane keeps
  constexpr int kLd = ROWS + 4;
  constexpr int kLdS = ROWS + 8;                  // 8 banks from column to column
  constexpr int kRowX = kSplit == 4 ? 24 : 16;    // the rows that lanes read side by side in different banks
  let_successor_start();
  const int col0 = blockIdx.x * kColumns, own_head = blockIdx.y, head = from.head0 + own_head, seq = blockIdx.z;
  const int start = seq_q_start[seq], len = seq_q_len[seq];
  const int columns = padded_columns(dv);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* tile = chunk_smem + 2 * walk_stage(ROWS);  // [16 columns][kLdS]: S, transposed
  float* xs = tile + walk_tile(ROWS);               // [C][kRowX]: U
  const int chunks = (len + C - 1) / C;
  auto fetch = [&](int chunk) {
    float* ys = chunk_smem + (chunk & 1) * walk_stage(ROWS);
    float* kds = ys + C * kLd;
    float* ws = kds + C * kLd;
    float* es = ws + C * kColumns;
    const int n = min(C, len - chunk * C);
    const int64_t first = static_cast<int64_t>(start) + chunk * C;
#pragma unroll
    for (int idx = tid; idx < C * ROWS / 4; idx += kThreads) {
      const int r = idx / (ROWS / 4), c = idx % (ROWS / 4) * 4;
      const int64_t at = r < n ? ((first + r) * from.heads + own_head) * ROWS + c : 0;
      stage_copy<16>(ys + r * kLd + c, from.y + at, r < n);
      stage_copy<16>(kds + r * kLd + c, from.kd + at, r < n);
    }
    if (tid < C * kColumns / 4) {
      const int r = tid / 4, c = tid % 4 * 4;
      stage_copy<16>(ws + r * kColumns + c, from.x + (r < n ? ((first + r) * from.heads + own_head) * columns + col0 + c : 0), r < n);
    } else if (tid < C * kColumns / 4 + ROWS / 4) {
      const int c = (tid - C * kColumns / 4) * 4;
      stage_copy<16>(es + c, from.e + (chunk_place(start, seq, chunk) * from.heads + own_head) * ROWS + c, true);
    }
    commit_copies();
  };
  const int jp = lane % kSplit, cg = lane / kSplit % 4;
  const int quad = warp * (ROWS / kWarps) + lane / (4 * kSplit) * 4;  // the lane's tile: rows quad .. + 3, columns 4 cg .. + 3
  const int row0 = quad + jp * kPer;                                  // the rows it keeps
  float* s_base = state + (static_cast<int64_t>(seq_slot[seq]) * heads + head) * dk * dv + col0;
  float s[kPer][4];
  wait_for_predecessor();
  if (chunks > 0) fetch(0);
#pragma unroll
  for (int r = 0; r < kPer; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      s[r][c] = row0 + r < dk && col0 + cg * 4 + c < dv ? s_base[static_cast<int64_t>(row0 + r) * dv + cg * 4 + c] : 0.f;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int n = min(C, len - chunk * C);
    const int64_t first = static_cast<int64_t>(start) + chunk * C;
    float* s_out = from.s + ((chunk_place(start, seq, chunk) * from.heads + own_head) * ROWS + row0) * columns + col0 + cg * 4;
    float4 own[kPer];
    if (ADD) {
#pragma unroll
      for (int r = 0; r < kPer; ++r) own[r] = *reinterpret_cast<const float4*>(s_out + static_cast<int64_t>(r) * columns);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float* to = tile + (cg * 4 + c) * kLdS + row0;
      if (kPer == 4) *reinterpret_cast<float4*>(to) = make_float4(s[0][c], s[kPer / 4][c], s[kPer / 2][c], s[kPer - 1][c]);
      else if (kPer == 2) *reinterpret_cast<float2*>(to) = make_float2(s[0][c], s[kPer - 1][c]);
      else *to = s[0][c];
    }
    wait_copies<0>();
    __syncthreads();  // S and the chunk's operands are there, and nobody reads the other stage any more
    if (chunk + 1 < chunks) fetch(chunk + 1);
    const float* ys = chunk_smem + (chunk & 1) * walk_stage(ROWS);
    const float* kds = ys + C * kLd;
    const float* ws = kds + C * kLd;
    const float* es = ws + C * kColumns;
    {
      // Tokens 4 warp .. + 3, columns ct, ct + 4, .., every eighth group of four rows; sums over even and odd rows side by side.
      const int ct = lane & 3, part = lane >> 2;
      const float* y = ys + warp * 4 * kLd + part * 4;
      const float* t = tile + ct * kLdS + part * 4;
      pair_t acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0;
#pragma unroll
      for (int k = 0; k < ROWS; k += 32) {
        quad_t a[4], b[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          a[x] = load_quad(y + x * kLd + k);
          b[x] = load_quad(t + x * 4 * kLdS + k);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][c] = fma_pair(a[i].hi, b[c].hi, fma_pair(a[i].lo, b[c].lo, acc[i][c]));
      }
      // The eight parts meet: a lane ends with two columns of one token.
      const bool b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
      float sum[4][4], two[2][4], row[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[i][c] = sum_pair(acc[i][c]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) two[i][c] = from_pair(b2 ? sum[i][c] : sum[i + 2][c], b2 ? sum[i + 2][c] : sum[i][c], 4);
#pragma unroll
      for (int c = 0; c < 4; ++c) row[c] = from_pair(b3 ? two[0][c] : two[1][c], b3 ? two[1][c] : two[0][c], 8);
      const int i = warp * 4 + (b2 ? 2 : 0) + (b3 ? 1 : 0), c = ct + (b4 ? 8 : 0);
      const float u0 = from_pair(b4 ? row[0] : row[2], b4 ? row[2] : row[0], 16) + ws[i * kColumns + c];
      const float u1 = from_pair(b4 ? row[1] : row[3], b4 ? row[3] : row[1], 16) + ws[i * kColumns + c + 4];
      xs[i * kRowX + c] = u0, xs[i * kRowX + c + 4] = u1;
      if (i < n) {
        float* to = from.x + ((first + i) * from.heads + own_head) * columns + col0 + c;
        to[0] = u0, to[4] = u1;
      }
    }
    // The state in front of the chunk, for `chunk_out`.
#pragma unroll
    for (int r = 0; r < kPer; ++r) *reinterpret_cast<float4*>(s_out + static_cast<int64_t>(r) * columns) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
    __syncthreads();
    {
      float add[4][4];  // summed apart from the state, which is rounded once a chunk
#pragma unroll
      for (int r = 0; r < 4; ++r) add[r][0] = add[r][1] = add[r][2] = add[r][3] = 0.f;
      const float* kd = kds + jp * kLd + quad;
      const float* x = xs + jp * kRowX + cg * 4;
#pragma unroll 4
      for (int j = 0; j < C; j += kSplit) {
        const float4 u = *reinterpret_cast<const float4*>(x + j * kRowX);
        const float4 kj = *reinterpret_cast<const float4*>(kd + j * kLd);
        const float f[4] = {kj.x, kj.y, kj.z, kj.w};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          add[r][0] = fmaf(f[r], u.x, add[r][0]), add[r][1] = fmaf(f[r], u.y, add[r][1]);
          add[r][2] = fmaf(f[r], u.z, add[r][2]), add[r][3] = fmaf(f[r], u.w, add[r][3]);
        }
      }
      // The lanes of a tile meet, each keeping kPer rows.
      if (kSplit == 4) {
        const bool high = jp & 2;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) add[r][c] = from_pair(high ? add[r][c] : add[r + 2][c], high ? add[r + 2][c] : add[r][c], 2);
      }
      if (kSplit >= 2) {
        const bool high = jp & 1;
#pragma unroll
        for (int r = 0; r < kPer; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) add[r][c] = from_pair(high ? add[r][c] : add[r + kPer][c], high ? add[r + kPer][c] : add[r][c], 1);
      }
#pragma unroll
      for (int r = 0; r < kPer; ++r) {
        const float e = es[row0 + r];
        if (ADD) add[r][0] += own[r].x, add[r][1] += own[r].y, add[r][2] += own[r].z, add[r][3] += own[r].w;
#pragma unroll
        for (int c = 0; c < 4; ++c) s[r][c] = fmaf(e, s[r][c], add[r][c]);
      }
    }
  }
  if (chunks > 0) {
#pragma unroll
    for (int r = 0; r < kPer; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (row0 + r < dk && col0 + cg * 4 + c < dv) s_base[static_cast<int64_t>(row0 + r) * dv + cg * 4 + c] = s[r][c];
  }
}

// --- outputs ---------------------------------------------------------------------------------------------------------------------------
//
// One block per (chunk, head, request and COLS columns): O = Qt S (+ A U) (+ Av V) as one product over rows + 32 (+ 32) numbers, 32 of
// them at a time by cp.async in two stages. A thread has eight tokens and four neighbouring columns: 12 numbers read for 32 FMAs, since
// what an SM takes out of shared memory (32 numbers a cycle, however many lanes want the same one) bounds this kernel.
constexpr int kLdSlab = C + 4;
constexpr size_t out_smem(int cols) { return sizeof(float) * 2 * (C * kLdSlab + C * (cols + 4)); }

template <int COLS, bool WITH_U, bool WITH_V>
__global__ void __launch_bounds__(COLS)
chunk_out_kernel(const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int heads, int dv, int rows, int tiles, Scratch from, const float* v,
                 int64_t v_ld, int v_wide, float* out, float* den) {
  extern __shared__ __align__(16) float chunk_smem[];
  constexpr int kLdOut = COLS + 4, kStage = C * kLdSlab + C * kLdOut;
  let_successor_start();
  const int seq = blockIdx.z / tiles, col0 = blockIdx.z % tiles * COLS, own_head = blockIdx.y, head = from.head0 + own_head, chunk = blockIdx.x;
  const int start = seq_q_start[seq], n = min(C, seq_q_len[seq] - chunk * C);
  if (n <= 0) return;
  const int64_t first = static_cast<int64_t>(start) + chunk * C;
  const int columns = padded_columns(dv), width = min(COLS, columns - col0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* states = from.s + (chunk_place(start, seq, chunk) * from.heads + own_head) * rows * columns + col0;
  const int state_slabs = rows / C, slabs = state_slabs + (WITH_U ? 1 : 0) + (WITH_V ? 1 : 0);
  wait_for_predecessor();
  auto fetch = [&](int slab) {
    float* left = chunk_smem + (slab & 1) * kStage;
    float* right = left + C * kLdSlab;
    const bool in_state = slab < state_slabs, is_u = WITH_U && slab == state_slabs;
    const float* pairs = is_u ? from.a : from.av;
#pragma unroll
    for (int r = tid >> 3; r < C; r += COLS / 8) {
      const int c = (tid & 7) * 4;
      const int64_t row = (first + r) * from.heads + own_head;
      stage_copy<16>(left + r * kLdSlab + c, r < n ? (in_state ? from.qt + row * rows + slab * C + c : pairs + row * C + c) : from.qt, r < n);
    }
    if (in_state || is_u) {
#pragma unroll
      for (int r = tid / (COLS / 4); r < C; r += 4) {
        const int c = tid % (COLS / 4) * 4;
        const bool valid = c < width && (in_state || r < n);
        const float* at = in_state ? states + static_cast<int64_t>(slab * C + r) * columns + c : from.x + ((first + r) * from.heads + own_head) * columns + col0 + c;
        stage_copy<16>(right + r * kLdOut + c, valid ? at : from.qt, valid);
      }
    } else if (v_wide) {
#pragma unroll
      for (int r = tid / (COLS / 4); r < C; r += 4) {
        const int c = tid % (COLS / 4) * 4;
        const bool valid = col0 + c < dv && r < n;
        stage_copy<16>(right + r * kLdOut + c, valid ? v + (first + r) * v_ld + static_cast<int64_t>(head) * dv + col0 + c : v, valid);
      }
    } else {
      for (int r = 0; r < C; ++r) {
        const bool valid = col0 + tid < dv && r < n;
        stage_copy<4>(right + r * kLdOut + tid, valid ? v + (first + r) * v_ld + static_cast<int64_t>(head) * dv + col0 + tid : v, valid);
      }
    }
    commit_copies();
  };
  const int ct = (lane & 7) + 8 * warp, it = lane >> 3;  // columns 4 ct .. + 3, tokens it, it + 4, ..
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  fetch(0);
  if (den != nullptr && col0 == 0) {  // the normaliser read out as the state is: n . (e q) + the chunk's own pairs
    const float* n0 = from.n + (chunk_place(start, seq, chunk) * from.heads + own_head) * rows;
    for (int r = warp; r < n; r += COLS / 32) {
      const int64_t row = (first + r) * from.heads + own_head;
      float sum = from.av[row * C + lane];
      for (int c = lane; c < rows; c += 32) sum = fmaf(from.qt[row * rows + c], n0[c], sum);
      sum = warp_sum(sum);
      if (lane == 0) den[(first + r) * heads + head] = sum;
    }
  }
  for (int slab = 0; slab < slabs; ++slab) {
    if (slab + 1 < slabs) {
      fetch(slab + 1);
      wait_copies<1>();
    } else {
      wait_copies<0>();
    }
    __syncthreads();
    const float* left = chunk_smem + (slab & 1) * kStage + it * kLdSlab;
    const float* right = chunk_smem + (slab & 1) * kStage + C * kLdSlab + ct * 4;
    float sum[8][4];  // one slab's sum by itself: fewer roundings of the whole
#pragma unroll
    for (int i = 0; i < 8; ++i) sum[i][0] = sum[i][1] = sum[i][2] = sum[i][3] = 0.f;
    // Pairs of tokens form a triangle: a token leaves out those behind it (a value there that is not finite times a pair's zero is
    // not zero). Tokens 4 i .. + 3 of a warp stand against tokens k .. k + 3, so only one group of four looks at its lanes.
    auto multiply = [&](auto triangle) {
      constexpr bool kTriangle = decltype(triangle)::value;
#pragma unroll 2
      for (int k = 0; k < C; k += 4) {
        float4 b[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) b[x] = *reinterpret_cast<const float4*>(right + (k + x) * kLdOut);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (kTriangle && k > 4 * i) continue;
          const float4 a = *reinterpret_cast<const float4*>(left + i * 4 * kLdSlab + k);
          const float f[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if (kTriangle && k == 4 * i && x > it) continue;
            sum[i][0] = fmaf(f[x], b[x].x, sum[i][0]), sum[i][1] = fmaf(f[x], b[x].y, sum[i][1]);
            sum[i][2] = fmaf(f[x], b[x].z, sum[i][2]), sum[i][3] = fmaf(f[x], b[x].w, sum[i][3]);
          }
        }
      }
    };
    if (slab < state_slabs) multiply(std::false_type{});
    else multiply(std::true_type{});
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] += sum[i][0], acc[i][1] += sum[i][1], acc[i][2] += sum[i][2], acc[i][3] += sum[i][3];
    __syncthreads();
  }
  const int c = col0 + ct * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = it + 4 * i;
    if (row >= n) continue;
    float* to = out + ((first + row) * heads + head) * dv + c;
    if (dv % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
      if (c < dv) *reinterpret_cast<float4*>(to) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (c + x < dv) to[x] = acc[i][x];
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
  const int64_t rows = padded_rows(z.dk), columns = padded_columns(z.dv), per_head = static_cast<int64_t>(z.tokens) * heads;
  const int64_t chunks = (static_cast<int64_t>(z.tokens) / C + z.seqs + 1) * heads;
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
            raise_smem(chunk_walk_kernel<ROWS, false>, walk_smem(ROWS));
  if constexpr (ROWS <= kMaxLinearRows) {
    const size_t general = linear_prepare_smem(ROWS, kGeneralDelta), linear = linear_prepare_smem(ROWS, kLinear), memory = linear_prepare_smem(ROWS, kMemory);
    ok = ok && raise_smem(linear_chunk_prepare_kernel<ROWS, 1, kLinear>, linear) && raise_smem(linear_chunk_prepare_kernel<ROWS, 4, kLinear>, linear) &&
         raise_smem(linear_chunk_prepare_kernel<ROWS, 1, kGeneralDelta>, general) && raise_smem(linear_chunk_prepare_kernel<ROWS, 4, kGeneralDelta>, general) &&
         raise_smem(linear_chunk_prepare_kernel<ROWS, 1, kMemory>, memory) && raise_smem(linear_chunk_prepare_kernel<ROWS, 4, kMemory>, memory) &&
         raise_smem(chunk_walk_kernel<ROWS, true>, walk_smem(ROWS));
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
// with one decay per head take 418 us in one part, 481 in two, 627 in three, 786 in four (token by token 810), 24 heads of 64 x 64 under the
// generalized rule 236, 335, 417 and 544 (465).
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
  launch_kernel_as(true, walk, dim3(padded_columns(z.dv) / kColumns, scratch.heads, z.seqs), dim3(kThreads), walk_smem(rows), stream, req.q_start, req.q_len, req.slot,
                   z.heads, z.dk, z.dv, scratch, state);
  return b200_check_launch("chunk_walk");
}

template <bool WITH_U, bool WITH_V>
int launch_out(const Sizes& z, const Requests& req, const Scratch& scratch, const float* v, int64_t v_ld, float* out, float* den, cudaStream_t stream) {
  const int columns = padded_columns(z.dv), cols = columns <= 64 ? 64 : 128, tiles = (columns + cols - 1) / cols;
  launch_kernel(cols == 64 ? chunk_out_kernel<64, WITH_U, WITH_V> : chunk_out_kernel<128, WITH_U, WITH_V>, dim3((z.max_q_len + C - 1) / C, scratch.heads, z.seqs * tiles),
                dim3(cols), out_smem(cols), stream, req.q_start, req.q_len, z.heads, z.dv, padded_rows(z.dk), tiles, scratch, v,
                v_ld, z.dv % 4 == 0 && v_ld % 4 == 0 && aligned16(v) ? 1 : 0, out, den);
  return b200_check_launch("chunk_out");
}

int launch_linear_prepare(const Sizes& z, const Requests& req, int rule, bool wide, const LinearRule& in, const Scratch& scratch, cudaStream_t stream) {
  const int rows = padded_rows(z.dk);
  launch_kernel(rows == 64 ? linear_prepare_form<64>(wide, rule) : linear_prepare_form<128>(wide, rule), dim3((z.max_q_len + C - 1) / C, scratch.heads, z.seqs),
                dim3(kThreads), linear_prepare_smem(rows, rule), stream, in, req.q_start, req.q_len, z.heads, z.dk, z.dv, scratch);
  return b200_check_launch("linear_chunk_prepare");
}

int launch_scan(const Sizes& z, const Requests& req, const Scratch& scratch, float* state, float* normaliser, cudaStream_t stream) {
  const int rows = padded_rows(z.dk), blocks = (rows * padded_columns(z.dv) / 4 + kThreads - 1) / kThreads;
  launch_kernel(chunk_scan_kernel, dim3(blocks + (normaliser != nullptr ? (rows + kThreads - 1) / kThreads : 0), scratch.heads, z.seqs), dim3(kThreads), 0, stream, req.q_start,
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
