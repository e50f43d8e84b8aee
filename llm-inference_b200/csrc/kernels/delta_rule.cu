// The gated delta rule with one decay per head and key channel, and what surrounds it.
//
// Per head, with a state S [dk][dv] that starts at zero and is carried from token to token:
//   S <- g (.) S (g scales the rows of S, one factor per key channel);  u = beta (v - S^T k);
//   S <- S + k u^T;  o = S^T q   (the read-out sees the token's own write).
// q and k are unit vectors per head (q also times dk^-1/2) made from projections that first pass
// a short causal convolution over time and silu; g = exp(-exp(A_log[h]) softplus(a + dt_bias));
// beta = sigmoid(b). The state and the convolution's last taps - 1 inputs live in per-request
// slots. Everything that enters the recurrence is 32-bit. The form with one decay per head has a
// recurrence of its own (delta_head.cu); `delta_prepare` and `delta_output` serve both, the latter
// with a sigmoid or a silu of the gate.
//
// Kernels: `delta_prepare` (one block per token: convolution, silu, unit vectors, beta, decay,
// and k . q where the recurrence wants it),
// `conv_state_update` (one block per request: the slot's last inputs), `delta_recurrence` (the
// columns of S are independent, so a thread group owns a column and walks the request's tokens),
// `delta_output` (o / rms(o) * w * sigmoid(gate)).
#include <type_traits>

#include "common.cuh"
#include "packs.cuh"

namespace {

__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float silu_f(float x) { return x * sigmoid_quick(x); }
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// `proj` rows: [q (kv_heads*dk) | k (kv_heads*dk) | v (heads*dv) | b (heads)]; the first
// `channels` = 2 kv_heads dk + heads dv columns pass the convolution. `conv_state`
// [slots][taps-1][channels] holds each request's last inputs, oldest first. `decay_in`
// [tokens][heads * span] is the projection the decays come from. Without `kq_out` there is a decay per head and key
// channel (span = dk) and `decay_out` takes the factors; with it there is one per head (span = 1), `decay_out` takes
// their logarithms, and `kq_out` k . q per kv head, of the vectors as they are written.
template <typename T>
__global__ void delta_prepare_kernel(const T* proj, int ld, const T* decay_in, int decay_ld,
                                     const float* __restrict__ taps_w, int taps, const T* conv_state,
                                     const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                     const int* token_seq, const int* seq_q_start, const int* seq_slot, int heads,
                                     int kv_heads, int dk, int dv, float* q_out, float* k_out, float* v_out, float* beta_out,
                                     float* decay_out, float* kq_out) {
  extern __shared__ float y[];  // [channels]
  wait_for_predecessor();
  let_successor_start();
  const int t = blockIdx.x, tid = threadIdx.x;
  const int qk = kv_heads * dk, vw = heads * dv;
  const int channels = 2 * qk + vw;
  const int seq = token_seq[t];
  const int run = t - seq_q_start[seq];  // tokens of this request in front of t within the step
  const T* state = conv_state + static_cast<int64_t>(seq_slot[seq]) * (taps - 1) * channels;
  for (int c = tid; c < channels; c += blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < taps; ++j) {
      const int back = taps - 1 - j;  // how many tokens before t
      const float x = back <= run ? to_f32<T>(proj[static_cast<int64_t>(t - back) * ld + c])
                                  : to_f32<T>(state[static_cast<int64_t>(taps - 1 + run - back) * channels + c]);
      acc = fmaf(taps_w[c * taps + j], x, acc);
    }
    y[c] = acc * sigmoid_f(acc);
  }
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  // unit vectors: one warp per (q or k, kv head); k . q is worked out beside k
  for (int item = warp; item < 2 * kv_heads; item += warps) {
    const float* src = y + item * dk;
    float ss = 0.f;
    for (int i = lane; i < dk; i += 32) ss = fmaf(src[i], src[i], ss);
    ss = warp_sum(ss);
    const bool is_q = item < kv_heads;
    const float factor = (1.f / sqrtf(ss + 1e-6f)) * (is_q ? 1.f / sqrtf(static_cast<float>(dk)) : 1.f);
    const int head = is_q ? item : item - kv_heads;
    float* dst = (is_q ? q_out : k_out) + static_cast<int64_t>(t) * qk + head * dk;
    for (int i = lane; i < dk; i += 32) dst[i] = src[i] * factor;
    if (kq_out != nullptr && !is_q) {
      const float* q = y + head * dk;
      float q_ss = 0.f, dot = 0.f;
      for (int i = lane; i < dk; i += 32) q_ss = fmaf(q[i], q[i], q_ss), dot = fmaf(q[i], src[i], dot);
      q_ss = warp_sum(q_ss);
      dot = warp_sum(dot);
      if (lane == 0)
        kq_out[static_cast<int64_t>(t) * kv_heads + head] = dot * factor * ((1.f / sqrtf(q_ss + 1e-6f)) * (1.f / sqrtf(static_cast<float>(dk))));
    }
  }
  for (int i = tid; i < vw; i += blockDim.x) v_out[static_cast<int64_t>(t) * vw + i] = y[2 * qk + i];
  for (int h = tid; h < heads; h += blockDim.x)
    beta_out[static_cast<int64_t>(t) * heads + h] = sigmoid_f(to_f32<T>(proj[static_cast<int64_t>(t) * ld + channels + h]));
  const bool per_head = kq_out != nullptr;
  const int span = per_head ? 1 : dk;
  for (int i = tid; i < heads * span; i += blockDim.x) {
    const float step = softplus_f(to_f32<T>(decay_in[static_cast<int64_t>(t) * decay_ld + i]) + dt_bias[i]);
    const float log_decay = -expf(a_log[i / span]) * step;
    decay_out[static_cast<int64_t>(t) * heads * span + i] = per_head ? log_decay : expf(log_decay);
  }
}

// The same for prompt portions and four taps. A warp takes four neighbouring tokens and up to 128 channels: a q and a k head, or a piece of
// the values or of the decays, four neighbouring channels a lane, so that nothing passes through shared memory, rows and taps
// are read once for the four tokens that want them, and a lane's seven rows are asked for together. Only tokens next to a request's
// start look into its slot.
// What bounds it: instructions (exponentials, logarithms, quotients). One block for four tokens of all channels held 128 registers a thread, so
// two blocks an SM, and went through a token's rows with a look at its request for every tap: on a B200 2,048 tokens of 12 heads of 128 took, the
// slots' update with them, 56 us with a decay per channel and 45 with one per head, now 28 and 21
// (with divisions nearly what they took before: their code, in line sixteen times, does not fit what an SM holds of it).
// Heads of more than 256 channels do not fit a warp's registers: the four warps of a block share one, and its numbers wait for their factors where they
// go (4 heads of 512, 2,048 tokens: 78 us with a decay per channel and 59 with one per head in the form for single tokens, 55 and 41 in the block for all
// channels, now 40 and 27; 300 tokens 21 and 17, 24 and 20, now 11 and 9; one warp a head 23 and 23).
constexpr int kWideTokens = 4, kWideTaps = 4, kWideChannels = 128;

struct WidePrepare {
  int ld, decay_ld, tokens, heads, kv_heads, dk, dv;
  const float* taps_w;
  const float* a_log;
  const float* dt_bias;
  const int* token_seq;
  const int* seq_q_start;
  const int* seq_slot;
  float* q_out;
  float* k_out;
  float* v_out;
  float* beta_out;
  float* decay_out;
  float* kq_out;
  int v_pieces, decay_pieces;
};

// Channels c .. + 3 of tokens t0 .. + 3 behind the convolution and silu. `inside`: all of them at least three tokens into one request.
template <typename T>
__device__ __forceinline__ void convolve_wide(float4 (&y)[kWideTokens], const WidePrepare& p, const T* proj, const T* conv_state, int t0, int count, bool inside, int c) {
  float4 rows[kWideTokens + kWideTaps - 1];  // inputs of tokens t0 - 3 .. t0 + 3
#pragma unroll
  for (int i = 0; i < kWideTokens + kWideTaps - 1; ++i) {
    const int t = t0 - (kWideTaps - 1) + i;
    rows[i] = t >= 0 && t < p.tokens ? load4<T>(proj + static_cast<int64_t>(t) * p.ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float4 taps[4];  // of channel c + x
#pragma unroll
  for (int x = 0; x < 4; ++x) taps[x] = *reinterpret_cast<const float4*>(p.taps_w + (c + x) * kWideTaps);
  const float* w[4] = {&taps[0].x, &taps[1].x, &taps[2].x, &taps[3].x};
#pragma unroll
  for (int i = 0; i < kWideTokens; ++i) {
    float4 in[kWideTaps];
#pragma unroll
    for (int j = 0; j < kWideTaps; ++j) in[j] = rows[i + j];
    if (!inside && i < count) {
      const int seq = p.token_seq[t0 + i], run = t0 + i - p.seq_q_start[seq];  // tokens of this request in front of t within the step
      const int64_t slot = static_cast<int64_t>(p.seq_slot[seq]) * (kWideTaps - 1);
#pragma unroll
      for (int j = 0; j < kWideTaps - 1; ++j)
        if (kWideTaps - 1 - j > run) in[j] = load4<T>(conv_state + (slot + run + j) * (2 * p.kv_heads * p.dk + p.heads * p.dv) + c);
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kWideTaps; ++j) {
      acc.x = fmaf(w[0][j], in[j].x, acc.x), acc.y = fmaf(w[1][j], in[j].y, acc.y);
      acc.z = fmaf(w[2][j], in[j].z, acc.z), acc.w = fmaf(w[3][j], in[j].w, acc.w);
    }
    y[i] = make_float4(silu_f(acc.x), silu_f(acc.y), silu_f(acc.z), silu_f(acc.w));
  }
}

template <typename T, int QUADS>  // QUADS: a q or k head has up to 128 QUADS channels; 0: any number, a block's four warps a head
__global__ void __launch_bounds__(128, QUADS == 1 ? 6 : 4)
delta_prepare_wide_kernel(const WidePrepare p, const T* proj, const T* decay_in, const T* conv_state) {
  const int items = p.kv_heads + p.v_pieces + p.decay_pieces + 1;
  // Tokens run fastest: what an SM works on at a time is then of one kind, whose code it holds.
  const int groups = (p.tokens + kWideTokens - 1) / kWideTokens, lane = threadIdx.x & 31, own = threadIdx.x >> 5;
  const int64_t warp = static_cast<int64_t>(blockIdx.x) * 4 + own;
  const int t0 = static_cast<int>((QUADS == 0 ? blockIdx.x : warp) % groups) * kWideTokens;
  int item = static_cast<int>(warp / groups);
  if (QUADS == 0) {
    item = blockIdx.x / groups;
    if (item >= p.kv_heads) item += 3 * (item - p.kv_heads) + own;
  }
  if (item >= items) return;
  const int count = min(kWideTokens, p.tokens - t0);
  const int qk = p.kv_heads * p.dk, vw = p.heads * p.dv;
  const int seq = p.token_seq[t0];
  const bool inside = p.token_seq[t0 + count - 1] == seq && t0 - p.seq_q_start[seq] >= kWideTaps - 1;
  wait_for_predecessor();
  let_successor_start();
  if (QUADS == 0 && item < p.kv_heads) {
    float q_ss[kWideTokens] = {}, k_ss[kWideTokens] = {}, dot[kWideTokens] = {};
    float* q_to = p.q_out + static_cast<int64_t>(t0) * qk + item * p.dk;
    float* k_to = p.k_out + static_cast<int64_t>(t0) * qk + item * p.dk;
#pragma unroll 1
    for (int c = threadIdx.x * 4; c < p.dk; c += 4 * kWideChannels) {
      float4 q[kWideTokens], k[kWideTokens];
      convolve_wide<T>(q, p, proj, conv_state, t0, count, inside, item * p.dk + c);
      convolve_wide<T>(k, p, proj, conv_state, t0, count, inside, qk + item * p.dk + c);
#pragma unroll
      for (int i = 0; i < kWideTokens; ++i) {
        const float4 a = q[i], b = k[i];
        q_ss[i] = square_sum(a, q_ss[i]), k_ss[i] = square_sum(b, k_ss[i]);
        dot[i] = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, dot[i]))));
        if (i < count) *reinterpret_cast<float4*>(q_to + static_cast<int64_t>(i) * qk + c) = a, *reinterpret_cast<float4*>(k_to + static_cast<int64_t>(i) * qk + c) = b;
      }
    }
    __shared__ float sums[kWideTokens][3][4];
#pragma unroll
    for (int i = 0; i < kWideTokens; ++i) {
      q_ss[i] = warp_sum(q_ss[i]), k_ss[i] = warp_sum(k_ss[i]), dot[i] = warp_sum(dot[i]);
      if (lane == 0) sums[i][0][own] = q_ss[i], sums[i][1][own] = k_ss[i], sums[i][2][own] = dot[i];
    }
    __syncthreads();
    const auto whole = [&](int i, int kind) { return (sums[i][kind][0] + sums[i][kind][1]) + (sums[i][kind][2] + sums[i][kind][3]); };
#pragma unroll 1
    for (int i = 0; i < count; ++i) {
      const float q_factor = (1.f / sqrtf(whole(i, 0) + 1e-6f)) * (1.f / sqrtf(static_cast<float>(p.dk))), k_factor = 1.f / sqrtf(whole(i, 1) + 1e-6f);
      for (int c = threadIdx.x * 4; c < p.dk; c += 4 * kWideChannels) {  // a thread's own numbers again
        float4* q = reinterpret_cast<float4*>(q_to + static_cast<int64_t>(i) * qk + c);
        float4* k = reinterpret_cast<float4*>(k_to + static_cast<int64_t>(i) * qk + c);
        *q = scale_each(*q, q_factor), *k = scale_each(*k, k_factor);
      }
      if (p.kq_out != nullptr && threadIdx.x == 0) p.kq_out[static_cast<int64_t>(t0 + i) * p.kv_heads + item] = whole(i, 2) * k_factor * q_factor;
    }
    return;
  }
  if (QUADS > 0 && item < p.kv_heads) {  // unit vectors, and k . q
    float q_factor[kWideTokens], k_factor[kWideTokens], dot[kWideTokens];
    float4 q[QUADS + (QUADS == 0)][kWideTokens], k[QUADS + (QUADS == 0)][kWideTokens];
#pragma unroll
    for (int x = 0; x < QUADS; ++x) {
      const int c = x * kWideChannels + lane * 4;
      if (c < p.dk) {
        convolve_wide<T>(q[x], p, proj, conv_state, t0, count, inside, item * p.dk + c);
        convolve_wide<T>(k[x], p, proj, conv_state, t0, count, inside, qk + item * p.dk + c);
      } else {
#pragma unroll
        for (int i = 0; i < kWideTokens; ++i) q[x][i] = k[x][i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int i = 0; i < kWideTokens; ++i) {
      float q_ss = 0.f, k_ss = 0.f;
      dot[i] = 0.f;
#pragma unroll
      for (int x = 0; x < QUADS; ++x) {
        const float4 a = q[x][i], b = k[x][i];
        q_ss = square_sum(a, q_ss), k_ss = square_sum(b, k_ss);
        dot[i] = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, dot[i]))));
      }
      q_ss = warp_sum(q_ss), k_ss = warp_sum(k_ss);
      q_factor[i] = (1.f / sqrtf(q_ss + 1e-6f)) * (1.f / sqrtf(static_cast<float>(p.dk))), k_factor[i] = 1.f / sqrtf(k_ss + 1e-6f);
    }
#pragma unroll
    for (int i = 0; i < kWideTokens; ++i) {
      if (i >= count) break;
      const int64_t t = t0 + i;
#pragma unroll
      for (int x = 0; x < QUADS; ++x) {
        const int c = x * kWideChannels + lane * 4;
        if (c >= p.dk) break;
        *reinterpret_cast<float4*>(p.q_out + t * qk + item * p.dk + c) = scale_each(q[x][i], q_factor[i]);
        *reinterpret_cast<float4*>(p.k_out + t * qk + item * p.dk + c) = scale_each(k[x][i], k_factor[i]);
      }
      if (p.kq_out != nullptr) {
        const float whole = warp_sum(dot[i]);
        if (lane == 0) p.kq_out[t * p.kv_heads + item] = whole * k_factor[i] * q_factor[i];
      }
    }
    return;
  }
  item -= p.kv_heads;
  if (item < p.v_pieces) {
    const int c = item * kWideChannels + lane * 4;
    if (c >= vw) return;
    float4 y[kWideTokens];
    convolve_wide<T>(y, p, proj, conv_state, t0, count, inside, 2 * qk + c);
#pragma unroll
    for (int i = 0; i < kWideTokens; ++i)
      if (i < count) *reinterpret_cast<float4*>(p.v_out + static_cast<int64_t>(t0 + i) * vw + c) = y[i];
    return;
  }
  item -= p.v_pieces;
  if (item < p.decay_pieces) {  // one per head and key channel
    const int c = item * kWideChannels + lane * 4;
    if (c >= p.heads * p.dk) return;
    const float rate = -expf(p.a_log[c / p.dk]);
    const float4 bias = *reinterpret_cast<const float4*>(p.dt_bias + c);
    float4 next = load4<T>(decay_in + static_cast<int64_t>(t0) * p.decay_ld + c);
#pragma unroll 1
    for (int i = 0; i < count; ++i) {
      const float4 z = next;
      if (i + 1 < count) next = load4<T>(decay_in + static_cast<int64_t>(t0 + i + 1) * p.decay_ld + c);
      *reinterpret_cast<float4*>(p.decay_out + static_cast<int64_t>(t0 + i) * p.heads * p.dk + c) =
          make_float4(expf(rate * softplus_f(z.x + bias.x)), expf(rate * softplus_f(z.y + bias.y)), expf(rate * softplus_f(z.z + bias.z)),
                      expf(rate * softplus_f(z.w + bias.w)));
    }
    return;
  }
  for (int idx = lane; idx < count * p.heads; idx += 32) {
    const int64_t t = t0 + idx / p.heads;
    const int h = idx % p.heads;
    p.beta_out[t * p.heads + h] = sigmoid_f(to_f32<T>(proj[t * p.ld + 2 * qk + vw + h]));
    if (p.kq_out != nullptr) p.decay_out[t * p.heads + h] = -expf(p.a_log[h]) * softplus_f(to_f32<T>(decay_in[t * p.decay_ld + h]) + p.dt_bias[h]);
  }
}

// After a step the slot holds the last taps - 1 inputs of [old slot | the step's inputs].
template <typename T>
__global__ void conv_state_update_kernel(const T* proj, int ld, int channels, int taps, const int* seq_q_start,
                                         const int* seq_q_len, const int* seq_slot, T* conv_state) {
  wait_for_predecessor();
  let_successor_start();
  const int seq = blockIdx.x;
  const int start = seq_q_start[seq], len = seq_q_len[seq];
  const int keep = taps - 1;
  T* state = conv_state + static_cast<int64_t>(seq_slot[seq]) * keep * channels;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
    for (int r = 0; r < keep; ++r) {
      const int at = len + r;  // index into [old slot (keep) | inputs (len)]
      state[static_cast<int64_t>(r) * channels + c] =
          at < keep ? state[static_cast<int64_t>(at) * channels + c] : proj[static_cast<int64_t>(start + at - keep) * ld + c];
    }
  }
}

// A block owns `cols` columns of one head of one request; a column's dk rows are spread over
// `lanes_per_col` neighbouring lanes (row r on lane r % lanes_per_col), PER rows per lane in
// registers: few rows per lane keep the two dot products' chains of dependent FMAs short, which
// is what a token's latency is made of. The tokens' q, k, g, v and beta arrive kStage at a time
// by cp.async in a ring of two stages, so the next tokens load while these are worked on.
constexpr int kRecurrenceThreads = 128;
constexpr int kStage = 8;

// `bytes` (4 or 16) global -> shared; with `valid` false zeros are written and nothing is read.
template <int kBytes>
__device__ __forceinline__ void stage_copy(float* smem, const float* gmem, bool valid) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? kBytes : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(kBytes), "r"(bytes) : "memory");
}

template <int PER, int LANES>
__global__ void __launch_bounds__(kRecurrenceThreads)
delta_recurrence_kernel(const float* q, const float* k, const float* v, const float* beta, const float* decay,
                        const int* seq_q_start, const int* seq_q_len, const int* seq_slot, int heads, int kv_heads, int dk,
                        int dv, int vec, float* state, float* out) {
  extern __shared__ __align__(16) float stage[];
  let_successor_start();
  constexpr int lanes_per_col = LANES;
  constexpr int cols = kRecurrenceThreads / lanes_per_col;
  const int seq = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * cols;
  const int tid = threadIdx.x;
  const int part = tid % lanes_per_col, col = col0 + tid / lanes_per_col;
  constexpr int padded = PER * lanes_per_col;
  constexpr int per_stage = kStage * (3 * padded + cols) + kStage;
  const int start = seq_q_start[seq], len = seq_q_len[seq];
  const int kvh = head / (heads / kv_heads);
  const bool live = col < dv;
  float* s_base = state + (static_cast<int64_t>(seq_slot[seq]) * heads + head) * dk * dv;
  wait_for_predecessor();
  // Rows past dk (when dk is no multiple of the lanes) hold zeros in q, k and g and stay zero.
  auto fetch = [&](int buffer, int t0) {
    float* sq = stage + buffer * per_stage;
    float* sk = sq + kStage * padded;
    float* sg = sk + kStage * padded;
    float* sv = sg + kStage * padded;
    float* sb = sv + kStage * cols;
    const int count = min(kStage, len - t0);
    const int64_t first = static_cast<int64_t>(start) + t0;
    if (vec) {
      for (int idx = tid * 4; idx < count * padded; idx += kRecurrenceThreads * 4) {
        const int j = idx / padded, r = idx % padded;
        const int64_t tok = first + j;
        const bool in = r < dk;
        const int rr = in ? r : 0;
        stage_copy<16>(sq + idx, q + (tok * kv_heads + kvh) * dk + rr, in);
        stage_copy<16>(sk + idx, k + (tok * kv_heads + kvh) * dk + rr, in);
        stage_copy<16>(sg + idx, decay + (tok * heads + head) * dk + rr, in);
      }
      for (int idx = tid * 4; idx < count * cols; idx += kRecurrenceThreads * 4) {
        const int j = idx / cols, c = col0 + idx % cols;
        stage_copy<16>(sv + idx, v + ((first + j) * heads + head) * dv + (c < dv ? c : 0), c < dv);
      }
    } else {
      for (int idx = tid; idx < count * padded; idx += kRecurrenceThreads) {
        const int j = idx / padded, r = idx % padded;
        const int64_t tok = first + j;
        const bool in = r < dk;
        const int rr = in ? r : 0;
        stage_copy<4>(sq + idx, q + (tok * kv_heads + kvh) * dk + rr, in);
        stage_copy<4>(sk + idx, k + (tok * kv_heads + kvh) * dk + rr, in);
        stage_copy<4>(sg + idx, decay + (tok * heads + head) * dk + rr, in);
      }
      for (int idx = tid; idx < count * cols; idx += kRecurrenceThreads) {
        const int j = idx / cols, c = col0 + idx % cols;
        stage_copy<4>(sv + idx, v + ((first + j) * heads + head) * dv + (c < dv ? c : 0), c < dv);
      }
    }
    if (tid < count) stage_copy<4>(sb + tid, beta + (first + tid) * heads + head, true);
  };
  float s[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int r = i * lanes_per_col + part;
    s[i] = (live && r < dk) ? s_base[static_cast<int64_t>(r) * dv + col] : 0.f;
  }
  if (len > 0) fetch(0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int t0 = 0, buffer = 0; t0 < len; t0 += kStage, buffer ^= 1) {
    if (t0 + kStage < len) fetch(buffer ^ 1, t0 + kStage);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float* sq = stage + buffer * per_stage;
    const float* sk = sq + kStage * padded;
    const float* sg = sk + kStage * padded;
    const float* sv = sg + kStage * padded;
    const float* sb = sv + kStage * cols;
    const int count = min(kStage, len - t0);
    for (int j = 0; j < count; ++j) {
      const float* kj = sk + j * padded + part;
      const float* gj = sg + j * padded + part;
      const float* qj = sq + j * padded + part;
      float kr[PER];
      float ks0 = 0.f, ks1 = 0.f;
#pragma unroll
      for (int i = 0; i < PER; i += 2) {
        kr[i] = kj[i * lanes_per_col], kr[i + 1] = kj[(i + 1) * lanes_per_col];
        s[i] *= gj[i * lanes_per_col], s[i + 1] *= gj[(i + 1) * lanes_per_col];
        ks0 = fmaf(kr[i], s[i], ks0), ks1 = fmaf(kr[i + 1], s[i + 1], ks1);
      }
      float ks = ks0 + ks1;
#pragma unroll
      for (int o = lanes_per_col >> 1; o > 0; o >>= 1) ks += __shfl_xor_sync(0xffffffffu, ks, o);
      const float u = sb[j] * (sv[j * cols + tid / lanes_per_col] - ks);
      float qs0 = 0.f, qs1 = 0.f;
#pragma unroll
      for (int i = 0; i < PER; i += 2) {
        s[i] = fmaf(kr[i], u, s[i]), s[i + 1] = fmaf(kr[i + 1], u, s[i + 1]);
        qs0 = fmaf(qj[i * lanes_per_col], s[i], qs0), qs1 = fmaf(qj[(i + 1) * lanes_per_col], s[i + 1], qs1);
      }
      float qs = qs0 + qs1;
#pragma unroll
      for (int o = lanes_per_col >> 1; o > 0; o >>= 1) qs += __shfl_xor_sync(0xffffffffu, qs, o);
      if (live && part == 0) out[(static_cast<int64_t>(start) + t0 + j) * heads * dv + head * dv + col] = qs;
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int r = i * lanes_per_col + part;
    if (live && r < dk) s_base[static_cast<int64_t>(r) * dv + col] = s[i];
  }
}

// out[t, h, :] = o / rms(o) * w * sigmoid(gate[t, h, :]), or silu of the gate; one warp per (token, head).
template <typename T, bool SILU>
__global__ void delta_output_kernel(const float* o, const float* __restrict__ weight, const T* gate, int gate_ld, int rows,
                                    int heads, int dv, float eps, T* out) {
  wait_for_predecessor();
  let_successor_start();
  const int lane = threadIdx.x & 31;
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= rows * heads) return;
  const int t = item / heads, h = item % heads;
  const float* src = o + static_cast<int64_t>(item) * dv;
  float ss = 0.f;
  for (int i = lane; i < dv; i += 32) ss = fmaf(src[i], src[i], ss);
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / static_cast<float>(dv) + eps);
  const T* g = gate + static_cast<int64_t>(t) * gate_ld + h * dv;
  T* dst = out + static_cast<int64_t>(item) * dv;
  for (int i = lane; i < dv; i += 32) {
    const float x = to_f32<T>(g[i]);
    dst[i] = from_f32<T>(src[i] * inv * weight[i] * (SILU ? x * sigmoid_f(x) : sigmoid_f(x)));
  }
}

// The same with four numbers a thread: 2^n lanes hold one (token, head), dv = 4 x 2^n up to 128.
template <typename T, bool SILU>
__global__ void __launch_bounds__(256)
delta_output_wide_kernel(const float* o, const float* __restrict__ weight, const T* gate, int gate_ld, int rows, int heads, int dv, float eps, T* out) {
  wait_for_predecessor();
  let_successor_start();
  const int lanes = dv / 4;
  const int64_t quad = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool live = quad < static_cast<int64_t>(rows) * heads * lanes;
  const int64_t item = live ? quad / lanes : 0;
  const int i = static_cast<int>(quad % lanes) * 4, h = static_cast<int>(item % heads);
  const float4 x = *reinterpret_cast<const float4*>(o + item * dv + i);
  const float4 g = load4<T>(gate + item / heads * gate_ld + h * dv + i), w = *reinterpret_cast<const float4*>(weight + i);
  float ss = square_sum(x, 0.f);
  for (int step = lanes >> 1; step > 0; step >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, step);
  const float inv = 1.f / sqrtf(ss / static_cast<float>(dv) + eps);
  const auto gated = [](float z) { return SILU ? silu_f(z) : sigmoid_quick(z); };
  if (live)
    store4<T>(out + item * dv + i, make_float4(x.x * inv * w.x * gated(g.x), x.y * inv * w.y * gated(g.y), x.z * inv * w.z * gated(g.z), x.w * inv * w.w * gated(g.w)));
}

}  // namespace

B200_API int b200_delta_prepare(const void* proj, int ld, const void* decay_in, int decay_ld, const float* taps_w, int taps,
                                void* conv_state, const float* a_log, const float* dt_bias, const int* token_seq,
                                const int* seq_q_start, const int* seq_q_len, const int* seq_slot, int tokens, int seqs,
                                int heads, int kv_heads, int dk, int dv, float* q_out, float* k_out, float* v_out,
                                float* beta_out, float* decay_out, float* kq_out, int dtype, cudaStream_t stream) {
  if (tokens == 0) return 0;
  B200_REQUIRE(tokens > 0 && seqs > 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dk > 0 && dv > 0 && taps >= 1,
               "delta_prepare: bad sizes");
  const int channels = 2 * kv_heads * dk + heads * dv;
  const size_t smem = sizeof(float) * channels;
  B200_REQUIRE(smem <= 200 * 1024, "delta_prepare: %d convolved channels do not fit shared memory", channels);
  const int threads = 256;
  const int update_blocks = (channels + threads - 1) / threads;  // a thread per channel: the slots' update is a tail of its own
  // The wide form from half a block an SM on, with rows, taps and results on 16-byte (bfloat16 rows: 8-byte) boundaries.
  const auto on = [](const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; };
  const int in_bytes = dtype == DTYPE_F32 ? 16 : 8;
  const bool wide = taps == kWideTaps && tokens >= kWideTokens * b200_sm_count_host() / 2 && ld % 4 == 0 && dk % 4 == 0 && dv % 4 == 0 &&
                    on(proj, in_bytes) && on(conv_state, in_bytes) && on(taps_w, 16) && on(q_out, 16) && on(k_out, 16) && on(v_out, 16) &&
                    (kq_out != nullptr || (decay_ld % 4 == 0 && on(decay_in, in_bytes) && on(dt_bias, 16) && on(decay_out, 16)));
  auto launch_wide = [&](auto kernel, auto* typed) {
    using T = typename std::remove_pointer<decltype(typed)>::type;
    const auto pieces = [](int64_t n) { return static_cast<int>((n + kWideChannels - 1) / kWideChannels); };
    const WidePrepare p = {ld, decay_ld, tokens, heads, kv_heads, dk, dv, taps_w, a_log, dt_bias, token_seq, seq_q_start, seq_slot, q_out, k_out, v_out, beta_out,
                           decay_out, kq_out, pieces(static_cast<int64_t>(heads) * dv), kq_out != nullptr ? 0 : pieces(static_cast<int64_t>(heads) * dk)};
    const int64_t groups = (tokens + kWideTokens - 1) / kWideTokens, pieces_a_group = p.v_pieces + p.decay_pieces + 1;
    const int64_t blocks = dk > 2 * kWideChannels ? groups * (kv_heads + (pieces_a_group + 3) / 4) : (groups * (kv_heads + pieces_a_group) + 3) / 4;
    launch_kernel(kernel, dim3(static_cast<unsigned>(blocks)), dim3(128), 0, stream, p, typed, static_cast<const T*>(decay_in), static_cast<const T*>(conv_state));
  };
  if (wide && (dtype == DTYPE_F32 || dtype == DTYPE_BF16)) {
    const auto form = [&](auto one, auto two, auto any) { return dk <= kWideChannels ? one : (dk <= 2 * kWideChannels ? two : any); };
    if (dtype == DTYPE_F32)
      launch_wide(form(delta_prepare_wide_kernel<float, 1>, delta_prepare_wide_kernel<float, 2>, delta_prepare_wide_kernel<float, 0>), static_cast<const float*>(proj));
    else
      launch_wide(form(delta_prepare_wide_kernel<__nv_bfloat16, 1>, delta_prepare_wide_kernel<__nv_bfloat16, 2>, delta_prepare_wide_kernel<__nv_bfloat16, 0>),
                  static_cast<const __nv_bfloat16*>(proj));
    if (int status = b200_check_launch("delta_prepare")) return status;
    if (dtype == DTYPE_F32)
      launch_kernel(conv_state_update_kernel<float>, dim3(seqs, update_blocks), dim3(threads), 0, stream, static_cast<const float*>(proj), ld, channels, taps,
                    seq_q_start, seq_q_len, seq_slot, static_cast<float*>(conv_state));
    else
      launch_kernel(conv_state_update_kernel<__nv_bfloat16>, dim3(seqs, update_blocks), dim3(threads), 0, stream, static_cast<const __nv_bfloat16*>(proj), ld,
                    channels, taps, seq_q_start, seq_q_len, seq_slot, static_cast<__nv_bfloat16*>(conv_state));
    return b200_check_launch("conv_state_update");
  }
  if (dtype == DTYPE_F32) {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(delta_prepare_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    launch_kernel(delta_prepare_kernel<float>, dim3(tokens), dim3(threads), smem, stream, static_cast<const float*>(proj), ld,
                  static_cast<const float*>(decay_in), decay_ld, taps_w, taps, static_cast<const float*>(conv_state), a_log,
                  dt_bias, token_seq, seq_q_start, seq_slot, heads, kv_heads, dk, dv, q_out, k_out, v_out, beta_out, decay_out, kq_out);
    if (int status = b200_check_launch("delta_prepare")) return status;
    launch_kernel(conv_state_update_kernel<float>, dim3(seqs, update_blocks), dim3(threads), 0, stream, static_cast<const float*>(proj), ld,
                  channels, taps, seq_q_start, seq_q_len, seq_slot, static_cast<float*>(conv_state));
  } else if (dtype == DTYPE_BF16) {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(delta_prepare_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem));
    launch_kernel(delta_prepare_kernel<__nv_bfloat16>, dim3(tokens), dim3(threads), smem, stream,
                  static_cast<const __nv_bfloat16*>(proj), ld, static_cast<const __nv_bfloat16*>(decay_in), decay_ld, taps_w,
                  taps, static_cast<const __nv_bfloat16*>(conv_state), a_log, dt_bias, token_seq, seq_q_start, seq_slot, heads,
                  kv_heads, dk, dv, q_out, k_out, v_out, beta_out, decay_out, kq_out);
    if (int status = b200_check_launch("delta_prepare")) return status;
    launch_kernel(conv_state_update_kernel<__nv_bfloat16>, dim3(seqs, update_blocks), dim3(threads), 0, stream,
                  static_cast<const __nv_bfloat16*>(proj), ld, channels, taps, seq_q_start, seq_q_len, seq_slot,
                  static_cast<__nv_bfloat16*>(conv_state));
  } else {
    return b200_fail("delta_prepare: unknown dtype %d", dtype);
  }
  return b200_check_launch("conv_state_update");
}

B200_API int b200_delta_recurrence(const float* q, const float* k, const float* v, const float* beta, const float* decay,
                                   const int* seq_q_start, const int* seq_q_len, const int* seq_slot, int seqs, int heads,
                                   int kv_heads, int dk, int dv, float* state, float* out, cudaStream_t stream) {
  if (seqs == 0) return 0;
  B200_REQUIRE(seqs > 0 && heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0 && dk > 0 && dv > 0,
               "delta_recurrence: bad sizes");
  B200_REQUIRE(dk <= 1024, "delta_recurrence: %d key channels per head, at most 1024", dk);
  // Lanes per column: enough that a lane holds at most 8 rows (up to 32 rows when even a whole warp
  // per column leaves more).
  int lanes = 1;
  while ((dk + lanes - 1) / lanes > 8 && lanes < 32) lanes *= 2;
  const int rows = (dk + lanes - 1) / lanes;
  B200_REQUIRE(rows <= 32, "delta_recurrence: %d key channels per head, at most 1024", dk);
  const int per = rows <= 8 ? 8 : (rows <= 16 ? 16 : 32);
  const int cols = kRecurrenceThreads / lanes;
  const dim3 grid(seqs, heads, (dv + cols - 1) / cols);
  B200_REQUIRE(grid.z <= 65535, "delta_recurrence: too many columns");
  const size_t smem = sizeof(float) * 2 * (kStage * (3 * per * lanes + cols) + kStage);
  const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  // 16-byte copies when every staged row starts on a 16-byte boundary.
  const int vec = dk % 4 == 0 && dv % 4 == 0 && aligned(q) && aligned(k) && aligned(v) && aligned(decay) ? 1 : 0;
  B200_REQUIRE(smem <= 200 * 1024, "delta_recurrence: the staged tokens do not fit shared memory");
  auto launch = [&](auto kernel) {
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    launch_kernel(kernel, grid, dim3(kRecurrenceThreads), smem, stream, q, k, v, beta, decay, seq_q_start, seq_q_len, seq_slot,
                  heads, kv_heads, dk, dv, vec, state, out);
  };
  if (per == 32) launch(delta_recurrence_kernel<32, 32>);
  else if (per == 16) launch(delta_recurrence_kernel<16, 32>);
  else if (lanes == 32) launch(delta_recurrence_kernel<8, 32>);
  else if (lanes == 16) launch(delta_recurrence_kernel<8, 16>);
  else if (lanes == 8) launch(delta_recurrence_kernel<8, 8>);
  else if (lanes == 4) launch(delta_recurrence_kernel<8, 4>);
  else if (lanes == 2) launch(delta_recurrence_kernel<8, 2>);
  else launch(delta_recurrence_kernel<8, 1>);
  return b200_check_launch("delta_recurrence");
}

B200_API int b200_delta_output(const float* o, const float* weight, const void* gate, int gate_ld, int rows, int heads, int dv,
                               float eps, int silu, void* out, int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200_REQUIRE(rows > 0 && heads > 0 && dv > 0, "delta_output: bad sizes");
  const int threads = 128;
  const int64_t items = static_cast<int64_t>(rows) * heads;
  const unsigned blocks = static_cast<unsigned>((items + 3) / 4);
  const int lanes = dv / 4, in_bytes = dtype == DTYPE_F32 ? 16 : 8;
  const auto on = [](const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; };
  if (dv % 4 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && gate_ld % 4 == 0 && on(o, 16) && on(weight, 16) && on(gate, in_bytes) && on(out, in_bytes) &&
      (dtype == DTYPE_F32 || dtype == DTYPE_BF16)) {
    const dim3 grid(static_cast<unsigned>((items * lanes + 255) / 256));
    if (dtype == DTYPE_F32)
      launch_kernel(silu ? delta_output_wide_kernel<float, true> : delta_output_wide_kernel<float, false>, grid, dim3(256), 0, stream, o, weight,
                    static_cast<const float*>(gate), gate_ld, rows, heads, dv, eps, static_cast<float*>(out));
    else
      launch_kernel(silu ? delta_output_wide_kernel<__nv_bfloat16, true> : delta_output_wide_kernel<__nv_bfloat16, false>, grid, dim3(256), 0, stream, o, weight,
                    static_cast<const __nv_bfloat16*>(gate), gate_ld, rows, heads, dv, eps, static_cast<__nv_bfloat16*>(out));
    return b200_check_launch("delta_output");
  }
  if (dtype == DTYPE_F32) {
    launch_kernel(silu ? delta_output_kernel<float, true> : delta_output_kernel<float, false>, dim3(blocks), dim3(threads), 0, stream, o, weight,
                  static_cast<const float*>(gate), gate_ld, rows, heads, dv, eps, static_cast<float*>(out));
  } else if (dtype == DTYPE_BF16) {
    launch_kernel(silu ? delta_output_kernel<__nv_bfloat16, true> : delta_output_kernel<__nv_bfloat16, false>, dim3(blocks), dim3(threads), 0, stream,
                  o, weight, static_cast<const __nv_bfloat16*>(gate), gate_ld, rows, heads, dv, eps, static_cast<__nv_bfloat16*>(out));
  } else {
    return b200_fail("delta_output: unknown dtype %d", dtype);
  }
  return b200_check_launch("delta_output");
}
