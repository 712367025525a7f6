// The gated delta rule: a linear-attention mixer whose per-head state is a matrix S [dim, vdim] that forgets by a
// per-token decay and is corrected towards each new value.
//
// The step's fused input projection is [T, 2 G dim + 2 H vdim] in the compute type: queries and keys of G groups,
// values of H heads, then the output gate (H vdim).  A second small product gives, in float32, the pre-activations
// of the write strength and of the decay, [T, 2 H].
//
// delta_prepare_kernel (a block per token and query group, key group or value head): every query, key and value channel goes through a short causal
// convolution over its last K inputs (weights [channels, K], the last column the current token's, no bias, zeros
// before the start of the sequence; inputs from before the portion are read from the request's slot) and SiLU.
// Queries and keys are made unit vectors per group, x / sqrt(sum x^2 + 1e-6), queries also times dim^-1/2.  Per
// head, beta = sigmoid(b) and decay = exp(-exp(A_log) softplus(a + dt_bias)).  Everything after the projection is
// float32 and leaves the kernel as float32.
//
// delta_rule_kernel: per request and head, token by token,
//     S <- decay S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q,
// so the read-out sees the current token's write (computed as decay (S_old^T q) + (q.k) u, which is the same).  The columns of S (one per value channel) never meet: R lanes of
// a warp hold one column between them (dim / R numbers each, in registers), so a warp carries 32 / R columns, and
// the two dot products of a token are finished by a butterfly among the R lanes.  The order of every sum depends on
// R and dim only, never on the batch.  What a run of tokens brings is staged in shared memory for the whole block, one
// run ahead of the arithmetic.  The state is read from the request's slot at the portion's start and written back at its end; one block
// per request also brings the slot's convolution inputs up to date (the last K-1 rows of the projection, or what
// was there before, moved up, when the portion is shorter).
//
// Portions of eight tokens and more of bfloat16 projections (keys of up to 128 numbers in fours) go through the kernels of
// delta_chunks.cu instead, which need neither the single steps nor:
//
// delta_cross_kernel (a warp per token and head): q.k, and k.k' and q.k' with the key of the token before.
//
// channel_delta_rule_kernel: the same rule with a decay per head and key channel, g [T, H, dim], which multiplies the rows
// of S.  delta_prepare_kernel then takes the write strength's pre-activation from the projection itself (the row is
// [q | k | v | ...], ``ld`` numbers to the next), and delta_cross_kernel gives (k g).k' and (q g).k' instead of k.k' and q.k'.
//
// delta_finish_kernel (a warp per token and head): o / sqrt(mean(o^2) + eps) * gain[vdim] * silu(gate), rounded to
// the compute type for the output projection.
//
// Slot layout (float32): [K-1, C] convolution inputs, oldest first (C = 2 G dim + H vdim), then S as [H, dim, vdim].
#include "delta_common.cuh"

namespace {

using namespace delta;

// A block per (token, unit); a unit is one query group, one key group (dim channels each) or one value head (vdim).
template <typename T>
__global__ void __launch_bounds__(128)
delta_prepare_kernel(const T* __restrict__ proj, const float* __restrict__ ba, const float* __restrict__ taps,
                     const float* __restrict__ a_log, const float* __restrict__ dt_bias, const float* __restrict__ state,
                     const int32_t* __restrict__ positions, const int32_t* __restrict__ token_item,
                     const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots, float* __restrict__ qkv,
                     float* __restrict__ bd, int G, int H, int dim, int vdim, int K, int num_slots, size_t slot_floats,
                     int T_tokens, int tokens_per_block, long long P, int beta_at) {
  extern __shared__ float row[];  // the unit's convolved, activated channels
  __shared__ float scratch[4];
  const int unit = blockIdx.y;
  const int C = 2 * G * dim + H * vdim;  // (P: numbers from one row of the projection to the next)
  const int c0 = unit < 2 * G ? unit * dim : 2 * G * dim + (unit - 2 * G) * vdim;
  const int len = unit < 2 * G ? dim : vdim;
  pdl_wait();
  for (int t = blockIdx.x * tokens_per_block; t < min(T_tokens, (blockIdx.x + 1) * tokens_per_block); ++t) {
  __syncthreads();  // the last token's row and sums have been read
  const int item = token_item[t];
  const int p = positions[t], p0 = positions[item_start[item]];
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  const float* tail = state + (size_t)slot * slot_floats;
  float ss = 0.f;
  for (int i = threadIdx.x; i < len; i += blockDim.x) {
    const int c = c0 + i;
    float x[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {  // the inputs under the taps, asked for together
      if (k >= K) break;
      const int src = p - (K - 1) + k;
      x[k] = 0.f;
      if (src >= p0) x[k] = to_float<T>(proj[(size_t)(t - (p - src)) * P + c]);
      else if (src >= 0) x[k] = tail[(size_t)(src - p0 + K - 1) * C + c];
    }
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K) break;
      acc = fmaf(taps[(size_t)c * K + k], x[k], acc);
    }
    const float v = siluf_(acc);
    row[i] = v;
    ss = fmaf(v, v, ss);
  }
  float factor = 1.f;
  if (unit < 2 * G) {  // unit vectors; queries also times dim^-1/2
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = ss;
    __syncthreads();
    const float total = scratch[0] + scratch[1] + scratch[2] + scratch[3];
    factor = unit_factor(total, unit < G ? dim : 1);
  }
  float* out = qkv + (size_t)t * C + c0;
  for (int i = threadIdx.x; i < len; i += blockDim.x) out[i] = row[i] * factor;  // a thread reads back what it wrote
  if (unit == 0) {
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
      if (!ba) {  // write strengths only, from the projection; the decays are somebody else's
        bd[(size_t)t * BD * H + h] = sigmoidf_(to_float<T>(proj[(size_t)t * P + beta_at + h]));
        continue;
      }
      bd[(size_t)t * BD * H + h] = sigmoidf_(ba[(size_t)t * 2 * H + h]);
      bd[(size_t)t * BD * H + H + h] = expf(-expf(a_log[h]) * softplusf_(ba[(size_t)t * 2 * H + H + h] + dt_bias[h]));
    }
  }
  }
  // At the end, not at the start: the recurrence behind this kernel has few blocks that live long.  Let in while this
  // kernel's blocks fill the SMs, they crowd onto the few SMs with room and stay there, several to a scheduler; a
  // 2,048-token portion then took 1.4 ms a layer instead of 0.7.
  pdl_trigger();
}

// The same for long steps: a block takes eight tokens and a unit, a thread a channel (two for units of up to 256), holds the
// inputs of the run in registers (each is read once, not once a tap) and the eight tokens' sums of squares are finished
// together.  K <= RUN_TAPS; rows before a portion come from the slot as above.
constexpr int RUN_TOKENS = 8, RUN_TAPS = 4;

template <typename T, int CH>
__global__ void __launch_bounds__(128)
delta_prepare_run_kernel(const T* __restrict__ proj, const float* __restrict__ ba, const float* __restrict__ taps,
                         const float* __restrict__ a_log, const float* __restrict__ dt_bias, const float* __restrict__ state,
                         const int32_t* __restrict__ positions, const int32_t* __restrict__ token_item,
                         const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots, float* __restrict__ qkv,
                         float* __restrict__ bd, int G, int H, int dim, int vdim, int K, int num_slots, size_t slot_floats,
                         int T_tokens, long long P, int beta_at) {
  __shared__ float scratch[RUN_TOKENS][4];
  const int unit = blockIdx.y;
  const int C = 2 * G * dim + H * vdim;
  const int c0 = unit < 2 * G ? unit * dim : 2 * G * dim + (unit - 2 * G) * vdim;
  const int len = unit < 2 * G ? dim : vdim;
  const int t0 = blockIdx.x * RUN_TOKENS, n = min(RUN_TOKENS, T_tokens - t0);
  pdl_wait();
  // per token of the run: how many of the inputs in front of it lie in its own portion (at most RUN_TAPS - 1), its position
  // capped alike, and the slot that holds the others
  int own[RUN_TOKENS], pos[RUN_TOKENS], slot[RUN_TOKENS];
#pragma unroll
  for (int i = 0; i < RUN_TOKENS; ++i) {
    if (i >= n) break;
    const int item = token_item[t0 + i];
    own[i] = min(t0 + i - item_start[item], RUN_TAPS - 1);
    pos[i] = min(positions[t0 + i], RUN_TAPS - 1);
    slot[i] = min(max(slots[item], 0), num_slots - 1);
  }
  float y[CH][RUN_TOKENS];
#pragma unroll
  for (int u = 0; u < CH; ++u) {
    const int i0 = threadIdx.x + u * 128;
    const int c = c0 + i0;
    if (i0 >= len) {
#pragma unroll
      for (int i = 0; i < RUN_TOKENS; ++i) y[u][i] = 0.f;
      continue;
    }
    float x[RUN_TOKENS + RUN_TAPS - 1], w[RUN_TAPS];  // x[i + RUN_TAPS - 1]: token t0 + i's input
#pragma unroll
    for (int i = 0; i < RUN_TOKENS + RUN_TAPS - 1; ++i) {
      const int t = t0 + i - (RUN_TAPS - 1);
      x[i] = (t >= 0 && t < T_tokens) ? to_float<T>(proj[(size_t)t * P + c]) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < RUN_TAPS; ++k) w[k] = k < K ? taps[(size_t)c * K + K - 1 - k] : 0.f;  // w[k]: the input k positions back
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i) {
      float acc = 0.f;
      if (i < n) {
#pragma unroll
        for (int k = RUN_TAPS - 1; k >= 0; --k) {  // oldest first, as in delta_prepare_kernel
          if (k >= K) continue;
          float v = x[i + RUN_TAPS - 1 - k];
          if (k > own[i])  // before the portion: the slot's row of that position, zero before the sequence
            v = k <= pos[i] ? state[(size_t)slot[i] * slot_floats + (size_t)(K - 1 - (k - own[i])) * C + c] : 0.f;
          acc = fmaf(w[k], v, acc);
        }
      }
      y[u][i] = siluf_(acc);
    }
  }
  float factor[RUN_TOKENS];
#pragma unroll
  for (int i = 0; i < RUN_TOKENS; ++i) factor[i] = 1.f;
  if (unit < 2 * G) {
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i) {
      float ss = 0.f;
#pragma unroll
      for (int u = 0; u < CH; ++u) ss = fmaf(y[u][i], y[u][i], ss);
      ss = warp_sum(ss);
      if ((threadIdx.x & 31) == 0) scratch[i][threadIdx.x >> 5] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i)
      factor[i] = unit_factor(scratch[i][0] + scratch[i][1] + scratch[i][2] + scratch[i][3], unit < G ? dim : 1);
  }
#pragma unroll
  for (int u = 0; u < CH; ++u) {
    const int i0 = threadIdx.x + u * 128;
    if (i0 < len) {
#pragma unroll
      for (int i = 0; i < RUN_TOKENS; ++i)
        if (i < n) qkv[(size_t)(t0 + i) * C + c0 + i0] = y[u][i] * factor[i];
    }
  }
  if (unit == 0) {
    for (int j = threadIdx.x; j < n * H; j += blockDim.x) {
      const int t = t0 + j / H, h = j % H;
      if (!ba) {
        bd[(size_t)t * BD * H + h] = sigmoidf_(to_float<T>(proj[(size_t)t * P + beta_at + h]));
        continue;
      }
      bd[(size_t)t * BD * H + h] = sigmoidf_(ba[(size_t)t * 2 * H + h]);
      bd[(size_t)t * BD * H + H + h] = expf(-expf(a_log[h]) * softplusf_(ba[(size_t)t * 2 * H + H + h] + dt_bias[h]));
    }
  }
  pdl_trigger();  // at the end, as in delta_prepare_kernel
}

// The same again where units are of up to 128 channels in fours and everything lies on the boundaries of wide accesses (the usual
// sizes): a warp takes a unit and a run of eight tokens, four neighbouring channels a lane, so that the inputs come in 8 (16) bytes a
// lane, the results leave in 16 and the sums of squares need no barrier.  What a token's place in its portion decides is asked for once
// a warp, and only a run at a portion's start looks at the slot.  Bound by what its warps issue (the taps and the SiLU of every
// channel).  2,000 tokens of 16 heads over 8 groups of 128: 21 us (28 with a division for every SiLU and each sum of squares by itself), with a channel a thread 47.
template <typename T>
__device__ __forceinline__ void load_four(const T* p, float (&v)[4]) {
  if constexpr (sizeof(T) == 2) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
}

constexpr int WIDE_WARPS = 4;

template <typename T>
__global__ void __launch_bounds__(WIDE_WARPS * 32)
delta_prepare_wide_kernel(const T* __restrict__ proj, const float* __restrict__ ba, const float* __restrict__ taps,
                          const float* __restrict__ a_log, const float* __restrict__ dt_bias, const float* __restrict__ state,
                          const int32_t* __restrict__ positions, const int32_t* __restrict__ token_item,
                          const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots, float* __restrict__ qkv,
                          float* __restrict__ bd, int G, int H, int dim, int vdim, int K, int num_slots, size_t slot_floats,
                          int T_tokens, long long P, int beta_at) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = blockIdx.y * WIDE_WARPS + warp;
  const int C = 2 * G * dim + H * vdim;
  const int t0 = blockIdx.x * RUN_TOKENS, n = min(RUN_TOKENS, T_tokens - t0);
  const bool there = unit < 2 * G + H;
  const int c0 = unit < 2 * G ? unit * dim : 2 * G * dim + (unit - 2 * G) * vdim;
  const int len = unit < 2 * G ? dim : vdim, c = c0 + 4 * lane;
  const bool mine = there && 4 * lane < len;
  float w[4][RUN_TAPS];  // w[.][k]: the weight of the input k positions back
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (K == RUN_TAPS) {
      const float4 v = mine ? *reinterpret_cast<const float4*>(taps + (size_t)(c + j) * RUN_TAPS) : make_float4(0.f, 0.f, 0.f, 0.f);
      w[j][3] = v.x;
      w[j][2] = v.y;
      w[j][1] = v.z;
      w[j][0] = v.w;
    } else {
#pragma unroll
      for (int k = 0; k < RUN_TAPS; ++k) w[j][k] = mine && k < K ? taps[(size_t)(c + j) * K + K - 1 - k] : 0.f;
    }
  }
  pdl_wait();
  // lane i: token i's item, how many inputs in front of it lie in its own portion (at most RUN_TAPS - 1), its position, capped
  int own = RUN_TAPS - 1, pos = RUN_TAPS - 1, slot = 0;
  if (lane < n) {
    const int item = token_item[t0 + lane];
    own = min(t0 + lane - item_start[item], RUN_TAPS - 1);
    pos = min(positions[t0 + lane], RUN_TAPS - 1);
    slot = min(max(slots[item], 0), num_slots - 1);
  }
  const bool inside = __all_sync(0xffffffffu, own == RUN_TAPS - 1);
  float x[RUN_TOKENS + RUN_TAPS - 1][4];  // x[i + RUN_TAPS - 1]: token t0 + i's inputs
#pragma unroll
  for (int i = 0; i < RUN_TOKENS + RUN_TAPS - 1; ++i) {
    const int t = t0 + i - (RUN_TAPS - 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) x[i][j] = 0.f;
    if (mine && t >= 0 && t < T_tokens) load_four<T>(proj + (size_t)t * P + c, x[i]);
  }
  float y[RUN_TOKENS][4];
  if (inside && K == RUN_TAPS) {  // most runs: nothing to ask about
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float acc = 0.f;
#pragma unroll
        for (int k = RUN_TAPS - 1; k >= 0; --k) acc = fmaf(w[j][k], x[i + RUN_TAPS - 1 - k][j], acc);
        y[i][j] = acc;  // (zero where there is no channel)
      }
  } else {
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i) {
      const int own_i = __shfl_sync(0xffffffffu, own, i), pos_i = __shfl_sync(0xffffffffu, pos, i), slot_i = __shfl_sync(0xffffffffu, slot, i);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float acc = 0.f;
#pragma unroll
        for (int k = RUN_TAPS - 1; k >= 0; --k) {  // oldest first, as in delta_prepare_kernel
          if (k >= K) continue;
          float v = x[i + RUN_TAPS - 1 - k][j];
          if (k > own_i)  // before the portion: the slot's row of that position, zero before the sequence
            v = mine && k <= pos_i ? state[(size_t)slot_i * slot_floats + (size_t)(K - 1 - (k - own_i)) * C + c + j] : 0.f;
          acc = fmaf(w[j][k], v, acc);
        }
        y[i][j] = mine ? acc : 0.f;
      }
    }
  }
  silu_all(y);
  if (there && unit < 2 * G) {  // unit vectors; queries also times dim^-1/2
    float ss[RUN_TOKENS];
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i) {
      ss[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) ss[i] = fmaf(y[i][j], y[i][j], ss[i]);
    }
    // all tokens' sums over the warp at a time: four lanes end up with each, and make its factor
    static_assert(RUN_TOKENS == 8, "a token per four lanes");
#pragma unroll
    for (int m = 4, off = 16; m > 0; m >>= 1, off >>= 1) {
      const bool up = lane & off;
#pragma unroll
      for (int e = 0; e < m; ++e) ss[e] = (up ? ss[e + m] : ss[e]) + __shfl_xor_sync(0xffffffffu, up ? ss[e] : ss[e + m], off);
    }
    ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 2);
    ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);
    const float factor = unit_factor(ss[0], unit < G ? dim : 1);
#pragma unroll
    for (int i = 0; i < RUN_TOKENS; ++i) {
      const float f = __shfl_sync(0xffffffffu, factor, 4 * i);
#pragma unroll
      for (int j = 0; j < 4; ++j) y[i][j] *= f;
    }
  }
#pragma unroll
  for (int i = 0; i < RUN_TOKENS; ++i)
    if (mine && i < n) *reinterpret_cast<float4*>(qkv + (size_t)(t0 + i) * C + c) = make_float4(y[i][0], y[i][1], y[i][2], y[i][3]);
  if (blockIdx.y == 0) {
    for (int j = threadIdx.x; j < n * H; j += blockDim.x) {
      const int t = t0 + j / H, h = j % H;
      if (!ba) {
        bd[(size_t)t * BD * H + h] = sigmoidf_(to_float<T>(proj[(size_t)t * P + beta_at + h]));
        continue;
      }
      bd[(size_t)t * BD * H + h] = sigmoidf_(ba[(size_t)t * 2 * H + h]);
      bd[(size_t)t * BD * H + H + h] = expf(-expf(a_log[h]) * softplusf_(ba[(size_t)t * 2 * H + H + h] + dt_bias[h]));
    }
  }
  pdl_trigger();  // at the end, as in delta_prepare_kernel
}

// A warp per (token, head): the three state-free dot products of the unit vectors delta_prepare_kernel left; with ``decay``
// (float32 [T, H, dim]) the two with the token before carry it, sum_d (k g)_d k'_d and sum_d (q g)_d k'_d.
__global__ void __launch_bounds__(128)
delta_cross_kernel(const float* __restrict__ qkv, const int32_t* __restrict__ token_item, const int32_t* __restrict__ item_start,
                   float* __restrict__ bd, long long units, int G, int H, int dim, int vdim, const float* __restrict__ decay) {
  pdl_wait();  // (no early trigger: the recurrence comes next, see the end of delta_prepare_kernel)
  const long long unit = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (unit >= units) return;
  const long long t = unit / H;
  const int h = (int)(unit - t * H), g = h / (H / G);
  const int C = 2 * G * dim + H * vdim;
  const float* q = qkv + (size_t)t * C + (size_t)g * dim;
  const float* k = q + (size_t)G * dim;
  const bool first = t == item_start[token_item[t]];  // no token before it in this step's portion
  const float* kp = first ? k : k - C;
  float qk = 0.f, kk = 0.f, qkp = 0.f;
  for (int d = lane; d < dim; d += 32) {
    const float qv = q[d], kv = k[d], pv = kp[d] * (decay ? decay[(size_t)unit * dim + d] : 1.f);
    qk = fmaf(qv, kv, qk);
    kk = fmaf(kv, pv, kk);
    qkp = fmaf(qv, pv, qkp);
  }
  qk = warp_sum(qk); kk = warp_sum(kk); qkp = warp_sum(qkp);
  if (lane == 0) {
    float* out = bd + (size_t)t * BD * H + h;
    out[2 * H] = qk;
    out[3 * H] = first ? 0.f : kk;
    out[4 * H] = first ? 0.f : qkp;
  }
}

constexpr int RULE_WARPS = 4;

// PER: numbers of a column one lane holds; R: lanes per column.  R * PER >= dim.  What the tokens of a stage bring
// (queries, keys, the block's value columns, beta, decay) is copied into shared memory one stage ahead of the
// arithmetic (cp.async into the other of two buffers), so the chain from token to token never waits for memory.
//
// The chain itself is kept short: with S the state before the token, the sums k.S and q.S (per column) are finished by
// one butterfly, q.k comes ready-made (it does not depend on the state: delta_cross_kernel), and then
//     u = beta (v - dec k.S),   o = dec q.S + (q.k) u,   S <- dec S + k u^T,
// which is the read-out of the updated state written so that it does not wait for the update.  Tokens go two a round
// (see the loop): one butterfly for both.
template <typename T, int PER, int R>
__global__ void __launch_bounds__(RULE_WARPS * 32)
delta_rule_kernel(const float* __restrict__ qkv, const float* __restrict__ bd, const T* __restrict__ proj,
                  float* __restrict__ state, const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots,
                  float* __restrict__ o, int G, int H, int dim, int vdim, int K, int num_slots, size_t slot_floats,
                  int stage_tokens, int max_tokens) {
  extern __shared__ __align__(16) float staged[];  // [2][stage_tokens][W]
  constexpr int COLS = 32 / R;  // columns a warp holds
  constexpr int RP = R * PER, BC = RULE_WARPS * COLS, W = (2 * RP + BC + BD + 3) / 4 * 4;
  static_assert(RP % 4 == 0, "queries and keys of a token start on 16 bytes");
  const int C = 2 * G * dim + H * vdim, P = C + H * vdim;
  const int h = blockIdx.y, item = blockIdx.z;
  const int g = h / (H / G);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane % R;
  const int col0 = blockIdx.x * BC, in_block = warp * COLS + lane / R;
  const int col = col0 + in_block;
  const bool live = col < vdim;
  // 16-byte copies of queries and keys need their rows on 16 bytes in the [T, C] array
  const bool wide = dim % 4 == 0 && C % 4 == 0 && (((uintptr_t)qkv) & 15) == 0;
  pdl_wait();
  const int t0 = item_start[item], t1 = item_start[item + 1];
  if (t1 - t0 > max_tokens) return;  // a portion of the kernels that work in chunks
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  float* base = state + (size_t)slot * slot_floats;
  float* S = base + (size_t)(K - 1) * C + (size_t)h * dim * vdim;

  auto stage = [&](int ts, float* buf) {  // tokens ts .. ts + stage_tokens - 1 (those before t1) into buf
    const int n = min(stage_tokens, t1 - ts);
    if (wide) {
      constexpr int PIECES = 2 * RP / 4;  // 16-byte pieces of a token's queries and keys
      for (int i = threadIdx.x; i < n * PIECES; i += blockDim.x) {
        const int tok = i / PIECES, e = (i - tok * PIECES) * 4;
        const int which = e / RP, d = e - which * RP;
        float* dst = buf + tok * W + e;
        if (d < dim) copy_async16(dst, qkv + (size_t)(ts + tok) * C + (size_t)which * G * dim + g * dim + d);
        else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int i = threadIdx.x; i < n * 2 * RP; i += blockDim.x) {
        const int tok = i / (2 * RP), e = i - tok * 2 * RP;
        const int which = e / RP, d = e - which * RP;
        if (d < dim) copy_async4(buf + tok * W + e, qkv + (size_t)(ts + tok) * C + (size_t)which * G * dim + g * dim + d);
        else buf[tok * W + e] = 0.f;
      }
    }
    for (int i = threadIdx.x; i < n * (BC + BD); i += blockDim.x) {
      const int tok = i / (BC + BD), e = i - tok * (BC + BD);
      float* dst = buf + tok * W + 2 * RP + e;
      if (e >= BC) copy_async4(dst, bd + (size_t)(ts + tok) * BD * H + (e - BC) * H + h);
      else if (col0 + e < vdim) copy_async4(dst, qkv + (size_t)(ts + tok) * C + 2 * G * dim + h * vdim + col0 + e);
      else *dst = 0.f;
    }
  };

  if (t1 > t0) stage(t0, staged);
  float s[PER];
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int d = r * PER + e;
    s[e] = (live && d < dim) ? S[(size_t)d * vdim + col] : 0.f;
  }
  int which_buf = 0;
  for (int ts = t0; ts < t1; ts += stage_tokens, which_buf ^= 1) {
    const int n = min(stage_tokens, t1 - ts);
    copy_async_wait();
    __syncthreads();  // this stage has landed for everybody, and everybody has left the other buffer
    if (ts + stage_tokens < t1) stage(ts + stage_tokens, staged + (size_t)(which_buf ^ 1) * stage_tokens * W);
    const float* buf = staged + (size_t)which_buf * stage_tokens * W;
    auto load_qk = [&](const float* tokrow, float (&qq)[PER], float (&kk)[PER]) {
      if constexpr (PER % 4 == 0) {
#pragma unroll
        for (int e = 0; e < PER; e += 4) {
          const float4 a = *reinterpret_cast<const float4*>(tokrow + r * PER + e);
          const float4 b4 = *reinterpret_cast<const float4*>(tokrow + RP + r * PER + e);
          qq[e] = a.x; qq[e + 1] = a.y; qq[e + 2] = a.z; qq[e + 3] = a.w;
          kk[e] = b4.x; kk[e + 1] = b4.y; kk[e + 2] = b4.z; kk[e + 3] = b4.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          qq[e] = tokrow[r * PER + e];
          kk[e] = tokrow[RP + r * PER + e];
        }
      }
    };
    int i = 0;
    // Two tokens a round.  With S the state before token a and b = a + 1, the four sums k_a.S, q_a.S, k_b.S, q_b.S are
    // finished by one butterfly; what token b needs of token a's write comes through the state-free products:
    //   u_a = beta_a (v_a - dec_a k_a.S),                              o_a = dec_a q_a.S + (q_a.k_a) u_a,
    //   u_b = beta_b (v_b - dec_b (dec_a k_b.S + (k_a.k_b) u_a)),      o_b = dec_b (dec_a q_b.S + (q_b.k_a) u_a) + (q_b.k_b) u_b,
    //   S <- dec_b dec_a S + k_a (dec_b u_a)^T + k_b u_b^T.
    for (; i + 1 < n; i += 2) {
      const float* ra = buf + i * W;
      const float* rb = ra + W;
      float qa[PER], ka[PER], qb[PER], kb[PER];
      load_qk(ra, qa, ka);
      load_qk(rb, qb, kb);
      const float va = ra[2 * RP + in_block], vb = rb[2 * RP + in_block];
      const float beta_a = ra[2 * RP + BC], dec_a = ra[2 * RP + BC + 1], qk_a = ra[2 * RP + BC + 2];
      const float beta_b = rb[2 * RP + BC], dec_b = rb[2 * RP + BC + 1], qk_b = rb[2 * RP + BC + 2];
      const float kk_ab = rb[2 * RP + BC + 3], qk_ba = rb[2 * RP + BC + 4];
      float kas = 0.f, qas = 0.f, kbs = 0.f, qbs = 0.f;
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        kas = fmaf(ka[e], s[e], kas);
        qas = fmaf(qa[e], s[e], qas);
        kbs = fmaf(kb[e], s[e], kbs);
        qbs = fmaf(qb[e], s[e], qbs);
      }
#pragma unroll
      for (int off = 1; off < R; off <<= 1) {
        kas += __shfl_xor_sync(0xffffffffu, kas, off);
        qas += __shfl_xor_sync(0xffffffffu, qas, off);
        kbs += __shfl_xor_sync(0xffffffffu, kbs, off);
        qbs += __shfl_xor_sync(0xffffffffu, qbs, off);
      }
      const float ua = beta_a * (va - dec_a * kas);
      const float ub = beta_b * (vb - dec_b * fmaf(kk_ab, ua, dec_a * kbs));
      const float dd = dec_b * dec_a, wa = dec_b * ua;
#pragma unroll
      for (int e = 0; e < PER; ++e) s[e] = fmaf(kb[e], ub, fmaf(ka[e], wa, dd * s[e]));
      if (live && r == 0) {
        float* orow = o + ((size_t)(ts + i) * H + h) * vdim + col;
        orow[0] = fmaf(qk_a, ua, dec_a * qas);
        orow[(size_t)H * vdim] = fmaf(qk_b, ub, dec_b * fmaf(qk_ba, ua, dec_a * qbs));
      }
    }
    for (; i < n; ++i) {  // a portion's last token when their number is odd (a single decoded token)
      const float* tokrow = buf + i * W;
      float qq[PER], kk[PER];
      load_qk(tokrow, qq, kk);
      const float v = tokrow[2 * RP + in_block];
      const float beta = tokrow[2 * RP + BC], dec = tokrow[2 * RP + BC + 1], qk = tokrow[2 * RP + BC + 2];
      float ks0 = 0.f, ks1 = 0.f, qs0 = 0.f, qs1 = 0.f;
#pragma unroll
      for (int e = 0; e < PER; e += 2) {
        ks0 = fmaf(kk[e], s[e], ks0);
        qs0 = fmaf(qq[e], s[e], qs0);
        if (e + 1 < PER) {
          ks1 = fmaf(kk[e + 1], s[e + 1], ks1);
          qs1 = fmaf(qq[e + 1], s[e + 1], qs1);
        }
      }
      float ksum = ks0 + ks1, qsum = qs0 + qs1;
#pragma unroll
      for (int off = 1; off < R; off <<= 1) {
        ksum += __shfl_xor_sync(0xffffffffu, ksum, off);
        qsum += __shfl_xor_sync(0xffffffffu, qsum, off);
      }
      const float u = beta * (v - dec * ksum);
#pragma unroll
      for (int e = 0; e < PER; ++e) s[e] = fmaf(kk[e], u, dec * s[e]);
      if (live && r == 0) o[((size_t)(ts + i) * H + h) * vdim + col] = fmaf(qk, u, dec * qsum);
    }
  }
  // Only now may the next kernel's blocks come: this kernel has two warps a scheduler and is bound by their chains of
  // dependent instructions, and the next kernel reads what the last token writes anyway.
  pdl_trigger();
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int d = r * PER + e;
    if (live && d < dim) S[(size_t)d * vdim + col] = s[e];
  }
  if (blockIdx.x == 0 && h == 0) keep_conv_inputs<T>(proj, P, base, t0, t1, C, K);
}

// The rule with a decay per key channel.  A lane holds PER rows of a column in runs of four, 4 R apart (so that the lanes'
// 16-byte reads of a token's vectors lie side by side).  Tokens go two a round, as above: with S the state before token a,
//   u_a = beta_a (v_a - (k_a g_a).S),                                  o_a = (q_a g_a).S + (q_a.k_a) u_a,
//   u_b = beta_b (v_b - (k_b g_b g_a).S - ((k_b g_b).k_a) u_a),        o_b = (q_b g_b g_a).S + ((q_b g_b).k_a) u_a + (q_b.k_b) u_b,
//   S <- g_b (g_a S + k_a u_a^T) + k_b u_b^T,
// four sums finished by one butterfly; the products in parentheses without S come from delta_cross_kernel.
template <int PER, int R>
__device__ __forceinline__ int channel_row(int r, int e) {
  return PER % 4 == 0 ? (e >> 2) * (4 * R) + r * 4 + (e & 3) : e * R + r;
}
template <int PER, int R>
__device__ __forceinline__ void channel_vector(const float* __restrict__ v, int r, float (&o)[PER]) {
  if constexpr (PER % 4 == 0) {
#pragma unroll
    for (int e = 0; e < PER; e += 4) {
      const float4 a = *reinterpret_cast<const float4*>(v + channel_row<PER, R>(r, e));
      o[e] = a.x; o[e + 1] = a.y; o[e + 2] = a.z; o[e + 3] = a.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < PER; ++e) o[e] = v[channel_row<PER, R>(r, e)];
  }
}

template <typename T, int PER, int R>
__global__ void __launch_bounds__(RULE_WARPS * 32)
channel_delta_rule_kernel(const float* __restrict__ qkv, const float* __restrict__ bd, const float* __restrict__ decay,
                          const T* __restrict__ proj, long long P, float* __restrict__ state, const int32_t* __restrict__ item_start,
                          const int32_t* __restrict__ slots, float* __restrict__ o, int G, int H, int dim, int vdim, int K,
                          int num_slots, long long slot_floats, int stage_tokens, int max_tokens) {
  extern __shared__ __align__(16) float staged[];  // [2][stage_tokens][W]: q, k, g (RP each, zeros beyond dim), values, bd
  constexpr int COLS = 32 / R, RP = R * PER, BC = RULE_WARPS * COLS, W = (3 * RP + BC + BD + 3) / 4 * 4;
  static_assert(RP % 4 == 0, "a token's vectors start on 16 bytes");
  const int C = 2 * G * dim + H * vdim;
  const int h = blockIdx.y, item = blockIdx.z;
  const int g = h / (H / G);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane % R;
  const int col0 = blockIdx.x * BC, in_block = warp * COLS + lane / R;
  const int col = col0 + in_block;
  const bool live = col < vdim;
  const bool wide = dim % 4 == 0 && C % 4 == 0 && (((uintptr_t)qkv | (uintptr_t)decay) & 15) == 0;
  pdl_wait();
  const int t0 = item_start[item], t1 = item_start[item + 1];
  if (t1 - t0 > max_tokens) return;  // a portion of the kernels that work in chunks
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  float* base = state + (size_t)slot * slot_floats;
  float* S = base + (size_t)(K - 1) * C + (size_t)h * dim * vdim;

  auto stage = [&](int ts, float* buf) {  // tokens ts .. ts + stage_tokens - 1 (those before t1) into buf
    const int n = min(stage_tokens, t1 - ts);
    if (wide) {
      constexpr int PIECES = 3 * RP / 4;
      for (int i = threadIdx.x; i < n * PIECES; i += blockDim.x) {
        const int tok = i / PIECES, e = (i - tok * PIECES) * 4;
        const int which = e / RP, d = e - which * RP;
        float* dst = buf + tok * W + e;
        const float* src = which == 2 ? decay + ((size_t)(ts + tok) * H + h) * dim + d
                                      : qkv + (size_t)(ts + tok) * C + (size_t)which * G * dim + (size_t)g * dim + d;
        if (d < dim) copy_async16(dst, src);
        else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int i = threadIdx.x; i < n * 3 * RP; i += blockDim.x) {
        const int tok = i / (3 * RP), e = i - tok * 3 * RP;
        const int which = e / RP, d = e - which * RP;
        const float* src = which == 2 ? decay + ((size_t)(ts + tok) * H + h) * dim + d
                                      : qkv + (size_t)(ts + tok) * C + (size_t)which * G * dim + (size_t)g * dim + d;
        if (d < dim) copy_async4(buf + tok * W + e, src);
        else buf[tok * W + e] = 0.f;
      }
    }
    for (int i = threadIdx.x; i < n * (BC + BD); i += blockDim.x) {
      const int tok = i / (BC + BD), e = i - tok * (BC + BD);
      float* dst = buf + tok * W + 3 * RP + e;
      if (e >= BC) copy_async4(dst, bd + (size_t)(ts + tok) * BD * H + (e - BC) * H + h);
      else if (col0 + e < vdim) copy_async4(dst, qkv + (size_t)(ts + tok) * C + 2 * (size_t)G * dim + (size_t)h * vdim + col0 + e);
      else *dst = 0.f;
    }
  };

  if (t1 > t0) stage(t0, staged);
  float s[PER];
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int d = channel_row<PER, R>(r, e);
    s[e] = (live && d < dim) ? S[(size_t)d * vdim + col] : 0.f;
  }
  int which_buf = 0;
  for (int ts = t0; ts < t1; ts += stage_tokens, which_buf ^= 1) {
    const int n = min(stage_tokens, t1 - ts);
    copy_async_wait();
    __syncthreads();  // this stage has landed for everybody, and everybody has left the other buffer
    if (ts + stage_tokens < t1) stage(ts + stage_tokens, staged + (size_t)(which_buf ^ 1) * stage_tokens * W);
    const float* buf = staged + (size_t)which_buf * stage_tokens * W;
    int i = 0;
    if constexpr (PER <= 16) {
      for (; i + 1 < n; i += 2) {
        const float* ra = buf + i * W;
        const float* rb = ra + W;
        float ka[PER], ga[PER], kb[PER], gb[PER], q[PER];
        channel_vector<PER, R>(ra + RP, r, ka);
        channel_vector<PER, R>(ra + 2 * RP, r, ga);
        channel_vector<PER, R>(rb + RP, r, kb);
        channel_vector<PER, R>(rb + 2 * RP, r, gb);
        const float va = ra[3 * RP + in_block], vb = rb[3 * RP + in_block];
        const float beta_a = ra[3 * RP + BC], qk_a = ra[3 * RP + BC + 2];
        const float beta_b = rb[3 * RP + BC], qk_b = rb[3 * RP + BC + 2], kk_ab = rb[3 * RP + BC + 3], qk_ba = rb[3 * RP + BC + 4];
        float kas[2] = {}, qas[2] = {}, kbs[2] = {}, qbs[2] = {};
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          s[e] *= ga[e];                       // g_a S, which is all that is needed of S from here on
          ga[e] = gb[e] * s[e];                // g_b g_a S
          kas[e & 1] = fmaf(ka[e], s[e], kas[e & 1]);
          kbs[e & 1] = fmaf(kb[e], ga[e], kbs[e & 1]);
        }
        channel_vector<PER, R>(ra, r, q);
#pragma unroll
        for (int e = 0; e < PER; ++e) qas[e & 1] = fmaf(q[e], s[e], qas[e & 1]);
        channel_vector<PER, R>(rb, r, q);
#pragma unroll
        for (int e = 0; e < PER; ++e) qbs[e & 1] = fmaf(q[e], ga[e], qbs[e & 1]);
        float ks_a = kas[0] + kas[1], ks_b = kbs[0] + kbs[1], qs_a = qas[0] + qas[1], qs_b = qbs[0] + qbs[1];
#pragma unroll
        for (int off = 1; off < R; off <<= 1) {
          ks_a += __shfl_xor_sync(0xffffffffu, ks_a, off);
          ks_b += __shfl_xor_sync(0xffffffffu, ks_b, off);
          qs_a += __shfl_xor_sync(0xffffffffu, qs_a, off);
          qs_b += __shfl_xor_sync(0xffffffffu, qs_b, off);
        }
        const float ua = beta_a * (va - ks_a);
        const float ub = beta_b * (vb - fmaf(kk_ab, ua, ks_b));
#pragma unroll
        for (int e = 0; e < PER; ++e) s[e] = fmaf(kb[e], ub, fmaf(gb[e] * ka[e], ua, ga[e]));
        if (live && r == 0) {
          float* orow = o + ((size_t)(ts + i) * H + h) * vdim + col;
          orow[0] = fmaf(qk_a, ua, qs_a);
          orow[(size_t)H * vdim] = fmaf(qk_b, ub, fmaf(qk_ba, ua, qs_b));
        }
      }
    }
    for (; i < n; ++i) {  // a portion's last token when their number is odd (a single decoded token)
      const float* row = buf + i * W;
      float v4[PER];
      channel_vector<PER, R>(row + 2 * RP, r, v4);
#pragma unroll
      for (int e = 0; e < PER; ++e) s[e] *= v4[e];
      float ks[2] = {}, qs[2] = {};
      channel_vector<PER, R>(row, r, v4);
#pragma unroll
      for (int e = 0; e < PER; ++e) qs[e & 1] = fmaf(v4[e], s[e], qs[e & 1]);
      channel_vector<PER, R>(row + RP, r, v4);
#pragma unroll
      for (int e = 0; e < PER; ++e) ks[e & 1] = fmaf(v4[e], s[e], ks[e & 1]);
      float ksum = ks[0] + ks[1], qsum = qs[0] + qs[1];
#pragma unroll
      for (int off = 1; off < R; off <<= 1) {
        ksum += __shfl_xor_sync(0xffffffffu, ksum, off);
        qsum += __shfl_xor_sync(0xffffffffu, qsum, off);
      }
      const float u = row[3 * RP + BC] * (row[3 * RP + in_block] - ksum);
#pragma unroll
      for (int e = 0; e < PER; ++e) s[e] = fmaf(v4[e], u, s[e]);
      if (live && r == 0) o[((size_t)(ts + i) * H + h) * vdim + col] = fmaf(row[3 * RP + BC + 2], u, qsum);
    }
  }
  pdl_trigger();  // at the end, as in delta_rule_kernel
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int d = channel_row<PER, R>(r, e);
    if (live && d < dim) S[(size_t)d * vdim + col] = s[e];
  }
  if (blockIdx.x == 0 && h == 0) keep_conv_inputs<T>(proj, P, base, t0, t1, C, K);
}

// The same rule for long portions and keys of 129 to 256 numbers, sixteen tokens at a time (shorter keys: delta_chunks.cu).
// Within a chunk, with c_i = g_1 ... g_i (the decays from the chunk's start up to token i, each a product of numbers of at most
// one, nothing is ever divided by a decay) and S the state before the chunk,
//
//     A_ij = sum_d k_i k_j g_(j+1) .. g_i   (j < i),      B_ij = the same with q_i   (j <= i),
//     (I + diag(beta) A) U = diag(beta) (V - (k c) S),    O = (q c) S + B U,    S <- c_16 S + sum_j (k_j g_(j+1) .. g_16) u_j^T.
//
// W = (I + diag(beta) A)^-1 diag(beta) is a triangular 16 x 16 matrix that does not depend on the state, so
//     U = W V - (W (k c)) S.
// channel_delta_chunk_kernel (a block per chunk and head, all chunks of the step side by side) leaves a record of what the
// chain needs: M = W (k c), Q = q c, K = k g .. (16 rows of RP numbers each), c_16 [RP], B [16][B_PITCH], W V [16][vpad].
// channel_delta_chain_kernel (a block per 16 columns, head and request) walks the chunks: one butterfly over the warp for the
// 32 products with S, then U, O and the new S.  A chain step costs sixteen tokens one such round instead of sixteen.
// Chunks are counted through the step's items in order; a portion's last chunk is filled up with tokens of beta 0, key 0
// and decay 1.
constexpr int CH = 16, B_PITCH = 20, CHAIN_COLS = 16, LR = 8, RP = 32 * LR;  // LR rows of S a lane, RP of them in all

struct ChunkRecord {
  int vpad;
  __host__ __device__ int b_at() const { return (3 * CH + 1) * RP; }
  __host__ __device__ int wv_at() const { return b_at() + CH * B_PITCH; }
  __host__ __device__ int floats() const { return wv_at() + CH * vpad; }
};

__device__ __forceinline__ bool find_delta_chunk(const int32_t* __restrict__ item_start, int items, int at, int& t0, int& n) {
  for (int i = 0; i < items; ++i) {
    const int a = item_start[i], b = item_start[i + 1];
    const int c = (b - a + CH - 1) / CH;
    if (at < c) {
      t0 = a + at * CH;
      n = min(CH, b - t0);
      return true;
    }
    at -= c;
  }
  return false;
}

// v[0..31] of every lane -> lane L gets the sum over the lanes of v[L].
__device__ __forceinline__ float reduce32(float (&v)[32], int lane) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int r = 0; r < off; ++r) {
      const float give = up ? v[r] : v[r + off], keep = up ? v[r + off] : v[r];
      v[r] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
  return v[0];
}

__global__ void __launch_bounds__(128)
channel_delta_chunk_kernel(const float* __restrict__ qkv, const float* __restrict__ bd, const float* __restrict__ decay,
                           const int32_t* __restrict__ item_start, float* __restrict__ records, int items, int G, int H, int dim,
                           int vdim, int vpad) {
  extern __shared__ __align__(16) float chunk_smem[];  // k, q, g: [CH][RP] each
  __shared__ float As[CH][CH + 1], Ws[CH][CH + 1], beta[CH];
  float *ks = chunk_smem, *qs = ks + CH * RP, *gs = qs + CH * RP;
  pdl_wait();
  int t0, n;
  if (!find_delta_chunk(item_start, items, blockIdx.x, t0, n)) return;
  const int h = blockIdx.y, g = h / (H / G);
  const int C = 2 * G * dim + H * vdim;
  const ChunkRecord rec{vpad};
  float* out = records + ((size_t)blockIdx.x * H + h) * rec.floats();
  for (int i = threadIdx.x; i < CH * RP; i += blockDim.x) {
    const int t = i / RP, d = i - t * RP;
    const bool there = t < n && d < dim;
    const float* row = qkv + (size_t)(t0 + t) * C + (size_t)g * dim + d;
    qs[i] = there ? row[0] : 0.f;
    ks[i] = there ? row[(size_t)G * dim] : 0.f;
    gs[i] = there ? decay[((size_t)(t0 + t) * H + h) * dim + d] : 1.f;
  }
  if (threadIdx.x < CH) beta[threadIdx.x] = (int)threadIdx.x < n ? bd[(size_t)(t0 + threadIdx.x) * BD * H + h] : 0.f;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j = warp; j < CH; j += 4) {
    float run[LR], v[32];
#pragma unroll
    for (int e = 0; e < LR; ++e) run[e] = ks[j * RP + e * 32 + lane];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      float a = 0.f, b = 0.f;
      if (i >= j) {
#pragma unroll
        for (int e = 0; e < LR; ++e) {
          const int at = i * RP + e * 32 + lane;
          if (i > j) run[e] *= gs[at];
          a = fmaf(ks[at], run[e], a);
          b = fmaf(qs[at], run[e], b);
        }
      }
      v[i] = i > j ? a : 0.f;
      v[CH + i] = b;
    }
    const float mine = reduce32(v, lane);
    if (lane < CH) As[lane][j] = mine;
    else out[rec.b_at() + (lane - CH) * B_PITCH + j] = mine;
  }
  __syncthreads();
  if (threadIdx.x < CH) {  // a column of W a thread, by forward substitution
    const int j = threadIdx.x;
    float w[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      float acc = i == j ? 1.f : 0.f;
#pragma unroll
      for (int l = 0; l < i; ++l) acc = fmaf(-As[i][l], w[l], acc);
      w[i] = beta[i] * acc;
      Ws[i][j] = w[i];
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RP; d += blockDim.x) {
    float kc[CH], c = 1.f;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      c *= gs[i * RP + d];
      kc[i] = ks[i * RP + d] * c;
      out[(CH + i) * RP + d] = qs[i * RP + d] * c;
    }
    out[3 * CH * RP + d] = c;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      float m = 0.f;
#pragma unroll
      for (int l = 0; l <= i; ++l) m = fmaf(Ws[i][l], kc[l], m);
      out[i * RP + d] = m;
    }
    c = 1.f;
#pragma unroll
    for (int i = CH - 1; i >= 0; --i) {
      out[(2 * CH + i) * RP + d] = ks[i * RP + d] * c;
      c *= gs[i * RP + d];
    }
  }
  for (int col = threadIdx.x; col < vpad; col += blockDim.x) {
    float v[CH];
#pragma unroll
    for (int l = 0; l < CH; ++l)
      v[l] = (l < n && col < vdim) ? qkv[(size_t)(t0 + l) * C + 2 * (size_t)G * dim + (size_t)h * vdim + col] : 0.f;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      float m = 0.f;
#pragma unroll
      for (int l = 0; l <= i; ++l) m = fmaf(Ws[i][l], v[l], m);
      out[rec.wv_at() + i * vpad + col] = m;
    }
  }
  pdl_trigger();  // at the end, as in delta_prepare_kernel: the chain's blocks are few and long
}

struct Four {
  float v[4];
};

// The four columns' sums of vectors BASE .. BASE + N - 1 (rows of RP numbers at ``rows``) with the lane's rows of S, brought
// together over the warp so that the lane whose low bits are r holds vector BASE + r's.
template <int N, int BASE>
__device__ __forceinline__ Four chain_products(const float* __restrict__ rows, const float (&s)[4][LR], int lane) {
  Four out;
  if constexpr (N == 1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) out.v[j] = 0.f;
#pragma unroll
    for (int e = 0; e < LR; e += 4) {
      const float4 m = *reinterpret_cast<const float4*>(rows + BASE * RP + e * 32 + lane * 4);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        out.v[j] = fmaf(m.w, s[j][e + 3], fmaf(m.z, s[j][e + 2], fmaf(m.y, s[j][e + 1], fmaf(m.x, s[j][e], out.v[j]))));
    }
  } else {
    const Four a = chain_products<N / 2, BASE>(rows, s, lane), b = chain_products<N / 2, BASE + N / 2>(rows, s, lane);
    const bool up = lane & (N / 2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float give = up ? a.v[j] : b.v[j], keep = up ? b.v[j] : a.v[j];
      out.v[j] = keep + __shfl_xor_sync(0xffffffffu, give, N / 2);
    }
  }
  return out;
}

// A block: 16 columns of a request's and head's state, four a warp; lane's rows of S: e / 4 * 128 + lane * 4 + e % 4.
template <typename T>
__global__ void __launch_bounds__(RULE_WARPS * 32)
channel_delta_chain_kernel(const float* __restrict__ records, const T* __restrict__ proj, long long P, float* __restrict__ state,
                           const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots, float* __restrict__ o, int G,
                           int H, int dim, int vdim, int vpad, int K, int num_slots, long long slot_floats) {
  const ChunkRecord rec{vpad};
  constexpr int HEAD = (3 * CH + 1) * RP + CH * B_PITCH, BUF = HEAD + CH * CHAIN_COLS;  // floats: the record up to B, then W V's columns
  extern __shared__ __align__(16) float chain_smem[];  // [2][BUF]
  __shared__ __align__(16) float us[RULE_WARPS][CH][4];
  const int C = 2 * G * dim + H * vdim;
  const int h = blockIdx.y, item = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col0 = blockIdx.x * CHAIN_COLS, col = col0 + warp * 4;
  pdl_wait();
  const int t0 = item_start[item], t1 = item_start[item + 1];
  int first = 0;
  for (int i = 0; i < item; ++i) first += (item_start[i + 1] - item_start[i] + CH - 1) / CH;
  const int chunks = (t1 - t0 + CH - 1) / CH;
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  float* base = state + (size_t)slot * slot_floats;
  float* S = base + (size_t)(K - 1) * C + (size_t)h * dim * vdim;

  auto stage = [&](int c, float* buf) {
    const float* src = records + ((size_t)(first + c) * H + h) * rec.floats();
    for (int i = threadIdx.x; i < HEAD / 4; i += blockDim.x) copy_async16(buf + i * 4, src + i * 4);
    for (int i = threadIdx.x; i < CH * CHAIN_COLS / 4; i += blockDim.x) {
      const int row = i / (CHAIN_COLS / 4), piece = i - row * (CHAIN_COLS / 4);
      copy_async16(buf + HEAD + i * 4, src + rec.wv_at() + row * vpad + col0 + piece * 4);
    }
  };

  if (chunks > 0) stage(0, chain_smem);
  float s[4][LR];
#pragma unroll
  for (int e = 0; e < LR; ++e) {
    const int d = e / 4 * 128 + lane * 4 + e % 4;
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j][e] = (d < dim && col + j < vdim) ? S[(size_t)d * vdim + col + j] : 0.f;
  }
  for (int c = 0; c < chunks; ++c) {
    copy_async_wait();
    __syncthreads();  // this chunk has landed for everybody, and everybody has left the other buffer
    if (c + 1 < chunks) stage(c + 1, chain_smem + ((c + 1) & 1) * BUF);
    const float* buf = chain_smem + (c & 1) * BUF;
    const Four y = chain_products<32, 0>(buf, s, lane);
    if (lane < CH) {
      const float4 wv = *reinterpret_cast<const float4*>(buf + HEAD + lane * CHAIN_COLS + warp * 4);
      *reinterpret_cast<float4*>(us[warp][lane]) = make_float4(wv.x - y.v[0], wv.y - y.v[1], wv.z - y.v[2], wv.w - y.v[3]);
    }
    __syncwarp();
    // the state first: the next chunk waits for it
    const float* krows = buf + 2 * CH * RP;
#pragma unroll
    for (int e = 0; e < LR; e += 4) {
      const float4 gc = *reinterpret_cast<const float4*>(buf + 3 * CH * RP + e * 32 + lane * 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[j][e] *= gc.x;
        s[j][e + 1] *= gc.y;
        s[j][e + 2] *= gc.z;
        s[j][e + 3] *= gc.w;
      }
    }
#pragma unroll
    for (int l = 0; l < CH; ++l) {
      const float4 u4 = *reinterpret_cast<const float4*>(us[warp][l]);
      const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
      for (int e = 0; e < LR; e += 4) {
        const float4 k = *reinterpret_cast<const float4*>(krows + l * RP + e * 32 + lane * 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[j][e] = fmaf(k.x, u[j], s[j][e]);
          s[j][e + 1] = fmaf(k.y, u[j], s[j][e + 1]);
          s[j][e + 2] = fmaf(k.z, u[j], s[j][e + 2]);
          s[j][e + 3] = fmaf(k.w, u[j], s[j][e + 3]);
        }
      }
    }
    if (lane >= CH) {
      const int i = lane - CH, t = t0 + c * CH + i;
      float acc[4] = {y.v[0], y.v[1], y.v[2], y.v[3]};
      const float* brow = buf + (3 * CH + 1) * RP + i * B_PITCH;
#pragma unroll
      for (int l = 0; l < CH; l += 4) {
        const float4 b = *reinterpret_cast<const float4*>(brow + l);
        const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 u4 = *reinterpret_cast<const float4*>(us[warp][l + q]);
          acc[0] = fmaf(bb[q], u4.x, acc[0]);
          acc[1] = fmaf(bb[q], u4.y, acc[1]);
          acc[2] = fmaf(bb[q], u4.z, acc[2]);
          acc[3] = fmaf(bb[q], u4.w, acc[3]);
        }
      }
      if (t < t1) {
        float* dst = o + ((size_t)t * H + h) * vdim + col;
        if (vdim % 4 == 0 && col < vdim) *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        else
          for (int j = 0; j < 4; ++j)
            if (col + j < vdim) dst[j] = acc[j];
      }
    }
    __syncwarp();
  }
  pdl_trigger();
#pragma unroll
  for (int e = 0; e < LR; ++e) {
    const int d = e / 4 * 128 + lane * 4 + e % 4;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (d < dim && col + j < vdim) S[(size_t)d * vdim + col + j] = s[j][e];
  }
  if (blockIdx.x == 0 && h == 0) keep_conv_inputs<T>(proj, P, base, t0, t1, C, K);
}

template <typename T>
__global__ void __launch_bounds__(128)
delta_finish_kernel(const float* __restrict__ o, const T* __restrict__ proj, const float* __restrict__ gain,
                    T* __restrict__ out, long long units, int G, int H, int dim, int vdim, float eps) {
  pdl_trigger();
  pdl_wait();
  const long long unit = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (unit >= units) return;
  const long long t = unit / H;
  const int h = (int)(unit - t * H);
  const int C = 2 * G * dim + H * vdim, P = C + H * vdim;
  const float* orow = o + (size_t)unit * vdim;
  const T* gate = proj + (size_t)t * P + C + (size_t)h * vdim;
  float ss = 0.f;
  for (int j = lane; j < vdim; j += 32) ss = fmaf(orow[j], orow[j], ss);
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / (float)vdim + eps);
  T* orow_out = out + (size_t)unit * vdim;
  for (int j = lane; j < vdim; j += 32) orow_out[j] = from_float<T>(orow[j] * inv * gain[j] * siluf_(to_float<T>(gate[j])));
}

// The same for up to 128 values in fours, four heads of a token (or of neighbouring tokens) a warp: what they read is asked for at once.
constexpr int FINISH_UNITS = 4;

template <typename T>
__global__ void __launch_bounds__(128)
delta_finish_wide_kernel(const float* __restrict__ o, const T* __restrict__ proj, const float* __restrict__ gain,
                         T* __restrict__ out, unsigned units, int G, int H, int dim, int vdim, float eps) {
  pdl_trigger();
  pdl_wait();
  const unsigned first = (blockIdx.x * 4 + (threadIdx.x >> 5)) * FINISH_UNITS;
  const int lane = threadIdx.x & 31;
  const bool mine = 4 * lane < vdim;
  const int C = 2 * G * dim + H * vdim, P = C + H * vdim;
  float x[FINISH_UNITS][4], z[FINISH_UNITS][4], g[4];
#pragma unroll
  for (int u = 0; u < FINISH_UNITS; ++u) {
    const unsigned unit = first + u, t = unit / (unsigned)H;
#pragma unroll
    for (int j = 0; j < 4; ++j) x[u][j] = z[u][j] = 0.f;
    if (mine && unit < units) {
      load_four<float>(o + (size_t)unit * vdim + 4 * lane, x[u]);
      load_four<T>(proj + (size_t)t * P + C + (size_t)(unit - t * H) * vdim + 4 * lane, z[u]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) g[j] = mine ? gain[4 * lane + j] : 0.f;
  silu_all(z);
#pragma unroll
  for (int u = 0; u < FINISH_UNITS; ++u) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) ss = fmaf(x[u][j], x[u][j], ss);
    const float inv = 1.f / sqrtf(warp_sum(ss) / (float)vdim + eps);
    if (!mine || first + u >= units) continue;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = x[u][j] * inv * g[j] * z[u][j];
    T* dst = out + (size_t)(first + u) * vdim + 4 * lane;
    if constexpr (sizeof(T) == 2) {
      __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    } else {
      *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
}

template <typename T, int PER, int R>
void launch_rule(dim3 grid, cudaStream_t stream, const float* qkv, const float* bd, const T* proj, float* state,
                 const int32_t* item_start, const int32_t* slots, float* o, int G, int H, int dim, int vdim, int K,
                 int num_slots, size_t slot_floats, int max_tokens) {
  constexpr int W = (2 * R * PER + RULE_WARPS * (32 / R) + BD + 3) / 4 * 4;
  // two buffers within the 48 KB a kernel has without asking: 16 tokens a stage for keys up to 128 numbers, 4 beyond
  const int stage_tokens = 2 * 16 * W * (int)sizeof(float) <= 48 * 1024 ? 16 : 4;
  static_assert(2 * 4 * W * sizeof(float) <= 48 * 1024, "a stage of four tokens fits the default shared memory twice");
  psb_launch(delta_rule_kernel<T, PER, R>, grid, dim3(RULE_WARPS * 32), (size_t)2 * stage_tokens * W * sizeof(float), stream, qkv,
             bd, proj, state, item_start, slots, o, G, H, dim, vdim, K, num_slots, slot_floats, stage_tokens, max_tokens);
}

}  // namespace

PSB_API int psb_delta_max_taps() { return MAX_TAPS; }

// ``ba`` null: the write strengths' pre-activations are the projection's columns beta_at .. beta_at + H - 1 and the decays come
// from elsewhere; ``decay`` (float32 [T, H, dim] or null) then goes into the products with the key of the token before.
// (proj, dtype, ld, beta_at, ba, decay, taps, a_log, dt_bias, state, positions, token_item, item_start, slots, qkv_out, bd_out, T, G,
//  H, dim, vdim, K, num_slots, slot_floats, cross, stream); ``cross`` 0: no token goes through a kernel that reads those products
PSB_API int psb_delta_prepare(const void* proj, int dtype, long long ld, int beta_at, const void* ba, const void* decay,
                              const void* taps, const void* a_log, const void* dt_bias, const void* state, const void* positions, const void* token_item,
                              const void* item_start, const void* slots, void* qkv, void* bd, int T, int G, int H, int dim,
                              int vdim, int K, int num_slots, long long slot_floats, int cross, cudaStream_t stream) {
  if (T < 0 || G < 1 || H < 1 || H % G || dim < 1 || vdim < 1) PSB_REFUSE("delta_prepare: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS) PSB_REFUSE("delta_prepare: %d taps are outside [1, %d]", K, MAX_TAPS);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  if (ld < C || (!ba && (beta_at < 0 || ld < (long long)beta_at + H))) PSB_REFUSE("delta_prepare: row stride %lld is shorter than the row", ld);
  if (slot_floats != (K - 1) * C + (long long)H * dim * vdim) PSB_REFUSE("delta_prepare: a slot of %lld numbers does not fit the sizes", slot_floats);
  const size_t smem = (size_t)(dim > vdim ? dim : vdim) * sizeof(float);
  if (smem > 48 * 1024 || 2 * G + H > 65535) PSB_REFUSE("delta_prepare: sizes exceed the kernel's shared memory or grid");
  if (T == 0) return 0;
  PSB_DISPATCH_DTYPE(dtype, T_, {
    const int widest = dim > vdim ? dim : vdim;
    // Runs of eight tokens: a step of few tokens fills too few warps with them, a block a token and unit is done first (12 us either way
    // at 40 tokens of 64 units and at 85 of 32; 23 us against 36 at 150 of 64).
    if ((long long)T * (2 * G + H) >= 2560 && K <= RUN_TAPS && widest <= 128 && dim % 4 == 0 && vdim % 4 == 0 && ld % 4 == 0 && ((uintptr_t)proj & (4 * sizeof(T_) - 1)) == 0
        && (((uintptr_t)qkv | (uintptr_t)taps) & 15) == 0) {
      psb_launch(delta_prepare_wide_kernel<T_>, dim3((T + RUN_TOKENS - 1) / RUN_TOKENS, (2 * G + H + WIDE_WARPS - 1) / WIDE_WARPS), dim3(WIDE_WARPS * 32),
                 0, stream, (const T_*)proj, (const float*)ba, (const float*)taps, (const float*)a_log, (const float*)dt_bias, (const float*)state,
                 (const int32_t*)positions, (const int32_t*)token_item, (const int32_t*)item_start, (const int32_t*)slots, (float*)qkv, (float*)bd,
                 G, H, dim, vdim, K, num_slots, (size_t)slot_floats, T, ld, beta_at);
    } else if (T >= 256 && K <= RUN_TAPS && widest <= 256) {
      auto launch = [&](auto kernel) {
        psb_launch(kernel, dim3((T + RUN_TOKENS - 1) / RUN_TOKENS, 2 * G + H), dim3(128), 0, stream, (const T_*)proj, (const float*)ba,
                   (const float*)taps, (const float*)a_log, (const float*)dt_bias, (const float*)state, (const int32_t*)positions,
                   (const int32_t*)token_item, (const int32_t*)item_start, (const int32_t*)slots, (float*)qkv, (float*)bd, G, H, dim,
                   vdim, K, num_slots, (size_t)slot_floats, T, ld, beta_at);
      };
      if (widest <= 128) launch(delta_prepare_run_kernel<T_, 1>);
      else launch(delta_prepare_run_kernel<T_, 2>);
    } else {
    const int per_block = T >= 1024 ? 8 : 1;  // long steps: a block stays with its unit for eight tokens
    psb_launch(delta_prepare_kernel<T_>, dim3((T + per_block - 1) / per_block, 2 * G + H), dim3(128), smem, stream, (const T_*)proj,
               (const float*)ba, (const float*)taps, (const float*)a_log, (const float*)dt_bias, (const float*)state,
               (const int32_t*)positions, (const int32_t*)token_item, (const int32_t*)item_start, (const int32_t*)slots,
               (float*)qkv, (float*)bd, G, H, dim, vdim, K, num_slots, (size_t)slot_floats, T, per_block, ld, beta_at);
    }
  });
  PSB_LAUNCH_CHECK("delta_prepare");
  if (!cross || (!ba && !decay)) return 0;  // the chunked forms make their own products
  const long long units = (long long)T * H;
  psb_launch(delta_cross_kernel, dim3((unsigned)((units + 3) / 4)), dim3(128), 0, stream, (const float*)qkv, (const int32_t*)token_item,
             (const int32_t*)item_start, (float*)bd, units, G, H, dim, vdim, (const float*)decay);
  PSB_LAUNCH_CHECK("delta_cross");
  return 0;
}

// (qkv, bd, proj, dtype, state, item_start, slots, o_out, items, G, H, dim, vdim, K, num_slots, slot_floats, lanes, max_tokens,
//  stream).  Portions of more than ``max_tokens`` tokens, and their slots, are left untouched.
// ``lanes``: lanes of a warp that share a column of the state (4: a warp reads whole sectors of the state, for steps
// of single tokens; 16 or 32: short chains per token and more warps, for long portions).
PSB_API int psb_delta_rule(const void* qkv, const void* bd, const void* proj, int dtype, void* state, const void* item_start,
                           const void* slots, void* o, int items, int G, int H, int dim, int vdim, int K, int num_slots,
                           long long slot_floats, int lanes, int max_tokens, cudaStream_t stream) {
  if (items < 0 || G < 1 || H < 1 || H % G || dim < 1 || vdim < 1) PSB_REFUSE("delta_rule: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS) PSB_REFUSE("delta_rule: %d taps are outside [1, %d]", K, MAX_TAPS);
  if (lanes != 4 && lanes != 16 && lanes != 32) PSB_REFUSE("delta_rule: %d lanes a column is not built (4, 16 or 32)", lanes);
  if (dim > 64 * lanes) PSB_REFUSE("delta_rule: key size %d exceeds %d", dim, 64 * lanes);
  if (H > 65535 || items > 65535) PSB_REFUSE("delta_rule: too many heads or requests for one launch");
  if (items == 0) return 0;
  const int per = (dim + lanes - 1) / lanes;
  const int cols = RULE_WARPS * (32 / lanes);
  const dim3 grid((vdim + cols - 1) / cols, H, items);
#define RULE(PER_, R_)                                                                                                \
  launch_rule<T_, PER_, R_>(grid, stream, (const float*)qkv, (const float*)bd, (const T_*)proj, (float*)state,       \
                            (const int32_t*)item_start, (const int32_t*)slots, (float*)o, G, H, dim, vdim, K, num_slots, \
                            (size_t)slot_floats, max_tokens)
  PSB_DISPATCH_DTYPE(dtype, T_, {
    if (lanes == 4) {
      if (per <= 4) RULE(4, 4);
      else if (per <= 8) RULE(8, 4);
      else if (per <= 16) RULE(16, 4);
      else if (per <= 32) RULE(32, 4);
      else RULE(64, 4);
    } else if (lanes == 16) {
      if (per <= 2) RULE(2, 16);
      else if (per <= 4) RULE(4, 16);
      else if (per <= 8) RULE(8, 16);
      else RULE(16, 16);
    } else {
      if (per <= 1) RULE(1, 32);
      else if (per <= 2) RULE(2, 32);
      else if (per <= 4) RULE(4, 32);
      else RULE(8, 32);
    }
  });
#undef RULE
  PSB_LAUNCH_CHECK("delta_rule");
  return 0;
}

// (qkv, bd, decay, proj, dtype, ld, state, item_start, slots, o_out, items, G, H, dim, vdim, K, num_slots, slot_floats, lanes, max_tokens,
//  stream)  ``lanes`` (4, 8, 16 or 32) and ``max_tokens`` as for psb_delta_rule.
PSB_API int psb_channel_delta_rule(const void* qkv, const void* bd, const void* decay, const void* proj, int dtype, long long ld,
                                   void* state, const void* item_start, const void* slots, void* o, int items, int G, int H, int dim,
                                   int vdim, int K, int num_slots, long long slot_floats, int lanes, int max_tokens, cudaStream_t stream) {
  if (items < 0 || G < 1 || H < 1 || H % G || dim < 1 || vdim < 1) PSB_REFUSE("channel_delta_rule: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS) PSB_REFUSE("channel_delta_rule: %d taps are outside [1, %d]", K, MAX_TAPS);
  if (lanes != 4 && lanes != 8 && lanes != 16 && lanes != 32) PSB_REFUSE("channel_delta_rule: %d lanes a column is not built (4, 8, 16 or 32)", lanes);
  const int per = (dim + lanes - 1) / lanes;
  if (per > 32) PSB_REFUSE("channel_delta_rule: key size %d exceeds %d", dim, 32 * lanes);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  if (ld < C || slot_floats != (K - 1) * C + (long long)H * dim * vdim) PSB_REFUSE("channel_delta_rule: the slot or the rows do not fit the sizes");
  if (H > 65535 || items > 65535) PSB_REFUSE("channel_delta_rule: too many heads or requests for one launch");
  if (items == 0) return 0;
  const int cols = RULE_WARPS * (32 / lanes);
  const dim3 grid((vdim + cols - 1) / cols, H, items);
#define PSB_RULE(PER_, R_)                                                                                                         \
  do {                                                                                                                             \
    constexpr int W = (3 * R_ * PER_ + RULE_WARPS * (32 / R_) + BD + 3) / 4 * 4;                                                   \
    constexpr int stage_tokens = 2 * 16 * W * (int)sizeof(float) <= 64 * 1024 ? 16 : (2 * 8 * W * (int)sizeof(float) <= 64 * 1024 ? 8 : 2); \
    constexpr int smem = 2 * stage_tokens * W * (int)sizeof(float);                                                                 \
    auto kernel = channel_delta_rule_kernel<T_, PER_, R_>;                                                                          \
    if (smem > 48 * 1024) {                                                                                                        \
      static PsbPerDevice configured;                                                                                              \
      if (!configured.get()) {                                                                                                     \
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)                        \
          PSB_REFUSE("channel_delta_rule: cannot raise the shared-memory limit");                                                  \
        configured.set();                                                                                                          \
      }                                                                                                                            \
    }                                                                                                                              \
    psb_launch(kernel, grid, dim3(RULE_WARPS * 32), (size_t)smem, stream, (const float*)qkv, (const float*)bd, (const float*)decay, \
               (const T_*)proj, ld, (float*)state, (const int32_t*)item_start, (const int32_t*)slots, (float*)o, G, H, dim, vdim, K, \
               num_slots, slot_floats, stage_tokens, max_tokens);                                                                  \
  } while (0)
  PSB_DISPATCH_DTYPE(dtype, T_, {
    if (lanes == 4) {
      if (per <= 4) PSB_RULE(4, 4); else if (per <= 8) PSB_RULE(8, 4); else if (per <= 16) PSB_RULE(16, 4); else PSB_RULE(32, 4);
    } else if (lanes == 8) {
      if (per <= 4) PSB_RULE(4, 8); else if (per <= 8) PSB_RULE(8, 8); else if (per <= 16) PSB_RULE(16, 8); else PSB_RULE(32, 8);
    } else if (lanes == 16) {
      if (per <= 2) PSB_RULE(2, 16); else if (per <= 4) PSB_RULE(4, 16); else if (per <= 8) PSB_RULE(8, 16);
      else if (per <= 16) PSB_RULE(16, 16); else PSB_RULE(32, 16);
    } else {
      if (per <= 4) PSB_RULE(4, 32); else if (per <= 8) PSB_RULE(8, 32); else if (per <= 16) PSB_RULE(16, 32); else PSB_RULE(32, 32);
    }
  });
#undef PSB_RULE
  PSB_LAUNCH_CHECK("channel_delta_rule");
  return 0;
}

// (dim, vdim) -> float32 numbers of a chunk's record, 0 if the chunked form does not take the sizes (keys of up to 128 numbers go through
// the kernels of delta_chunks.cu)
PSB_API int psb_channel_delta_record(int dim, int vdim) {
  if (dim <= 128 || vdim < 1 || dim > 256 || vdim > 4096) return 0;
  return ChunkRecord{(vdim + CHAIN_COLS - 1) / CHAIN_COLS * CHAIN_COLS}.floats();
}

// The chunked form: (qkv, bd, decay, proj, dtype, ld, state, item_start, slots, records, o_out, items, chunks, G, H, dim, vdim, K,
// num_slots, slot_floats, stream); records [chunks, H, psb_channel_delta_record] float32, chunks at least sum ceil(tokens / 16)
PSB_API int psb_channel_delta_chunks(const void* qkv, const void* bd, const void* decay, const void* proj, int dtype, long long ld,
                                     void* state, const void* item_start, const void* slots, void* records, void* o, int items,
                                     int chunks, int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats,
                                     cudaStream_t stream) {
  if (items < 0 || G < 1 || H < 1 || H % G || !psb_channel_delta_record(dim, vdim)) PSB_REFUSE("channel_delta_chunks: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS) PSB_REFUSE("channel_delta_chunks: %d taps are outside [1, %d]", K, MAX_TAPS);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  if (ld < C || slot_floats != (K - 1) * C + (long long)H * dim * vdim) PSB_REFUSE("channel_delta_chunks: the slot or the rows do not fit the sizes");
  if (H > 65535 || items > 65535 || chunks < items) PSB_REFUSE("channel_delta_chunks: too many heads or requests, or too few chunks");
  if (((uintptr_t)records | (uintptr_t)o) & 15) PSB_REFUSE("channel_delta_chunks: records and read-out must be 16-byte aligned");
  if (items == 0) return 0;
  const int vpad = (vdim + CHAIN_COLS - 1) / CHAIN_COLS * CHAIN_COLS;
  constexpr int chunk_bytes = 3 * CH * RP * (int)sizeof(float);
  constexpr int chain_bytes = 2 * ((3 * CH + 1) * RP + CH * B_PITCH + CH * CHAIN_COLS) * (int)sizeof(float);
  PSB_DISPATCH_DTYPE(dtype, T_, {
    auto chunk = channel_delta_chunk_kernel;
    auto chain = channel_delta_chain_kernel<T_>;
    static PsbPerDevice configured;
    if (!configured.get()) {
      if (cudaFuncSetAttribute(chunk, cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_bytes) != cudaSuccess ||
          cudaFuncSetAttribute(chain, cudaFuncAttributeMaxDynamicSharedMemorySize, chain_bytes) != cudaSuccess)
        PSB_REFUSE("channel_delta_chunks: cannot raise the shared-memory limit");
      configured.set();
    }
    psb_launch(chunk, dim3(chunks, H), dim3(128), (size_t)chunk_bytes, stream, (const float*)qkv, (const float*)bd,
               (const float*)decay, (const int32_t*)item_start, (float*)records, items, G, H, dim, vdim, vpad);
    PSB_LAUNCH_CHECK("channel_delta_chunk");
    psb_launch(chain, dim3(vpad / CHAIN_COLS, H, items), dim3(RULE_WARPS * 32), (size_t)chain_bytes, stream, (const float*)records,
               (const T_*)proj, ld, (float*)state, (const int32_t*)item_start, (const int32_t*)slots, (float*)o, G, H, dim, vdim,
               vpad, K, num_slots, slot_floats);
    PSB_LAUNCH_CHECK("channel_delta_chain");
  });
  return 0;
}

// (o, proj, dtype, gain, out, T, G, H, dim, vdim, eps, stream)
PSB_API int psb_delta_finish(const void* o, const void* proj, int dtype, const void* gain, void* out, int T, int G, int H,
                             int dim, int vdim, float eps, cudaStream_t stream) {
  if (T < 0 || G < 1 || H < 1 || dim < 1 || vdim < 1) PSB_REFUSE("delta_finish: bad sizes");
  if (T == 0) return 0;
  const long long units = (long long)T * H;
  PSB_DISPATCH_DTYPE(dtype, T_, {
    // (a unit a warp: 3.3 us against 4.9 at 2,900 units, 17 against 13 at 32,000)
    if (units >= 12288 && units < (1LL << 31) && vdim <= 128 && vdim % 4 == 0 && dim % 4 == 0 && (((uintptr_t)o | (uintptr_t)proj | (uintptr_t)out) & 15) == 0)
      psb_launch(delta_finish_wide_kernel<T_>, dim3((unsigned)((units + 4 * FINISH_UNITS - 1) / (4 * FINISH_UNITS))), dim3(128), 0, stream,
                 (const float*)o, (const T_*)proj, (const float*)gain, (T_*)out, (unsigned)units, G, H, dim, vdim, eps);
    else
      psb_launch(delta_finish_kernel<T_>, dim3((unsigned)((units + 3) / 4)), dim3(128), 0, stream, (const float*)o, (const T_*)proj,
                 (const float*)gain, (T_*)out, units, G, H, dim, vdim, eps);
  });
  PSB_LAUNCH_CHECK("delta_finish");
  return 0;
}
