// The delta rules over portions, 32 tokens at a time, float32 throughout: the gated one (a decay per head; bfloat16 projections) and
// the one with a decay per head and key channel.
//
// Within a chunk, with g_l the decays (a vector over the key channels; the gated rule's are all alike), c_i = g_1 .. g_i (from the
// chunk's start up to token i), r_j = g_(j+1) .. g_32 and S the state before the chunk, the writes u_i of its tokens are the rows of
//
//     U = W V - M S,         W = (I + diag(beta) A)^-1 diag(beta),  M = W (K c),   A_ij = sum_d k_i k_j g_(j+1) .. g_i   (j < i),
//     O = (Q c) S + B U,     B_ij = sum_d q_i k_j g_(j+1) .. g_i   (j <= i),
//     S <- c_32 S + (K r)^T U.
//
// (Decays are only ever multiplied, never divided by, and their running products carry what the roundings lose, but for A and B within sixteen
// tokens where the decays are per channel: plain float32, up to fifteen factors.)  All but the products with S and U is made beforehand:
//   delta_chunk_kernel, channel_delta_chunk_kernel   a block per chunk and head, all chunks of the step side by side: A, B and W (forward
//                        substitution, a column a lane), then M, Q c, K r, B, c_32 and W V, 98 KB a chunk and head;
//   delta_chain_kernel   a block per 16 or 32 columns of a head's state and request walks the chunks, on the tensor cores.  Eight warps hold
//                        16 key channels of S each, in registers, as the left operand of the first product and the sums of the second;
//                        what a chunk brings each asks for a chunk ahead, straight into registers.  [M; Q c] S comes out in eight shares that go through shared
//                        memory; eight more warps make U of M's while the first multiply Q c, and the read-outs while those bring S up to date.
// Operands of the tensor cores are three bfloat16 terms a float32 number, to its last bit: the sums of the six products of terms that count are as
// accurate as float32's own (the products of first terms are added up in float32 with rounding to nearest, sixteen tokens or channels
// at a time, since the instruction cuts its sums off; the rest is smaller by 2^8).  M, Q, K and B are taken apart once, where they are made.
// W and B are zero above the diagonal, and zero times what is not finite is not zero: M and W V are summed over the tokens up to their own, and
// a read-out that comes out not finite is made again from those, so that a token reaches later ones only.
// Chunks are counted through the step's portions of at least ``min_tokens`` tokens in order; a portion's last chunk is filled up
// with tokens of beta 0, key 0 and decay 1.
//
// Distances from float64 for the same unit vectors, strengths and decays, the gated rule token by token and here (9, 31, 64, 700 and 2,000 tokens of 16
// heads): read-outs before they are rounded to bfloat16 0.95, 1.12, 0.93, 1.74 and 1.73e-7 and 0.82, 0.99, 1.02, 1.13 and 1.11e-7; states 0.92, 1.33, 0.90, 2.05
// and 2.04e-7 and 0.64, 0.80, 0.98, 0.96 and 0.99e-7.  The rule with a decay per channel over 1,200 tokens, whole: read-outs 1.6e-7, states 1.4e-7;
// sixteen tokens at a time on the CUDA cores, as it was, 2.1e-7 and 1.9e-7.
//
// What bounds it: the chain, by the latency of its steps one after the other (in clocks, a block of 16 columns: a share of [M; Q c] S 900, U 500 beside the other
// half, the new state 1,000, and two barriers; the tensor cores are busy 1,280 of 3,000).  2,000 tokens of 16 heads: chunk kernel 44 us, chain 110; two portions of
// 1,200 and 960 tokens with decays per channel 66 and 112.  The chain was 135 and 125 with four warps beside the workers, who then waited for U and for the
// read-outs (1,750), with W V asked for just before its use, and with records that came from DRAM no more than a chunk ahead; products of up to six TF32 terms
// whose operands every block split for itself took 201 us, sixteen tokens at a time on the CUDA cores 211, register tiles of fma.rn.f32x2 193, bound by
// what shared memory hands to the registers; two chunks ahead through shared memory: no faster.
#include "chunk_products.cuh"

namespace {
using namespace delta;
using namespace chunks;

// A chunk's record of a head, 32-bit words.  What the tensor cores take lies as their right operands' fragments, a lane's four words of a term
// together (16 channels or tokens by 8, see mma_bf16), 128 words a term, three terms one after the other:
//   M and Q c   per 16 channels w, per two eights of tokens (0, 1: M; 2, 3: Q c): both fragments of either eight;
//   K r         per 16 channels, per eight of them: both fragments of tokens 0 .. 15, then of 16 .. 31;
//   B           per eight of its rows: the same;
// then c_32 [128], and W V [columns in runs of 16][32] as float32.
constexpr int MQ_AT = 0, K_AT = MQ_AT + (RP / 16) * 4 * UNIT, B_AT = K_AT + (RP / 16) * 2 * UNIT, G_AT = B_AT + (CHUNK / 8) * UNIT, V_AT = G_AT + RP;
constexpr int RUN = 16;
__host__ __device__ constexpr int record_floats(int vdim) { return V_AT + (vdim + RUN - 1) / RUN * RUN * CHUNK; }

// W in A's place (the whole warp, a column a lane): row i of A is used up when W's is known.  ``beta``: of the lane's token.
__device__ __forceinline__ void solve(float (*as)[TP], float beta, int lane) {
  float w[CHUNK];
#pragma unroll
  for (int i = 0; i < CHUNK; ++i) {
    float acc[4] = {};
#pragma unroll
    for (int l = 0; l < i; l += 4) {
      const float4 a = *reinterpret_cast<const float4*>(&as[i][l]);  // zeros from the diagonal on
      acc[0] = fmaf(a.x, w[l], acc[0]);
      if (l + 1 < i) acc[1] = fmaf(a.y, w[l + 1], acc[1]);
      if (l + 2 < i) acc[2] = fmaf(a.z, w[l + 2], acc[2]);
      if (l + 3 < i) acc[3] = fmaf(a.w, w[l + 3], acc[3]);
    }
    const float b = __shfl_sync(0xffffffffu, beta, i);
    w[i] = b * ((i == lane ? 1.f : 0.f) - ((acc[0] + acc[1]) + (acc[2] + acc[3])));
    __syncwarp();
    as[i][lane] = w[i];
  }
  __syncwarp();
}
// 16 columns of X as a thread's share of right operands: [tokens 16 k + 8 r + 2 tg + 0, 1][columns 8 n + gr]
struct Columns {
  float v[2][2][2][2];  // [k][n][r][token]
  template <typename X>
  __device__ __forceinline__ void fetch(X x, int gr, int tg) {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int t = 0; t < 2; ++t) v[k][n][r][t] = x(16 * k + 8 * r + 2 * tg + t, 8 * n + gr);
  }
};
// W X: rows gr and gr + 8 of either half, columns 2 tg and 2 tg + 1 of either eight, in out[half][eight][4].  W is zero above the diagonal, and a row that
// comes out not finite is made again from the tokens up to its own, ``x(l, column)``.
template <typename X>
__device__ __forceinline__ void times_w(const float (*ws)[TP], const Left (&w)[3], const Columns& have, X x, float (&out)[2][2][4], int gr, int tg) {
  float sum[2][2][4] = {}, small[2][2][4] = {};
  Right b[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) b[n].put(r, split3(have.v[k][n][r][0], have.v[k][n][r][1]));
    if (k == 0) step<2>(sum[0], small[0], w[0], b);
    step<2>(sum[1], small[1], w[1 + k], b);
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) out[m][n][e] = sum[m][n][e] + small[m][n][e];
  bool fine = true;
#pragma unroll
  for (int i = 0; i < 16; ++i) fine = fine && is_finite(out[i >> 3][(i >> 2) & 1][i & 3]);
  if (!fine) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      const int row = 16 * (i >> 3) + gr + 8 * ((i >> 1) & 1), col = 8 * ((i >> 2) & 1) + 2 * tg + (i & 1);
      float again = 0.f;
#pragma unroll 1
      for (int l = 0; l <= row; ++l) again = fmaf(ws[row][l], x(l, col), again);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j == i && !is_finite(out[j >> 3][(j >> 2) & 1][j & 3])) out[j >> 3][(j >> 2) & 1][j & 3] = again;
    }
  }
}
// M and W V of a head, 16 channels or columns a warp at a time.  K c is ``kc(l, d)``; ``ahead``: this warp's first columns of V (16 warp ..).
template <int WARPS, typename KC, typename V>
__device__ __forceinline__ void put_m_and_values(const float (*ws)[TP], KC kc, V v, Columns& ahead, int vdim, float* __restrict__ out, int warp, int lane) {
  const int gr = lane >> 2, tg = lane & 3;
  const Left w[3] = {left_rows(&ws[0][0], TP, gr, tg), left_rows(&ws[16][0], TP, gr, tg), left_rows(&ws[16][16], TP, gr, tg)};
  float y[2][2][4];
#pragma unroll 1
  for (int u = warp; u < RP / 16; u += WARPS) {
    auto x = [&](int l, int d) { return kc(l, 16 * u + d); };
    Columns have;
    have.fetch(x, gr, tg);
    times_w(ws, w, have, x, y, gr, tg);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const Terms t[4] = {split3(y[m][0][0], y[m][0][1]), split3(y[m][1][0], y[m][1][1]), split3(y[m][0][2], y[m][0][3]), split3(y[m][1][2], y[m][1][3])};
      put_terms(out + MQ_AT + (u * 4 + m) * UNIT + 4 * lane, t);
    }
  }
#pragma unroll 1
  for (int col0 = 16 * warp; col0 < vdim; col0 += 16 * WARPS) {
    const Columns have = ahead;
    if (col0 + 16 * WARPS < vdim) ahead.fetch([&](int l, int c) { return v(l, col0 + 16 * WARPS + c); }, gr, tg);
    times_w(ws, w, have, [&](int l, int c) { return v(l, col0 + c); }, y, gr, tg);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) out[V_AT + (col0 + 8 * c + 2 * tg + (e & 1)) * CHUNK + 16 * m + gr + 8 * (e >> 1)] = y[m][c][e];
  }
}
struct ChunkShape {
  static constexpr int Q = CHUNK * KP, AS = 2 * CHUNK * KP, BS = AS + CHUNK * TP, CR = BS + CHUNK * TP, FLOATS = CR + 2 * CHUNK;
};

// (The heads of a group each make K K^T and Q K^T again: a block per group had too few warps, and too few blocks, to hide one step's latency behind
// another's.)
__global__ void __launch_bounds__(CHUNK_THREADS, 4)
delta_chunk_kernel(const float* __restrict__ qkv, const float* __restrict__ bd, const int32_t* __restrict__ item_start,
                   float* __restrict__ records, int items, int min_tokens, int G, int H, int dim, int vdim) {
  using Sh = ChunkShape;
  extern __shared__ __align__(16) float chunk_smem[];
  float *ks = chunk_smem, *qs = chunk_smem + Sh::Q;
  float(*as)[TP] = reinterpret_cast<float(*)[TP]>(chunk_smem + Sh::AS);
  float(*bs)[TP] = reinterpret_cast<float(*)[TP]>(chunk_smem + Sh::BS);
  float *cs = chunk_smem + Sh::CR, *rs = cs + CHUNK;  // c and r of every token
  const int h = blockIdx.x % H, chunk = (int)(gridDim.x / H) - 1 - (int)(blockIdx.x / H);  // the first chunks last: the chain starts with them
  pdl_wait();
  int t0, n;
  if (!portions::find_chunk<CHUNK>(item_start, items, min_tokens, chunk, t0, n)) return;
  const int g = h / (H / G), C = 2 * G * dim + H * vdim;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  float* out = records + ((size_t)chunk * H + h) * record_floats(vdim);
  bring_rows(qs, qkv + (size_t)t0 * C + (size_t)g * dim, C, n, dim, true);
  bring_rows(ks, qkv + (size_t)t0 * C + (size_t)(G + g) * dim, C, n, dim, true);
  const float* mine = bd + (size_t)(t0 + min(lane, n - 1)) * BD * H + h;
  const float beta = lane < n ? mine[0] : 0.f, decay = lane < n ? mine[H] : 1.f;
  copy_async_wait();
  __syncthreads();
  {  // K K^T and Q K^T, 16 rows a warp
    static_assert(CHUNK_THREADS == 128, "four warps");
    const float* rows = (warp < 2 ? ks : qs) + 16 * (warp & 1) * KP;
    float sum[4][4] = {}, small[4][4] = {};
#pragma unroll 1
    for (int k = 0; k < RP; k += 16) {
      Right b[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) b[m] = right_rows(ks + 8 * m * KP + k, KP, gr, tg);
      step<4>(sum, small, left_rows(rows + k, KP, gr, tg), b);
    }
    float* to = (warp < 2 ? as : bs)[16 * (warp & 1) + gr] + 2 * tg;
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) to[8 * (e >> 1) * TP + 8 * m + (e & 1)] = sum[m][e] + small[m][e];
  }
  __syncthreads();
  if (warp < 2) {  // (either warp of A and B, both with all the products)
    float(*at)[TP] = warp ? bs : as;
    Product run, before, behind;  // lane j: products over the tokens between j and i, up to j, behind j
#pragma unroll 4
    for (int i = 0; i < CHUNK; ++i) {
      const float d = __shfl_sync(0xffffffffu, decay, i);
      if (i <= lane) before.times(d);
      if (i > lane) {
        run.times(d);
        behind.times(d);
      }
      at[i][lane] = i + warp > lane ? run.value() * at[i][lane] : 0.f;
    }
    if (warp) {
      cs[lane] = before.value();
      rs[lane] = behind.value();
    }
  }
  __syncthreads();
  const float* values = qkv + (size_t)t0 * C + 2 * (size_t)G * dim + (size_t)h * vdim;
  auto v = [&](int l, int c) { return l < n && c < vdim ? values[(size_t)l * C + c] : 0.f; };
  Columns ahead;
  ahead.fetch([&](int l, int c) { return v(l, 16 * warp + c); }, gr, tg);
  if (warp == 0) {
    solve(as, beta, lane);
  } else {  // what does not wait for W
    put_rows(qs, out + MQ_AT + 2 * UNIT, 4, threadIdx.x - 32, CHUNK_THREADS - 32, [&](int t) { return cs[t]; });
    put_keys(ks, out + K_AT, threadIdx.x - 32, CHUNK_THREADS - 32, [&](int t) { return rs[t]; });
    put_b(bs, out + B_AT, threadIdx.x - 32, CHUNK_THREADS - 32);
    for (int d = threadIdx.x - 32; d < RP; d += CHUNK_THREADS - 32) out[G_AT + d] = cs[CHUNK - 1];
  }
  __syncthreads();
  put_m_and_values<CHUNK_THREADS / 32>(as, [&](int l, int d) { return ks[l * KP + d] * cs[l]; }, v, ahead, vdim, out, warp, lane);
  pdl_trigger();  // at the end: the chain's blocks are few and long (see delta_prepare_kernel)
}

// ---- a decay per channel -------------------------------------------------------------------------------------------------
struct ChannelShape {
  static constexpr int Q = CHUNK * KP, G = 2 * CHUNK * KP, AS = 3 * CHUNK * KP, BS = AS + CHUNK * TP, FLOATS = BS + CHUNK * TP;
};

// A and B in halves of 16 tokens: on the diagonal a running product a column, behind it as products of q_i (k_i) times the decays from the
// half's start and k_j times those to its half's end.
__global__ void __launch_bounds__(CHUNK_THREADS, 3)
channel_delta_chunk_kernel(const float* __restrict__ qkv, const float* __restrict__ bd, const float* __restrict__ decay,
                           const int32_t* __restrict__ item_start, float* __restrict__ records, int items, int min_tokens, int G, int H,
                           int dim, int vdim, bool wide, bool wide_decay) {
  using Sh = ChannelShape;
  extern __shared__ __align__(16) float chunk_smem[];
  float *ks = chunk_smem, *qs = chunk_smem + Sh::Q, *gs = chunk_smem + Sh::G;
  float(*as)[TP] = reinterpret_cast<float(*)[TP]>(chunk_smem + Sh::AS);
  float(*bs)[TP] = reinterpret_cast<float(*)[TP]>(chunk_smem + Sh::BS);
  const int h = blockIdx.x % H, chunk = (int)(gridDim.x / H) - 1 - (int)(blockIdx.x / H);  // the first chunks last: the chain starts with them
  pdl_wait();
  int t0, n;
  if (!portions::find_chunk<CHUNK>(item_start, items, min_tokens, chunk, t0, n)) return;
  const int g = h / (H / G), C = 2 * G * dim + H * vdim;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* out = records + ((size_t)chunk * H + h) * record_floats(vdim);
  bring_rows(qs, qkv + (size_t)t0 * C + (size_t)g * dim, C, n, dim, wide);
  bring_rows(ks, qkv + (size_t)t0 * C + (size_t)(G + g) * dim, C, n, dim, wide);
  bring_rows(gs, decay + ((size_t)t0 * H + h) * dim, (long long)H * dim, n, dim, wide_decay);  // (0 where there is none: the key is 0 too)
  const float beta = lane < n ? bd[(size_t)(t0 + lane) * BD * H + h] : 0.f;
  copy_async_wait();
  __syncthreads();
  products_on_diagonal<true, false>(ks, qs, gs, as, bs, warp, lane);
  __syncthreads();
  // a channel a thread: the running products
  const int d = threadIdx.x;
  float kc[CHUNK], qc[CHUNK];  // K c, Q c
  {
    Product c, front, tail, upto;
    float f[CHUNK];
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) f[i] = i < n && d < dim ? gs[i * KP + d] : 1.f;
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
      const float q = qs[i * KP + d], k = ks[i * KP + d];
      c.times(f[i]);
      kc[i] = k * c.value();
      qc[i] = q * c.value();
      if (i >= HALF) {
        front.times(f[i]);
        qs[i * KP + d] = q * front.value();
        qs[(i - HALF) * KP + d] = k * front.value();   // (the first half's queries are done with)
      }
    }
    out[G_AT + d] = c.value();
#pragma unroll
    for (int i = CHUNK - 1; i >= 0; --i) {
      const float k = ks[i * KP + d];
      if (i < HALF) {
        gs[i * KP + d] = k * upto.value();  // to the end of the first half
        upto.times(f[i]);
      }
      ks[i * KP + d] = k * tail.value();
      tail.times(f[i]);
    }
  }
  __syncthreads();
  products_behind<true>(qs, gs, as, bs);  // (rows 0 .. 15 of the queries' place are the second half's keys now, 16 .. 31 its queries)
  __syncthreads();
#pragma unroll
  for (int i = 0; i < CHUNK; ++i) {
    qs[i * KP + d] = qc[i];
    gs[i * KP + d] = kc[i];
  }
  __syncthreads();
  const float* values = qkv + (size_t)t0 * C + 2 * (size_t)G * dim + (size_t)h * vdim;
  auto v = [&](int l, int c) { return l < n && c < vdim ? values[(size_t)l * C + c] : 0.f; };
  Columns ahead;
  ahead.fetch([&](int l, int c) { return v(l, 16 * warp + c); }, lane >> 2, lane & 3);
  if (warp == 0) {
    solve(as, beta, lane);
  } else {
    auto one = [](int) { return 1.f; };
    put_rows(qs, out + MQ_AT + 2 * UNIT, 4, threadIdx.x - 32, CHUNK_THREADS - 32, one);
    put_keys(ks, out + K_AT, threadIdx.x - 32, CHUNK_THREADS - 32, one);
    put_b(bs, out + B_AT, threadIdx.x - 32, CHUNK_THREADS - 32);
  }
  __syncthreads();
  put_m_and_values<CHUNK_THREADS / 32>(as, [&](int l, int c) { return gs[l * KP + c]; }, v, ahead, vdim, out, warp, lane);
  pdl_trigger();  // at the end, as in delta_chunk_kernel
}

// ---- the chain -----------------------------------------------------------------------------------------------------------
constexpr int PP = 2 * CHUNK + 8;   // of the shares: columns first
template <int TILES>
struct Chain {
  static constexpr int COLS = 16 * TILES;
  static constexpr int U_AT = WORKERS / 32 * COLS * PP, FLOATS = U_AT + TILES * 2 * UNIT;  // U per 16 columns and 16 tokens: fragments, as in a record
  static_assert(FLOATS * 4 <= 227 * 1024, "beyond a block's shared memory");
};


// Eight warps beside the workers make U, two columns of every 16 each, and the read-outs, eight tokens of 16 columns each.  A block is launched with 128 registers
// a thread; who gets how many of them, us for 2,000 tokens (16 columns a block) and for portions of 1,200 and 960 (32): workers 168 and makers 88 205 and 222, 152
// and 104 197 and 206, 144 and 112 189 and 214, 136 and 120 196 and 215.
constexpr int MAKERS = 256, DELTA_THREADS = WORKERS + MAKERS;
template <int TILES>
struct Registers {
  static constexpr int WORKER = TILES == 1 ? 144 : 152, MAKER = 256 - WORKER;
  static_assert(WORKERS == MAKERS, "what the workers get beyond 128 the makers give");
};

template <int TILES, typename T>
__global__ void __launch_bounds__(DELTA_THREADS, 1)
delta_chain_kernel(const float* __restrict__ records, const T* __restrict__ proj, long long P, float* __restrict__ state,
                   const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots, float* __restrict__ o, int items,
                   int all_chunks, int min_tokens, int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats) {
  using Sh = Chain<TILES>;
  constexpr int COLS = Sh::COLS, SHARES = WORKERS / 32;
  extern __shared__ __align__(16) float chain[];
  float* parts = chain;                                               // [SHARES][COLS][PP]: M S of the chunk's tokens, then Q c S
  uint32_t* us = reinterpret_cast<uint32_t*>(chain + Sh::U_AT);       // [TILES][2][3][32 lanes][4]
  const int C = 2 * G * dim + H * vdim;
  const int h = blockIdx.y, col0 = blockIdx.x * COLS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  pdl_wait();
  int item, first;  // (a block per portion: blocks for requests that have none would only be in the way, one fills an SM)
  if (!portions::find_portion<CHUNK>(item_start, items, min_tokens, blockIdx.z, item, first)) return;
  const int t0 = item_start[item], t1 = item_start[item + 1];
  const int chunks = (t1 - t0 + CHUNK - 1) / CHUNK;
  if (first + chunks > all_chunks) return;  // (the caller counted fewer than there are: no records for them)
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  float* base = state + (size_t)slot * slot_floats;
  float* S = base + (size_t)(K - 1) * C + (size_t)h * dim * vdim;
  const size_t size = record_floats(vdim);
  auto record_of = [&](int c) { return records + ((size_t)(first + c) * H + h) * size; };
  auto left_of = [&](int at) {  // 16 columns of U, 16 tokens
    Left u;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint4 x = *reinterpret_cast<const uint4*>(us + at * UNIT + p * TERM + 4 * lane);
      u.v[p][0] = x.x, u.v[p][1] = x.y, u.v[p][2] = x.z, u.v[p][3] = x.w;
    }
    return u;
  };
  auto unit = [&](const float* at, uint4 (&to)[3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p)  // (volatile: where they are asked for, not where they are used)
      asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(to[p].x), "=r"(to[p].y), "=r"(to[p].z), "=r"(to[p].w) : "l"(at + p * TERM + 4 * lane));
  };

  if (threadIdx.x < WORKERS) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Registers<TILES>::WORKER));
    uint4 mq[4][3], kr[2][3];  // asked for a chunk ahead, each as soon as the last one's is used up
    float2 g[2];
    const float* r = record_of(0);
    const size_t stride = (size_t)H * size;
    auto fetch_mq = [&](int first) {
#pragma unroll
      for (int p = 0; p < 2; ++p) unit(r + MQ_AT + (warp * 4 + first + p) * UNIT, mq[first + p]);
    };
    auto fetch_rest = [&] {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        unit(r + K_AT + (warp * 2 + m) * UNIT, kr[m]);
        g[m] = __ldg(reinterpret_cast<const float2*>(r + G_AT + 16 * warp + 8 * m + 2 * tg));
      }
    };
    fetch_mq(0);
    fetch_mq(2);
    fetch_rest();
    // S, columns first: columns gr and gr + 8 of every 16, channels 16 warp + 8 m + 2 tg and + 1
    float s[TILES][2][4];
    Left a[TILES];
    auto at = [&](int tile, int m, int e) -> float* {
      const int d = 16 * warp + 8 * m + 2 * tg + (e & 1), col = col0 + 16 * tile + gr + 8 * (e >> 1);
      return d < dim && col < vdim ? S + (size_t)d * vdim + col : nullptr;
    };
    auto take_apart = [&](int tile) {  // the sums of the second product lie as the left operand of the first
#pragma unroll
      for (int r = 0; r < 4; ++r) a[tile].put(r, split3(s[tile][r >> 1][2 * (r & 1)], s[tile][r >> 1][2 * (r & 1) + 1]));
    };
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float* p = at(tile, m, e);
          s[tile][m][e] = p ? *p : 0.f;
        }
      take_apart(tile);
    }
    auto share = [&](int half) {  // this warp's share of M S, or of Q c S
      Right b[4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          const uint4 v = mq[2 * half + (n >> 1)][p];
          b[n].v[p][0] = n & 1 ? v.z : v.x;
          b[n].v[p][1] = n & 1 ? v.w : v.y;
        }
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        float sum[4][4] = {}, small[4][4] = {};
        step<4>(sum, small, a[tile], b);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          float* to = parts + (warp * COLS + 16 * tile + gr) * PP + 8 * (4 * half + n) + 2 * tg;
          *reinterpret_cast<float2*>(to) = make_float2(sum[n][0] + small[n][0], sum[n][1] + small[n][1]);
          *reinterpret_cast<float2*>(to + 8 * PP) = make_float2(sum[n][2] + small[n][2], sum[n][3] + small[n][3]);
        }
      }
    };
    for (int c = 0; c < chunks; ++c) {
      share(0);
      if (c + 1 < chunks) {
        r += stride;
        fetch_mq(0);
      }
      __syncthreads();  // the others make U of it
      share(1);
      if (c + 1 < chunks) fetch_mq(2);
      __syncthreads();
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        float sum[2][2][4], small[2][2][4] = {};  // of either half of the tokens
        const Left u[2] = {left_of(2 * tile), left_of(2 * tile + 1)};
        Right b[2][2];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            b[0][m].v[p][0] = kr[m][p].x, b[0][m].v[p][1] = kr[m][p].y;
            b[1][m].v[p][0] = kr[m][p].z, b[1][m].v[p][1] = kr[m][p].w;
          }
        step_halves(sum, small, u, b);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            s[tile][m][e] = fmaf(e & 1 ? g[m].y : g[m].x, s[tile][m][e], (sum[0][m][e] + sum[1][m][e]) + (small[0][m][e] + small[1][m][e]));
        take_apart(tile);
      }
      if (c + 1 < chunks) fetch_rest();
    }
    pdl_trigger();  // at the end, as in delta_chunk_kernel
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (float* p = at(tile, m, e)) *p = s[tile][m][e];
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Registers<TILES>::MAKER));
    const int mine = warp - WORKERS / 32;
    const int tile = mine / (CHUNK / 8), eight = mine % (CHUNK / 8);  // of the read-outs: tokens 8 eight .. + 7 of every chunk, the tile's columns
    const int column = 2 * mine + (lane >> 4), vp = lane & 15;        // of U: this thread's column of every 16 and its pair of tokens
    uint4 b[3];
    float2 wv[TILES];
    auto fetch_b = [&](int c) {
      if (tile < TILES) unit(record_of(c) + B_AT + eight * UNIT, b);
    };
    auto fetch_values = [&](int c) {
#pragma unroll
      for (int n = 0; n < TILES; ++n) {
        const int col = col0 + 16 * n + column;
        wv[n] = col < (vdim + RUN - 1) / RUN * RUN ? __ldg(reinterpret_cast<const float2*>(record_of(c) + V_AT + (size_t)col * CHUNK) + vp) : make_float2(0.f, 0.f);
      }
    };
    auto sum_of_shares = [&](int col, int token) {
      float2 v[SHARES];
#pragma unroll
      for (int q = 0; q < SHARES; ++q) v[q] = *reinterpret_cast<const float2*>(parts + (q * COLS + col) * PP + token);
#pragma unroll
      for (int m = SHARES / 2; m > 0; m >>= 1)
#pragma unroll
        for (int q = 0; q < m; ++q) v[q].x += v[q + m].x, v[q].y += v[q + m].y;
      return v[0];
    };
    // A record's way from DRAM takes longer than a chunk: every block of a head asks for its share of the one after the next into L2.
    const size_t bytes = size * sizeof(float), share_bytes = (bytes / gridDim.x + 15) & ~(size_t)15, share_at = share_bytes * blockIdx.x;
    auto ask_for = [&](int c) {
      if (threadIdx.x == WORKERS && c < chunks && share_at < bytes)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const char*>(record_of(c)) + share_at),
                     "r"((uint32_t)min(share_bytes, bytes - share_at)) : "memory");
    };
    fetch_b(0);
    fetch_values(0);
    ask_for(1);
    for (int c = 0; c < chunks; ++c) {
      ask_for(c + 2);
      __syncthreads();
      const int n = t1 - (t0 + c * CHUNK);  // tokens left
#pragma unroll
      for (int m = 0; m < TILES; ++m) {  // U = W V - M S
        const float2 y = sum_of_shares(16 * m + column, 2 * vp);
        const Terms t = split3(2 * vp < n ? wv[m].x - y.x : 0.f, 2 * vp + 1 < n ? wv[m].y - y.y : 0.f);
        uint32_t* to = us + (m * 2 + (vp >> 3)) * UNIT + ((column & 7) * 4 + (vp & 3)) * 4 + (column >> 3) + 2 * ((vp >> 2) & 1);
#pragma unroll
        for (int p = 0; p < 3; ++p) to[p * TERM] = t.v[p];
      }
      __syncthreads();
      if (c + 1 < chunks) fetch_values(c + 1);  // as early as their registers are free: U is what all the others wait for
      if (tile < TILES) {
        float sum[2][1][4] = {}, small[2][1][4] = {};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (k && eight < 2) break;  // B is triangular
          Right x[1];
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            x[0].v[p][0] = k ? b[p].z : b[p].x;
            x[0].v[p][1] = k ? b[p].w : b[p].y;
          }
          step<1>(sum[k], small[k], left_of(tile * 2 + k), x);
        }
        float v[4];
        bool fine = true;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[e] = (sum[0][0][e] + sum[1][0][e]) + (small[0][0][e] + small[1][0][e]);
          fine = fine && is_finite(v[e]);
        }
        if (!fine) {
#pragma unroll 1
          for (int e = 0; e < 4; ++e) {
            const int in = gr + 8 * (e >> 1), i = 8 * eight + 2 * tg + (e & 1);
            float again = 0.f;
            const uint32_t* rec = reinterpret_cast<const uint32_t*>(record_of(c)) + B_AT + eight * UNIT;
#pragma unroll 1
            for (int j = 0; j <= i; ++j) {
              const int q = (j & 7) >> 1, k = j >> 4, h8 = (j >> 3) & 1;
              float x = 0.f, y = 0.f;
              for (int p = 2; p >= 0; --p) {
                x += term(rec[p * TERM + ((i & 7) * 4 + q) * 4 + 2 * k + h8], j & 1);
                y += term(us[(tile * 2 + k) * UNIT + p * TERM + ((in & 7) * 4 + q) * 4 + (in >> 3) + 2 * h8], j & 1);
              }
              again = fmaf(x, y, again);
            }
#pragma unroll
            for (int f = 0; f < 4; ++f)
              if (f == e && !is_finite(v[f])) v[f] = again;
          }
        }
        float* row = o + ((size_t)(t0 + c * CHUNK + 8 * eight + 2 * tg) * H + h) * vdim + col0 + 16 * tile + gr;
        const int left = n - (8 * eight + 2 * tg);  // tokens from this thread's first on
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float2 read = sum_of_shares(16 * tile + gr + 8 * r, CHUNK + 8 * eight + 2 * tg);  // Q c S
          if (col0 + 16 * tile + gr + 8 * r >= vdim) continue;
          if (left > 0) row[8 * r] = read.x + v[2 * r];
          if (left > 1) row[(size_t)H * vdim + 8 * r] = read.y + v[2 * r + 1];
        }
      }
      if (c + 1 < chunks) fetch_b(c + 1);
    }
    pdl_trigger();
  }
  if (blockIdx.x == 0 && h == 0) keep_conv_inputs<T>(proj, P, base, t0, t1, C, K);
}

template <int TILES, typename T>
int launch_chain(const float* records, const T* proj, long long ld, float* state, const int32_t* item_start, const int32_t* slots, float* o,
                 int items, int portions, int chunks, int min_tokens, int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats,
                 cudaStream_t stream) {
  constexpr int COLS = 16 * TILES, bytes = Chain<TILES>::FLOATS * (int)sizeof(float);
  auto kernel = delta_chain_kernel<TILES, T>;
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) PSB_REFUSE("delta_chain: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(kernel, dim3((vdim + COLS - 1) / COLS, H, portions), dim3(DELTA_THREADS), (size_t)bytes, stream, records, proj, ld, state, item_start, slots, o,
             items, chunks, min_tokens, G, H, dim, vdim, K, num_slots, slot_floats);
  PSB_LAUNCH_CHECK("delta_chain");
  return 0;
}

// Runs of columns a block takes.  One block fills an SM, so by rounds over the SMs: a chunk takes a block of one run 1.75 us and one of two 2.95 (the gated
// rule over 2,000 tokens of 16 heads, 128 blocks, and the other over 1,200 and 960 tokens, 128 blocks).
template <typename T>
int chain_of(const void* records, const void* proj, long long ld, void* state, const void* item_start, const void* slots, void* o, int items,
             int portions, int chunks, int min_tokens, int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats, cudaStream_t stream) {
  const long long heads = (long long)H * portions, sms = psb_current_sms();
  const long long rounds16 = (heads * ((vdim + 15) / 16) + sms - 1) / sms, rounds32 = (heads * ((vdim + 31) / 32) + sms - 1) / sms;
  auto launch = rounds32 * 59 < rounds16 * 35 ? launch_chain<2, T> : launch_chain<1, T>;
  return launch((const float*)records, (const T*)proj, ld, (float*)state, (const int32_t*)item_start, (const int32_t*)slots, (float*)o, items, portions, chunks,
                min_tokens, G, H, dim, vdim, K, num_slots, slot_floats, stream);
}

}  // namespace

// (dim, vdim) -> float32 numbers of a chunk's record of a head, 0 if the kernels are not built for the sizes
PSB_API int psb_delta_chunk_record(int dim, int vdim) {
  return dim >= 4 && dim <= RP && dim % 4 == 0 && vdim >= 4 && vdim % 4 == 0 && vdim <= (1 << 20) ? record_floats(vdim) : 0;
}

// () -> tokens of a chunk
PSB_API int psb_delta_chunk_tokens() { return CHUNK; }

// The rule over every portion of at least ``min_tokens`` tokens, from what psb_delta_prepare left; other tokens, and the slots of
// other portions, are left untouched.  records [chunks, H, psb_delta_chunk_record] float32, portions and chunks at least the number of these
// portions and of their chunks.
// (qkv, bd, proj bfloat16, ld, state, item_start, slots, records, o_out, items, portions, chunks, min_tokens, G, H, dim, vdim, K,
//  num_slots, slot_floats, stream)
PSB_API int psb_delta_chunks(const void* qkv, const void* bd, const void* proj, long long ld, void* state, const void* item_start,
                             const void* slots, void* records, void* o, int items, int portions, int chunks, int min_tokens, int G, int H,
                             int dim, int vdim, int K, int num_slots, long long slot_floats, cudaStream_t stream) {
  if (items < 0 || G < 1 || H < 1 || H % G || !psb_delta_chunk_record(dim, vdim)) PSB_REFUSE("delta_chunks: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS || min_tokens < 1 || num_slots < 1) PSB_REFUSE("delta_chunks: %d taps are outside [1, %d], or no tokens or slots", K, MAX_TAPS);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  if (ld < C || slot_floats != (K - 1) * C + (long long)H * dim * vdim) PSB_REFUSE("delta_chunks: the slot or the rows do not fit the sizes");
  if (H > 65535 || portions > 65535 || chunks < 0 || (long long)chunks * H > 0x7fffffffLL) PSB_REFUSE("delta_chunks: too many heads or requests for one launch");
  if (((uintptr_t)qkv | (uintptr_t)records | (uintptr_t)o) & 15) PSB_REFUSE("delta_chunks: operands must be 16-byte aligned");
  if (items == 0 || portions < 1 || chunks == 0) return 0;
  constexpr int bytes = ChunkShape::FLOATS * (int)sizeof(float);
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) PSB_REFUSE("delta_chunks: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(delta_chunk_kernel, dim3((unsigned)chunks * H), dim3(CHUNK_THREADS), (size_t)bytes, stream, (const float*)qkv, (const float*)bd, (const int32_t*)item_start,
             (float*)records, items, min_tokens, G, H, dim, vdim);
  PSB_LAUNCH_CHECK("delta_chunk");
  return chain_of<__nv_bfloat16>(records, proj, ld, state, item_start, slots, o, items, portions, chunks, min_tokens, G, H, dim, vdim, K, num_slots, slot_floats, stream);
}

// (dim, vdim) -> float32 numbers of a chunk's record of a head for the rule with a decay per channel, 0 if the kernels are not built for the sizes
PSB_API int psb_channel_delta_chunk_record(int dim, int vdim) { return dim >= 1 && dim <= RP && vdim >= 1 && vdim <= 4096 ? record_floats(vdim) : 0; }

// The rule with a decay per channel: as above, with decay float32 [T, H, dim] and a projection of either type.
// (qkv, bd, decay, proj, dtype, ld, state, item_start, slots, records, o_out, items, portions, chunks, min_tokens, G, H, dim, vdim, K,
//  num_slots, slot_floats, stream)
PSB_API int psb_channel_delta_chunks32(const void* qkv, const void* bd, const void* decay, const void* proj, int dtype, long long ld, void* state,
                                       const void* item_start, const void* slots, void* records, void* o, int items, int portions, int chunks, int min_tokens,
                                       int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats, cudaStream_t stream) {
  if (items < 0 || G < 1 || H < 1 || H % G || !psb_channel_delta_chunk_record(dim, vdim)) PSB_REFUSE("channel_delta_chunks: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS || min_tokens < 1 || num_slots < 1) PSB_REFUSE("channel_delta_chunks: %d taps are outside [1, %d], or no tokens or slots", K, MAX_TAPS);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  if (ld < C || slot_floats != (K - 1) * C + (long long)H * dim * vdim) PSB_REFUSE("channel_delta_chunks: the slot or the rows do not fit the sizes");
  if (H > 65535 || portions > 65535 || chunks < 0 || (long long)chunks * H > 0x7fffffffLL) PSB_REFUSE("channel_delta_chunks: too many heads or requests for one launch");
  if (((uintptr_t)records | (uintptr_t)o) & 15) PSB_REFUSE("channel_delta_chunks: records and read-out must be 16-byte aligned");
  if (items == 0 || portions < 1 || chunks == 0) return 0;
  constexpr int bytes = ChannelShape::FLOATS * (int)sizeof(float);
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(channel_delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
      PSB_REFUSE("channel_delta_chunks: cannot raise the shared-memory limit");
    configured.set();
  }
  const bool wide_decay = dim % 4 == 0 && ((uintptr_t)decay & 15) == 0, wide = dim % 4 == 0 && C % 4 == 0 && ((uintptr_t)qkv & 15) == 0;
  psb_launch(channel_delta_chunk_kernel, dim3((unsigned)chunks * H), dim3(CHUNK_THREADS), (size_t)bytes, stream, (const float*)qkv, (const float*)bd, (const float*)decay,
             (const int32_t*)item_start, (float*)records, items, min_tokens, G, H, dim, vdim, wide, wide_decay);
  PSB_LAUNCH_CHECK("channel_delta_chunk");
  PSB_DISPATCH_DTYPE(dtype, T_, {
    return chain_of<T_>(records, proj, ld, state, item_start, slots, o, items, portions, chunks, min_tokens, G, H, dim, vdim, K, num_slots, slot_floats, stream);
  });
  return 0;
}
