// Gated linear attention (linear_attention.cu) over long portions of bfloat16 projections, 32 tokens at a time on the tensor cores,
// float32 throughout:
//
//     S <- diag(alpha_t) S + k_t v_t^T,    o_t = S^T q_t * scale.
//
// With c_i = alpha_1 .. alpha_i from a chunk's start, r_j = alpha_(j+1) .. alpha_32, per key channel, and S the state before the chunk,
//     O = (Q c) S + P V,  P_ij = sum_d q_i k_j alpha_(j+1) .. alpha_i  (j <= i),    S <- diag(c_32) S + (K r)^T V.
//   linear_chunk_kernel   a block per chunk and head, all chunks of the step side by side: P, Q c, K r, c_32 and V as the chain takes them, 64 KB;
//   linear_chain_kernel   a block per 16 or 32 columns of a head's state and portion walks the chunks: eight warps hold 16 key channels of S
//                         each, in registers, multiply Q c by it (eight shares, through shared memory) and bring it up to date, four more
//                         add the shares and P V up behind them.  What a chunk brings goes straight into the registers of those who use it, a chunk ahead.
// Decays are only ever multiplied, never divided by, and the running ones of a chunk carry what the roundings lose.  float32 numbers enter the tensor cores in three
// terms (chunk_products.cuh), the values, which are bfloat16, as they are.
// P is zero above the diagonal, and zero times a value that is not finite is not zero: a result that comes out not finite is made
// again from the tokens up to its own, and from the state as it is, whose terms are no sum where it is infinite.
// A float32 projection's values would need terms too; those stay with the other kernels.
//
// Distances from float64, token by token and here (150 and 700 tokens): read-outs 1.2e-7 and 1.0e-7, states 0.95e-7 and 0.59e-7.  A decay product between two
// tokens of the same sixteen is rounded once (in plain float32, 5 us less for the call below, it was up to 3.9 times as far off).
//
// What bounds it: the chain, by what a chunk brings from L2 (64 KB an SM and chunk, 1.1 us) and the latency of its steps.  1,811 tokens of 16 heads of 128:
// chunk kernel 47 us, chain 64; chunks of 64 tokens all side by side, the states they start from in a pass between two kernels, took 31, 11 and 87 us
// and were bound by the read-out's phases, one block an SM, in four rounds.  Two chunks ahead through shared memory: no faster.
#include "chunk_products.cuh"

namespace {
using namespace chunks;

// A chunk's record of a head, 32-bit words: Q c (per 16 channels, per two eights of tokens, both fragments of either), K r (per 16 channels, per eight
// of them, the fragments of either half of the tokens), P (per eight of its rows, the same), c_32 [128], and V per 16 columns and half of the tokens as
// left operands' fragments.
constexpr int Q_AT = 0, K_AT = Q_AT + (RP / 16) * 2 * UNIT, P_AT = K_AT + (RP / 16) * 2 * UNIT, G_AT = P_AT + (CHUNK / 8) * UNIT, V_AT = G_AT + RP;
__host__ __device__ constexpr int record_floats(int vdim) { return V_AT + (vdim + 15) / 16 * 2 * TERM; }

// 32 rows of bfloat16 (row pitch ld, ``dim`` numbers in fours, zeros beyond them and beyond n rows) as float32 [32][KP]
__device__ __forceinline__ void widen_rows(float* dst, const __nv_bfloat16* __restrict__ src, long long ld, int n, int dim) {
  constexpr int EACH = CHUNK * RP / 4 / CHUNK_THREADS;
  uint2 raw[EACH];
#pragma unroll
  for (int e = 0; e < EACH; ++e) {  // asked for together
    const int i = threadIdx.x + e * CHUNK_THREADS, t = i / (RP / 4), d = (i % (RP / 4)) * 4;
    raw[e] = make_uint2(0, 0);
    if (t < n && d < dim) raw[e] = *reinterpret_cast<const uint2*>(src + (size_t)t * ld + d);
  }
#pragma unroll
  for (int e = 0; e < EACH; ++e) {
    const int i = threadIdx.x + e * CHUNK_THREADS, t = i / (RP / 4), d = (i % (RP / 4)) * 4;
    *reinterpret_cast<float4*>(dst + t * KP + d) = make_float4(__uint_as_float(raw[e].x << 16), __uint_as_float(raw[e].x & 0xffff0000u),
                                                               __uint_as_float(raw[e].y << 16), __uint_as_float(raw[e].y & 0xffff0000u));
  }
}

struct ChunkShape {
  static constexpr int Q = CHUNK * KP, G = 2 * CHUNK * KP, PS = 3 * CHUNK * KP, FLOATS = PS + CHUNK * TP;
};

__global__ void __launch_bounds__(CHUNK_THREADS, 3)
linear_chunk_kernel(const __nv_bfloat16* __restrict__ proj, long long ld, const float* __restrict__ alpha, const int32_t* __restrict__ item_start,
                    float* __restrict__ records, int items, int min_tokens, int H, int dim, int vdim) {
  using Sh = ChunkShape;
  extern __shared__ __align__(16) float chunk_smem[];
  float *ks = chunk_smem, *qs = chunk_smem + Sh::Q, *gs = chunk_smem + Sh::G;
  float(*ps)[TP] = reinterpret_cast<float(*)[TP]>(chunk_smem + Sh::PS);
  pdl_wait();
  int t0, n;
  const int h = blockIdx.x % H, chunk = blockIdx.x / H;
  if (!portions::find_chunk<CHUNK>(item_start, items, min_tokens, chunk, t0, n)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  float* out = records + ((size_t)chunk * H + h) * record_floats(vdim);
  const __nv_bfloat16* rows = proj + (size_t)t0 * ld;
  bring_rows(gs, alpha + ((size_t)t0 * H + h) * dim, (long long)H * dim, n, dim, true);  // (0 where there is none: q and k are 0 too)
  widen_rows(qs, rows + (size_t)h * dim, ld, n, dim);
  widen_rows(ks, rows + (size_t)(H + h) * dim, ld, n, dim);
  delta::copy_async_wait();
  __syncthreads();
  products_on_diagonal<false, true>(ks, qs, gs, nullptr, ps, warp, lane);
  // the values, columns first: nobody else waits for them
  const uint16_t* values = reinterpret_cast<const uint16_t*>(rows + 2 * (size_t)H * dim + (size_t)h * vdim);
#pragma unroll 2
  for (int i = threadIdx.x; i < (vdim + 15) / 16 * 2 * 32; i += CHUNK_THREADS) {
    const int col0 = (i >> 6) * 16, k = (i >> 5) & 1;  // (i & 31 is the lane)
    uint32_t w[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int col = col0 + gr + 8 * (r & 1), t = 16 * k + 8 * (r >> 1) + 2 * tg;
      const uint32_t a = t < n && col < vdim ? values[(size_t)t * ld + col] : 0, b = t + 1 < n && col < vdim ? values[(size_t)(t + 1) * ld + col] : 0;
      w[r] = a | b << 16;
    }
    *reinterpret_cast<uint4*>(out + V_AT + (i >> 5) * TERM + 4 * lane) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  __syncthreads();
  // a channel a thread: the running products
  const int d = threadIdx.x;
  float qc[CHUNK];  // Q c
  {
    Product c, front, tail, upto;
    float f[CHUNK];
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) f[i] = i < n && d < dim ? gs[i * KP + d] : 1.f;
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
      const float q = qs[i * KP + d];
      c.times(f[i]);
      qc[i] = q * c.value();
      if (i >= HALF) {
        front.times(f[i]);
        qs[i * KP + d] = q * front.value();
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
  products_behind<false>(qs + HALF * KP, gs, nullptr, ps);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < CHUNK; ++i) qs[i * KP + d] = qc[i];
  __syncthreads();
  auto one = [](int) { return 1.f; };
  put_rows(qs, out + Q_AT, 2, threadIdx.x, CHUNK_THREADS, one);
  put_keys(ks, out + K_AT, threadIdx.x, CHUNK_THREADS, one);
  put_b(ps, out + P_AT, threadIdx.x, CHUNK_THREADS);
  pdl_trigger();  // at the end: the chain's blocks are few and long
}

constexpr int PP = CHUNK + 8;  // of the shares: columns first
constexpr int SP = RP + 8;     // of the state: columns first, as pairs of channels
template <int TILES>
struct Chain {
  static constexpr int COLS = 16 * TILES, SHARES = WORKERS / 32, S_AT = 2 * SHARES * COLS * PP, FLOATS = S_AT + 2 * COLS * SP;  // of two chunks
  static_assert(FLOATS * 4 <= 227 * 1024, "beyond a block's shared memory");
};
// One step of sixteen terms of N sums whose left operand is bfloat16 as it is (see step).
template <int N>
__device__ __forceinline__ void step_whole(float (&sum)[N][4], float (&small)[N][4], const uint32_t (&a)[4], const Right (&b)[N]) {
  const float zero[4] = {};
  float d[N][4];
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a, b[n].v[2][0], b[n].v[2][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(d[n], a, b[n].v[0][0], b[n].v[0][1], zero);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a, b[n].v[1][0], b[n].v[1][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[n][e] += d[n][e];
}

// the number whose first term lies in this word of a record
__device__ __forceinline__ float number(const uint32_t* word, int half) {
  const float first = term(word[0], half);
  return is_finite(first) ? first + (term(word[TERM], half) + term(word[2 * TERM], half)) : first;
}

template <int TILES>
__global__ void __launch_bounds__(CHAIN_THREADS, 1)
linear_chain_kernel(const float* __restrict__ records, float* __restrict__ state, long long slot_floats, const int32_t* __restrict__ item_start,
                    const int32_t* __restrict__ slots, float* __restrict__ o, int items, int all_chunks, int min_tokens, int H, int dim, int vdim,
                    int num_slots, float scale) {
  using Sh = Chain<TILES>;
  constexpr int COLS = Sh::COLS, SHARES = Sh::SHARES;
  extern __shared__ __align__(16) float chain[];  // [2][SHARES][COLS][PP], and the state each chunk starts from, [2][COLS][SP]
  const int h = blockIdx.y, col0 = blockIdx.x * COLS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  pdl_wait();
  int item, first;
  if (!portions::find_portion<CHUNK>(item_start, items, min_tokens, blockIdx.z, item, first)) return;
  const int t0 = item_start[item], t1 = item_start[item + 1];
  const int chunks = (t1 - t0 + CHUNK - 1) / CHUNK;
  if (first + chunks > all_chunks) return;  // (the caller counted fewer than there are: no records for them)
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  float* S = state + (size_t)slot * slot_floats + (size_t)h * dim * vdim;
  const size_t size = record_floats(vdim), stride = (size_t)H * size;
  const float* r = records + ((size_t)first * H + h) * size;
  auto fetch4 = [&](const float* at) {  // (volatile: where it is asked for, not where it is used)
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(at + 4 * lane));
    return v;
  };
  auto unit = [&](const float* at, uint4 (&to)[3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) to[p] = fetch4(at + p * TERM);
  };
  uint4 vt[TILES][2];  // V of the chunk: columns gr and gr + 8 of every 16
  auto fetch_values = [&] {
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
      for (int k = 0; k < 2; ++k)
        vt[tile][k] = col0 + 16 * tile < vdim ? fetch4(r + V_AT + ((size_t)(col0 / 16 + tile) * 2 + k) * TERM) : make_uint4(0, 0, 0, 0);
  };

  if (threadIdx.x < WORKERS) {
    uint4 qc[2][3], kr[2][3];
    float2 g[2];
    auto fetch_queries = [&] {
#pragma unroll
      for (int p = 0; p < 2; ++p) unit(r + Q_AT + (warp * 2 + p) * UNIT, qc[p]);
    };
    auto fetch_keys = [&] {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        unit(r + K_AT + (warp * 2 + m) * UNIT, kr[m]);
        g[m] = __ldg(reinterpret_cast<const float2*>(r + G_AT + 16 * warp + 8 * m + 2 * tg));
      }
    };
    fetch_queries();
    fetch_keys();
    fetch_values();
    // S, columns first: columns gr and gr + 8 of every 16, channels 16 warp + 8 m + 2 tg and + 1
    float s[TILES][2][4];
    auto at = [&](int tile, int m, int e) -> float* {
      const int d = 16 * warp + 8 * m + 2 * tg + (e & 1), col = col0 + 16 * tile + gr + 8 * (e >> 1);
      return d < dim && col < vdim ? S + (size_t)d * vdim + col : nullptr;
    };
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float* p = at(tile, m, e);
          s[tile][m][e] = p ? *p : 0.f;
        }
    for (int c = 0; c < chunks; ++c) {
      float* parts = chain + (c & 1) * SHARES * COLS * PP;
      {  // this warp's share of Q c S
        Right b[4];
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            const uint4 v = qc[n >> 1][p];
            b[n].v[p][0] = n & 1 ? v.z : v.x;
            b[n].v[p][1] = n & 1 ? v.w : v.y;
          }
#pragma unroll
        for (int tile = 0; tile < TILES; ++tile) {
          float* held = chain + Sh::S_AT + ((c & 1) * COLS + 16 * tile + gr) * SP + 16 * warp + 2 * tg;  // for read-outs that are made again
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) *reinterpret_cast<float2*>(held + 8 * r * SP + 8 * m) = make_float2(s[tile][m][2 * r], s[tile][m][2 * r + 1]);
          Left a;  // the state's sums lie as a left operand
#pragma unroll
          for (int e = 0; e < 4; ++e) a.put(e, split3(s[tile][e >> 1][2 * (e & 1)], s[tile][e >> 1][2 * (e & 1) + 1]));
          float sum[4][4] = {}, small[4][4] = {};
          step<4>(sum, small, a, b);
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            float* to = parts + (warp * COLS + 16 * tile + gr) * PP + 8 * n + 2 * tg;
            *reinterpret_cast<float2*>(to) = make_float2(sum[n][0] + small[n][0], sum[n][1] + small[n][1]);
            *reinterpret_cast<float2*>(to + 8 * PP) = make_float2(sum[n][2] + small[n][2], sum[n][3] + small[n][3]);
          }
        }
      }
      const float* next = r + stride;
      if (c + 1 < chunks) {
        r = next;
        fetch_queries();
      }
      __syncthreads();  // (the shares of the chunk before last have been added up)
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        float sum[2][2][4] = {}, small[2][2][4] = {};  // of either half of the tokens
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint32_t a[4] = {vt[tile][k].x, vt[tile][k].y, vt[tile][k].z, vt[tile][k].w};
          Right b[2];
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int p = 0; p < 3; ++p) {
              b[m].v[p][0] = k ? kr[m][p].z : kr[m][p].x;
              b[m].v[p][1] = k ? kr[m][p].w : kr[m][p].y;
            }
          step_whole<2>(sum[k], small[k], a, b);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            s[tile][m][e] = fmaf(e & 1 ? g[m].y : g[m].x, s[tile][m][e], (sum[0][m][e] + sum[1][m][e]) + (small[0][m][e] + small[1][m][e]));
      }
      if (c + 1 < chunks) {
        fetch_keys();
        fetch_values();
      }
    }
    pdl_trigger();  // at the end, as in linear_chunk_kernel
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (float* p = at(tile, m, e)) *p = s[tile][m][e];
  } else {
    const int eight = warp - WORKERS / 32;  // tokens 8 eight .. + 7 of every chunk
    uint4 b[3];
    unit(r + P_AT + eight * UNIT, b);
    fetch_values();
    for (int c = 0; c < chunks; ++c) {
      const float* parts = chain + (c & 1) * SHARES * COLS * PP;
      float of_values[TILES][4];  // P V: columns gr and gr + 8, tokens 2 tg and 2 tg + 1
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        float sum[2][1][4] = {}, small[2][1][4] = {};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (k && eight < 2) break;  // P is triangular
          const uint32_t a[4] = {vt[tile][k].x, vt[tile][k].y, vt[tile][k].z, vt[tile][k].w};
          Right x[1];
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            x[0].v[p][0] = k ? b[p].z : b[p].x;
            x[0].v[p][1] = k ? b[p].w : b[p].y;
          }
          step_whole<1>(sum[k], small[k], a, x);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) of_values[tile][e] = (sum[0][0][e] + sum[1][0][e]) + (small[0][0][e] + small[1][0][e]);
      }
      const uint32_t* record = reinterpret_cast<const uint32_t*>(r);
      if (c + 1 < chunks) {
        r += stride;
        unit(r + P_AT + eight * UNIT, b);
        fetch_values();
      }
      __syncthreads();
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
          const int in = gr + 8 * e2, col = col0 + 16 * tile + in;
          float2 v[SHARES];
#pragma unroll
          for (int q = 0; q < SHARES; ++q) v[q] = *reinterpret_cast<const float2*>(parts + (q * COLS + 16 * tile + in) * PP + 8 * eight + 2 * tg);
#pragma unroll
          for (int m = SHARES / 2; m > 0; m >>= 1)
#pragma unroll
            for (int q = 0; q < m; ++q) v[q].x += v[q + m].x, v[q].y += v[q + m].y;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = 8 * eight + 2 * tg + e, t = t0 + c * CHUNK + i;
            float of_state = e ? v[0].y : v[0].x;
            float y = of_state + of_values[tile][2 * e2 + e];
            if (!is_finite(y) && col < vdim) {
              if (!is_finite(of_state)) {  // an infinite number's lower terms are not zero: the state as it is, until it is not a number
                const float* held = chain + Sh::S_AT + ((c & 1) * COLS + 16 * tile + in) * SP;
                of_state = 0.f;
#pragma unroll 1
                for (int d = 0; d < RP && of_state == of_state; ++d)
                  of_state = fmaf(number(record + Q_AT + ((d >> 4) * 2 + (i >> 4)) * UNIT + ((i & 7) * 4 + ((d & 7) >> 1)) * 4 + 2 * ((i >> 3) & 1) + ((d >> 3) & 1), d & 1),
                                  held[d], of_state);
              }
              float again = 0.f;
#pragma unroll 1
              for (int j = 0; j <= i; ++j) {
                const int q = (j & 7) >> 1, k = j >> 4, h8 = (j >> 3) & 1;
                again = fmaf(number(record + P_AT + eight * UNIT + ((i & 7) * 4 + q) * 4 + 2 * k + h8, j & 1),
                             term(record[V_AT + ((size_t)(col0 / 16 + tile) * 2 + k) * TERM + ((in & 7) * 4 + q) * 4 + (in >> 3) + 2 * h8], j & 1), again);
              }
              y = of_state + again;
            }
            if (t < t1 && col < vdim) o[((size_t)t * H + h) * vdim + col] = y * scale;
          }
        }
    }
    pdl_trigger();
  }
}

template <int TILES>
int launch_chain(const float* records, float* state, long long slot_floats, const int32_t* item_start, const int32_t* slots, float* o, int items, int portions,
                 int chunks, int min_tokens, int H, int dim, int vdim, int num_slots, float scale, cudaStream_t stream) {
  constexpr int bytes = Chain<TILES>::FLOATS * (int)sizeof(float), COLS = Chain<TILES>::COLS;
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(linear_chain_kernel<TILES>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) PSB_REFUSE("linear_chunks: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(linear_chain_kernel<TILES>, dim3((vdim + COLS - 1) / COLS, H, portions), dim3(CHAIN_THREADS), (size_t)bytes, stream, records, state, slot_floats,
             item_start, slots, o, items, chunks, min_tokens, H, dim, vdim, num_slots, scale);
  PSB_LAUNCH_CHECK("linear_chain");
  return 0;
}

}  // namespace

// (dim, vdim) -> float32 numbers of a chunk's record of a head, 0 if these kernels do not take the sizes
PSB_API int psb_linear_chunk_record(int dim, int vdim) { return dim >= 4 && dim <= RP && dim % 4 == 0 && vdim >= 4 && vdim <= RP && vdim % 4 == 0 ? record_floats(vdim) : 0; }

// () -> tokens of a chunk
PSB_API int psb_linear_chunk_tokens() { return CHUNK; }

// Every portion of at least ``min_tokens`` tokens, and its slot; other tokens and slots are left untouched.  records [chunks, H,
// psb_linear_chunk_record] float32 is scratch, portions and chunks at least the number of these portions and of their chunks.
// (proj bfloat16, ld, alpha, state, slot_floats, item_start, slots, records, o, items, portions, chunks, min_tokens, H, dim, vdim, num_slots,
//  scale, stream)
PSB_API int psb_linear_chunks(const void* proj, long long ld, const void* alpha, void* state, long long slot_floats,
                              const void* item_start, const void* slots, void* records, void* o, int items, int portions, int chunks,
                              int min_tokens, int H, int dim, int vdim, int num_slots, float scale, cudaStream_t stream) {
  if (items < 0 || H < 1 || num_slots < 1 || min_tokens < 1 || !psb_linear_chunk_record(dim, vdim)) PSB_REFUSE("linear_chunks: bad sizes H=%d dim=%d vdim=%d", H, dim, vdim);
  if (ld < 2LL * H * dim + (long long)H * vdim || ld % 4) PSB_REFUSE("linear_chunks: row stride %lld is shorter than the row or no multiple of 4", ld);
  if (slot_floats < (long long)H * dim * vdim) PSB_REFUSE("linear_chunks: a slot of %lld numbers does not hold the state", slot_floats);
  if (((uintptr_t)proj & 7) || (((uintptr_t)alpha | (uintptr_t)records) & 15)) PSB_REFUSE("linear_chunks: operands are not aligned");
  if (H > 65535 || portions > 65535 || (long long)chunks * H > 0x7fffffffLL) PSB_REFUSE("linear_chunks: too many heads, requests or chunks for one launch");
  if (items == 0 || portions < 1 || chunks < 1) return 0;
  constexpr int bytes = ChunkShape::FLOATS * (int)sizeof(float);
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(linear_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) PSB_REFUSE("linear_chunks: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(linear_chunk_kernel, dim3((unsigned)chunks * H), dim3(CHUNK_THREADS), (size_t)bytes, stream, (const __nv_bfloat16*)proj, ld, (const float*)alpha,
             (const int32_t*)item_start, (float*)records, items, min_tokens, H, dim, vdim);
  PSB_LAUNCH_CHECK("linear_chunk");
  // runs of columns a block takes: as for the delta rules' chain (delta_chunks.cu)
  const long long heads = (long long)H * portions, sms = psb_current_sms();
  const long long rounds16 = (heads * ((vdim + 15) / 16) + sms - 1) / sms, rounds32 = (heads * ((vdim + 31) / 32) + sms - 1) / sms;
  auto launch = rounds32 * 31 < rounds16 * 20 ? launch_chain<2> : launch_chain<1>;
  return launch((const float*)records, (float*)state, slot_floats, (const int32_t*)item_start, (const int32_t*)slots, (float*)o, items, portions, chunks,
                min_tokens, H, dim, vdim, num_slots, scale, stream);
}
