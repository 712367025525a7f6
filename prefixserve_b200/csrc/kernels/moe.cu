// A routed feed-forward (mixture of experts): router, grouping of the chosen (token, expert) pairs by expert, the two
// products of every expert over its own rows, and the weighted sum.
//
// moe_route_kernel (a warp per token): scores s of the float32 router logits z [T, E(+1)]: sigmoid(z), or
// (``softmax_scores``) the softmax of z over all experts; the choice is made on s + correction, the weights on s.
// With ``groups`` > 1 the experts form that many equal groups of neighbours; a group's score is the sum of its two
// largest choice scores, or (``group_by_max``) its largest, and only the experts of the ``keep`` best groups can be
// chosen.  The ``top`` largest choice scores win (the lower index on a tie); their weights are
// s / (sum of the chosen s + 1e-20) * scale, or (``normalize`` 0) s * scale as it is.
//
// moe_group_kernel (one block or one cluster): counts the pairs of every expert, lays the experts' rows out one after the other
// (offsets [E + 1]; every expert's first row a multiple of ``pad``, the rows in between belong to nobody) and gives
// every pair its row: row_pair[row] = t * top + slot (-1: nobody's), pair_row[t * top + slot] = row; tile_expert
// names the expert of every run of ``pad`` rows (-1 beyond the last).  Which row of its expert a pair gets does not
// matter: every row of the products below is computed by itself.
//
// moe_gather_kernel: the rows of x in that order (nobody's rows are not written), for the tensor-core product that reads
// its left operand through a tensor map (gemm_tcgen05.cu, grouped).
//
// moe_gemm_kernel: C[row] = act(A[src(row)] . W[e]^T) for the rows of expert e, float32 sums over k in increasing
// order on the CUDA cores, in 64 x 64 tiles; a row tile never spans two experts (the grid has one row tile more per
// expert than the rows alone would need, whatever the routing turns out to be, so its shape does not depend on it).
// ``gather``: A's row is the pair's token (first product) or the row itself (second).  act: none or relu squared.
//
// ``glu`` (second product of gated experts): A holds, per row, K gate values followed by K up values as the first
// product left them, and the operand is g * sigmoid(alpha g) * (u + offset) with g = min(gate, limit), u = clamp(up,
// -limit, limit), taken in float32 as the row is read and rounded to A's type: the gate costs no pass of its own, and a
// row that belongs to nobody is never read.
//
// ``glu`` 2 is the SiLU gate, silu(r g) * (r u), with r the row's weight where a pair's weight multiplies what its expert
// reads (``row_weight``, by row: the first product is linear, so the weight may as well multiply its sums) and one otherwise.
//
// moe_mma_kernel: the same product for bfloat16 operands on the tensor cores (mma.sync m16n8k16, float32 sums).
// moe_fewrows_kernel: the same for steps with no more than eight rows an expert on average (see there).
//
// moe_combine_kernel: out[t] = sum over slots of weight[t, slot] * Y[pair_row[t, slot]]  (+ sigmoid(gate[t]) *
// shared[t] for a shared expert that every token uses), float32 sums in slot order, rounded to the compute type; without
// weights the rows are added as they are.
#include <algorithm>
#include <cfloat>

#include "common.cuh"

namespace {

constexpr int MAX_EXPERTS = 512;
constexpr int MAX_TOP = 32;

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }

constexpr int ROUTE_WARPS = 4;

__global__ void __launch_bounds__(ROUTE_WARPS * 32)
moe_route_kernel(const float* __restrict__ z, int ldz, const float* __restrict__ correction, int32_t* __restrict__ chosen,
                 float* __restrict__ weight, int T, int E, int top, int groups, int keep, float scale, int softmax_scores,
                 int group_by_max, int normalize) {
  extern __shared__ float sm[];  // per warp: s[E], choice[E], group score[groups]
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * ROUTE_WARPS + warp;
  if (t >= T) return;
  float* s = sm + (size_t)warp * (2 * E + groups);
  float* choice = s + E;
  float* gscore = choice + E;
  float z_top = -FLT_MAX, z_sum = 1.f;
  if (softmax_scores) {
    for (int e = lane; e < E; e += 32) z_top = fmaxf(z_top, z[(size_t)t * ldz + e]);
    z_top = warp_max(z_top);
    float part = 0.f;
    for (int e = lane; e < E; e += 32) part += expf(z[(size_t)t * ldz + e] - z_top);
    z_sum = warp_sum(part);
  }
  for (int e = lane; e < E; e += 32) {
    const float v = softmax_scores ? expf(z[(size_t)t * ldz + e] - z_top) / z_sum : sigmoidf_(z[(size_t)t * ldz + e]);
    s[e] = v;
    choice[e] = v + (correction ? correction[e] : 0.f);
  }
  __syncwarp();
  const int per = E / groups;
  if (groups > 1 && keep < groups) {
    for (int g = lane; g < groups; g += 32) {
      float a = -FLT_MAX, b = -FLT_MAX;  // the two largest of the group
      for (int e = g * per; e < (g + 1) * per; ++e) {
        const float c = choice[e];
        if (c > a) { b = a; a = c; }
        else if (c > b) b = c;
      }
      gscore[g] = (per > 1 && !group_by_max) ? a + b : a;
    }
    __syncwarp();
    // a group is dropped when at least ``keep`` groups come before it (larger score, or equal and a lower index)
    for (int g = lane; g < groups; g += 32) {
      int before = 0;
      const float mine = gscore[g];
      for (int o = 0; o < groups; ++o) before += (gscore[o] > mine) || (gscore[o] == mine && o < g);
      if (before >= keep)
        for (int e = g * per; e < (g + 1) * per; ++e) choice[e] = -INFINITY;
    }
    __syncwarp();
  }
  // the ``top`` best, one after the other: every lane looks at its share, a butterfly finds the winner
  float total = 0.f;
  int mine_e = -1;
  float mine_s = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float c = choice[e];
      if (c > best || (c == best && e < at && c != -INFINITY)) { best = c; at = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
    if (at >= E) at = 0;  // fewer candidates than ``top`` (refused on the host); keep the index inside the table
    const float sv = s[at];
    total += sv;
    if (lane == k % 32 && k / 32 == 0) { mine_e = at; mine_s = sv; }
    __syncwarp();
    if (lane == 0) choice[at] = -INFINITY;
    __syncwarp();
  }
  if (lane < top) {
    chosen[(size_t)t * top + lane] = mine_e;
    weight[(size_t)t * top + lane] = (normalize ? mine_s / (total + 1e-20f) : mine_s) * scale;
  }
}

// Long steps: the pairs are dealt out among the CTAs of one cluster.  Each counts its own, learns the others' counts through distributed shared memory and so
// knows where its pairs of every expert start.  Bound by the latency of its steps: 8,148 pairs of 32 experts 5.9 us, 15 as a single block; with counters
// a warp and match_any instead of atomics 19.
constexpr int GROUP_CTAS = 8, GROUP_THREADS = 512, GROUP_HELD = 4;

__global__ void __launch_bounds__(GROUP_THREADS)
moe_group_kernel(const int32_t* __restrict__ chosen, int32_t* __restrict__ offsets, int32_t* __restrict__ row_pair,
                 int32_t* __restrict__ pair_row, int32_t* __restrict__ tile_expert, int pairs, int E, int pad, int rows_room,
                 const float* __restrict__ weight, float* __restrict__ row_weight) {
  __shared__ int count[MAX_EXPERTS];
  __shared__ int cursor[MAX_EXPERTS];
  __shared__ int first_row[MAX_EXPERTS];
  pdl_trigger();
  pdl_wait();
  const int ctas = gridDim.x, rank = blockIdx.x;  // the cluster is the grid
  for (int e = threadIdx.x; e < E; e += GROUP_THREADS) count[e] = 0;
  __syncthreads();
  const int per = (pairs + ctas - 1) / ctas, first = rank * per, last = min(pairs, first + per);
  int held[GROUP_HELD];  // the experts of this thread's first pairs
  auto expert_of = [&](int i) { return min(max(chosen[i], 0), E - 1); };
#pragma unroll
  for (int k = 0; k < GROUP_HELD; ++k) {
    const int i = first + k * GROUP_THREADS + threadIdx.x;
    held[k] = i < last ? expert_of(i) : -1;
  }
#pragma unroll
  for (int k = 0; k < GROUP_HELD; ++k)
    if (held[k] >= 0) atomicAdd(&count[held[k]], 1);
  for (int i = first + GROUP_HELD * GROUP_THREADS + threadIdx.x; i < last; i += GROUP_THREADS) atomicAdd(&count[expert_of(i)], 1);
  for (int r = rank * GROUP_THREADS + threadIdx.x; r < rows_room; r += ctas * GROUP_THREADS) {
    row_pair[r] = -1;
    if (row_weight) row_weight[r] = 0.f;
    if (tile_expert && r < (rows_room + pad - 1) / pad) tile_expert[r] = -1;
  }
  if (ctas > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else __syncthreads();
  for (int e = threadIdx.x; e < E; e += GROUP_THREADS) {
    int before = 0, all = 0;
    for (int q = 0; q < ctas; ++q) {
      int n;
      if (ctas > 1) {
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&count[e])), "r"(q));
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(n) : "r"(at));
      } else {
        n = count[e];
      }
      if (q < rank) before += n;
      all += n;
    }
    cursor[e] = before;
    first_row[e] = (all + pad - 1) / pad * pad;  // rows it takes, until the sum over the experts before it is known
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int at = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + (int)threadIdx.x, rows = e < E ? first_row[e] : 0;
      int upto = rows;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, off);
        if ((int)threadIdx.x >= off) upto += v;
      }
      if (e < E) {
        first_row[e] = at + upto - rows;
        cursor[e] += at + upto - rows;
        if (rank == 0) {
          offsets[e] = at + upto - rows;
          if (tile_expert)
            for (int t = 0; t < rows / pad; ++t) tile_expert[(at + upto - rows) / pad + t] = e;
        }
      }
      at += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (threadIdx.x == 0 && rank == 0) offsets[E] = at;
  }
  __syncthreads();
  auto place = [&](int i, int e) {
    const int row = atomicAdd(&cursor[e], 1);
    row_pair[row] = i;
    pair_row[i] = row;
    if (row_weight) row_weight[row] = weight[i];
  };
#pragma unroll
  for (int k = 0; k < GROUP_HELD; ++k)
    if (held[k] >= 0) place(first + k * GROUP_THREADS + threadIdx.x, held[k]);
  for (int i = first + GROUP_HELD * GROUP_THREADS + threadIdx.x; i < last; i += GROUP_THREADS) place(i, expert_of(i));
  // (nobody leaves while another may still read its counts)
  if (ctas > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A warp a row, all of what a lane copies (up to 4 KB a row) asked for together.  Rows of nobody are left as they are: no row of a product depends on
// another's.  8,148 rows of 2,048 numbers among 12,212: 8.6 us, 14 with a block a row that cleared nobody's.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* __restrict__ row_pair,
                  __nv_bfloat16* __restrict__ out, int rows, int K, int top) {
  constexpr int EACH = 8;
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int pair = row < rows ? row_pair[row] : -1;
  if (pair < 0) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(pair / top) * K);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row * K);
  for (int i0 = lane; i0 < K / 8; i0 += 32 * EACH) {
    uint4 v[EACH];
#pragma unroll
    for (int k = 0; k < EACH; ++k)
      if (i0 + 32 * k < K / 8) v[k] = src[i0 + 32 * k];
#pragma unroll
    for (int k = 0; k < EACH; ++k)
      if (i0 + 32 * k < K / 8) dst[i0 + 32 * k] = v[k];
  }
}

// Which expert and which of its rows the row tile ``tile`` covers (tiles of ``rows_per_tile`` rows are numbered
// through the experts in order, an expert's last tile may be partly filled).  False beyond the last tile.
__device__ __forceinline__ bool find_tile(const int32_t* __restrict__ offsets, int E, int rows_per_tile, int tile, int& expert,
                                          int& row0, int& row1) {
  for (int e = 0; e < E; ++e) {
    const int a = offsets[e], b = offsets[e + 1];
    const int n = (b - a + rows_per_tile - 1) / rows_per_tile;
    if (tile < n) {
      expert = e;
      row0 = a + tile * rows_per_tile;
      row1 = min(b, row0 + rows_per_tile);
      return true;
    }
    tile -= n;
  }
  return false;
}

enum : int { MOE_ACT_NONE = 0, MOE_ACT_RELU2 = 1 };

__device__ __forceinline__ float moe_act(float v, int act) {
  if (act == MOE_ACT_RELU2) { v = fmaxf(v, 0.f); return v * v; }
  return v;
}

enum : int { GLU_NONE = 0, GLU_CLIPPED = 1, GLU_SILU = 2 };

__device__ __forceinline__ float glu_value(float g, float u, int glu, float r, const GluClip& c) {
  return glu == GLU_SILU ? gate_act(r * g, PSB_ACT_SILU) * (r * u) : clipped_gate_value(g, u, c);
}

// eight gated values from eight gate and eight up values (bfloat16), rounded to bfloat16
__device__ __forceinline__ uint4 glu8(const uint4& g4, const uint4& u4, int glu, float r, const GluClip& c) {
  const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&g4);
  const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&u4);
  uint4 o4;
  __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o4);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 g = __bfloat1622float2(g2[k]), u = __bfloat1622float2(u2[k]);
    o2[k] = __floats2bfloat162_rn(glu_value(g.x, u.x, glu, r, c), glu_value(g.y, u.y, glu, r, c));
  }
  return o4;
}

constexpr int TILE = 64;
constexpr int BK = 16;
constexpr int THREADS = 256;

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(THREADS)
moe_gemm_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, const int32_t* __restrict__ offsets,
                const int32_t* __restrict__ row_pair, int E, int N, int K, int top, int gather, int act, int glu,
                const GluClip clip, const float* __restrict__ row_weight) {
  __shared__ float sa[BK][TILE + 4];
  __shared__ float sw[BK][TILE + 4];
  __shared__ int src[TILE];
  pdl_trigger();
  pdl_wait();
  int expert, row0, row1;
  if (!find_tile(offsets, E, TILE, blockIdx.y, expert, row0, row1)) return;
  const int M = row1 - row0;
  W += (size_t)expert * N * K;
  for (int i = threadIdx.x; i < TILE; i += blockDim.x) {
    const int pair = i < M ? row_pair[row0 + i] : -1;  // -1: a row that belongs to nobody
    src[i] = pair < 0 ? -1 : (gather ? pair / top : row0 + i);
  }
  __syncthreads();
  const int n0 = blockIdx.x * TILE;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  const int lrow = threadIdx.x >> 2, lcol = (threadIdx.x & 3) * 4;
  const int arow = src[lrow];
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lcol + j;
      const int n = n0 + lrow;
      float av = 0.f;
      if (arow >= 0 && k < K) {
        if (glu) {
          const TA* ar = A + (size_t)arow * 2 * K;
          av = to_float<TA>(from_float<TA>(glu_value(to_float<TA>(ar[k]), to_float<TA>(ar[K + k]), glu, row_weight ? row_weight[arow] : 1.f, clip)));
        } else {
          av = to_float<TA>(A[(size_t)arow * K + k]);
        }
      }
      sa[lcol + j][lrow] = av;
      sw[lcol + j][lrow] = (n < N && k < K) ? to_float<TW>(W[(size_t)n * K + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = sa[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = sw[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)(row0 + m) * N + n] = from_float<TC>(moe_act(acc[i][j], act));
    }
  }
}

// bfloat16 on the tensor cores: a block of four warps computes 64 rows x 64 columns; warp w takes rows 16w..16w+15.
// Operands go through shared memory as bfloat16 [64][BKM + 8] (the padding keeps the fragment loads off each other's
// banks).  K in steps of 32; K must be a multiple of 8 (16-byte loads).
constexpr int BKM = 32;

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <typename TC>
__global__ void __launch_bounds__(128)
moe_mma_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W, TC* __restrict__ C,
               const int32_t* __restrict__ offsets, const int32_t* __restrict__ row_pair, int E, int N, int K, int top,
               int gather, int act, int glu, const GluClip clip, const float* __restrict__ row_weight) {
  __shared__ __align__(16) __nv_bfloat16 sa[TILE][BKM + 8];
  __shared__ __align__(16) __nv_bfloat16 sw[TILE][BKM + 8];
  __shared__ int src[TILE];
  pdl_trigger();
  pdl_wait();
  int expert, row0, row1;
  if (!find_tile(offsets, E, TILE, blockIdx.y, expert, row0, row1)) return;
  const int M = row1 - row0;
  W += (size_t)expert * N * K;
  for (int i = threadIdx.x; i < TILE; i += blockDim.x) {
    const int pair = i < M ? row_pair[row0 + i] : -1;  // -1: a row that belongs to nobody
    src[i] = pair < 0 ? -1 : (gather ? pair / top : row0 + i);
  }
  __syncthreads();
  const int n0 = blockIdx.x * TILE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, tig = lane & 3;
  float acc[8][4] = {};
  for (int k0 = 0; k0 < K; k0 += BKM) {
    // 64 rows x 32 columns = 256 pieces of 8 elements per operand; 128 threads take two of each
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int piece = threadIdx.x + it * 128;
      const int r = piece >> 2, c = (piece & 3) * 8;
      uint4 va = make_uint4(0, 0, 0, 0), vw = make_uint4(0, 0, 0, 0);
      if (k0 + c < K) {
        if (src[r] >= 0) {
          if (glu) {
            const __nv_bfloat16* ar = A + (size_t)src[r] * 2 * K + k0 + c;
            va = glu8(*reinterpret_cast<const uint4*>(ar), *reinterpret_cast<const uint4*>(ar + K), glu, row_weight ? row_weight[src[r]] : 1.f, clip);
          } else {
            va = *reinterpret_cast<const uint4*>(A + (size_t)src[r] * K + k0 + c);
          }
        }
        if (n0 + r < N) vw = *reinterpret_cast<const uint4*>(W + (size_t)(n0 + r) * K + k0 + c);
      }
      *reinterpret_cast<uint4*>(&sa[r][c]) = va;
      *reinterpret_cast<uint4*>(&sw[r][c]) = vw;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BKM; kk += 16) {
      uint32_t a[4];
      a[0] = *reinterpret_cast<const uint32_t*>(&sa[warp * 16 + gid][kk + tig * 2]);
      a[1] = *reinterpret_cast<const uint32_t*>(&sa[warp * 16 + gid + 8][kk + tig * 2]);
      a[2] = *reinterpret_cast<const uint32_t*>(&sa[warp * 16 + gid][kk + tig * 2 + 8]);
      a[3] = *reinterpret_cast<const uint32_t*>(&sa[warp * 16 + gid + 8][kk + tig * 2 + 8]);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        uint32_t b[2];
        b[0] = *reinterpret_cast<const uint32_t*>(&sw[nt * 8 + gid][kk + tig * 2]);
        b[1] = *reinterpret_cast<const uint32_t*>(&sw[nt * 8 + gid][kk + tig * 2 + 8]);
        mma_bf16(acc[nt], a, b);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int m = warp * 16 + gid + half * 8;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int n = n0 + nt * 8 + tig * 2 + j;
        if (n < N) C[(size_t)(row0 + m) * N + n] = from_float<TC>(moe_act(acc[nt][half * 2 + j], act));
      }
    }
  }
}

// Some rows per expert (decoding): what matters is that every chosen expert's matrix is read once, as fast as memory gives it.
// The work is cut into units of an expert, eight of its rows and a slab of 32 output columns; two blocks an SM take equal runs of
// units, expert by expert, so that rows are staged once per expert and no block is left over at the end.  In a unit a warp takes 16
// columns and every fourth 128 of K.  mma.sync m16n8k16 with the weights as the left operand: which k an instruction's places stand
// for is free as long as both operands agree, so a lane's 16 bytes of a weight row, and the same 16 of a token's, are the places of two
// instructions, straight out of memory.  A warp asks for its next 128 of K, and at the end of a unit for the next unit's first ones,
// before it works on the ones it has.  The four shares of K are added up in shared memory, in order.
//
// Bound by memory.  12 tokens of 4 of 32 gated experts (4,096 in and out, 2,048 between): 142 and 81 us, 5.8 TB/s of the matrices.  A
// block per expert and slab on the CUDA cores, four rows at a time, took 199 and 121; a block per expert and slab with these products
// 158 and 97 (too few turns a block to keep memory busy, and a last round of blocks).
constexpr int FEW_ROWS = 8, FEW_WARPS = 8, FEW_COLS = 32, FEW_SHARES = 4, FEW_STEPS = 4, FEW_TURN = 32 * FEW_STEPS;
// Up to so many pairs an expert on average: all of the layer at 4,096 and 45 tokens (5.6 an expert) 327 us and 829 with moe_mma_kernel,
// at 2,048 and 63 tokens (7.9) 126 and 234.
constexpr int FEW_PAIRS = 8;
constexpr int FEW_SMEM = 192 * 1024;
// rows lie half a line off one another, so that a lane's pieces meet every bank once
__host__ __device__ constexpr int few_pitch(int K) { return (K + 63) / 64 * 64 + 32; }

// 16 terms of each sum.  The instruction cuts its sums off instead of rounding them, so what it makes of a turn's terms is added up
// outside, in pairs, and turns after one another.
__device__ __forceinline__ void few_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

template <typename TC>
__global__ void __launch_bounds__(FEW_WARPS * 32, 2)
moe_fewrows_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W, TC* __restrict__ C,
                   const int32_t* __restrict__ offsets, const int32_t* __restrict__ row_pair, int E, int N, int K, int top, int gather,
                   int act, int glu, const GluClip clip, const float* __restrict__ row_weight, int rows_at_once) {
  extern __shared__ __align__(16) unsigned char few_smem[];
  __shared__ float shares[2][FEW_WARPS][FEW_ROWS][16];
  __shared__ int32_t passes[MAX_EXPERTS * (1 + FEW_PAIRS * 2 / FEW_ROWS)];  // expert and first row of every pass over a matrix
  __shared__ int passes_n;
  static_assert(FEW_ROWS % 2 == 0, "rows_at_once is all or half of them");
  __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(few_smem);  // [rows_at_once][pitch]
  pdl_trigger();
  const int pitch = few_pitch(K);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  const int share = warp & (FEW_SHARES - 1);
  pdl_wait();
  if (warp == 0) {
    int at = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, a = e < E ? offsets[e] : 0, n = e < E ? offsets[e + 1] - a : 0;
      const int mine = (n + rows_at_once - 1) / rows_at_once;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += below;
      }
      for (int p = 0; p < mine; ++p) passes[at + sum - mine + p] = e | (p * rows_at_once) << 9;
      at += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) passes_n = at;
  }
  __syncthreads();
  const int slabs = (N + FEW_COLS - 1) / FEW_COLS;
  const long long units = (long long)passes_n * slabs;
  const int first = (int)(units * blockIdx.x / gridDim.x), last = (int)(units * (blockIdx.x + 1) / gridDim.x);
  if (first >= last) return;
  const __nv_bfloat16 *w0, *w1;  // this lane's two weight rows of the unit
  auto aim = [&](int unit) {
    const int e = passes[unit / slabs] & (MAX_EXPERTS - 1), n1 = unit % slabs * FEW_COLS + warp / FEW_SHARES * 16;
    w0 = W + ((size_t)e * N + min(N - 1, n1 + gr)) * K;
    w1 = W + ((size_t)e * N + min(N - 1, n1 + gr + 8)) * K;
  };
  auto fetch = [&](int k0, uint4 (&x)[FEW_STEPS][2]) {
#pragma unroll
    for (int u = 0; u < FEW_STEPS; ++u) {
      const int k = k0 + 32 * u + 8 * tg;
      x[u][0] = k < K ? __ldg(reinterpret_cast<const uint4*>(w0 + k)) : make_uint4(0, 0, 0, 0);
      x[u][1] = k < K ? __ldg(reinterpret_cast<const uint4*>(w1 + k)) : make_uint4(0, 0, 0, 0);
    }
  };
  uint4 now[FEW_STEPS][2], next[FEW_STEPS][2];
  aim(first);
  fetch(share * FEW_TURN, now);
  int staged = -1, r0 = 0, m = 0;
  for (int unit = first; unit < last; ++unit) {
    const int pass = unit / slabs, n0 = unit % slabs * FEW_COLS;
    if (pass != staged) {  // (everybody is through with the rows that lie there: the barrier of the unit before)
      staged = pass;
      const int e = passes[pass] & (MAX_EXPERTS - 1);
      r0 = offsets[e] + (passes[pass] >> 9);
      m = min(rows_at_once, offsets[e + 1] - r0);
      for (int i = threadIdx.x; i < m * (K / 8); i += blockDim.x) {
        const int r = i / (K / 8), c = i - r * (K / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        const int pair = row_pair[r0 + r];
        const int src = pair < 0 ? -1 : (gather ? pair / top : r0 + r);
        if (src >= 0) {
          if (glu) {
            const uint4* ar = reinterpret_cast<const uint4*>(A + (size_t)src * 2 * K);
            v = glu8(ar[c], ar[K / 8 + c], glu, row_weight ? row_weight[src] : 1.f, clip);
          } else {
            v = reinterpret_cast<const uint4*>(A + (size_t)src * K)[c];
          }
        }
        *reinterpret_cast<uint4*>(rows + (size_t)r * pitch + 8 * c) = v;
      }
      __syncthreads();
    }
    float acc[4] = {};
    const __nv_bfloat16* mine = rows + (size_t)min(gr, m - 1) * pitch;  // (a row that is not there: its sums are not used)
    for (int k0 = share * FEW_TURN; k0 < K; k0 += FEW_SHARES * FEW_TURN) {
      const bool over = k0 + FEW_SHARES * FEW_TURN >= K;
      if (over && unit + 1 < last) aim(unit + 1);
      fetch(!over ? k0 + FEW_SHARES * FEW_TURN : unit + 1 < last ? share * FEW_TURN : K, next);
      static_assert(FEW_STEPS == 4, "pairs of pairs");
      float part[2][4];
#pragma unroll
      for (int u = 0; u < FEW_STEPS; ++u) {
        const int k = k0 + 32 * u + 8 * tg;
        const uint4 b = k < K ? *reinterpret_cast<const uint4*>(mine + k) : make_uint4(0, 0, 0, 0);
        const uint4 a = now[u][0], e = now[u][1];
        float d0[4], d1[4];
        few_mma(d0, a.x, e.x, a.y, e.y, b.x, b.y);
        few_mma(d1, a.z, e.z, a.w, e.w, b.z, b.w);
#pragma unroll
        for (int x = 0; x < 4; ++x) part[u / 2][x] = u % 2 ? part[u / 2][x] + (d0[x] + d1[x]) : d0[x] + d1[x];
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[x] += part[0][x] + part[1][x];
#pragma unroll
      for (int u = 0; u < FEW_STEPS; ++u) {
        now[u][0] = next[u][0];
        now[u][1] = next[u][1];
      }
    }
    auto& buf = shares[unit & 1];
#pragma unroll
    for (int x = 0; x < 4; ++x)  // columns gr and gr + 8, rows 2 tg and 2 tg + 1
      buf[warp][2 * tg + (x & 1)][gr + 8 * (x >> 1)] = acc[x];
    __syncthreads();
    {
      const int r = threadIdx.x / FEW_COLS, n = threadIdx.x % FEW_COLS, at = n / 16 * FEW_SHARES;
      float v = 0.f;
#pragma unroll
      for (int q = 0; q < FEW_SHARES; ++q) v += buf[at + q][r][n % 16];
      if (r < m && n0 + n < N) C[(size_t)(r0 + r) * N + n0 + n] = from_float<TC>(moe_act(v, act));
    }
  }
}
static_assert(FEW_WARPS * 32 == FEW_ROWS * FEW_COLS && FEW_WARPS == FEW_SHARES * FEW_COLS / 16, "a thread an output");
static_assert(MAX_EXPERTS == 1 << 9, "an expert is nine bits of a pass");

PsbPerDevice fewrows_attr[2];

template <typename TY, typename TS, typename TO>
__global__ void moe_combine_kernel(const TY* __restrict__ Y, const int32_t* __restrict__ pair_row, const float* __restrict__ weight,
                                   const TS* __restrict__ shared, const float* __restrict__ gate, int ldg, TO* __restrict__ out,
                                   int H, int top) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const float sg = shared ? sigmoidf_(gate ? gate[(size_t)t * ldg] : FLT_MAX) : 0.f;
  for (int j = threadIdx.x; j < H; j += blockDim.x) {
    float v = 0.f;
    for (int k = 0; k < top; ++k) {
      const int row = pair_row[(size_t)t * top + k];
      v = fmaf(weight ? weight[(size_t)t * top + k] : 1.f, to_float<TY>(Y[(size_t)row * H + j]), v);
    }
    if (shared) v = fmaf(sg, to_float<TS>(shared[(size_t)t * H + j]), v);
    out[(size_t)t * H + j] = from_float<TO>(v);
  }
}

// Eight numbers as they lie in memory.
template <typename T>
struct Eight;
template <>
struct Eight<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) { a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4); }
  __device__ __forceinline__ void add_to(float (&v)[8], float w) const {
    v[0] = fmaf(w, a.x, v[0]); v[1] = fmaf(w, a.y, v[1]); v[2] = fmaf(w, a.z, v[2]); v[3] = fmaf(w, a.w, v[3]);
    v[4] = fmaf(w, b.x, v[4]); v[5] = fmaf(w, b.y, v[5]); v[6] = fmaf(w, b.z, v[6]); v[7] = fmaf(w, b.w, v[7]);
  }
};
template <>
struct Eight<__nv_bfloat16> {
  uint4 raw;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { raw = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void add_to(float (&v)[8], float w) const {
    const uint32_t x[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = fmaf(w, __uint_as_float(x[i] << 16), v[2 * i]);
      v[2 * i + 1] = fmaf(w, __uint_as_float(x[i] & 0xffff0000u), v[2 * i + 1]);
    }
  }
};

// The same with eight columns a thread; the rows of four slots, of TOKENS tokens each, and the shared expert's are asked for together.  H % 8 == 0, rows on 16
// bytes.  Bound by how much is under way: 2,037 tokens of four slots and 2,048 columns 16 to 18 us a token at a time, the shared row behind the others, 12 so.
template <int TOKENS, typename TY, typename TS, typename TO>
__global__ void __launch_bounds__(256)
moe_combine_vec_kernel(const TY* __restrict__ Y, const int32_t* __restrict__ pair_row, const float* __restrict__ weight,
                       const TS* __restrict__ shared, const float* __restrict__ gate, int ldg, TO* __restrict__ out, int T, int H, int top) {
  pdl_trigger();
  pdl_wait();
  const int t0 = blockIdx.x * TOKENS;
  for (int j = threadIdx.x * 8; j < H; j += blockDim.x * 8) {
    float v[TOKENS][8] = {};
    Eight<TS> of_shared[TOKENS];
    if (shared) {
#pragma unroll
      for (int u = 0; u < TOKENS; ++u)
        if (t0 + u < T) of_shared[u].load(shared + (size_t)(t0 + u) * H + j);
    }
    for (int k0 = 0; k0 < top; k0 += 4) {
      Eight<TY> y[TOKENS][4];
      float w[TOKENS][4];
#pragma unroll
      for (int u = 0; u < TOKENS; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k0 + k >= top || t0 + u >= T) continue;
          const size_t at = (size_t)(t0 + u) * top + k0 + k;
          w[u][k] = weight ? weight[at] : 1.f;
          y[u][k].load(Y + (size_t)pair_row[at] * H + j);
        }
#pragma unroll
      for (int u = 0; u < TOKENS; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k0 + k < top && t0 + u < T) y[u][k].add_to(v[u], w[u][k]);
    }
#pragma unroll
    for (int u = 0; u < TOKENS; ++u) {
      const int t = t0 + u;
      if (t >= T) break;
      if (shared) of_shared[u].add_to(v[u], sigmoidf_(gate ? gate[(size_t)t * ldg] : FLT_MAX));
      TO* o = out + (size_t)t * H + j;
      if constexpr (sizeof(TO) == 4) {
        *reinterpret_cast<float4*>(o) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
        *reinterpret_cast<float4*>(o + 4) = make_float4(v[u][4], v[u][5], v[u][6], v[u][7]);
      } else {
        uint4 raw;
        __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) h2[i] = __floats2bfloat162_rn(v[u][2 * i], v[u][2 * i + 1]);
        *reinterpret_cast<uint4*>(o) = raw;
      }
    }
  }
}

}  // namespace

// (z, ldz, correction, chosen, weight, T, E, top, groups, keep, scale, softmax_scores, group_by_max, normalize, stream)
PSB_API int psb_moe_route(const void* z, int ldz, const void* correction, void* chosen, void* weight, int T, int E, int top,
                          int groups, int keep, float scale, int softmax_scores, int group_by_max, int normalize,
                          cudaStream_t stream) {
  if (T < 0 || E < 1 || E > MAX_EXPERTS || top < 1 || top > MAX_TOP || top > E || ldz < E) PSB_REFUSE("moe_route: bad sizes E=%d top=%d", E, top);
  if (groups < 1 || E % groups || keep < 1 || keep > groups) PSB_REFUSE("moe_route: %d experts cannot form %d groups of which %d are kept", E, groups, keep);
  if ((E / groups) * keep < top) PSB_REFUSE("moe_route: %d kept groups of %d experts cannot give %d choices", keep, E / groups, top);
  if (T == 0) return 0;
  const size_t smem = sizeof(float) * ROUTE_WARPS * (2 * (size_t)E + groups);
  psb_launch(moe_route_kernel, dim3((T + ROUTE_WARPS - 1) / ROUTE_WARPS), dim3(ROUTE_WARPS * 32), smem, stream, (const float*)z, ldz,
             (const float*)correction, (int32_t*)chosen, (float*)weight, T, E, top, groups, keep, scale, softmax_scores,
             group_by_max, normalize);
  PSB_LAUNCH_CHECK("moe_route");
  return 0;
}

// (chosen, offsets, row_pair [rows_room], pair_row [pairs], tile_expert [rows_room / pad rounded up] or null, pairs, E, pad,
//  rows_room, weight [pairs] and row_weight [rows_room] or both null, stream); rows_room >= pairs + E * (pad - 1)
PSB_API int psb_moe_group(const void* chosen, void* offsets, void* row_pair, void* pair_row, void* tile_expert, int pairs, int E,
                          int pad, int rows_room, const void* weight, void* row_weight, cudaStream_t stream) {
  if ((weight == nullptr) != (row_weight == nullptr)) PSB_REFUSE("moe_group: weights by pair and by row come together");
  if (pairs < 0 || E < 1 || E > MAX_EXPERTS || pad < 1) PSB_REFUSE("moe_group: bad sizes pairs=%d E=%d pad=%d", pairs, E, pad);
  if ((long long)rows_room < (long long)pairs + (long long)E * (pad - 1)) PSB_REFUSE("moe_group: %d rows cannot hold %d pairs of %d experts padded to %d", rows_room, pairs, E, pad);
  // (a step of few pairs is done by one CTA before a cluster's have met: 48 pairs 3.0 us)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pairs >= 1024 ? GROUP_CTAS : 1);
  cfg.blockDim = dim3(GROUP_THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cfg.gridDim.x;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (psb_pdl_enabled) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cudaLaunchKernelEx(&cfg, moe_group_kernel, (const int32_t*)chosen, (int32_t*)offsets, (int32_t*)row_pair, (int32_t*)pair_row, (int32_t*)tile_expert,
                     pairs, E, pad, rows_room, (const float*)weight, (float*)row_weight);
  PSB_LAUNCH_CHECK("moe_group");
  return 0;
}

// (x bfloat16 [T, K], row_pair [rows], out bfloat16 [rows, K], rows, K, top, stream); K a multiple of 8, 16-byte aligned
PSB_API int psb_moe_gather(const void* x, const void* row_pair, void* out, int rows, int K, int top, cudaStream_t stream) {
  if (rows < 0 || K < 8 || K % 8 || top < 1 || (((uintptr_t)x | (uintptr_t)out) & 15)) PSB_REFUSE("moe_gather: needs rows of a multiple of 8 numbers, 16-byte aligned");
  if (rows == 0) return 0;
  psb_launch(moe_gather_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, (const __nv_bfloat16*)x, (const int32_t*)row_pair,
             (__nv_bfloat16*)out, rows, K, top);
  PSB_LAUNCH_CHECK("moe_gather");
  return 0;
}

// ``pairs``: the rows the layout has room for (every expert may have one partly filled tile more than its rows need).
// ``glu`` 1 (with gather 0): a's rows are [gate (K) | up (K)] and the clipped gate (limit, alpha, offset) is taken as they are read;
// 2: the SiLU gate, with row_weight (by row, or null) multiplying both halves first.
// (a, a_dtype, w, w_dtype, c, c_dtype, offsets, row_pair, pairs, E, N, K, top, gather, act, glu, limit, alpha, offset, row_weight, stream)
PSB_API int psb_moe_gemm(const void* a, int a_dtype, const void* w, int w_dtype, void* c, int c_dtype, const void* offsets,
                         const void* row_pair, int pairs, int E, int N, int K, int top, int gather, int act, int glu, float limit,
                         float alpha, float offset, const void* row_weight, cudaStream_t stream) {
  if (pairs < 0 || E < 1 || E > MAX_EXPERTS || N < 1 || K < 1 || top < 1) PSB_REFUSE("moe_gemm: bad sizes");
  if (glu < GLU_NONE || glu > GLU_SILU) PSB_REFUSE("moe_gemm: gate code %d is not built", glu);
  if (glu && (gather || (glu == GLU_CLIPPED && !(limit > 0.f)))) PSB_REFUSE("moe_gemm: the gate on the rows goes with the second product and a positive limit");
  if (row_weight && glu != GLU_SILU) PSB_REFUSE("moe_gemm: weights by row go with the SiLU gate");
  const GluClip clip{limit, alpha, offset};
  if (act != MOE_ACT_NONE && act != MOE_ACT_RELU2) PSB_REFUSE("moe_gemm: activation code %d is not built", act);
  if (pairs == 0) return 0;
  const long long row_tiles = (pairs + TILE - 1) / TILE + E;
  if (row_tiles > 65535) PSB_REFUSE("moe_gemm: too many rows for one launch");
  const dim3 grid((N + TILE - 1) / TILE, (unsigned)row_tiles);
  const size_t few_row = few_pitch(K) * sizeof(__nv_bfloat16);
  const int few_rows = FEW_ROWS * few_row <= FEW_SMEM ? FEW_ROWS : FEW_ROWS / 2;
  const size_t few_smem = few_rows * few_row;
  if (a_dtype == PSB_BF16 && w_dtype == PSB_BF16 && K % 8 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0 &&
      pairs <= FEW_PAIRS * E && few_smem <= FEW_SMEM) {
    const dim3 few_grid(2 * psb_current_sms());
    PSB_DISPATCH_DTYPE(c_dtype, TC, {
      auto kernel = moe_fewrows_kernel<TC>;
      PsbPerDevice& done = fewrows_attr[c_dtype == PSB_F32 ? 0 : 1];
      if (!done.get()) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_SMEM) != cudaSuccess)
          PSB_REFUSE("moe_gemm: cannot raise the shared-memory limit");
        done.set();
      }
      psb_launch(kernel, few_grid, dim3(FEW_WARPS * 32), few_smem, stream, (const __nv_bfloat16*)a, (const __nv_bfloat16*)w, (TC*)c,
                 (const int32_t*)offsets, (const int32_t*)row_pair, E, N, K, top, gather, act, glu, clip, (const float*)row_weight,
                 few_rows);
    });
    PSB_LAUNCH_CHECK("moe_gemm");
    return 0;
  }
  if (a_dtype == PSB_BF16 && w_dtype == PSB_BF16 && K % 8 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0) {
    PSB_DISPATCH_DTYPE(c_dtype, TC, {
      psb_launch(moe_mma_kernel<TC>, grid, dim3(128), 0, stream, (const __nv_bfloat16*)a, (const __nv_bfloat16*)w, (TC*)c,
                 (const int32_t*)offsets, (const int32_t*)row_pair, E, N, K, top, gather, act, glu, clip, (const float*)row_weight);
    });
    PSB_LAUNCH_CHECK("moe_gemm");
    return 0;
  }
  PSB_DISPATCH_DTYPE(a_dtype, TA, {
    PSB_DISPATCH_DTYPE(w_dtype, TW, {
      PSB_DISPATCH_DTYPE(c_dtype, TC, {
        psb_launch(moe_gemm_kernel<TA, TW, TC>, grid, dim3(THREADS), 0, stream, (const TA*)a, (const TW*)w, (TC*)c,
                   (const int32_t*)offsets, (const int32_t*)row_pair, E, N, K, top, gather, act, glu, clip, (const float*)row_weight);
      });
    });
  });
  PSB_LAUNCH_CHECK("moe_gemm");
  return 0;
}

// (y, y_dtype, pair_row, weight, shared, shared_dtype, gate, ldg, out, out_dtype, T, H, top, stream)
PSB_API int psb_moe_combine(const void* y, int y_dtype, const void* pair_row, const void* weight, const void* shared,
                            int shared_dtype, const void* gate, int ldg, void* out, int out_dtype, int T, int H, int top,
                            cudaStream_t stream) {
  if (T < 0 || H < 1 || top < 1) PSB_REFUSE("moe_combine: bad sizes");
  if (T == 0) return 0;
  const bool vec = H % 8 == 0 && (((uintptr_t)y | (uintptr_t)shared | (uintptr_t)out) & 15) == 0;
  PSB_DISPATCH_DTYPE(y_dtype, TY, {
    PSB_DISPATCH_DTYPE(shared_dtype, TS, {
      PSB_DISPATCH_DTYPE(out_dtype, TO, {
        if (vec) {
          // two tokens a block where there are enough of them for every place on the SMs (four blocks each) and the rows are of 16 bits
          constexpr int PAIR = sizeof(TY) == 2 ? 2 : 1;
          const bool pairs = PAIR == 2 && T >= 8 * psb_current_sms();
          auto kernel = pairs ? moe_combine_vec_kernel<PAIR, TY, TS, TO> : moe_combine_vec_kernel<1, TY, TS, TO>;
          psb_launch(kernel, dim3(pairs ? (T + 1) / 2 : T), dim3(H >= 2048 ? 256 : 128), 0, stream, (const TY*)y, (const int32_t*)pair_row,
                     (const float*)weight, (const TS*)shared, (const float*)gate, ldg, (TO*)out, T, H, top);
          PSB_LAUNCH_CHECK("moe_combine");
          return 0;
        }
        psb_launch(moe_combine_kernel<TY, TS, TO>, dim3(T), dim3(256), 0, stream, (const TY*)y, (const int32_t*)pair_row,
                   (const float*)weight, (const TS*)shared, (const float*)gate, ldg, (TO*)out, H, top);
      });
    });
  });
  PSB_LAUNCH_CHECK("moe_combine");
  return 0;
}
