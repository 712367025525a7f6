// Attention of single tokens in the latent space on the tensor cores: all heads of a token read the same cached rows
// [latent of RANK numbers | rotated key part of ROT], so a block takes 16 or 32 heads of one token and a run of its keys,
// and every row it brings in serves all of them.
//
// A block walks its run 32 rows at a time; the rows come in with cp.async, STAGES tiles deep.  Eight warps make the products of a tile:
//   S = Q K^T   four groups of warps take a quarter of the row's 576 numbers each (144: nine steps of mma.sync m16n8k16) and
//               leave their partial scores in shared memory; the queries stay in registers for the whole run;
//   O += P V    every warp takes 64 of the 512 value columns;
// and four more bring the rows in and do the softmax between the two: a thread adds the quarters of a few scores of one head, in float32, and keeps the
// head's maximum and sum.  While they work on one tile, the others make S of the next and P V of the one before.
// Queries and weights are float32 and stay so: each goes in as three bfloat16 terms whose sum is the number to its last bit
// (8 + 8 + 8 bits), against rows that are bfloat16 to begin with, so every product is exact.  The instruction cuts its sums off
// instead of rounding them, so its accumulators hold 32 numbers' (or keys') terms at a time, the smallest terms first, and what
// comes out is added up in float32: 1.5e-7 from float64 over 3,500 keys (1.4e-6 with a chain of instructions over a block's
// keys; 1.6e-7 on the CUDA cores).  A block that shares a token's keys with others leaves maximum, sum and unscaled result for
// the merge kernel.
//
// What bounds it: the tensor cores' legacy path (three terms: 108 + 96 instructions a warp and tile, 1,024 multiply-adds a clock and SM: 1.7 us a tile of
// 32 heads, of which it takes 3.4; two chains of instructions a warp side by side are what the registers hold).  16 tokens of 32 heads over up to 3,500 keys and the
// merge 41 us on the device, 32 tokens 77, 16 tokens of 16 heads 26; with the softmax on the products' own warps, which waited for it, 47, 91 and 31.  The kernel on the CUDA
// cores beside it (latent_attention_rows_kernel, still used for other sizes) reads every row once for each pair of heads: 402 us.
#include "common.cuh"

#include <cfloat>

namespace {

constexpr int RANK = 512, ROT = 64, D = RANK + ROT;
constexpr int WARPS = 8, SOFTMAX = 128, THREADS = 32 * WARPS + SOFTMAX;  // warps of the products; threads of the softmax, behind them
constexpr int QUARTERS = 4, STEPS = D / 16 / QUARTERS;   // steps of 16 numbers a group of warps takes of a row
constexpr int PITCH = D + 8;                             // elements from row to row: an odd number of 16-byte pieces
constexpr int KEYS = 32;                                 // of a tile
constexpr int MAX_SPLITS = 32;
static_assert(D % (16 * QUARTERS) == 0 && RANK == 64 * WARPS, "shares of the warps");

// HEADS 32: the two halves of the block take 16 heads each.  HEADS 16: they take the two halves of a tile's keys.
template <int HEADS>
struct LatentShape {
  static constexpr int MG = HEADS / 16;
  // A block is launched with 168 registers a thread, of which the softmax's threads hand some to the products' warps (32 heads with 224 and 56: 42 us
  // instead of 41).
  static constexpr int PRODUCT_REGISTERS = MG == 2 ? 232 : 224, SOFTMAX_REGISTERS = MG == 2 ? 40 : 56;
  static_assert(32 * WARPS * PRODUCT_REGISTERS + SOFTMAX * SOFTMAX_REGISTERS <= THREADS * 168, "more registers than the block is launched with");
  static constexpr int KT = KEYS, STAGES = 4;
  static constexpr int SPT = HEADS * KT / SOFTMAX;  // scores a thread has in the softmax
  static constexpr int S_PITCH = KT + 8, P_PITCH = KT + 8;
  static constexpr int TILE_BYTES = KT * PITCH * 2;
  static constexpr int S_OFF = STAGES * TILE_BYTES;
  // scores, weights and factors of two tiles, in turn
  static constexpr int S_FLOATS = QUARTERS * HEADS * S_PITCH, P_WORDS = 3 * HEADS * P_PITCH / 2;
  static constexpr int P_OFF = S_OFF + 2 * S_FLOATS * 4;
  static constexpr int A_OFF = P_OFF + 2 * P_WORDS * 4;          // per head: the factor of the tile, at the end the result's
  static constexpr int L_OFF = A_OFF + 2 * HEADS * 4;            // per stage and row: whether the row counts
  static constexpr int BYTES = L_OFF + STAGES * KT * 4;
  static_assert(KT % (SOFTMAX / 32) == 0 && KT % SPT == 0 && BYTES <= 227 * 1024, "rows of a tile");
};

__device__ __forceinline__ void latent_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c = a b, from nothing
__device__ __forceinline__ void latent_mma_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void latent_ldmatrix(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void latent_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void latent_copy16(uint32_t dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// (x, y) as three pairs of bfloat16, the largest term first; the sum of a number's terms is the number
__device__ __forceinline__ void three_terms(float x, float y, uint32_t (&out)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(x, y);
    out[i] = *reinterpret_cast<const uint32_t*>(&t);
    const float2 f = __bfloat1622float2(t);
    x -= f.x;
    y -= f.y;
  }
}

// How the tokens' keys are shared out: every share is a run of at most ``per`` tiles of one token, with the smallest ``per`` for
// which no more than ``shares`` are needed (and no more than MAX_SPLITS of a token).  Every warp finds it from the positions, so
// that a captured step of other lengths is shared out anew.  With the same number of shares for every token, the blocks of the
// shorter ones were done early: 16 tokens of 3,500 keys down to half, 55 us -> 45.  That is for a single round of blocks: the
// search costs a block 0.7 us with 16 tokens and 1.5 with 90, and in several rounds the blocks that are done early make room for
// others anyway (90 tokens of 3,400 keys down to half: 231 us so, 205 with equal numbers), so there every token gets ``each``, its shares
// side by side (226 with the tokens side by side).
struct LatentRun {
  int token, position, item;
  int first, count;  // the token's shares
  int per;           // tiles of a share
};
__device__ __forceinline__ int latent_lowest(int p, int window) { return (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0; }
// tiles of a token's keys; one that has none is given a share all the same
__device__ __forceinline__ int latent_tiles(int p, int window) { return max(1, (p - latent_lowest(p, window) + KEYS) / KEYS); }

// the run that share ``mine`` is of (token -1: nobody needs that share)
__device__ __forceinline__ LatentRun latent_share(const int32_t* positions, const int32_t* token_item, int tokens, int window, int shares,
                                                  int mine, int lane) {
  int p = lane < tokens ? positions[lane] : 0, item = lane < tokens ? token_item[lane] : 0;  // of the first 32 tokens
  const int n0 = lane < tokens ? latent_tiles(p, window) : 0;
  int total = n0, most = n0;
  for (int t = lane + 32; t < tokens; t += 32) {
    const int n = latent_tiles(positions[t], window);
    total += n;
    most = max(most, n);
  }
  total = __reduce_add_sync(0xffffffffu, total);
  most = __reduce_max_sync(0xffffffffu, most);
  int lo = max((total + shares - 1) / shares, (most + MAX_SPLITS - 1) / MAX_SPLITS);
  // enough: total / (shares - tokens) tiles each
  int hi = max(lo, min(most, (total + shares - tokens - 1) / (shares - tokens)));
  while (lo < hi) {
    const int per = (lo + hi) >> 1;
    int needed = (n0 + per - 1) / per;
    for (int t = lane + 32; t < tokens; t += 32) needed += (latent_tiles(positions[t], window) + per - 1) / per;
    if (__reduce_add_sync(0xffffffffu, needed) <= shares) hi = per;
    else lo = per + 1;
  }
  int before = 0;
  for (int t0 = 0; t0 < tokens; t0 += 32) {
    if (t0 > 0 && t0 + lane < tokens) p = positions[t0 + lane], item = token_item[t0 + lane];
    const int n = t0 + lane < tokens ? (latent_tiles(p, window) + lo - 1) / lo : 0;
    int upto = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, off);
      if (lane >= off) upto += x;
    }
    const unsigned beyond = __ballot_sync(0xffffffffu, mine < before + upto);
    if (beyond) {
      const int who = __ffs(beyond) - 1;
      const int count = __shfl_sync(0xffffffffu, n, who);
      return {t0 + who, __shfl_sync(0xffffffffu, p, who), __shfl_sync(0xffffffffu, item, who),
              before + __shfl_sync(0xffffffffu, upto, who) - count, count, lo};
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  return {-1, 0, 0, 0, 0, lo};
}

template <int HEADS>
__global__ void __launch_bounds__(THREADS, 1)
latent_attention_mma_kernel(const float* __restrict__ q_lat, const __nv_bfloat16* __restrict__ cache, const int32_t* __restrict__ table,
                            int table_width, const int32_t* __restrict__ positions, const int32_t* __restrict__ token_item,
                            const float* __restrict__ gate, __nv_bfloat16* __restrict__ out, float* __restrict__ partial, int tokens,
                            int shares, int each, int heads, int page_size, int num_pages, int window, float scale,
                            const float* __restrict__ sink) {
  using Sh = LatentShape<HEADS>;
  constexpr int KT = Sh::KT, MG = Sh::MG;
  extern __shared__ __align__(16) unsigned char latent_smem[];
  float* scores = reinterpret_cast<float*>(latent_smem + Sh::S_OFF);
  uint32_t* weights = reinterpret_cast<uint32_t*>(latent_smem + Sh::P_OFF);
  float* factors = reinterpret_cast<float*>(latent_smem + Sh::A_OFF);
  int* counts = reinterpret_cast<int*>(latent_smem + Sh::L_OFF);
  const uint32_t tiles_at = (uint32_t)__cvta_generic_to_shared(latent_smem);
  const uint32_t weights_at = tiles_at + Sh::P_OFF;
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = heads / HEADS;
  const int share = blockIdx.x / groups, h0 = (blockIdx.x - share * groups) * HEADS;
  LatentRun run;
  if (each > 0) {
    const int t = share / each;
    if (t >= tokens) return;  // what the tokens leave over
    const int p = positions[t];
    run = LatentRun{t, p, token_item[t], t * each, each, (latent_tiles(p, window) + each - 1) / each};
  } else {
    run = latent_share(positions, token_item, tokens, window, shares, share, lane);
    if (run.token < 0) return;
  }
  const int t = run.token, split = share - run.first, splits = run.count, p = run.position, per = run.per;
  const int32_t* pages = table + (size_t)run.item * table_width;
  const int lo = latent_lowest(p, window);
  const int first = lo + split * per * KT;
  const int end = p + 1 - first > per * KT ? first + per * KT : p + 1;
  const int ntiles = max(0, (end - first + KT - 1) / KT);

  // Tile i's scores are made in turn i - 1, its weights in turn i and its part of the result in turn i + 1, so that products and softmax always have
  // something to do; it is asked for in turn i - 2 and its stage is free again behind turn i + 1.
  if (warp < WARPS) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Sh::PRODUCT_REGISTERS));
    const int quarter = warp & 3, half = warp >> 2;        // half: of the heads (32) or of a tile's keys (16)
    const int gr = lane >> 2, gc = 2 * (lane & 3);
    uint32_t q[STEPS][3][4];
    {
      const float* rows = q_lat + ((size_t)t * heads + h0 + (MG == 2 ? 16 * half : 0) + gr) * D + quarter * STEPS * 16 + gc;
#pragma unroll
      for (int k = 0; k < STEPS; ++k) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 x = *reinterpret_cast<const float2*>(rows + (size_t)(j & 1) * 8 * D + k * 16 + (j >> 1) * 8);
          uint32_t terms[3];
          three_terms(x.x, x.y, terms);
#pragma unroll
          for (int e = 0; e < 3; ++e) q[k][e][j] = terms[e];
        }
      }
    }
    float o[MG][8][4];
#pragma unroll
    for (int m = 0; m < MG; ++m)
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[m][n][e] = 0.f;
    auto products = [&](int i) {  // this warp's share of the scores of tile i
      constexpr int NT = MG == 2 ? KT / 8 : KT / 16;
      const uint32_t tile = tiles_at + (i % Sh::STAGES) * Sh::TILE_BYTES;
      const int key0 = MG == 2 ? 0 : KT / 2 * half;
      float s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
      const uint32_t at = tile + ((key0 + (lane & 7) + 8 * (lane >> 4)) * PITCH + quarter * STEPS * 16 + 8 * ((lane >> 3) & 1)) * 2;
#pragma unroll
      for (int k = 0; k < STEPS; k += 2) {
        constexpr int LAST = STEPS - 1;
        const int steps = k < LAST ? 2 : 1;
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
          uint32_t b[2][4];
          float d0[4], d1[4];
#pragma unroll
          for (int x = 0; x < steps; ++x) latent_ldmatrix(b[x], at + (n * 8 * PITCH + (k + x) * 16) * 2);
          latent_mma_first(d0, q[k][2], b[0][0], b[0][1]);
          latent_mma_first(d1, q[k][2], b[0][2], b[0][3]);
#pragma unroll
          for (int e = 2; e >= 0; --e)
#pragma unroll
            for (int x = e == 2 ? 1 : 0; x < steps; ++x) {
              latent_mma(d0, q[k + x][e], b[x][0], b[x][1]);
              latent_mma(d1, q[k + x][e], b[x][2], b[x][3]);
            }
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            s[n][x] += d0[x];
            s[n + 1][x] += d1[x];
          }
        }
      }
      float* dst = scores + (i & 1) * Sh::S_FLOATS + (quarter * HEADS + (MG == 2 ? 16 * half : 0) + gr) * Sh::S_PITCH + key0 + gc;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        *reinterpret_cast<float2*>(dst + n * 8) = make_float2(s[n][0], s[n][1]);
        *reinterpret_cast<float2*>(dst + 8 * Sh::S_PITCH + n * 8) = make_float2(s[n][2], s[n][3]);
      }
    };
    auto weighted = [&](int i) {  // O += P V of tile i
      const uint32_t tile = tiles_at + (i % Sh::STAGES) * Sh::TILE_BYTES;
      static_assert(KT == 32, "two steps of keys");
      const uint32_t at = tile + ((lane & 15) * PITCH + 64 * warp + 8 * (lane >> 4)) * 2;
      const uint32_t wat = weights_at + (i & 1) * Sh::P_WORDS * 4 + ((lane & 15) * Sh::P_PITCH + 8 * (lane >> 4)) * 2;
#pragma unroll
      for (int m = 0; m < MG; ++m) {
        const float f0 = factors[(i & 1) * HEADS + 16 * m + gr], f1 = factors[(i & 1) * HEADS + 16 * m + gr + 8];
        uint32_t a[2][3][4];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int e = 0; e < 3; ++e) latent_ldmatrix(a[k][e], wat + ((e * HEADS + 16 * m) * Sh::P_PITCH + k * 16) * 2);
#pragma unroll
        for (int n = 0; n < 8; n += 2) {
          uint32_t b[2][4];
          float d0[4], d1[4];
#pragma unroll
          for (int k = 0; k < 2; ++k) latent_ldmatrix_trans(b[k], at + (k * 16 * PITCH + n * 8) * 2);
          latent_mma_first(d0, a[0][2], b[0][0], b[0][1]);
          latent_mma_first(d1, a[0][2], b[0][2], b[0][3]);
#pragma unroll
          for (int e = 2; e >= 0; --e)
#pragma unroll
            for (int k = e == 2 ? 1 : 0; k < 2; ++k) {
              latent_mma(d0, a[k][e], b[k][0], b[k][1]);
              latent_mma(d1, a[k][e], b[k][2], b[k][3]);
            }
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            o[m][n][x] = fmaf(o[m][n][x], x < 2 ? f0 : f1, d0[x]);
            o[m][n + 1][x] = fmaf(o[m][n + 1][x], x < 2 ? f0 : f1, d1[x]);
          }
        }
      }
    };
    __syncthreads();  // tile 0 is there
    if (ntiles > 0) products(0);
    __syncthreads();
    for (int i = 0; i <= ntiles; ++i) {
      if (i + 1 < ntiles) products(i + 1);
      if (i > 0) weighted(i - 1);
      if (i < ntiles) __syncthreads();
    }
    if (shares > tokens) {  // a token's shares together: [heads, splits, RANK + 2]
      float* mine = partial + ((size_t)run.first * heads + (size_t)h0 * splits + split) * (RANK + 2);
#pragma unroll
      for (int m = 0; m < MG; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float* row = mine + (size_t)(16 * m + gr + 8 * r) * splits * (RANK + 2) + 2 + 64 * warp + gc;
#pragma unroll
          for (int n = 0; n < 8; ++n) *reinterpret_cast<float2*>(row + n * 8) = make_float2(o[m][n][2 * r], o[m][n][2 * r + 1]);
        }
      return;
    }
    __syncthreads();  // the results' factors are there
#pragma unroll
    for (int m = 0; m < MG; ++m)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int h = 16 * m + gr + 8 * r;
        const float f = factors[(ntiles & 1) * HEADS + h];
        __nv_bfloat16* row = out + ((size_t)t * heads + h0 + h) * RANK + 64 * warp + gc;
#pragma unroll
        for (int n = 0; n < 8; ++n) *reinterpret_cast<__nv_bfloat162*>(row + n * 8) = __floats2bfloat162_rn(o[m][n][2 * r] * f, o[m][n][2 * r + 1] * f);
      }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Sh::SOFTMAX_REGISTERS));
    // A warp brings in eight neighbouring rows of a tile; where they lie is looked up one tile earlier (lane r: row r), so that
    // the copies never wait for the page table.
    constexpr int MINE = KT / (SOFTMAX / 32);
    const int first_row = (warp - WARPS) * MINE;
    auto look_up = [&](int i) -> long long {
      const int key = first + i * KT + first_row + (lane & (MINE - 1));
      if (i >= ntiles || key >= end) return -1;
      const int page = pages[key / page_size];
      return page >= 0 && page < num_pages ? ((long long)page * page_size + key % page_size) * D : -1;
    };
    auto bring = [&](int i, long long rows) {
      const int stage = i % Sh::STAGES;
      if (i < ntiles) {
        if (lane < MINE) counts[stage * KT + first_row + lane] = rows >= 0;
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
          const long long at = __shfl_sync(0xffffffffu, rows, j);
          const __nv_bfloat16* src = cache + (at < 0 ? 0 : at);
          const uint32_t dst = tiles_at + stage * Sh::TILE_BYTES + (first_row + j) * PITCH * 2;
#pragma unroll
          for (int c = 0; c < D / 8; c += 32)
            if (c + lane < D / 8) latent_copy16(dst + (c + lane) * 16, src + (c + lane) * 8, at >= 0);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    bring(0, look_up(0));
    bring(1, look_up(1));
    long long next_rows = look_up(2);
    // the softmax's share of a thread: SPT neighbouring keys of one head
    constexpr int SPT = Sh::SPT, PER_HEAD = KT / SPT;
    const int head = (threadIdx.x - 32 * WARPS) / PER_HEAD, key_at = ((threadIdx.x - 32 * WARPS) % PER_HEAD) * SPT;
    float m_run = -FLT_MAX, l_run = 0.f;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // tile 0 is there
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // its scores and tile 1 are
    for (int i = 0; i < ntiles; ++i) {
      bring(i + 2, next_rows);
      next_rows = look_up(i + 3);
      {
        float s[SPT];
#pragma unroll
        for (int j = 0; j < SPT; ++j) s[j] = 0.f;
        bool on[SPT];
#pragma unroll
        for (int j = 0; j < SPT; j += 2) {
#pragma unroll
          for (int e = 0; e < QUARTERS; ++e) {
            const float2 part = *reinterpret_cast<const float2*>(scores + (i & 1) * Sh::S_FLOATS + (e * HEADS + head) * Sh::S_PITCH + key_at + j);
            s[j] += part.x;
            s[j + 1] += part.y;
          }
          const int2 live = *reinterpret_cast<const int2*>(counts + (i % Sh::STAGES) * KT + key_at + j);
          on[j] = live.x != 0;
          on[j + 1] = live.y != 0;
        }
        // An infinity of the row times a term that is 0 is NaN, and so is a query beyond bfloat16's range: such a score is made again
        // from the numbers themselves, and -inf drops out as it should.  (A value that is infinite may still come out as NaN.)
#pragma unroll
        for (int j = 0; j < SPT; ++j) {
          if (!on[j] || s[j] == s[j]) continue;
          const float* query = q_lat + ((size_t)t * heads + h0 + head) * D;
          const __nv_bfloat16* row = reinterpret_cast<const __nv_bfloat16*>(latent_smem + (i % Sh::STAGES) * Sh::TILE_BYTES) + (key_at + j) * PITCH;
          float sum = 0.f;
#pragma unroll 1
          for (int d = 0; d < D; ++d) sum = fmaf(query[d], __bfloat162float(row[d]), sum);
          s[j] = sum;
        }
        float m_new = m_run;
#pragma unroll
        for (int e = 0; e < SPT; ++e) {
          s[e] *= scale;
          if (on[e]) m_new = fmaxf(m_new, s[e]);
        }
#pragma unroll
        for (int off = 1; off < PER_HEAD; off <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, off));
        const float alpha = expf(m_run - m_new);  // first tile: exp(-huge) = 0; no key that counts so far: 1, of nothing
        float w[SPT], add = 0.f;
#pragma unroll
        for (int e = 0; e < SPT; ++e) {
          w[e] = on[e] ? expf(s[e] - m_new) : 0.f;
          add += w[e];
        }
        l_run = fmaf(l_run, alpha, add);
        m_run = m_new;
#pragma unroll
        for (int j = 0; j < SPT; j += 2) {
          uint32_t a[3];
          three_terms(w[j], w[j + 1], a);
#pragma unroll
          for (int e = 0; e < 3; ++e) weights[(i & 1) * Sh::P_WORDS + ((e * HEADS + head) * Sh::P_PITCH + key_at + j) / 2] = a[e];
        }
        if (key_at == 0) factors[(i & 1) * HEADS + head] = alpha;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
#pragma unroll
    for (int off = 1; off < PER_HEAD; off <<= 1) l_run += __shfl_xor_sync(0xffffffffu, l_run, off);
    if (shares > tokens) {
      float* mine = partial + ((size_t)run.first * heads + (size_t)h0 * splits + split) * (RANK + 2);
      // where a token's shares are stands in its rows of the result, if that's to be found
      const int at = threadIdx.x - 32 * WARPS;
      if (each == 0 && split == 0 && at < HEADS) *reinterpret_cast<int2*>(out + ((size_t)t * heads + h0 + at) * RANK) = make_int2(run.first, splits);
      if (key_at == 0) *reinterpret_cast<float2*>(mine + (size_t)head * splits * (RANK + 2)) = make_float2(m_run, l_run);
      return;
    }
    if (key_at == 0) {
      float by = 1.f / l_run;
      if (sink) {
        const float sk = sink[h0 + head], top = fmaxf(m_run, sk), down = expf(m_run - top);
        by = down / fmaf(l_run, down, expf(sk - top));
      }
      factors[(ntiles & 1) * HEADS + head] = by * (gate ? gate[(size_t)t * heads + h0 + head] : 1.f);  // (not the last tile's place)
    }
    __syncthreads();
  }
}

// A block per (token, head): the shares of the blocks that split its keys, every other one a group of threads, asked for before
// their weights are known (up to ten of them): 16 tokens of 32 heads, 9 shares each, 5.9 us by itself with cold caches; with one group of threads and
// a share after the other 1.3 us more.
constexpr int MERGE_AHEAD = 5, MERGE_COLS = RANK / 4;
template <int GROUPS>
__global__ void __launch_bounds__(GROUPS * MERGE_COLS)
latent_attention_mma_merge_kernel(const float* __restrict__ partial, const float* __restrict__ gate, __nv_bfloat16* out, int each,
                                  const float* __restrict__ sink, int heads) {
  __shared__ float by[MAX_SPLITS];
  __shared__ float4 sums[GROUPS > 1 ? GROUPS - 1 : 1][MERGE_COLS];
  pdl_trigger();
  pdl_wait();
  const size_t unit = blockIdx.x;
  // first share and number of shares; what stands in the result is overwritten at the end
  const int2 run = each > 0 ? make_int2((int)(unit / heads) * each, each) : *reinterpret_cast<const int2*>(out + unit * RANK);
  const int splits = run.y;
  const float* mine = partial + ((size_t)run.x * heads + unit % heads * splits) * (RANK + 2);
  const int group = threadIdx.x / MERGE_COLS, column = threadIdx.x % MERGE_COLS, lane = threadIdx.x & 31;
  const float* src = mine + 2 + 4 * column;  // rows start on 8 bytes
  float2 a[MERGE_AHEAD], b[MERGE_AHEAD];
  auto ask = [&](int s0) {
#pragma unroll
    for (int j = 0; j < MERGE_AHEAD; ++j) {
      const int s = s0 + j * GROUPS;
      a[j] = b[j] = make_float2(0.f, 0.f);
      if (s >= splits) continue;
      a[j] = *reinterpret_cast<const float2*>(src + (size_t)s * (RANK + 2));
      b[j] = *reinterpret_cast<const float2*>(src + (size_t)s * (RANK + 2) + 2);
    }
  };
  ask(group);
  if (threadIdx.x < 32) {
    const float2 ml = lane < splits ? *reinterpret_cast<const float2*>(mine + (size_t)lane * (RANK + 2)) : make_float2(-FLT_MAX, 0.f);
    const float sk = sink ? sink[unit % heads] : -FLT_MAX;
    const float top = fmaxf(warp_max(ml.x), sk);
    const float f = ml.y > 0.f ? expf(ml.x - top) : 0.f;
    const float sum = warp_sum(ml.y * f) + (sink ? expf(sk - top) : 0.f);
    by[lane] = f * (gate ? gate[unit] : 1.f) / sum;
  }
  __syncthreads();
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = group; s0 < splits; s0 += MERGE_AHEAD * GROUPS) {
    if (s0 > group) ask(s0);
#pragma unroll
    for (int j = 0; j < MERGE_AHEAD; ++j) {
      if (s0 + j * GROUPS >= splits) break;
      const float f = by[s0 + j * GROUPS];
      v.x = fmaf(a[j].x, f, v.x); v.y = fmaf(a[j].y, f, v.y);
      v.z = fmaf(b[j].x, f, v.z); v.w = fmaf(b[j].y, f, v.w);
    }
  }
  if constexpr (GROUPS > 1) {
    if (group) sums[group - 1][column] = v;
    __syncthreads();
    if (group) return;
#pragma unroll
    for (int g = 0; g < GROUPS - 1; ++g) {
      const float4 x = sums[g][column];
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
  }
  __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(out + unit * RANK + 4 * column) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

template <int HEADS>
int launch_latent_mma(const float* q, const __nv_bfloat16* cache, const int32_t* table, int width, const int32_t* positions,
                      const int32_t* token_item, const float* gate, __nv_bfloat16* out, float* partial, int T, int heads, int page_size,
                      int num_pages, int window, float scale, int shares, int each, const float* sink, cudaStream_t stream) {
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(latent_attention_mma_kernel<HEADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, LatentShape<HEADS>::BYTES) != cudaSuccess)
      PSB_REFUSE("latent_attention_mma: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(latent_attention_mma_kernel<HEADS>, dim3((unsigned)(shares * (heads / HEADS))), dim3(THREADS), (size_t)LatentShape<HEADS>::BYTES,
             stream, q, cache, table, width, positions, token_item, gate, out, partial, T, shares, each, heads, page_size, num_pages, window,
             scale, sink);
  PSB_LAUNCH_CHECK("latent_attention_mma");
  return 0;
}

}  // namespace

// (rank, rot, heads) -> heads a block takes of a token, 0 if the kernel is not built for the sizes
PSB_API int psb_latent_attention_mma_heads(int rank, int rot, int heads) {
  if (rank != RANK || rot != ROT || heads < 1) return 0;
  return heads % 32 == 0 ? 32 : heads % 16 == 0 ? 16 : 0;
}

// bfloat16 cache and output, float32 queries [T, heads, RANK + ROT]; ``shares`` (T..32 T) blocks share out the tokens' keys, for
// every group of heads, with ``partial`` float32 [shares, heads, RANK + 2] as their meeting place if they are more than the tokens.
PSB_API int psb_latent_attention_mma(const void* q_lat, const void* cache, const void* table, int table_width, const void* positions,
                                     const void* token_item, const void* gate, void* out, int T, int heads, int rank, int rot, int page_size,
                                     int num_pages, int window, float scale, int shares, void* partial, const void* sink, cudaStream_t stream) {
  const int per_block = psb_latent_attention_mma_heads(rank, rot, heads);
  if (!per_block || T < 0) PSB_REFUSE("latent_attention_mma: not built for T=%d heads=%d rank=%d rot=%d", T, heads, rank, rot);
  if (page_size < 1 || num_pages < 1 || table_width < 1) PSB_REFUSE("latent_attention_mma: bad paging (page_size=%d pages=%d width=%d)", page_size, num_pages, table_width);
  if (window < 0) PSB_REFUSE("latent_attention_mma: negative window");
  if (((uintptr_t)cache | (uintptr_t)q_lat | (uintptr_t)out | (uintptr_t)partial) & 15) PSB_REFUSE("latent_attention_mma: queries, cache, scratch and output must be 16-byte aligned");
  if (T == 0) return 0;
  if (shares < T || shares > (long long)T * MAX_SPLITS || (shares > T && !partial))
    PSB_REFUSE("latent_attention_mma: 1 to %d shares a token (with their scratch), not %d for %d", MAX_SPLITS, shares, T);
  if ((long long)T * heads > 0x7fffffffLL || (long long)shares * (heads / per_block) > 0x7fffffffLL) PSB_REFUSE("latent_attention_mma: batch too large");
  const int each = shares == T || (long long)shares * (heads / per_block) > psb_current_sms() ? shares / T : 0;
  auto launch = per_block == 32 ? launch_latent_mma<32> : launch_latent_mma<16>;
  const int status = launch((const float*)q_lat, (const __nv_bfloat16*)cache, (const int32_t*)table, table_width, (const int32_t*)positions,
                            (const int32_t*)token_item, (const float*)gate, (__nv_bfloat16*)out, (float*)partial, T, heads, page_size,
                            num_pages, window, scale, shares, each, (const float*)sink, stream);
  if (status) return status;
  if (shares > T) {
    const auto merge = each > 0 ? latent_attention_mma_merge_kernel<1> : latent_attention_mma_merge_kernel<2>;
    psb_launch(merge, dim3((unsigned)(T * heads)), dim3((each > 0 ? 1 : 2) * MERGE_COLS), 0, stream, (const float*)partial, (const float*)gate,
               (__nv_bfloat16*)out, each, (const float*)sink, heads);
    PSB_LAUNCH_CHECK("latent_attention_mma_merge");
  }
  return 0;
}
