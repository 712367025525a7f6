// C[M,N] = A[M,K] * W[N,K]^T in bfloat16 on the 5th-generation tensor cores, for many rows (prefill).
//
// Persistent, warp-specialised CTAs (one per SM), 320 threads, output tiles of 128 rows by BN columns (256, 192 or
// 128: the widest that still gives every SM a tile; a few hundred rows against a narrow matrix take the narrow ones):
//   warp 0      producer: one lane issues TMA loads (cp.async.bulk.tensor.2d) of a 128x64 tile of A and two
//               (BN/2)x64 tiles of W per stage into 128-byte-swizzled shared memory; completion by mbarrier
//               transaction bytes;
//   warp 1      MMA: an elected lane issues tcgen05.mma (cta_group::1, kind::f16, M=128, N=BN, K=16; four per stage)
//               with shared-memory matrix descriptors; accumulators are float32 in tensor memory (two buffers 256
//               columns apart, so the epilogue of one tile overlaps the main loop of the next); tcgen05.commit hands
//               stages back to the producer and finished accumulators to the epilogue;
//   warps 2..9  epilogue: tcgen05.ld (32 lanes x 32 columns per instruction) -> registers -> bfloat16 -> global.
// Products of many tiles go two CTAs to a tile of 256 rows (gemm_tcgen05_pair_kernel below).
// The two W tiles of a stage are rows [n0, n0+BN/2) and [n1, n1+BN/2): for a plain product n1 = n0 + BN/2; for the
// gated feed-forward n0 indexes the gate rows and n1 the matching up rows, and the epilogue writes
// silu(gate) * up, so the [T, 2I] intermediate never exists (prefixserve/model/llama.py:120-121 of PrefixServe;
// F.linear at :113, :117).  For the projection of an attention layer the epilogue does the rotary kernel's job
// (rope.cu) on the sums and stores queries, keys and values where they belong (llama.py:113-116 and
// prefixserve/model/attention.py:105-106 of PrefixServe), so the [T, (hq + 2 hkv) D] matrix never exists either.
//
// Rows of A past M, rows of W past N and columns past K are filled with zeros by the TMA unit (K only needs to be a
// multiple of 8: a 16-byte row pitch).  No load is multicast: every CTA brings its own tiles, the two of a pair each its part.
//
// Every wait on an mbarrier is bounded.  If one runs out, the CTA raises a flag that all its warps poll, stops
// issuing work, pauses long enough for copies in flight to land, frees its tensor memory and returns; the host finds
// a non-zero status word (psb_tcgen05_status) and raises.  That path has never been taken in testing; it exists so
// that a defect cannot hang the GPU.
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;        // 16 KB
// Warps that store a tile: two on each quarter of its rows, half the columns each; four where a row's angles fill the registers.  With four, and a
// division and a choice of the activation a number, the epilogue was what bounded products with short contractions: 8,148 rows of 32 experts, K 2,048
// gated and 1,024 plain, 208 us with four and 129 with eight (two CTAs a tile both).
constexpr int store_warps(int hb) { return hb > 0 ? 4 : 8; }
constexpr int threads(int hb) { return 32 * (2 + store_warps(hb)); }
// Columns of a tile that are one warp's (as many as loads from tensor memory bring; the last warp's may be fewer).
__host__ __device__ constexpr int part_columns(int bn, int parts) { return (bn / parts + 31) / 32 * 32; }
constexpr int TMEM_COLS = 512;              // two accumulator buffers, 256 float32 columns apart
constexpr int ACC_STRIDE = 256;
constexpr int MAX_STAGES = 6;
// What a storing warp of two CTAs' tiles has of shared memory: 32 rows of 32 results, on their way out (see leave_rows).
constexpr int LEAVING_WARP = 32 * 32 * 2, LEAVING_BYTES = 8 * LEAVING_WARP;

// The output tile is 128 rows by BN columns: 256 where that fills the SMs evenly, 192 where it does not (a product of
// 192 tiles of 256 columns takes 148 CTAs two rounds, as 256 tiles of 192 columns two rounds of three quarters the size),
// 240 for plain products that 256 would cut into a few tiles less than there are SMs (2,048 rows by 2,048 columns:
// 128 tiles of 256 leave 20 SMs idle, 144 tiles of 240 do the same work in one round of 15/16 the length).
template <int BN>
struct Tile {
  static_assert(BN == 256 || BN == 240 || BN == 192 || BN == 128, "tile widths built");
  static constexpr int HALF = BN / 2;                  // rows of W per TMA load
  static constexpr int B_BYTES = BN * BK * 2;          // 32 to 16 KB, a multiple of 1,024 (the swizzle's period)
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN >= 240 ? 4 : (BN == 192 ? 5 : 6);
  static_assert(B_BYTES % 1024 == 0 && (HALF * BK * 2) % 1024 == 0, "operand tiles start on the swizzle's period");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
  static_assert(STAGES <= MAX_STAGES && SMEM_BYTES <= 227 * 1024, "beyond a CTA's shared memory");
};

// shared memory: [stages][A | B] (1024-byte aligned), then barriers and the tensor-memory address
struct Barriers {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  uint32_t abort;
};
static_assert(sizeof(Barriers) <= 256, "room kept for the barriers");

// status word: 0 ok; otherwise which wait gave up (1 producer, 2 mma, 3 epilogue, 4 mma/acc)
using namespace tc;

// mode: 0 plain (C[M, N], tile columns [n0, n0+BN/2) and [n0+BN/2, n0+BN)); 1 gated (C[M, I], W = [gate; up], tile
// columns [n0, n0+128) of the gate and the same of the up rows); 2 the projection of an attention layer (columns as in
// 0; the epilogue rotates queries and keys and stores queries, keys and values where RopeArgs says, C is not used).
enum : int { MODE_PLAIN = 0, MODE_GATED = 1, MODE_ROPE = 2, MODE_GATED_GELU = 3, MODE_RELU2 = 4, MODE_GATED_CLIPPED = 5, MODE_GATED_SCALED = 6,
             MODE_SILU = 7, MODE_GELU = 8 };
// gated: SiLU, the tanh form of GELU, or (clipped) g * sigmoid(alpha g) * (u + offset) with g = min(gate, limit) and
// u = clamp(up, -limit, limit), the three numbers in a GluClip (common.cuh).
using GluArgs = GluClip;
__device__ __forceinline__ bool mode_is_gated(int mode) { return mode == MODE_GATED || mode == MODE_GATED_GELU || mode == MODE_GATED_CLIPPED || mode == MODE_GATED_SCALED; }
// MODE_RELU2: columns as in 0, the epilogue stores max(sum, 0)^2.  MODE_SILU, MODE_GELU: the same with SiLU or the tanh form of
// GELU of the sum.
//
// Grouped products (``tile_expert`` given): W is a stack of matrices [experts * N_out, K] and every 128-row tile of A
// belongs to one of them, named by tile_expert[row tile] (-1: the tile holds no rows and is skipped by all three
// roles alike); the W rows of the tile start at expert * N_out (gated: at expert * 2 N_out, the expert's gate rows
// followed by its up rows).  Columns of a tile beyond N_out read the next matrix's
// rows and are never stored.
//
// MODE_GATED_SCALED (SiLU): ``row_scale`` gives a number per row that multiplies both branches before the activation (the weight of a
// (token, expert) pair that acts on what the expert reads: the product is linear, so it may act on the sums).

// One thread's row of a 128 x BN tile of sums, for the projection of an attention layer: 16 columns are 8 pairs of one
// head (first-half elements, then the ones they are rotated with), so the job of the rotary kernel is done on the sums
// while they are in registers.  Each value is first rounded to bfloat16, which is what a separate projection would have
// stored for the rotary kernel to read.  HB > 0: a head is HB blocks of 16 columns and the caller holds the angles of
// the row's position in registers (cs, sn); HB == 0: any head size, angles fetched block by block, and two warps share the
// columns.
template <int BN, int HB>
__device__ __forceinline__ void rope_store_row(uint32_t taddr, int row, int M, int n0, int N_out, const RopeArgs& rope, int pos,
                                               int page, const float (&cs)[HB > 0 ? HB : 1][8],
                                               const float (&sn)[HB > 0 ? HB : 1][8], int part) {
  static_assert(HB % 2 == 0 && BN % (16 * (HB > 0 ? HB : 1)) == 0, "tiles must start at a head's first column");
  constexpr int SPAN = HB > 0 ? 16 * HB : 32;  // columns per round: one head, or one load from tensor memory
  constexpr int MINE = part_columns(BN, store_warps(HB) / 4);
  const int D = rope.D, q_cols = rope.hq * D, k_cols = rope.hkv * D;
  const int safe = pos < 0 ? 0 : (pos >= rope.max_positions ? rope.max_positions - 1 : pos);
  const bool page_ok = page >= 0 && page < rope.num_pages;  // the host checks tables before launch; a bad id is skipped
  const size_t in_page = (size_t)(pos & ((1 << rope.page_shift) - 1)) * D;
#pragma unroll 1
  for (int c0 = part * MINE; c0 < BN && c0 < (part + 1) * MINE; c0 += SPAN) {
#pragma unroll
    for (int cc = 0; cc < SPAN; cc += 32) {
      uint32_t v[32];
      tmem_ld32(taddr + c0 + cc, v);
      tmem_ld_wait();
      if (row >= M) continue;
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int col = n0 + c0 + cc + 16 * b;
        if (col >= N_out) continue;
        float lo[8], hi[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          lo[j] = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[16 * b + j])));
          hi[j] = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[16 * b + 8 + j])));
        }
        __nv_bfloat16* dst = nullptr;
        if (col < q_cols + k_cols) {
          const int within = col < q_cols ? col : col - q_cols;
          const int head = within / D;
          const int blk = HB > 0 ? cc / 16 + b : (within - head * D) >> 4;
          if (rope.cos_t) {
            if constexpr (HB > 0) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float a, r;
                rotate_pair(lo[j], hi[j], cs[cc / 16 + b][j], sn[cc / 16 + b][j], a, r);
                lo[j] = a; hi[j] = r;
              }
            } else {
              const float4* cp = reinterpret_cast<const float4*>(rope.cos_t + (size_t)safe * (D >> 1) + blk * 8);
              const float4* sp = reinterpret_cast<const float4*>(rope.sin_t + (size_t)safe * (D >> 1) + blk * 8);
              const float4 c0v = __ldg(cp), c1v = __ldg(cp + 1), s0v = __ldg(sp), s1v = __ldg(sp + 1);
              const float cv[8] = {c0v.x, c0v.y, c0v.z, c0v.w, c1v.x, c1v.y, c1v.z, c1v.w};
              const float sv[8] = {s0v.x, s0v.y, s0v.z, s0v.w, s1v.x, s1v.y, s1v.z, s1v.w};
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float a, r;
                rotate_pair(lo[j], hi[j], cv[j], sv[j], a, r);
                lo[j] = a; hi[j] = r;
              }
            }
          }
          if (col < q_cols) dst = rope.q_out + ((size_t)row * rope.hq + head) * D + blk * 16;
          else if (page_ok) dst = rope.kv + ((((size_t)page * 2) * rope.hkv + head) << rope.page_shift) * D + in_page + blk * 16;
        } else {
          const int within = col - q_cols - k_cols;
          const int head = within / D, d0 = within - head * D;
          if (page_ok) dst = rope.kv + ((((size_t)page * 2 + 1) * rope.hkv + head) << rope.page_shift) * D + in_page + d0;
        }
        if (dst) {
          reinterpret_cast<uint4*>(dst)[0] = make_uint4(pack2(lo[0], lo[1]), pack2(lo[2], lo[3]), pack2(lo[4], lo[5]), pack2(lo[6], lo[7]));
          reinterpret_cast<uint4*>(dst)[1] = make_uint4(pack2(hi[0], hi[1]), pack2(hi[2], hi[3]), pack2(hi[4], hi[5]), pack2(hi[6], hi[7]));
        }
      }
    }
  }
}

// 32 columns of the warp's rows, a thread a row, from ``col`` on as far as there are columns (``limit``); rows from M on stay.  They go through shared memory
// (pieces of 16 bytes, piece j of row r at j ^ (r / 2 % 4)) to where four lanes have a row's 64 bytes: stored by the thread that has the row, every 16 bytes are
// half a sector on a line of their own.  Where a CTA's tiles follow one another and their stores are in the way, as in two CTAs a tile: routed experts on 2,037
// tokens (8,148 rows of 2,048 by 1,024 in the second product: 50 us -> 42) 159 us a call -> 154, 142 -> 133 without gates; 1,979 tokens of feed-forward as before.
// A CTA's only tile leaves sooner straight from the registers (300 rows of 8,192 gated and 2,048 columns 44.0 us instead of 43.5).
__device__ __forceinline__ void leave_rows(uint4* leaving, const uint32_t (&packed)[4][4], __nv_bfloat16* __restrict__ C, int row, int M, int col, int limit, int ldc) {
  const int lane = threadIdx.x & 31, row0 = row - lane;
  if (col + 32 <= limit && (ldc & 7) == 0) {
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j) leaving[lane * 4 + (j ^ ((lane >> 1) & 3))] = make_uint4(packed[j][0], packed[j][1], packed[j][2], packed[j][3]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int in = 8 * i + (lane >> 2), piece = lane & 3;
      if (row0 + in < M) *reinterpret_cast<uint4*>(C + (size_t)(row0 + in) * ldc + col + 8 * piece) = leaving[in * 4 + (piece ^ ((in >> 1) & 3))];
    }
    __syncwarp();
  } else if (row < M) {
    __nv_bfloat16* crow = C + (size_t)row * ldc;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (col + 8 * j + 8 <= limit && (ldc & 7) == 0) {  // a last run of fewer than 32: its whole eights
        *reinterpret_cast<uint4*>(crow + col + 8 * j) = make_uint4(packed[j][0], packed[j][1], packed[j][2], packed[j][3]);
      } else {
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(packed[j]);
        for (int q = 0; q < 8; ++q)
          if (col + 8 * j + q < limit) crow[col + 8 * j + q] = e[q];
      }
    }
  }
}

// One thread's row of a tile of sums: what the epilogue does, in two parts around the wait for the sums.  LEAVE: results go through shared memory.
template <int BN, int HB, bool LEAVE = false>
struct Epilogue {
  static constexpr int BN_HALF = BN / 2, PARTS = store_warps(HB) / 4;
  int pos = 0, page = -1;
  float cs[HB > 0 ? HB : 1][8], sn[HB > 0 ? HB : 1][8];  // HB > 0: the angles of this row's position, all of a head's pairs

  __device__ __forceinline__ void before(int row, int M, int mode, const RopeArgs& rope) {
    if (mode == MODE_ROPE && row < M) {  // this row's token: where it stands and which page takes it (inputs of the step)
      pos = rope.positions[row];
      page = rope.table[(size_t)rope.token_item[row] * rope.table_width + (pos >> rope.page_shift)];
      if (HB > 0 && rope.cos_t) {
        const int safe = pos < 0 ? 0 : (pos >= rope.max_positions ? rope.max_positions - 1 : pos);
        const float4* cp = reinterpret_cast<const float4*>(rope.cos_t + (size_t)safe * (rope.D >> 1));
        const float4* sp = reinterpret_cast<const float4*>(rope.sin_t + (size_t)safe * (rope.D >> 1));
#pragma unroll
        for (int b = 0; b < (HB > 0 ? HB : 1); ++b) {
          const float4 c0 = __ldg(cp + 2 * b), c1 = __ldg(cp + 2 * b + 1), s0 = __ldg(sp + 2 * b), s1 = __ldg(sp + 2 * b + 1);
          cs[b][0] = c0.x; cs[b][1] = c0.y; cs[b][2] = c0.z; cs[b][3] = c0.w; cs[b][4] = c1.x; cs[b][5] = c1.y; cs[b][6] = c1.z; cs[b][7] = c1.w;
          sn[b][0] = s0.x; sn[b][1] = s0.y; sn[b][2] = s0.z; sn[b][3] = s0.w; sn[b][4] = s1.x; sn[b][5] = s1.y; sn[b][6] = s1.z; sn[b][7] = s1.w;
        }
      }
    }
  }
  // two results of a plain product with an activation
  __device__ __forceinline__ static uint32_t activated(float v0, float v1, int mode) {
    if (mode == MODE_RELU2) {
      v0 = fmaxf(v0, 0.f), v1 = fmaxf(v1, 0.f);
      v0 *= v0, v1 *= v1;
    } else if (mode == MODE_SILU || mode == MODE_GELU) {
      const int act = mode == MODE_SILU ? PSB_ACT_SILU : PSB_ACT_GELU_TANH;
      v0 = quick_act(v0, act), v1 = quick_act(v1, act);
    }
    return pack2(v0, v1);
  }
  // ``value``: of the two rounded sums; ``quick`` the same where every |gate sum| * ``rate`` of the 32 is at most QUICK_UP_TO
  template <typename Quick, typename Value>
  __device__ __forceinline__ static void gated_columns(uint32_t taddr, int row, int M, int n0, __nv_bfloat16* crow, int N_out, int ldc, int part, float rate,
                                                       Quick quick, Value value) {
#pragma unroll 1
    for (int c = part * (BN_HALF / PARTS); c < (part + 1) * (BN_HALF / PARTS); c += 32) {
      uint32_t g[32], u[32];
      tmem_ld32(taddr + c, g);
      tmem_ld32(taddr + BN_HALF + c, u);
      tmem_ld_wait();
      if (row >= M) continue;
      auto columns = [&](auto of) {
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          const int col = n0 + c + j;
          uint32_t packed[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            // the reference rounds both projections to bfloat16 before the activation
            const uint32_t gb = pack2(__uint_as_float(g[j + 2 * q]), __uint_as_float(g[j + 2 * q + 1]));
            const uint32_t ub = pack2(__uint_as_float(u[j + 2 * q]), __uint_as_float(u[j + 2 * q + 1]));
            packed[q] = pack2(of(__uint_as_float(gb << 16), __uint_as_float(ub << 16)),
                              of(__uint_as_float(gb & 0xffff0000u), __uint_as_float(ub & 0xffff0000u)));
          }
          if (col + 8 <= N_out && (ldc & 7) == 0) {
            *reinterpret_cast<uint4*>(crow + col) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          } else {
            const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(packed);
            for (int q = 0; q < 8; ++q)
              if (col + q < N_out) crow[col + q] = e[q];
          }
        }
      };
      float top = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) top = fmaxf(top, fabsf(__uint_as_float(g[j])));
      if (top * rate <= QUICK_UP_TO) columns(quick);
      else columns(value);
    }
  }
  // the same, through shared memory
  template <typename Quick, typename Value>
  __device__ __forceinline__ static void gated_columns_leave(uint32_t taddr, int row, int M, int n0, __nv_bfloat16* __restrict__ C, int N_out, int ldc, int part, float rate,
                                                             uint4* leaving, Quick quick, Value value) {
#pragma unroll 1
    for (int c = part * (BN_HALF / PARTS); c < (part + 1) * (BN_HALF / PARTS); c += 32) {
      uint32_t g[32], u[32];
      tmem_ld32(taddr + c, g);
      tmem_ld32(taddr + BN_HALF + c, u);
      tmem_ld_wait();
      if (row - (int)(threadIdx.x & 31) >= M) continue;
      uint32_t packed[4][4] = {};
      auto columns = [&](auto of) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t gb = pack2(__uint_as_float(g[8 * j + 2 * q]), __uint_as_float(g[8 * j + 2 * q + 1]));
            const uint32_t ub = pack2(__uint_as_float(u[8 * j + 2 * q]), __uint_as_float(u[8 * j + 2 * q + 1]));
            packed[j][q] = pack2(of(__uint_as_float(gb << 16), __uint_as_float(ub << 16)),
                                 of(__uint_as_float(gb & 0xffff0000u), __uint_as_float(ub & 0xffff0000u)));
          }
      };
      if (row < M) {
        float top = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) top = fmaxf(top, fabsf(__uint_as_float(g[j])));
        if (top * rate <= QUICK_UP_TO) columns(quick);
        else columns(value);
      }
      leave_rows(leaving, packed, C, row, M, n0 + c, N_out, ldc);
    }
  }
  // (M: rows there are; the tile's columns start at n0; part: which half of the columns, where two warps share the rows)
  __device__ __forceinline__ void store(uint32_t taddr, int row, int M, int n0, __nv_bfloat16* __restrict__ C, int N_out, int ldc, int mode, bool gated,
                                        const RopeArgs& rope, const GluArgs& glu, const float* __restrict__ row_scale, int part, uint4* leaving = nullptr) const {
    __nv_bfloat16* crow = C + (size_t)row * ldc;
    if (mode == MODE_ROPE) {
      rope_store_row<BN, HB>(taddr, row, M, n0, N_out, rope, pos, page, cs, sn, part);
    } else if (gated) {
      // the activation is chosen once a tile, not once a number
      const float rs = mode == MODE_GATED_SCALED && row < M ? row_scale[row] : 1.f;
      auto gate = [&](float rate, auto quick, auto value) {
        if constexpr (LEAVE) gated_columns_leave(taddr, row, M, n0, C, N_out, ldc, part, rate, leaving, quick, value);
        else gated_columns(taddr, row, M, n0, crow, N_out, ldc, part, rate, quick, value);
      };
      if (mode == MODE_GATED) {
        gate(1.f, [](float g, float u) { return divided(g, 1.f + __expf(-g)) * u; }, [](float g, float u) { return g / (1.f + __expf(-g)) * u; });
      } else if (mode == MODE_GATED_SCALED) {
        gate(fabsf(rs), [rs](float g, float u) { return divided(rs * g, 1.f + __expf(-rs * g)) * (rs * u); },
             [rs](float g, float u) { return rs * g / (1.f + __expf(-rs * g)) * (rs * u); });
      } else if (mode == MODE_GATED_CLIPPED) {
        gate(fabsf(glu.alpha), [&](float g, float u) {
          g = fminf(g, glu.limit);
          return divided(g, 1.f + expf(-glu.alpha * g)) * (fminf(fmaxf(u, -glu.limit), glu.limit) + glu.offset);
        }, [&](float g, float u) { return clipped_gate_value(g, u, glu); });
      } else {
        auto value = [](float g, float u) { return gate_act(g, PSB_ACT_GELU_TANH) * u; };
        gate(1.f, value, value);
      }
    } else {
      constexpr int MINE = part_columns(BN, PARTS);
#pragma unroll 1
      for (int c = part * MINE; c < BN && c < (part + 1) * MINE; c += 32) {
        uint32_t v[32];
        tmem_ld32(taddr + c, v);  // (a tile of 240 columns: the last load reads 16 columns beyond it, which nobody stores)
        tmem_ld_wait();
        if constexpr (LEAVE) {
          static_assert(BN % 32 == 0, "whole runs of columns");
          if (row - (int)(threadIdx.x & 31) >= M) continue;
          uint32_t packed[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) packed[j][q] = activated(__uint_as_float(v[8 * j + 2 * q]), __uint_as_float(v[8 * j + 2 * q + 1]), mode);
          leave_rows(leaving, packed, C, row, M, n0 + c, N_out, ldc);
        } else if (row < M) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (BN % 32 != 0 && c + j >= BN) break;
            const int col = n0 + c + j;
            uint32_t packed[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) packed[q] = activated(__uint_as_float(v[j + 2 * q]), __uint_as_float(v[j + 2 * q + 1]), mode);
            if (col + 8 <= N_out && (ldc & 7) == 0) {
              *reinterpret_cast<uint4*>(crow + col) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            } else {
              const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(packed);
              for (int q = 0; q < 8; ++q)
                if (col + q < N_out) crow[col + q] = e[q];
            }
          }
        }
      }
    }
  }
};

// BN: see Tile.  HB: see rope_store_row (0 unless mode is MODE_ROPE and the head size is 16 * HB).
template <int BN, int HB>
__global__ void __launch_bounds__(threads(HB), 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    __nv_bfloat16* __restrict__ C, int M, int N_out, int K, int ldc, int up_offset, int mode,
                    const RopeArgs rope, const int32_t* __restrict__ tile_expert, const GluArgs glu,
                    const float* __restrict__ row_scale) {
  using T = Tile<BN>;
  constexpr int BN_HALF = T::HALF, STAGES = T::STAGES, STAGE_BYTES = T::STAGE_BYTES;
  constexpr uint32_t INSTR_DESC = instr_desc(BM, BN, false);  // M=128, N=BN, both operands K-major
  const bool gated = mode_is_gated(mode);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(tiles + STAGES * STAGE_BYTES);
  volatile uint32_t* abort = &bars->abort;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;  // the warp's role is the same for all its lanes

  const int n_span = gated ? BN_HALF : BN;  // output columns one tile covers
  const int m_blocks = (M + BM - 1) / BM;
  const int n_blocks = (N_out + n_span - 1) / n_span;
  const int tiles_total = m_blocks * n_blocks;
  const int k_blocks = (K + BK - 1) / BK;

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], store_warps(HB));  // one arrival per epilogue warp
    }
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {  // one warp allocates (and later frees) the tensor memory
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();  // A is the preceding kernel's output

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < tiles_total; tile += gridDim.x) {
        const int m0 = (tile % m_blocks) * BM;
        int n0 = (tile / m_blocks) * n_span;
        if (tile_expert) {
          const int expert = tile_expert[tile % m_blocks];
          if (expert < 0) continue;
          n0 += expert * (gated ? 2 * N_out : N_out);  // a gated expert holds its gate rows, then its up rows
        }
        const int n1 = gated ? up_offset + n0 : n0 + BN_HALF;
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait(&bars->empty[stage], phase ^ 1, abort, 1);
          if (!ok) break;
          unsigned char* a_dst = tiles + stage * STAGE_BYTES;
          unsigned char* b_dst = a_dst + A_BYTES;
          mbar_expect_tx(&bars->full[stage], STAGE_BYTES);
          tma_load_2d(a_dst, &map_a, kb * BK, m0, &bars->full[stage]);
          tma_load_2d(b_dst, &map_w, kb * BK, n0, &bars->full[stage]);
          tma_load_2d(b_dst + BN_HALF * BK * 2, &map_w, kb * BK, n1, &bars->full[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------------- MMA
    // The whole warp runs this loop and waits on the barriers; each tensor-core instruction is issued by one elected
    // lane (tcgen05.cuh says why).
    {
      uint32_t stage = 0, phase = 0, local = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < tiles_total; tile += gridDim.x) {
        if (tile_expert && tile_expert[tile % m_blocks] < 0) continue;  // an empty tile uses no accumulator buffer
        const uint32_t buf = local & 1, use = local >> 1;  // accumulator buffer and how often it has been used
        ++local;
        ok = mbar_wait(&bars->acc_empty[buf], (use & 1) ^ 1, abort, 4);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        fence_after();
        const uint32_t acc = tmem_base + buf * ACC_STRIDE;
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait(&bars->full[stage], phase, abort, 2);  // filled by TMA: no tensor-memory fence needed
          if (!ok) break;
          const uint64_t da = smem_desc(smem_u32(tiles + stage * STAGE_BYTES));
          const uint64_t db = smem_desc(smem_u32(tiles + stage * STAGE_BYTES + A_BYTES));
          const uint32_t hi = (uint32_t)(da >> 32), a_lo = (uint32_t)da, b_lo = (uint32_t)db;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            // 16 elements = 32 bytes further along K inside the swizzled 128-byte rows: 2 in the address field
            if (elect_one()) mma_f16_split(acc, a_lo + 2 * k, hi, b_lo + 2 * k, hi, INSTR_DESC, (kb | k) != 0);
          }
          if (elect_one()) mma_commit(&bars->empty[stage]);  // arrives when the MMAs that read this stage are done
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && elect_one()) mma_commit(&bars->acc_full[buf]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3;  // a warp may only read tensor-memory lanes [32*(warp%4), +32)
    uint32_t local = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < tiles_total; tile += gridDim.x) {
      if (tile_expert && tile_expert[tile % m_blocks] < 0) continue;
      const uint32_t buf = local & 1, use = local >> 1;
      ++local;
      const int m0 = (tile % m_blocks) * BM;
      const int n0 = (tile / m_blocks) * n_span;
      const int row = m0 + quarter * 32 + lane;
      Epilogue<BN, HB> epilogue;
      epilogue.before(row, M, mode, rope);
      ok = mbar_wait(&bars->acc_full[buf], use & 1, abort, 3);
      if (!ok) break;
      fence_after();
      const uint32_t taddr = tmem_base + buf * ACC_STRIDE + ((uint32_t)(quarter * 32) << 16);
      epilogue.store(taddr, row, M, n0, C, N_out, ldc, mode, gated, rope, glu, row_scale, (warp - 2) >> 2);
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[buf]);  // this warp has read its part of the buffer
    }
  }

  if (*abort) {
    // something gave up: give copies in flight time to land before the shared memory is handed to another CTA
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  fence_before();
  __syncthreads();
  if (warp == 2) {
    fence_after();
    tmem_free(tmem_base, TMEM_COLS);
  }
}

// ---- two CTAs on a tile of 256 rows by 256 columns ---------------------------------------------------------------------
//
// The same roles, in clusters of two CTAs (tcgen05 cta_group::2): each CTA brings its 128 rows of A and half of the tile's rows of W (the
// gate's and the up rows, for the gated forms), the first one's MMA warp multiplies for both (M=256, N=256, K=16), and each CTA's
// epilogue stores its own rows.  A stage is 32 KB instead of 48 for the same work, an operand of W crosses from L2 once for 256 rows, and six
// stages are in flight.  The first CTA's full barriers count the bytes of both; commits arrive at both CTAs' barriers.
//
// Grouped products: a tile is a row tile of 128 and the next one if that is the same expert's (an expert's odd last one is a tile by itself whose other
// half is computed against the wrong matrix and not stored); the CTAs list the tiles that hold rows first, so that every pair gets as many (dealt out
// by the grid's stride with the empty ones among them, some CTAs had six and others two: 160 and 55 us for the products above, one CTA a tile).
//
// 1,979 tokens, K 4,096, 14,336 gated columns: 305 us on a cool GPU and 312 with one CTA a tile; in a loop, where power is the limit, both products of
// the feed-forward take 557 us instead of 580.
constexpr int PAIR_STAGES = 6, PAIR_STAGE = A_BYTES + 128 * BK * 2, MAX_UNITS = 2048;
constexpr int PAIR_SMEM = PAIR_STAGES * PAIR_STAGE + 1024 + 256 + MAX_UNITS * 2 + LEAVING_BYTES;
constexpr int ALONE = 1 << 15;  // the unit's second row tile is another expert's
static_assert(PAIR_STAGES <= MAX_STAGES && PAIR_SMEM <= 227 * 1024, "beyond a CTA's shared memory");

template <int HB>
__global__ void __launch_bounds__(threads(HB), 1)
gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                         __nv_bfloat16* __restrict__ C, int M, int N_out, int K, int ldc, int up_offset, int mode,
                         const RopeArgs rope, const int32_t* __restrict__ tile_expert, const GluArgs glu,
                         const float* __restrict__ row_scale) {
  constexpr int BN = 256, BN_HALF = BN / 2, STAGES = PAIR_STAGES;
  constexpr uint32_t INSTR_DESC = instr_desc(2 * BM, BN, false);
  const bool gated = mode_is_gated(mode);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(tiles + STAGES * PAIR_STAGE);
  uint16_t* units = reinterpret_cast<uint16_t*>(tiles + STAGES * PAIR_STAGE + 256);
  volatile uint32_t* abort = &bars->abort;
  __shared__ int listed;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  const int n_span = gated ? BN_HALF : BN;
  const int m_tiles = (M + BM - 1) / BM;
  const int n_blocks = (N_out + n_span - 1) / n_span;
  const int k_blocks = (K + BK - 1) / BK;

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], 2 * store_warps(HB));  // one arrival per epilogue warp of either CTA
    }
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) tmem_alloc_pair(&bars->tmem_base, TMEM_COLS);
  fence_before();
  pdl_wait();  // A and the tiles' experts are the preceding kernels' output
  if (tile_expert && warp == 0) {
    int count = 0, run = 0, last = -1;  // units listed; row tiles of ``last`` so far
    for (int t0 = 0; t0 < m_tiles; t0 += 32) {
      const int t = t0 + lane;
      const int expert = t < m_tiles ? tile_expert[t] : -1, next = t + 1 < m_tiles ? tile_expert[t + 1] : -1;
      int before = __shfl_up_sync(0xffffffffu, expert, 1);
      if (lane == 0) before = last;
      const uint32_t starts = __ballot_sync(0xffffffffu, expert != before), upto = starts & (0xffffffffu >> (31 - lane));
      const int place = upto ? lane - (31 - __clz(upto)) : run + lane;  // of its expert's row tiles
      const bool opens = expert >= 0 && !(place & 1);
      const uint32_t opening = __ballot_sync(0xffffffffu, opens);
      const int at = count + __popc(opening & ((1u << lane) - 1));
      if (opens && at < MAX_UNITS) units[at] = (uint16_t)(t | (next == expert ? 0 : ALONE));
      count += __popc(opening);
      last = __shfl_sync(0xffffffffu, expert, 31);
      run = __shfl_sync(0xffffffffu, place, 31) + 1;
    }
    if (lane == 0) listed = count < MAX_UNITS ? count : MAX_UNITS;
  }
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are there
  fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  const int m_units = tile_expert ? listed : (m_tiles + 1) / 2;
  const int tiles_total = m_units * n_blocks;
  // Tile -> row tile (its first), column tile, expert, and whether the second row tile counts.  Ungrouped, neighbours in time share a run of W and all of A
  // is in use; grouped, they share an expert's rows, and its matrix is read from one end to the other.
  struct Where {
    int m0, n0, expert;
    bool both;
  };
  auto where = [&](int tile) {
    Where w;
    if (tile_expert) {
      const int u = units[tile / n_blocks];
      w.n0 = tile % n_blocks * n_span;
      w.both = !(u & ALONE);
      w.m0 = (u & (ALONE - 1)) * BM;
      w.expert = tile_expert[u & (ALONE - 1)];
    } else {
      w.m0 = tile % m_units * 2 * BM;
      w.n0 = tile / m_units * n_span;
      w.both = true;
      w.expert = 0;
    }
    return w;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < tiles_total; tile += pairs) {
        const Where w = where(tile);
        const int m0 = w.m0 + rank * BM;
        int n0 = w.n0 + w.expert * (gated ? 2 * N_out : N_out);  // a gated expert holds its gate rows, then its up rows
        if (rank) n0 += gated ? up_offset : BN_HALF;
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait(&bars->empty[stage], phase ^ 1, abort, 1);
          if (!ok) break;
          unsigned char* a_dst = tiles + stage * PAIR_STAGE;
          if (rank == 0) mbar_expect_tx(&bars->full[stage], 2 * PAIR_STAGE);
          const uint32_t full = cluster_address(&bars->full[stage], 0);
          tma_load_2d_pair(a_dst, &map_a, kb * BK, m0, full);
          tma_load_2d_pair(a_dst + A_BYTES, &map_w, kb * BK, n0, full);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------------- MMA
    if (rank == 0) {
      uint32_t stage = 0, phase = 0, local = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < tiles_total; tile += pairs) {
        const uint32_t buf = local & 1, use = local >> 1;
        ++local;
        ok = mbar_wait(&bars->acc_empty[buf], (use & 1) ^ 1, abort, 4);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        fence_after();
        const uint32_t acc = tmem_base + buf * ACC_STRIDE;
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait(&bars->full[stage], phase, abort, 2);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const uint64_t da = smem_desc(smem_u32(tiles + stage * PAIR_STAGE));
          const uint64_t db = smem_desc(smem_u32(tiles + stage * PAIR_STAGE + A_BYTES));
          const uint32_t hi = (uint32_t)(da >> 32), a_lo = (uint32_t)da, b_lo = (uint32_t)db;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            if (elect_one()) mma_f16_split_pair(acc, a_lo + 2 * k, hi, b_lo + 2 * k, hi, INSTR_DESC, (kb | k) != 0);
          if (elect_one()) mma_commit_pair(&bars->empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && elect_one()) mma_commit_pair(&bars->acc_full[buf]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    uint32_t local = 0;
    bool ok = true;
    for (int tile = pair; ok && tile < tiles_total; tile += pairs) {
      const uint32_t buf = local & 1, use = local >> 1;
      ++local;
      const Where w = where(tile);
      const int row = w.m0 + rank * BM + quarter * 32 + lane, rows = rank && !w.both ? 0 : M;
      Epilogue<BN, HB, true> epilogue;
      epilogue.before(row, rows, mode, rope);
      ok = mbar_wait(&bars->acc_full[buf], use & 1, abort, 3);
      if (!ok) break;
      fence_after();
      epilogue.store(tmem_base + buf * ACC_STRIDE + ((uint32_t)(quarter * 32) << 16), row, rows, w.n0, C, N_out, ldc, mode, gated, rope, glu, row_scale, (warp - 2) >> 2,
                     reinterpret_cast<uint4*>(tiles + PAIR_STAGES * PAIR_STAGE + 256 + MAX_UNITS * 2 + (warp - 2) * LEAVING_WARP));
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_address(&bars->acc_empty[buf], 0));
    }
  }
  __syncwarp();
  if (*abort) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight, as above
  }
  fence_before();
  __syncthreads();
  cluster_sync_all();  // the first CTA's instructions read the other's shared memory, and both arrive at each other's barriers
  if (warp == 2) {
    fence_after();
    tmem_free_pair(tmem_base, TMEM_COLS);
  }
}

// ---- host side -----------------------------------------------------------------------------------------------
// row-major [rows, K] bfloat16 matrix, box of 64 columns x box_rows rows
int make_map(CUtensorMap* map, const void* base, int rows, int K, int box_rows) {
  const int r = make_map_bf16(map, base, (uint64_t)rows, (uint64_t)K, (uint64_t)K, box_rows);
  if (r == -1) PSB_REFUSE("gemm_tcgen05: the driver does not export cuTensorMapEncodeTiled");
  if (r != 0) PSB_REFUSE("gemm_tcgen05: cuTensorMapEncodeTiled failed with code %d (rows=%d K=%d)", r, rows, K);
  return 0;
}

int g_forced_width = 0;  // 0: the launcher chooses the tile width; 128, 192 or 256: tests compare them

// The tile width for a product: the one that gets it done in the fewest, shortest rounds over the SMs.  A round of
// tiles costs its width in tensor-core time plus a fixed share (first loads, the epilogue of the last tile).  The gated
// form needs an even split into gate and up columns and heads of 128 held in registers need whole heads: no 192.
int choose_width(int M, int N_out, bool gated, bool rope, int D, int sms) {
  const int m_blocks = (M + BM - 1) / BM;
  int best = 256;
  long best_cost = -1;
  for (int bn : {256, 240, 192, 128}) {
    if (bn == 192 && (gated || (rope && D == 128))) continue;
    if (bn == 240 && (gated || rope)) continue;  // whole heads and even halves want a power of two or 192
    if (g_forced_width && g_forced_width != 512 && bn != g_forced_width) continue;
    const int span = gated ? bn / 2 : bn;
    const long tiles = (long)m_blocks * ((N_out + span - 1) / span);
    const long cost = ((tiles + sms - 1) / sms) * (bn + 24);
    // from the widest down: a narrower tile has to pay for itself (240 against 256 is the same kernel but for the width)
    if (best_cost < 0 || (bn == 240 ? cost < best_cost : cost * 10 <= best_cost * 9)) {
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}

// Whether two CTAs a tile get the product done sooner, by rounds: theirs of 256 x 256 takes about six sevenths of a single CTA's of 128 x 256 (the same work
// an SM), the narrower tiles' as in choose_width.  Columns by K, rows, two CTAs against the best single width in us: 4,096 by 14,336, 1,979 rows 152 and
// 176, 1,024 82 and 96, 700 (one round of 192 columns) 81 and 77; 2,048 by 8,192, 1,979 rows 53 and 61; 6,144 by 4,096, 1,979 rows 74 and 83;
// 3,072 by 2,048, 1,979 rows (two rounds of 192) 35 and 30; gated 14,336 by 4,096, 1,024 rows 158 and 174.
//
// Grouped products (``experts`` > 0; the rows hold up to 127 of nobody an expert): rounds depend on the routing, which is not known here, so for rows dealt out
// evenly, half of the experts with an odd last row tile.  A pair brings W in once for 256 rows, but an expert's only (or odd last) row tile keeps just one of
// its CTAs busy.  What a tile costs beside its K, in columns, was fitted to experts of 4 to 256 rows on average, columns by K, us in pairs and single:
// 32 of 2,048 by 2,048, 8 rows 76 and 70, 48 rows 76 and 81, 256 rows 84 and 116; 32 of 2,048 by 1,024 47 and 43, 48 and 49, 55 and 66; 8 of 2,048 by 2,048,
// 32 rows 31 and 27; 64 of 1,536 by 2,048, 8 rows 104 and 102, 64 rows 104 and 113; 128 of them, 4 rows 173 and 205; 32 of 4,096 by 4,096, 8 rows 215 and 217,
// 64 rows 215 and 245.  Short contractions are bounded by the stores of their tiles, of which pairs do half as many at once: 64 of 1,024 by 512, 8 rows
// 39 and 29, 256 rows 51 and 44.
bool pairs_pay(int M, int N_out, int K, bool gated, int bn, int experts, int sms) {
  if (sms < 2 || (M + BM - 1) / BM > MAX_UNITS) return false;
  if (g_forced_width) return g_forced_width == 512;
  const long m_blocks = (M + BM - 1) / BM, span = gated ? bn / 2 : bn, span2 = gated ? 128 : 256, n_blocks = (N_out + span2 - 1) / span2;
  const long rounds = (m_blocks * ((N_out + span - 1) / span) + sms - 1) / sms;
  if (experts > 0) {
    if (K < 768) return false;
    const long rows = std::max(1L, (long)M - 127L * experts), units = std::min(rows, std::max((long)experts, (rows + 255) / 256 + experts / 2));
    const long rounds2 = (units * n_blocks + sms / 2 - 1) / (sms / 2);
    return (10 * rounds2 + 11) * (115 + 36000 / K) <= 10 * rounds * (bn + 24);
  }
  const long rounds2 = ((m_blocks + 1) / 2 * n_blocks + sms / 2 - 1) / (sms / 2);
  return rounds2 * (256 + 24) * 6 <= rounds * (bn + 24) * 7;
}

// ``tiles``: at most so many.  As many pairs as the device holds at once (asked once per device), no more than sms / 2.
template <int HB>
int launch_pairs(int tiles, int sms, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_w, void* c, int M, int N_out, int K, int ldc,
                 int up_offset, int mode, const RopeArgs& rope, const int32_t* tile_expert, const GluArgs& glu, const float* row_scale) {
  static PsbPerDevice configured;
  static int resident[PsbPerDevice::kMaxDevices] = {};
  auto kernel = gemm_tcgen05_pair_kernel<HB>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (sms / 2));
  cfg.blockDim = dim3(threads(HB));
  cfg.dynamicSmemBytes = PAIR_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int dev = PsbPerDevice::current();
  if (!configured.get()) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM);
    if (e != cudaSuccess) PSB_REFUSE("gemm_tcgen05: cannot reserve %d bytes of shared memory: %s", PAIR_SMEM, cudaGetErrorString(e));
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = sms / 2;
    }
    if (dev >= 0) resident[dev] = n;
    configured.set();
  }
  int pairs = dev >= 0 && resident[dev] > 0 && resident[dev] < sms / 2 ? resident[dev] : sms / 2;
  if (tiles < pairs) pairs = tiles;
  cfg.gridDim = dim3(2 * pairs);
  if (psb_pdl_enabled) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cudaLaunchKernelEx(&cfg, kernel, map_a, map_w, (__nv_bfloat16*)c, M, N_out, K, ldc, up_offset, mode, rope, tile_expert, glu, row_scale);
  PSB_LAUNCH_CHECK("gemm_tcgen05");
  return 0;
}

int launch(const void* a, const void* w, void* c, int M, int w_rows, int N_out, int K, int up_offset, int mode, int sms,
           cudaStream_t stream, const RopeArgs& rope = RopeArgs{}, const int32_t* tile_expert = nullptr,
           const GluArgs& glu = GluArgs{}, const float* row_scale = nullptr, int ldc = 0) {
  const bool gated = mode == MODE_GATED || mode == MODE_GATED_GELU || mode == MODE_GATED_CLIPPED || mode == MODE_GATED_SCALED;
  if (ldc == 0) ldc = N_out;
  if (ldc < N_out) PSB_REFUSE("gemm_tcgen05: output rows %d numbers apart do not hold %d", ldc, N_out);
  if (M < 1 || N_out < 1 || K < 8 || K % 8) PSB_REFUSE("gemm_tcgen05: needs K a multiple of 8 (M=%d N=%d K=%d)", M, N_out, K);
  if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)c) & 15) PSB_REFUSE("gemm_tcgen05: operands must be 16-byte aligned");
  const int experts = tile_expert ? w_rows / (gated ? 2 * N_out : N_out) : 0;
  const int m_blocks = (M + BM - 1) / BM;
  const int bn = choose_width(M, N_out, gated, mode == MODE_ROPE, rope.D, sms);
  CUtensorMap map_a, map_w;
  if (int rc = make_map(&map_a, a, M, K, BM)) return rc;
  if (pairs_pay(M, N_out, K, gated, bn, experts, sms)) {
    if (int rc = make_map(&map_w, w, w_rows, K, 128)) return rc;
    const int span = gated ? 128 : 256, most = (tile_expert ? m_blocks : (m_blocks + 1) / 2) * ((N_out + span - 1) / span);
    if (mode == MODE_ROPE && rope.D == 128) return launch_pairs<8>(most, sms, stream, map_a, map_w, c, M, N_out, K, ldc, up_offset, mode, rope, tile_expert, glu, row_scale);
    if (mode == MODE_ROPE && rope.D == 64) return launch_pairs<4>(most, sms, stream, map_a, map_w, c, M, N_out, K, ldc, up_offset, mode, rope, tile_expert, glu, row_scale);
    return launch_pairs<0>(most, sms, stream, map_a, map_w, c, M, N_out, K, ldc, up_offset, mode, rope, tile_expert, glu, row_scale);
  }
  if (int rc = make_map(&map_w, w, w_rows, K, bn / 2)) return rc;
  const int n_span = gated ? bn / 2 : bn;
  const int tiles = m_blocks * ((N_out + n_span - 1) / n_span);
  const int grid = tiles < sms ? tiles : sms;
#define PSB_TCGEN05(BN, HB)                                                                                          \
  do {                                                                                                               \
    static PsbPerDevice configured;  /* more than 48 KB of dynamic shared memory has to be asked for once */           \
    if (!configured.get()) {                                                                                               \
      cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, HB>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                           Tile<BN>::SMEM_BYTES);                                                    \
      if (e != cudaSuccess) PSB_REFUSE("gemm_tcgen05: cannot reserve %d bytes of shared memory: %s", Tile<BN>::SMEM_BYTES, cudaGetErrorString(e)); \
      configured.set();                                                                                              \
    }                                                                                                                \
    psb_launch(gemm_tcgen05_kernel<BN, HB>, dim3(grid), dim3(threads(HB)), (size_t)Tile<BN>::SMEM_BYTES, stream, map_a,   \
               map_w, (__nv_bfloat16*)c, M, N_out, K, ldc, up_offset, mode, rope, tile_expert, glu, row_scale);      \
  } while (0)
  // the usual head sizes keep a row's angles in registers; every other multiple of 16 fetches them block by block
  if (mode == MODE_ROPE && rope.D == 128) { if (bn == 128) PSB_TCGEN05(128, 8); else PSB_TCGEN05(256, 8); }
  else if (mode == MODE_ROPE && rope.D == 64) { if (bn == 128) PSB_TCGEN05(128, 4); else if (bn == 192) PSB_TCGEN05(192, 4); else PSB_TCGEN05(256, 4); }
  else if (bn == 128) PSB_TCGEN05(128, 0);
  else if (bn == 192) PSB_TCGEN05(192, 0);
  else if (bn == 240) PSB_TCGEN05(240, 0);
  else PSB_TCGEN05(256, 0);
#undef PSB_TCGEN05
  PSB_LAUNCH_CHECK("gemm_tcgen05");
  return 0;
}

}  // namespace

// C[M,N] = A[M,K] W[N,K]^T, all bfloat16 row-major, K % 8 == 0.  sms: CTAs to launch at most (the SM count).
PSB_API int psb_gemm_tcgen05(const void* a, const void* w, void* c, int M, int N, int K, int sms, cudaStream_t stream) {
  return launch(a, w, c, M, N, N, K, 0, MODE_PLAIN, sms, stream);
}

// C[M,N] = f(A W^T), f the activation named by its code (PsbAct), in rows ldc numbers apart.
PSB_API int psb_gemm_tcgen05_unary(const void* a, const void* w, void* c, int M, int N, int K, int ldc, int sms, int activation,
                                   cudaStream_t stream) {
  if (!psb_activation_known(activation)) PSB_REFUSE("gemm_tcgen05_unary: activation code %d is not built", activation);
  return launch(a, w, c, M, N, N, K, 0, activation == PSB_ACT_SILU ? MODE_SILU : MODE_GELU, sms, stream, RopeArgs{}, nullptr, GluArgs{}, nullptr, ldc);
}

// act[M,I] = f(A Wg^T) * (A Wu^T) for W = [Wg; Wu] of shape [2I, K], f the activation named by its code (PsbAct).
PSB_API int psb_gemm_tcgen05_gated(const void* a, const void* w, void* act, int M, int I, int K, int sms, int activation,
                                   cudaStream_t stream) {
  if (!psb_activation_known(activation)) PSB_REFUSE("gemm_tcgen05_gated: activation code %d is not built", activation);
  return launch(a, w, act, M, 2 * I, I, K, I, activation == PSB_ACT_SILU ? MODE_GATED : MODE_GATED_GELU, sms, stream);
}

// The same with both branches clipped before they meet: act = g * sigmoid(alpha g) * (u + offset), g = min(A Wg^T, limit),
// u = clamp(A Wu^T, -limit, limit), both rounded to bfloat16 first, as the product without the activation would leave them.
PSB_API int psb_gemm_tcgen05_gated_clipped(const void* a, const void* w, void* act, int M, int I, int K, int sms, float limit,
                                           float alpha, float offset, cudaStream_t stream) {
  if (!(limit > 0.f)) PSB_REFUSE("gemm_tcgen05_gated_clipped: the limit must be positive");
  return launch(a, w, act, M, 2 * I, I, K, I, MODE_GATED_CLIPPED, sms, stream, RopeArgs{}, nullptr, GluArgs{limit, alpha, offset});
}

// Grouped: C[M, N] = act(A[M, K] W[e]^T) where W is [experts, N, K] and the rows of A lie expert by expert, every
// expert's rows starting at a multiple of 128; tile_expert [M / 128 rounded up] (device) names the expert of every
// 128-row tile or -1 for a tile without rows.  relu2: store max(sum, 0)^2.
PSB_API int psb_gemm_tcgen05_grouped(const void* a, const void* w, void* c, int M, int N, int K, int experts, const void* tile_expert,
                                     int relu2, int sms, cudaStream_t stream) {
  if (experts < 1 || !tile_expert) PSB_REFUSE("gemm_tcgen05_grouped: needs the experts and the tiles' experts");
  if ((long long)experts * N > 0x7fffffffLL) PSB_REFUSE("gemm_tcgen05_grouped: too many rows in the stack of matrices");
  return launch(a, w, c, M, experts * N, N, K, 0, relu2 ? MODE_RELU2 : MODE_PLAIN, sms, stream, RopeArgs{}, (const int32_t*)tile_expert);
}

// Grouped and gated: act[M, I] = g * sigmoid(alpha g) * (u + offset) with g = min(A Wg[e]^T, limit), u = clamp(A Wu[e]^T,
// -limit, limit) for W = [experts, 2 I, K], an expert's gate rows followed by its up rows; rows of A and tile_expert as above.
PSB_API int psb_gemm_tcgen05_grouped_gated_clipped(const void* a, const void* w, void* act, int M, int I, int K, int experts,
                                                   const void* tile_expert, float limit, float alpha, float offset, int sms,
                                                   cudaStream_t stream) {
  if (experts < 1 || !tile_expert) PSB_REFUSE("gemm_tcgen05_grouped_gated_clipped: needs the experts and the tiles' experts");
  if ((long long)experts * 2 * I > 0x7fffffffLL) PSB_REFUSE("gemm_tcgen05_grouped_gated_clipped: too many rows in the stack of matrices");
  if (!(limit > 0.f)) PSB_REFUSE("gemm_tcgen05_grouped_gated_clipped: the limit must be positive");
  return launch(a, w, act, M, experts * 2 * I, I, K, I, MODE_GATED_CLIPPED, sms, stream, RopeArgs{}, (const int32_t*)tile_expert,
                GluArgs{limit, alpha, offset});
}

// Grouped and gated with SiLU: act[M, I] = silu(r g) * (r u) with g = A Wg[e]^T, u = A Wu[e]^T and r = row_weight[row] (float32
// [M], or null: one).
PSB_API int psb_gemm_tcgen05_grouped_gated_silu(const void* a, const void* w, void* act, int M, int I, int K, int experts,
                                                const void* tile_expert, const void* row_weight, int sms, cudaStream_t stream) {
  if (experts < 1 || !tile_expert) PSB_REFUSE("gemm_tcgen05_grouped_gated_silu: needs the experts and the tiles' experts");
  if ((long long)experts * 2 * I > 0x7fffffffLL) PSB_REFUSE("gemm_tcgen05_grouped_gated_silu: too many rows in the stack of matrices");
  return launch(a, w, act, M, experts * 2 * I, I, K, I, row_weight ? MODE_GATED_SCALED : MODE_GATED, sms, stream, RopeArgs{}, (const int32_t*)tile_expert, GluArgs{},
                (const float*)row_weight);
}

// The projection of an attention layer for many tokens: A W^T with W = [queries; keys; values] [(hq + 2 hkv) D, K] in the
// pair-interleaved row order described at RopeArgs (common.cuh); queries rotated into q_out [M, hq, D], keys rotated
// and values as they are stored at the tokens' positions in the pages: what psb_gemm_tcgen05 followed by
// psb_rope_append in its paired form would do, without the [M, (hq + 2 hkv) D] matrix in between.
PSB_API int psb_gemm_tcgen05_rope(const void* a, const void* w, int M, int K, int sms, const void* positions, const void* token_item,
                                  const void* table, int table_width, const void* cos_t, const void* sin_t, void* kv, void* q_out,
                                  int hq, int hkv, int D, int page_size, int num_pages, int max_positions, cudaStream_t stream) {
  if (hq < 1 || hkv < 1 || D < 16 || D % 16) PSB_REFUSE("gemm_tcgen05_rope: needs a head size that is a multiple of 16 (hq=%d hkv=%d D=%d)", hq, hkv, D);
  if (page_size < 1 || (page_size & (page_size - 1)) || num_pages < 1 || table_width < 1) PSB_REFUSE("gemm_tcgen05_rope: page size %d must be a power of two (pages=%d, width=%d)", page_size, num_pages, table_width);
  if (!positions || !token_item || !table || !kv || !q_out) PSB_REFUSE("gemm_tcgen05_rope: cache arguments missing");
  if ((cos_t == nullptr) != (sin_t == nullptr) || (cos_t && max_positions < 1)) PSB_REFUSE("gemm_tcgen05_rope: angle tables incomplete");
  if (((uintptr_t)kv | (uintptr_t)q_out | (uintptr_t)cos_t | (uintptr_t)sin_t) & 31) PSB_REFUSE("gemm_tcgen05_rope: cache, queries and angle tables must be 32-byte aligned");
  RopeArgs rope;
  rope.positions = (const int32_t*)positions; rope.token_item = (const int32_t*)token_item; rope.table = (const int32_t*)table;
  rope.cos_t = (const float*)cos_t; rope.sin_t = (const float*)sin_t; rope.kv = (__nv_bfloat16*)kv; rope.q_out = (__nv_bfloat16*)q_out;
  rope.table_width = table_width; rope.hq = hq; rope.hkv = hkv; rope.D = D; rope.num_pages = num_pages; rope.max_positions = max_positions;
  rope.page_shift = 0;
  while ((1 << rope.page_shift) < page_size) ++rope.page_shift;
  const int N = (hq + 2 * hkv) * D;
  return launch(a, w, q_out, M, N, N, K, 0, MODE_ROPE, sms, stream, rope);
}

// For tests: 128, 192, 240 or 256 makes every later product use that tile width where the shape allows it, 512 two CTAs a tile of 256 x 256, 0 gives
// the choice back.
PSB_API int psb_gemm_tcgen05_tile_width(int width) {
  if (width != 0 && width != 128 && width != 192 && width != 240 && width != 256 && width != 512) PSB_REFUSE("gemm_tcgen05: tile widths are 128, 192, 240, 256 and 512, not %d", width);
  g_forced_width = width;
  return 0;
}

// (M, N, K, experts, gated, sms) -> 1 if the product goes two CTAs a tile (experts 0: not grouped; N: columns of the result; not for the rotating one)
PSB_API int psb_gemm_tcgen05_pairs(int M, int N_out, int K, int experts, int gated, int sms) {
  if (M < 1 || N_out < 1 || K < 8 || experts < 0 || sms < 1) return 0;
  return pairs_pay(M, N_out, K, gated != 0, choose_width(M, N_out, gated != 0, false, 0, sms), experts, sms) ? 1 : 0;
}

// How many output tiles the kernel would cut a product into (kind: 0 plain [M, N], 1 gated [M, N] from 2N rows, 2 the
// projection that rotates, with heads of D).  The host sends products with too few tiles for the SMs elsewhere.
PSB_API int psb_gemm_tcgen05_tiles(int M, int N_out, int kind, int D, int sms) {
  if (M < 1 || N_out < 1 || sms < 1) return 0;
  const int bn = choose_width(M, N_out, kind == 1, kind == 2, D, sms);
  const int span = kind == 1 ? bn / 2 : bn;
  return ((M + BM - 1) / BM) * ((N_out + span - 1) / span);
}

// 0 while no bounded wait has ever run out on the current device; reading it synchronises with the device.
PSB_API int psb_tcgen05_status() {
  return tc::read_status();
}
