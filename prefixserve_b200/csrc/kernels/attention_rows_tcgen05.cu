// Causal attention of prompt portions over cache rows that hold a key and then its value, on the 5th-generation tensor cores:
// heads of 128 over pages [pages, hkv, page_size, 128 + 128], with a window (and kept first keys), a chunk mask, a cap on the
// scores or a distance bias, a sink and an output gate, as attention_biased.cu defines them.
//
// A CTA owns 128 consecutive new tokens of one request, for two query heads that read the same key/value head (one where no
// two do): two tiles of 128 rows over the same keys, which alternate on the tensor cores.  Keys come in blocks of 64 aligned
// to absolute positions.  352 threads:
//   warp 0      TMA: the tiles' queries once, then per block the keys and the values of its pages into a ring of stages;
//   warp 10     S = Q K^T (tcgen05.mma, M = 128, N = 64) into four tensor-memory buffers in turn;
//   warp 1      O += P V (A from tensor memory), both tiles' O in tensor memory.  The weights are float32 and keep 16 bits:
//               they enter as hi + lo, two bfloat16 numbers each, in two products, as in the kernel on mma.sync;
//   warps 2..5  softmax of tile 0, warps 6..9 of tile 1, a thread a row.  The weights go over the scores they came from (32
//               scores' 32 columns hold 16 columns of hi pairs and 16 of lo pairs).  A row's reference maximum follows the
//               true one only when that has grown by 2^8, and only then is its row of O rescaled.
// All pages a CTA reads belong to its request: positions outside the tile's reach are taken from a page inside it, the scores
// of their keys are masked and the rows of their values cleared in shared memory (0 x a page nobody has written must be 0).
//
// What bounds it: the chain of a block through its warps (scores, softmax, P V) beside the two tiles' products (the tensor
// pipe is busy 47 % of the time).  A 2,000-token prompt of 16 heads over windows of 1,024 takes 36 us, 48 with capped scores;
// the kernel on mma.sync, which issues every product from the softmax's own warps, 149 with capped scores.
//
// A launch takes as many rounds over the SMs as it has CTAs for, and a last round that is nearly empty costs as much as a full
// one.  The units (128 tokens, two heads) of such a round are therefore cut into ranges of keys, a CTA each, which leave
// unnormalised results for attention_rows_merge_kernel; so are those of a step that is small to begin with (two portions of
// 1,500 and 1,200 tokens, 176 units for 148 SMs: 91 -> 76 us, 79 since masked scores have no say in the form of the cap and the
// gate is exact, 76 since results leave by whole rows; 256 tokens behind 2,000: 49 -> 24, 22).
//
// Every wait on an mbarrier is bounded (tcgen05.cuh).
#include "tcgen05.cuh"

namespace {
using namespace tc;

constexpr int D = 128, KB = 64, TILE_M = 128, TILES = 2, NB = 4;
constexpr int SOFTMAX_WARPS = 4;
constexpr int S_WARP = 2 + SOFTMAX_WARPS * TILES;
constexpr int THREADS = 32 * (3 + SOFTMAX_WARPS * TILES);
constexpr int TMEM_COLS = 512, O_COL = NB * KB;
constexpr int Q_TILE_BYTES = TILE_M * D * 2, Q_SUB_BYTES = TILE_M * 128;
constexpr int KV_STAGE_BYTES = KB * D * 2, KV_SUB_BYTES = KB * 128;
constexpr int MAX_RANGES = 16;
// distances whose bias a CTA keeps in shared memory for each of its heads, behind as many places for keys of the tile's last
// block that lie after a row (their scores are masked, but looked up)
constexpr int NEAR_BIAS = 3904, AHEAD = TILE_M + KB;
enum Scores { PLAIN, CAPPED, BIASED };

template <int MODE>
struct Shape {
  static constexpr int STAGES = MODE == BIASED ? 4 : 5;  // the bias takes a stage's place
  static constexpr int K_OFF = TILES * Q_TILE_BYTES;
  static constexpr int V_OFF = K_OFF + STAGES * KV_STAGE_BYTES;
  static constexpr int BIAS_OFF = V_OFF + STAGES * KV_STAGE_BYTES;
  static constexpr int BAR_OFF = BIAS_OFF + (MODE == BIASED ? TILES * (AHEAD + NEAR_BIAS) * 4 : 0);
};
static_assert(O_COL + TILES * D <= TMEM_COLS, "tensor memory");

constexpr int MAX_STAGES = 5;
struct Barriers {
  uint64_t q_full;
  uint64_t kv_full[MAX_STAGES], kv_empty[MAX_STAGES];
  uint64_t s_full[NB], p_ready[NB], p_used[NB], o_full[TILES];  // of an S buffer (scores, weights there, weights used); of a tile
  uint32_t tmem_base;
  uint32_t abort;
};
template <int MODE>
constexpr int smem_bytes() { return Shape<MODE>::BAR_OFF + 1024 /* alignment slack */ + (int)sizeof(Barriers); }

struct RowsArgs {
  const int32_t *table, *positions, *item_start;
  const float *bias, *sink;
  const __nv_bfloat16* gate;
  __nv_bfloat16* out;
  long long ldg, ldo;
  float *part_o, *part_ml;  // of a unit cut into ranges: [unit - whole, range, head, row] results of D numbers / (exponent, sum)
  int table_width, items, min_tokens, hq, hkv, heads_here, page_shift, window, chunk, reach, keep_first;
  int whole, ranges;        // units before ``whole`` are a CTA's, later ones ``ranges`` CTAs'
  float scale, softcap, out_scale;
};

// The tokens of a unit: the last 128 of the last request come first.  n = 0: there is no such unit.
__device__ __forceinline__ void unit_tokens(const RowsArgs& args, int unit, int& item, int& t0, int& n, int& h0) {
  const int groups = args.hq / args.heads_here;
  h0 = unit % groups * args.heads_here;
  item = n = t0 = 0;
  int tiles = 0;
  for (int i = 0; i < args.items; ++i) {
    const int ni = args.item_start[i + 1] - args.item_start[i];
    if (ni >= args.min_tokens) tiles += (ni + TILE_M - 1) / TILE_M;
  }
  int left = tiles - 1 - unit / groups;
  for (int i = 0; i < args.items && left >= 0; ++i) {
    const int a = args.item_start[i], ni = args.item_start[i + 1] - a;
    if (ni < args.min_tokens) continue;
    const int mine = (ni + TILE_M - 1) / TILE_M;
    if (left < mine) {
      item = i;
      t0 = a + left * TILE_M;
      n = min(TILE_M, ni - left * TILE_M);
      return;
    }
    left -= mine;
  }
}

__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void halves_of(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// cap tanh(u) for |u| <= 1/4 as an odd polynomial, u = x * rate (the series up to u^9: the next term is 8e-9 of the value);
// larger scores as cap - 2 cap / (exp(2 u) + 1), which takes two more instructions of the unit that does the exponentials.
constexpr float CAP_SMALL = 0.25f;
__device__ __forceinline__ uint64_t capped_pair(uint64_t x, uint64_t rate, uint64_t slope) {
  const uint64_t u = mul_pair(x, rate), t = mul_pair(u, u);
  uint64_t p = fma_pair(t, pair_of(62.f / 2835.f, 62.f / 2835.f), pair_of(-17.f / 315.f, -17.f / 315.f));
  p = fma_pair(t, p, pair_of(2.f / 15.f, 2.f / 15.f));
  p = fma_pair(t, p, pair_of(-1.f / 3.f, -1.f / 3.f));
  const uint64_t y = mul_pair(x, slope);
  return fma_pair(mul_pair(t, p), y, y);
}
__device__ __forceinline__ float capped_far(float x, float rate2, float cap) { return fmaf(-2.f * cap, __fdividef(1.f, exp2f(x * rate2) + 1.f), cap); }

// The output gate's factor 1 / (1 + exp(-g)).  expf and a reciprocal improved by a Newton step to the last place, as good as the
// division in attention_biased.cu: the quick exponential and division lose bits, and give 0 where the sum is beyond 2^126.  (The sum
// is taken 2^-8 of, so that its reciprocal is a normal number; the division proper cost 6 us of rows of 2,700 tokens' 77.)
__device__ __forceinline__ float gate_of(float g) {
  const float x = (1.f + expf(-g)) * 0x1p-8f;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  r = fmaf(r, fmaf(-x, r, 1.f), r);
  return x > 0x1p120f ? 0.f : r * 0x1p-8f;  // (only an infinite sum is that large)
}
__device__ __forceinline__ float2 gates_of(uint32_t pair) {
  return make_float2(gate_of(__uint_as_float(pair << 16)), gate_of(__uint_as_float(pair & 0xffff0000u)));
}

// bits ``at`` and up, and bits up to ``at``, of 32; ``at`` may lie outside
__device__ __forceinline__ uint32_t bits_from(int at) { return at <= 0 ? ~0u : at > 31 ? 0u : ~0u << at; }
__device__ __forceinline__ uint32_t bits_upto(int at) { return at < 0 ? 0u : at > 30 ? ~0u : (2u << at) - 1u; }

// blocks of a CTA from which on its tiles start apart (see the softmax)
template <int MODE>
constexpr int FEWEST_APART = MODE == CAPPED ? 2 : 3;

// status codes: 1 producer, 2 MMA, 3 softmax
template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
attention_rows_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, const RowsArgs args) {
  using Sh = Shape<MODE>;
  constexpr int STAGES = Sh::STAGES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + Sh::BAR_OFF);
  volatile uint32_t* abort = &bars->abort;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;

  pdl_wait();
  pdl_trigger();  // (behind the wait: the kernel that joins the ranges reads the step's lengths and the gates before its own)
  const bool cut = (int)blockIdx.x >= args.whole;
  const int unit = cut ? args.whole + ((int)blockIdx.x - args.whole) / args.ranges : (int)blockIdx.x;
  const int range = cut ? ((int)blockIdx.x - args.whole) % args.ranges : 0;
  int item, t0, n, h0;
  unit_tokens(args, unit, item, t0, n, h0);
  if (n == 0) return;  // uniform for the CTA, before anything is allocated
  const int ntiles = args.heads_here;
  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->kv_full[s], 1);
      mbar_init(&bars->kv_empty[s], 1);
    }
    for (int j = 0; j < NB; ++j) {
      mbar_init(&bars->s_full[j], 1);
      mbar_init(&bars->p_used[j], 1);
      mbar_init(&bars->p_ready[j], SOFTMAX_WARPS);
    }
    for (int t = 0; t < TILES; ++t) mbar_init(&bars->o_full[t], 1);
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) tmem_alloc(&bars->tmem_base, TMEM_COLS);
  const int near_len = min(NEAR_BIAS, args.reach);
  if constexpr (MODE == BIASED) {
    float* near = reinterpret_cast<float*>(smem + Sh::BIAS_OFF);
    for (int i = threadIdx.x; i < ntiles * (AHEAD + near_len); i += THREADS) {
      const int t = i / (AHEAD + near_len), d = i - t * (AHEAD + near_len) - AHEAD;
      near[t * (AHEAD + NEAR_BIAS) + AHEAD + d] = d < 0 ? 0.f : args.bias[(size_t)(h0 + t) * args.reach + d] * PSB_LOG2E;
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  const int p_first = args.positions[t0], p_last = p_first + n - 1;
  const int kvl = p_last + 1 + (args.item_start[item + 1] - t0 - n);  // keys the request holds after this step
  const int kvh = h0 / (args.hq / args.hkv);
  auto low_of = [&](int p) {
    int low = args.window > 0 ? max(p - args.window + 1, 0) : 0;
    if (args.chunk > 0) low = max(low, p / args.chunk * args.chunk);
    return args.keep_first > 0 && low <= args.keep_first ? 0 : low;
  };
  const int lo_tile = low_of(p_first), low_last = low_of(p_last);
  // kept first keys: one stretch from 0 while the tile's first token still reaches them; else their blocks come first
  const int kept_blocks = (args.keep_first > 0 && lo_tile > 0) ? (args.keep_first + KB - 1) / KB : 0;
  const int main0 = lo_tile / KB;
  const int all = kept_blocks + p_last / KB - main0 + 1;
  const int per = cut ? (all + args.ranges - 1) / args.ranges : all, i0 = range * per;  // this CTA's blocks
  const int nblk = max(0, min(per, all - i0));
  auto is_kept = [&](int i) { return i0 + i < kept_blocks; };
  auto base_of = [&](int i) { return KB * (is_kept(i) ? i0 + i : main0 + i0 + i - kept_blocks); };
  const int total = ntiles * nblk;  // the tiles' blocks in the order their S is computed: (0,0) (1,0) (0,1) (1,1) ...

  if (warp == 0) {
    // ---------------------------------------------------------------------------------------------- producer
    const int page = 1 << args.page_shift, pages_per_block = KB >> args.page_shift;
    const int32_t* pages = args.table + (size_t)item * args.table_width;
    if (lane == 0) {
      mbar_expect_tx(&bars->q_full, (uint32_t)(ntiles * Q_TILE_BYTES));
      for (int t = 0; t < ntiles; ++t)
#pragma unroll
        for (int j = 0; j < D / 64; ++j)
          tma_load_2d(smem + t * Q_TILE_BYTES + j * Q_SUB_BYTES, &map_q, (h0 + t) * D + 64 * j, t0, &bars->q_full);
    }
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int i = 0; ok && i < nblk; ++i) {
      int row = 0;
      if (lane < pages_per_block) {
        const int at = (base_of(i) >> args.page_shift) + lane;
        const int first = is_kept(i) ? 0 : lo_tile >> args.page_shift;
        const int last = (is_kept(i) ? args.keep_first - 1 : kvl - 1) >> args.page_shift;
        row = (__ldg(pages + min(max(at, first), last)) * args.hkv + kvh) * page;
      }
      ok = mbar_wait(&bars->kv_empty[stage], phase ^ 1, abort, 1);  // P V of the block that used this stage has finished
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(&bars->kv_full[stage], 2u * (uint32_t)KV_STAGE_BYTES);
      __syncwarp();
      if (lane < pages_per_block) {
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          unsigned char* dst = smem + (which ? Sh::V_OFF : Sh::K_OFF) + stage * KV_STAGE_BYTES + lane * page * 128;
#pragma unroll
          for (int j = 0; j < D / 64; ++j) tma_load_2d(dst + j * KV_SUB_BYTES, &map_kv, which * D + 64 * j, row, &bars->kv_full[stage]);
        }
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1 || warp == S_WARP) {
    // --------------------------------------------------------------------------------------------------- MMA
    // S of event e takes the buffer that holds the weights of event e - NB, so its warp waits until that P V has completed.
    // A block's keys are no longer needed once P V of its last tile has been issued.
    constexpr uint32_t IDESC_S = instr_desc(TILE_M, KB, false);
    constexpr uint32_t IDESC_O = instr_desc(TILE_M, D, true);
    const uint64_t d_q = smem_desc(smem_u32(smem)), d_k = smem_desc(smem_u32(smem + Sh::K_OFF));
    const uint64_t d_v = smem_desc_mn(smem_u32(smem + Sh::V_OFF), KV_SUB_BYTES);
    const uint32_t hi_q = (uint32_t)(d_q >> 32), hi_v = (uint32_t)(d_v >> 32);
    const uint32_t q_lo = (uint32_t)d_q, k_lo = (uint32_t)d_k, v_lo = (uint32_t)d_v;
    int kv_seen = 0, v_seen = 0;
    auto tile_of = [&](int e) { return ntiles == 1 ? 0 : (e & 1); };
    auto block_of = [&](int e) { return ntiles == 1 ? e : (e >> 1); };
    auto block_ready = [&](int i) {  // waits (once) for every block up to i
      while (kv_seen <= i) {
        bool got = mbar_wait(&bars->kv_full[kv_seen % STAGES], (kv_seen / STAGES) & 1, abort, 2);
        got = __all_sync(0xffffffffu, got);
        if (!got) return false;
        ++kv_seen;
      }
      return true;
    };
    if (warp == S_WARP) {
      bool ok = mbar_wait(&bars->q_full, 0, abort, 2);
      ok = __all_sync(0xffffffffu, ok);
      for (int e = 0; ok && e < total; ++e) {
        if (e >= NB) {
          ok = mbar_wait(&bars->p_used[e % NB], ((e / NB) - 1) & 1, abort, 2);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          fence_after();
        }
        ok = block_ready(block_of(e));
        if (!ok) break;
        if (elect_one()) {
          const uint32_t a = q_lo + tile_of(e) * (Q_TILE_BYTES >> 4), bk = k_lo + (block_of(e) % STAGES) * (KV_STAGE_BYTES >> 4);
          const uint32_t dst = tmem_base + (e % NB) * KB;
#pragma unroll
          for (int j = 0; j < D / 64; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              mma_f16_split(dst, a + ((j * Q_SUB_BYTES + k * 32) >> 4), hi_q, bk + ((j * KV_SUB_BYTES + k * 32) >> 4), hi_q, IDESC_S, (j | k) != 0);
          mma_commit(&bars->s_full[e % NB]);
        }
        __syncwarp();
      }
    } else {
      auto values_ready = [&](int i) {  // every block up to i: arrived, and the rows outside the reach cleared
        while (v_seen <= i) {
          if (!block_ready(v_seen)) return false;
          const int base = base_of(v_seen);
          const int from = is_kept(v_seen) ? 0 : max(lo_tile - base, 0);
          const int upto = min((is_kept(v_seen) ? args.keep_first : kvl) - base, KB);
          if (from > 0 || upto < KB) {
            unsigned char* stage = smem + Sh::V_OFF + (v_seen % STAGES) * KV_STAGE_BYTES;
            for (int idx = lane; idx < KB * 16; idx += 32) {
              const int row = idx >> 4, rest = idx & 15;
              if (row < from || row >= upto)
                *reinterpret_cast<uint4*>(stage + (rest >> 3) * KV_SUB_BYTES + row * 128 + (rest & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            fence_async_smem();
            __syncwarp();
          }
          ++v_seen;
        }
        return true;
      };
      bool ok = true;
      for (int e = 0; ok && e < total; ++e) {
        const int t = tile_of(e), i = block_of(e);
        ok = values_ready(i);
        if (!ok) break;
        ok = mbar_wait(&bars->p_ready[e % NB], (e / NB) & 1, abort, 2);  // the weights of this block are written (over its S)
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        fence_after();
        if (elect_one()) {
          const uint32_t bv = v_lo + (i % STAGES) * (KV_STAGE_BYTES >> 4);
          const uint32_t dst = tmem_base + O_COL + t * D, src = tmem_base + (e % NB) * KB;
#pragma unroll
          for (int kk = 0; kk < KB / 16; ++kk) {  // the lo terms first
            mma_f16_tmem_a(dst, src + (kk >> 1) * 32 + 16 + (kk & 1) * 8, bv + ((kk * 2048) >> 4), hi_v, IDESC_O, (i | kk) != 0);
            mma_f16_tmem_a(dst, src + (kk >> 1) * 32 + (kk & 1) * 8, bv + ((kk * 2048) >> 4), hi_v, IDESC_O, 1);
          }
          mma_commit(&bars->o_full[t]);
          mma_commit(&bars->p_used[e % NB]);
          if (t == ntiles - 1) mma_commit(&bars->kv_empty[i % STAGES]);
        }
        __syncwarp();
      }
    }
  } else {
    // ----------------------------------------------------------------------------------------------- softmax
    const int t = (warp - 2) / SOFTMAX_WARPS;
    const int quarter = warp & 3;  // a warp may only touch tensor-memory lanes [32*(warp%4), +32)
    const int r = quarter * 32 + lane;
    if (t < ntiles) {
      const bool valid = r < n;
      const int pr = min(p_first + r, p_last);  // an absent row (its query is another request's, or zeros) is masked as the last one; nobody stores it
      const int low = low_of(pr), head = h0 + t;
      const float cap = args.softcap * PSB_LOG2E, rate = MODE == CAPPED ? args.scale / args.softcap : 0.f;
      const float factor = args.scale * PSB_LOG2E;
      const float c = MODE == PLAIN ? factor : 1.f;  // from what the scores are after their function to powers of two
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
      const uint32_t o_addr = lane_addr + O_COL + t * D;
      const float* near = reinterpret_cast<const float*>(smem + Sh::BIAS_OFF) + t * (AHEAD + NEAR_BIAS) + AHEAD;
      float m_run = -INFINITY, l_run = 0.f;
      bool ok = true;
      float sv[2][32];
      auto seq_of = [&](int i) { return ntiles == 1 ? i : 2 * i + t; };
      auto load_scores = [&](int e) {
        fence_after();
        const uint32_t s_addr = lane_addr + (e % NB) * KB;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) tmem_ld32(s_addr + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&sv[cc][0]));
      };
      auto request_scores = [&](int i) {  // false: a wait gave up
        const int e = seq_of(i);
        bool got = mbar_wait(&bars->s_full[e % NB], (e / NB) & 1, abort, 3);
        got = __all_sync(0xffffffffu, got);
        if (!got) return false;
        load_scores(e);
        return true;
      };
      auto request_scores_if_there = [&](int i) {  // asks for them only if they are computed already (the whole warp agrees)
        const int e = seq_of(i);
        if (!__all_sync(0xffffffffu, mbar_test_wait(&bars->s_full[e % NB], (e / NB) & 1))) return false;
        load_scores(e);
        return true;
      };
      if (nblk > 0) ok = request_scores(0);
      // Left to themselves both tiles make the same step of a block at the same time: the products of both, then the caps (or biases) of both, then the
      // exponentials, each on a unit of its own that is idle meanwhile.  A start half a block apart keeps them apart: 1,500 and 1,200 capped tokens 76.2 us ->
      // 72.0 (1,200 to 1,600 clocks; 800 73.9, 2,000 73.0), with a bias 71.6 -> 69.6; plain scores, whose steps are the products and the exponentials, no difference.
      // Only where there are blocks to keep apart: 8 units of 128 tokens, us without and with it by blocks 1, 2, 3, 4, 8 of a CTA, capped 13.8 16.5 18.6 20.5 28.1
      // and 13.8 16.1 17.8 19.5 26.0, in two ranges 13.0 15.2 17.6 19.6 27.1 and 13.1 15.2 16.9 18.6 25.2; with a bias 12.0 14.2 16.1 17.7 23.6 and 12.3 14.2 15.5 17.0
      // 22.8, in two ranges 13.9 15.7 17.7 19.4 25.6 and 14.4 15.9 17.3 18.7 24.5.
      if (MODE != PLAIN && t == 1) {
        const int apart = nblk >= FEWEST_APART<MODE> ? 1300 : 0;
        const long long from = clock64();
        while (clock64() - from < apart) {}
      }
      for (int i = 0; ok && i < nblk; ++i) {
        const bool kept = is_kept(i);
        const int key0 = base_of(i);
        const uint32_t s_addr = lane_addr + (seq_of(i) % NB) * KB;
        const bool need_mask = kept ? key0 + KB > args.keep_first : (key0 + KB - 1 > p_first || key0 < low_last);
        uint32_t counts[2];  // the row's keys that count, a bit each (only where need_mask)
        if (need_mask) {
          // (without kept blocks of their own the kept keys lie inside the ordinary blocks)
          const int first = kept ? 0 : low, last = kept ? args.keep_first - 1 : pr, also = kept || kept_blocks ? 0 : args.keep_first;
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const int at = key0 + cc * 32;
            counts[cc] = bits_upto(last - at) & (bits_from(first - at) | bits_upto(also - 1 - at));
          }
        }
        tmem_ld_wait();
        if constexpr (MODE == CAPPED) {
          // Only scores that count have a say in the form: those of masked keys (later ones, rows of a page that nobody has written)
          // and of rows behind the portion (another request's queries) do not, or a result would depend on them.
          float top = 0.f;
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            if (need_mask) {
#pragma unroll
              for (int k = 0; k < 32; k += 2)
                top = max3(top, counts[cc] & (1u << k) ? fabsf(sv[cc][k]) : 0.f, counts[cc] & (2u << k) ? fabsf(sv[cc][k + 1]) : 0.f);
            } else {
#pragma unroll
              for (int k = 0; k < 32; k += 2) top = max3(top, fabsf(sv[cc][k]), fabsf(sv[cc][k + 1]));
            }
          }
          if (!valid) top = 0.f;
          if (__all_sync(0xffffffffu, top * rate <= CAP_SMALL)) {
            const uint64_t rate2 = pair_of(rate, rate), slope = pair_of(factor, factor);
#pragma unroll
            for (int cc = 0; cc < 2; ++cc)
#pragma unroll
              for (int k = 0; k < 32; k += 2) halves_of(capped_pair(pair_of(sv[cc][k], sv[cc][k + 1]), rate2, slope), sv[cc][k], sv[cc][k + 1]);
          } else {
            const float twice = 2.f * PSB_LOG2E * rate;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc)
#pragma unroll
              for (int k = 0; k < 32; ++k) sv[cc][k] = capped_far(sv[cc][k], twice, cap);
          }
        } else if constexpr (MODE == BIASED) {
          const int dist = pr - key0;
          if (p_last - key0 < near_len) {  // every distance of the block has its own place in shared memory
#pragma unroll
            for (int cc = 0; cc < 2; ++cc)
#pragma unroll
              for (int k = 0; k < 32; ++k) sv[cc][k] = fmaf(sv[cc][k], factor, near[dist - cc * 32 - k]);
          } else {
            const float* far = args.bias + (size_t)head * args.reach;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc)
#pragma unroll
              for (int k = 0; k < 32; ++k) {
                const int d = min(dist - cc * 32 - k, args.reach - 1);
                const float b = d < near_len ? near[d] : __ldg(far + d) * PSB_LOG2E;
                sv[cc][k] = fmaf(sv[cc][k], factor, b);
              }
          }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float(&x)[32] = sv[cc];
          if (need_mask) {
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (!(counts[cc] & (1u << k))) x[k] = -INFINITY;
          }
#pragma unroll
          for (int k = 0; k < 32; k += 8) {
            mx0 = max3(mx0, x[k], x[k + 1]); mx1 = max3(mx1, x[k + 2], x[k + 3]);
            mx2 = max3(mx2, x[k + 4], x[k + 5]); mx3 = max3(mx3, x[k + 6], x[k + 7]);
          }
        }
        const float m_new = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
        const bool grow = (m_new - m_run) * c > 8.f;  // false while the row has seen nothing (-inf - -inf)
        // A parity wait can only tell the phase in progress from the one before it.  With two tiles the scores of block i
        // exist, so P V of block i - 2 has completed (it had their buffer), and o_full is at most one phase behind: it is
        // waited for where O has to be rescaled, and before the last block is handed over.  With one tile, whose scores run
        // further ahead, every phase is waited for once.  (The weights have a barrier a buffer: a tile may hand over two
        // blocks before the warp that issues P V has looked at the first.)
        bool waited = i == 0 || (ntiles == 2 && i + 1 < nblk);
        const bool any_grow = __any_sync(0xffffffffu, grow);
        if (i > 0 && any_grow) {
          ok = mbar_wait(&bars->o_full[t], (i - 1) & 1, abort, 3);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          waited = true;
        }
        if (any_grow) {
          const float alpha = grow ? ex2((m_run - m_new) * c) : 1.f;  // 0 from -inf
          if (grow) { m_run = m_new; l_run *= alpha; }
          if (i > 0) {
            fence_after();
#pragma unroll 1
            for (int cc = 0; cc < D / 32; ++cc) {
              uint32_t v[32];
              tmem_ld32(o_addr + cc * 32, v);
              tmem_ld_wait();
#pragma unroll
              for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * alpha);
              tmem_st32(o_addr + cc * 32, v);
            }
            tmem_st_wait();
          }
        }
        const float mc = (m_run == -INFINITY ? 0.f : m_run) * c;
        const uint64_t c_pair = pair_of(c, c), mc_pair = pair_of(-mc, -mc);
        uint64_t sum_pair = pair_of(0.f, 0.f);  // even and odd keys add up apart
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int k = 0; k < 32; k += 2) {
            float x0, x1;
            if constexpr (MODE == PLAIN) halves_of(fma_pair(pair_of(sv[cc][k], sv[cc][k + 1]), c_pair, mc_pair), x0, x1);
            else halves_of(add_pair(pair_of(sv[cc][k], sv[cc][k + 1]), mc_pair), x0, x1);
            const float p0 = ex2(x0), p1 = ex2(x1);  // masked entries are -inf: 0
            const uint64_t p = pair_of(p0, p1);
            sum_pair = add_pair(sum_pair, p);
            hi[k >> 1] = pack2(p0, p1);
            const uint64_t back = pair_of(-__uint_as_float(hi[k >> 1] << 16), -__uint_as_float(hi[k >> 1] & 0xffff0000u));
            float r0, r1;
            halves_of(add_pair(p, back), r0, r1);
            lo[k >> 1] = pack2(r0, r1);
          }
          tmem_st16(s_addr + cc * 32, hi);
          tmem_st16(s_addr + cc * 32 + 16, lo);
        }
        const bool asked = i + 1 < nblk && request_scores_if_there(i + 1);
        tmem_st_wait();
        float sum0, sum1;
        halves_of(sum_pair, sum0, sum1);
        l_run += sum0 + sum1;
        if (!waited) {
          ok = mbar_wait(&bars->o_full[t], (i - 1) & 1, abort, 3);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        fence_before();       // weights written, O rescaled
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_ready[seq_of(i) % NB]);
        if (i + 1 < nblk && !asked) {
          ok = request_scores(i + 1);
          if (!ok) break;
        }
      }
      if (ok && nblk > 0) {
        ok = mbar_wait(&bars->o_full[t], (nblk - 1) & 1, abort, 3);
        ok = __all_sync(0xffffffffu, ok);
      }
      // Results leave by whole rows: a thread has a row, and 32 rows at a time touch 32 lines an instruction.  The warp's 32 rows go through shared memory (the
      // place of the tile's queries, which nobody reads any more), 64 columns at a time: [32][16] pieces of 16 bytes, piece j of row r at j ^ (r % 16).
      // (Two portions of 1,500 and 1,200 tokens with gates 79 us -> 76, 300 tokens behind 1,500 23 -> 21.)
      float4* const staging = reinterpret_cast<float4*>(smem + t * Q_TILE_BYTES) + quarter * 32 * 16;
      auto staged = [&](int row, int piece) { return staging[row * 16 + (piece ^ (row & 15))]; };
      auto stage_results = [&](int pass, float factor) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t v[32];
          tmem_ld32(o_addr + pass * 64 + cc * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            staging[lane * 16 + ((8 * cc + k) ^ (lane & 15))] = make_float4(__uint_as_float(v[4 * k]) * factor, __uint_as_float(v[4 * k + 1]) * factor,
                                                                            __uint_as_float(v[4 * k + 2]) * factor, __uint_as_float(v[4 * k + 3]) * factor);
        }
        __syncwarp();
      };
      if (ok && cut) {
        fence_after();
        const size_t slot = (((size_t)(unit - args.whole) * args.ranges + range) * ntiles + t) * TILE_M + r;
        const bool some = nblk > 0 && m_run != -INFINITY;
        *reinterpret_cast<float2*>(args.part_ml + slot * 2) = make_float2(some ? m_run * c : -INFINITY, some ? l_run : 0.f);
        if (nblk > 0) {
          float* dst = args.part_o + (slot - lane) * D;  // of the warp's first row
#pragma unroll 1
          for (int pass = 0; pass < D / 64; ++pass) {
            stage_results(pass, 1.f);
#pragma unroll 4
            for (int at = lane; at < 32 * 16; at += 32)
              *reinterpret_cast<float4*>(dst + (size_t)(at >> 4) * D + 64 * pass + 4 * (at & 15)) = staged(at >> 4, at & 15);
            __syncwarp();
          }
        }
        fence_before();
      } else if (ok) {
        fence_after();
        // a sink joins the denominator here, where the row's sum is complete
        const float inv = (l_run > 0.f ? (args.sink ? sink_quotient2(m_run * c, l_run, args.sink[head] * PSB_LOG2E) : 1.f / l_run) : 0.f) * args.out_scale;
        const int row0 = t0 + quarter * 32, column = head * D + 8 * (lane & 7);
#pragma unroll 1
        for (int pass = 0; pass < D / 64; ++pass) {
          uint4 g[8];  // the gates this lane needs: rows lane / 8 + 4 i
          if (args.gate) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int row = 4 * i + (lane >> 3);
              if (quarter * 32 + row < n) g[i] = *reinterpret_cast<const uint4*>(args.gate + (size_t)(row0 + row) * args.ldg + column + 64 * pass);
            }
          }
          stage_results(pass, inv);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row = 4 * i + (lane >> 3);
            const float4 a = staged(row, 2 * (lane & 7)), b = staged(row, 2 * (lane & 7) + 1);
            float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            if (quarter * 32 + row >= n) continue;
            if (args.gate) {
              const uint32_t gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                const float2 f = gates_of(gw[w]);
                v[2 * w] *= f.x;
                v[2 * w + 1] *= f.y;
              }
            }
            *reinterpret_cast<uint4*>(args.out + (size_t)(row0 + row) * args.ldo + column + 64 * pass) = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
          }
          __syncwarp();
        }
        fence_before();
      }
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

// A warp per row of the units that were cut: out = sum_s w_s O_s / sum_s w_s l_s with w_s = 2^(e_s - max e), the sink one
// more range with a sum of one and no result; then the factor and the gate.
__global__ void __launch_bounds__(128)
attention_rows_merge_kernel(const RowsArgs args) {
  pdl_trigger();
  const int at = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int in_unit = at % (args.heads_here * TILE_M), t = in_unit / TILE_M, r = in_unit % TILE_M;
  const int rest = at / (args.heads_here * TILE_M);
  int item, t0, n, h0;
  unit_tokens(args, args.whole + rest, item, t0, n, h0);
  const int head = h0 + t;
  uint2 g = make_uint2(0, 0);
  if (args.gate && r < n) g = *reinterpret_cast<const uint2*>(args.gate + (size_t)(t0 + r) * args.ldg + (size_t)head * D + 4 * lane);
  pdl_wait();
  if (r >= n) return;
  const size_t step = (size_t)args.heads_here * TILE_M;  // from range to range
  const size_t slot0 = (size_t)rest * args.ranges * step + (size_t)t * TILE_M + r;
  // four ranges' results at a time, asked for before their weights are known (28 units in five ranges 10 us, one behind the other; 300 tokens behind 1,500, the
  // whole call, 21.1 -> 19.6)
  constexpr int AHEAD = 4;
  float4 v[AHEAD];
  auto ask = [&](int s0) {
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)
      if (s0 + k < args.ranges) v[k] = *reinterpret_cast<const float4*>(args.part_o + (slot0 + (s0 + k) * step) * D + 4 * lane);
  };
  ask(0);
  const float2 ml = lane < args.ranges ? *reinterpret_cast<const float2*>(args.part_ml + (slot0 + lane * step) * 2) : make_float2(-INFINITY, 0.f);
  const float s2 = args.sink ? args.sink[head] * PSB_LOG2E : -INFINITY;
  const float top = fmaxf(warp_max(ml.x), s2);
  const float w = ml.y > 0.f ? exp2f(ml.x - top) : 0.f;
  const float sum = warp_sum(w * ml.y) + (args.sink ? exp2f(s2 - top) : 0.f);
  const float inv = (sum > 0.f ? 1.f / sum : 0.f) * args.out_scale;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int s0 = 0; s0 < args.ranges; s0 += AHEAD) {
    if (s0) ask(s0);
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      if (s0 + k >= args.ranges) break;
      const float ws = __shfl_sync(0xffffffffu, w, s0 + k);
      if (ws == 0.f) continue;  // a range that saw nothing has left nothing
      acc[0] = fmaf(ws, v[k].x, acc[0]); acc[1] = fmaf(ws, v[k].y, acc[1]);
      acc[2] = fmaf(ws, v[k].z, acc[2]); acc[3] = fmaf(ws, v[k].w, acc[3]);
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] *= inv;
  if (args.gate) {
    const uint32_t gw[2] = {g.x, g.y};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 f = gates_of(gw[e]);
      acc[2 * e] *= f.x;
      acc[2 * e + 1] *= f.y;
    }
  }
  *reinterpret_cast<uint2*>(args.out + (size_t)(t0 + r) * args.ldo + (size_t)head * D + 4 * lane) = make_uint2(pack2(acc[0], acc[1]), pack2(acc[2], acc[3]));
}

template <int MODE>
int launch(const CUtensorMap& map_q, const CUtensorMap& map_kv, const RowsArgs& args, dim3 grid, cudaStream_t stream) {
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(attention_rows_tcgen05_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<MODE>()) != cudaSuccess)
      PSB_REFUSE("attention_rows_tcgen05: cannot reserve %d bytes of shared memory", smem_bytes<MODE>());
    configured.set();
  }
  psb_launch(attention_rows_tcgen05_kernel<MODE>, grid, dim3(THREADS), (size_t)smem_bytes<MODE>(), stream, map_q, map_kv, args);
  PSB_LAUNCH_CHECK("attention_rows_tcgen05");
  return 0;
}

}  // namespace

// (hq, hkv, dim, vdim, page_size, capped, biased) -> 1 if the kernel takes them
PSB_API int psb_attention_rows_tcgen05_supported(int hq, int hkv, int dim, int vdim, int page_size, int capped, int biased) {
  if (hq < 1 || hkv < 1 || hq % hkv || dim != D || vdim != D || (capped && biased)) return 0;
  return page_size >= 8 && page_size <= KB && (page_size & (page_size - 1)) == 0 ? 1 : 0;
}

// (hq, hkv) -> query heads a unit takes
PSB_API int psb_attention_rows_tcgen05_heads(int hq, int hkv) { return hkv > 0 && (hq / hkv) % 2 == 0 ? 2 : 1; }

// Every portion of at least ``min_tokens`` tokens; other tokens are left untouched.  ``tiles``: at least the number of runs of
// 128 tokens these portions make up.  A unit is such a run for psb_attention_rows_tcgen05_heads() heads; the first ``whole`` of
// them, or all (whole < 0), are a CTA's each and the others ``ranges`` CTAs', with part_o float32 [units - whole, ranges, heads * 128, 128]
// and part_ml [.., heads * 128, 2] as their scratch.
// (q, kv, num_pages, table, table_width, positions, item_start, items, T, min_tokens, tiles, bias, sink, out, hq, hkv, dim, vdim,
//  page_size, window, chunk, reach, scale, keep_first, gate, ldg, ldo, out_scale, softcap, whole, ranges, part_o, part_ml, stream)
PSB_API int psb_attention_rows_tcgen05(const void* q, const void* kv, long long num_pages, const void* table, int table_width,
                                       const void* positions, const void* item_start, int items, int T, int min_tokens, int tiles,
                                       const void* bias, const void* sink, void* out, int hq, int hkv, int dim, int vdim, int page_size,
                                       int window, int chunk, int reach, float scale, int keep_first, const void* gate, long long ldg,
                                       long long ldo, float out_scale, float softcap, int whole, int ranges, void* part_o,
                                       void* part_ml, cudaStream_t stream) {
  // (the largest raw score stands for the largest scaled one, and the cap's vote is on their size)
  if (!(scale > 0.f)) PSB_REFUSE("attention_rows_tcgen05: scores are multiplied by a positive scale, not %g", scale);
  if (softcap < 0.f || !psb_attention_rows_tcgen05_supported(hq, hkv, dim, vdim, page_size, softcap > 0.f, bias != nullptr))
    PSB_REFUSE("attention_rows_tcgen05: %d heads over %d of %d and %d in pages of %d are not taken", hq, hkv, dim, vdim, page_size);
  if (ldo < (long long)hq * D || ldo % 8 || (gate && (ldg < (long long)hq * D || ldg % 8))) PSB_REFUSE("attention_rows_tcgen05: bad output or gate rows");
  if (keep_first < 0 || (keep_first > 0 && (window < 1 || chunk > 0))) PSB_REFUSE("attention_rows_tcgen05: kept first keys go with a window and no chunk mask");
  if (table_width < 1 || window < 0 || chunk < 0 || (bias && reach < 1) || num_pages < 1) PSB_REFUSE("attention_rows_tcgen05: bad arguments");
  if (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)out | (uintptr_t)gate) & 15) PSB_REFUSE("attention_rows_tcgen05: operands must be 16-byte aligned");
  if (items < 1 || T < 1 || min_tokens < 1 || tiles < 1) return 0;
  const int heads_here = psb_attention_rows_tcgen05_heads(hq, hkv);
  const long long units = (long long)tiles * (hq / heads_here);
  if (whole < 0 || whole > units) whole = (int)units;
  if (whole < units && (ranges < 1 || ranges > MAX_RANGES || !part_o || !part_ml || (((uintptr_t)part_o | (uintptr_t)part_ml) & 15)))
    PSB_REFUSE("attention_rows_tcgen05: 1 to %d ranges with their scratch, not %d", MAX_RANGES, ranges);
  const long long kv_rows = num_pages * hkv * page_size;
  if (units > 0xffffff || kv_rows > 0x7fffffffLL) PSB_REFUSE("attention_rows_tcgen05: %d runs of tokens or %lld cache rows are too many for one launch", tiles, kv_rows);
  RowsArgs args{};
  args.table = (const int32_t*)table; args.positions = (const int32_t*)positions; args.item_start = (const int32_t*)item_start;
  args.bias = (const float*)bias; args.sink = (const float*)sink; args.gate = (const __nv_bfloat16*)gate; args.out = (__nv_bfloat16*)out;
  args.ldg = ldg; args.ldo = ldo; args.table_width = table_width; args.items = items; args.min_tokens = min_tokens; args.hq = hq;
  args.hkv = hkv; args.heads_here = heads_here; args.window = window; args.chunk = chunk; args.reach = bias ? reach : 0;
  args.keep_first = keep_first; args.scale = scale; args.softcap = softcap; args.out_scale = out_scale;
  while ((1 << args.page_shift) < page_size) ++args.page_shift;
  CUtensorMap map_q, map_kv;
  int r = make_map_bf16(&map_q, q, (uint64_t)T, (uint64_t)hq * D, (uint64_t)hq * D, TILE_M);
  if (r == 0) r = make_map_bf16(&map_kv, kv, (uint64_t)kv_rows, (uint64_t)2 * D, (uint64_t)2 * D, page_size);
  if (r != 0) PSB_REFUSE("attention_rows_tcgen05: no tensor map (%d)", r);
  args.whole = whole; args.ranges = whole < units ? ranges : 1; args.part_o = (float*)part_o; args.part_ml = (float*)part_ml;
  const unsigned rest = (unsigned)(units - whole);
  const dim3 grid((unsigned)whole + rest * args.ranges);
  const int status = softcap > 0.f ? launch<CAPPED>(map_q, map_kv, args, grid, stream)
                     : bias        ? launch<BIASED>(map_q, map_kv, args, grid, stream)
                                   : launch<PLAIN>(map_q, map_kv, args, grid, stream);
  if (status || !rest) return status;
  psb_launch(attention_rows_merge_kernel, dim3(rest * heads_here * TILE_M / 4), dim3(128), 0, stream, args);
  PSB_LAUNCH_CHECK("attention_rows_merge");
  return 0;
}

// 0 while no bounded wait of this kernel has ever run out on the current device; reading it synchronises with the device.
PSB_API int psb_attention_rows_tcgen05_status() { return tc::read_status(); }
