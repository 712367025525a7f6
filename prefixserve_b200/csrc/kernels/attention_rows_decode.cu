// Attention of steps of single tokens over cache rows that hold a key and then its value, heads of 128 in bfloat16, fed by the TMA
// unit: what attention_rows_single_kernel (attention_biased.cu) computes, where up to eight query heads read a key/value head.
//
// A block takes an equal share of all tokens' runs of 16 keys, piece by piece (a piece is of one token and key/value head), or, where
// tokens see few keys, a token and a key/value head.  One producer warp asks for the runs, aligned to absolute
// positions (four boxes of 64 columns with 128-byte swizzle, keys then values) into a ring of eight stages, four consumer warps take
// the runs in turn: ldmatrix out of the swizzled rows, S = Q K^T (mma.sync m16n8k16: heads in rows, keys in columns), scale, cap,
// bias, masks and the online softmax in float32.  The weights are float32 and keep 16 bits: hi + lo, two bfloat16 numbers.  With at
// most eight heads half of an instruction's rows would be empty, so rows 0..7 carry the hi terms and rows 8..15 the lo terms of the
// same heads, and one instruction does both; the two halves of the result are added up at the end.  O is rescaled only when a row's
// maximum has grown.  Pieces that are not all of a (token, key/value head) are joined by attention_rows_decode_merge_kernel.
//
// What bounds it: the cached rows (512 bytes a key and head).  32 tokens that read 255 MB of rows together: 52 us by itself and the merge
// 3, 54 one call behind the other, 4.9 TB/s (56, 6 and 61 with the same number of blocks for every token and key/value head; the kernel it
// stands in for 119 us: it copied every row with a lane's own cp.async and spent two products on the weights).
// Calls that read few rows stay with that one (ROWS_DECODE_LEAST in ops/kernels.py).
//
// Every wait on an mbarrier is bounded (tcgen05.cuh).
#include <cfloat>

#include "tcgen05.cuh"

namespace {
using namespace tc;

constexpr int D = 128, CONSUMERS = 4, THREADS = 32 * (CONSUMERS + 1), RUN = 16, STAGES = 8, HEADS = 8, BLOCKS = 3;
constexpr int BOX_BYTES = RUN * 128, STAGE_BYTES = 4 * BOX_BYTES;  // two boxes of keys, two of values
// Every stage belongs to one consumer warp: a warp that got ahead of the others would take the phase before a stage's for its own.
static_assert(STAGES % CONSUMERS == 0, "every stage belongs to one consumer warp");
constexpr int JOIN_PITCH = D + 4, JOINED = CONSUMERS / 2, JOIN_BYTES = JOINED * HEADS * (JOIN_PITCH + 2) * 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + JOIN_BYTES + 1024 + 2 * STAGES * 8 + 16;
static_assert(BLOCKS * (SMEM_BYTES + 1024) <= 228 * 1024, "blocks of an SM");
constexpr int PART = D + 2;  // what a share leaves of a head: maximum in powers of two, sum, result

struct DecodeArgs {
  const __nv_bfloat16 *q, *gate;
  const int32_t *table, *positions, *token_item;
  const float *bias, *sink;
  __nv_bfloat16* out;
  int4* found;      // per (token, key/value head): first and last block that has a share of it, and where the first one's lies
  float* partial;   // two a block: [2 blocks, heads of a key/value head, PART]
  long long ldg, ldo;
  int tokens, table_width, hq, hkv, page_shift, window, chunk, reach, keep_first, least_runs;
  float scale, softcap, out_scale;
};

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// the 16-byte piece ``piece`` (8 columns) of row ``row`` of two swizzled boxes
__device__ __forceinline__ uint32_t piece_at(uint32_t base, int row, int piece) {
  return base + (uint32_t)((piece >> 3) * BOX_BYTES + row * 128 + (((piece & 7) ^ (row & 7)) << 4));
}
// cap tanh(x / cap) with x = s scale (see attention_biased.cu); ``rate`` = 2 log2(e) scale / cap
__device__ __forceinline__ float quick_cap(float s, float rate, float cap) { return fmaf(-2.f * cap, __fdividef(1.f, exp2f(s * rate) + 1.f), cap); }

// A token's runs of keys: kept first keys in runs of their own in front, if the window does not reach them, then the window's.
struct TokenRuns {
  int p, lo, kept, first, count;
  __device__ __forceinline__ TokenRuns(const DecodeArgs& args, int position) : p(position) {
    lo = (args.window > 0 && p - args.window + 1 > 0) ? p - args.window + 1 : 0;
    if (args.chunk > 0) lo = max(lo, p / args.chunk * args.chunk);
    kept = 0;
    if (args.keep_first > 0) {
      if (lo <= args.keep_first) lo = 0;
      else kept = (args.keep_first + RUN - 1) / RUN;
    }
    first = lo / RUN;
    count = max(1, kept + p / RUN - first + 1);
  }
  __device__ __forceinline__ int base(int run) const { return RUN * (run < kept ? run : first + run - kept); }
};

// The walk of a block over its share of all tokens' runs, laid end to end (a token's, once for every key/value head): pieces of one
// (token, key/value head) each.  Every warp makes it by itself.  The ring goes on from piece to piece; with a block for every
// (token, key/value head, share) instead, 32 tokens of 8 key/value heads took three rounds of blocks that each filled their rings anew.
struct Walk {
  int t = 0, at = 0, end = 0;        // the token, where its runs start, and where the block's share ends
  int begin = 0, pos = 0, total = 0, blocks = 0;
  int g = 0, r0 = 0, runs = 0;       // the piece
  int p = 0, next_p = 0, item = 0, next_item = 0;

  __device__ __forceinline__ void ask(const DecodeArgs& args) {
    const int next = min(t + 1, args.tokens - 1);
    next_p = args.positions[next];
    next_item = args.token_item[next];
  }
  // false: nothing to do
  __device__ __forceinline__ bool start(const DecodeArgs& args, int lane) {
    if (args.least_runs == 0) {  // a (token, key/value head) a block
      t = blockIdx.x / args.hkv;
      p = args.positions[t];
      item = args.token_item[t];
      const TokenRuns runs_of(args, p);
      begin = pos = (blockIdx.x - t * args.hkv) * runs_of.count;
      end = pos + runs_of.count;
      return true;
    }
    int mine = 0;
    for (int i = lane; i < args.tokens; i += 32) mine += TokenRuns(args, args.positions[i]).count;
    total = __reduce_add_sync(0xffffffffu, mine) * args.hkv;
    blocks = min((int)gridDim.x, max(1, total / args.least_runs));
    if ((int)blockIdx.x >= blocks) return false;
    begin = pos = (int)((long long)blockIdx.x * total / blocks);
    end = (int)((long long)(blockIdx.x + 1) * total / blocks);
    for (int i0 = 0; i0 < args.tokens; i0 += 32) {
      const int position = i0 + lane < args.tokens ? args.positions[i0 + lane] : 0;
      const int n = i0 + lane < args.tokens ? TokenRuns(args, position).count * args.hkv : 0;
      int upto = n;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, off);
        if (lane >= off) upto += x;
      }
      const unsigned beyond = __ballot_sync(0xffffffffu, pos < at + upto);
      if (beyond) {
        const int who = __ffs(beyond) - 1;
        t = i0 + who;
        at += __shfl_sync(0xffffffffu, upto - n, who);
        p = __shfl_sync(0xffffffffu, position, who);
        break;
      }
      at += __shfl_sync(0xffffffffu, upto, 31);
    }
    item = args.token_item[t];
    ask(args);
    return true;
  }
  __device__ __forceinline__ bool more() const { return pos < end; }
  __device__ __forceinline__ TokenRuns piece(const DecodeArgs& args) {
    TokenRuns all(args, p);
    if (pos >= at + all.count * args.hkv) {
      at += all.count * args.hkv;
      ++t;
      p = next_p;
      item = next_item;
      ask(args);
      all = TokenRuns(args, p);
    }
    g = (pos - at) / all.count;
    r0 = pos - at - g * all.count;
    runs = min(all.count - r0, end - pos);
    pos += runs;
    return all;
  }
  // the block that has run x of all
  __device__ __forceinline__ int block_of(int x) const { return (int)(((long long)(x + 1) * blocks - 1) / total); }
};

// four columns of a head's result: divided by the sum, gated
__device__ __forceinline__ void finish(const DecodeArgs& args, int t, int h, int d, const float (&acc)[4], float sum) {
  const float by = args.out_scale / sum;
  const __nv_bfloat16* gate = args.gate ? args.gate + (size_t)t * args.ldg + (size_t)h * D + d : nullptr;
  __nv_bfloat16* dst = args.out + (size_t)t * args.ldo + (size_t)h * D + d;
#pragma unroll
  for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16_rn(acc[e] * (gate ? by / (1.f + expf(-__bfloat162float(gate[e]))) : by));
}
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// status codes: 1 producer, 2 consumer
__global__ void __launch_bounds__(THREADS, BLOCKS)
attention_rows_decode_kernel(const __grid_constant__ CUtensorMap map_kv, const DecodeArgs args) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* join = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES);  // results of a piece, [two warps' each][head][D + 4 | m | l]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + JOIN_BYTES);
  uint64_t* empty = full + STAGES;
  volatile uint32_t* abort = reinterpret_cast<volatile uint32_t*>(empty + STAGES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  const int share = args.hq / args.hkv;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (args.least_runs == 0) pdl_trigger();  // (else the joining kernel's blocks, and what comes behind it, would take places of these: 77 us instead of 54)
  pdl_wait();
  Walk walk;
  if (!walk.start(args, lane)) return;

  int done = 0;  // runs of the pieces before
  if (warp == CONSUMERS) {
    bool ok = true;
    while (ok && walk.more()) {
      const TokenRuns all = walk.piece(args);
      const int32_t* pages = args.table + (size_t)walk.item * args.table_width;
      int ids = 0;
      for (int k = 0; k < walk.runs; ++k) {
        if ((k & 31) == 0) {  // page ids of the next 32 runs, one a lane
          const int ahead = k + lane;
          ids = ahead < walk.runs ? __ldg(pages + (all.base(walk.r0 + ahead) >> args.page_shift)) : 0;
        }
        const int page = __shfl_sync(0xffffffffu, ids, k & 31), i = done + k, stage = i % STAGES;
        if (i >= STAGES) {
          ok = mbar_wait(&empty[stage], ((i / STAGES) - 1) & 1, abort, 1);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        if (lane == 0) {
          const int row = ((page * args.hkv + walk.g) << args.page_shift) + (all.base(walk.r0 + k) & ((1 << args.page_shift) - 1));
          mbar_expect_tx(&full[stage], (uint32_t)STAGE_BYTES);
#pragma unroll
          for (int b = 0; b < 4; ++b) tma_load_2d(smem + stage * STAGE_BYTES + b * BOX_BYTES, &map_kv, 64 * b, row, &full[stage]);
        }
        __syncwarp();
      }
      done += walk.runs;
    }
  }
  bool ok = true;  // a consumer that has given up goes on to the pieces' barriers
  while (warp < CONSUMERS && walk.more()) {
    const TokenRuns all = walk.piece(args);
    const int t = walk.t, p = all.p, h0 = walk.g * share;
    float m = -FLT_MAX, l = 0.f;   // of head gr, in powers of two
    float o[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    uint32_t qa[D / 16][2];  // rows 0..7: the heads' queries
    const uint32_t* qrow = gr < share ? reinterpret_cast<const uint32_t*>(args.q + ((size_t)t * args.hq + h0 + gr) * D) : nullptr;
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
      qa[k][0] = qrow ? qrow[8 * k + tg] : 0u;
      qa[k][1] = qrow ? qrow[8 * k + 4 + tg] : 0u;
    }
    const float factor = args.scale * PSB_LOG2E, cap = args.softcap * PSB_LOG2E;
    const float rate = args.softcap > 0.f ? 2.f * PSB_LOG2E * args.scale / args.softcap : 0.f;
    const float* bias = args.bias && gr < share ? args.bias + (size_t)(h0 + gr) * args.reach : nullptr;
    const int lm = lane >> 3, lr = lane & 7;
    for (int k = (warp - done) & (CONSUMERS - 1); ok && k < walk.runs; k += CONSUMERS) {  // run i of the block is warp i % CONSUMERS's
      const int run = walk.r0 + k, i = done + k, stage = i % STAGES, key0 = all.base(run);
      const bool kept = run < all.kept;
      const int from = kept ? 0 : all.lo - key0, upto = (kept ? args.keep_first : p + 1) - key0;  // rows that count
      ok = mbar_wait(&full[stage], (i / STAGES) & 1, abort, 2);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const uint32_t kbase = smem_u32(smem) + stage * STAGE_BYTES, vbase = kbase + 2 * BOX_BYTES;
      if (from > 0 || upto < RUN) {  // 0 x (what an earlier owner of the page left) must be 0
        for (int idx = lane; idx < RUN * (D / 8); idx += 32) {
          const int row = idx / (D / 8);
          if (row < from || row >= upto) asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(piece_at(vbase, row, idx % (D / 8))), "r"(0u) : "memory");
        }
        fence_async_smem();  // these writes come before the TMA unit's next use of the stage
        __syncwarp();
      }
      float s[2][4] = {};
#pragma unroll
      for (int k = 0; k < D / 16; k += 2) {
        uint32_t b0[4], b1[4];
        ldmatrix4(b0, piece_at(kbase, lr, 2 * k + lm));
        ldmatrix4(b1, piece_at(kbase, 8 + lr, 2 * k + lm));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t a[4] = {qa[k + e][0], 0u, qa[k + e][1], 0u};
          mma_16816(s[0], a, b0[2 * e], b0[2 * e + 1]);
          mma_16816(s[1], a, b1[2 * e], b1[2 * e + 1]);
        }
      }
      float x[4], top = -FLT_MAX;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = 8 * (e >> 1) + 2 * tg + (e & 1);
        float v = s[e >> 1][e & 1];
        v = args.softcap > 0.f ? quick_cap(v, rate, cap) : v * factor;
        if (bias) {  // (the lowest finite bias stays finite in powers of two: keys that all have it weigh the same)
          const float b = bias[max(0, min(p - key0 - row, args.reach - 1))];
          v += b == -INFINITY ? b : fmaxf(b * PSB_LOG2E, -FLT_MAX);
        }
        if (row < from || row >= upto) v = -INFINITY;
        x[e] = v;
        top = fmaxf(top, v);
      }
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      if (__any_sync(0xffffffffu, top > m)) {
        const float m_new = fmaxf(m, top), alpha = exp2f(m - m_new);
        m = m_new;
        l *= alpha;
#pragma unroll
        for (int j = 0; j < D / 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[j][e] *= alpha;
      }
      uint32_t a[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float w0 = exp2f(x[2 * e] - m), w1 = exp2f(x[2 * e + 1] - m);  // a masked score is -inf: weight 0
        l += w0 + w1;
        const uint32_t hi = pack2(w0, w1);
        a[2 * e] = hi;                                                                                     // row gr
        a[2 * e + 1] = pack2(w0 - __uint_as_float(hi << 16), w1 - __uint_as_float(hi & 0xffff0000u));  // row gr + 8
      }
#pragma unroll
      for (int c = 0; c < D / 8; c += 2) {
        uint32_t b[4];
        ldmatrix4_trans(b, piece_at(vbase, (lm & 1) * 8 + lr, c + (lm >> 1)));
        mma_16816(o[c], a, b[0], b[1]);
        mma_16816(o[c + 1], a, b[2], b[3]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
    }
    done += walk.runs;
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    constexpr int ROW = JOIN_PITCH + 2;
    float* mine = join + ((warp % JOINED) * HEADS + gr) * ROW;  // warps 0 and 2 meet here, 1 and 3 there
    auto leave = [&](float mx, float sum, auto value) {
#pragma unroll
      for (int j = 0; j < D / 8; ++j) *reinterpret_cast<float2*>(mine + 8 * j + 2 * tg) = value(j);
      if (tg == 0) *reinterpret_cast<float2*>(mine + JOIN_PITCH) = make_float2(mx, sum);
    };
    if (warp >= JOINED) leave(m, l, [&](int j) { return make_float2(o[j][0] + o[j][2], o[j][1] + o[j][3]); });
    named_barrier(1, 32 * CONSUMERS);
    if (warp < JOINED) {
      const float2 theirs = *reinterpret_cast<const float2*>(mine + JOIN_PITCH);
      const float both = fmaxf(m, theirs.x), f0 = exp2f(m - both), f1 = exp2f(theirs.x - both);  // (a warp without runs has a sum and a result of 0)
      __syncwarp();  // everybody has read the maximum and the sum
      leave(both, fmaf(f0, l, f1 * theirs.y), [&](int j) {
        const float2 x = *reinterpret_cast<const float2*>(mine + 8 * j + 2 * tg);
        return make_float2(fmaf(f0, o[j][0] + o[j][2], f1 * x.x), fmaf(f0, o[j][1] + o[j][3], f1 * x.y));
      });
    }
    named_barrier(1, 32 * CONSUMERS);
    const bool whole = walk.runs == all.count;
    const int slot = 2 * blockIdx.x + (walk.pos - walk.runs == walk.begin ? 0 : 1);
    if (args.least_runs > 0 && walk.r0 == 0 && threadIdx.x == 0)
      args.found[(size_t)t * args.hkv + walk.g] =
          make_int4(blockIdx.x, whole ? -1 : walk.block_of(walk.pos - walk.runs + all.count - 1), slot, 0);
    for (int idx = threadIdx.x; idx < share * (D / 4); idx += 32 * CONSUMERS) {
      const int row = idx / (D / 4), d = (idx % (D / 4)) * 4, h = h0 + row;
      const float* src = join + row * ROW;
      const float s2 = whole && args.sink ? args.sink[h] * PSB_LOG2E : -INFINITY;
      float top = s2;
#pragma unroll
      for (int w = 0; w < JOINED; ++w) top = fmaxf(top, src[w * HEADS * ROW + JOIN_PITCH]);
      float sum = whole && args.sink ? exp2f(s2 - top) : 0.f, acc[4] = {};
#pragma unroll
      for (int w = 0; w < JOINED; ++w) {
        const float* mine = src + w * HEADS * ROW;
        const float f = exp2f(mine[JOIN_PITCH] - top);
        sum = fmaf(f, mine[JOIN_PITCH + 1], sum);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] = fmaf(f, mine[d + e], acc[e]);
      }
      if (whole) finish(args, t, h, d, acc, sum);
      else {
        float* dst = args.partial + ((size_t)slot * share + row) * PART;
        if (d == 0) *reinterpret_cast<float2*>(dst) = make_float2(top, sum);
        *reinterpret_cast<float2*>(dst + 2 + d) = make_float2(acc[0], acc[1]);
        *reinterpret_cast<float2*>(dst + 4 + d) = make_float2(acc[2], acc[3]);
      }
    }
    named_barrier(1, 32 * CONSUMERS);  // the next piece's results may come
  }
  if (*abort) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight must land before the memory changes hands
  }
}

// The shares that several blocks left of a (token, key/value head), a warp a head of it.
__global__ void __launch_bounds__(32 * HEADS)
attention_rows_decode_merge_kernel(const DecodeArgs args) {
  pdl_trigger();
  pdl_wait();
  const int4 found = args.found[blockIdx.x];
  const int n = found.y - found.x + 1;
  if (n < 2) return;  // one block had it all
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, share = args.hq / args.hkv;
  const int t = blockIdx.x / args.hkv, h = (blockIdx.x - t * args.hkv) * share + warp;
  auto part = [&](int j) { return args.partial + ((size_t)(j == 0 ? found.z : 2 * (found.x + j)) * share + warp) * PART; };
  constexpr int AHEAD = 4;
  float2 ml[AHEAD], a[AHEAD], b[AHEAD];
  float top = args.sink ? args.sink[h] * PSB_LOG2E : -INFINITY;
  float sum = args.sink ? 1.f : 0.f, acc[4] = {};
  for (int j0 = 0; j0 < n; j0 += AHEAD) {
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      ml[j] = make_float2(-INFINITY, 0.f);
      a[j] = b[j] = make_float2(0.f, 0.f);
      if (j0 + j >= n) continue;
      const float* from = part(j0 + j);
      ml[j] = *reinterpret_cast<const float2*>(from);
      a[j] = *reinterpret_cast<const float2*>(from + 2 + 4 * lane);
      b[j] = *reinterpret_cast<const float2*>(from + 4 + 4 * lane);
    }
    float now = top;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) now = fmaxf(now, ml[j].x);
    const float down = exp2f(top - now);  // (a share's maximum is finite)
    top = now;
    sum *= down;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] *= down;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      const float f = exp2f(ml[j].x - top);
      sum = fmaf(f, ml[j].y, sum);
      acc[0] = fmaf(f, a[j].x, acc[0]); acc[1] = fmaf(f, a[j].y, acc[1]);
      acc[2] = fmaf(f, b[j].x, acc[2]); acc[3] = fmaf(f, b[j].y, acc[3]);
    }
  }
  finish(args, t, h, 4 * lane, acc, sum);
}

void set_scratch(DecodeArgs& args, void* scratch) {
  args.found = (int4*)scratch;
  args.partial = (float*)scratch + (size_t)4 * args.tokens * args.hkv;
}

}  // namespace

// (hq, hkv, dim, vdim, page_size) -> 1 if the kernel takes them
PSB_API int psb_attention_rows_decode_supported(int hq, int hkv, int dim, int vdim, int page_size) {
  return hq >= 1 && hkv >= 1 && hq % hkv == 0 && hq / hkv <= HEADS && dim == D && vdim == D && page_size >= RUN && (page_size & (page_size - 1)) == 0 ? 1 : 0;
}

// () -> blocks an SM holds
PSB_API int psb_attention_rows_decode_blocks() { return BLOCKS; }

// Tokens one by one.  ``blocks`` 0: a block per (token, key/value head).  Else up to so many blocks share out all of their runs of 16
// keys, at least ``least_runs`` each, and what is left in ``scratch`` (float32 [4 T hkv + 2 blocks hq/hkv 130]) the caller has joined
// (psb_attention_rows_decode_merge).
// (q, kv, num_pages, table, table_width, positions, token_item, bias, sink, out, T, hq, hkv, dim, vdim, page_size, window, chunk, reach,
//  scale, keep_first, scratch, blocks, least_runs, gate, ldg, ldo, out_scale, softcap, stream)
PSB_API int psb_attention_rows_decode(const void* q, const void* kv, long long num_pages, const void* table, int table_width,
                                      const void* positions, const void* token_item, const void* bias, const void* sink, void* out, int T,
                                      int hq, int hkv, int dim, int vdim, int page_size, int window, int chunk, int reach, float scale,
                                      int keep_first, void* scratch, int blocks, int least_runs, const void* gate, long long ldg,
                                      long long ldo, float out_scale, float softcap, cudaStream_t stream) {
  if (!psb_attention_rows_decode_supported(hq, hkv, dim, vdim, page_size))
    PSB_REFUSE("attention_rows_decode: %d heads over %d of %d and %d in pages of %d are not taken", hq, hkv, dim, vdim, page_size);
  if (ldo < (long long)hq * D || (gate && ldg < (long long)hq * D) || softcap < 0.f) PSB_REFUSE("attention_rows_decode: bad output or gate rows, or a negative cap");
  if (keep_first < 0 || (keep_first > 0 && (window < 1 || chunk > 0))) PSB_REFUSE("attention_rows_decode: kept first keys go with a window and no chunk mask");
  if (table_width < 1 || window < 0 || chunk < 0 || (bias && reach < 1) || num_pages < 1) PSB_REFUSE("attention_rows_decode: bad arguments");
  if (blocks < 0 || (blocks > 0 && (!scratch || least_runs < 1))) PSB_REFUSE("attention_rows_decode: %d blocks of at least %d runs, or their scratch is missing", blocks, least_runs);
  if (((uintptr_t)kv & 15) || ((uintptr_t)q & 3) || ((uintptr_t)scratch & 15)) PSB_REFUSE("attention_rows_decode: operands are not aligned");
  if (T <= 0) return 0;
  const long long kv_rows = num_pages * hkv * page_size;
  if (kv_rows > 0x7fffffffLL || (long long)T * hkv > 0x7fffffffLL) PSB_REFUSE("attention_rows_decode: too many cache rows or tokens");
  DecodeArgs args{};
  args.q = (const __nv_bfloat16*)q; args.gate = (const __nv_bfloat16*)gate; args.table = (const int32_t*)table;
  args.positions = (const int32_t*)positions; args.token_item = (const int32_t*)token_item; args.bias = (const float*)bias;
  args.sink = (const float*)sink; args.out = (__nv_bfloat16*)out; args.ldg = ldg; args.ldo = ldo; args.tokens = T;
  args.least_runs = blocks > 0 ? least_runs : 0;
  args.table_width = table_width; args.hq = hq; args.hkv = hkv; args.window = window; args.chunk = chunk; args.reach = reach;
  args.keep_first = keep_first; args.scale = scale; args.softcap = softcap; args.out_scale = out_scale;
  set_scratch(args, scratch);
  while ((1 << args.page_shift) < page_size) ++args.page_shift;
  CUtensorMap map;
  const int r = make_map_bf16(&map, kv, (uint64_t)kv_rows, (uint64_t)2 * D, (uint64_t)2 * D, RUN);
  if (r != 0) PSB_REFUSE("attention_rows_decode: no tensor map (%d)", r);
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(attention_rows_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
      PSB_REFUSE("attention_rows_decode: cannot reserve %d bytes of shared memory", SMEM_BYTES);
    configured.set();
  }
  psb_launch(attention_rows_decode_kernel, dim3((unsigned)(blocks > 0 ? blocks : T * hkv)), dim3(THREADS), (size_t)SMEM_BYTES, stream, map, args);
  PSB_LAUNCH_CHECK("attention_rows_decode");
  return 0;
}

// (scratch of the launch before, sink, out, T, hq, hkv, gate, ldg, ldo, out_scale, stream)
PSB_API int psb_attention_rows_decode_merge(void* scratch, const void* sink, void* out, int T, int hq, int hkv, const void* gate,
                                            long long ldg, long long ldo, float out_scale, cudaStream_t stream) {
  if (T < 0 || !psb_attention_rows_decode_supported(hq, hkv, D, D, RUN) || !scratch || ((uintptr_t)scratch & 15) || ldo < (long long)hq * D ||
      (gate && ldg < (long long)hq * D))
    PSB_REFUSE("attention_rows_decode_merge: bad arguments");
  if (T == 0) return 0;
  DecodeArgs args{};
  args.gate = (const __nv_bfloat16*)gate; args.sink = (const float*)sink; args.out = (__nv_bfloat16*)out; args.ldg = ldg; args.ldo = ldo;
  args.tokens = T; args.hq = hq; args.hkv = hkv; args.out_scale = out_scale;
  set_scratch(args, scratch);
  psb_launch(attention_rows_decode_merge_kernel, dim3((unsigned)(T * hkv)), dim3(32 * (hq / hkv)), 0, stream, args);
  PSB_LAUNCH_CHECK("attention_rows_decode_merge");
  return 0;
}

// 0 while no bounded wait of this kernel has ever run out on the current device; reading it synchronises with the device.
PSB_API int psb_attention_rows_decode_status() { return tc::read_status(); }
