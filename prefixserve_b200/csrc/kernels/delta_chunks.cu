// The gated delta rule over long portions of bfloat16 projections, 32 tokens at a time, float32 throughout.
//
// Distances from float64 for the same inputs, token by token and here: read-outs, before they are rounded to bfloat16, 1.10e-7 to
// 1.30e-7 and 1.08e-7 to 1.24e-7 (9, 31, 64, 700 and 2,000 tokens); states 0.9e-7 to 1.5e-7 and 0.7e-7 to 1.1e-7.  That takes products
// of U, of B U and of the new state to their last bit (tf32_terms.cuh), and K K^T and Q K^T added up in pairs; with two terms throughout
// and a chain over the numbers it was 1.8e-7 and 1.5e-7, 182 us for 2,000 tokens instead of 220.  Float32 projections stay with the
// token-by-token kernel.
//
// Within a chunk, with g_l the decays, c_i = g_1 .. g_i (from the chunk's start up to token i), r_j = g_(j+1) .. g_32 and S the
// state before the chunk, the writes u_i of its tokens are the rows of
//
//     U = W (V - diag(c) K S),   W = (I + diag(beta) A)^-1 diag(beta),   A_ij = (k_i . k_j) g_(j+1) .. g_i   (j < i),
//     O = diag(c) Q S + B U,     B_ij = (q_i . k_j) g_(j+1) .. g_i   (j <= i),
//     S <- c_32 S + K^T diag(r) U.
//
// (Decays are only ever multiplied, never divided by.)  W and B do not depend on the state:
//   delta_chunk_kernel   a block per chunk and query/key group, all chunks of the step side by side: K K^T and Q K^T of the group
//                        once, then a warp per head its decays, B and W (forward substitution, a column a lane).  Leaves W, B, c
//                        and r, 8.4 KB a chunk and head;
//   delta_chain_kernel   a block of 16 warps per 16 columns of a head's state and request walks the chunks; what a chunk brings
//                        comes in with cp.async one chunk ahead.  [K; Q] S (16 rows and a quarter of the keys' numbers a warp),
//                        V - .. and W (..) by four warps while four others make the last chunk's O, then the new state (16 x 8
//                        of its numbers a warp, which stay in its registers as float32), all on the tensor cores with operands
//                        in terms.
// W and B are zero above the diagonal, and zero times what is not finite is not zero: a sum that comes out not finite is made again from
// its own terms, the tokens up to its own, so that a token reaches later ones only.
// Chunks are counted through the step's portions of at least ``min_tokens`` tokens in order; a portion's last chunk is filled up
// with tokens of beta 0, key 0 and decay 1.
//
// What bounds it: the chain, by what its warps issue (53 % of the slots busy; splitting operands is the largest share) and the
// barriers between its three phases, on as many SMs as there are heads and runs of 16 columns.  2,000 tokens of 16 heads:
// 220 us, all but about 20 of them the chain.  The same chain on the CUDA cores was bound by what shared memory hands to registers (238 us); the
// token-by-token kernel (delta_rule.cu) waits for a butterfly every two tokens (611 us).  Eight warps a block and two blocks an
// SM took as long.
#include "delta_common.cuh"
#include "portions.cuh"
#include "tf32_terms.cuh"

namespace {
using namespace delta;
using namespace terms;

constexpr int CHUNK = 32, COLS = 16;
constexpr int RP = 128;                  // keys are filled up to so many numbers
// pitches in shared memory, such that fragments of the products meet every bank once; SP: of rows of (hi, lo) pairs
constexpr int KP = RP + 8, TP = CHUNK + 4, CP = COLS + 8, SP = COLS + 4;
constexpr int CHAIN_THREADS = 512, CHUNK_THREADS = 128;

// a chunk's record of a head: W, B [32][32], c, r [32]
constexpr int W_AT = 0, B_AT = CHUNK * CHUNK, C_AT = 2 * CHUNK * CHUNK, R_AT = C_AT + CHUNK, RECORD = R_AT + CHUNK;

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ float both(uint64_t v) {  // the sum of a pair
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
struct Pairs {
  uint64_t lo, hi;
};
__device__ __forceinline__ Pairs load4(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}

__global__ void __launch_bounds__(CHUNK_THREADS)
delta_chunk_kernel(const float* __restrict__ qkv, const float* __restrict__ bd, const int32_t* __restrict__ item_start,
                   float* __restrict__ records, int items, int min_tokens, int G, int H, int dim, int vdim) {
  constexpr int WARPS = CHUNK_THREADS / 32;
  __shared__ __align__(16) float rows[2 * CHUNK * KP];
  __shared__ float kk[CHUNK][CHUNK + 1], qk[CHUNK][CHUNK + 1];
  float *ks = rows, *qs = rows + CHUNK * KP;
  float(*as)[CHUNK][TP] = reinterpret_cast<float(*)[CHUNK][TP]>(rows);  // A of a warp's head, where the keys and queries were
  static_assert(WARPS * CHUNK * TP <= 2 * CHUNK * KP, "room for every warp's A");
  pdl_wait();
  int t0, n;
  if (!portions::find_chunk<CHUNK>(item_start, items, min_tokens, blockIdx.x, t0, n)) return;
  const int g = blockIdx.y, C = 2 * G * dim + H * vdim;
  for (int i = threadIdx.x; i < CHUNK * RP / 4; i += CHUNK_THREADS) {
    const int t = i / (RP / 4), d = (i - t * (RP / 4)) * 4;
    const bool there = t < n && d < dim;
    const float* src = qkv + (size_t)(t0 + (there ? t : 0)) * C + (size_t)g * dim + (there ? d : 0);
    copy_async16_or_zero(qs + t * KP + d, src, there);
    copy_async16_or_zero(ks + t * KP + d, src + (size_t)G * dim, there);
  }
  copy_async_wait();
  __syncthreads();
  {
    // a thread: rows ti + 8a of K (or Q) against rows tj + 8b of K (rows eight apart, so that neighbours meet other banks)
    const int ti = (threadIdx.x & 63) >> 3, tj = threadIdx.x & 7;
    const bool query = threadIdx.x >= 64;
    const float* left = (query ? qs : ks) + ti * KP;
    const float* right = ks + tj * KP;
    // 16 numbers at a time, then in pairs: a single chain over the 128 was what lost most of a read-out
    auto block = [&](int d0, float (&out)[4][4]) {
      uint64_t acc[4][4] = {};
#pragma unroll
      for (int d = d0; d < d0 + 16; d += 4) {
        Pairs a[4], b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          a[e] = load4(left + e * 8 * KP + d);
          b[e] = load4(right + e * 8 * KP + d);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            fma2(acc[x][y], a[x].lo, b[y].lo);
            fma2(acc[x][y], a[x].hi, b[y].hi);
          }
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) out[x][y] = both(acc[x][y]);
    };
    auto add = [](float (&to)[4][4], const float (&what)[4][4]) {
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) to[x][y] += what[x][y];
    };
    float total[4][4] = {};
#pragma unroll 1
    for (int d = 0; d < RP; d += 64) {
      float p[4][4], r[4][4], u[4][4];
      block(d, p);
      block(d + 16, r);
      add(p, r);
      block(d + 32, r);
      block(d + 48, u);
      add(r, u);
      add(p, r);
      add(total, p);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) (query ? qk : kk)[ti + 8 * x][tj + 8 * y] = total[x][y];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per = H / G;
  for (int hh = warp; hh < per; hh += WARPS) {
    const int h = g * per + hh;
    float* out = records + ((size_t)blockIdx.x * H + h) * RECORD;
    const float* mine = bd + (size_t)(t0 + min(lane, n - 1)) * BD * H + h;
    const float beta = lane < n ? mine[0] : 0.f, decay = lane < n ? mine[H] : 1.f;
    Product run, before, behind;  // lane j: products over the tokens between j and i, up to j, behind j
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
      const float d = __shfl_sync(0xffffffffu, decay, i);
      if (i <= lane) before.times(d);
      if (i > lane) {
        run.times(d);
        behind.times(d);
      }
      as[warp][i][lane] = i > lane ? run.value() * kk[i][lane] : 0.f;
      out[B_AT + i * CHUNK + lane] = i >= lane ? run.value() * qk[i][lane] : 0.f;
    }
    out[C_AT + lane] = before.value();
    out[R_AT + lane] = behind.value();
    __syncwarp();
    float w[CHUNK];  // lane j: column j of W
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
      float acc[4] = {};
#pragma unroll
      for (int l = 0; l < i; l += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&as[warp][i][l]);  // zeros from the diagonal on
        acc[0] = fmaf(a.x, w[l], acc[0]);
        if (l + 1 < i) acc[1] = fmaf(a.y, w[l + 1], acc[1]);
        if (l + 2 < i) acc[2] = fmaf(a.z, w[l + 2], acc[2]);
        if (l + 3 < i) acc[3] = fmaf(a.w, w[l + 3], acc[3]);
      }
      const float b = __shfl_sync(0xffffffffu, beta, i);
      w[i] = b * ((i == lane ? 1.f : 0.f) - ((acc[0] + acc[1]) + (acc[2] + acc[3])));
      out[W_AT + i * CHUNK + lane] = w[i];
    }
    __syncwarp();
  }
  pdl_trigger();  // at the end: the chain's blocks are few and long (see delta_prepare_kernel)
}

// ---- the chain, on the tensor cores, operands in terms (tf32_terms.cuh) --------------------------------------------------
struct ChainShape {
  static constexpr int K_AT = 0, Q_AT = K_AT + CHUNK * KP, SW_AT = Q_AT + CHUNK * KP, V_AT = SW_AT + CHUNK * TP;
  static constexpr int STAGE = V_AT + CHUNK * CP;                          // floats of a stage
  static constexpr int B_SIZE = CHUNK * TP + 2 * CHUNK;                    // B, then c and r: read one chunk longer than the rest
  static constexpr int RING_AT = 2 * STAGE, S_AT = RING_AT + 3 * B_SIZE;   // the state in (hi, lo) pairs
  static constexpr int UU_AT = S_AT + RP * 2 * SP, U_AT = UU_AT + CHUNK * 2 * SP;  // U times r in (hi, lo) pairs; U of two chunks
  static constexpr int PART_AT = U_AT + 2 * CHUNK * CP, FLOATS = PART_AT + 2 * 4 * 2 * CHUNK * CP;  // quarters of [K; Q] S, of two chunks
};

__device__ __forceinline__ void store_split(float* at, float x, float y) {  // two neighbours of a row of pairs
  const Split a = split(x), b = split(y);
  *reinterpret_cast<uint4*>(at) = make_uint4(a.hi, a.lo, b.hi, b.lo);
}
__device__ __forceinline__ Split load_split(const float* at) {
  const uint2 v = *reinterpret_cast<const uint2*>(at);
  return {v.x, v.y};
}
__global__ void __launch_bounds__(CHAIN_THREADS, 1)
delta_chain_kernel(const float* __restrict__ qkv, const float* __restrict__ records, const __nv_bfloat16* __restrict__ proj, long long P,
                   float* __restrict__ state, const int32_t* __restrict__ item_start, const int32_t* __restrict__ slots,
                   float* __restrict__ o, int items, int all_chunks, int min_tokens, int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats) {
  using Sh = ChainShape;
  extern __shared__ __align__(16) float chain[];
  float *st = chain + Sh::S_AT, *uu = chain + Sh::UU_AT;
  const int C = 2 * G * dim + H * vdim;
  const int h = blockIdx.y, g = h / (H / G);
  const int col0 = blockIdx.x * COLS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gr = lane >> 2, tg = lane & 3;  // the lane's row (or column) and place in a fragment
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

  auto stage = [&](int c, int thread, int threads) {
    float *buf = chain + (c & 1) * Sh::STAGE, *ring = chain + Sh::RING_AT + c % 3 * Sh::B_SIZE;
    const int ts = t0 + c * CHUNK, n = min(CHUNK, t1 - ts);
    const float* rows = qkv + (size_t)ts * C;
    const float* record = records + ((size_t)(first + c) * H + h) * RECORD;
    for (int i = thread; i < CHUNK * RP / 4; i += threads) {
      const int t = i / (RP / 4), d = (i % (RP / 4)) * 4;
      const bool there = t < n && d < dim;
      const float* src = rows + (there ? (size_t)t * C + d : 0) + (size_t)g * dim;
      copy_async16_or_zero(buf + Sh::K_AT + t * KP + d, src + (size_t)G * dim, there);
      copy_async16_or_zero(buf + Sh::Q_AT + t * KP + d, src, there);
    }
    for (int i = thread; i < CHUNK * CHUNK / 4; i += threads) {
      const int row = i / (CHUNK / 4), piece = (i % (CHUNK / 4)) * 4;
      copy_async16(buf + Sh::SW_AT + row * TP + piece, record + W_AT + row * CHUNK + piece);
      copy_async16(ring + row * TP + piece, record + B_AT + row * CHUNK + piece);
    }
    for (int i = thread; i < CHUNK * COLS / 4; i += threads) {
      const int t = i / (COLS / 4), v = (i % (COLS / 4)) * 4;
      const bool there = t < n && col0 + v < vdim;
      copy_async16_or_zero(buf + Sh::V_AT + t * CP + v, rows + (there ? (size_t)t * C + 2 * (size_t)G * dim + (size_t)h * vdim + col0 + v : 0), there);
    }
    for (int i = thread; i < 2 * CHUNK / 4; i += threads)  // c and r
      copy_async16(ring + CHUNK * TP + 4 * i, record + C_AT + 4 * i);
  };
  auto part_of = [&](int c) { return chain + Sh::PART_AT + (c & 1) * 4 * 2 * CHUNK * CP; };
  auto u_of = [&](int c) { return chain + Sh::U_AT + (c & 1) * CHUNK * CP; };

  // the read-out of chunk c, 16 rows and 8 columns a warp: while the next chunk's U is made
  auto read_out = [&](int c) {
    const int i0 = 16 * ((warp >> 1) & 1) + gr, oc = 8 * (warp & 1);
    const float *ring = chain + Sh::RING_AT + c % 3 * Sh::B_SIZE, *part = part_of(c) + (CHUNK + i0) * CP + oc + 2 * tg;
    const float *a = ring + i0 * TP + tg, *b = u_of(c) + tg * CP + oc + gr;
    Sum y;
#pragma unroll
    for (int k = 0; k < CHUNK / 8; ++k) {
      if (k >= 2 && i0 < 16) break;  // B is triangular
      uint32_t ah[4], al[4];
      load_rows(a + 8 * k, 8 * TP, 4, ah, al);
      y.step<6>(ah, al, split(b[8 * k * CP]), split(b[(8 * k + 4) * CP]));
    }
    float total[4];
    y.totals(total);
    if (!all_finite(total)) {
#pragma unroll 1
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + 8 * (e >> 1);
        float sum = 0.f;
#pragma unroll 1
        for (int j = 0; j <= i; ++j) sum = fmaf(ring[i * TP + j], u_of(c)[j * CP + oc + 2 * tg + (e & 1)], sum);
        if (!is_finite(pick(total, e))) place(total, e, sum);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = t0 + c * CHUNK + i0 + 8 * r, col = col0 + oc + 2 * tg;
      float2 v = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 p = *reinterpret_cast<const float2*>(part + (q * 2 * CHUNK + 8 * r) * CP);
        v.x += p.x;
        v.y += p.y;
      }
      const float ci = ring[CHUNK * TP + i0 + 8 * r];
      if (t < t1 && col < vdim)
        *reinterpret_cast<float2*>(o + ((size_t)t * H + h) * vdim + col) = make_float2(fmaf(ci, v.x, total[2 * r]), fmaf(ci, v.y, total[2 * r + 1]));
    }
  };

  stage(0, threadIdx.x, CHAIN_THREADS);
  // the state: rows 16 (warp / 2) + gr and + 8, columns 8 (warp % 2) + 2 tg and + 1 are this thread's
  float s[4];
  const int d0 = 16 * (warp >> 1) + gr, sc = 8 * (warp & 1) + 2 * tg;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int d = d0 + 8 * (e >> 1), col = col0 + sc + (e & 1);
    s[e] = (d < dim && col < vdim) ? S[(size_t)d * vdim + col] : 0.f;
  }
  store_split(st + (d0 * SP + sc) * 2, s[0], s[1]);
  store_split(st + ((d0 + 8) * SP + sc) * 2, s[2], s[3]);
  // [K; Q] S: 16 rows (of K: mt 0 and 1, of Q: 2 and 3) over a quarter of the keys' numbers
  const int mt = warp >> 2, quarter = warp & 3;

  for (int c = 0; c < chunks; ++c) {
    copy_async_wait();
    __syncthreads();  // this chunk and the state have landed, and everybody has left the other buffer
    const float* buf = chain + (c & 1) * Sh::STAGE;
    const float* ring = chain + Sh::RING_AT + c % 3 * Sh::B_SIZE;
    {
      Sum y[2];
      const float* a = buf + (mt < 2 ? Sh::K_AT : Sh::Q_AT) + ((mt & 1) * 16 + gr) * KP + quarter * (RP / 4) + tg;
      const float* b = st + ((quarter * (RP / 4) + tg) * SP + gr) * 2;
#pragma unroll
      for (int k = 0; k < RP / 32; ++k) {
        uint32_t ah[4], al[4];
        load_rows(a + 8 * k, 8 * KP, 4, ah, al);
#pragma unroll
        for (int n = 0; n < 2; ++n) y[n].step<4>(ah, al, load_split(b + (8 * k * SP + 8 * n) * 2), load_split(b + ((8 * k + 4) * SP + 8 * n) * 2));
      }
      float* part = part_of(c) + (quarter * 2 * CHUNK + mt * 16 + gr) * CP + 2 * tg;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        *reinterpret_cast<float2*>(part + 8 * n) = make_float2(y[n].total(0), y[n].total(1));
        *reinterpret_cast<float2*>(part + 8 * CP + 8 * n) = make_float2(y[n].total(2), y[n].total(3));
      }
    }
    __syncthreads();
    if (warp < 4) {  // U = W (V - ..): 16 rows and 8 columns a warp, which puts the right side together itself
      const int i0 = 16 * (warp >> 1) + gr, uc = 8 * (warp & 1);
      const float *a = buf + Sh::SW_AT + i0 * TP + tg, *v = buf + Sh::V_AT + tg * CP + uc + gr, *part = part_of(c) + tg * CP + uc + gr;
      Sum u;
#pragma unroll
      for (int k = 0; k < CHUNK / 8; ++k) {
        if (k >= 2 && i0 < 16) break;  // W is triangular
        uint32_t ah[4], al[4];
        load_rows(a + 8 * k, 8 * TP, 4, ah, al);
        Split x[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = (8 * k + 4 * e) * CP;
          const float y = (part[i] + part[2 * CHUNK * CP + i]) + (part[4 * CHUNK * CP + i] + part[6 * CHUNK * CP + i]);
          x[e] = split(fmaf(-ring[CHUNK * TP + 8 * k + 4 * e + tg], y, v[i]));
        }
        u.step<6>(ah, al, x[0], x[1]);
      }
      float total[4];
      u.totals(total);
      if (!all_finite(total)) {
#pragma unroll 1
        for (int e = 0; e < 4; ++e) {
          const int i = i0 + 8 * (e >> 1), col = uc + 2 * tg + (e & 1);
          float sum = 0.f;
#pragma unroll 1
          for (int j = 0; j <= i; ++j) {
            const float* q = part_of(c) + j * CP + col;
            const float y = (q[0] + q[2 * CHUNK * CP]) + (q[4 * CHUNK * CP] + q[6 * CHUNK * CP]);
            sum = fmaf(buf[Sh::SW_AT + i * TP + j], fmaf(-ring[CHUNK * TP + j], y, buf[Sh::V_AT + j * CP + col]), sum);
          }
          if (!is_finite(pick(total, e))) place(total, e, sum);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + 8 * r, col = uc + 2 * tg;
        const float ri = ring[CHUNK * TP + CHUNK + i];
        *reinterpret_cast<float2*>(u_of(c) + i * CP + col) = make_float2(total[2 * r], total[2 * r + 1]);
        store_split(uu + (i * SP + col) * 2, total[2 * r] * ri, total[2 * r + 1] * ri);
      }
    } else if (warp < 8) {
      if (c > 0) read_out(c - 1);
    } else if (c + 1 < chunks) {
      stage(c + 1, threadIdx.x - 256, CHAIN_THREADS - 256);
    }
    __syncthreads();
    {
      Sum d;
      const float* a = buf + Sh::K_AT + tg * KP + d0;
      const float* b = uu + (tg * SP + 8 * (warp & 1) + gr) * 2;
#pragma unroll
      for (int k = 0; k < CHUNK / 8; ++k) {
        uint32_t ah[4], al[4];
        load_rows(a + 8 * k * KP, 8, 4 * KP, ah, al);
        d.step<6>(ah, al, load_split(b + 8 * k * SP * 2), load_split(b + (8 * k + 4) * SP * 2));
      }
      const float all = ring[CHUNK * TP + CHUNK - 1];
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = fmaf(all, s[e], d.total(e));
      store_split(st + (d0 * SP + sc) * 2, s[0], s[1]);
      store_split(st + ((d0 + 8) * SP + sc) * 2, s[2], s[3]);
    }
  }
  if (warp >= 4 && warp < 8 && chunks > 0) read_out(chunks - 1);
  pdl_trigger();  // at the end, as in delta_chunk_kernel
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int d = d0 + 8 * (e >> 1), col = col0 + sc + (e & 1);
    if (d < dim && col < vdim) S[(size_t)d * vdim + col] = s[e];
  }
  if (blockIdx.x == 0 && h == 0) keep_conv_inputs<__nv_bfloat16>(proj, P, base, t0, t1, C, K);
}

}  // namespace

// (dim, vdim) -> float32 numbers of a chunk's record of a head, 0 if the kernels are not built for the sizes
PSB_API int psb_delta_chunk_record(int dim, int vdim) {
  return dim >= 4 && dim <= RP && dim % 4 == 0 && vdim >= 4 && vdim % 4 == 0 ? RECORD : 0;
}

// () -> tokens of a chunk
PSB_API int psb_delta_chunk_tokens() { return CHUNK; }

// The rule over every portion of at least ``min_tokens`` tokens, from what psb_delta_prepare left; other tokens, and the slots of
// other portions, are left untouched.  records [chunks, H, RECORD] float32, portions and chunks at least the number of these portions
// and of their chunks.
// (qkv, bd, proj bfloat16, ld, state, item_start, slots, records, o_out, items, portions, chunks, min_tokens, G, H, dim, vdim, K,
//  num_slots, slot_floats, stream)
PSB_API int psb_delta_chunks(const void* qkv, const void* bd, const void* proj, long long ld, void* state, const void* item_start,
                             const void* slots, void* records, void* o, int items, int portions, int chunks, int min_tokens, int G, int H,
                             int dim, int vdim, int K, int num_slots, long long slot_floats, cudaStream_t stream) {
  if (items < 0 || G < 1 || H < 1 || H % G || !psb_delta_chunk_record(dim, vdim)) PSB_REFUSE("delta_chunks: bad sizes G=%d H=%d dim=%d vdim=%d", G, H, dim, vdim);
  if (K < 1 || K > MAX_TAPS || min_tokens < 1 || num_slots < 1) PSB_REFUSE("delta_chunks: %d taps are outside [1, %d], or no tokens or slots", K, MAX_TAPS);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  if (ld < C || slot_floats != (K - 1) * C + (long long)H * dim * vdim) PSB_REFUSE("delta_chunks: the slot or the rows do not fit the sizes");
  if (H > 65535 || portions > 65535 || chunks < 0) PSB_REFUSE("delta_chunks: too many heads or requests for one launch");
  if (((uintptr_t)qkv | (uintptr_t)records) & 15) PSB_REFUSE("delta_chunks: operands must be 16-byte aligned");
  if (items == 0 || portions < 1 || chunks == 0) return 0;
  constexpr int bytes = ChainShape::FLOATS * (int)sizeof(float);
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(delta_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
      PSB_REFUSE("delta_chunks: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(delta_chunk_kernel, dim3(chunks, G), dim3(CHUNK_THREADS), 0, stream, (const float*)qkv, (const float*)bd, (const int32_t*)item_start,
             (float*)records, items, min_tokens, G, H, dim, vdim);
  PSB_LAUNCH_CHECK("delta_chunk");
  psb_launch(delta_chain_kernel, dim3((vdim + COLS - 1) / COLS, H, portions), dim3(CHAIN_THREADS), (size_t)bytes, stream, (const float*)qkv,
             (const float*)records, (const __nv_bfloat16*)proj, ld, (float*)state, (const int32_t*)item_start, (const int32_t*)slots, (float*)o,
             items, chunks, min_tokens, G, H, dim, vdim, K, num_slots, slot_floats);
  PSB_LAUNCH_CHECK("delta_chain");
  return 0;
}
