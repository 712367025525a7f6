// Gated linear attention (linear_attention.cu) over long portions of bfloat16 projections, 64 tokens at a time on the tensor cores,
// float32 throughout:
//
//     S <- diag(alpha_t) S + k_t v_t^T,    o_t = S^T q_t * scale.
//
// With c_i = alpha_1 .. alpha_i from a chunk's start and r_j = alpha_(j+1) .. alpha_64, per key channel,
//   linear_local_kernel    every chunk from a zero state: B = sum_j (k_j r_j) v_j^T, and A = c_64;
//   linear_starts_kernel   per portion, chunk by chunk: the state every chunk starts from (over B), and the slot's new state;
//   linear_read_kernel     O = (Q c) S + P V,  P_ij = sum_d q_i k_j alpha_(j+1) .. alpha_i  (j <= i).
// Decays are only ever multiplied, never divided by, so P is made in blocks of 16 x 16 tokens: off the diagonal as products of
// q_i alpha_(start of i's run) .. alpha_i and k_j alpha_(j+1) .. alpha_(end of j's run) with whole runs' decays between them, on the
// diagonal with a running product a column (four columns a warp, four channels a lane).
// Products of float32 numbers enter the tensor cores in terms (tf32_terms.cuh: all of them for P, those of lo lo too for (Q c) S, P to
// its last bit for P V), the values, which are bfloat16, as they are.
// P is zero above the diagonal, and zero times a value that is not finite is not zero: a result that comes out not finite is made
// again from the tokens up to its own.
// Running products of decays carry what their roundings lose.  With that read-outs lie at 1.15e-7 to 1.18e-7 from float64, token by
// token at 1.21e-7 to 1.25e-7 (100, 300 and 1,811 tokens), states at 0.80e-7 and 0.95e-7; with two terms throughout read-outs came out
// at 1.28e-7 to 1.30e-7, 1,811 tokens in 119 us instead of 129.  A float32 projection's values would need terms too; those stay with the
// other kernels.
//
// What bounds it: the read-out, by what its warps issue and by its five phases one after the other, one block of 16 warps an SM
// (190 KB of shared memory).  1,811 tokens of 16 heads of 128: local 31 us, starts 11, read-out 87; the token-by-token kernels took
// 73, 13 and 114.  Eight warps a block took 112 us for the read-out.
#include <type_traits>

#include "portions.cuh"
#include "tf32_terms.cuh"

namespace {
using namespace terms;

constexpr int CHUNK = 64, RUN = 16, RUNS = CHUNK / RUN, RP = 128, KP = RP + 8, VP = RP + 4, PP = CHUNK + 8, THREADS = 512;

// Products over k take the places 2 tg and 2 tg + 1 of every eight (instead of tg and tg + 4) of both operands: rows give them as one
// 8-byte load.  Pitches are such that such loads (KP, PP), and loads down a column (VP), meet every bank once.
__device__ __forceinline__ void load_row_pairs(const float* a, int down, float2 factor, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float2 x = *reinterpret_cast<const float2*>(a + e * down);
    const Split u = split_product(x.x, factor.x), v = split_product(x.y, factor.y);
    hi[e] = u.hi;
    lo[e] = u.lo;
    hi[2 + e] = v.hi;
    lo[2 + e] = v.lo;
  }
}

// 64 rows of ``src`` (row pitch ld, ``width`` numbers, zeros beyond them and beyond n rows) as float32
template <typename T, int PITCH>
__device__ __forceinline__ void bring(float* dst, const T* __restrict__ src, long long ld, int n, int width) {
  constexpr int EACH = CHUNK * RP / 4 / THREADS;
  using Raw = typename std::conditional<sizeof(T) == 2, uint2, float4>::type;
  Raw raw[EACH];
#pragma unroll
  for (int e = 0; e < EACH; ++e) {  // asked for together
    const int i = threadIdx.x + e * THREADS, t = i / (RP / 4), d = (i % (RP / 4)) * 4;
    raw[e] = Raw{};
    if (t < n && d < width) raw[e] = *reinterpret_cast<const Raw*>(src + (size_t)t * ld + d);
  }
#pragma unroll
  for (int e = 0; e < EACH; ++e) {
    const int i = threadIdx.x + e * THREADS, t = i / (RP / 4), d = (i % (RP / 4)) * 4;
    float4 v;
    if constexpr (sizeof(T) == 2) {
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[e].x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[e].y));
      v = make_float4(a.x, a.y, b.x, b.y);
    } else {
      v = raw[e];
    }
    *reinterpret_cast<float4*>(dst + t * PITCH + d) = v;
  }
}

__global__ void __launch_bounds__(THREADS, 2)
linear_local_kernel(const __nv_bfloat16* __restrict__ proj, long long ld, const float* __restrict__ alpha, const int32_t* __restrict__ item_start,
                    float* __restrict__ local_b, float* __restrict__ local_a, int items, int min_tokens, int H, int dim, int vdim) {
  extern __shared__ __align__(16) float linear_smem[];
  float *kr = linear_smem, *vs = kr + CHUNK * KP, *whole = vs + CHUNK * KP;  // [64][KP] each, [RUNS][RP]
  pdl_trigger();
  pdl_wait();
  int t0, n;
  if (!portions::find_chunk<CHUNK>(item_start, items, min_tokens, blockIdx.y, t0, n)) return;
  const int h = blockIdx.x;
  bring<__nv_bfloat16, KP>(kr, proj + (size_t)t0 * ld + (size_t)H * dim + (size_t)h * dim, ld, n, dim);
  bring<__nv_bfloat16, KP>(vs, proj + (size_t)t0 * ld + 2 * (size_t)H * dim + (size_t)h * vdim, ld, n, vdim);
  const int d = threadIdx.x & (RP - 1), at = threadIdx.x / RP;
  float a[RUN];  // this thread's channel over a quarter of the tokens
#pragma unroll
  for (int i = 0; i < RUN; ++i) {
    const int t = at * RUN + i;
    a[i] = t < n && d < dim ? alpha[((size_t)(t0 + t) * H + h) * dim + d] : 1.f;
  }
  Product all;
#pragma unroll
  for (int i = 0; i < RUN; ++i) all.times(a[i]);
  whole[at * RP + d] = all.value();
  __syncthreads();
  Product run;
  for (int r = RUNS - 1; r > at; --r) run.times(whole[r * RP + d]);
#pragma unroll
  for (int i = RUN - 1; i >= 0; --i) {
    kr[(at * RUN + i) * KP + d] *= run.value();
    run.times(a[i]);
  }
  if (at == 0 && d < dim) local_a[((size_t)blockIdx.y * H + h) * dim + d] = run.value();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  const int d0 = 16 * (warp & 7) + gr;
  float* dst = local_b + ((size_t)blockIdx.y * H + h) * dim * vdim;
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {  // 16 rows and 16 columns a warp
    const int c0 = (warp >> 3) * 64 + pass * 16;
    if (c0 >= vdim || 16 * (warp & 7) >= dim) break;
    Sum y[2];
#pragma unroll
    for (int k = 0; k < CHUNK / 8; ++k) {
      uint32_t ah[4], al[4];
      load_rows(kr + (8 * k + tg) * KP + d0, 8, 4 * KP, ah, al);
      const float* b = vs + (8 * k + tg) * KP + c0 + gr;
#pragma unroll
      for (int m = 0; m < 2; ++m) y[m].step<false>(ah, al, b[8 * m], b[4 * KP + 8 * m]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int col = c0 + 8 * m + 2 * tg;
        if (d0 + 8 * r < dim && col < vdim) *reinterpret_cast<float2*>(dst + (size_t)(d0 + 8 * r) * vdim + col) = make_float2(y[m].total(2 * r), y[m].total(2 * r + 1));
      }
  }
}

// A thread per four numbers of a portion's state: B of every chunk becomes the state the chunk starts from, the slot gets the last one.
__global__ void __launch_bounds__(128)
linear_starts_kernel(float* __restrict__ state, long long slot_floats, const int32_t* __restrict__ item_start,
                     const int32_t* __restrict__ slots, float* __restrict__ local_b, const float* __restrict__ local_a, int chunks,
                     int min_tokens, int H, int dim, int vdim, int num_slots) {
  pdl_trigger();
  pdl_wait();
  const int item = blockIdx.y, tokens = item_start[item + 1] - item_start[item];
  if (tokens < min_tokens) return;
  int first = 0;
  for (int i = 0; i < item; ++i) {
    const int ni = item_start[i + 1] - item_start[i];
    if (ni >= min_tokens) first += (ni + CHUNK - 1) / CHUNK;
  }
  const int n = (tokens + CHUNK - 1) / CHUNK;
  if (first + n > chunks) return;  // (the caller counted fewer than there are: no room for them)
  const long long per_chunk = (long long)H * dim * vdim, at = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (at >= per_chunk) return;
  int slot = slots[item];
  slot = slot < 0 ? 0 : (slot >= num_slots ? num_slots - 1 : slot);
  float4 run = *reinterpret_cast<const float4*>(state + (size_t)slot * slot_floats + at);
  const long long hd = at / vdim;
  constexpr int AHEAD = 8;
  for (int c0 = 0; c0 < n; c0 += AHEAD) {
    float4 b[AHEAD];
    float a[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {  // asked for together
      const int c = min(c0 + j, n - 1);
      b[j] = *reinterpret_cast<const float4*>(local_b + (size_t)(first + c) * per_chunk + at);
      a[j] = local_a[(size_t)(first + c) * H * dim + hd];
    }
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      if (c0 + j >= n) break;
      *reinterpret_cast<float4*>(local_b + (size_t)(first + c0 + j) * per_chunk + at) = run;
      run.x = fmaf(a[j], run.x, b[j].x);
      run.y = fmaf(a[j], run.y, b[j].y);
      run.z = fmaf(a[j], run.z, b[j].z);
      run.w = fmaf(a[j], run.w, b[j].w);
    }
  }
  *reinterpret_cast<float4*>(state + (size_t)slot * slot_floats + at) = run;
}

struct ReadShape {
  static constexpr int Q_AT = 0, K_AT = Q_AT + CHUNK * KP, V_AT = K_AT + CHUNK * KP, S_AT = V_AT + CHUNK * VP;
  static constexpr int P_AT = S_AT + RP * VP, W_AT = P_AT + CHUNK * PP;      // W: decays of whole runs
  static constexpr int F_AT = W_AT + RUNS * RP, FLOATS = F_AT + 7 * RP;      // F: products of those
};

__global__ void __launch_bounds__(THREADS, 1)
linear_read_kernel(const __nv_bfloat16* __restrict__ proj, long long ld, const float* __restrict__ alpha, const int32_t* __restrict__ item_start,
                   const float* __restrict__ starts, float* __restrict__ o, int items, int min_tokens, int H, int dim, int vdim, float scale) {
  using Sh = ReadShape;
  extern __shared__ __align__(16) float linear_smem[];
  float *qs = linear_smem + Sh::Q_AT, *ks = linear_smem + Sh::K_AT, *vs = linear_smem + Sh::V_AT, *ss = linear_smem + Sh::S_AT;
  float *ps = linear_smem + Sh::P_AT, *whole = linear_smem + Sh::W_AT, *fs = linear_smem + Sh::F_AT;
  float* as = ss;  // the decays, [64][KP], until the state takes their place
  pdl_trigger();
  pdl_wait();
  int t0, n;
  if (!portions::find_chunk<CHUNK>(item_start, items, min_tokens, blockIdx.y, t0, n)) return;
  const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  const __nv_bfloat16* rows = proj + (size_t)t0 * ld;
  bring<__nv_bfloat16, KP>(qs, rows + (size_t)h * dim, ld, n, dim);
  bring<__nv_bfloat16, KP>(ks, rows + (size_t)H * dim + (size_t)h * dim, ld, n, dim);
  bring<__nv_bfloat16, VP>(vs, rows + 2 * (size_t)H * dim + (size_t)h * vdim, ld, n, vdim);
  bring<float, KP>(as, alpha + ((size_t)t0 * H + h) * dim, (long long)H * dim, n, dim);  // (channels and tokens that are not there: q and k are 0)
  for (int i = threadIdx.x; i < CHUNK * PP; i += THREADS) ps[i] = 0.f;
  __syncthreads();
  // P on the diagonal: columns j0 .. j0 + 3 of a run, the lane's four channels, down the run's rows
  static_assert(THREADS / 32 == RUNS * RUN / 4, "a warp per four columns");
  {
    const int j0 = ((warp + (warp >> 2)) & 3) * 4, base = (warp >> 2) * RUN;
    Product run[4][4];  // with what the roundings lose: up to fifteen decays a product
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 row = *reinterpret_cast<const float4*>(ks + (base + j0 + j) * KP + 4 * lane);
      run[j][0].hi = row.x;
      run[j][1].hi = row.y;
      run[j][2].hi = row.z;
      run[j][3].hi = row.w;
    }
#pragma unroll 2
    for (int i = j0; i < RUN; ++i) {
      const float4 q = *reinterpret_cast<const float4*>(qs + (base + i) * KP + 4 * lane), a = *reinterpret_cast<const float4*>(as + (base + i) * KP + 4 * lane);
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i > j0 + j) {
          run[j][0].times(a.x);
          run[j][1].times(a.y);
          run[j][2].times(a.z);
          run[j][3].times(a.w);
        }
        v[j] = fmaf(q.x, run[j][0].value(), q.y * run[j][1].value()) + fmaf(q.z, run[j][2].value(), q.w * run[j][3].value());
      }
      // the four sums over the warp: lane's bits 3 and 4 choose which of them it ends up with
      const bool up4 = lane & 16, up3 = lane & 8;
      const float x0 = (up4 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up4 ? v[0] : v[2], 16);
      const float x1 = (up4 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up4 ? v[1] : v[3], 16);
      float y = (up3 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, up3 ? x0 : x1, 8);
      y += __shfl_xor_sync(0xffffffffu, y, 4);
      y += __shfl_xor_sync(0xffffffffu, y, 2);
      y += __shfl_xor_sync(0xffffffffu, y, 1);
      const int j = j0 + (up4 ? 2 : 0) + (up3 ? 1 : 0);
      if ((lane & 7) == 0 && j <= i) ps[(base + i) * PP + base + j] = y;
    }
  }
  __syncthreads();
  {  // queries times the decays from their run's start, keys times those to their run's end
    const int d = threadIdx.x & (RP - 1), base = threadIdx.x / RP * RUN;
    float a[RUN];
#pragma unroll
    for (int i = 0; i < RUN; ++i) a[i] = base + i < n && d < dim ? as[(base + i) * KP + d] : 1.f;
    Product front, behind;
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      front.times(a[i]);
      qs[(base + i) * KP + d] *= front.value();
    }
    whole[(base / RUN) * RP + d] = front.value();
#pragma unroll
    for (int i = RUN - 1; i >= 0; --i) {
      ks[(base + i) * KP + d] *= behind.value();
      behind.times(a[i]);
    }
  }
  __syncthreads();
  {  // the state the chunk starts from, in the decays' place
    const float* S = starts + ((size_t)blockIdx.y * H + h) * dim * vdim;
    for (int i = threadIdx.x; i < RP * RP / 4; i += THREADS) {
      const int d = i / (RP / 4), c = (i % (RP / 4)) * 4;
      const bool there = d < dim && c < vdim;
      const float* src = S + (there ? (size_t)d * vdim + c : 0);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(ss + d * VP + c)), "l"(src), "r"(there ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (threadIdx.x < RP) {
    const int d = threadIdx.x;
    const float w0 = whole[d], w1 = whole[RP + d], w2 = whole[2 * RP + d];
    fs[d] = 1.f;                        // 0 .. 3: in front of run 0, 1, 2, 3
    fs[RP + d] = w0;
    fs[2 * RP + d] = w0 * w1;
    fs[3 * RP + d] = w0 * w1 * w2;
    fs[4 * RP + d] = w1;                // between runs 0 and 2
    fs[5 * RP + d] = w2;                // ... 1 and 3
    fs[6 * RP + d] = w1 * w2;           // ... 0 and 3
  }
  __syncthreads();
  // a fragment of the queries of run m times a vector of F
  auto queries = [&](int m, const float* f, int k, uint32_t (&ah)[4], uint32_t (&al)[4]) {
    load_row_pairs(qs + (m * RUN + gr) * KP + 8 * k + 2 * tg, 8 * KP, *reinterpret_cast<const float2*>(f + 8 * k + 2 * tg), ah, al);
  };
  if (warp < 12) {  // P off the diagonal: runs (1,0) (2,0) (2,1) (3,0) (3,1) (3,2), eight columns a warp
    const int pair = warp >> 1, m = pair < 1 ? 1 : pair < 3 ? 2 : 3, j = pair - m * (m - 1) / 2, c0 = 8 * (warp & 1);
    const float* f = fs + (m - j == 1 ? 0 : m - j == 3 ? 6 : m == 2 ? 4 : 5) * RP;
    Sums<2> y;
#pragma unroll 4
    for (int k = 0; k < RP / 8; ++k) {
      uint32_t ah[4], al[4];
      queries(m, f, k, ah, al);
      const float2 b = *reinterpret_cast<const float2*>(ks + (j * RUN + c0 + gr) * KP + 8 * k + 2 * tg);
      y.step<6>(ah, al, split(b.x), split(b.y), k & 1);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
      *reinterpret_cast<float2*>(ps + (m * RUN + gr + 8 * r) * PP + j * RUN + c0 + 2 * tg) = make_float2(y.total(2 * r), y.total(2 * r + 1));
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // O: the 16 rows of run m, 32 columns a warp (the runs in turn, so that no scheduler gets all the long ones)
  const int m = (warp + (warp >> 2)) & 3, c0 = (warp >> 2) * 32;
  if (m * RUN >= n || c0 >= vdim) return;
  Sums<2> y[4];
#pragma unroll 4
  for (int k = 0; k < RP / 8; ++k) {
    uint32_t ah[4], al[4];
    queries(m, fs + m * RP, k, ah, al);
    const float* b = ss + (8 * k + 2 * tg) * VP + c0 + gr;
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c].step<4>(ah, al, split(b[8 * c]), split(b[VP + 8 * c]), k & 1);
  }
#pragma unroll 2
  for (int k = 0; k < 2 * (m + 1); ++k) {
    uint32_t ah[4], al[4];
    load_row_pairs(ps + (m * RUN + gr) * PP + 8 * k + 2 * tg, 8 * PP, make_float2(1.f, 1.f), ah, al);
    const float* b = vs + (8 * k + 2 * tg) * VP + c0 + gr;
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c].step<true>(ah, al, b[8 * c], b[VP + 8 * c], k & 1);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int i = m * RUN + gr + 8 * r;
    if (i >= n) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int col = c0 + 8 * c + 2 * tg;
      if (col >= vdim) continue;
      float v[2] = {y[c].total(2 * r), y[c].total(2 * r + 1)};
      if (!is_finite(v[0]) || !is_finite(v[1])) {
        float again[2] = {0.f, 0.f};
#pragma unroll 1
        for (int d = 0; d < dim; ++d) {
          const float q = qs[i * KP + d] * fs[m * RP + d];
          again[0] = fmaf(q, ss[d * VP + col], again[0]);
          again[1] = fmaf(q, ss[d * VP + col + 1], again[1]);
        }
#pragma unroll 1
        for (int j = 0; j <= i; ++j) {
          again[0] = fmaf(ps[i * PP + j], vs[j * VP + col], again[0]);
          again[1] = fmaf(ps[i * PP + j], vs[j * VP + col + 1], again[1]);
        }
        if (!is_finite(v[0])) v[0] = again[0];
        if (!is_finite(v[1])) v[1] = again[1];
      }
      *reinterpret_cast<float2*>(o + ((size_t)(t0 + i) * H + h) * vdim + col) = make_float2(v[0] * scale, v[1] * scale);
    }
  }
}

}  // namespace

// (dim, vdim) -> 1 if these kernels take the sizes
PSB_API int psb_linear_chunks_supported(int dim, int vdim) { return dim >= 4 && dim <= RP && dim % 4 == 0 && vdim >= 4 && vdim <= RP && vdim % 4 == 0 ? 1 : 0; }

// () -> tokens of a chunk
PSB_API int psb_linear_chunk_tokens() { return CHUNK; }

// Every portion of at least ``min_tokens`` tokens, and its slot; other tokens and slots are left untouched.  local_b [chunks, H, dim,
// vdim] and local_a [chunks, H, dim] float32 are scratch, chunks at least the number of these portions' chunks.
// (proj bfloat16, ld, alpha, state, slot_floats, item_start, slots, local_b, local_a, o, items, chunks, min_tokens, H, dim, vdim, num_slots,
//  scale, stream)
PSB_API int psb_linear_chunks(const void* proj, long long ld, const void* alpha, void* state, long long slot_floats,
                              const void* item_start, const void* slots, void* local_b, void* local_a, void* o, int items, int chunks,
                              int min_tokens, int H, int dim, int vdim, int num_slots, float scale, cudaStream_t stream) {
  if (items < 0 || H < 1 || num_slots < 1 || min_tokens < 1 || !psb_linear_chunks_supported(dim, vdim)) PSB_REFUSE("linear_chunks: bad sizes H=%d dim=%d vdim=%d", H, dim, vdim);
  if (ld < 2LL * H * dim + (long long)H * vdim || ld % 4) PSB_REFUSE("linear_chunks: row stride %lld is shorter than the row or no multiple of 4", ld);
  if (slot_floats < (long long)H * dim * vdim || slot_floats % 4) PSB_REFUSE("linear_chunks: a slot of %lld numbers does not hold the state, or is no multiple of 4", slot_floats);
  if (((uintptr_t)proj & 7) || (((uintptr_t)alpha | (uintptr_t)state | (uintptr_t)local_b | (uintptr_t)o) & 15))
    PSB_REFUSE("linear_chunks: operands are not aligned");
  if (H > 65535 || chunks > 65535 || items > 65535) PSB_REFUSE("linear_chunks: too many heads, requests or chunks for one launch");
  if (items == 0 || chunks < 1) return 0;
  constexpr int local_bytes = (2 * CHUNK * KP + RUNS * RP) * (int)sizeof(float), read_bytes = ReadShape::FLOATS * (int)sizeof(float);
  static PsbPerDevice configured;
  if (!configured.get()) {
    if (cudaFuncSetAttribute(linear_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, local_bytes) != cudaSuccess ||
        cudaFuncSetAttribute(linear_read_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, read_bytes) != cudaSuccess)
      PSB_REFUSE("linear_chunks: cannot raise the shared-memory limit");
    configured.set();
  }
  psb_launch(linear_local_kernel, dim3(H, chunks), dim3(THREADS), (size_t)local_bytes, stream, (const __nv_bfloat16*)proj, ld, (const float*)alpha,
             (const int32_t*)item_start, (float*)local_b, (float*)local_a, items, min_tokens, H, dim, vdim);
  PSB_LAUNCH_CHECK("linear_local");
  const long long fours = (long long)H * dim * vdim / 4;
  psb_launch(linear_starts_kernel, dim3((unsigned)((fours + 127) / 128), items), dim3(128), 0, stream, (float*)state, slot_floats,
             (const int32_t*)item_start, (const int32_t*)slots, (float*)local_b, (const float*)local_a, chunks, min_tokens, H, dim, vdim,
             num_slots);
  PSB_LAUNCH_CHECK("linear_starts");
  psb_launch(linear_read_kernel, dim3(H, chunks), dim3(THREADS), (size_t)read_bytes, stream, (const __nv_bfloat16*)proj, ld, (const float*)alpha,
             (const int32_t*)item_start, (const float*)local_b, (float*)o, items, min_tokens, H, dim, vdim, scale);
  PSB_LAUNCH_CHECK("linear_read");
  return 0;
}
