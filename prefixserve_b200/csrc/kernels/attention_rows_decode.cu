// Attention of steps of single tokens over cache rows that hold a key and then its value, heads of 128 in bfloat16, fed by the TMA
// unit: what attention_rows_single_kernel (attention_biased.cu) computes, where up to eight query heads read a key/value head.
//
// A block takes a token, a key/value head and a share of the keys: one producer warp asks for runs of 16 keys aligned to absolute
// positions (four boxes of 64 columns with 128-byte swizzle, keys then values) into a ring of eight stages, four consumer warps take
// the runs in turn: ldmatrix out of the swizzled rows, S = Q K^T (mma.sync m16n8k16: heads in rows, keys in columns), scale, cap,
// bias, masks and the online softmax in float32.  The weights are float32 and keep 16 bits: hi + lo, two bfloat16 numbers.  With at
// most eight heads half of an instruction's rows would be empty, so rows 0..7 carry the hi terms and rows 8..15 the lo terms of the
// same heads, and one instruction does both; the two halves of the result are added up at the end.  O is rescaled only when a row's
// maximum has grown.  Blocks that share a token's keys leave partial results for attention_biased_merge_kernel.
//
// What bounds it: the cached rows (512 bytes a key and head).  32 tokens that read 255 MB of rows together: 56 us and the merge 6, 4.6
// TB/s (the kernel it stands in for 119 us: it copied every row with a lane's own cp.async and spent two products on the weights).
// Calls that read few rows stay with that one (ROWS_DECODE_LEAST in ops/kernels.py).
//
// Every wait on an mbarrier is bounded (tcgen05.cuh).
#include <cfloat>

#include "tcgen05.cuh"

namespace {
using namespace tc;

constexpr int D = 128, CONSUMERS = 4, THREADS = 32 * (CONSUMERS + 1), RUN = 16, STAGES = 8, HEADS = 8;
constexpr int BOX_BYTES = RUN * 128, STAGE_BYTES = 4 * BOX_BYTES;  // two boxes of keys, two of values
static_assert(STAGES % CONSUMERS == 0, "every stage belongs to one consumer warp");
constexpr int JOIN_PITCH = D + 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 2 * STAGES * 8 + 16;
static_assert(CONSUMERS * HEADS * (JOIN_PITCH + 2) * 4 <= STAGES * STAGE_BYTES, "the warps' results take the ring's place");

struct DecodeArgs {
  const __nv_bfloat16 *q, *gate;
  const int32_t *table, *positions, *token_item;
  const float *bias, *sink;
  __nv_bfloat16* out;
  float* partial;
  long long ldg, ldo;
  int table_width, hq, hkv, page_shift, window, chunk, reach, keep_first, splits;
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

// status codes: 1 producer, 2 consumer
__global__ void __launch_bounds__(THREADS, 3)
attention_rows_decode_kernel(const __grid_constant__ CUtensorMap map_kv, const DecodeArgs args) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  volatile uint32_t* abort = reinterpret_cast<volatile uint32_t*>(empty + STAGES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  const int share = args.hq / args.hkv, split = blockIdx.y;
  const int t = blockIdx.x / args.hkv, g = blockIdx.x - t * args.hkv, h0 = g * share;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  const int p = args.positions[t];
  const int32_t* pages = args.table + (size_t)args.token_item[t] * args.table_width;
  int lo = (args.window > 0 && p - args.window + 1 > 0) ? p - args.window + 1 : 0;
  if (args.chunk > 0) lo = max(lo, p / args.chunk * args.chunk);
  int kept_runs = 0;  // kept first keys: one stretch from 0 while the window reaches them, else runs of their own in front
  if (args.keep_first > 0) {
    if (lo <= args.keep_first) lo = 0;
    else kept_runs = (args.keep_first + RUN - 1) / RUN;
  }
  const int first_run = lo / RUN, all = kept_runs + p / RUN - first_run + 1;
  const int per = (all + args.splits - 1) / args.splits, r0 = split * per, runs = max(0, min(per, all - r0));
  auto is_kept = [&](int i) { return r0 + i < kept_runs; };
  auto base_of = [&](int i) { return RUN * (is_kept(i) ? r0 + i : first_run + r0 + i - kept_runs); };

  float m = -FLT_MAX, l = 0.f;   // of head gr, in powers of two
  float o[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  if (warp == CONSUMERS) {
    int ids = 0;
    bool ok = true;
    for (int i = 0; ok && i < runs; ++i) {
      if ((i & 31) == 0) {  // page ids of the next 32 runs, one a lane
        const int ii = i + lane;
        ids = ii < runs ? __ldg(pages + (base_of(ii) >> args.page_shift)) : 0;
      }
      const int page = __shfl_sync(0xffffffffu, ids, i & 31), stage = i % STAGES;
      if (i >= STAGES) {
        ok = mbar_wait(&empty[stage], ((i / STAGES) - 1) & 1, abort, 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      if (lane == 0) {
        const int row = ((page * args.hkv + g) << args.page_shift) + (base_of(i) & ((1 << args.page_shift) - 1));
        mbar_expect_tx(&full[stage], (uint32_t)STAGE_BYTES);
#pragma unroll
        for (int b = 0; b < 4; ++b) tma_load_2d(smem + stage * STAGE_BYTES + b * BOX_BYTES, &map_kv, 64 * b, row, &full[stage]);
      }
      __syncwarp();
    }
  } else {
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
    bool ok = true;
    for (int i = warp; ok && i < runs; i += CONSUMERS) {
      const int stage = i % STAGES, key0 = base_of(i);
      const int from = is_kept(i) ? 0 : lo - key0, upto = (is_kept(i) ? args.keep_first : p + 1) - key0;  // rows that count
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
  }
  if (*abort) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies in flight must land before the memory changes hands
  }
  __syncthreads();  // every run has been used: the ring now carries the warps' results, [warp][head][D + 4 | m | l]
  float* join = reinterpret_cast<float*>(smem);
  constexpr int ROW = JOIN_PITCH + 2;
  if (warp < CONSUMERS) {
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    float* dst = join + (warp * HEADS + gr) * ROW;
#pragma unroll
    for (int j = 0; j < D / 8; ++j) *reinterpret_cast<float2*>(dst + 8 * j + 2 * tg) = make_float2(o[j][0] + o[j][2], o[j][1] + o[j][3]);
    if (tg == 0) {
      dst[JOIN_PITCH] = m;
      dst[JOIN_PITCH + 1] = l;
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < share * (D / 4); idx += THREADS) {
    const int row = idx / (D / 4), d = (idx % (D / 4)) * 4, h = h0 + row;
    const float* src = join + row * ROW;
    const bool whole = args.splits == 1;
    const float s2 = whole && args.sink ? args.sink[h] * PSB_LOG2E : -INFINITY;
    float top = s2;
#pragma unroll
    for (int w = 0; w < CONSUMERS; ++w) top = fmaxf(top, src[w * HEADS * ROW + JOIN_PITCH]);
    float sum = whole && args.sink ? exp2f(s2 - top) : 0.f, acc[4] = {};
#pragma unroll
    for (int w = 0; w < CONSUMERS; ++w) {
      const float* mine = src + w * HEADS * ROW;
      const float f = exp2f(mine[JOIN_PITCH] - top);  // (a warp without runs has a sum and a result of 0)
      sum = fmaf(f, mine[JOIN_PITCH + 1], sum);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = fmaf(f, mine[d + e], acc[e]);
    }
    if (whole) {
      const float by = args.out_scale / sum;
      const __nv_bfloat16* gate = args.gate ? args.gate + (size_t)t * args.ldg + (size_t)h * D + d : nullptr;
      __nv_bfloat16* dst = args.out + (size_t)t * args.ldo + (size_t)h * D + d;
#pragma unroll
      for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16_rn(acc[e] * (gate ? by / (1.f + expf(-__bfloat162float(gate[e]))) : by));
    } else {
      float* dst = args.partial + (((size_t)t * args.hq + h) * args.splits + split) * (D + 2);
      if (d == 0) {
        dst[0] = top == -INFINITY ? -FLT_MAX : fmaxf(top * 0.6931471805599453f, -FLT_MAX);
        dst[1] = sum;
      }
      *reinterpret_cast<float2*>(dst + 2 + d) = make_float2(acc[0], acc[1]);
      *reinterpret_cast<float2*>(dst + 4 + d) = make_float2(acc[2], acc[3]);
    }
  }
}

}  // namespace

// (hq, hkv, dim, vdim, page_size) -> 1 if the kernel takes them
PSB_API int psb_attention_rows_decode_supported(int hq, int hkv, int dim, int vdim, int page_size) {
  return hq >= 1 && hkv >= 1 && hq % hkv == 0 && hq / hkv <= HEADS && dim == D && vdim == D && page_size >= RUN && (page_size & (page_size - 1)) == 0 ? 1 : 0;
}

// () -> blocks an SM holds
PSB_API int psb_attention_rows_decode_blocks() { return 3; }

// Tokens one by one.  With several ``splits`` the shares are left in partial [T * hq, splits, 130] float32 and the caller joins them
// (psb_attention_rows_merge).
// (q, kv, num_pages, table, table_width, positions, token_item, bias, sink, out, T, hq, hkv, dim, vdim, page_size, window, chunk, reach,
//  scale, keep_first, partial, splits, gate, ldg, ldo, out_scale, softcap, stream)
PSB_API int psb_attention_rows_decode(const void* q, const void* kv, long long num_pages, const void* table, int table_width,
                                      const void* positions, const void* token_item, const void* bias, const void* sink, void* out, int T,
                                      int hq, int hkv, int dim, int vdim, int page_size, int window, int chunk, int reach, float scale,
                                      int keep_first, void* partial, int splits, const void* gate, long long ldg, long long ldo,
                                      float out_scale, float softcap, cudaStream_t stream) {
  if (!psb_attention_rows_decode_supported(hq, hkv, dim, vdim, page_size))
    PSB_REFUSE("attention_rows_decode: %d heads over %d of %d and %d in pages of %d are not taken", hq, hkv, dim, vdim, page_size);
  if (ldo < (long long)hq * D || (gate && ldg < (long long)hq * D) || softcap < 0.f) PSB_REFUSE("attention_rows_decode: bad output or gate rows, or a negative cap");
  if (keep_first < 0 || (keep_first > 0 && (window < 1 || chunk > 0))) PSB_REFUSE("attention_rows_decode: kept first keys go with a window and no chunk mask");
  if (table_width < 1 || window < 0 || chunk < 0 || (bias && reach < 1) || num_pages < 1) PSB_REFUSE("attention_rows_decode: bad arguments");
  if (splits < 1 || splits > 65535 || (splits > 1 && !partial)) PSB_REFUSE("attention_rows_decode: %d shares, or their scratch is missing", splits);
  if (((uintptr_t)kv & 15) || ((uintptr_t)q & 3) || ((uintptr_t)partial & 7)) PSB_REFUSE("attention_rows_decode: operands are not aligned");
  if (T <= 0) return 0;
  const long long kv_rows = num_pages * hkv * page_size;
  if (kv_rows > 0x7fffffffLL || (long long)T * hkv > 0x7fffffffLL) PSB_REFUSE("attention_rows_decode: too many cache rows or tokens");
  DecodeArgs args{};
  args.q = (const __nv_bfloat16*)q; args.gate = (const __nv_bfloat16*)gate; args.table = (const int32_t*)table;
  args.positions = (const int32_t*)positions; args.token_item = (const int32_t*)token_item; args.bias = (const float*)bias;
  args.sink = (const float*)sink; args.out = (__nv_bfloat16*)out; args.partial = (float*)partial; args.ldg = ldg; args.ldo = ldo;
  args.table_width = table_width; args.hq = hq; args.hkv = hkv; args.window = window; args.chunk = chunk; args.reach = reach;
  args.keep_first = keep_first; args.splits = splits; args.scale = scale; args.softcap = softcap; args.out_scale = out_scale;
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
  psb_launch(attention_rows_decode_kernel, dim3((unsigned)(T * hkv), splits), dim3(THREADS), (size_t)SMEM_BYTES, stream, map, args);
  PSB_LAUNCH_CHECK("attention_rows_decode");
  return 0;
}

// 0 while no bounded wait of this kernel has ever run out on the current device; reading it synchronises with the device.
PSB_API int psb_attention_rows_decode_status() { return tc::read_status(); }
