// Both delta rules over steps of single tokens, everything in one kernel: the short convolution and SiLU of the token's channels, its unit vectors, write
// strength and decay, the state's turn, the read-out (the gated rule's normed and gated) and the convolution inputs the slot keeps (delta_rule.cu says
// what each of these is).
//
// A CTA per request and head: the copy engine brings the head's state into shared memory (one copy, under way while the convolution is made), a warp
// takes every eighth of its rows and a lane four neighbouring columns, and the copy engine takes the new state back.  With S the state (times its channels'
// decays, where they have their own) and dec the head's decay (or 1)
//     u = beta (v - dec S^T k),   o = dec S^T q + (q.k) u,   S <- dec S + k u^T,
// so both sums over S are taken from one reading.  The heads of a group are a cluster: each makes the group's queries and keys for itself from
// the slot's convolution inputs, which the cluster's first CTA brings up to date when all have read them.
//
// Bound by memory from some sixteen requests on (64 KB read and written a request and head, three CTAs an SM: 32 requests of 32 heads 4.2 TB/s); below, by the
// launch and the chain of its steps.  On the device, us a call, kernels for preparing, the products of neighbouring tokens, the rule and the finish
// before, and this one: the gated rule, 16 heads, 4, 16 and 32 requests 24, 33, 46 and 8.5, 13, 20; 32 heads 38, 58, 89 and 11, 20, 32; a decay per channel 21, 28, 38 and
// 9, 13, 20; 33, 50, 72 and 12, 20, 32.  With the state in registers (two CTAs an SM) 32 heads took 10, 20, 37 and 13, 24, 48.
#include "delta_common.cuh"
#include "tcgen05.cuh"

namespace {
using namespace delta;

constexpr int WIDEST = 128, WARPS = 8, THREADS = 32 * WARPS, ROWS = WIDEST / WARPS;  // rows of the state a warp takes
constexpr int MAX_CLUSTER = 8;

struct SingleArgs {
  const float *ba, *taps, *a_log, *dt_bias, *decay, *gain;
  float* state;
  const int32_t *positions, *item_start, *slots;
  void* out;  // gated: [T, H vdim] of the compute type; a decay per channel: float32 [T, H, vdim]
  long long P, slot_floats;
  int beta_at, G, H, dim, vdim, K, num_slots;
  float eps;
  int* gives_up;  // not null: the wait gives up at once and says so there
};

template <typename T, bool CHANNEL>
__global__ void __launch_bounds__(THREADS, 3)
delta_single_kernel(const T* __restrict__ proj, const SingleArgs a) {
  extern __shared__ __align__(128) float held[];  // the state [dim][vdim]
  __shared__ float x[3 * WIDEST];  // queries, keys, values
  __shared__ float decays[CHANNEL ? WIDEST : 1];
  __shared__ uint64_t arrived;
  __shared__ uint32_t abort;
  __shared__ __align__(16) float part[WARPS][2][WIDEST], us[WIDEST];
  __shared__ float sums[3], squares[WIDEST / 32];
  const int h = blockIdx.y, each = a.H / a.G, g = h / each, dim = a.dim, vdim = a.vdim, K = a.K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int C = 2 * a.G * dim + a.H * vdim;
  pdl_trigger();
  pdl_wait();
  const int t = a.item_start[blockIdx.x];
  if (a.item_start[blockIdx.x + 1] != t + 1) return;  // (the same for the whole cluster)
  int slot = a.slots[blockIdx.x];
  slot = slot < 0 ? 0 : (slot >= a.num_slots ? a.num_slots - 1 : slot);
  float* base = a.state + (size_t)slot * a.slot_floats;
  float* S = base + (size_t)(K - 1) * C + (size_t)h * dim * vdim;
  const bool mine = 4 * lane < vdim;
  const uint32_t bytes = (uint32_t)(dim * vdim) * 4u;
  if (threadIdx.x == 0) {
    abort = 0;
    tc::mbar_init(&arrived, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_expect_tx(&arrived, bytes);
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::smem_u32(held)), "l"(S), "r"(bytes), "r"(tc::smem_u32(&arrived)) : "memory");
  }
  // channel j of queries, keys and values, one after the other: its column of the projection
  auto column = [&](int j) { return j < dim ? g * dim + j : j < 2 * dim ? (a.G + g) * dim + j - dim : 2 * a.G * dim + h * vdim + j - 2 * dim; };
  const int p = a.positions[t], channels = 2 * dim + vdim;
  for (int j = threadIdx.x; j < channels; j += THREADS) {
    const int c = column(j);
    float in[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K) break;
      if (k == K - 1) in[k] = to_float<T>(proj[(size_t)t * a.P + c]);
      else in[k] = p - (K - 1) + k >= 0 ? base[(size_t)k * C + c] : 0.f;
    }
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K) break;
      acc = fmaf(a.taps[(size_t)c * K + k], in[k], acc);
    }
    x[j] = siluf_(acc);
  }
  if constexpr (CHANNEL) {
    if (threadIdx.x < dim) decays[threadIdx.x] = a.decay[((size_t)t * a.H + h) * dim + threadIdx.x];
  }
  float beta, dec = 1.f;
  if (a.ba) {
    beta = sigmoidf_(a.ba[(size_t)t * 2 * a.H + h]);
    dec = expf(-expf(a.a_log[h]) * softplusf_(a.ba[(size_t)t * 2 * a.H + a.H + h] + a.dt_bias[h]));
  } else {
    beta = sigmoidf_(to_float<T>(proj[(size_t)t * a.P + a.beta_at + h]));
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // this CTA has read the slot's convolution inputs
  if (warp < 3) {  // q.q, k.k, q.k
    const float *l = x + (warp == 1 ? dim : 0), *r = x + (warp == 0 ? 0 : dim);
    float sum = 0.f;
    for (int d = lane; d < dim; d += 32) sum = fmaf(l[d], r[d], sum);
    sum = warp_sum(sum);
    if (lane == 0) sums[warp] = sum;
  }
  __syncthreads();
  const float fq = unit_factor(sums[0], dim), fk = unit_factor(sums[1], 1);
  float4* const rows = reinterpret_cast<float4*>(held) + lane;  // row d: (vdim / 4) d further
  // A wait that gives up (never seen) leaves the head's state, the slot's inputs that this CTA keeps and the result as they were, but for
  // the copy, which is waited for once more: it must not land in another CTA's shared memory.
  if (!tc::mbar_wait_limited(&arrived, 0, &abort, 1, a.gives_up ? 0 : tc::SPIN_LIMIT, a.gives_up ? a.gives_up : &tc::g_status))
    for (uint32_t spin = 0; spin < tc::SPIN_LIMIT && !tc::mbar_try_wait(&arrived, 0); ++spin) {}
  const bool fine = __syncthreads_and(abort == 0);
  {
    float4 sk = make_float4(0.f, 0.f, 0.f, 0.f), sq = sk;
#pragma unroll 4
    for (int d = warp; d < dim; d += WARPS) {
      if (!mine) continue;
      const float f = CHANNEL ? decays[d] : 1.f, q = x[d] * fq, k = x[dim + d] * fk;
      float4 s = rows[d * (vdim / 4)];
      if constexpr (CHANNEL) s.x *= f, s.y *= f, s.z *= f, s.w *= f;
      sk.x = fmaf(k, s.x, sk.x); sk.y = fmaf(k, s.y, sk.y); sk.z = fmaf(k, s.z, sk.z); sk.w = fmaf(k, s.w, sk.w);
      sq.x = fmaf(q, s.x, sq.x); sq.y = fmaf(q, s.y, sq.y); sq.z = fmaf(q, s.z, sq.z); sq.w = fmaf(q, s.w, sq.w);
    }
    *reinterpret_cast<float4*>(&part[warp][0][4 * lane]) = sk;
    *reinterpret_cast<float4*>(&part[warp][1][4 * lane]) = sq;
  }
  __syncthreads();
  float o = 0.f;
  if (threadIdx.x < WIDEST) {  // a column a thread
    const int c = threadIdx.x;
    float sk[WARPS], sq[WARPS];
#pragma unroll
    for (int w = 0; w < WARPS; ++w) sk[w] = part[w][0][c], sq[w] = part[w][1][c];
#pragma unroll
    for (int m = WARPS / 2; m > 0; m >>= 1)
#pragma unroll
      for (int w = 0; w < m; ++w) sk[w] += sk[w + m], sq[w] += sq[w + m];
    const float u = c < vdim ? beta * (x[2 * dim + c] - dec * sk[0]) : 0.f;
    us[c] = u;
    o = fmaf(sums[2] * fq * fk, u, dec * sq[0]);
    if constexpr (CHANNEL) {
      if (fine && c < vdim) static_cast<float*>(a.out)[((size_t)t * a.H + h) * vdim + c] = o;
    } else {
      const float ss = warp_sum(c < vdim ? o * o : 0.f);
      if (lane == 0) squares[warp] = ss;
    }
  }
  __syncthreads();
  const float4 u = *reinterpret_cast<const float4*>(us + 4 * lane);
#pragma unroll 4
  for (int d = warp; d < dim; d += WARPS) {
    if (!mine) continue;
    const float k = x[dim + d] * fk, f = CHANNEL ? decays[d] : dec;
    float4 s = rows[d * (vdim / 4)];
    s.x = fmaf(k, u.x, f * s.x); s.y = fmaf(k, u.y, f * s.y); s.z = fmaf(k, u.z, f * s.z); s.w = fmaf(k, u.w, f * s.w);
    rows[d * (vdim / 4)] = s;
  }
  tc::fence_async_smem();
  __syncthreads();
  if (threadIdx.x == 0 && fine)
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;"
                 ::"l"(S), "r"(tc::smem_u32(held)), "r"(bytes) : "memory");
  if constexpr (!CHANNEL) {
    if (fine && threadIdx.x < vdim) {
      const int c = threadIdx.x;
      const float inv = 1.f / sqrtf(((squares[0] + squares[1]) + (squares[2] + squares[3])) / (float)vdim + a.eps);
      const size_t at = (size_t)h * vdim + c;
      const float gate = to_float<T>(proj[(size_t)t * a.P + C + at]);
      static_cast<T*>(a.out)[(size_t)t * a.H * vdim + at] = from_float<T>(o * inv * a.gain[c] * siluf_(gate));
    }
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  // the slot's convolution inputs move up by one; a group's queries and keys by its first head
  for (int j = (h % each == 0 ? 0 : 2 * dim) + threadIdx.x; fine && j < channels; j += THREADS) {
    const int c = column(j);
    float keep[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K - 1) break;
      keep[k] = k == K - 2 ? to_float<T>(proj[(size_t)t * a.P + c]) : base[(size_t)(k + 1) * C + c];
    }
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K - 1) break;
      base[(size_t)k * C + c] = keep[k];
    }
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // (written: what follows this kernel reads it)
}

}  // namespace

// (G, H, dim, vdim, K) -> 1 if psb_delta_single is built for the sizes
PSB_API int psb_delta_single_supported(int G, int H, int dim, int vdim, int K) {
  if (G < 1 || H < 1 || H % G || H / G > MAX_CLUSTER || H > 65535 || dim < 1 || dim > WIDEST || vdim < 4 || vdim > WIDEST || vdim % 4 || K < 1 || K > MAX_TAPS) return 0;
  const long long C = 2LL * G * dim + (long long)H * vdim;
  return (K - 1) * C % 4 == 0 ? 1 : 0;
}

// Requests of one token each; others are left untouched.  The gated rule (gain given): proj of either type [T, ld] with q | k | v | gate in its first columns, ba
// float32 [T, 2 H], out [T, H vdim] of proj's type.  The other: decay float32 [T, H, dim], the write strengths in proj's columns from beta_at on,
// out float32 [T, H, vdim].  gives_up (an int32 on the device, null as a rule): the wait for the state gives up without a poll and leaves its code there.
// (proj, dtype, ld, beta_at, ba, decay, taps, a_log, dt_bias, state, positions, item_start, slots, gain, out, items, G, H, dim, vdim, K, num_slots,
//  slot_floats, eps, gives_up, stream)
PSB_API int psb_delta_single(const void* proj, int dtype, long long ld, int beta_at, const void* ba, const void* decay, const void* taps, const void* a_log,
                             const void* dt_bias, void* state, const void* positions, const void* item_start, const void* slots, const void* gain, void* out,
                             int items, int G, int H, int dim, int vdim, int K, int num_slots, long long slot_floats, float eps, void* gives_up, cudaStream_t stream) {
  if (!psb_delta_single_supported(G, H, dim, vdim, K)) PSB_REFUSE("delta_single: sizes G=%d H=%d dim=%d vdim=%d K=%d are not built", G, H, dim, vdim, K);
  const long long C = 2LL * G * dim + (long long)H * vdim;
  const bool gated = gain != nullptr;
  if (gated ? !ba || !a_log || !dt_bias || decay || ld < C + (long long)H * vdim : !decay || ba || beta_at < C || ld < (long long)beta_at + H)
    PSB_REFUSE("delta_single: the gates, decays or the row of %lld numbers do not fit the sizes", ld);
  if (num_slots < 1 || slot_floats != (K - 1) * C + (long long)H * dim * vdim || slot_floats % 4) PSB_REFUSE("delta_single: a slot of %lld numbers does not fit the sizes", slot_floats);
  if ((uintptr_t)state & 15) PSB_REFUSE("delta_single: the state must be 16-byte aligned");
  if (items <= 0) return 0;
  SingleArgs args{};
  args.ba = (const float*)ba; args.taps = (const float*)taps; args.a_log = (const float*)a_log; args.dt_bias = (const float*)dt_bias;
  args.decay = (const float*)decay; args.gain = (const float*)gain; args.state = (float*)state; args.positions = (const int32_t*)positions;
  args.item_start = (const int32_t*)item_start; args.slots = (const int32_t*)slots; args.out = out; args.P = ld; args.slot_floats = slot_floats;
  args.beta_at = beta_at; args.G = G; args.H = H; args.dim = dim; args.vdim = vdim; args.K = K; args.num_slots = num_slots; args.eps = eps; args.gives_up = (int*)gives_up;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)items, (unsigned)H);
  cfg.blockDim = dim3(THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
  attr[0].val.clusterDim.y = (unsigned)(H / G);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (psb_pdl_enabled) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cfg.dynamicSmemBytes = (size_t)dim * vdim * 4;
  PSB_DISPATCH_DTYPE(dtype, T_, {
    auto kernel = gated ? delta_single_kernel<T_, false> : delta_single_kernel<T_, true>;
    static PsbPerDevice configured[2];
    if (!configured[gated].get()) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WIDEST * WIDEST * 4) != cudaSuccess)
        PSB_REFUSE("delta_single: cannot raise the shared-memory limit");
      configured[gated].set();
    }
    cudaLaunchKernelEx(&cfg, kernel, (const T_*)proj, (const SingleArgs)args);
  });
  PSB_LAUNCH_CHECK("delta_single");
  return 0;
}

// 0 while no bounded wait of this kernel has ever run out on the current device; reading it synchronises with the device.
PSB_API int psb_delta_single_status() { return tc::read_status(); }
