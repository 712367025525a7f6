// What the recurrences that work 32 tokens at a time share (delta_chunks.cu, linear_attention_chunks.cu): float32 products on the tensor cores in three
// bfloat16 terms a number, how their operands lie in a chunk's record, and the products of a chunk's queries and keys with a decay per channel.
//
// A float32 number is the sum of three bfloat16 numbers, to its last bit, and six of the nine products of terms count.  Products of first terms are
// exact, and their sums leave the tensor cores every sixteen terms and are added up in float32 with rounding to nearest (the instruction cuts its sums
// off); the rest is smaller by 2^8.  As many terms as float32's own accuracy takes in TF32 (six products of eleven bits) take twice as long, and
// fma.rn.f32x2 as long as these, but for what shared memory has to hand to the registers (16 bytes a lane: four cycles a warp).
#pragma once
#include "delta_common.cuh"
#include "portions.cuh"

namespace chunks {
using delta::copy_async16_or_zero;

__device__ __forceinline__ bool is_finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// A running product of decays with what its roundings lose carried along, rounded once where it is read.
struct Product {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float a) {
    const float p = hi * a;
    lo = fmaf(lo, a, fmaf(hi, a, -p));
    hi = p;
  }
  __device__ __forceinline__ float value() const { return hi + lo; }
};

constexpr int CHUNK = 32;
constexpr int RP = 128;                            // keys are filled up to so many numbers
constexpr int KP = RP + 4, TP = CHUNK + 4;         // pitches in shared memory: 16-byte reads of eight neighbouring rows meet every bank once
constexpr int CHUNK_THREADS = 128;

// What the tensor cores take lies in a record as their right operands' fragments, a lane's four words of a term together (16 channels or tokens by 8,
// see mma_bf16): 128 words a term, three terms a unit.
constexpr int TERM = 128, UNIT = 3 * TERM;

// x and y as three terms each, packed in pairs (x in the low half)
struct Terms {
  uint32_t v[3];
};
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&p);
}
__device__ __forceinline__ Terms split3(float x, float y) {
  Terms t;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t.v[i] = pack_bf16(x, y);
    x -= __uint_as_float(t.v[i] << 16);
    y -= __uint_as_float(t.v[i] & 0xffff0000u);
  }
  return t;
}

// D = A B + C: A [16][16] (lane: rows gr and gr + 8, two neighbours at 2 tg, then at 2 tg + 8), B [16][8] (column gr, rows as A's), C and D
// [16][8] (rows gr and gr + 8, columns 2 tg and 2 tg + 1), with gr = lane / 4 and tg = lane % 4
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
struct Left {  // a left operand's three terms
  uint32_t v[3][4];
  __device__ __forceinline__ void put(int r, const Terms& t) {
#pragma unroll
    for (int p = 0; p < 3; ++p) v[p][r] = t.v[p];
  }
};
struct Right {
  uint32_t v[3][2];
  __device__ __forceinline__ void put(int r, const Terms& t) {
#pragma unroll
    for (int p = 0; p < 3; ++p) v[p][r] = t.v[p];
  }
};
// One step of sixteen terms of N sums: sum += first terms' products, rounded to nearest; small += the others that count, the smallest first.  The
// sums' instructions take turns: each of one sum waits for the last of it.
template <int N>
__device__ __forceinline__ void step(float (&sum)[N][4], float (&small)[N][4], const Left& a, const Right (&b)[N]) {
  const float zero[4] = {};
  float d[N][4];
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a.v[2], b[n].v[0][0], b[n].v[0][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(d[n], a.v[0], b[n].v[0][0], b[n].v[0][1], zero);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a.v[0], b[n].v[2][0], b[n].v[2][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a.v[1], b[n].v[1][0], b[n].v[1][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a.v[1], b[n].v[0][0], b[n].v[0][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) mma_bf16(small[n], a.v[0], b[n].v[1][0], b[n].v[1][1], small[n]);
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[n][e] += d[n][e];
}

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

__device__ __forceinline__ void put_terms(float* at, const Terms (&t)[4]) {
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(at + p * TERM) = make_uint4(t[0].v[p], t[1].v[p], t[2].v[p], t[3].v[p]);
}
// The same for two left operands with their own right ones (b[k][n]), sums apart.
__device__ __forceinline__ void step_halves(float (&sum)[2][2][4], float (&small)[2][2][4], const Left (&a)[2], const Right (&b)[2][2]) {
  const float zero[4] = {};
  auto round = [&](int p, int q) {
#pragma unroll
    for (int i = 0; i < 4; ++i) mma_bf16(small[i >> 1][i & 1], a[i >> 1].v[p], b[i >> 1][i & 1].v[q][0], b[i >> 1][i & 1].v[q][1], small[i >> 1][i & 1]);
  };
  round(2, 0);
#pragma unroll
  for (int i = 0; i < 4; ++i) mma_bf16(sum[i >> 1][i & 1], a[i >> 1].v[0], b[i >> 1][i & 1].v[0][0], b[i >> 1][i & 1].v[0][1], zero);
  round(0, 2);
  round(1, 1);
  round(1, 0);
  round(0, 1);
}

// 32 rows of numbers [32][KP] (times a number a row) as right operands' columns: per 16 of their numbers, ``apart`` units from the last, two units
template <typename Factor>
__device__ __forceinline__ void put_rows(const float* rows, float* __restrict__ at, int apart, int thread, int threads, Factor factor) {
#pragma unroll 2
  for (int i = thread; i < RP / 16 * 2 * 32; i += threads) {
    const int lane = i & 31, pair = (i >> 5) & 1, w = i >> 6, gr = lane >> 2, tg = lane & 3;
    Terms t[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = 8 * (2 * pair + (r >> 1)) + gr;
      const float f = factor(row);
      const float2 v = *reinterpret_cast<const float2*>(rows + row * KP + 16 * w + 8 * (r & 1) + 2 * tg);
      t[r] = split3(v.x * f, v.y * f);
    }
    put_terms(at + (w * apart + pair) * UNIT + 4 * lane, t);
  }
}
// 32 tokens' keys [32][KP], times a number a token, as K r
template <typename Factor>
__device__ __forceinline__ void put_keys(const float* rows, float* __restrict__ at, int thread, int threads, Factor factor) {
#pragma unroll 2
  for (int i = thread; i < RP / 16 * 2 * 32; i += threads) {
    const int lane = i & 31, gr = lane >> 2, tg = lane & 3, eight = i >> 5;
    Terms t[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int j = 8 * r + 2 * tg;
      const float* k = rows + j * KP + 8 * eight + gr;
      t[r] = split3(k[0] * factor(j), k[KP] * factor(j + 1));
    }
    put_terms(at + eight * UNIT + 4 * lane, t);
  }
}
// B [32][TP]
__device__ __forceinline__ void put_b(const float (*bs)[TP], float* __restrict__ at, int thread, int threads) {
#pragma unroll 2
  for (int i = thread; i < CHUNK / 8 * 32; i += threads) {
    const int lane = i & 31, row = 8 * (i >> 5) + (lane >> 2), tg = lane & 3;
    Terms t[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) t[r] = split3(bs[row][8 * r + 2 * tg], bs[row][8 * r + 2 * tg + 1]);
    put_terms(at + (i >> 5) * UNIT + 4 * lane, t);
  }
}
// Fragments of rows in shared memory: 16 rows from ``rows`` and 16 of their numbers as a left operand; eight rows and 16 numbers as a right one.
__device__ __forceinline__ Left left_rows(const float* rows, int pitch, int gr, int tg) {
  Left a;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float* at = rows + (gr + 8 * (r & 1)) * pitch + 8 * (r >> 1) + 2 * tg;
    a.put(r, split3(at[0], at[1]));
  }
  return a;
}
__device__ __forceinline__ Right right_rows(const float* rows, int pitch, int gr, int tg) {
  Right b;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float* at = rows + gr * pitch + 8 * r + 2 * tg;
    b.put(r, split3(at[0], at[1]));
  }
  return b;
}
// 32 rows of ``src`` (rows C numbers apart, ``dim`` numbers, zeros beyond them and beyond n rows)
__device__ __forceinline__ void bring_rows(float* dst, const float* src, long long C, int n, int dim, bool wide) {
  if (wide) {
    for (int i = threadIdx.x; i < CHUNK * RP / 4; i += CHUNK_THREADS) {
      const int t = i / (RP / 4), d = (i % (RP / 4)) * 4;
      const bool there = t < n && d < dim;
      copy_async16_or_zero(dst + t * KP + d, src + (there ? (size_t)t * C + d : 0), there);
    }
  } else {
    for (int i = threadIdx.x; i < CHUNK * RP; i += CHUNK_THREADS) {
      const int t = i / RP, d = i % RP;
      dst[t * KP + d] = t < n && d < dim ? src[(size_t)t * C + d] : 0.f;
    }
  }
}

__device__ __forceinline__ float term(uint32_t word, int half) { return __uint_as_float(half ? word & 0xffff0000u : word << 16); }

constexpr int HALF = CHUNK / 2;
// A_ij = sum_d k_i k_j g_(j+1) .. g_i (j < i; WITH_A) and B_ij with q_i (j <= i) for 32 tokens' keys, queries and decays [32][KP] each, where the decays are per
// channel, in halves of 16 tokens.  On the diagonal: a running product a column (COMPENSATED: with what its roundings lose); ends with the warp's own.
template <bool WITH_A, bool COMPENSATED>
__device__ __forceinline__ void products_on_diagonal(const float* ks, const float* qs, const float* gs, float (*as)[TP], float (*bs)[TP], int warp, int lane) {
  // on the diagonal: a warp takes two times four columns of a half, a lane four channels
#pragma unroll 1
  for (int turn = 0; turn < 2; ++turn) {
    const int base = HALF * (warp & 1), j0 = 4 * (turn ? 3 - (warp >> 1) : (warp >> 1));  // (a long run and a short one)
    Product run[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 key = *reinterpret_cast<const float4*>(ks + (base + j0 + j) * KP + 4 * lane);
      run[j][0].hi = key.x, run[j][1].hi = key.y, run[j][2].hi = key.z, run[j][3].hi = key.w;
    }
#pragma unroll 2
    for (int i = j0; i < HALF; ++i) {
      const int at = (base + i) * KP + 4 * lane;
      const float4 f = *reinterpret_cast<const float4*>(gs + at), k = *reinterpret_cast<const float4*>((WITH_A ? ks : qs) + at), q = *reinterpret_cast<const float4*>(qs + at);
      const float fs[4] = {f.x, f.y, f.z, f.w};
      float v[WITH_A ? 8 : 4];  // A's and B's row i, columns j0 .. j0 + 3
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (i > j0 + j) {
            if constexpr (COMPENSATED) run[j][e].times(fs[e]);
            else run[j][e].hi *= fs[e];
          }
          x[e] = COMPENSATED ? run[j][e].value() : run[j][e].hi;
        }
        if constexpr (WITH_A) v[j] = fmaf(k.x, x[0], k.y * x[1]) + fmaf(k.z, x[2], k.w * x[3]);
        v[(WITH_A ? 4 : 0) + j] = fmaf(q.x, x[0], q.y * x[1]) + fmaf(q.z, x[2], q.w * x[3]);
      }
      // the sums over the warp: lane's bits (4, then) 3 and 2, or 4 and 3, choose which of them it ends up with
      constexpr int FIRST = WITH_A ? 4 : 2;
#pragma unroll
      for (int m = FIRST, off = 16; m > 0; m >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int e = 0; e < m; ++e) v[e] = (up ? v[e + m] : v[e]) + __shfl_xor_sync(0xffffffffu, up ? v[e] : v[e + m], off);
      }
#pragma unroll
      for (int off = WITH_A ? 2 : 4; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
      const int j = j0 + (WITH_A ? (lane >> 2) & 3 : lane >> 3);
      if ((lane & (WITH_A ? 3 : 7)) == 0) {
        if (!WITH_A || (lane & 16)) bs[base + i][base + j] = j <= i ? v[0] : 0.f;
        else as[base + i][base + j] = j < i ? v[0] : 0.f;
      }
    }
    // above the diagonal: this warp's columns in the rows before j0, and (those of the second half) in the first half's
    auto clear = [&](int i) {
      bs[i][base + j0 + (lane & 3)] = 0.f;
      if constexpr (WITH_A) as[i][base + j0 + (lane & 3)] = 0.f;
    };
    for (int i = lane >> 2; i < j0; i += 8) clear(base + i);
    if (base)
      for (int i = lane >> 2; i < HALF; i += 8) clear(i);
  }
}
// Rows m HALF of ``left`` with rows 8 c of ``right``, N channels: sixteen at a time, then in pairs (a single chain over the 128 loses most of a read-out).
template <int ROWS, int N>
__device__ __forceinline__ void sums_in_pairs(const float* left, const float* right, float (&out)[ROWS][2]) {
  if constexpr (N == 16) {
    uint64_t acc[ROWS][2] = {};
#pragma unroll
    for (int e = 0; e < N; e += 4) {
      Pairs a[ROWS], b[2];
#pragma unroll
      for (int m = 0; m < ROWS; ++m) a[m] = load4(left + HALF * m * KP + e);
#pragma unroll
      for (int c = 0; c < 2; ++c) b[c] = load4(right + 8 * c * KP + e);
#pragma unroll
      for (int m = 0; m < ROWS; ++m)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          fma2(acc[m][c], a[m].lo, b[c].lo);
          fma2(acc[m][c], a[m].hi, b[c].hi);
        }
    }
#pragma unroll
    for (int m = 0; m < ROWS; ++m)
#pragma unroll
      for (int c = 0; c < 2; ++c) out[m][c] = both(acc[m][c]);
  } else {
    float half[ROWS][2];
    sums_in_pairs<ROWS, N / 2>(left, right, out);
    sums_in_pairs<ROWS, N / 2>(left + N / 2, right + N / 2, half);
#pragma unroll
    for (int m = 0; m < ROWS; ++m)
#pragma unroll
      for (int c = 0; c < 2; ++c) out[m][c] += half[m][c];
  }
}
// Behind the diagonal: queries and keys of the second half (rows of ``left``: its keys, WITH_A, then its queries) times the decays from its start, and keys of
// the first (``right``) times those to its end.
template <bool WITH_A>
__device__ __forceinline__ void products_behind(const float* left, const float* right, float (*as)[TP], float (*bs)[TP]) {
  const int ri = threadIdx.x >> 3, cj = threadIdx.x & 7;
  constexpr int ROWS = WITH_A ? 2 : 1;
  float total[ROWS][2];
  sums_in_pairs<ROWS, RP>(left + ri * KP, right + cj * KP, total);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if constexpr (WITH_A) as[HALF + ri][cj + 8 * c] = total[0][c];
    bs[HALF + ri][cj + 8 * c] = total[ROWS - 1][c];
  }
}

// ---- the chain that walks a portion's chunks
constexpr int WORKERS = 256, READERS = 128, CHAIN_THREADS = WORKERS + READERS;
static_assert(WORKERS / 32 == RP / 16 && READERS / 32 == CHUNK / 8, "a worker warp per 16 channels, a reader warp per eight tokens");

}  // namespace chunks
