// The general path: forward and backward flash-attention blocks with fp32 accuracy. It serves (1) fp32 inputs, with or
// without a dense additive bias (the reference's bias_func protocol, lv_xattn/attn.py:386-389: S = scale * q.k + bias,
// bias [B, 1 or H, Sq, Skv] fp32), and (2) the backward of fp16 inputs with a bias.
//
// Every product runs on the tensor core as three tf32 products (mma.sync.m16n8k8): an operand x is taken as hi + lo, hi =
// x rounded to tf32's 11 bits, lo = the next 11, and a*b as hi*lo + lo*hi + hi*hi; what is dropped is 2^-22 of a
// product. The tensor core only ever sums the three products of one k-step of eight, onto zero; that sum is added to the
// fp32 accumulator by the FMA pipe, so the long sums keep fp32's own rounding (and take a sixteenth of the additions that a
// plain FMA loop takes: the error against 64 bits at 512 x 8,192 is 5.9e-7 where an FMA loop's was 1.1e-6). 16-bit
// inputs are exact in tf32 and take no lo.
// Measured at 32 heads, 512 x 8,192: forward 2.47 -> 1.34 ms, backward 5.84 -> 3.65 ms.
// What bounds it: mma.sync runs tf32 at 484 FMA/clk/SM here, i.e. 161 a clock for three products, against 128 (with
// packed arithmetic, 104 without) on the FMA pipe, where moreover every operand of a register tile has to come through
// shared memory at 4 bytes a lane and clock: the FMA kernels that this replaces sat at 48. tcgen05 is not used: it takes
// its operands from shared memory, where hi and lo of all five tiles of the backward do not fit, and MN-major 32-bit tiles
// only in a swizzle of their own; fragments in registers are split after they have been read.
// Infinities, NaN and values up to the largest float come out where a plain sum has them: hi is kept finite, and an
// infinity goes into lo. (Only an infinity times a value of 4,096 or more may give NaN for infinity: hi times the other's lo
// can then overflow with the other sign.)
//
// Fragment layout (lane = 4*g + t): A is rows g, g+8 by k = t, t+4; B is k = t, t+4 by column g; C is rows g, g+8 by columns
// 2t, 2t+1. Where a C tile becomes an A operand (P, dS) the k axis is taken in the order 2t, 2t+1 instead, for A and B
// alike: a thread's own C values are then its A fragment. Rows of the 128-wide tiles are 132 floats apart, which makes
// both ways of reading a B fragment free of bank conflicts (4g+t, and 8t+g with k = 2t).
#include "lvx_internal.h"
#include "sm100_prims.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>
#include <type_traits>

namespace lvx {

constexpr int GT_LD = 132;                 // row stride of a [rows][128] tile (floats)
constexpr int GT_LDP = 68;                 // row stride of a [64][64] P / dS tile
constexpr int GT_TILE = 64 * GT_LD;
constexpr int GT_PTILE = 64 * GT_LDP;

__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }
__device__ __forceinline__ void from_f32(float* p, float x) { *p = x; }
__device__ __forceinline__ void from_f32(__half* p, float x) { *p = __float2half_rn(x); }

// Rows [row0, row0 + nrows_tile) of a dense [nrows, 128] matrix into a padded fp32 tile; rows past nrows are zero. fp32
// rows are copied asynchronously (the caller commits and waits), 16-bit ones are converted on the way.
template <typename T>
__device__ __forceinline__ void load_rows(float* dst, const T* src, int row0, int nrows, int tile_rows, int tid) {
  if constexpr (sizeof(T) == 4) {
    for (int idx = tid; idx < tile_rows * 32; idx += 256) {
      const int r = idx >> 5, c = (idx & 31) * 4, gr = row0 + r;
      const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst + r * GT_LD + c));
      const T* s = src + size_t(min(gr, nrows - 1)) * 128 + c;
      const int bytes = gr < nrows ? 16 : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(s), "r"(bytes) : "memory");
    }
  } else {
    for (int idx = tid; idx < tile_rows * 128; idx += 256) {
      const int r = idx >> 7, c = idx & 127, gr = row0 + r;
      dst[r * GT_LD + c] = gr < nrows ? to_f32(src[size_t(gr) * 128 + c]) : 0.f;
    }
  }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Values beyond tf32's largest (infinities, and what rounding has taken to one) and NaN become that largest, with their sign:
// one instruction.
__device__ __forceinline__ uint32_t clamp_tf32(uint32_t x) {
  float r;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(__uint_as_float(x)), "f"(__uint_as_float(0x7f7fe000u)));
  return __float_as_uint(r);
}
// x = hi + lo (+ at most 2^-22 of x), both in tf32: hi rounded, so that what lo cuts off has a sign of its own. Near the
// largest float rounding gives infinity, and lo the other one; every product with such a value, or with an infinite one,
// is then NaN. With CLAMP hi is always finite: near the largest float lo takes the rest, and for an infinite x (or NaN) lo
// is x, so that lo*b is what x*b is and nothing of the other sign or NaN is added to it.
// A CTA walks over its tiles without CLAMP first, and again with it where NaN came out: of 512 x 8,192, forward and
// backward, that takes 0.7 %, against 5.7 % with the clamp in every split and 4 % with a look at the values of every tile
// as it arrives. A result that is NaN by right takes both walks.
struct Split {
  uint32_t hi, lo;
};
template <bool CLAMP>
__device__ __forceinline__ Split split_tf32(float x) {
  Split s;
  s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  if (CLAMP) s.hi = clamp_tf32(s.hi);
  s.lo = __float_as_uint(x - __uint_as_float(s.hi)) & 0xffffe000u;
  return s;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// A fragment, split once and used for a row of n-tiles. EXACT: the values are tf32 already.
template <bool EXACT, bool CLAMP>
struct AFrag {
  uint32_t hi[4], lo[4];
  __device__ __forceinline__ void set(float a0, float a1, float a2, float a3) {
    const float a[4] = {a0, a1, a2, a3};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (EXACT) {
        hi[i] = __float_as_uint(a[i]);
      } else {
        const Split s = split_tf32<CLAMP>(a[i]);
        hi[i] = s.hi;
        lo[i] = s.lo;
      }
    }
  }
};
// acc[n] += A * B[n] over one k-step of eight, for four n-tiles; b(n, i) is the i-th value of a B fragment. The three
// products of an n-tile depend on one another, so the four tiles take turns.
template <bool EXA, bool EXB, bool CLAMP, typename LoadB>
__device__ __forceinline__ void mma3x4(float (*acc)[4], const AFrag<EXA, CLAMP>& a, LoadB b) {
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  float t[4][4];
  Split s[4][2];
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (EXB) s[n][i].hi = __float_as_uint(b(n, i));
      else s[n][i] = split_tf32<CLAMP>(b(n, i));
    }
  static_assert(EXB || !EXA, "an exact A comes with an exact B");
  if constexpr (EXA) {
#pragma unroll
    for (int n = 0; n < 4; ++n) mma_tf32(t[n], a.hi, s[n][0].hi, s[n][1].hi, zero);
  } else {
    // an exact B keeps its infinities in hi; they belong to the product with A's hi alone
    auto beside_lo = [](uint32_t hi) { return EXB && CLAMP ? clamp_tf32(hi) : hi; };
#pragma unroll
    for (int n = 0; n < 4; ++n) mma_tf32(t[n], a.lo, beside_lo(s[n][0].hi), beside_lo(s[n][1].hi), zero);
    if constexpr (!EXB) {
#pragma unroll
      for (int n = 0; n < 4; ++n) mma_tf32(t[n], a.hi, s[n][0].lo, s[n][1].lo, t[n]);
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) mma_tf32(t[n], a.hi, s[n][0].hi, s[n][1].hi, t[n]);
  }
  // packed additions: with three products and the splits of B the issue slots are nearly as busy as the tensor core
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    f32x2_get(add2(f32x2(acc[n][0], acc[n][1]), f32x2(t[n][0], t[n][1])), acc[n][0], acc[n][1]);
    f32x2_get(add2(f32x2(acc[n][2], acc[n][3]), f32x2(t[n][2], t[n][3])), acc[n][2], acc[n][3]);
  }
}

// NaN if any of them is (or where infinities of both signs meet)
template <int N>
__device__ __forceinline__ bool has_nan(const float (&v)[N][4]) {
  uint64_t a = 0, b = 0;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    a = add2(a, f32x2(v[n][0], v[n][1]));
    b = add2(b, f32x2(v[n][2], v[n][3]));
  }
  float x, y;
  f32x2_get(add2(a, b), x, y);
  return isnan(x + y);
}
template <int N>
__device__ __forceinline__ void set_zero(float (&v)[N][4]) {
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) v[n][e] = 0.f;
}

// pointer to the bias row of packed row `r` of query slab `slab` (kv slab `kvs`), or nullptr
__device__ __forceinline__ const float* bias_row(const BiasView& b, int slab, int kvs, int kv_slabs, int hkv, int r) {
  if (b.base == nullptr) return nullptr;
  const int blk = slab / kv_slabs, batch = kvs / hkv, hk = kvs % hkv;
  const int h = hk * b.g + r / b.sq, i = r % b.sq;
  return b.base + blk * b.s_blk + batch * b.s_b + h * b.s_h + i * b.s_q;
}

struct Fp32FwdParams {
  const float *q, *k, *v;
  BiasView bias;
  const int32_t* kv_valid_len;
  int rows, skv, hkv, kv_slabs, nsplit, tiles_per_split;   // tiles_per_split counts 128-row tiles, as in the 16-bit plan
  float scale_log2;
  float *o_part, *ml_part;
  const int* status;   // device status word: non-zero => return at once
};

// A CTA owns 128 packed rows (a warp 16 of them) and a range of keys, 64 at a time through two stages. Scores and P stay in
// the warp that made them.
constexpr int GF_SMEM = (128 * GT_LD + 4 * GT_TILE) * sizeof(float);

// BIAS: a thread's 32 values of a tile are all requested before the products, under which they arrive. Requested one by one
// between the products and the softmax they took nearly as long as the products: 32 slabs of 130 rows x 1,601 keys 289 -> 188
// us (168 without a bias), 8 slabs of 160 rows x 6,404 keys 196 -> 160. Without a bias the kernel carries none of it.
template <bool BIAS>
__global__ void __launch_bounds__(256, 1)
fp32_fwd_kernel(const Fp32FwdParams p) {
  if (p.status && *reinterpret_cast<const volatile int*>(p.status) != 0) return;
  extern __shared__ __align__(16) float sm[];
  float* sQ = sm;
  float* sKV = sQ + 128 * GT_LD;               // stage s: K at +2*s*TILE, V right after
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int mb = blockIdx.x, slab = blockIdx.y, split = blockIdx.z;
  const int kvs = slab % p.kv_slabs;          // several query blocks may share one K/V batch entry
  int valid = p.skv;
  if (p.kv_valid_len) valid = min(valid, max(0, p.kv_valid_len[kvs / p.hkv]));
  const int kv_begin = min(valid, split * p.tiles_per_split * 128);
  const int kv_end = min(valid, (split + 1) * p.tiles_per_split * 128);
  const float* ks = p.k + size_t(kvs) * p.skv * 128;
  const float* vs = p.v + size_t(kvs) * p.skv * 128;
  const int row0 = mb * 128 + warp * 16 + g;  // fragment rows row0, row0 + 8
  const bool has_rows = mb * 128 + warp * 16 < p.rows;      // a warp without any only loads: its share of the CTA stays free
  const float* brow[2];                       // (rows that do not exist: the last one's)
#pragma unroll
  for (int i = 0; i < 2; ++i)
    brow[i] = BIAS ? bias_row(p.bias, slab, kvs, p.kv_slabs, p.hkv, min(row0 + 8 * i, p.rows - 1)) : nullptr;

  float m[2], l[2], o[16][4];
  // the walk over the keys; a second one with CLAMP where NaN came out
  auto walk = [&](auto cl) {
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
    set_zero(o);
    if (kv_begin < kv_end) {
      load_rows(sQ, p.q + size_t(slab) * p.rows * 128, mb * 128, p.rows, 128, tid);
      load_rows(sKV, ks, kv_begin, p.skv, 64, tid);
      load_rows(sKV + GT_TILE, vs, kv_begin, p.skv, 64, tid);
      cp_commit();
    }
    const float* qa = sQ + (warp * 16 + g) * GT_LD + t;
    int st = 0;
    for (int kv0 = kv_begin; kv0 < kv_end; kv0 += 64, st ^= 1) {
      if (kv0 + 64 < kv_end) {
        float* nxt = sKV + 2 * (st ^ 1) * GT_TILE;
        load_rows(nxt, ks, kv0 + 64, p.skv, 64, tid);
        load_rows(nxt + GT_TILE, vs, kv0 + 64, p.skv, 64, tid);
      }
      cp_commit();                               // possibly empty: the group before it is then complete after cp_wait<1>
      cp_wait<1>();
      __syncthreads();
      if (!has_rows) {
        __syncthreads();
        continue;
      }
      const float* tile = sKV + 2 * st * GT_TILE;
      const float* kb = tile + g * GT_LD + t;
      const float* vb = tile + GT_TILE + 2 * t * GT_LD + g;
      float bv[BIAS ? 8 : 1][4];
      if constexpr (BIAS) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) bv[n][e] = __ldg(brow[e >> 1] + min(kv0 + n * 8 + 2 * t + (e & 1), kv_end - 1) * p.bias.s_kv);
      }
      float s[8][4];
      set_zero(s);
#pragma unroll 2
      for (int d = 0; d < 128; d += 8) {
        AFrag<false, cl.value> a;
        a.set(qa[d], qa[8 * GT_LD + d], qa[d + 4], qa[8 * GT_LD + d + 4]);
#pragma unroll
        for (int n = 0; n < 8; n += 4)
          mma3x4<false, false, cl.value>(s + n, a, [&](int u, int i) { return kb[(n + u) * 8 * GT_LD + d + 4 * i]; });
      }
      // online softmax in base 2; a row is spread over the four lanes of a quad
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = kv0 + n * 8 + 2 * t + (e & 1), i = e >> 1;
          float sc = -INFINITY;
          if (col < kv_end) {
            sc = s[n][e] * p.scale_log2;
            if constexpr (BIAS) sc = fmaf(bv[n][e], 1.4426950408889634f, sc);              // scale*q.k + bias, base 2
          }
          s[n][e] = sc;
          mx[i] = fmaxf(mx[i], sc);
        }
      float off[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        const float m_new = fmaxf(m[i], mx[i]);
        off[i] = m_new == -INFINITY ? 0.f : m_new;
        const float alpha = exp2f(m[i] - off[i]);       // m = -inf -> 0
        m[i] = m_new;
        l[i] *= alpha;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          o[n][2 * i] *= alpha;
          o[n][2 * i + 1] *= alpha;
        }
      }
      float sum[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[n][e] = exp2f(s[n][e] - off[e >> 1]);
          sum[e >> 1] += s[n][e];
        }
      l[0] += sum[0];
      l[1] += sum[1];
      // O += P V, eight keys at a time in the order 2t, 2t+1
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        AFrag<false, cl.value> a;
        a.set(s[n][0], s[n][2], s[n][1], s[n][3]);
        const float* v0 = vb + n * 8 * GT_LD;
#pragma unroll
        for (int c = 0; c < 16; c += 4)
          mma3x4<false, false, cl.value>(o + c, a, [&](int u, int i) { return v0[i * GT_LD + (c + u) * 8]; });
      }
      __syncthreads();                           // the stage may be loaded again
    }
  };
  walk(std::false_type{});
  if (__syncthreads_or(has_nan(o))) walk(std::true_type{});
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    const int row = row0 + 8 * i;
    if (row >= p.rows) continue;
    const size_t prow = (size_t(slab) * p.nsplit + split) * p.rows + row;
#pragma unroll
    for (int n = 0; n < 16; ++n)
      *reinterpret_cast<float2*>(p.o_part + prow * 128 + n * 8 + 2 * t) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
    if (t == 0) *reinterpret_cast<float2*>(p.ml_part + prow * 2) = make_float2(m[i], l[i]);
  }
}

struct Fp32BwdParams {
  const void *q, *d_o, *k, *v;
  const float *lse, *delta;
  BiasView bias;
  const int32_t* kv_valid_len;
  int rows, skv, hkv, nblk, kv_slabs;
  float scale, scale_log2;
  float *dq_acc;
  void *dk_acc, *dv_acc;   // fp32 for accumulate 0/1; the input dtype for accumulate 2
  int accumulate;
  const int* status;   // device status word: non-zero => return at once
};

// A CTA owns 64 keys (K, V in shared memory, dK, dV in registers) and walks over the packed query rows 64 at a time: S and
// dP (warp: 16 rows x 32 keys), P and dS to shared memory, dV += P^T dO and dK += dS^T Q (warp: 16 keys x 64 columns), dQ =
// dS K (16 rows x 64 columns) reduce-added. Q has two stages; dO has one, free after dV, so that its successor arrives
// while dK and dQ are computed.
constexpr int GB_SMEM = (5 * GT_TILE + 2 * GT_PTILE) * sizeof(float);

template <typename T>
__global__ void __launch_bounds__(256, 1)
fp32_bwd_kernel(const Fp32BwdParams p) {
  constexpr bool EX = sizeof(T) == 2;          // 16-bit inputs are exact in tf32
  // This kernel ends an fp32 backward (dQ is accumulated where it is wanted), so it also tells the host.
  if (p.status && __syncthreads_or(*reinterpret_cast<const volatile int*>(p.status) != 0)) {
    if (threadIdx.x == 0) publish_status(p.status);
    return;
  }
  extern __shared__ __align__(16) float sm[];
  float* sK = sm;
  float* sV = sK + GT_TILE;
  float* sQ = sV + GT_TILE;                    // two stages
  float* sDO = sQ + 2 * GT_TILE;
  float* sP = sDO + GT_TILE;                   // [q][kv]
  float* sDS = sP + GT_PTILE;                  // [q][kv]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wm = warp & 3, wn = warp >> 2;
  const int kv0 = blockIdx.x * 64, slab = blockIdx.y;
  int valid = p.skv;
  if (p.kv_valid_len) valid = min(valid, max(0, p.kv_valid_len[slab / p.hkv]));
  const bool live = kv0 < valid;
  const int tiles_per_block = (p.rows + 63) / 64, ntot = live ? tiles_per_block * p.nblk : 0;
  auto qslab_of = [&](int it) { return slab + (it / tiles_per_block) * p.kv_slabs; };
  auto load_q = [&](int it) {
    load_rows(sQ + (it & 1) * GT_TILE, static_cast<const T*>(p.q) + size_t(qslab_of(it)) * p.rows * 128,
              (it % tiles_per_block) * 64, p.rows, 64, tid);
  };
  auto load_do = [&](int it) {
    load_rows(sDO, static_cast<const T*>(p.d_o) + size_t(qslab_of(it)) * p.rows * 128, (it % tiles_per_block) * 64, p.rows,
              64, tid);
  };

  float dk[8][4], dv[8][4];      // keys wm*16 + g (+8), columns wn*64 + 8n + 2t (+1)
  if (ntot > 0) {
    load_rows(sK, static_cast<const T*>(p.k) + size_t(slab) * p.skv * 128, kv0, p.skv, 64, tid);
    load_rows(sV, static_cast<const T*>(p.v) + size_t(slab) * p.skv * 128, kv0, p.skv, 64, tid);
  }
  // The walk over the query rows, and a second one with CLAMP where NaN came out. dQ leaves with every tile: from the first
  // tile whose dQ holds NaN a warp adds nothing more, and the second walk adds from there.
  int redo_from = ntot;
  auto walk = [&](auto cl) {
    constexpr bool CL = cl.value;
    set_zero(dk);
    set_zero(dv);
    if (ntot > 0) {
      load_q(0);
      load_do(0);
      cp_commit();
    }
    for (int it = 0; it < ntot; ++it) {
      const int qslab = qslab_of(it), q0 = (it % tiles_per_block) * 64;
      float l2[2], dl[2];
      const float* br[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int qrow = q0 + wm * 16 + g + 8 * i;
        l2[i] = INFINITY;                        // rows that do not exist, or that have no valid key anywhere
        dl[i] = 0.f;
        br[i] = nullptr;
        if (qrow < p.rows) {
          l2[i] = p.lse[size_t(qslab) * p.rows + qrow] * 1.4426950408889634f;
          if (l2[i] == -INFINITY) l2[i] = INFINITY;
          dl[i] = p.delta[size_t(qslab) * p.rows + qrow];
          br[i] = bias_row(p.bias, qslab, slab, p.kv_slabs, p.hkv, qrow);
        }
      }
      cp_wait<0>();
      __syncthreads();                           // Q and dO are here; the previous tile is done with P, dS and its Q
      if (it + 1 < ntot) load_q(it + 1);
      cp_commit();
      const float* q = sQ + (it & 1) * GT_TILE;
      {
        float s[4][4], dp[4][4];
        const float *qa = q + (wm * 16 + g) * GT_LD + t, *da = sDO + (wm * 16 + g) * GT_LD + t;
        const float *kb = sK + (wn * 32 + g) * GT_LD + t, *vb = sV + (wn * 32 + g) * GT_LD + t;
        set_zero(s);
        set_zero(dp);
#pragma unroll 2
        for (int d = 0; d < 128; d += 8) {
          AFrag<EX, CL> a, b;
          a.set(qa[d], qa[8 * GT_LD + d], qa[d + 4], qa[8 * GT_LD + d + 4]);
          b.set(da[d], da[8 * GT_LD + d], da[d + 4], da[8 * GT_LD + d + 4]);
          mma3x4<EX, EX, CL>(s, a, [&](int u, int i) { return kb[u * 8 * GT_LD + d + 4 * i]; });
          mma3x4<EX, EX, CL>(dp, b, [&](int u, int i) { return vb[u * 8 * GT_LD + d + 4 * i]; });
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float pv[2], ds[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int col = kv0 + wn * 32 + n * 8 + 2 * t + e;
              const bool ok = col < valid;
              float sc = s[n][2 * i + e] * p.scale_log2;
              if (ok && br[i]) sc = fmaf(br[i][col * p.bias.s_kv], 1.4426950408889634f, sc);
              pv[e] = ok ? exp2f(sc - l2[i]) : 0.f;
              ds[e] = pv[e] * (dp[n][2 * i + e] - dl[i]);
            }
            const int at = (wm * 16 + g + 8 * i) * GT_LDP + wn * 32 + n * 8 + 2 * t;
            *reinterpret_cast<float2*>(sP + at) = make_float2(pv[0], pv[1]);
            *reinterpret_cast<float2*>(sDS + at) = make_float2(ds[0], ds[1]);
          }
      }
      __syncthreads();
      // acc[key][d] += X[q][key]^T B[q][d], eight query rows at a time in the order 2t, 2t+1
      auto transposed = [&](float (&acc)[8][4], const float* x, const float* b) {
        const float* xa = x + 2 * t * GT_LDP + wm * 16 + g;
        const float* bb = b + 2 * t * GT_LD + wn * 64 + g;
#pragma unroll 2
        for (int k8 = 0; k8 < 64; k8 += 8) {
          AFrag<false, CL> a;
          a.set(xa[k8 * GT_LDP], xa[k8 * GT_LDP + 8], xa[(k8 + 1) * GT_LDP], xa[(k8 + 1) * GT_LDP + 8]);
#pragma unroll
          for (int n = 0; n < 8; n += 4)
            mma3x4<false, EX, CL>(acc + n, a, [&](int u, int i) { return bb[(k8 + i) * GT_LD + (n + u) * 8]; });
        }
      };
      transposed(dv, sP, sDO);
      __syncthreads();                           // dO may be loaded again
      if (it + 1 < ntot) load_do(it + 1);
      cp_commit();
      transposed(dk, sDS, q);
      float dq[8][4];
      set_zero(dq);
      const float* xa = sDS + (wm * 16 + g) * GT_LDP + 2 * t;
      const float* kb = sK + 2 * t * GT_LD + wn * 64 + g;
#pragma unroll 2
      for (int k8 = 0; k8 < 64; k8 += 8) {
        const float2 r0 = *reinterpret_cast<const float2*>(xa + k8);
        const float2 r1 = *reinterpret_cast<const float2*>(xa + 8 * GT_LDP + k8);
        AFrag<false, CL> a;
        a.set(r0.x, r1.x, r0.y, r1.y);
#pragma unroll
        for (int n = 0; n < 8; n += 4)
          mma3x4<false, EX, CL>(dq + n, a, [&](int u, int i) { return kb[(k8 + i) * GT_LD + (n + u) * 8]; });
      }
      if (CL) {
        if (it < redo_from) continue;
      } else {
        if (redo_from == ntot && __any_sync(0xffffffffu, has_nan(dq))) redo_from = it;
        if (it >= redo_from) continue;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int qrow = q0 + wm * 16 + g + 8 * i;
        if (qrow >= p.rows) continue;
        float* dst = p.dq_acc + (size_t(qslab) * p.rows + qrow) * 128 + wn * 64 + 2 * t;
#pragma unroll
        for (int n = 0; n < 8; ++n)
          asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(dst + n * 8), "f"(dq[n][2 * i] * p.scale),
                       "f"(dq[n][2 * i + 1] * p.scale)
                       : "memory");
      }
    }
  };
  walk(std::false_type{});
  if (__syncthreads_or(redo_from < ntot || has_nan(dk) || has_nan(dv))) walk(std::true_type{});
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = kv0 + wm * 16 + g + 8 * i;
    if (row >= p.skv || (!live && p.accumulate == 1)) continue;
    const size_t off = (size_t(slab) * p.skv + row) * 128 + wn * 64 + 2 * t;
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float a = dk[n][2 * i + e] * p.scale, b = dv[n][2 * i + e];
        if (p.accumulate == 2) {                          // finished gradients in the input dtype
          from_f32(static_cast<T*>(p.dk_acc) + off + n * 8 + e, a);
          from_f32(static_cast<T*>(p.dv_acc) + off + n * 8 + e, b);
        } else {
          float* dkp = static_cast<float*>(p.dk_acc) + off + n * 8 + e;
          float* dvp = static_cast<float*>(p.dv_acc) + off + n * 8 + e;
          *dkp = p.accumulate == 1 ? *dkp + a : a;
          *dvp = p.accumulate == 1 ? *dvp + b : b;
        }
      }
  }
}

int launch_fwd_block_general(const lvx_shape& s, const FwdPlan& pl, const void* q, const void* k, const void* v,
                          const int32_t* kv_valid_len, const lvx_bias* bias, float sm_scale, float* o_part,
                          float* ml_part, cudaStream_t st) {
  Fp32FwdParams p;
  p.q = static_cast<const float*>(q);
  p.k = static_cast<const float*>(k);
  p.v = static_cast<const float*>(v);
  p.bias = make_bias(s, bias);
  p.kv_valid_len = kv_valid_len;
  p.rows = pl.rows;
  p.skv = s.Skv;
  p.hkv = s.Hkv;
  p.kv_slabs = s.B * s.Hkv;
  p.nsplit = pl.nsplit;
  p.tiles_per_split = pl.tiles_per_split;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.o_part = o_part;
  p.ml_part = ml_part;
  p.status = device_status_ptr();
  dim3 grid(pl.m_blocks, q_blocks_of(s) * s.B * s.Hkv, pl.nsplit);
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GF_SMEM);
    if (e == cudaSuccess) kern<<<grid, 256, GF_SMEM, st>>>(p);
  };
  if (bias) go(fp32_fwd_kernel<true>);
  else go(fp32_fwd_kernel<false>);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(fp32 fwd)");
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fp32 fwd kernel launch");
  return LVX_OK;
}

int launch_bwd_block_general(const lvx_shape& s, const void* q, const void* d_o, const float* lse, const float* delta,
                          const void* k, const void* v, const int32_t* kv_valid_len, const lvx_bias* bias,
                          float sm_scale, float* dq_acc, void* dk_acc, void* dv_acc, int accumulate_dkdv,
                          cudaStream_t st) {
  Fp32BwdParams p;
  p.q = q;
  p.d_o = d_o;
  p.lse = lse;
  p.delta = delta;
  p.k = k;
  p.v = v;
  p.bias = make_bias(s, bias);
  p.kv_valid_len = kv_valid_len;
  p.rows = (s.Hq / s.Hkv) * s.Sq;
  p.skv = s.Skv;
  p.hkv = s.Hkv;
  p.nblk = q_blocks_of(s);
  p.kv_slabs = s.B * s.Hkv;
  p.scale = sm_scale;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.dq_acc = dq_acc;
  p.dk_acc = dk_acc;
  p.dv_acc = dv_acc;
  p.accumulate = accumulate_dkdv;
  p.status = device_status_ptr();
  dim3 grid((s.Skv + 63) / 64, s.B * s.Hkv, 1);
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GB_SMEM);
    if (e == cudaSuccess) kern<<<grid, 256, GB_SMEM, st>>>(p);
  };
  if (s.dtype == LVX_FP32) go(fp32_bwd_kernel<float>);
  else go(fp32_bwd_kernel<__half>);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(fp32 bwd)");
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fp32 bwd kernel launch");
  return LVX_OK;
}

}  // namespace lvx
