// Forward block for few packed query rows (g * Sq <= 64): one new token, or a handful, against a long K/V shard.
//
// Such a call is a stream over K and V (2 x 256 bytes per key and KV head, read once), so what counts is bytes in
// flight, not tensor throughput. The 256-row kernel of fwd_sm100.cu spends the same ~3,400 cycles on a K/V tile
// however few of its rows exist, which holds it to about 4 TB/s. Here a CTA keeps three 64 KB stages (128 keys of K and
// V) in flight and eight warps share a tile without any hand-over between them: a warp owns 16 query rows (an
// mma.m16n8k16 tile) and 128 * RG / 8 keys of every tile, with a running (max, sum, O) of its own; the warps that share
// rows merge once, at the end of the CTA's key range. The legacy mma.sync form is used on purpose: its operands come
// from and go to registers, so the scores never leave the warp, and at <= 64 rows its rate is not what bounds the call.
// K and V tiles are the same 128-byte-swizzled boxes as in the 256-row kernel and are read with conflict-free ldmatrix.
// Measured: one token, 32 heads on 8 KV heads, 409,856 keys (1.68 GB of K and V): 427-449 -> 249-252 us a call, block and
// combine together, i.e. 6.7 TB/s (a copy reaches 6.5).
// The line at 64 rows, block and combine in us, 256-row kernel -> this one, at 1 / 32 / 33 / 64 rows per KV head:
//    8 KV heads x    300 keys    10.1 ->   5.9    11.0 ->   8.1    11.3 ->   8.7    11.5 ->   9.7
//    8 KV heads x  6,404 keys    21.7 ->  11.1    21.9 ->  12.8    22.0 ->  15.3    21.6 ->  17.2
//    8 KV heads x 102,464 keys   99.0 ->  66.2    99.3 ->  69.5    98.7 ->  93.8    98.0 ->  96.1
//  128 KV heads x  1,601 keys    37.0 ->  22.2    37.2 ->  25.4    37.6 ->  34.5    40.0 ->  36.6
//  128 KV heads x  6,404 keys   105.8 ->  64.6   106.2 ->  69.0   106.2 -> 105.6   108.6 -> 107.5
// Up to 32 rows the call runs at the rate of its bytes; with 64 the mma work of a tile takes longer than they do, and where
// the grid is large both kernels are even. More rows would be slower here than there.
// The partials have the layout of that kernel, so the combine kernel does not care which of the two ran.
#include "lvx_internal.h"
#include "sm100_prims.cuh"
#include <math.h>
#include <type_traits>

namespace lvx {

constexpr int FR_STAGES = 3;
constexpr int FR_HALF = 128 * 128;               // 64 columns of 128 keys, 16-bit
constexpr int FR_STAGE = 4 * FR_HALF;            // K then V
constexpr int FR_OFF_BAR = FR_STAGES * FR_STAGE;
constexpr int FR_SMEM = FR_OFF_BAR + 256 + 1024; // + barriers + alignment slack
constexpr int FR_WARPS = 8;
constexpr int FR_THREADS = (FR_WARPS + 1) * 32;
constexpr int FR_LDO = 132;                      // row stride (floats) of the merge buffer, which reuses the stages

enum { FR_K_FULL = 0, FR_V_FULL = FR_STAGES, FR_EMPTY = 2 * FR_STAGES, FR_COUNT = 3 * FR_STAGES };
#define FR_CODE(role, bar) (LVX_DEV_TIMEOUT_BASE | 0x180 | ((role) << 5) | (bar))

struct RowsParams {
  const void* q;
  int rows, skv, hkv, nsplit, tiles_per_split;
  const int32_t* kv_valid_len;
  float scale_log2;
  float *o_part, *ml_part;
  int* status;
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <bool IS_BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (IS_BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// RG: groups of 16 query rows (1, 2 or 4); the other 8 / RG warps of a group split the keys of a tile.
template <bool IS_BF16, int RG>
__global__ void __launch_bounds__(FR_THREADS, 1)
fwd_rows_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const RowsParams p) {
  constexpr int KG = FR_WARPS / RG;          // warps that share a row group
  constexpr int KPW = 128 / KG;              // keys of a tile per warp
  constexpr int CH = KPW < 32 ? KPW : 32;    // keys per softmax step
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FR_OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + FR_COUNT);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x, slab = blockIdx.y;
  // The status word may be set by another CTA or stream at any moment: one thread reads it, and the CTA leaves or stays as
  // a whole. Warps that went on alone would meet barriers that nobody initialised and wait for the others at bar.sync.
  int word = 0;
  if (tid == 0) word = *reinterpret_cast<volatile int*>(p.status);
  int valid = p.skv;
  if (p.kv_valid_len) valid = min(valid, max(0, p.kv_valid_len[slab / p.hkv]));
  const int valid_tiles = (valid + 127) >> 7;
  const int tile0 = split * p.tiles_per_split;
  const int n = max(0, min(tile0 + p.tiles_per_split, valid_tiles) - tile0);
  if (tid == 0) {
    for (int s = 0; s < FR_STAGES; ++s) {
      mbar_init(&bars[FR_K_FULL + s], 1);
      mbar_init(&bars[FR_V_FULL + s], 1);
      mbar_init(&bars[FR_EMPTY + s], FR_WARPS);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (__syncthreads_or(word)) return;

  float* o_dst = p.o_part + (size_t(slab) * p.nsplit + split) * p.rows * 128;
  float* ml_dst = p.ml_part + (size_t(slab) * p.nsplit + split) * p.rows * 2;
  if (n == 0) {      // nothing valid in this key range: the empty partial (O = 0, max = -inf, sum = 0)
    for (int i = tid; i < p.rows * 32; i += FR_THREADS) reinterpret_cast<float4*>(o_dst)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < p.rows; i += FR_THREADS) reinterpret_cast<float2*>(ml_dst)[i] = make_float2(-INFINITY, 0.f);
    return;
  }

  if (warp == FR_WARPS) {
    // =========================== TMA producer ===========================
    if (lane == 0) {
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      int issued = 0;
      for (int j = 0; j < n; ++j) {
        const int s = j % FR_STAGES, y = (tile0 + j) * 128;
        if (!mbar_wait(&bars[FR_EMPTY + s], ((j / FR_STAGES) & 1) ^ 1, abort_flag, p.status, FR_CODE(2, FR_EMPTY),
                       LVX_SPIN_LIMIT_CYCLES))
          break;
        uint8_t* dst = smem + s * FR_STAGE;
        mbar_arrive_expect_tx(&bars[FR_K_FULL + s], 2 * FR_HALF);
        tma_load_3d(dst, &tmK, &bars[FR_K_FULL + s], 0, y, slab);
        tma_load_3d(dst + FR_HALF, &tmK, &bars[FR_K_FULL + s], 64, y, slab);
        mbar_arrive_expect_tx(&bars[FR_V_FULL + s], 2 * FR_HALF);
        tma_load_3d(dst + 2 * FR_HALF, &tmV, &bars[FR_V_FULL + s], 0, y, slab);
        tma_load_3d(dst + 3 * FR_HALF, &tmV, &bars[FR_V_FULL + s], 64, y, slab);
        issued = j + 1;
      }
      if (*abort_flag) {   // a CTA that is giving up must not leave while a copy into its shared memory is in flight
        for (int j = max(0, issued - FR_STAGES); j < issued; ++j)
          for (int b = FR_K_FULL; b <= FR_V_FULL; b += FR_STAGES) {
            const long long t0 = clock64();
            while (!mbar_try_wait(&bars[b + j % FR_STAGES], (j / FR_STAGES) & 1) && clock64() - t0 < LVX_SPIN_LIMIT_CYCLES) {}
          }
      }
    }
    return;
  }

  // =========================== compute warps ===========================
  const int rg = warp % RG, kg = warp / RG;
  const int r0 = rg * 16 + (lane >> 2), cq = (lane & 3) * 2;   // fragment rows r0, r0 + 8; column pair cq
  uint32_t qf[8][4];
  {
    const uint32_t* qs = reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.q) + size_t(slab) * p.rows * 128);
    const bool ok0 = r0 < p.rows, ok1 = r0 + 8 < p.rows;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const int c = (kk * 16 + cq) >> 1;
      qf[kk][0] = ok0 ? qs[r0 * 64 + c] : 0u;
      qf[kk][1] = ok1 ? qs[(r0 + 8) * 64 + c] : 0u;
      qf[kk][2] = ok0 ? qs[r0 * 64 + c + 4] : 0u;
      qf[kk][3] = ok1 ? qs[(r0 + 8) * 64 + c + 4] : 0u;
    }
  }
  const float c = p.scale_log2;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float o[16][4];
#pragma unroll
  for (int t = 0; t < 16; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[t][e] = 0.f;
  // ldmatrix lane addresses inside a tile: K takes (keys 0-7 | 8-15) x (d 0-7 | 8-15) with d running first, V keys first
  const uint32_t sbase = smem_u32(smem);
  const int k_row = kg * KPW + ((lane >> 4) << 3) + (lane & 7), k_ch = (lane >> 3) & 1;
  const int v_row = kg * KPW + (((lane >> 3) & 1) << 3) + (lane & 7), v_ch = lane >> 4;
  const uint32_t sw = lane & 7;              // row % 8 of every address this lane forms
  bool alive = true;
  for (int j = 0; alive && j < n; ++j) {
    const int s = j % FR_STAGES;
    const uint32_t ph = (j / FR_STAGES) & 1;
    const uint32_t tk = sbase + s * FR_STAGE, tv = tk + 2 * FR_HALF;
    alive = mbar_wait(&bars[FR_K_FULL + s], ph, abort_flag, p.status, FR_CODE(0, FR_K_FULL), LVX_SPIN_LIMIT_CYCLES);
    alive = __all_sync(0xffffffffu, alive);
    if (!alive) break;
    const int left = valid - (tile0 + j) * 128 - kg * KPW;   // valid keys from this warp's first key on
#pragma unroll
    for (int c0 = 0; c0 < KPW; c0 += CH) {
      float sc[CH / 8][4];
#pragma unroll
      for (int t = 0; t < CH / 8; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[t][e] = 0.f;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
#pragma unroll
        for (int g = 0; g < CH / 16; ++g) {
          uint32_t b[4];
          ldsm4(tk + (kk >> 2) * FR_HALF + (k_row + c0 + g * 16) * 128 + ((((kk & 3) * 2 + k_ch) ^ sw) << 4), b);
          mma_16816<IS_BF16>(sc[2 * g], qf[kk], b[0], b[1]);
          mma_16816<IS_BF16>(sc[2 * g + 1], qf[kk], b[2], b[3]);
        }
      if (left < c0 + CH) {
#pragma unroll
        for (int t = 0; t < CH / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c0 + t * 8 + cq + (e & 1) >= left) sc[t][e] = -INFINITY;
      }
      // online softmax in base 2; a row is spread over four lanes. The running max is a reference point only: it is
      // raised when it would grow by more than 2^8, so that P stays below 256 and O is rarely rescaled.
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int t = 0; t < CH / 8; ++t) {
        mx[0] = fmaxf(mx[0], fmaxf(sc[t][0], sc[t][1]));
        mx[1] = fmaxf(mx[1], fmaxf(sc[t][2], sc[t][3]));
      }
      bool grow = false;
      float alpha[2] = {1.f, 1.f};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2)) * c;
        if (mx[i] > m[i] + 8.f) {
          alpha[i] = ex2f(m[i] - mx[i]);
          m[i] = mx[i];
          l[i] *= alpha[i];
          grow = true;
        }
      }
      if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          o[t][0] *= alpha[0];
          o[t][1] *= alpha[0];
          o[t][2] *= alpha[1];
          o[t][3] *= alpha[1];
        }
      }
      const float off0 = m[0] == -INFINITY ? 0.f : m[0], off1 = m[1] == -INFINITY ? 0.f : m[1];
      uint32_t pf[CH / 16][4];
#pragma unroll
      for (int t = 0; t < CH / 8; ++t) {
        const float p0 = ex2f(fmaf(sc[t][0], c, -off0)), p1 = ex2f(fmaf(sc[t][1], c, -off0));
        const float p2 = ex2f(fmaf(sc[t][2], c, -off1)), p3 = ex2f(fmaf(sc[t][3], c, -off1));
        l[0] += p0 + p1;
        l[1] += p2 + p3;
        pf[t >> 1][(t & 1) * 2] = IS_BF16 ? pack_bf16x2(p0, p1) : pack_f16x2(p0, p1);
        pf[t >> 1][(t & 1) * 2 + 1] = IS_BF16 ? pack_bf16x2(p2, p3) : pack_f16x2(p2, p3);
      }
      if (c0 == 0) {
        alive = mbar_wait(&bars[FR_V_FULL + s], ph, abort_flag, p.status, FR_CODE(0, FR_V_FULL), LVX_SPIN_LIMIT_CYCLES);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) break;
      }
#pragma unroll
      for (int g = 0; g < CH / 16; ++g)
#pragma unroll
        for (int dn = 0; dn < 8; ++dn) {
          uint32_t b[4];
          ldsm4_t(tv + (dn >> 2) * FR_HALF + (v_row + c0 + g * 16) * 128 + ((((dn & 3) * 2 + v_ch) ^ sw) << 4), b);
          mma_16816<IS_BF16>(o[2 * dn], pf[g], b[0], b[1]);
          mma_16816<IS_BF16>(o[2 * dn + 1], pf[g], b[2], b[3]);
        }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[FR_EMPTY + s]);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
  // ---- merge of the KG warps of a row group, through the stage buffers (every copy has landed: every warp has waited
  // for every tile; a warp that gave up has set the abort flag) ----
  float* mo = reinterpret_cast<float*>(smem);
  float* mml = mo + FR_WARPS * 16 * FR_LDO;
  asm volatile("bar.sync 1, %0;" ::"n"(FR_WARPS * 32) : "memory");
  if (*abort_flag) return;
  {
    float* dst = mo + (warp * 16 + (lane >> 2)) * FR_LDO + cq;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      *reinterpret_cast<float2*>(dst + t * 8) = make_float2(o[t][0], o[t][1]);
      *reinterpret_cast<float2*>(dst + 8 * FR_LDO + t * 8) = make_float2(o[t][2], o[t][3]);
    }
    if ((lane & 3) == 0) {
      float* d = mml + (warp * 16 + (lane >> 2)) * 2;
      d[0] = m[0];
      d[1] = l[0];
      d[16] = m[1];
      d[17] = l[1];
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(FR_WARPS * 32) : "memory");
  for (int i = tid; i < RG * 16 * 32; i += FR_WARPS * 32) {
    const int row = i >> 5, c4 = i & 31;
    if (row >= p.rows) break;
    const int w0 = row >> 4, rr = row & 15;
    float mm = -INFINITY;
#pragma unroll
    for (int g = 0; g < KG; ++g) mm = fmaxf(mm, mml[((g * RG + w0) * 16 + rr) * 2]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float ls = 0.f;
    const float moff = mm == -INFINITY ? 0.f : mm;
#pragma unroll
    for (int g = 0; g < KG; ++g) {
      const int wr = (g * RG + w0) * 16 + rr;
      const float w = ex2f(mml[wr * 2] - moff);
      const float4 v = *reinterpret_cast<const float4*>(mo + wr * FR_LDO + c4 * 4);
      ls = fmaf(mml[wr * 2 + 1], w, ls);
      acc.x = fmaf(v.x, w, acc.x);
      acc.y = fmaf(v.y, w, acc.y);
      acc.z = fmaf(v.z, w, acc.z);
      acc.w = fmaf(v.w, w, acc.w);
    }
    reinterpret_cast<float4*>(o_dst)[row * 32 + c4] = acc;
    if (c4 == 0) *reinterpret_cast<float2*>(ml_dst + row * 2) = make_float2(mm, ls);
  }
}

int launch_fwd_rows(const lvx_shape& s, const FwdPlan& pl, const void* q, const void* k, const void* v,
                    const int32_t* kv_valid_len, float sm_scale, float* o_part, float* ml_part, int* status,
                    cudaStream_t st) {
  CUtensorMap tmK, tmV;
  const uint64_t row_bytes = 256, slabs = uint64_t(s.B) * s.Hkv;
  const uint64_t kvrows = s.Skv > 0 ? s.Skv : 1;     // no rows: every CTA writes the empty partial, nothing is loaded
  int rc = make_tmap_3d(&tmK, s.dtype, s.Skv > 0 ? k : q, 128, kvrows, slabs, row_bytes, row_bytes * kvrows, 64, 128);
  if (rc) return rc;
  rc = make_tmap_3d(&tmV, s.dtype, s.Skv > 0 ? v : q, 128, kvrows, slabs, row_bytes, row_bytes * kvrows, 64, 128);
  if (rc) return rc;
  RowsParams p;
  p.q = q;
  p.rows = pl.rows;
  p.skv = s.Skv;
  p.hkv = s.Hkv;
  p.nsplit = pl.nsplit;
  p.tiles_per_split = pl.tiles_per_split;
  p.kv_valid_len = kv_valid_len;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.o_part = o_part;
  p.ml_part = ml_part;
  p.status = status;
  dim3 grid(pl.nsplit, unsigned(slabs), 1);
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FR_SMEM);
    if (e == cudaSuccess) kern<<<grid, FR_THREADS, FR_SMEM, st>>>(tmK, tmV, p);
  };
  auto pick = [&](auto bf16) {
    constexpr bool B16 = decltype(bf16)::value;
    if (pl.rows <= 16) go(fwd_rows_kernel<B16, 1>);
    else if (pl.rows <= 32) go(fwd_rows_kernel<B16, 2>);
    else go(fwd_rows_kernel<B16, 4>);
  };
  if (s.dtype == LVX_BF16) pick(std::true_type{});
  else pick(std::false_type{});
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(fwd rows)");
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fwd_rows_kernel launch");
  return LVX_OK;
}

}  // namespace lvx
