// HBM-bound helper kernels around the two tensor-core blocks:
//   fwd_combine_kernel  split-KV partials (+) travelling (O, lse)  ->  (O, lse)
//   bwd_prep_kernel     delta = rowsum(O * dO)
//   add_cast_kernel     out = cast(a + b)
// A row of 128 values is read by one warp (fp32) or half a warp (16 bits), 16 bytes a lane, so that every access is a full
// coalesced 512- or 256-byte row. Where rows are few, eight warps share one in the combine.
#include "lvx_internal.h"
#include "sm100_prims.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

namespace lvx {

constexpr float kLn2 = 0.6931471805599453f;
constexpr float kLog2e = 1.4426950408889634f;

// While the device status word is set (a bounded wait ran out somewhere) every kernel returns at once, so that
// nothing is computed from buffers an aborted kernel left unwritten.
__device__ __forceinline__ bool poisoned(const int* status) {
  return status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
}

template <int OUT>  // 0 bf16, 1 fp16, 2 fp32
__device__ __forceinline__ void store4(void* base, size_t idx4, float4 v) {
  if (OUT == 2) {
    reinterpret_cast<float4*>(base)[idx4] = v;
  } else if (OUT == 0) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<uint32_t*>(&a);
    u.y = *reinterpret_cast<uint32_t*>(&b);
    reinterpret_cast<uint2*>(base)[idx4] = u;
  } else {
    __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<uint32_t*>(&a);
    u.y = *reinterpret_cast<uint32_t*>(&b);
    reinterpret_cast<uint2*>(base)[idx4] = u;
  }
}

// Partials live in the packed-row order of the forward block: slab (b*Hkv + hk), split, row r = hg*Sq + i
// where the query head is h = hk*g + hg. A [B,Hq,Sq,D] tensor has exactly the same row order
// (row index (b*Hq + h)*Sq + i = slab*rows + r), so "global row" below indexes both.
//
// The partials are read once, four splits of a row at a time with their (max, sum) beside them: a first walk over the
// statistics alone would be a second round trip to memory for every row. WPR warps share a row: one where there are rows
// enough to fill the GPU, eight (each with every eighth group of four splits) for the few rows and many splits of a
// decoding call, where a single warp's walk is a chain of round trips. The status word is requested together with the
// data and looked at before anything is stored. Measured: 65,536 rows of 4 splits 44 -> 36 us; 32 rows of
// 18 splits 14 -> 5 us.
struct RowAcc {
  float m, l;      // running max (base 2, already scaled) and sum
  float4 v;
};
__device__ __forceinline__ void row_merge(RowAcc& a, const RowAcc& b) {
  const float m = fmaxf(a.m, b.m);
  if (m == -INFINITY) return;
  const float wa = exp2f(a.m - m), wb = exp2f(b.m - m);      // an empty side (max -inf) gets weight 0
  a.m = m;
  a.l = a.l * wa + b.l * wb;
  a.v.x = a.v.x * wa + b.v.x * wb;
  a.v.y = a.v.y * wa + b.v.y * wb;
  a.v.z = a.v.z * wa + b.v.z * wb;
  a.v.w = a.v.w * wa + b.v.w * wb;
}

template <int OUT, int WPR>
__global__ void __launch_bounds__(256)
fwd_combine_kernel(const float* __restrict__ o_part, const float* __restrict__ ml_part, const float* __restrict__ o_in,
                   const float* __restrict__ lse_in, void* __restrict__ o_out, float* __restrict__ lse_out,
                   int rows_per_slab, int nsplit, long total_rows, const int* status) {
  const int bad = status ? *reinterpret_cast<const volatile int*>(status) : 0;
  const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) % WPR;
  const long grow = ((long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) / WPR;
  if (grow >= total_rows) return;                 // WPR > 1: a block is one row, so its warps leave together
  const long slab = grow / rows_per_slab;
  const int r = int(grow - slab * rows_per_slab);

  RowAcc a;
  a.m = -INFINITY;
  a.l = 0.f;
  a.v = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = part * 4; s0 < nsplit; s0 += WPR * 4) {
    float2 ml[4];
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int s = min(s0 + u, nsplit - 1);
      const size_t prow = (size_t(slab) * nsplit + s) * rows_per_slab + r;
      ml[u] = *reinterpret_cast<const float2*>(ml_part + prow * 2);
      v[u] = reinterpret_cast<const float4*>(o_part + prow * 128)[lane];
      if (s0 + u >= nsplit) ml[u].x = -INFINITY;
    }
    const float m = fmaxf(fmaxf(a.m, fmaxf(ml[0].x, ml[1].x)), fmaxf(ml[2].x, ml[3].x));
    if (m == -INFINITY) continue;
    const float wa = exp2f(a.m - m);
    a.m = m;
    a.l *= wa;
    a.v.x *= wa; a.v.y *= wa; a.v.z *= wa; a.v.w *= wa;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (ml[u].x == -INFINITY) continue;
      const float w = exp2f(ml[u].x - m);
      a.l += ml[u].y * w;
      a.v.x += v[u].x * w;
      a.v.y += v[u].y * w;
      a.v.z += v[u].z * w;
      a.v.w += v[u].w * w;
    }
  }
  if constexpr (WPR > 1) {
    __shared__ float4 s_v[WPR][32];
    __shared__ float2 s_ml[WPR];
    s_v[part][lane] = a.v;
    if (lane == 0) s_ml[part] = make_float2(a.m, a.l);
    __syncthreads();
    if (part > 0) return;
#pragma unroll
    for (int w = 1; w < WPR; ++w) {
      RowAcc b;
      b.m = s_ml[w].x;
      b.l = s_ml[w].y;
      b.v = s_v[w][lane];
      row_merge(a, b);
    }
  }
  if (bad) {
    if (lane == 0) publish_status(status);
    return;
  }
  float4 acc = a.v;
  const float mmax = a.m, lsum = a.l;
  // (O_loc, lse_loc) of this shard
  float lse_loc = -INFINITY;
  if (lsum > 0.f) {
    const float inv = 1.f / lsum;
    acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
    lse_loc = (mmax + log2f(lsum)) * kLn2;
  } else {
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // merge with the travelling accumulator
  float lse_new = lse_loc;
  if (o_in != nullptr) {
    const float lse_old = lse_in[grow];
    const float mx = fmaxf(lse_old, lse_loc);
    if (mx == -INFINITY) {
      lse_new = -INFINITY;
      acc = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      const float wo = expf(lse_old - mx), wl = expf(lse_loc - mx);
      const float tot = wo + wl;
      lse_new = mx + logf(tot);
      const float co = wo / tot, cl = wl / tot;
      const float4 vo = reinterpret_cast<const float4*>(o_in)[size_t(grow) * 32 + lane];
      acc.x = vo.x * co + acc.x * cl;
      acc.y = vo.y * co + acc.y * cl;
      acc.z = vo.z * co + acc.z * cl;
      acc.w = vo.w * co + acc.w * cl;
    }
  }
  store4<OUT>(o_out, size_t(grow) * 32 + lane, acc);
  if (lane == 0) lse_out[grow] = lse_new;
}

int launch_fwd_combine(const lvx_shape& s, const FwdPlan& p, const float* o_part, const float* ml_part,
                       const float* o_in, const float* lse_in, void* o_out, float* lse_out, int out_is_final,
                       cudaStream_t st) {
  const long total_rows = long(q_blocks_of(s)) * s.B * s.Hq * s.Sq;
  const int threads = 256;
  const int* sp = device_status_ptr();
  const long blocks = (total_rows * 32 + threads - 1) / threads;
  const int out = out_is_final ? s.dtype : LVX_FP32;
  // Eight warps per row while the rows alone leave SMs empty and a warp would walk more than two groups of four splits.
  const bool wide = total_rows <= 148 * 8 && p.nsplit > 8;
  auto go = [&](auto one, auto eight) {
    if (wide) eight<<<total_rows, threads, 0, st>>>(o_part, ml_part, o_in, lse_in, o_out, lse_out, p.rows, p.nsplit, total_rows, sp);
    else one<<<blocks, threads, 0, st>>>(o_part, ml_part, o_in, lse_in, o_out, lse_out, p.rows, p.nsplit, total_rows, sp);
  };
  if (out == LVX_BF16) go(fwd_combine_kernel<0, 1>, fwd_combine_kernel<0, 8>);
  else if (out == LVX_FP16) go(fwd_combine_kernel<1, 1>, fwd_combine_kernel<1, 8>);
  else go(fwd_combine_kernel<2, 1>, fwd_combine_kernel<2, 8>);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fwd_combine launch");
  return LVX_OK;
}

// ---------------------------------------------------------------------------------------------
// Merge of `count` normalised partial results (O fp32, lse) of the same rows; one warp per row.
template <int OUT>
__global__ void __launch_bounds__(256)
fwd_merge_parts_kernel(const float* __restrict__ o_parts, const float* __restrict__ lse_parts, int count,
                       size_t stride_o, size_t stride_lse, void* __restrict__ o_out, float* __restrict__ lse_out,
                       long total_rows, const int* status) {
  if (poisoned(status)) return;
  const int lane = threadIdx.x & 31;
  const long row = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (row >= total_rows) return;
  float mx = -INFINITY;
  for (int c = 0; c < count; ++c) mx = fmaxf(mx, lse_parts[c * stride_lse + row]);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float tot = 0.f;
  if (mx != -INFINITY) {
    for (int c = 0; c < count; ++c) {
      const float l = lse_parts[c * stride_lse + row];
      if (l == -INFINITY) continue;
      const float w = expf(l - mx);
      tot += w;
      const float4 v = reinterpret_cast<const float4*>(o_parts + c * stride_o)[size_t(row) * 32 + lane];
      acc.x += v.x * w; acc.y += v.y * w; acc.z += v.z * w; acc.w += v.w * w;
    }
    const float inv = 1.f / tot;
    acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
  }
  store4<OUT>(o_out, size_t(row) * 32 + lane, acc);
  if (lane == 0) lse_out[row] = mx == -INFINITY ? -INFINITY : mx + logf(tot);
}

int launch_fwd_merge_parts(const lvx_shape& s, const float* o_parts, const float* lse_parts, int count,
                           size_t stride_o, size_t stride_lse, void* o_out, float* lse_out, cudaStream_t st) {
  const long total_rows = long(q_blocks_of(s)) * s.B * s.Hq * s.Sq;
  const int threads = 256;
  const int* sp = device_status_ptr();
  const long blocks = (total_rows * 32 + threads - 1) / threads;
  if (s.dtype == LVX_BF16)
    fwd_merge_parts_kernel<0><<<blocks, threads, 0, st>>>(o_parts, lse_parts, count, stride_o, stride_lse, o_out, lse_out, total_rows, sp);
  else if (s.dtype == LVX_FP16)
    fwd_merge_parts_kernel<1><<<blocks, threads, 0, st>>>(o_parts, lse_parts, count, stride_o, stride_lse, o_out, lse_out, total_rows, sp);
  else
    fwd_merge_parts_kernel<2><<<blocks, threads, 0, st>>>(o_parts, lse_parts, count, stride_o, stride_lse, o_out, lse_out, total_rows, sp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fwd_merge_parts launch");
  return LVX_OK;
}

// ---------------------------------------------------------------------------------------------
// delta = rowsum(O * dO): 16 bytes a lane (a half-warp per 16-bit row), four rows in flight per lane group: 65,536 rows of
// bf16 in 7.6 us against 23 with one row per warp.
template <int IN>
__global__ void __launch_bounds__(256)
bwd_prep_kernel(const void* __restrict__ o, const void* __restrict__ d_o, float* __restrict__ delta, long total_rows,
                const int* status) {
  constexpr int LANES = IN == 2 ? 32 : 16, GROUPS = 256 / LANES, U = 4;
  const int bad = status ? *reinterpret_cast<const volatile int*>(status) : 0;
  const int l = threadIdx.x % LANES, grp = threadIdx.x / LANES;
  const long row0 = long(blockIdx.x) * (GROUPS * U) + grp;
  uint4 a[U], b[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const size_t at = size_t(min(row0 + u * GROUPS, total_rows - 1)) * LANES + l;
    a[u] = reinterpret_cast<const uint4*>(o)[at];
    b[u] = reinterpret_cast<const uint4*>(d_o)[at];
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t x[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, y[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (IN == 2) {
        v = fmaf(__uint_as_float(x[i]), __uint_as_float(y[i]), v);
      } else {
        const float2 p = unpack16x2<IN == 0>(x[i]), q = unpack16x2<IN == 0>(y[i]);
        v = fmaf(p.x, q.x, v);
        v = fmaf(p.y, q.y, v);
      }
    }
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (l == 0 && row0 + u * GROUPS < total_rows && !bad) delta[row0 + u * GROUPS] = v;
  }
}

int launch_bwd_prep(const lvx_shape& s, const void* o, const void* d_o, float* delta, cudaStream_t st) {
  const long total_rows = long(q_blocks_of(s)) * s.B * s.Hq * s.Sq;
  const int threads = 256;
  const int* sp = device_status_ptr();
  const long per_block = (s.dtype == LVX_FP32 ? 8 : 16) * 4;
  const long blocks = (total_rows + per_block - 1) / per_block;
  if (s.dtype == LVX_BF16) bwd_prep_kernel<0><<<blocks, threads, 0, st>>>(o, d_o, delta, total_rows, sp);
  else if (s.dtype == LVX_FP16) bwd_prep_kernel<1><<<blocks, threads, 0, st>>>(o, d_o, delta, total_rows, sp);
  else bwd_prep_kernel<2><<<blocks, threads, 0, st>>>(o, d_o, delta, total_rows, sp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "bwd_prep launch");
  return LVX_OK;
}

// ---------------------------------------------------------------------------------------------
template <int OUT>
__global__ void __launch_bounds__(256)
add_cast_kernel(const float* __restrict__ a, const float* __restrict__ b, void* __restrict__ out, size_t n4, size_t n,
                const int* status) {
  if (poisoned(status)) {
    if ((threadIdx.x & 31) == 0) publish_status(status);
    return;
  }
  const size_t stride = size_t(gridDim.x) * blockDim.x;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
    float4 v = reinterpret_cast<const float4*>(a)[i];
    if (b) {
      const float4 w = reinterpret_cast<const float4*>(b)[i];
      v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    store4<OUT>(out, i, v);
  }
  // tail (n not a multiple of 4)
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const size_t i = n4 * 4 + threadIdx.x;
    const float v = a[i] + (b ? b[i] : 0.f);
    if (OUT == 2) reinterpret_cast<float*>(out)[i] = v;
    else if (OUT == 0) reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(v);
    else reinterpret_cast<__half*>(out)[i] = __float2half_rn(v);
  }
}

int launch_add_cast(const float* a, const float* b, void* out, int out_dtype, size_t n, cudaStream_t st) {
  const size_t n4 = n / 4;
  const int threads = 256;
  const int* sp = device_status_ptr();
  size_t blocks = (n4 + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks == 0) blocks = 1;
  if (out_dtype == LVX_BF16) add_cast_kernel<0><<<blocks, threads, 0, st>>>(a, b, out, n4, n, sp);
  else if (out_dtype == LVX_FP16) add_cast_kernel<1><<<blocks, threads, 0, st>>>(a, b, out, n4, n, sp);
  else add_cast_kernel<2><<<blocks, threads, 0, st>>>(a, b, out, n4, n, sp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "add_cast launch");
  return LVX_OK;
}

// ---------------------------------------------------------------------------------------------
template <int OUT>
__global__ void __launch_bounds__(256)
sum_cast_kernel(const float* __restrict__ parts, int count, size_t stride, void* __restrict__ out, size_t n4,
                const int* status) {
  if (poisoned(status)) return;
  const size_t gstride = size_t(gridDim.x) * blockDim.x;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += gstride) {
    float4 v = reinterpret_cast<const float4*>(parts)[i];
    for (int c = 1; c < count; ++c) {
      const float4 w = reinterpret_cast<const float4*>(parts + c * stride)[i];
      v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    store4<OUT>(out, i, v);
  }
}

int launch_sum_cast(const float* parts, int count, size_t stride, void* out, int out_dtype, size_t n, cudaStream_t st) {
  const size_t n4 = n / 4;
  const int threads = 256;
  const int* sp = device_status_ptr();
  size_t blocks = (n4 + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks == 0) blocks = 1;
  if (out_dtype == LVX_BF16) sum_cast_kernel<0><<<blocks, threads, 0, st>>>(parts, count, stride, out, n4, sp);
  else if (out_dtype == LVX_FP16) sum_cast_kernel<1><<<blocks, threads, 0, st>>>(parts, count, stride, out, n4, sp);
  else sum_cast_kernel<2><<<blocks, threads, 0, st>>>(parts, count, stride, out, n4, sp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "sum_cast launch");
  return LVX_OK;
}

}  // namespace lvx
