// Reading activations with an optional prologue (shared by the kernels that prepare x).
#pragma once
#include "bqq_common.cuh"

namespace bqq {

// Where the activation comes from, and what is applied to it on the way in (BqqFusion::prologue):
// nothing, RMS normalisation (x * inv_rms * w[n]; inv_rms of the row is computed by the caller of
// xprep_pair), or SwiGLU (silu(x[n]) * x[n + n_in], x holding [gate | up] rows of 2 * n_in elements).
struct XSource {
  const void* x;
  const void* w;
  int64_t ld;
  int dtype, w_dtype, mode, n_in;
  float eps;
};
__device__ __forceinline__ float load_x(const XSource& s, int m, int n, float inv_rms) {
  float v = load_as_float(s.x, (size_t)m * s.ld + n, s.dtype);
  if (s.mode == BQQ_PRO_RMSNORM) {
    v = v * inv_rms * load_as_float(s.w, n, s.w_dtype);
  } else if (s.mode == BQQ_PRO_SWIGLU) {
    const float u = load_as_float(s.x, (size_t)m * s.ld + s.n_in + n, s.dtype);
    v = v / (1.f + __expf(-v)) * u;
  }
  return v;
}
// Four consecutive elements n0 .. n0+3 of a tensor of type `dt` as floats; one 8- or 16-byte load when the
// address allows it, four element loads otherwise.
__device__ __forceinline__ void load_quad(const void* base, size_t idx, int dt, float (&v)[4]) {
  if (dt == BQQ_F32) {
    const float* p = reinterpret_cast<const float*>(base) + idx;
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
      const float4 q = *reinterpret_cast<const float4*>(p);
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = p[e];
    }
    return;
  }
  const uint16_t* p = reinterpret_cast<const uint16_t*>(base) + idx;
  uint32_t w0, w1;
  if ((reinterpret_cast<uintptr_t>(p) & 7) == 0) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    w0 = q.x; w1 = q.y;
  } else {
    w0 = (uint32_t)p[0] | ((uint32_t)p[1] << 16);
    w1 = (uint32_t)p[2] | ((uint32_t)p[3] << 16);
  }
  if (dt == BQQ_BF16) {
    v[0] = __uint_as_float(w0 << 16); v[1] = __uint_as_float(w0 & 0xFFFF0000u);
    v[2] = __uint_as_float(w1 << 16); v[3] = __uint_as_float(w1 & 0xFFFF0000u);
  } else {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w0));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&w1));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}
// x[m, n0 .. n0+3] after the prologue (all four columns exist)
__device__ __forceinline__ void load_x_quad(const XSource& s, int m, int n0, float inv_rms, float (&v)[4]) {
  load_quad(s.x, (size_t)m * s.ld + n0, s.dtype, v);
  if (s.mode == BQQ_PRO_RMSNORM) {
    float w[4];
    load_quad(s.w, n0, s.w_dtype, w);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = v[e] * inv_rms * w[e];
  } else if (s.mode == BQQ_PRO_SWIGLU) {
    float u[4];
    load_quad(s.x, (size_t)m * s.ld + s.n_in + n0, s.dtype, u);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = v[e] / (1.f + __expf(-v[e])) * u[e];
  }
}
// Four consecutive elements as they lie in memory (aligned to four elements), and as floats: several loads can be under way
// before the first is converted.
__device__ __forceinline__ uint4 load_raw4(const void* base, size_t idx, bool f32) {
  if (f32) return *reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(base) + idx);
  const uint2 q = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(base) + idx);
  return make_uint4(q.x, q.y, 0u, 0u);
}
__device__ __forceinline__ void raw4_to_float(const uint4& r, int dt, float (&v)[4]) {
  if (dt == BQQ_F32) {
    v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
  } else if (dt == BQQ_BF16) {
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xFFFF0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xFFFF0000u);
  } else {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}
// whether quads at multiples of four elements behind element `idx` can be read with load_raw4
__device__ __forceinline__ bool raw4_aligned(const void* base, size_t idx, int dt) {
  return dt == BQQ_F32 ? ((reinterpret_cast<uintptr_t>(base) + 4 * idx) & 15) == 0
                       : ((reinterpret_cast<uintptr_t>(base) + 2 * idx) & 7) == 0;
}
// Sum of squares of row m over this thread's share of the columns (threads tid, tid + n, ...).
__device__ __forceinline__ float row_sumsq_share(const XSource& s, int m, int tid, int nthreads) {
  float acc = 0.f;
  if ((s.n_in & 3) == 0 && raw4_aligned(s.x, (size_t)m * s.ld, s.dtype)) {
    // eight quads in flight: one round trip for 4096 columns and 128 threads
    constexpr int kAhead = 8;
    for (int n0 = 4 * tid; n0 < s.n_in; n0 += 4 * kAhead * nthreads) {
      uint4 r[kAhead];
      const bool f32 = s.dtype == BQQ_F32;
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int n = n0 + 4 * k * nthreads;
        r[k] = n < s.n_in ? load_raw4(s.x, (size_t)m * s.ld + n, f32) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        float v[4];
        raw4_to_float(r[k], s.dtype, v);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc = fmaf(v[e], v[e], acc);
      }
    }
  } else {
    for (int n = tid; n < s.n_in; n += nthreads) {
      const float v = load_as_float(s.x, (size_t)m * s.ld + n, s.dtype);
      acc = fmaf(v, v, acc);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;                                       // the warp's share, in every lane
}

}  // namespace bqq
