// Prefill forward: y[M,N] = x[M,K] @ W[N,K]^T with W rebuilt once from the packed
// planes into scratch memory, then a TMA + tcgen05 tensor-core GEMM with the fp32
// accumulator in tensor memory.  W is stored in the 16-bit format of the
// activations: fp16 (scaled by a power of two so that the bound on |W| maps to
// 2^14) for fp16 x, or as a bf16 pair hi + lo for bf16 x, in which case the K
// loop runs once per (x part, W part) pass into the same accumulator; fp32 x is
// split into bf16 hi + lo the same way (passes hi*hi, hi*lo, lo*hi).  Replaces reconstruct_W_kernel + torch::mm of
// the reference (neural_network_compression/src/bqq_cuda.cu:198-246, 367-383).
//
// GEMM kernel, one (128 MT) x BN output tile per CTA or, with a K split, per cluster of S CTAs (BN a multiple of 32 up to
// 256; MT = 1 or 2 row halves that share the B tile; plan_gemm below says which), 6 warps:
//   warp 0   TMA producer: ring of {A (128 MT)x64, B BNx64} 16-bit tiles (as many stages as fit, at most 6),
//            128-byte swizzle, completion on mbarriers
//   warp 1   allocates tensor memory (MT accumulators of BN columns); one lane issues tcgen05.mma
//            (M=128, N=BN, K=16 per instruction) and commits stage releases to mbarriers
//   warps 2-5 epilogue: tcgen05.ld 32 lanes x 32 columns, scale, bias, convert, store
// With a K split every CTA of the cluster sweeps its share of K; then the 32-column pieces of the tile are dealt out over the
// CTAs, each sends its sums of a piece to the CTA that owns it (distributed shared memory, over the operand
// ring, which is empty by then), and the owner adds them in CTA order, so results are reproducible.
// Bound: the tensor pipe for large M x N (at the clock that the power limit leaves), else operand traffic from the L2
// (64 bytes per SM and clock) and, for few tiles, the length of the K sweep.
// Every mbarrier wait is bounded by a clock budget; on expiry the kernel records
// a status code in global memory, drains its copies and returns.
//
// The call is a chain of programmatic dependent launches over column panels of W (one wave of
// GEMM tiles each): bound, rebuild panel 0, stage x, then alternately multiply panel p and rebuild
// panel p+1.  A GEMM waits for everything before it and then lets the next rebuild start at once, so the
// rebuild of a panel (ALU work) runs beside the GEMM of the previous one (TMA and tensor pipe).
#include <algorithm>
#include <cmath>

#include "bqq_tc.cuh"

namespace bqq {

constexpr int kBM = 128;
constexpr int kBK = 64;          // 64 x 2 bytes = one 128-byte swizzle row
constexpr int kGemmThreads = 192;
constexpr int kMaxStages = 6;
constexpr int kGemmSmem = 226 * 1024;    // operand ring, barriers, alignment

struct GemmParams {
  void* y;
  const void* bias;
  const float* bound_parts;  // coefficient maxima (coef_bound_kernel) when W was scaled (fp16), else NULL
  float bound_mult;          // bw * r
  const float* row_unscale;  // optional per-row factor of y (activation rows were scaled on staging)
  unsigned* status;          // device word, set nonzero when a wait timed out
  int64_t ldy;
  int y_dtype, bias_dtype;
  int M, N, K;
  int passes;                // K sweeps accumulated into one tile (1..3)
  int a_sel[3];              // per pass: 0 = first activation map, 1 = second (low half of fp32 x)
  int b_row[3];              // per pass: row offset into the stacked W map (0 = hi / only part, N = lo part)
  uint32_t idesc;
  int BN, stages, split;     // columns of a tile (a multiple of 32), ring stages, CTAs that share its K sweep (the cluster)
  int n_tile0;               // first BN-column tile of this launch (column panels of W are multiplied one after the other)
};

__device__ __forceinline__ uint32_t cluster_address(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// 32 finished sums of row m, columns nb .. of which those below n_end exist
__device__ __forceinline__ void gemm_store(const GemmParams& p, const float (&f)[32], int m, int nb, int n_end) {
  const size_t row = (size_t)m * p.ldy;
  if (nb + 32 <= n_end && p.y_dtype != BQQ_F32 && (((row + nb) * 2 + (uintptr_t)p.y) & 15) == 0) {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.y) + row + nb);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float f0 = f[g * 8 + 2 * e], f1 = f[g * 8 + 2 * e + 1];
        if (p.bias) {
          f0 += load_as_float(p.bias, nb + g * 8 + 2 * e, p.bias_dtype);
          f1 += load_as_float(p.bias, nb + g * 8 + 2 * e + 1, p.bias_dtype);
        }
        if (p.y_dtype == BQQ_BF16) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1);
          w[e] = *reinterpret_cast<const uint32_t*>(&h);
        } else {
          const __half2 h = __floats2half2_rn(f0, f1);
          w[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
      }
      dst[g] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  } else if (nb + 32 <= n_end && p.y_dtype == BQQ_F32 && (((row + nb) * 4 + (uintptr_t)p.y) & 15) == 0) {
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.y) + row + nb);
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = f[4 * g + e] + (p.bias ? load_as_float(p.bias, nb + 4 * g + e, p.bias_dtype) : 0.f);
      dst[g] = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else {
#pragma unroll
    for (int e = 0; e < 32; ++e)
      if (nb + e < n_end)
        store_from_float(p.y, row + nb + e, p.y_dtype, f[e] + (p.bias ? load_as_float(p.bias, nb + e, p.bias_dtype) : 0.f));
  }
}

template <int MT, bool PAIR>
__global__ void __launch_bounds__(kGemmThreads, 1)
bqq_gemm_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
  extern __shared__ __align__(1024) uint8_t gsm[];
  constexpr uint32_t kAHalf = kBM * kBK * 2;              // one 128-row half of the A tile
  constexpr uint32_t kABytes = MT * kAHalf;
  const int BN = p.BN;
  const int brows = PAIR ? BN / 2 : BN;                   // rows of the B tile that this CTA holds
  const uint32_t kBBytes = (uint32_t)brows * kBK * 2;
  const uint32_t acc_cols = (uint32_t)BN;                 // tensor-memory columns of one accumulator
  uint32_t tmem_cols = 32;
  while (tmem_cols < acc_cols * MT) tmem_cols *= 2;
  // 1024-byte aligned tiles (required by the 128-byte swizzle); the same offset in every CTA of a cluster
  uint8_t* base = gsm + ((1024u - (smem_u32(gsm) & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(base);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* acc_bar = empty_bar + kMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile uint32_t* failed = tmem_slot + 1;
  uint8_t* sA = base + 1024;
  uint8_t* sB = sA + p.stages * kABytes;

  // everything before this launch (the rebuilt panel of W, the staged x) has to be complete; the next kernel of the
  // stream (the rebuild of the following panel) may start now and run beside this one
  pdl_enter(kPdlWaitFirst);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned csize = (unsigned)p.split * (PAIR ? 2 : 1);
  const int crank = (int)(blockIdx.x % csize);             // rank in the cluster: (share of K, half of a pair)
  const int rank = PAIR ? crank >> 1 : crank, half = PAIR ? crank & 1 : 0;
  const int n0 = (int)(blockIdx.x / csize + p.n_tile0) * BN;
  const int n_end = min(p.N, n0 + BN);
  // row half mt of this CTA starts at m0 + mt * mstep
  constexpr int mstep = PAIR ? 2 * kBM : kBM;
  const int m0 = blockIdx.y * (kBM * MT * (PAIR ? 2 : 1)) + half * kBM;
  const int kblocks = (p.K + kBK - 1) / kBK;
  const int all = kblocks * p.passes;
  const int it0 = (int)((long long)all * rank / p.split), it1 = (int)((long long)all * (rank + 1) / p.split);
  const int iters = it1 - it0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
    mbar_init(acc_bar, 1);
    *failed = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();                  // the leader's barriers are initialised before the other half's copies report
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0, issued = 0;
      uint32_t ph = 1u;
      int kb = it0 % kblocks, pass = it0 / kblocks;
      for (int it = 0; it < iters; ++it) {
        if (*failed || !mbar_wait(empty_bar + s, ph)) { *failed = 1; break; }
        const CUtensorMap* ma = p.a_sel[pass] == 0 ? &map_a0 : &map_a1;
        if (PAIR) {
          if (half == 0) mbar_expect_tx(full_bar + s, 2 * (kABytes + kBBytes));
          const uint32_t bar = cluster_address(smem_u32(full_bar + s), (uint32_t)(crank & ~1));
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
            tma_load_2d_pair(sA + s * kABytes + mt * kAHalf, ma, bar, kb * kBK, m0 + mt * mstep);
          tma_load_2d_pair(sB + s * kBBytes, &map_b, bar, kb * kBK, p.b_row[pass] + n0 + half * brows);
        } else {
          mbar_expect_tx(full_bar + s, kABytes + kBBytes);
          tma_load_2d(sA + s * kABytes, ma, full_bar + s, kb * kBK, m0);
          tma_load_2d(sB + s * kBBytes, &map_b, full_bar + s, kb * kBK, p.b_row[pass] + n0);
        }
        issued = it + 1;
        if (++kb == kblocks) { kb = 0; ++pass; }
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
      if (*failed && half == 0) {
        // drain: copies already issued must land before the CTA exits (the leader's barriers count those of both halves,
        // which leave together)
        int first = issued > p.stages ? issued - p.stages : 0;
        for (int it = first; it < issued; ++it)
          mbar_wait(full_bar + it % p.stages, (uint32_t)(it / p.stages) & 1u);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && half == 0) {
      const uint16_t both = (uint16_t)(3u << (crank & ~1));
      int s = 0;
      uint32_t ph = 0;
      for (int it = 0; it < iters; ++it) {
        if (*failed || !mbar_wait(full_bar + s, ph)) { *failed = 1; break; }
        tc_fence_after();
        const uint64_t bdesc = make_smem_desc(smem_u32(sB + s * kBBytes));
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const uint64_t adesc = make_smem_desc(smem_u32(sA + s * kABytes + mt * kAHalf));
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) { // 16 elements = 32 bytes = 2 descriptor units per step
            const uint32_t d = tmem_base + (uint32_t)mt * acc_cols, accum = (it | k) != 0 ? 1u : 0u;
            if (PAIR) tc_mma_f16_pair(d, adesc + 2 * k, bdesc + 2 * k, p.idesc, accum);
            else tc_mma_f16(d, adesc + 2 * k, bdesc + 2 * k, p.idesc, accum);
          }
        }
        // frees the stage when these MMAs have read it
        if (PAIR) tc_commit_pair(empty_bar + s, both);
        else tc_commit(empty_bar + s);
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
      // accumulators complete (or abandoned)
      if (PAIR) tc_commit_pair(acc_bar, both);
      else tc_commit(acc_bar);
    }
  } else {
    ok = mbar_wait(acc_bar, 0) && !*failed;
    if (!ok) *failed = 1;
    tc_fence_after();
  }
  __syncwarp();
  if (p.split > 1) cluster_sync();           // every CTA's ring is empty: it can take sums now

  const int quarter = warp & 3;              // epilogue warps 2..5 own tensor-memory lanes 32*(warp%4) .. +31
  const int cpt = BN / 32, pieces = MT * cpt;
  const uint32_t mine = tmem_base + ((uint32_t)(quarter * 32) << 16);
  float w_unscale = 1.f;
  if (warp >= 2 && p.bound_parts) w_unscale = 1.f / w_scale_from_maxima(p.bound_parts, p.bound_mult, lane);
  // sums of a piece from one CTA: [8 groups of 4 columns][128 rows][4], so that a warp's 16-byte accesses are adjacent
  constexpr uint32_t kPiece = 32 * kBM * 4;
  if (p.split == 1) {
    if (warp >= 2 && ok) {
#pragma unroll 1
      for (int q = 0; q < pieces; ++q) {
        const int mt = q / cpt, c = q - mt * cpt;
        const int m = m0 + mt * mstep + quarter * 32 + lane;
        uint32_t v[32];
        tc_ld32(mine + (uint32_t)mt * acc_cols + (uint32_t)(c * 32), v);
        tc_wait_ld();
        if (m < p.M && n0 + c * 32 < n_end) {
          const float f = w_unscale * (p.row_unscale ? p.row_unscale[m] : 1.f);
          float o[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __uint_as_float(v[e]) * f;
          gemm_store(p, o, m, n0 + c * 32, n_end);
        }
        __syncwarp();
      }
    }
  } else {
    if (warp >= 2) {
      const uint32_t slot0 = smem_u32(sA) + (uint32_t)rank * kPiece + (uint32_t)(quarter * 32 + lane) * 16;
#pragma unroll 1
      for (int q = 0; q < pieces; ++q) {
        const int mt = q / cpt, c = q - mt * cpt;
        uint32_t v[32];
        tc_ld32(mine + (uint32_t)mt * acc_cols + (uint32_t)(c * 32), v);
        tc_wait_ld();
        const uint32_t dst = cluster_address(slot0 + (uint32_t)(q / p.split) * (uint32_t)p.split * kPiece, (uint32_t)(q % p.split));
#pragma unroll
        for (int g = 0; g < 8; ++g)
          asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                       ::"r"(dst + g * (kBM * 16)), "r"(v[4 * g]), "r"(v[4 * g + 1]), "r"(v[4 * g + 2]), "r"(v[4 * g + 3]) : "memory");
      }
    }
    __syncwarp();
    cluster_sync();                          // all sums have arrived
    if (warp >= 2 && ok) {
#pragma unroll 1
      for (int q = rank; q < pieces; q += p.split) {
        const int mt = q / cpt, c = q - mt * cpt;
        const int m = m0 + mt * mstep + quarter * 32 + lane;
        if (m >= p.M || n0 + c * 32 >= n_end) continue;
        const uint8_t* src = sA + (size_t)(q / p.split) * p.split * kPiece + (quarter * 32 + lane) * 16;
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = 0.f;
#pragma unroll 1
        for (int r = 0; r < p.split; ++r, src += kPiece)
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float4 u = *reinterpret_cast<const float4*>(src + g * (kBM * 16));
            o[4 * g] += u.x; o[4 * g + 1] += u.y; o[4 * g + 2] += u.z; o[4 * g + 3] += u.w;
          }
        const float f = w_unscale * (p.row_unscale ? p.row_unscale[m] : 1.f);
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] *= f;
        gemm_store(p, o, m, n0 + c * 32, n_end);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
  if (threadIdx.x == 0 && *failed) atomicExch(p.status, 1u);
  if (PAIR) cluster_sync();                  // neither half leaves while the other may still signal it
}

// ---- x staging: any dtype / stride -> dense 16-bit rows (hi, lo for fp32) ----
// Bound: memory.  Four columns per thread (K is a multiple of 8), rows in steps of gridDim.y; one element per thread with a
// 64-bit division for its place cost 8 us of 106 (4096 x 4096, 1000 rows of fp32, whole call).
constexpr int kStageThreads = 128;
__global__ void __launch_bounds__(kStageThreads)
stage_x_kernel(const void* __restrict__ x, int x_dtype, int64_t ldx, int M, int K, int vec, uint16_t* __restrict__ hi,
               uint16_t* __restrict__ lo) {
  pdl_enter(kPdlOverlap);
  const int k = (blockIdx.x * kStageThreads + threadIdx.x) * 4;
  if (k < K)
    for (int m = blockIdx.y; m < M; m += gridDim.y) {
      const size_t from = (size_t)m * ldx + k, to = (size_t)m * K + k;
      if (x_dtype == BQQ_F32) {
        const float* row = reinterpret_cast<const float*>(x) + from;
        const float4 v = vec ? *reinterpret_cast<const float4*>(row) : make_float4(row[0], row[1], row[2], row[3]);
        const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
        const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - __low2float(h0), v.y - __high2float(h0));
        const __nv_bfloat162 l1 = __floats2bfloat162_rn(v.z - __low2float(h1), v.w - __high2float(h1));
        *reinterpret_cast<uint2*>(hi + to) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
        *reinterpret_cast<uint2*>(lo + to) = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
      } else {
        const uint16_t* row = reinterpret_cast<const uint16_t*>(x) + from;
        *reinterpret_cast<uint2*>(hi + to) = vec ? *reinterpret_cast<const uint2*>(row)
                                                 : make_uint2(row[0] | (uint32_t)row[1] << 16, row[2] | (uint32_t)row[3] << 16);
      }
    }
  pdl_exit(kPdlOverlap);
}

// bf16 rows -> fp16 rows scaled by a per-row power of two (max |x| of the row maps to at most 2^14,
// so nothing overflows and every bf16 value in range converts exactly); row_unscale[m] = 1 / scale.
// One block per row; with `vec` a thread moves 8 values per access and keeps its first kStageKeep
// accesses in registers, so rows up to 8 * kStageKeep * blockDim.x values are read once.
constexpr int kStageKeep = 4;
__global__ void __launch_bounds__(kStageThreads)
stage_x_bf16_to_f16_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, int M, int K,
                           __half* __restrict__ out, float* __restrict__ row_unscale, int vec) {
  __shared__ float warp_max[kStageThreads / 32];
  pdl_enter(kPdlOverlap);
  const int tid = threadIdx.x, lane = tid & 31;
  for (int m = blockIdx.x; m < M; m += gridDim.x) {
    const __nv_bfloat16* row = x + (size_t)m * ldx;
    const uint4* row8 = reinterpret_cast<const uint4*>(row);
    const int K8 = K >> 3;
    uint4 keep[kStageKeep];
    float amax = 0.f;
    if (vec) {
#pragma unroll
      for (int s = 0; s < kStageKeep; ++s) {
        const int k = tid + s * kStageThreads;
        keep[s] = k < K8 ? row8[k] : make_uint4(0u, 0u, 0u, 0u);
      }
      for (int k = tid + kStageKeep * kStageThreads; k < K8; k += kStageThreads) {
        const uint4 v = row8[k];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(w[e] << 16)), fabsf(__uint_as_float(w[e] & 0xFFFF0000u))));
      }
#pragma unroll
      for (int s = 0; s < kStageKeep; ++s) {
        const uint32_t w[4] = {keep[s].x, keep[s].y, keep[s].z, keep[s].w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(w[e] << 16)), fabsf(__uint_as_float(w[e] & 0xFFFF0000u))));
      }
    } else {
      for (int k = tid; k < K; k += kStageThreads) amax = fmaxf(amax, fabsf(__bfloat162float(row[k])));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    __syncthreads();                               // the previous row's readers are done with warp_max
    if (lane == 0) warp_max[tid >> 5] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kStageThreads / 32; ++w) amax = fmaxf(amax, warp_max[w]);
    float scale = 1.f;
    if (amax > 0.f && isfinite(amax)) {
      int e;
      frexpf(amax, &e);                        // amax = f * 2^e, f in [0.5, 1)
      scale = exp2f((float)max(-100, min(100, 14 - e)));
    }
    if (vec) {
      uint4* out8 = reinterpret_cast<uint4*>(out + (size_t)m * K);
      auto convert = [scale](const uint4& v) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t h[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __half2 t = __floats2half2_rn(__uint_as_float(w[e] << 16) * scale,
                                              __uint_as_float(w[e] & 0xFFFF0000u) * scale);
          h[e] = *reinterpret_cast<const uint32_t*>(&t);
        }
        return make_uint4(h[0], h[1], h[2], h[3]);
      };
#pragma unroll
      for (int s = 0; s < kStageKeep; ++s) {
        const int k = tid + s * kStageThreads;
        if (k < K8) out8[k] = convert(keep[s]);
      }
      for (int k = tid + kStageKeep * kStageThreads; k < K8; k += kStageThreads) out8[k] = convert(row8[k]);
    } else {
      for (int k = tid; k < K; k += kStageThreads) out[(size_t)m * K + k] = __float2half_rn(__bfloat162float(row[k]) * scale);
    }
    if (tid == 0) row_unscale[m] = 1.f / scale;
  }
  pdl_exit(kPdlOverlap);
}

// ---- host side -----------------------------------------------------------------
static inline size_t up256(size_t v) { return (v + 255) / 256 * 256; }

// workspace: [kPrefillHead bytes: status word, coefficient maxima at + 256][W parts 2 x N x K 16-bit][x hi M x K][x lo M x K]
constexpr size_t kPrefillHead = 256 + 2 * kBoundBlocks * 4;
size_t prefill_workspace_bytes(const BqqDims* dims, int M) {
  Geom g(*dims);
  const size_t K = g.in_features();
  const size_t need = kPrefillHead + up256((size_t)2 * g.out_features() * K * 2) + 2 * up256((size_t)M * K * 2);
  if (M > kFusedMaxM) return need;
  return std::max(need, kPrefillHead + up256(fused_counter_words(g) * 4) + fused_workspace_bytes(g, M));
}

struct GemmPlan {
  int BN, MT, split, pair, stages;
  size_t smem;
};

// Column panels: W is rebuilt and multiplied panel by panel, so that the rebuild of panel p + 1 runs beside the GEMM of panel
// p.  Tiles of a panel along N: what fills the SMs once, but at most eight panels.
static int panel_tiles(int tm, int tn) {
  if ((long long)tm * tn <= 222) return tn;                       // one wave and a half: not worth another rebuild launch
  const int tpp = std::max(std::max(1, 148 / tm), (tn + 7) / 8);
  const int panels = (tn + tpp - 1) / tpp;
  return (tn + panels - 1) / panels;
}
// CTA pairs (cta_group::2) load half of the B tile each.  That is worth the pairing where W does not fit the half of the L2 that
// is near an SM: 8192 x 4096 at 2048 rows 168.9 -> 164.5 us, 4096^2 at 1000 rows of fp32 118 -> 111, smaller W no difference.
constexpr size_t kPairBytes = 64u << 20;
// Tile and K split with the smallest estimated time, in SM clocks.  A k-block of 64 costs a CTA the largest of its products
// (3.5 clocks per column and row half; the tensor peak would be 2, the waits of the ring and the power limit are in it), its
// operands at 65 bytes per clock, and its share of the L2 (7300 bytes per clock for all SMs).  To that come the start of the
// CTA, the stores of a 32-column piece, for a K split (one row half only) two cluster barriers and the exchange of the
// pieces, and 43000 clocks per panel.  Clusters do not fill all 148 SMs (kSlots: what the occupancy query reports for this
// kernel).  The constants were fitted to 32 shapes (288 to 28672 outputs, 140 to 4096 rows, every tile and split timed): the
// choice is within 1 % of the best on average, 5 % at worst.
// Measured, whole forward, against the power-of-two tiles without a split (us): 2048 x 2048, 3 bit layers, 333 rows of fp32
// 57.6 -> 34; 1024 x 9632, 4 bit layers, 1422 rows of bf16 82.6 -> 61.  Panels of one wave each instead of at most four:
// 14336 x 4096, 2048 rows 335 -> 240; 8192 x 4096, 2048 rows 181 -> 141.
static GemmPlan plan_gemm(int M, int N, int kblocks, size_t w_bytes) {
  static const int kSlots[9] = {0, 148, 148, 135, 132, 130, 132, 105, 120};
  GemmPlan best = {};
  double best_cost = 0;
  for (int MT = 1; MT <= 2; ++MT)
    for (int BN = 32; BN <= 256; BN += 32) {
      const int tm = (M + kBM * MT - 1) / (kBM * MT), tn = (N + BN - 1) / BN;
      const size_t stage = (size_t)MT * kBM * kBK * 2 + (size_t)BN * kBK * 2;
      const int pieces = MT * BN / 32;
      for (int S = 1; S <= 8; ++S) {
        const size_t sums = S > 1 ? (size_t)((pieces + S - 1) / S) * S * 32 * kBM * 4 : 0;
        if (sums + 2048 > (size_t)kGemmSmem || (S > 1 && (MT > 1 || kblocks / S < 4))) continue;
        const double ctas = (double)tm * tn * S, slots = kSlots[S];
        const int tpp = S > 1 ? tn : panel_tiles(tm, tn);
        const int panels = (tn + tpp - 1) / tpp;
        const double waves = panels > 1 ? (double)panels * ((tpp * tm + 147) / 148) : std::ceil(ctas / slots);
        const double busy = std::min(panels > 1 ? (double)tpp * tm : ctas, slots);
        const double block = std::max(3.5 * BN * MT, stage * std::max(1 / 65.0, busy / 7300.0));
        const double tail = 7000.0 + 470.0 * pieces + (S > 1 ? 1750.0 + 180.0 * pieces : 0.0);
        const double cost = waves * ((kblocks + S - 1) / S * block + tail) + 43000.0 * panels;
        if (best.BN == 0 || cost < best_cost) {
          best_cost = cost;
          best = {BN, MT, S, (S == 1 && tm % 2 == 0 && w_bytes >= kPairBytes) ? 1 : 0, 0, 0};
        }
      }
    }
  const size_t stage = (size_t)best.MT * kBM * kBK * 2 + (size_t)best.BN / (best.pair ? 2 : 1) * kBK * 2;
  const int pieces = best.MT * best.BN / 32;
  best.stages = (int)std::min<size_t>(kMaxStages, (kGemmSmem - 2048) / stage);
  const size_t sums = best.split > 1 ? (size_t)((pieces + best.split - 1) / best.split) * best.split * 32 * kBM * 4 : 0;
  best.smem = 2048 + std::max((size_t)best.stages * stage, sums);
  // a CTA of a pair is alone on its SM: two pairs that wait for each other's tensor memory cannot meet
  if (best.pair) best.smem = std::max(best.smem, (size_t)116 * 1024);
  return best;
}

// tiles [tile0, tile0 + ntiles) along N, all of M
static int launch_gemm(const GemmPlan& pl, const CUtensorMap& a0, const CUtensorMap& a1, const CUtensorMap& b, GemmParams p,
                       int tile0, int ntiles, cudaStream_t st) {
  auto kern = pl.pair ? (pl.MT == 2 ? bqq_gemm_kernel<2, true> : bqq_gemm_kernel<1, true>)
                      : (pl.MT == 2 ? bqq_gemm_kernel<2, false> : bqq_gemm_kernel<1, false>);
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem) != cudaSuccess) return BQQ_ERR_CUDA;
  p.n_tile0 = tile0;
  cudaLaunchAttribute attr[2] = {pdl_attribute()};
  attr[1].id = cudaLaunchAttributeClusterDimension;
  const int cluster = pl.split * (pl.pair ? 2 : 1), rows = kBM * pl.MT * (pl.pair ? 2 : 1);
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ntiles * cluster, (p.M + rows - 1) / rows);
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kern, a0, a1, b, p) != cudaSuccess) { cudaGetLastError(); return BQQ_ERR_CUDA; }
  return launch_status();
}

int prefill_launch(const BqqLayer* L, const void* x, int x_dtype, int M, int64_t ldx, void* y, int y_dtype,
                   int64_t ldy, void* ws, size_t ws_bytes, cudaStream_t st) {
  Geom g(L->dims);
  const int N = g.out_features(), K = g.in_features();
  if (!ws || ws_bytes < prefill_workspace_bytes(&L->dims, M)) return BQQ_ERR_WORKSPACE;
  if (((uintptr_t)ws & 255) != 0) return BQQ_ERR_MISALIGNED;
  uint8_t* wsb = reinterpret_cast<uint8_t*>(ws);
  unsigned* status = reinterpret_cast<unsigned*>(wsb);
  uint16_t* W = reinterpret_cast<uint16_t*>(wsb + kPrefillHead);              // [2][N][K]: hi rows, then lo rows
  uint16_t* xhi = reinterpret_cast<uint16_t*>(wsb + kPrefillHead + up256((size_t)2 * N * K * 2));
  uint16_t* xlo = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(xhi) + up256((size_t)M * K * 2));
  float* bound_parts = reinterpret_cast<float*>(wsb + 256);
  if (M <= kFusedMaxM) {
    const size_t cw = up256(fused_counter_words(g) * 4);
    const int rc = fused_launch(L, x, x_dtype, M, ldx, y, y_dtype, ldy, reinterpret_cast<unsigned*>(wsb + kPrefillHead), status, true,
                                wsb + kPrefillHead + cw, nullptr, st);
    if (rc != BQQ_ERR_UNSUPPORTED) return rc;
  }
  if (K % 8 != 0) return BQQ_ERR_UNSUPPORTED;   // 16-byte row pitch for the TMA descriptors

  const bool f16 = x_dtype != BQQ_F32;
  const bool split_x = x_dtype == BQQ_F32;
  const GemmPlan pl = plan_gemm(M, N, (K + kBK - 1) / kBK * (split_x ? 3 : 1), (size_t)N * K * (split_x ? 4 : 2));
  const int BN = pl.BN;
  // a row patch that a panel border cuts is rebuilt with the first of the two panels
  const int tiles_n = (N + BN - 1) / BN, tiles_m = (M + kBM * pl.MT - 1) / (kBM * pl.MT);
  const int tiles_pp = pl.split > 1 ? tiles_n : panel_tiles(tiles_m, tiles_n);
  const int panels = (tiles_n + tiles_pp - 1) / tiles_pp;
  auto panel_rows = [&](int pnl, int* i0, int* i1) {           // row patches of panel pnl
    const int c0 = pnl * tiles_pp * BN, c1 = std::min(N, (pnl + 1) * tiles_pp * BN);
    *i0 = (c0 + g.P - 1) / g.P;
    *i1 = (c1 + g.P - 1) / g.P;
  };

  // x: fp16 is used in place when its pitch suits TMA; everything else is staged
  const bool direct = x_dtype == BQQ_F16 && (ldx % 8) == 0 && ((uintptr_t)x & 15) == 0;
  const void* a_ptr = direct ? x : (const void*)xhi;
  const int64_t a_ld = direct ? ldx : (int64_t)K;
  float* unscale = reinterpret_cast<float*>(xlo);            // the lo region is free when x has 16 bits
  const float* row_unscale = x_dtype == BQQ_BF16 ? unscale : nullptr;

  const uint32_t abox = pl.pair ? kBM : kBM * pl.MT;
  CUtensorMap ma0, ma1, mb;
  int rc = make_map(&ma0, a_ptr, !f16, (uint64_t)M, (uint64_t)K, (uint64_t)a_ld, abox);
  if (rc) return rc;
  rc = make_map(&ma1, split_x ? (const void*)xlo : a_ptr, !f16, (uint64_t)M, (uint64_t)K,
                split_x ? (uint64_t)K : (uint64_t)a_ld, abox);
  if (rc) return rc;
  rc = make_map(&mb, W, !f16, (uint64_t)(f16 ? N : 2 * N), (uint64_t)K, (uint64_t)K, (uint32_t)(pl.pair ? BN / 2 : BN));
  if (rc) return rc;

  GemmParams p;
  p.y = y; p.bias = L->bias; p.bound_parts = f16 ? bound_parts : nullptr; p.bound_mult = (float)(g.bw * g.r);
  p.status = status;
  p.row_unscale = row_unscale;
  p.ldy = ldy; p.y_dtype = y_dtype; p.bias_dtype = L->bias_dtype;
  p.M = M; p.N = N; p.K = K;
  p.n_tile0 = 0;
  p.BN = BN; p.stages = pl.stages; p.split = pl.split;
  for (int i = 0; i < 3; ++i) { p.a_sel[i] = 0; p.b_row[i] = 0; }
  if (f16) {
    p.passes = 1;
  } else {
    p.passes = 3; p.b_row[1] = N; p.a_sel[2] = 1;       // xhi*Whi + xhi*Wlo + xlo*Whi
  }
  // instruction descriptor: fp32 accumulate, A and B in the same 16-bit format, both K-major
  const uint32_t fmt = f16 ? 0u : 1u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((pl.pair ? 2 * kBM : kBM) >> 4) << 24);

  // 1. (16-bit x) bound on |W| for the power-of-two scale of the fp16 weight.  fp16 and bf16 activations use one
  //    fp16 W (bf16 rows are re-staged as scaled fp16, exact); fp32 activations use the bf16 hi + lo pair.
  //    The same kernel clears the status word.
  rc = coef_bound_launch(L, f16 ? bound_parts : nullptr, status, st);
  if (rc) return rc;
  // 2. panel 0 of W: waits for the bound (and for whatever preceded this call in the stream)
  auto rebuild = [&](int pnl, int pdl) {
    int i0, i1;
    panel_rows(pnl, &i0, &i1);
    return f16 ? reconstruct_launch(L, W, nullptr, BQQ_F16, 1.f, bound_parts, st, i0, i1, pdl, status)
               : reconstruct_launch(L, W, W + (size_t)N * K, BQQ_BF16, 1.f, nullptr, st, i0, i1, pdl, status);
  };
  rc = rebuild(0, kPdlWaitFirst);
  if (rc) return rc;
  // 3. x staging, beside the rebuild of panel 0
  if (x_dtype == BQQ_BF16) {
    const int vec = (K % 8 == 0 && ldx % 8 == 0 && ((uintptr_t)x & 15) == 0) ? 1 : 0;
    cudaLaunchAttribute attr[1] = {pdl_attribute()};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M);
    cfg.blockDim = dim3(kStageThreads);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, stage_x_bf16_to_f16_kernel, reinterpret_cast<const __nv_bfloat16*>(x), ldx, M, K,
                           reinterpret_cast<__half*>(xhi), unscale, vec) != cudaSuccess) { cudaGetLastError(); return BQQ_ERR_CUDA; }
  } else if (!direct) {
    const uintptr_t quad = 4 * (uintptr_t)dtype_size(x_dtype) - 1;
    const int vec = ldx % 4 == 0 && ((uintptr_t)x & quad) == 0;
    const int parts = (K / 4 + kStageThreads - 1) / kStageThreads;
    cudaLaunchAttribute attr[1] = {pdl_attribute()};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)parts, (unsigned)std::min(M, std::max(1, 148 * 16 / parts)));
    cfg.blockDim = dim3(kStageThreads);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, stage_x_kernel, x, x_dtype, ldx, M, K, vec, xhi, xlo) != cudaSuccess) {
      cudaGetLastError();
      return BQQ_ERR_CUDA;
    }
  }
  rc = launch_status();
  if (rc) return rc;
  // 4. alternately: multiply panel p (waits for everything before it, then lets its successor start), rebuild
  //    panel p+1 beside it (its last CTA waits for that GEMM, so the next GEMM's wait covers both)
  for (int pnl = 0; pnl < panels; ++pnl) {
    const int tile0 = pnl * tiles_pp, ntiles = std::min(tiles_pp, tiles_n - tile0);
    rc = launch_gemm(pl, ma0, ma1, mb, p, tile0, ntiles, st);
    if (rc) return rc;
    if (pnl + 1 < panels) {
      rc = rebuild(pnl + 1, kPdlOverlap);
      if (rc) return rc;
    }
  }
  return BQQ_OK;
}

}  // namespace bqq
