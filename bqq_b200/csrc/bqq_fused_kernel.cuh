// Forward for a few rows up to a few dozen: the dense weight exists only as tiles in tensor memory.
//   y[m, o] = sum_k W[o, k] x[m, k],  W rebuilt from the planes tile by tile and multiplied by tcgen05 at once.
// Replaces the M > 1 branch of bqq_forward (neural_network_compression/src/bqq_cuda.cu:327-383) for these batches.
//
// Bound: the rebuild (bqq_rebuild.cuh: issue slots and the int8 tensor pipe), which does not depend on the number of
// rows; the product with x is a few per cent of the tcgen05 rate.  The decode kernel pays per row of X (its second
// operand has to be cut into digits for every row), and a rebuild into memory pays for writing and re-reading W.
//
// A tile is 128 rows of W: four blocks of 32 rows (R = 4 tile + rb: row patch R / PT, block R % PT).  K is walked in
// stages of 128 columns: one super-group (four col patches) at one 32-column block position,
//   k' = ((jg QT + qt) 4 + sub) 32 + c   <->   column (4 jg + sub) Q + 32 qt + c,
// which is the order of x itself for patches of 32 columns; other patches have x staged in that order, zeros in the
// padding.  CTA = 16 compute warps (row block x col patch: one 32x32 block of W per stage each) and four
// helpers: plane words by TMA ([Y of all row blocks | Z of all] [bit] in a stage), coefficients as floats, x by TMA,
// tcgen05 issue.  W is operand A and lives in tensor memory (lane = row, two neighbouring k per column): the registers of a
// finished 32x32 block are what two 16x256b stores take, against sixteen 4-byte stores into swizzled shared memory, a
// proxy fence and up to 128 KB of buffers before.  Two to four W buffers, two sets of accumulators D[128 rows of W][N
// rows of x] beside them.
// Formats, accumulated in fp32 (NP products per tile):
//   1  W in fp16, x in fp16: 16-bit x of more than 16 rows.  Every block of 32 rows of an item is scaled by a power of two
//      (the bound on its entries maps to 2^14), bf16 rows of x are too; both are taken out of the sums.
//   2  W as bf16 hi + lo (16 bits), x in bf16 as it is;   3  the same with x as hi + lo.  Up to 16 rows, and fp32 x.
//
// Work items are (tile, chunk of K).  Chunks depend on K only, never on the number of rows of W, and their sums are added
// in order by the CTA that finishes a tile last, so a row shard gives the same bits as the whole layer.  CTAs walk the
// items; the sums of an item leave tensor memory while the next item is already being rebuilt, and the chunks are added up
// at the end.
// Measured (us, before -> with this kernel, W in shared memory -> in tensor memory): 8192 x 28672, 3 bit layers of rank 64,
// 32 rows 461 (rebuild into memory and GEMM) -> 375 -> 327; 4096 x 4096, 2 bit layers, 64 rows 43.3 -> 27.3 -> 26.0;
// 4096 x 14336, 3 bit layers, 16 rows 104.7 (decode kernel) -> 75.8 -> 66.4; P = 96, Q = 40, r = 33, 5 rows 25.0 -> 19.2.
#pragma once
#include "bqq_rebuild.cuh"
#include "bqq_tc.cuh"

namespace bqq {

constexpr int kFusedWarps = 16;
constexpr int kFusedThreads = (kFusedWarps + 8) * 32;
// registers: 768 threads are launched with 80 each; the helpers give some of theirs to the compute warps
constexpr int kFusedComputeRegs = 104, kFusedHelperRegs = 24, kFusedSumRegs = 40;
static_assert(kFusedWarps * kFusedComputeRegs + 4 * (kFusedHelperRegs + kFusedSumRegs) <= (kFusedWarps + 8) * 80, "more than was launched with");
constexpr int kFusedMaxItems = 48;                   // finished tiles that a CTA keeps for the end
constexpr int kFusedMaxPlaneStages = 4;
constexpr int kFusedBits = 8;                        // bit layers of a plane stage at most
constexpr int kFusedMaxN = 128;                      // rows of x (padded to 16)
constexpr int kFusedTile = 128;
constexpr int kFusedStageCols = 128;

struct FusedParams {
  const uint32_t* zp;
  const uint32_t* yp;
  const void *a, *b, *c, *d;
  const void* bias;
  const void* res;
  void* y;
  float* partial;              // [tile][chunk][N][128] when there are several chunks
  unsigned* counters;          // [tile], zero, left zero
  unsigned* status;            // set non-zero when a bounded wait gave up
  int64_t ldy, ld_res;
  int coef_dtype, bias_dtype, y_dtype, res_dtype;
  Geom g;
  int M, N;
  int nb, ns, nx;              // bit layers per plane stage; plane stages; x stages
  const float* row_unscale;    // NP = 1: factor of every row of x, or NULL
  int joint;                   // 1: one copy brings the planes of the tile's four row patches (PT = 1, all bit layers)
  int tiles, chunks, chunk_stages, stages;   // stages = JG * QT in all
  uint32_t idesc;
};

// Shared-memory layout in bytes, host and device.
struct FusedSmem {
  int x, planes, coef, total;
  int x_part, x_stage, plane_group, plane_stage, coef_stage;
  __host__ __device__ FusedSmem(int NP, int RT, int N, int nb, int ns, int nx) {
    x_part = N * kFusedStageCols * 2;
    x_stage = x_part * (NP == 3 ? 2 : 1);
    plane_group = nb * RT * 1024;
    plane_stage = 4 * plane_group;
    coef_stage = 4 * nb * kGroup * 16;
    int o = 1024;                                              // barriers and flags (the base is rounded up to 1024)
    x = o; o += nx * x_stage;
    planes = o; o += ns * plane_stage;
    coef = o; o += ns * coef_stage;
    total = o + 1024;
  }
};

__device__ __forceinline__ void store_shared_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Position in a ring of `n` slots.
struct RingPos {
  int slot;
  uint32_t phase;
  __device__ __forceinline__ RingPos() : slot(0), phase(0) {}
  __device__ __forceinline__ void next(int n) {
    if (++slot == n) { slot = 0; phase ^= 1u; }
  }
};

// One finished value of row m, local output row o (bias included by the caller).
__device__ __forceinline__ void fused_out(const FusedParams& p, int m, int o, float v) {
  if (p.res) v += load_as_float(p.res, (size_t)m * p.ld_res + o, p.res_dtype);
  store_from_float(p.y, (size_t)m * p.ldy + o, p.y_dtype, v);
}

// The sums of a finished tile: chunks added in order, four neighbouring rows of W per thread.  rowf: factors of the rows of x.
__device__ __forceinline__ void fused_reduce_tile(const FusedParams& p, int tile, int tid, int nthreads, const float* rowf) {
  const Geom& g = p.g;
  const float4* all = reinterpret_cast<const float4*>(p.partial) + (size_t)tile * p.chunks * p.N * (kFusedTile / 4);
  const size_t step = (size_t)p.N * (kFusedTile / 4);
  const int r4 = tid & 31;
  const int R = tile * 4 + (r4 >> 3), i = R / g.PT, pt = R - i * g.PT;
  const int p0 = 4 * (r4 & 7), left = i < g.rw ? min(4, g.P - 32 * pt - p0) : 0;       // rows of the four that exist
  const int o = i * g.P + 32 * pt + p0;
  float bias[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) bias[e] = p.bias && e < left ? load_as_float(p.bias, o + e, p.bias_dtype) : 0.f;
  const bool vec = left == 4 && !p.res && p.y_dtype != BQQ_F32 && ((((uintptr_t)p.y) | (uintptr_t)(2 * p.ldy) | (uintptr_t)(2 * o)) & 7) == 0;
  for (int m = tid >> 5; m < p.M; m += nthreads >> 5) {
    const float4* at = all + (size_t)m * 32 + r4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = 0; c < p.chunks; c += 4) {
      float4 u[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) u[e] = c + e < p.chunks ? __ldcg(at + (c + e) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int e = 0; e < 4; ++e) { v.x += u[e].x; v.y += u[e].y; v.z += u[e].z; v.w += u[e].w; }
    }
    const float f = rowf[m];
    const float w[4] = {fmaf(v.x, f, bias[0]), fmaf(v.y, f, bias[1]), fmaf(v.z, f, bias[2]), fmaf(v.w, f, bias[3])};
    if (vec) {
      uint32_t h[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (p.y_dtype == BQQ_BF16) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(w[2 * e], w[2 * e + 1]);
          h[e] = *reinterpret_cast<const uint32_t*>(&b);
        } else {
          const __half2 b = __floats2half2_rn(w[2 * e], w[2 * e + 1]);
          h[e] = *reinterpret_cast<const uint32_t*>(&b);
        }
      }
      *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.y) + (size_t)m * p.ldy + o) = make_uint2(h[0], h[1]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < left) fused_out(p, m, o + e, w[e]);
    }
  }
}

template <int NP, int RT>
__global__ void __launch_bounds__(kFusedThreads, 1)
bqq_fused_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                 const __grid_constant__ CUtensorMap map_y, const __grid_constant__ CUtensorMap map_z, const FusedParams p) {
  extern __shared__ __align__(1024) uint8_t fsm[];
  uint8_t* base = fsm + ((1024u - (smem_u32(fsm) & 1023u)) & 1023u);   // (pointer arithmetic: stays a shared address)
  const FusedSmem L(NP, RT, p.N, p.nb, p.ns, p.nx);
  uint64_t* full = reinterpret_cast<uint64_t*>(base);                   // planes and coefficients of a stage are there
  uint64_t* used = full + kFusedMaxPlaneStages;
  uint64_t* xfull = used + kFusedMaxPlaneStages;                        // x of a stage
  uint64_t* xfree = xfull + 4;
  uint64_t* wfull = xfree + 4;                                          // W buffer written / read by the MMAs
  uint64_t* wfree = wfull + 4;
  uint64_t* accfull = wfree + 4;                                        // accumulator set complete / read out
  uint64_t* accfree = accfull + 2;
  uint64_t* scaled = accfree + 2;                                       // scales of an item are there (NP = 1)
  float* wscale = reinterpret_cast<float*>(scaled + 2);                 // [set][row block]
  uint64_t* tail = reinterpret_cast<uint64_t*>(wscale + 8);             // the last item of this CTA has left tensor memory
  float* rowf = reinterpret_cast<float*>(tail + 1);                     // factor of every row of x
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rowf + kFusedMaxN);
  volatile uint32_t* failed = tmem_slot + 1;
  int* nfinished = reinterpret_cast<int*>(tmem_slot + 2);               // tiles that this CTA was the last to add to
  int* finished = nfinished + 1;
  constexpr int kBitBytes = RT * 1024;
  const Geom& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = p.tiles * p.chunks;
  const int nchunks = (g.bw + p.nb - 1) / p.nb;                         // plane stages of a block
  const uint32_t acc_cols = (uint32_t)(p.N <= 16 ? 16 : p.N <= 32 ? 32 : p.N <= 64 ? 64 : 128);
  constexpr uint32_t kWPart = kFusedStageCols / 2;                      // tensor-memory columns of a W buffer: hi, then lo
  constexpr uint32_t kWCols = NP == 1 ? kWPart : 2 * kWPart;
  const int wbufs = NP == 1 ? 4 : acc_cols > 64 ? 2 : 3;
  constexpr uint32_t tmem_cols = 512;
  static_assert(256 + 4 * kWPart <= tmem_cols && 256 + 2 * 2 * kWPart <= tmem_cols && 128 + 3 * 2 * kWPart <= tmem_cols, "");

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.ns; ++s) { mbar_init(full + s, 1 + 32); mbar_init(used + s, kFusedWarps); }
    for (int s = 0; s < p.nx; ++s) { mbar_init(xfull + s, 1); mbar_init(xfree + s, 1); }
    for (int s = 0; s < wbufs; ++s) { mbar_init(wfull + s, kFusedWarps); mbar_init(wfree + s, 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(scaled + s, 4);
      mbar_init(accfull + s, 1);
      mbar_init(accfree + s, 4);
    }
    mbar_init(tail, 1);
    *nfinished = 0;
    *failed = 0;
    mbar_init_fence();
  }
  if (warp == kFusedWarps + 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint64_t* bar, uint32_t phase) {                      // bounded; once one gave up, none waits any more
    if (mbar_try_wait(bar, phase)) return true;
    if (*failed) return false;
    if (mbar_wait(bar, phase)) return true;
    *failed = 1;
    return false;
  };
  // stages [t0, t1) of an item
  auto stage_range = [&](int item, int* t0, int* t1) {
    *t0 = (item % p.chunks) * p.chunk_stages;
    *t1 = min(p.stages, *t0 + p.chunk_stages);
  };

  if (warp < kFusedWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFusedComputeRegs));
    // ---- rebuild ---------------------------------------------------------------------------------------
    const int rb = warp & 3, sub = warp >> 2;                          // a warp reaches the tensor-memory lanes 32 (warp % 4) ...
    const RebuildLane RL = rebuild_lane(lane);
    const uint32_t wt = tmem + 2 * acc_cols + 16 * sub + ((uint32_t)(32 * rb) << 16);
    RebuildAcc r;
    float d = 0.f;
    RingPos ps, ws;
    int wn = 0, nitem = 0;                                             // W buffers filled, items begun
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      int t0, t1;
      stage_range(item, &t0, &t1);
      const int R = (item / p.chunks) * 4 + rb;
      const bool there = R < g.rw * g.PT;
      float f = 1.f;
      if (NP == 1) {
        wait(scaled + (nitem & 1), (uint32_t)(nitem >> 1) & 1u);
        f = wscale[4 * (nitem & 1) + rb];
        ++nitem;
      }
      for (int t = t0; t < t1; ++t) {
        for (int ch = 0; ch < nchunks; ++ch) {
          wait(full + ps.slot, ps.phase);
          if (there) {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(base + L.planes + ps.slot * L.plane_stage + rb * (L.plane_group / 2)) + sub;
            const uint32_t* z = w + L.plane_stage / 8;
            const float4* k4 = reinterpret_cast<const float4*>(base + L.coef + ps.slot * L.coef_stage) + rb * p.nb * kGroup + sub;
            const int nbits = min(p.nb, g.bw - ch * p.nb);
            if (ch == 0) d = k4[0].w;
            rebuild_bits<RT>(r, RL, w, z, RT * 128, k4, kGroup, f * kCoefScale, lane, nbits, ch == 0);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(used + ps.slot);
          ps.next(p.ns);
        }
        if (wn >= wbufs) wait(wfree + ws.slot, ws.phase ^ 1u);
        __syncwarp();
        tc_fence_after();
        if (there) {
          rebuild_end(r, d * f, lane);
          // entry pairs of rows g + 8 rr: 32-bit columns 8 qh + 2 t + x of the lane's quarter, which is their order in K
          auto rows16 = [&](auto MT) {
            constexpr int mt = decltype(MT)::value;
            uint32_t hi[8], lo[8];
            auto put = [&](auto K, float2 v) {
              constexpr int k = decltype(K)::value;
              if (NP == 1) {
                const __half2 h = __floats2half2_rn(v.x, v.y);
                hi[k] = *reinterpret_cast<const uint32_t*>(&h);
                return;
              }
              const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
              hi[k] = *reinterpret_cast<const uint32_t*>(&h);
              const __nv_bfloat162 l = __floats2bfloat162_rn(v.x - __uint_as_float(hi[k] << 16), v.y - __uint_as_float(hi[k] & 0xFFFF0000u));
              lo[k] = *reinterpret_cast<const uint32_t*>(&l);
            };
            put(std::integral_constant<int, 0>(), rebuild_entry<2 * mt, 0>(r));
            put(std::integral_constant<int, 1>(), rebuild_entry<2 * mt, 1>(r));
            put(std::integral_constant<int, 2>(), rebuild_entry<2 * mt + 1, 0>(r));
            put(std::integral_constant<int, 3>(), rebuild_entry<2 * mt + 1, 1>(r));
            put(std::integral_constant<int, 4>(), rebuild_entry<2 * mt, 2>(r));
            put(std::integral_constant<int, 5>(), rebuild_entry<2 * mt, 3>(r));
            put(std::integral_constant<int, 6>(), rebuild_entry<2 * mt + 1, 2>(r));
            put(std::integral_constant<int, 7>(), rebuild_entry<2 * mt + 1, 3>(r));
            const uint32_t at = wt + ws.slot * kWCols + ((uint32_t)(16 * mt) << 16);
            tc_st_16x256b_x2(at, hi);
            if (NP != 1) tc_st_16x256b_x2(at + kWPart, lo);
          };
          rows16(std::integral_constant<int, 0>());
          rows16(std::integral_constant<int, 1>());
          tc_wait_st();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(wfull + ws.slot);
        ws.next(wbufs);
        ++wn;
      }
    }
    // the next kernel of the stream may become resident: all that is left here are sums
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.chunks > 1 && wn && wait(tail, 0))                           // tiles completed by this CTA
      for (int k = 0; k < *nfinished; ++k) fused_reduce_tile(p, finished[k], threadIdx.x, kFusedWarps * 32, rowf);
  } else if (warp >= kFusedWarps + 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFusedSumRegs));
    // ---- sums of an item: tensor memory -> scratch or output, while the next item is rebuilt --------------------
    // everything that was in the stream before this kernel has to be complete before y and the scratch are touched
    const int quarter = warp & 3;
    // power of two that maps the bound on the entries of this warp's row block in item `it` to 2^14, given to the
    // compute warps; one item ahead
    auto scale_of = [&](int it, int set) {
      if (NP != 1 || it >= items) return 1.f;
      int t0, t1;
      stage_range(it, &t0, &t1);
      const int i = ((it / p.chunks) * 4 + quarter) / g.PT;
      const int j0 = (t0 / g.QT) * kGroup, j1 = min(g.cw, ((t1 - 1) / g.QT + 1) * kGroup);
      float bound = 0.f;
      if (i < g.rw)
        for (int j = j0 + lane; j < j1; j += 32) {
          float s = 0.f;
#pragma unroll 4
          for (int b = 0; b < g.bw; ++b) {
            const size_t at = ((size_t)b * g.rw + i) * g.cw + j;
            s += fabsf(load_as_float(p.a, at, p.coef_dtype)) + fabsf(load_as_float(p.b, at, p.coef_dtype)) +
                 fabsf(load_as_float(p.c, at, p.coef_dtype));
          }
          bound = fmaxf(bound, fmaf((float)g.r, s, fabsf(load_as_float(p.d, (size_t)i * g.cw + j, p.coef_dtype))));
        }
#pragma unroll
      for (int e = 16; e > 0; e >>= 1) bound = fmaxf(bound, __shfl_xor_sync(0xffffffffu, bound, e));
      const float s = scale_from_bound(bound);
      if (lane == 0) {
        wscale[4 * set + quarter] = s;
        mbar_arrive(scaled + set);
      }
      return s;
    };
    float next_scale = scale_of(blockIdx.x, 0);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int wtid = threadIdx.x - (kFusedWarps + 4) * 32;
    rowf[wtid] = NP == 1 && p.row_unscale && wtid < p.M ? p.row_unscale[wtid] : 1.f;
    asm volatile("bar.sync 2, 128;" ::: "memory");
    int nitem = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x, ++nitem) {
      const uint32_t set = (uint32_t)(nitem & 1);
      const float unscale = 1.f / next_scale;
      next_scale = scale_of(item + (int)gridDim.x, (int)(set ^ 1u));
      const bool ok = wait(accfull + set, (uint32_t)(nitem >> 1) & 1u);
      tc_fence_after();
      const int tile = item / p.chunks;
      const int R = tile * 4 + quarter;                                // row block of this warp's tensor-memory lanes
      const int i = R / g.PT, pt = R - i * g.PT;
      const bool row_ok = i < g.rw && 32 * pt + lane < g.P;
      const int o = i * g.P + 32 * pt + lane;
      const float bias = p.bias && row_ok ? load_as_float(p.bias, o, p.bias_dtype) : 0.f;
      float* part = p.partial + ((size_t)item * p.N) * kFusedTile + 32 * quarter + lane;
      for (int n0 = 0; n0 < p.N; n0 += 16) {
        uint32_t v[16];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                       "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(tmem + ((uint32_t)(quarter * 32) << 16) + set * acc_cols + (uint32_t)n0));
        tc_wait_ld();
        if (!ok) continue;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (n0 + e >= p.M) break;
          const float u = __uint_as_float(v[e]) * unscale;
          if (p.chunks > 1) part[(size_t)(n0 + e) * kFusedTile] = u;
          else if (row_ok) fused_out(p, n0 + e, o, fmaf(u, rowf[n0 + e], bias));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree + set);
      if (p.chunks > 1) {
        // the CTA that finishes a tile last adds its chunks, in order; its compute warps do so when all is rebuilt
        asm volatile("bar.sync 2, 128;" ::: "memory");
        if (wtid == 0) {
          unsigned t = 0xFFFFFFFFu;
          if (!*failed)
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(t) : "l"(p.counters + tile) : "memory");
          if (t == (unsigned)(p.chunks - 1)) {
            p.counters[tile] = 0u;
            finished[(*nfinished)++] = tile;
          }
          if (item + (int)gridDim.x >= items) mbar_arrive(tail);
        }
        if (nitem >= kFusedMaxItems - 1) {                             // the list may be full: work it off here
          asm volatile("bar.sync 2, 128;" ::: "memory");
          const int n = *nfinished;
          if (n == kFusedMaxItems && item + (int)gridDim.x < items) {
            for (int k = 0; k < n; ++k) fused_reduce_tile(p, finished[k], wtid, 128, rowf);
            asm volatile("bar.sync 2, 128;" ::: "memory");
            if (wtid == 0) *nfinished = 0;
          }
          asm volatile("bar.sync 2, 128;" ::: "memory");
        }
      }
    }
  } else {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFusedHelperRegs));
   if (warp == kFusedWarps) {
    // ---- plane words ---------------------------------------------------------------------------------------
    if (lane == 0) {
      RingPos ps;
      int n = 0;
      for (int item = blockIdx.x; item < items && !*failed; item += gridDim.x) {
        int t0, t1;
        stage_range(item, &t0, &t1);
        const int R0 = (item / p.chunks) * 4;
        const int groups = min(4, g.rw * g.PT - R0);
        int jg = t0 / g.QT, qt = t0 - jg * g.QT;
        for (int t = t0; t < t1; ++t) {
          for (int b0 = 0; b0 < g.bw; b0 += p.nb) {
            if (n >= p.ns && !wait(used + ps.slot, ps.phase ^ 1u)) break;
            mbar_expect_tx(full + ps.slot, (uint32_t)((p.joint ? 4 : groups) * p.nb * kBitBytes));
            uint8_t* dst = base + L.planes + ps.slot * L.plane_stage;
            if (p.joint) {                             // the four row patches of the tile at once
              tma_load_4d(dst, &map_y, full + ps.slot, 0, 0, jg, R0 * g.bw);
              tma_load_5d(dst + L.plane_stage / 2, &map_z, full + ps.slot, 0, qt, 0, jg, R0 * g.bw);
            } else {
              int i = R0 / g.PT, pt = R0 - i * g.PT;
#pragma unroll 1
              for (int rb = 0; rb < groups; ++rb) {
                tma_load_4d(dst + rb * (L.plane_group / 2), &map_y, full + ps.slot, 0, pt, jg, i * g.bw + b0);
                tma_load_5d(dst + L.plane_stage / 2 + rb * (L.plane_group / 2), &map_z, full + ps.slot, 0, qt, 0, jg, i * g.bw + b0);
                if (++pt == g.PT) { pt = 0; ++i; }
              }
            }
            ps.next(p.ns);
            ++n;
          }
          if (++qt == g.QT) { qt = 0; ++jg; }
        }
      }
      // the compute warps wait for every stage before they end; after a failure the copies in flight have to land first
      if (*failed)
        for (int k = 0; k < min(n, p.ns); ++k) {
          mbar_wait(full + ps.slot, ps.phase ^ 1u);
          ps.next(p.ns);
        }
    }
  } else if (warp == kFusedWarps + 1) {
    // ---- coefficients as floats ------------------------------------------------------------------------------
    // lane = (row block lane >> 4 and + 2, col patch, kind): kind 0, 1, 2 = a, b, c of every bit layer, 3 = d.  fp32 ones
    // are copied asynchronously (the barrier counts the copies), so nothing here waits for memory.
    const int sub = (lane >> 2) & 3, kind = lane & 3;
    const void* const src = kind == 0 ? p.a : kind == 1 ? p.b : kind == 2 ? p.c : p.d;
    const size_t bstep = (size_t)g.rw * g.cw;
    RingPos ps;
    int n = 0;
    for (int item = blockIdx.x; item < items && !*failed; item += gridDim.x) {
      int t0, t1;
      stage_range(item, &t0, &t1);
      const int R0 = (item / p.chunks) * 4 + (lane >> 4);
      const int i0 = R0 / g.PT, i1 = (R0 + 2) / g.PT;
      int jg = t0 / g.QT, qt = t0 - jg * g.QT;
      for (int t = t0; t < t1; ++t) {
        const int j = jg * kGroup + sub;
        for (int b0 = 0; b0 < g.bw; b0 += p.nb) {
          if (n >= p.ns && !wait(used + ps.slot, ps.phase ^ 1u)) break;
          uint32_t dst = smem_u32(base + L.coef + ps.slot * L.coef_stage) + (uint32_t)((((lane >> 4) * p.nb * kGroup + sub) * 4 + kind) * 4);
          const int some = kind < 3 ? min(p.nb, g.bw - b0) : (b0 == 0 ? 1 : 0);
#pragma unroll 1
          for (int h = 0; h < 2; ++h, dst += (uint32_t)(2 * p.nb * kGroup * 16)) {
            const int i = h ? i1 : i0;
            const int count = i < g.rw && j < g.cw ? some : 0;
            const size_t at = ((size_t)(kind < 3 ? b0 * g.rw : 0) + i) * g.cw + j;
            if (p.coef_dtype == BQQ_F32) {
              const float* from = reinterpret_cast<const float*>(src) + (count ? at : 0);
#pragma unroll 1
              for (int b = 0; b < p.nb; ++b) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                             ::"r"(dst + b * (kGroup * 16)), "l"(from), "r"(b < count ? 4 : 0) : "memory");
                if (b + 1 < count) from += bstep;
              }
            } else {
#pragma unroll 1
              for (int b = 0; b < p.nb; ++b)
                store_shared_u32(dst + b * (kGroup * 16),
                                 __float_as_uint(b < count ? load_as_float(src, at + b * bstep, p.coef_dtype) : 0.f));
            }
          }
          if (p.coef_dtype == BQQ_F32)
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(full + ps.slot)) : "memory");
          else
            mbar_arrive(full + ps.slot);
          ps.next(p.ns);
          ++n;
        }
        if (++qt == g.QT) { qt = 0; ++jg; }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == kFusedWarps + 2) {
    // ---- x ------------------------------------------------------------------------------------------------
    if (lane == 0) {
      asm volatile("griddepcontrol.wait;" ::: "memory");               // x comes from the kernels before this one
      RingPos xs;
      int n = 0;
      for (int item = blockIdx.x; item < items && !*failed; item += gridDim.x) {
        int t0, t1;
        stage_range(item, &t0, &t1);
        for (int t = t0; t < t1; ++t) {
          if (n >= p.nx && !wait(xfree + xs.slot, xs.phase ^ 1u)) break;
          mbar_expect_tx(xfull + xs.slot, (uint32_t)L.x_stage);
          uint8_t* dst = base + L.x + xs.slot * L.x_stage;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            tma_load_2d(dst + k * (L.x_part / 2), &map_hi, xfull + xs.slot, t * kFusedStageCols + 64 * k, 0);
            if (NP == 3) tma_load_2d(dst + L.x_part + k * (L.x_part / 2), &map_lo, xfull + xs.slot, t * kFusedStageCols + 64 * k, 0);
          }
          xs.next(p.nx);
          ++n;
        }
      }
      if (*failed)
        for (int k = 0; k < min(n, p.nx); ++k) {
          mbar_wait(xfull + xs.slot, xs.phase ^ 1u);
          xs.next(p.nx);
        }
    }
  } else {
    // ---- tensor core ---------------------------------------------------------------------------------------
    if (lane == 0) {
      RingPos xs, ws;
      int nitem = 0;
      for (int item = blockIdx.x; item < items && !*failed; item += gridDim.x, ++nitem) {
        int t0, t1;
        stage_range(item, &t0, &t1);
        const uint32_t set = (uint32_t)(nitem & 1);
        const uint32_t dtm = tmem + set * acc_cols;
        if (nitem >= 2 && !wait(accfree + set, (uint32_t)((nitem >> 1) - 1) & 1u)) break;
        for (int t = t0; t < t1; ++t) {
          if (!wait(xfull + xs.slot, xs.phase) || !wait(wfull + ws.slot, ws.phase)) break;
          tc_fence_after();
          const uint32_t wa = tmem + 2 * acc_cols + ws.slot * kWCols, xa = smem_u32(base + L.x + xs.slot * L.x_stage);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t whi = wa + 32 * k, wlo = whi + kWPart;
            const uint64_t xhi = make_smem_desc(xa + k * (L.x_part / 2));
#pragma unroll
            for (int e = 0; e < 4; ++e)                // 16 elements = 32 bytes: 8 columns of W, 2 descriptor units of x
              tc_mma_f16_ts(dtm, whi + 8 * e, xhi + 2 * e, p.idesc, (t != t0 || (k | e) != 0) ? 1u : 0u);
            if (NP >= 2) {
#pragma unroll
              for (int e = 0; e < 4; ++e) tc_mma_f16_ts(dtm, wlo + 8 * e, xhi + 2 * e, p.idesc, 1u);
            }
            if (NP == 3) {
              const uint64_t xlo = make_smem_desc(xa + L.x_part + k * (L.x_part / 2));
#pragma unroll
              for (int e = 0; e < 4; ++e) tc_mma_f16_ts(dtm, whi + 8 * e, xlo + 2 * e, p.idesc, 1u);
            }
          }
          tc_commit(wfree + ws.slot);
          tc_commit(xfree + xs.slot);
          xs.next(p.nx);
          ws.next(wbufs);
        }
        tc_commit(accfull + set);
      }
    }
  }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kFusedWarps + 3) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
  if (threadIdx.x == 0 && *failed) atomicExch(p.status, 1u);
}

}  // namespace bqq
