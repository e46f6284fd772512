// Dense weight from packed planes:
//   W[i*P+p, j*Q+q] = sum_b ( a_b popc(Yrow_b[p] & Zcol_b[q]) + b_b popc(Yrow_b[p])
//                             + c_b popc(Zcol_b[q]) ) + d
// i.e. BinaryQuadratic.get_weight (neural_network_compression/src/bqq_modules.py:48-55); replaces
// reconstruct_W_kernel (src/bqq_cuda.cu:198-246).
// A compute warp forms one 32x32 block of one patch at a time with int8 tensor-core products (bqq_rebuild.cuh, where the
// cost per bit layer is accounted for).  A stage of work is two super-groups at one block position: eight compute warps take
// their eight col patches (the plane words of a super-group's four are interleaved).  A producer warp runs a few stages
// ahead: it brings the plane words by bulk copies, the coefficients as floats and the place of the results, so that a step
// of a compute warp (one block, one bit layer) is four shared-memory loads and the arithmetic.  Measured, 4096 x 14336
// with 4 bit layers to bf16: 125.7 us with fp16 products, addresses and coefficients in every warp -> 64 us (53 us of
// it without the stores); 45 % of the tensor pipe, 65 % of the issue slots, 2.8 TB/s.
#include <algorithm>
#include <type_traits>

#include "bqq_async.cuh"
#include "bqq_rebuild.cuh"

namespace bqq {

constexpr int kReconGroups = 2;                    // super-groups of a stage
constexpr int kReconWarps = kReconGroups * kGroup; // compute warps
constexpr int kReconThreads = (kReconWarps + 2) * 32;
constexpr int kReconStages = 4;                    // stages in flight
constexpr int kReconBits = 8;                      // bit layers of a stage at most

struct ReconParams {
  const uint32_t* zp;
  const uint32_t* yp;
  const void *a, *b, *c, *d;
  void* W;
  void* W_lo;                  // optional second part: W - round(W), same type and layout
  const float* bound_parts;    // optional: entries are also scaled by w_scale_from_maxima
  float scale;
  int coef_dtype, w_dtype;
  int quads;                   // 1: four neighbouring entries of a row may be stored as one aligned word
  Geom g;
  int units;                   // super-groups of these row patches
  int step_i, step_jg;         // kReconGroups gridDim.x super-groups further: row patches and super-groups
  int i0, i1;                  // row patches [i0, i1) are rebuilt
  // How the launch takes part in a chain of programmatic dependent launches (kPdl* in bqq_common.cuh)
  int pdl;
  unsigned* status;            // optional word, set when a wait on a copy gave up
};

// element type of W as a compile-time choice
template <int DT> struct WType;
template <> struct WType<BQQ_F32> {
  using T = float;
  using T2 = float2;
  static __device__ __forceinline__ T cvt(float v) { return v; }
  static __device__ __forceinline__ T2 cvt2(float v0, float v1) { return make_float2(v0, v1); }
  static __device__ __forceinline__ float back(T v) { return v; }
};
template <> struct WType<BQQ_BF16> {
  using T = __nv_bfloat16;
  using T2 = __nv_bfloat162;
  static __device__ __forceinline__ T cvt(float v) { return __float2bfloat16_rn(v); }
  static __device__ __forceinline__ T2 cvt2(float v0, float v1) { return __floats2bfloat162_rn(v0, v1); }
  static __device__ __forceinline__ float back(T v) { return __bfloat162float(v); }
};
template <> struct WType<BQQ_F16> {
  using T = __half;
  using T2 = __half2;
  static __device__ __forceinline__ T cvt(float v) { return __float2half_rn(v); }
  static __device__ __forceinline__ T2 cvt2(float v0, float v1) { return __floats2half2_rn(v0, v1); }
  static __device__ __forceinline__ float back(T v) { return __half2float(v); }
};

// four neighbouring entries as one 8- or 16-byte store
__device__ __forceinline__ void store_quad(float* p, float2 a, float2 b) {
  *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
}
template <typename T, typename T2>
__device__ __forceinline__ void store_quad(T* p, T2 a, T2 b) {
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}

// The stages of one group of a CTA, in order: super-groups u = 2 (blockIdx.x + k gridDim.x) + group of the row patches
// [i0, i1) (counted row patch by row patch), their blocks, and up to kReconBits bit layers from bit0 at a time.
struct ReconWalk {
  int i, jg, pt, qt, bit0, u;
  __device__ __forceinline__ void start(const ReconParams& p, int group) {
    u = (int)blockIdx.x * kReconGroups + group;
    i = p.i0 + u / p.g.JG;
    jg = u % p.g.JG;
    pt = qt = bit0 = 0;
  }
  __device__ __forceinline__ bool there(const ReconParams& p) const { return u < p.units; }
  __device__ __forceinline__ void next(const ReconParams& p, int nb) {
    bit0 += nb;
    if (bit0 < p.g.bw) return;
    bit0 = 0;
    if (++qt < p.g.QT) return;
    qt = 0;
    if (++pt < p.g.PT) return;
    pt = 0;
    u += (int)gridDim.x * kReconGroups;
    i += p.step_i;
    jg += p.step_jg;
    if (jg >= p.g.JG) { jg -= p.g.JG; ++i; }
  }
};
// What a stage holds beside its plane words.
struct ReconHead {
  long long at;                // entry (0, 0) of the block of col patch 0 in W, in elements
  int rows, cols;              // rows and columns of the block that exist
  int patches;                 // col patches that exist (0: no super-group here)
  int pad[3];
};
struct ReconStage {
  ReconHead head[kReconGroups];
  float4 coef[kReconGroups][kReconBits][kGroup];   // {a, b, c, d}
};

template <int RT, int DT, bool LO>
__global__ void __launch_bounds__(kReconThreads, 2)
bqq_reconstruct_kernel(const ReconParams p) {
  using WT = typename WType<DT>::T;
  using WT2 = typename WType<DT>::T2;
  extern __shared__ __align__(128) uint8_t rsm[];    // planes: [stage][group][bit][Y RT x 512 | Z RT x 512 bytes]
  __shared__ uint64_t full[kReconStages], used[kReconStages];
  __shared__ __align__(16) ReconStage stage[kReconStages];
  constexpr int kBitBytes = RT * 1024;
  const Geom& g = p.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = min(g.bw, kReconBits), nchunks = (g.bw + nb - 1) / nb;   // bit layers of a stage, stages of a block
  const int blocks = g.PT * g.QT;
  const int pairs = (p.units + kReconGroups - 1) / kReconGroups;
  const int mine = ((int)blockIdx.x < pairs ? (pairs - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0);
  const int nstages = mine * blocks * nchunks;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kReconStages; ++s) { mbar_init(full + s, 2); mbar_init(used + s, kReconWarps); }
    mbar_init_fence();
  }
  __syncthreads();

  if (warp == kReconWarps) {
    // ---- producer of the plane words: one lane, a few stages ahead ---------------------------------------
    if (lane == 0) {
      ReconWalk w0, w1;
      w0.start(p, 0);
      w1.start(p, 1);
      for (int n = 0; n < nstages; ++n) {
        const int s = n % kReconStages;
        if (n >= kReconStages) mbar_wait(used + s, (uint32_t)(n / kReconStages - 1) & 1u);
        const int nbits = min(nb, g.bw - w0.bit0);
        mbar_expect_tx(full + s, (uint32_t)(nbits * kBitBytes) * (w1.there(p) ? 2u : 1u));
#pragma unroll
        for (int grp = 0; grp < kReconGroups; ++grp) {
          ReconWalk& w = grp ? w1 : w0;
          if (w.there(p)) {
            const size_t sg = (size_t)w.i * g.NS + (size_t)w.bit0 * g.JG + w.jg;
            const uint32_t* y = p.yp + (sg * g.PT + w.pt) * (RT * 128);
            const uint32_t* z = p.zp + (sg * RT * g.QT + w.qt) * 128;
            uint8_t* dst = rsm + (size_t)((s * kReconGroups + grp) * nb) * kBitBytes;
            for (int b = 0; b < nbits; ++b) {
              bulk_load(dst, y, RT * 512, full + s);
#pragma unroll
              for (int rt = 0; rt < RT; ++rt) bulk_load(dst + (RT + rt) * 512, z + rt * g.QT * 128, 512, full + s);
              dst += kBitBytes;
              y += (size_t)g.JG * g.PT * (RT * 128);
              z += (size_t)g.JG * RT * g.QT * 128;
            }
          }
          w.next(p, nb);
        }
      }
    }
    pdl_enter(p.pdl);
  } else if (warp == kReconWarps + 1) {
    // ---- producer of coefficients and places -------------------------------------------------------------
    // lane = (group, col patch, kind): its coefficient (kind 0, 1, 2: a, b, c of every bit layer of the stage; 3: d)
    const int grp = lane >> 4, sub = (lane >> 2) & 3, kind = lane & 3;
    const void* const base = kind == 0 ? p.a : kind == 1 ? p.b : kind == 2 ? p.c : p.d;
    ReconWalk w;
    w.start(p, grp);
    float v[kReconBits];
    auto load = [&](auto one) {                      // the coefficients of stage w
      const int j = w.jg * kGroup + sub;
      const bool there = w.there(p) && j < g.cw;
      const size_t at = ((size_t)(kind < 3 ? w.bit0 * g.rw : 0) + w.i) * g.cw + j, step = (size_t)g.rw * g.cw;
      const int count = !there ? 0 : kind < 3 ? min(nb, g.bw - w.bit0) : 1;
#pragma unroll
      for (int b = 0; b < kReconBits; ++b) {
        if (b >= nb) break;
        v[b] = b < count ? one(at + b * step) : 0.f;
      }
    };
    auto coefficients = [&]() {
      if (p.coef_dtype == BQQ_F32) load([&](size_t e) { return reinterpret_cast<const float*>(base)[e]; });
      else load([&](size_t e) { return load_as_float(base, e, p.coef_dtype); });
    };
    coefficients();
    pdl_enter(p.pdl);
    const float scale = p.bound_parts ? p.scale * w_scale_from_maxima(p.bound_parts, (float)(g.bw * g.r), lane) : p.scale;
    const float cscale = kind < 3 ? scale * kCoefScale : scale;
    for (int n = 0; n < nstages; ++n) {
      const int s = n % kReconStages;
      if (n >= kReconStages) mbar_wait(used + s, (uint32_t)(n / kReconStages - 1) & 1u);
      float* dst = reinterpret_cast<float*>(&stage[s].coef[grp][0][sub]) + kind;
#pragma unroll
      for (int b = 0; b < kReconBits; ++b) {
        if (b >= nb) break;
        dst[b * kGroup * 4] = v[b] * cscale;
      }
      if ((lane & 15) == 0) {
        ReconHead h;
        h.at = ((long long)w.i * g.P + 32 * w.pt) * ((long long)g.cw * g.Q) + (long long)w.jg * kGroup * g.Q + 32 * w.qt;
        h.rows = min(32, g.P - 32 * w.pt);
        h.cols = min(32, g.Q - 32 * w.qt);
        h.patches = w.there(p) ? min(kGroup, g.cw - w.jg * kGroup) : 0;
        stage[s].head[grp] = h;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(full + s);
      w.next(p, nb);
      coefficients();
    }
  } else {
    // ---- compute warps ---------------------------------------------------------------------------------
    pdl_enter(p.pdl);
    const int grp = warp / kGroup, sub = warp % kGroup;
    const int g8 = lane >> 2, t4 = lane & 3;
    const RebuildLane L = rebuild_lane(lane);
    const long long ldw = (long long)g.cw * g.Q;
    const long long here = (long long)sub * g.Q + g8 * ldw + 4 * t4;   // the lane's first entry inside a block
    RebuildAcc r;
    float d = 0.f;
    bool ok = true;
    int s = 0, chunk = 0;
    uint32_t phase = 0;
    for (int n = 0; n < nstages; ++n) {
      ok = ok && mbar_wait(full + s, phase);
      const ReconStage& st = stage[s];
      const ReconHead& h = st.head[grp];
      const int nbits = min(nb, g.bw - chunk * nb);
      const bool live = sub < h.patches;
      if (live) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(rsm + (size_t)((s * kReconGroups + grp) * nb) * kBitBytes) + sub;
        const float4* k = &st.coef[grp][0][sub];
        if (chunk == 0) d = k->w;
        rebuild_bits<RT>(r, L, w, w + RT * 128, kBitBytes / 4, k, kGroup, 1.f, lane, nbits, chunk == 0);
      }
      const long long at = h.at + here;
      const int rows = h.rows, cols = h.cols;
      __syncwarp();
      if (lane == 0) mbar_arrive(used + s);
      if (++s == kReconStages) { s = 0; phase ^= 1u; }
      if (++chunk < nchunks) continue;
      chunk = 0;
      if (!live) continue;

      // 32 x 32 entries: a lane holds four neighbouring columns of rows g8 + 8 rr in either half
      rebuild_end(r, d, lane);
      WT* wp = reinterpret_cast<WT*>(p.W) + at;
      WT* lp = LO ? reinterpret_cast<WT*>(p.W_lo) + at : nullptr;
      const bool quad0 = p.quads && 4 * t4 + 4 <= cols, quad1 = p.quads && 4 * t4 + 20 <= cols;
      auto half = [&](auto RR, auto QH, bool quad, float2 v01, float2 v23) {
        constexpr int rr = decltype(RR)::value, qh = decltype(QH)::value;
        WT* w = wp + 8 * rr * ldw + 16 * qh;
        WT* lo = LO ? lp + 8 * rr * ldw + 16 * qh : nullptr;
        if (quad) {
          const WT2 w01 = WType<DT>::cvt2(v01.x, v01.y), w23 = WType<DT>::cvt2(v23.x, v23.y);
          store_quad(w, w01, w23);
          if (LO)
            store_quad(lo, WType<DT>::cvt2(v01.x - WType<DT>::back(w01.x), v01.y - WType<DT>::back(w01.y)),
                       WType<DT>::cvt2(v23.x - WType<DT>::back(w23.x), v23.y - WType<DT>::back(w23.y)));
        } else {
          const float v[4] = {v01.x, v01.y, v23.x, v23.y};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (4 * t4 + 16 * qh + e < cols) {
              const WT t = WType<DT>::cvt(v[e]);
              w[e] = t;
              if (LO) lo[e] = WType<DT>::cvt(v[e] - WType<DT>::back(t));
            }
        }
      };
      auto each_row = [&](auto WHOLE) {
        auto row = [&](auto RR) {
          constexpr int rr = decltype(RR)::value;
          constexpr bool whole = decltype(WHOLE)::value;
          if (!whole && g8 + 8 * rr >= rows) return;
          half(RR, std::integral_constant<int, 0>(), whole || quad0, rebuild_entry<rr, 0>(r), rebuild_entry<rr, 1>(r));
          half(RR, std::integral_constant<int, 1>(), whole || quad1, rebuild_entry<rr, 2>(r), rebuild_entry<rr, 3>(r));
        };
        row(std::integral_constant<int, 0>());
        row(std::integral_constant<int, 1>());
        row(std::integral_constant<int, 2>());
        row(std::integral_constant<int, 3>());
      };
      if (p.quads && rows == 32 && cols == 32) each_row(std::true_type());
      else each_row(std::false_type());
    }
    if (!ok && p.status && lane == 0) atomicExch(p.status, 1u);   // a bounded wait gave up: the entries are invalid
  }
  pdl_exit(p.pdl);
}

template <typename K>
static int recon_launch_one(K kern, const ReconParams& p, dim3 blocks, cudaStream_t st) {
  const size_t smem = (size_t)kReconStages * kReconGroups * std::min(p.g.bw, kReconBits) * p.g.RT * 1024;
  if (smem > 32 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return BQQ_ERR_CUDA;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = blocks;
  cfg.blockDim = dim3(kReconThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = p.pdl != kPdlNone ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) { cudaGetLastError(); return BQQ_ERR_CUDA; }
  return launch_status();
}

template <int RT>
static int reconstruct_dispatch(const ReconParams& p, dim3 blocks, cudaStream_t st) {
  const bool lo = p.W_lo != nullptr;
  if (p.w_dtype == BQQ_F32) return recon_launch_one(bqq_reconstruct_kernel<RT, BQQ_F32, false>, p, blocks, st);
  if (p.w_dtype == BQQ_BF16)
    return lo ? recon_launch_one(bqq_reconstruct_kernel<RT, BQQ_BF16, true>, p, blocks, st)
              : recon_launch_one(bqq_reconstruct_kernel<RT, BQQ_BF16, false>, p, blocks, st);
  return lo ? recon_launch_one(bqq_reconstruct_kernel<RT, BQQ_F16, true>, p, blocks, st)
            : recon_launch_one(bqq_reconstruct_kernel<RT, BQQ_F16, false>, p, blocks, st);
}

int reconstruct_launch(const BqqLayer* L, void* W, void* W_lo, int w_dtype, float scale, const float* bound_parts,
                       cudaStream_t st, int i0, int i1, int pdl, unsigned* status) {
  ReconParams p;
  p.g = Geom(L->dims);
  p.i0 = i0;
  p.i1 = i1 < 0 ? p.g.rw : i1;
  p.pdl = pdl;
  p.status = status;
  p.zp = L->zplanes; p.yp = L->yplanes;
  p.a = L->a; p.b = L->b; p.c = L->c; p.d = L->d; p.coef_dtype = L->coef_dtype;
  p.W = W; p.W_lo = W_lo; p.scale = scale; p.bound_parts = bound_parts; p.w_dtype = w_dtype;
  const uintptr_t quad_mask = 4 * (uintptr_t)dtype_size(w_dtype) - 1;
  p.quads = (p.g.Q % 4 == 0 && ((uintptr_t)W & quad_mask) == 0 && ((uintptr_t)W_lo & quad_mask) == 0) ? 1 : 0;
  // resident CTAs walk the pairs of super-groups: 2 per SM on 148 SMs
  const long long units = (long long)p.g.JG * (p.i1 - p.i0);
  if (units <= 0) return BQQ_OK;
  if (units > (1ll << 30)) return BQQ_ERR_UNSUPPORTED;
  p.units = (int)units;
  const dim3 blocks((unsigned)std::min<long long>((units + kReconGroups - 1) / kReconGroups, 148LL * 2));
  p.step_i = (int)(blocks.x * kReconGroups) / p.g.JG;
  p.step_jg = (int)(blocks.x * kReconGroups) % p.g.JG;
  if (w_dtype == BQQ_F32 && W_lo) return BQQ_ERR_UNSUPPORTED;     // a second part only exists for 16-bit types
  if (p.g.RT == 1) return reconstruct_dispatch<1>(p, blocks, st);
  return reconstruct_dispatch<2>(p, blocks, st);
}

// maxima[block] = max(|a|+|b|+|c|), maxima[kBoundBlocks + block] = max|d| over the block's share of the coefficients
// (maxima may be NULL); clears *status.  Every block writes its pair, so nothing has to be cleared before.
__global__ void __launch_bounds__(256)
coef_bound_kernel(const void* a, const void* b, const void* c, const void* d, int dt, size_t nabc, size_t nd, float* maxima,
                  unsigned* status) {
  pdl_enter(kPdlWaitFirst);
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0u;
  if (!maxima) return;
  float m0 = 0.f, m1 = 0.f;
#pragma unroll 4
  for (size_t t = blockIdx.x * 256 + threadIdx.x; t < nabc; t += kBoundBlocks * 256)
    m0 = fmaxf(m0, fabsf(load_as_float(a, t, dt)) + fabsf(load_as_float(b, t, dt)) + fabsf(load_as_float(c, t, dt)));
#pragma unroll 4
  for (size_t t = blockIdx.x * 256 + threadIdx.x; t < nd; t += kBoundBlocks * 256)
    m1 = fmaxf(m1, fabsf(load_as_float(d, t, dt)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  __shared__ float part[2][8];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { part[0][warp] = m0; part[1][warp] = m1; }
  __syncthreads();
  if (threadIdx.x < 2) {
    float m = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) m = fmaxf(m, part[threadIdx.x][w]);
    maxima[threadIdx.x * kBoundBlocks + blockIdx.x] = m;
  }
}

int coef_bound_launch(const BqqLayer* L, float* maxima, unsigned* status, cudaStream_t st) {
  Geom g(L->dims);
  const size_t nabc = (size_t)g.bw * g.rw * g.cw, nd = (size_t)g.rw * g.cw;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(maxima ? kBoundBlocks : 1);
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, coef_bound_kernel, L->a, L->b, L->c, L->d, (int)L->coef_dtype, nabc, nd, maxima,
                         status) != cudaSuccess) { cudaGetLastError(); return BQQ_ERR_CUDA; }
  return launch_status();
}

}  // namespace bqq
