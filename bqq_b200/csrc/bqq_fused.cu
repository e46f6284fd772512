// Host side of the fused rebuild-and-multiply forward (algorithm and kernel in bqq_fused_kernel.cuh): plan, preparation of
// x, launch.
#include <algorithm>
#include <type_traits>

#include "bqq_fused_kernel.cuh"
#include "bqq_xsource.cuh"

namespace bqq {

// x in the kernel's column order, zeros in the padding; also clears the counters of the tiles for callers whose scratch is not
// kept clean.  Eight columns per thread.  NP (formats of bqq_fused_kernel.cuh) = 1: fp16, bf16 rows scaled by a power of
// two (the row's maximum maps to at most 2^14; unscale[m] = 1 / scale); 2: bf16; 3: bf16 hi and lo = the rest.
// Bound: two round trips to x, the row's maximum first, and what the SM does meanwhile.  A CTA of 128 threads and 32 registers
// (at most one per SM) shares the SM with a CTA of the fused kernel, which then rebuilds up to four stages of W beside it; one of
// 256 threads and 46 registers kept that CTA out until it was done (4096 x 4096, 2 bit layers, 64 rows: 24.8 -> 21.3 us in
// all; P = 96, Q = 40, r = 33, 5 rows 17.8 -> 14.3).  Rows of more than kPrepLong columns are more round trips
// than a rebuild of four stages hides: CTAs of 256 threads, in front of the fused kernel (28672 columns, 32 rows: 282
// against 293 us).
constexpr int kPrepThreads = 128, kPrepWide = 256, kPrepLong = 16384;
template <int NP, int T>
__global__ void __launch_bounds__(T, T == kPrepThreads ? 16 : 1)
fused_prep_kernel(const XSource xs, int M, Geom g, int Kp, uint16_t* __restrict__ hi, uint16_t* __restrict__ lo,
                  float* __restrict__ unscale, unsigned* __restrict__ zero, int nzero, unsigned* __restrict__ status) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (blockIdx.x == 0 && blockIdx.y == 0) {
    for (int e = threadIdx.x; e < nzero; e += T) zero[e] = 0u;
    if (status && threadIdx.x == 0) *status = 0u;
  }
  if (!hi) return;
  constexpr int kWarps = T / 32;
  __shared__ float part[kWarps];
  const int m = blockIdx.y;
  float inv_rms = 1.f, scale = 1.f;
  if (NP != 1 && xs.mode == BQQ_PRO_RMSNORM) {
    const float w = row_sumsq_share(xs, m, threadIdx.x, T);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = w;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) tot += part[k];
    inv_rms = rsqrtf(tot / (float)xs.n_in + xs.eps);
  }
  if (NP == 1 && unscale) {
    float top = 0.f;
    if ((xs.n_in & 3) == 0 && raw4_aligned(xs.x, (size_t)m * xs.ld, xs.dtype)) {
      const uint16_t* row = reinterpret_cast<const uint16_t*>(xs.x) + (size_t)m * xs.ld;
      constexpr int kAhead = 8;                       // in flight: one round trip for 4096 columns
      for (int n0 = 4 * threadIdx.x; n0 < xs.n_in; n0 += 4 * T * kAhead) {
        uint2 r[kAhead];                              // 16-bit types only
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
          r[k] = n0 + 4 * T * k < xs.n_in ? *reinterpret_cast<const uint2*>(row + n0 + 4 * T * k) : make_uint2(0u, 0u);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          float v[4];
          raw4_to_float(make_uint4(r[k].x, r[k].y, 0u, 0u), xs.dtype, v);
          top = fmaxf(top, fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
        }
      }
    } else {
      for (int n = threadIdx.x; n < xs.n_in; n += T) top = fmaxf(top, fabsf(load_as_float(xs.x, (size_t)m * xs.ld + n, xs.dtype)));
    }
#pragma unroll
    for (int e = 16; e > 0; e >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, e));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = top;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kWarps; ++k) top = fmaxf(top, part[k]);
    scale = scale_from_bound(top);
    if (threadIdx.x == 0 && blockIdx.x == 0) unscale[m] = 1.f / scale;
  }
  for (int k0 = (blockIdx.x * T + threadIdx.x) * 8; k0 < Kp; k0 += gridDim.x * (8 * T)) {
    const int blk = k0 >> 5, c0 = k0 & 31;
    const int sub = blk & 3, s = blk >> 2;
    const int jg = s / g.QT, qt = s - jg * g.QT;
    const int j = jg * kGroup + sub, q = 32 * qt + c0;
    float v[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float quad[4] = {0.f, 0.f, 0.f, 0.f};
      if (j < g.cw && q + 4 * h + 4 <= g.Q) {
        load_x_quad(xs, m, j * g.Q + q + 4 * h, inv_rms, quad);
      } else if (j < g.cw) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (q + 4 * h + e < g.Q) quad[e] = load_x(xs, m, j * g.Q + q + 4 * h + e, inv_rms);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) v[4 * h + e] = quad[e];
    }
    uint32_t wh[4], wl[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (NP == 1) {
        const __half2 b = __floats2half2_rn(v[2 * e] * scale, v[2 * e + 1] * scale);
        wh[e] = *reinterpret_cast<const uint32_t*>(&b);
        continue;
      }
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
      wh[e] = *reinterpret_cast<const uint32_t*>(&b);
      const __nv_bfloat162 r = __floats2bfloat162_rn(v[2 * e] - __uint_as_float(wh[e] << 16),
                                                     v[2 * e + 1] - __uint_as_float(wh[e] & 0xFFFF0000u));
      wl[e] = *reinterpret_cast<const uint32_t*>(&r);
    }
    *reinterpret_cast<uint4*>(hi + (size_t)m * Kp + k0) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
    if (NP == 3) *reinterpret_cast<uint4*>(lo + (size_t)m * Kp + k0) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
  }
}

namespace {

struct FusedPlan {
  bool ok;
  int N, nb, ns, nx, tiles, chunks, chunk_stages, stages, Kp;
  size_t smem, partial_bytes, x_bytes;
};

constexpr size_t kMaxSmem = 225 * 1024;            // leaves room for a CTA of the preparation
inline size_t up256(size_t v) { return (v + 255) / 256 * 256; }

// Estimated time (ns) of `tiles` tiles in chunks of `cs` stages, fitted to 27 layers and batches (8 to 224 tiles, 8 to 112
// stages, 16 to 128 rows) in up to nine chunk lengths each: rounds of items over 148 SMs, an item no shorter than what moves its
// sums, then the sum over the chunks of a tile by one CTA.
long long chunk_cost(const Geom& g, int stages, int tiles, int N, int cs) {
  const int chunks = (stages + cs - 1) / cs;
  const long long rounds = ((long long)tiles * chunks + 147) / 148;
  const long long item = cs * (870LL + g.bw * (g.RT == 1 ? 385 : 640)) + 1280 + 23 * N;
  if (chunks == 1) return rounds * item;
  return rounds * std::max(item, 3080LL + 25 * N) + 400 + (12LL * N * ((tiles + 147) / 148) + 30) * chunks;
}

// Chunk length of a layer, at most 32 chunks.  tiles = 0: the sum must not depend on the number of rows of W (a row shard
// reproduces the whole layer bit for bit), so it is the length that is good for 16 to 112 tiles (2048 to 14336 rows) alike.
// (us, length for 32 tiles -> this one, 16 rows: 2048 x 6144 b2 22.8 -> 15.6, 6144 x 2048 b3 19.1 -> 17.6, 14336 x 4096 b2
// 60.8 -> 56.5.)  A thread keeps the lengths it used last: the search takes about as long as a launch.
int chunk_length(const Geom& g, int stages, int tiles, int N) {
  constexpr int kSeen = 32;
  struct Seen { int stages, bw, RT, tiles, N, cs; };
  static thread_local Seen seen[kSeen] = {};
  Seen& m = seen[(unsigned)(stages * 31 + g.bw * 7 + g.RT + tiles * 13 + N) % kSeen];
  if (m.cs && m.stages == stages && m.bw == g.bw && m.RT == g.RT && m.tiles == tiles && m.N == N) return m.cs;
  static const int kTypical[4] = {16, 32, 48, 112};
  const int* const set = tiles ? &tiles : kTypical;
  const int n = tiles ? 1 : 4;
  double least[4];
  for (int k = 0; k < n; ++k) {
    long long lo = -1;
    for (int c = 1; c <= std::min(stages, 32); ++c) {
      const long long v = chunk_cost(g, stages, set[k], N, (stages + c - 1) / c);
      if (lo < 0 || v < lo) lo = v;
    }
    least[k] = (double)lo;
  }
  double best = -1.;
  int cs = stages;
  for (int c = std::min(stages, 32); c >= 1; --c) {
    const int len = (stages + c - 1) / c;
    double sum = 0.;
    for (int k = 0; k < n; ++k) sum += (double)chunk_cost(g, stages, set[k], N, len) / least[k];
    if (best < 0. || sum < best) { best = sum; cs = len; }
  }
  m = {stages, g.bw, g.RT, tiles, N, cs};
  return cs;
}

FusedPlan make_plan(const Geom& g, int M, int NP, bool any_rows) {
  FusedPlan pl = {};
  pl.N = (M + 15) / 16 * 16;
  if (pl.N > kFusedMaxN) return pl;
  // three products over columns that are a third or more padding cost more than a GEMM over those that exist (1600 x 6000,
  // Q = 40, fp32: 62 against 55 us at 128 rows, even at 96)
  if (NP == 3 && pl.N > 96 && 64 * g.QT > 3 * g.Q) return pl;
  const int RT = g.RT;
  // Shared memory: at least two of everything, with as many bit layers per plane stage as that leaves room for; then deeper
  // rings while there is room, x first (a round trip for x is longer than a stage).
  pl.nb = 0;
  auto fits = [&](int nb, int ns, int nx) { return (size_t)FusedSmem(NP, RT, pl.N, nb, ns, nx).total <= kMaxSmem; };
  for (int nb = std::min(g.bw, kFusedBits / RT); nb >= 1 && !pl.nb; --nb) {
    if (!fits(nb, 2, 2)) continue;
    pl.nb = nb;
    pl.ns = pl.nx = 2;
    for (bool more = true; more;) {
      more = false;
      if (pl.nx < 4 && fits(nb, pl.ns, pl.nx + 1)) { ++pl.nx; more = true; }
      if (pl.ns < kFusedMaxPlaneStages && fits(nb, pl.ns + 1, pl.nx)) { ++pl.ns; more = true; }
    }
    pl.smem = FusedSmem(NP, RT, pl.N, nb, pl.ns, pl.nx).total;
  }
  if (!pl.nb) return pl;
  pl.stages = g.JG * g.QT;
  pl.Kp = pl.stages * kFusedStageCols;
  pl.tiles = (g.rw * g.PT + 3) / 4;
  pl.chunk_stages = chunk_length(g, pl.stages, any_rows ? 0 : pl.tiles, pl.N);
  pl.chunks = (pl.stages + pl.chunk_stages - 1) / pl.chunk_stages;
  pl.partial_bytes = pl.chunks > 1 ? up256((size_t)pl.tiles * pl.chunks * pl.N * kFusedTile * 4) : 0;
  pl.x_bytes = up256((size_t)M * pl.Kp * 2) + 1024;         // and the factors of the rows
  pl.ok = true;
  return pl;
}

template <int NP, int RT>
int launch(const CUtensorMap& hi, const CUtensorMap& lo, const CUtensorMap& my, const CUtensorMap& mz, const FusedParams& p, const FusedPlan& pl, cudaStream_t st) {
  auto kern = bqq_fused_kernel<NP, RT>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess) return BQQ_ERR_CUDA;
  cudaLaunchAttribute attr[1] = {pdl_attribute()};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(pl.tiles * pl.chunks, 148));
  cfg.blockDim = dim3(kFusedThreads);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kern, hi, lo, my, mz, p) != cudaSuccess) { cudaGetLastError(); return BQQ_ERR_CUDA; }
  return launch_status();
}

}  // namespace

// Scratch beyond the counters: the larger of the ways x may come in (0: not for this many rows).
size_t fused_workspace_bytes(const Geom& g, int M) {
  size_t need = 0;
  for (int NP = 1; NP <= 3; ++NP) {
    const FusedPlan pl = make_plan(g, M, NP, M <= BQQ_DECODE_MAX_M);
    if (!pl.ok) continue;
    need = std::max(need, pl.partial_bytes + (size_t)(NP == 3 ? 2 : 1) * pl.x_bytes);
  }
  return need;
}
size_t fused_counter_words(const Geom& g) { return ((size_t)g.rw * g.PT + 3) / 4; }

int fused_launch(const BqqLayer* L, const void* x, int x_dtype, int M, int64_t ldx, void* y, int y_dtype, int64_t ldy,
                 unsigned* counters, unsigned* status, bool clear, void* scratch, const BqqFusion* fusion, cudaStream_t st) {
  const Geom g(L->dims);
  const bool prologue = fusion && fusion->prologue != BQQ_PRO_NONE;
  const int NP = x_dtype == BQQ_F32 || prologue ? 3 : M > BQQ_DECODE_MAX_M ? 1 : x_dtype == BQQ_BF16 ? 2 : 3;
  const FusedPlan pl = make_plan(g, M, NP, M <= BQQ_DECODE_MAX_M);
  if (!pl.ok) return BQQ_ERR_UNSUPPORTED;
  uint8_t* sc = reinterpret_cast<uint8_t*>(scratch);
  uint16_t* xhi = reinterpret_cast<uint16_t*>(sc + pl.partial_bytes);
  uint16_t* xlo = reinterpret_cast<uint16_t*>(sc + pl.partial_bytes + pl.x_bytes);
  float* unscale = reinterpret_cast<float*>(sc + pl.partial_bytes + pl.x_bytes - 1024);
  // rows in the kernel's own format and column order are read where they are
  const bool direct = x_dtype == (NP == 1 ? BQQ_F16 : BQQ_BF16) && NP != 3 && g.Q == 32 && ldx % 8 == 0 && ((uintptr_t)x & 15) == 0;

  FusedParams p;
  p.zp = L->zplanes; p.yp = L->yplanes;
  p.a = L->a; p.b = L->b; p.c = L->c; p.d = L->d; p.bias = L->bias;
  p.res = fusion ? fusion->residual : nullptr;
  p.ld_res = fusion ? fusion->ld_residual : 0;
  p.res_dtype = fusion ? fusion->residual_dtype : 0;
  p.y = y; p.ldy = ldy; p.y_dtype = y_dtype;
  p.partial = reinterpret_cast<float*>(sc);
  p.counters = counters;
  p.status = status;
  p.coef_dtype = L->coef_dtype; p.bias_dtype = L->bias_dtype;
  p.g = g;
  p.M = M; p.N = pl.N;
  p.nb = pl.nb; p.ns = pl.ns; p.nx = pl.nx;
  p.row_unscale = NP == 1 && x_dtype == BQQ_BF16 ? unscale : nullptr;
  p.tiles = pl.tiles; p.chunks = pl.chunks; p.chunk_stages = pl.chunk_stages; p.stages = pl.stages;
  // fp32 accumulators, both operands fp16 or bf16, K-major; M = 128, N rows of x
  const uint32_t fmt = NP == 1 ? 0u : 1u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(pl.N >> 3) << 17) | (8u << 24);

  p.joint = g.PT == 1 && pl.nb == g.bw;
  CUtensorMap hi, lo, my, mz;
  int rc = direct ? make_map(&hi, x, NP != 1, (uint64_t)M, (uint64_t)g.in_features(), (uint64_t)ldx, (uint32_t)pl.N)
                  : make_map(&hi, xhi, NP != 1, (uint64_t)M, (uint64_t)pl.Kp, (uint64_t)pl.Kp, (uint32_t)pl.N);
  if (rc) return rc;
  if (NP == 3) {
    rc = make_map(&lo, xlo, true, (uint64_t)M, (uint64_t)pl.Kp, (uint64_t)pl.Kp, (uint32_t)pl.N);
    if (rc) return rc;
  } else {
    lo = hi;
  }
  rc = make_plane_maps(&my, &mz, g, L->yplanes, L->zplanes, (uint32_t)(p.joint ? 4 * pl.nb : pl.nb));
  if (rc) return rc;
  if (!direct || clear) {
    const XSource xs = {x, fusion ? fusion->norm_weight : nullptr, ldx, x_dtype, fusion ? fusion->norm_dtype : 0,
                        prologue ? fusion->prologue : BQQ_PRO_NONE, g.in_features(), fusion ? fusion->eps : 0.f};
    cudaLaunchAttribute attr[1] = {pdl_attribute()};
    cudaLaunchConfig_t cfg = {};
    const bool wide = !direct && xs.n_in > kPrepLong;
    const int threads = wide ? kPrepWide : kPrepThreads, per = 8 * threads;
    const int parts = std::min((pl.Kp + per - 1) / per, wide ? 64 : 148 / M);
    cfg.gridDim = direct ? dim3(1) : dim3((unsigned)parts, (unsigned)M);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int nzero = clear ? pl.tiles : 0;
    uint16_t* h = direct ? nullptr : xhi;
    unsigned* stw = clear ? status : nullptr;
    float* un = const_cast<float*>(p.row_unscale);
    auto kern = wide ? (NP == 1 ? fused_prep_kernel<1, kPrepWide> : NP == 2 ? fused_prep_kernel<2, kPrepWide> : fused_prep_kernel<3, kPrepWide>)
                     : (NP == 1 ? fused_prep_kernel<1, kPrepThreads> : NP == 2 ? fused_prep_kernel<2, kPrepThreads> : fused_prep_kernel<3, kPrepThreads>);
    // an SM keeps its split of L1 and shared memory until it is empty: the one that the fused kernel needs
    if (cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess) {
      cudaGetLastError();
      return BQQ_ERR_CUDA;
    }
    if (cudaLaunchKernelEx(&cfg, kern, xs, M, g, pl.Kp, h, xlo, un, counters, nzero, stw) != cudaSuccess) {
      cudaGetLastError();
      return BQQ_ERR_CUDA;
    }
  }
  if (NP == 1) return g.RT == 1 ? launch<1, 1>(hi, lo, my, mz, p, pl, st) : launch<1, 2>(hi, lo, my, mz, p, pl, st);
  if (NP == 2) return g.RT == 1 ? launch<2, 1>(hi, lo, my, mz, p, pl, st) : launch<2, 2>(hi, lo, my, mz, p, pl, st);
  return g.RT == 1 ? launch<3, 1>(hi, lo, my, mz, p, pl, st) : launch<3, 2>(hi, lo, my, mz, p, pl, st);
}

}  // namespace bqq
