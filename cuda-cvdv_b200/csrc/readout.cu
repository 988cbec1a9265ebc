// Readouts: state I/O, norm, fidelities, marginals and <n>.
//
// Reductions are two-level and deterministic where they produce a scalar: a
// fixed grid writes one partial per block, a single block sums the partials in
// a fixed order.  Marginals of single registers have one owner per partial
// (k_marg_axis), several registers above a tile share one pass (k_marg_tiles), and
// those of registers above a row program's come from the row sums it wrote.  Joint
// marginals accumulate per-block shared-memory histograms with warp aggregation (one
// shared atomic per warp when every lane of the warp falls in the same bin, which is
// the case whenever the selected registers are not the lowest 5 index bits), then sum
// the per-block histograms bin by bin; past the histogram's size they use global atomics.

#include <cmath>
#include <cstring>
#include <mutex>

#include "../../include/cvdv.h"
#include "cvdv_internal.cuh"

using namespace cvdv;
struct CVDVContext : public cvdv::Context {};

namespace cvdv {

constexpr int kRedBlocks = 148 * 4;
constexpr int kRedThreads = 256;

template <typename C> __device__ __forceinline__ double2 tod(C v);
template <> __device__ __forceinline__ double2 tod<double2>(double2 v) { return v; }
template <> __device__ __forceinline__ double2 tod<float2>(float2 v) {
  return make_double2((double)v.x, (double)v.y);
}

__device__ __forceinline__ double2 block_sum2(double2 v) {
  __shared__ double2 ws[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) ws[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < (int)(blockDim.x >> 5) ? ws[lane] : make_double2(0.0, 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v.x += __shfl_down_sync(0xffffffffu, v.x, o);
      v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
  }
  return v;
}

__global__ void k_final_sum(const double2* __restrict__ part, int n, double2* out) {
  double2 a = make_double2(0.0, 0.0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    a.x += part[i].x;
    a.y += part[i].y;
  }
  a = block_sum2(a);
  if (threadIdx.x == 0) *out = a;
}

// ---- functors for the generic reduction: return a double2 per index
template <typename C>
struct OpNorm {  // sum |psi|^2    (measure.cu:276-300)
  const C* st;
  __device__ double2 operator()(uint64_t i) const {
    double2 v = tod<C>(st[i]);
    return make_double2(v.x * v.x + v.y * v.y, 0.0);
  }
};

template <typename C1, typename C2>
struct OpDot {  // sum conj(a) b   (kernelInnerProductStatevectors, measure.cuh:227-252)
  const C1* a;
  const C2* b;
  __device__ double2 operator()(uint64_t i) const {
    double2 x = tod<C1>(a[i]), y = tod<C2>(b[i]);
    return make_double2(x.x * y.x + x.y * y.y, x.x * y.y - x.y * y.x);
  }
};

template <typename C>
struct OpSep {  // sum conj(psi) * outer[i >> qLast] * last[i & m]   (measure.cuh:182-223)
  const C* st;
  const double2* outer;
  const double2* last;
  int qLast;
  __device__ double2 operator()(uint64_t i) const {
    double2 v = tod<C>(st[i]);
    double2 p = dmul(__ldg(last + (i & ((1ull << qLast) - 1))), __ldg(outer + (i >> qLast)));
    return make_double2(v.x * p.x + v.y * p.y, v.x * p.y - v.y * p.x);
  }
};

template <typename Op>
__global__ void __launch_bounds__(kRedThreads) k_reduce(Op op, uint64_t n, double2* part) {
  double2 a = make_double2(0.0, 0.0);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // four terms evaluated before they are added, so four loads are in flight
  for (; i + 3 * stride < n; i += 4 * stride) {
    const double2 v0 = op(i), v1 = op(i + stride), v2 = op(i + 2 * stride), v3 = op(i + 3 * stride);
    a.x += (v0.x + v1.x) + (v2.x + v3.x);
    a.y += (v0.y + v1.y) + (v2.y + v3.y);
  }
  for (; i < n; i += stride) {
    const double2 v = op(i);
    a.x += v.x;
    a.y += v.y;
  }
  a = block_sum2(a);
  if (threadIdx.x == 0) part[blockIdx.x] = a;
}

template <typename Op>
static bool reduce(Context* ctx, Op op, uint64_t n, double2* result) {
  double2* part = (double2*)arena_alloc(ctx, (kRedBlocks + 1) * sizeof(double2));
  if (!part) return false;
  double* hs = host_scratch(ctx, 2);
  if (!hs) return false;
  {
    LaunchScope _ls(ctx, kKReduce);
    k_reduce<Op><<<kRedBlocks, kRedThreads, 0, ctx->stream>>>(op, n, part);
  }
  {
    LaunchScope _ls(ctx, kKReduce);
    k_final_sum<<<1, 1024, 0, ctx->stream>>>(part, kRedBlocks, part + kRedBlocks);
  }
  if (!cuda_ok(ctx, cudaGetLastError(), "reduce launch")) return false;
  if (!cuda_ok(ctx, cudaMemcpyAsync(hs, part + kRedBlocks, sizeof(double2), cudaMemcpyDeviceToHost,
                                    ctx->stream),
               "reduce copy"))
    return false;
  if (!stream_sync(ctx, "reduce sync")) return false;
  *result = make_double2(hs[0], hs[1]);
  return true;
}

// ----------------------------------------------------------------- marginals
struct MargDesc {
  int nSel;
  int shift[16];
  int mask[16];
  long long stride[16];
  long long outSize;
};

__device__ __forceinline__ long long marg_bin(const MargDesc& D, uint64_t i) {
  long long oi = 0;
  for (int s = 0; s < D.nSel; ++s) oi += (long long)((i >> D.shift[s]) & (uint64_t)D.mask[s]) * D.stride[s];
  return oi;
}

// smem histogram per block -> part[block][bin]
template <typename C>
__global__ void __launch_bounds__(256) k_marg_smem(const C* __restrict__ st, uint64_t n,
                                                  MargDesc D, double* __restrict__ part) {
  extern __shared__ double hist[];
  for (int b = threadIdx.x; b < D.outSize; b += blockDim.x) hist[b] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t warpStride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n;
       base += warpStride) {
    uint64_t i = base + lane;
    double p = 0.0;
    long long bin = 0;
    if (i < n) {
      double2 v = tod<C>(st[i]);
      p = v.x * v.x + v.y * v.y;
      bin = marg_bin(D, i);
    }
    long long b0 = __shfl_sync(0xffffffffu, bin, 0);
    bool same = __all_sync(0xffffffffu, (i >= n) || bin == b0);
    if (same) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) p += __shfl_down_sync(0xffffffffu, p, o);
      if (lane == 0) atomicAdd(&hist[b0], p);
    } else if (i < n) {
      atomicAdd(&hist[bin], p);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < D.outSize; b += blockDim.x)
    part[(size_t)blockIdx.x * D.outSize + b] = hist[b];
}

// out[b] = sum over the nb blocks' partials, in a fixed order: 32 bins per CTA (x, so
// a warp reads a run of each block's row), kFinalY threads per bin that each add every
// kFinalY-th partial, then a fixed tree.  One thread per bin added the partials one
// after the other (up to 592 dependent adds: 33-66 us however few the bins).
constexpr int kFinalY = 32;
__device__ __forceinline__ double final_sum(const double* __restrict__ part, int nb, long long stride, long long b,
                                            bool ok) {
  __shared__ double red[kFinalY][33];
  double a = 0.0;
  if (ok) {
#pragma unroll 4
    for (int k = threadIdx.y; k < nb; k += kFinalY) a += part[(size_t)k * stride + b];
  }
  red[threadIdx.y][threadIdx.x] = a;
  __syncthreads();
#pragma unroll
  for (int o = kFinalY / 2; o > 0; o >>= 1) {
    if (threadIdx.y < o) red[threadIdx.y][threadIdx.x] += red[threadIdx.y + o][threadIdx.x];
    __syncthreads();
  }
  return red[0][threadIdx.x];
}

__global__ void __launch_bounds__(32 * kFinalY) k_marg_final(const double* __restrict__ part, int nb, long long outSize,
                                                            double* __restrict__ out) {
  const long long b = (long long)blockIdx.x * 32 + threadIdx.x;
  const double v = final_sum(part, nb, outSize, b, b < outSize);
  if (threadIdx.y == 0 && b < outSize) out[b] = v;
}
static void launch_marg_final(const double* part, int nb, long long outSize, double* out, cudaStream_t s) {
  k_marg_final<<<(unsigned)((outSize + 31) / 32), dim3(32, kFinalY), 0, s>>>(part, nb, outSize, out);
}

// large outputs: global atomics (warp-aggregated when the warp shares a bin)
template <typename C>
__global__ void __launch_bounds__(256) k_marg_global(const C* __restrict__ st, uint64_t n,
                                                    MargDesc D, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const uint64_t warpStride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n;
       base += warpStride) {
    uint64_t i = base + lane;
    double p = 0.0;
    long long bin = 0;
    if (i < n) {
      double2 v = tod<C>(st[i]);
      p = v.x * v.x + v.y * v.y;
      bin = marg_bin(D, i);
    }
    long long b0 = __shfl_sync(0xffffffffu, bin, 0);
    bool same = __all_sync(0xffffffffu, (i >= n) || bin == b0);
    if (same) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) p += __shfl_down_sync(0xffffffffu, p, o);
      if (lane == 0) atomicAdd(&out[b0], p);
    } else if (i < n) {
      atomicAdd(&out[bin], p);
    }
  }
}

// Tiled marginals: several outputs (each the joint marginal of some registers) in
// one pass.  A block reads tiles of 256 x 16 consecutive amplitudes.  An output
// whose registers all lie above the tile's 12 index bits has one bin per tile:
// the block sums the tile once and thread 0 adds it (no atomics at all, which
// is the case for every qubit register of a mode-last layout).  Other outputs
// bin each amplitude with warp-aggregated shared atomics.
constexpr int kMargLogV = 4;
constexpr int kMargLogTile = 8 + kMargLogV;
constexpr int kMargMaxOut = 16;
constexpr int kMargSmemBins = 4096;

struct MargOut {
  int nSel, sel0, off, high;
};
struct MargPlan {
  int nOut, nHigh, totalBins;
  int shift[16], mask[16], stride[16];
  MargOut out[kMargMaxOut];
};

__device__ __forceinline__ int marg_out_bin(const MargPlan& P, const MargOut& O, uint64_t i) {
  int b = 0;
  for (int s = 0; s < O.nSel; ++s)
    b += (int)((i >> P.shift[O.sel0 + s]) & (uint64_t)P.mask[O.sel0 + s]) * P.stride[O.sel0 + s];
  return b;
}

template <typename C>
__global__ void __launch_bounds__(256) k_marg_tiles(const C* __restrict__ st, uint64_t nTiles,
                                                   const __grid_constant__ MargPlan P,
                                                   double* __restrict__ part) {
  constexpr int V = 1 << kMargLogV;
  extern __shared__ double hist[];
  __shared__ double red[8];
  for (int b = threadIdx.x; b < P.totalBins; b += blockDim.x) hist[b] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint64_t tile = blockIdx.x; tile < nTiles; tile += gridDim.x) {
    const uint64_t t0 = tile << kMargLogTile;
    double p[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const double2 a = tod<C>(st[t0 + threadIdx.x + (v << 8)]);
      p[v] = a.x * a.x + a.y * a.y;
    }
    if (P.nHigh < P.nOut) {
      for (int o = 0; o < P.nOut; ++o) {
        const MargOut& O = P.out[o];
        if (O.high) continue;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int bin = marg_out_bin(P, O, t0 + threadIdx.x + (v << 8));
          const int b0 = __shfl_sync(0xffffffffu, bin, 0);
          if (__all_sync(0xffffffffu, bin == b0)) {
            double q = p[v];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) q += __shfl_down_sync(0xffffffffu, q, d);
            if (lane == 0) atomicAdd(&hist[O.off + b0], q);
          } else {
            atomicAdd(&hist[O.off + bin], p[v]);
          }
        }
      }
    }
    if (P.nHigh) {
      double q = 0.0;
#pragma unroll
      for (int v = 0; v < V; ++v) q += p[v];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) q += __shfl_down_sync(0xffffffffu, q, d);
      if (lane == 0) red[warp] = q;
      __syncthreads();
      if (threadIdx.x == 0) {
        double S = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) S += red[w];
        for (int o = 0; o < P.nOut; ++o)
          if (P.out[o].high) hist[P.out[o].off + marg_out_bin(P, P.out[o], t0)] += S;
      }
      __syncthreads();
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < P.totalBins; b += blockDim.x)
    part[(size_t)blockIdx.x * P.totalBins + b] = hist[b];
}

// One pass for `outs` (each a list of registers, first fastest); every output
// must have at most kMargSmemBins bins in total and the state at least one tile.
// dOut receives the outputs back to back.
static bool marginals_tiled(Context* ctx, const std::vector<std::vector<int>>& outs, double* dOut) {
  MargPlan P{};
  int sel = 0;
  for (const auto& regs : outs) {
    MargOut& O = P.out[P.nOut++];
    O.nSel = (int)regs.size();
    O.sel0 = sel;
    O.off = P.totalBins;
    O.high = 1;
    int stride = 1;
    for (int r : regs) {
      P.shift[sel] = ctx->flw[r];
      P.mask[sel] = (1 << ctx->q[r]) - 1;
      P.stride[sel] = stride;
      stride <<= ctx->q[r];
      if (ctx->flw[r] < kMargLogTile) O.high = 0;
      ++sel;
    }
    P.nHigh += O.high;
    P.totalBins += stride;
  }
  const uint64_t nTiles = ctx->size() >> kMargLogTile;
  uint64_t blocks = P.totalBins <= 256 ? 148ull * 4 : 148ull * 2;
  if (blocks > nTiles) blocks = nTiles;
  double* part = (double*)arena_alloc(ctx, (size_t)blocks * P.totalBins * sizeof(double));
  if (!part) return false;
  const size_t smem = (size_t)P.totalBins * sizeof(double);
  {
    LaunchScope _ls(ctx, kKReduce);
    if (ctx->precision == kC128)
      k_marg_tiles<double2><<<(unsigned)blocks, 256, smem, ctx->stream>>>((const double2*)ctx->state(), nTiles, P, part);
    else
      k_marg_tiles<float2><<<(unsigned)blocks, 256, smem, ctx->stream>>>((const float2*)ctx->state(), nTiles, P, part);
  }
  {
    LaunchScope _ls(ctx, kKReduce);
    launch_marg_final(part, (int)blocks, P.totalBins, dOut, ctx->stream);
  }
  return cuda_ok(ctx, cudaGetLastError(), "marginal launch");
}

// Marginals of single registers without atomics: every register is a job, all jobs
// of a readout share one launch, and a CTA works for one job.  With N = 2^q values
// and S = 2^s amplitudes below the register:
//   S >= 32: a value's amplitudes are runs of S; G threads (a CTA, or a warp where a
//     value has few amplitudes) add a slice of one value's amplitudes;
//   S < 32:  a thread keeps one position of the inner N S amplitudes (or of a CTA's
//     256) and adds it over a slice of the outer index; the S neighbours of a value
//     are added at the end.
// Either way a CTA's loads are contiguous and each partial has one owner.  The slices
// of a value are added by k_axis_final in a fixed order.  Binning each amplitude with
// shared-memory atomics, or with one global atomic past 4096 values, and adding the
// blocks' partials with one thread per value took 126 us for the four registers of a
// 2^20 complex128 state ([2, 8, 9, 1], now 29) and 589 us for both of a 2^26 one
// ([13, 13], now 337: two reads of the state, 330 at the copy rate).
struct AxisJob {
  int shift, q;
  int logG;     // S >= 32: log2 of the threads per value (5 or 8)
  int slices;   // partials per value
  int block0;   // first CTA
  double* dst;  // partial [slice][value], or the output itself with one slice
};
struct AxisPlan {
  int nJobs;
  AxisJob job[kMargMaxOut];
};

template <typename C>
__device__ __forceinline__ double prob_at(const C* __restrict__ st, uint64_t i) {
  const double2 v = tod<C>(st[i]);
  return v.x * v.x + v.y * v.y;
}

template <typename C>
__global__ void __launch_bounds__(256) k_marg_axis(const C* __restrict__ st, int logTotal,
                                                  const __grid_constant__ AxisPlan A) {
  __shared__ double red[256];
  int jb = 0;
  while (jb + 1 < A.nJobs && (int)blockIdx.x >= A.job[jb + 1].block0) ++jb;
  const AxisJob& J = A.job[jb];
  const uint64_t cta = (uint64_t)((int)blockIdx.x - J.block0);
  const int tid = threadIdx.x, s = J.shift, q = J.q;
  double a = 0.0;
  if (s >= 5) {
    // unit = (slice, value); its amplitudes u map to ((u >> s) << (s + q)) | j << s | (u mod S)
    const int G = 1 << J.logG;
    const uint64_t unit = (cta << (8 - J.logG)) + (uint64_t)(tid >> J.logG);
    const uint64_t j = unit & ((1ull << q) - 1), k = unit >> q;
    const uint64_t len = (1ull << (logTotal - q)) / (uint64_t)J.slices, sm = (1ull << s) - 1;
    const bool ok = k < (uint64_t)J.slices;
    if (ok) {
      const uint64_t end = (k + 1) * len;
#pragma unroll 4
      for (uint64_t u = k * len + (uint64_t)(tid & (G - 1)); u < end; u += G)
        a += prob_at(st, ((u & ~sm) << q) | (j << s) | (u & sm));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (G > 32) {
      if ((tid & 31) == 0) red[tid >> 5] = a;
      __syncthreads();
      a = ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
    }
    if (ok && (tid & (G - 1)) == 0) J.dst[unit] = a;
    return;
  }
  // positions of the inner block: a CTA holds 256 of them for one slice, or (shorter
  // blocks) 256 / P outer values at once
  const int logP = s + q;
  if (logP >= 8) {
    const uint64_t chunks = 1ull << (logP - 8), ch = cta & (chunks - 1), k = cta >> (logP - 8);
    const uint64_t outer = 1ull << (logTotal - logP), len = outer / (uint64_t)J.slices;
    const uint64_t pos = (ch << 8) + tid;
#pragma unroll 4
    for (uint64_t o = k * len; o < (k + 1) * len; ++o) a += prob_at(st, (o << logP) | pos);
    for (int o = 1; o < (1 << s); o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((tid & ((1 << s) - 1)) == 0) J.dst[(k << q) + (pos >> s)] = a;
    return;
  }
  const uint64_t total = 1ull << logTotal, len = total / (uint64_t)J.slices, end = (cta + 1) * len;
#pragma unroll 4
  for (uint64_t i = cta * len + tid; i < end; i += 256) a += prob_at(st, i);
  red[tid] = a;
  __syncthreads();
  if (tid < (1 << q)) {  // value tid: threads whose index has it in bits s .. s + q
    double b = 0.0;
    for (int u = 0; u < (256 >> q); ++u) b += red[((u >> s) << logP) | (tid << s) | (u & ((1 << s) - 1))];
    J.dst[(cta << q) + tid] = b;
  }
}

// The slices of every job that has more than one, to their outputs.
struct AxisFinal {
  int nJobs;
  struct {
    const double* part;
    double* out;
    int q, slices, block0;
  } job[kMargMaxOut];
};
__global__ void __launch_bounds__(32 * kFinalY) k_axis_final(const __grid_constant__ AxisFinal A) {
  int jb = 0;
  while (jb + 1 < A.nJobs && (int)blockIdx.x >= A.job[jb + 1].block0) ++jb;
  const long long N = 1ll << A.job[jb].q, b = (long long)((int)blockIdx.x - A.job[jb].block0) * 32 + threadIdx.x;
  const double v = final_sum(A.job[jb].part, A.job[jb].slices, N, b, b < N);
  if (threadIdx.y == 0 && b < N) A.job[jb].out[b] = v;
}

// Marginal of register regs[k] to dOut + pos[k], for all k (at most kMargMaxOut).
static bool marginals_axis(Context* ctx, const std::vector<int>& regs, const std::vector<size_t>& pos, double* dOut) {
  AxisPlan A{};
  AxisFinal F{};
  const int n = ctx->totalQbt;
  long long blocks = 0, finals = 0;
  for (size_t k = 0; k < regs.size(); ++k) {
    AxisJob& J = A.job[A.nJobs++];
    const int s = ctx->flw[regs[k]], q = ctx->q[regs[k]], logP = s + q;
    J.shift = s;
    J.q = q;
    // slices: CTAs for eight per SM, while a thread keeps at least four loads
    const long long want = 8ll * ctx->numSMs;
    int logSl = 0;
    long long ctas;
    if (s >= 5) {
      J.logG = n - q >= 10 ? 8 : 5;  // a CTA per slice where values have 2^10 amplitudes or more
      while ((((1ll << q) << logSl) >> (8 - J.logG)) < want && n - q - logSl > J.logG + 2) ++logSl;
      ctas = (((1ll << q) << logSl) + (256 >> J.logG) - 1) >> (8 - J.logG);
    } else if (logP >= 8) {
      while (((1ll << (logP - 8)) << logSl) < want && n - logP - logSl > 2) ++logSl;
      ctas = (1ll << (logP - 8)) << logSl;
    } else {
      while ((1ll << logSl) < want && n - logSl > 10) ++logSl;
      ctas = 1ll << logSl;
    }
    J.slices = 1 << logSl;
    J.block0 = (int)blocks;
    blocks += ctas;
    J.dst = dOut + pos[k];
    if (logSl == 0) continue;
    J.dst = (double*)arena_alloc(ctx, ((size_t)1 << (q + logSl)) * sizeof(double));
    if (!J.dst) return false;
    auto& f = F.job[F.nJobs++];
    f.part = J.dst;
    f.out = dOut + pos[k];
    f.q = q;
    f.slices = J.slices;
    f.block0 = (int)finals;
    finals += ((1ll << q) + 31) / 32;
  }
  {
    LaunchScope _ls(ctx, kKReduce);
    if (ctx->precision == kC128)
      k_marg_axis<double2><<<(unsigned)blocks, 256, 0, ctx->stream>>>((const double2*)ctx->state(), n, A);
    else
      k_marg_axis<float2><<<(unsigned)blocks, 256, 0, ctx->stream>>>((const float2*)ctx->state(), n, A);
  }
  if (finals) {
    LaunchScope _ls(ctx, kKReduce);
    k_axis_final<<<(unsigned)finals, dim3(32, kFinalY), 0, ctx->stream>>>(F);
  }
  return cuda_ok(ctx, cudaGetLastError(), "marginal launch");
}

// Marginals of registers above the last one from the row sums the flush's last
// row program wrote (a row = one value of every register but the last): the rows'
// partials are added in a fixed order, then one CTA per output bin adds the rows
// with that register value in a fixed tree.
__global__ void k_row_total(const double* __restrict__ parts, int P, uint64_t rows, double* __restrict__ tot) {
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (uint64_t)gridDim.x * blockDim.x) {
    double a = 0.0;
    for (int p = 0; p < P; ++p) a += parts[r * P + p];
    tot[r] = a;
  }
}

struct RowMarg {
  int nOut;
  int shift[kMargMaxOut], q[kMargMaxOut], off[kMargMaxOut];  // register field in the row index; output offset
};

__global__ void __launch_bounds__(256) k_row_marg(const double* __restrict__ tot, uint64_t rows,
                                                  const __grid_constant__ RowMarg M, double* __restrict__ out) {
  int o = 0;
  while (o + 1 < M.nOut && (int)blockIdx.x >= M.off[o + 1]) ++o;
  const uint64_t v = (uint64_t)(blockIdx.x - M.off[o]);
  const int sh = M.shift[o], q = M.q[o];
  const uint64_t cnt = rows >> q, low = (1ull << sh) - 1;
  double a = 0.0;
  for (uint64_t i = threadIdx.x; i < cnt; i += blockDim.x)
    a += tot[((i & ~low) << q) | (v << sh) | (i & low)];
  const double2 s = block_sum2(make_double2(a, 0.0));
  if (threadIdx.x == 0) out[blockIdx.x] = s.x;
}

static bool marginals_from_rows(Context* ctx, const std::vector<int>& regs, int parts, double* dOut) {
  const int last = ctx->numReg - 1;
  const uint64_t rows = ctx->size() >> ctx->q[last];
  RowMarg M{};
  int bins = 0;
  for (int r : regs) {
    M.shift[M.nOut] = ctx->flw[r] - ctx->q[last];
    M.q[M.nOut] = ctx->q[r];
    M.off[M.nOut++] = bins;
    bins += 1 << ctx->q[r];
  }
  double* tot = (double*)arena_alloc(ctx, rows * sizeof(double));
  if (!tot) return false;
  {
    LaunchScope _ls(ctx, kKReduce);
    k_row_total<<<(unsigned)((rows + 255) / 256 < 1184 ? (rows + 255) / 256 : 1184), 256, 0, ctx->stream>>>(
        ctx->rowSumBuf, parts, rows, tot);
  }
  {
    LaunchScope _ls(ctx, kKReduce);
    k_row_marg<<<bins, 256, 0, ctx->stream>>>(tot, rows, M, dOut);
  }
  return cuda_ok(ctx, cudaGetLastError(), "row-sum marginal launch");
}

// Ask the next flush for row sums when every register read is a single register
// above the last one; false (nothing asked) otherwise.
static bool request_row_sums(Context* c, const std::vector<int>& regs) {
  if (c->numReg < 2) return false;
  for (int r : regs)
    if (r == c->numReg - 1) return false;
  const size_t need = (c->size() >> c->q[c->numReg - 1]) * kRowSumMaxParts;
  if (need > c->rowSumCap) {
    cudaStreamSynchronize(c->stream);
    if (c->rowSumBuf) cudaFree(c->rowSumBuf);
    c->rowSumBuf = nullptr;
    c->rowSumCap = 0;
    if (cudaMalloc(&c->rowSumBuf, need * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    c->rowSumCap = need;
  }
  c->rowSums = c->rowSumBuf;
  c->rowSumParts = 0;
  return true;
}

// out[k] = sum_j m_k[j] x_j^2 of the two marginals m_0, m_1 of a register (block k), the
// second moment of a marginal in place of a weighted sum over the state
// (kernelExpectX2, measure.cuh:158-178), which converted every amplitude's index to x.
// With the transform as one row or column program instead of tile passes and one wait
// instead of two, the readouts of a 2^22 state (two photon numbers among them) take 518 us
// instead of 726.
__global__ void __launch_bounds__(256) k_second_moments(const double* __restrict__ m, int N, double dx,
                                                        double* __restrict__ out) {
  const double* p = m + (size_t)blockIdx.x * N;
  double a = 0.0;
  for (int j = threadIdx.x; j < N; j += 256) {
    const double x = ((double)j - (double)(N - 1) * 0.5) * dx;
    a += p[j] * x * x;
  }
  const double2 s = block_sum2(make_double2(a, 0.0));
  if (threadIdx.x == 0) out[blockIdx.x] = s.x;
}

static bool tiled_ok(Context* ctx, long long bins) {
  return bins <= kMargSmemBins && ctx->totalQbt >= kMargLogTile;
}

static bool marginal_device(Context* ctx, const int* regs, int nr, double** dOut, long long* outSize) {
  MargDesc D{};
  D.nSel = nr;
  long long stride = 1;
  for (int s = 0; s < nr; ++s) {
    D.shift[s] = ctx->flw[regs[s]];
    D.mask[s] = (1 << ctx->q[regs[s]]) - 1;
    D.stride[s] = stride;  // column-major: first selected register fastest (measure.cu:89-91)
    stride *= (long long)1 << ctx->q[regs[s]];
  }
  D.outSize = stride;
  *outSize = stride;
  uint64_t n = ctx->size();
  double* out = (double*)arena_alloc(ctx, (size_t)stride * sizeof(double));
  if (!out) return false;
  if (stride <= 4096) {
    int blocks = 148 * 2;
    uint64_t maxBlocks = (n + 255) / 256;
    if ((uint64_t)blocks > maxBlocks) blocks = (int)maxBlocks;
    double* part = (double*)arena_alloc(ctx, (size_t)blocks * stride * sizeof(double));
    if (!part) return false;
    size_t smem = (size_t)stride * sizeof(double);
    if (ctx->precision == kC128)
      {
        LaunchScope _ls(ctx, kKReduce);
        k_marg_smem<double2><<<blocks, 256, smem, ctx->stream>>>((const double2*)ctx->state(), n, D, part);
      }
    else
      {
        LaunchScope _ls(ctx, kKReduce);
        k_marg_smem<float2><<<blocks, 256, smem, ctx->stream>>>((const float2*)ctx->state(), n, D, part);
      }
    {
      LaunchScope _ls(ctx, kKReduce);
      launch_marg_final(part, blocks, stride, out, ctx->stream);
    }
  } else {
    if (!cuda_ok(ctx, cudaMemsetAsync(out, 0, (size_t)stride * sizeof(double), ctx->stream), "memset"))
      return false;
    int blocks = 148 * 8;
    if (ctx->precision == kC128)
      {
        LaunchScope _ls(ctx, kKReduce);
        k_marg_global<double2><<<blocks, 256, 0, ctx->stream>>>((const double2*)ctx->state(), n, D, out);
      }
    else
      {
        LaunchScope _ls(ctx, kKReduce);
        k_marg_global<float2><<<blocks, 256, 0, ctx->stream>>>((const float2*)ctx->state(), n, D, out);
      }
  }
  if (!cuda_ok(ctx, cudaGetLastError(), "marginal launch")) return false;
  *dOut = out;
  return true;
}

// ----------------------------------------------------------------- conversions
__global__ void k_c128_to_c64(const double2* __restrict__ s, float2* __restrict__ d, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    d[i] = make_float2((float)s[i].x, (float)s[i].y);
}

bool launch_convert_c128_to_c64(Context* ctx, const double2* src, float2* dst, uint64_t n) {
  {
    LaunchScope _ls(ctx, kKInit);
    k_c128_to_c64<<<148 * 8, 256, 0, ctx->stream>>>(src, dst, n);
  }
  return cuda_ok(ctx, cudaGetLastError(), "convert launch");
}

template <typename C>
__global__ void k_split(const C* __restrict__ st, uint64_t off, uint64_t cnt, double* __restrict__ re,
                        double* __restrict__ im) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += (uint64_t)gridDim.x * blockDim.x) {
    double2 v = tod<C>(st[off + i]);
    re[i] = v.x;
    im[i] = v.y;
  }
}

}  // namespace cvdv

// ====================================================================== C API
static Context* C(CVDVContext* p) { return static_cast<Context*>(p); }

// Doubles at src[at .. at + count) of a device buffer to host memory `to`.
struct HostPart {
  double* to;
  size_t at, count;
};
// Whether the host can write all parts itself: results may go to device memory too, by
// copy calls only.
static bool host_memory(const std::vector<HostPart>& parts) {
  const double* next = nullptr;
  for (const HostPart& p : parts) {
    if (p.to != next) {  // (parts that follow one another are one array)
      cudaPointerAttributes a{};
      if (cudaPointerGetAttributes(&a, p.to) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      if (a.type == cudaMemoryTypeDevice) return false;
    }
    next = p.to + p.count;
  }
  return true;
}
// Waits for the parts of a device buffer of `total` doubles: small buffers come back
// in one copy to the context's pinned block (a copy per register to pageable memory
// took 10 us each), large parts through copy_to_host.
static bool read_back(Context* c, const std::vector<HostPart>& parts, const double* src, size_t total, const char* what) {
  constexpr size_t kSmall = (Context::kPinnedBytes - Context::kPinnedScratchAt) / sizeof(double);
  constexpr size_t kLarge = (2u << 20) / sizeof(double);
  double* hs = total <= kSmall && host_memory(parts) ? host_scratch(c, total) : nullptr;
  if (hs) {
    if (!cuda_ok(c, cudaMemcpyAsync(hs, src, total * sizeof(double), cudaMemcpyDeviceToHost, c->stream), what) ||
        !stream_sync(c, what))
      return false;
    for (const HostPart& p : parts) memcpy(p.to, hs + p.at, p.count * sizeof(double));
    return true;
  }
  for (const HostPart& p : parts) {
    const bool ok = p.count >= kLarge ? copy_to_host(c, p.to, src + p.at, p.count * sizeof(double), what)
                                      : cuda_ok(c, cudaMemcpyAsync(p.to, src + p.at, p.count * sizeof(double),
                                                                   cudaMemcpyDeviceToHost, c->stream), what);
    if (!ok) return false;
  }
  return stream_sync(c, what);
}

static bool ready(Context* c, const char* what) {
  if (c->numReg == 0 || !c->initialized) {
    set_error(c, kErrNotInitialized, "%s: state not initialised", what);
    return false;
  }
  return flush(c);
}

extern "C" {

int cvdvGetLastError(CVDVContext* ctx, char* msg, int len);

void cvdvGetState(CVDVContext* ctx, double* realOut, double* imagOut) {
  if (!ctx) return;
  Context* c = C(ctx);
  if (!ready(c, "cvdvGetState") || !realOut || !imagOut) return;
  arena_reset(c);
  uint64_t n = c->size();
  const uint64_t chunk = 1ull << 22;
  uint64_t cnt0 = n < chunk ? n : chunk;
  double* dre = (double*)arena_alloc(c, 2 * cnt0 * sizeof(double));
  if (!dre) return;
  double* dim = dre + cnt0;
  for (uint64_t off = 0; off < n; off += chunk) {
    uint64_t cnt = n - off < chunk ? n - off : chunk;
    int blocks = (int)((cnt + 255) / 256 < 1184 ? (cnt + 255) / 256 : 1184);
    if (c->precision == kC128)
      {
        LaunchScope _ls(ctx, kKReduce);
        k_split<double2><<<blocks, 256, 0, c->stream>>>((const double2*)c->state(), off, cnt, dre, dim);
      }
    else
      {
        LaunchScope _ls(ctx, kKReduce);
        k_split<float2><<<blocks, 256, 0, c->stream>>>((const float2*)c->state(), off, cnt, dre, dim);
      }
    // (waits, so the next chunk may overwrite the split arrays)
    if (!read_back(c, {{realOut + off, 0, (size_t)cnt}, {imagOut + off, (size_t)cnt0, (size_t)cnt}}, dre, 2 * (size_t)cnt0,
                   "getState copy"))
      return;
  }
}

double cvdvGetNorm(CVDVContext* ctx) {
  if (!ctx) return 0.0;
  Context* c = C(ctx);
  if (!ready(c, "cvdvGetNorm")) return 0.0;
  arena_reset(c);
  double2 r;
  bool ok = c->precision == kC128
                ? reduce(c, OpNorm<double2>{(const double2*)c->state()}, c->size(), &r)
                : reduce(c, OpNorm<float2>{(const float2*)c->state()}, c->size(), &r);
  return ok ? r.x : 0.0;
}

static bool measure(Context* c, const int* regIdxs, int numRegs, double* probsOut, const char* w) {
  if (!regIdxs || numRegs <= 0 || !probsOut) {
    set_error(c, kErrInvalidArg, "%s: empty register list", w);
    return false;
  }
  if (numRegs > 16) {
    set_error(c, kErrInvalidArg, "%s: at most 16 registers", w);
    return false;
  }
  for (int s = 0; s < numRegs; ++s)
    if (regIdxs[s] < 0 || regIdxs[s] >= c->numReg) {
      set_error(c, kErrInvalidArg, "%s: invalid register index %d", w, regIdxs[s]);
      return false;
    }
  if (!ready(c, w)) return false;
  arena_reset(c);
  long long bins = 1;
  for (int s = 0; s < numRegs; ++s) bins <<= c->q[regIdxs[s]];
  double* dOut;
  long long outSize = bins;
  if (numRegs == 1) {
    dOut = (double*)arena_alloc(c, (size_t)bins * sizeof(double));
    if (!dOut || !marginals_axis(c, {regIdxs[0]}, {0}, dOut)) return false;
  } else if (tiled_ok(c, bins)) {
    dOut = (double*)arena_alloc(c, (size_t)bins * sizeof(double));
    if (!dOut || !marginals_tiled(c, {std::vector<int>(regIdxs, regIdxs + numRegs)}, dOut)) return false;
  } else if (!marginal_device(c, regIdxs, numRegs, &dOut, &outSize)) {
    return false;
  }
  return read_back(c, {{probsOut, 0, (size_t)outSize}}, dOut, (size_t)outSize, "marginal");
}

void cvdvMeasureMultiple(CVDVContext* ctx, const int* regIdxs, int numRegs, double* probsOut) {
  if (!ctx) return;
  measure(C(ctx), regIdxs, numRegs, probsOut, "cvdvMeasureMultiple");
}

void cvdvMeasureMultipleCT(CVDVContext* ctx, const int* regIdxs, int numRegs, double* probsOut) {
  if (!ctx) return;
  measure(C(ctx), regIdxs, numRegs, probsOut, "cvdvMeasureMultipleCT");
}

void cvdvMeasureEach(CVDVContext* ctx, const int* regIdxs, int numRegs, double* probsOut) {
  if (!ctx) return;
  Context* c = C(ctx);
  const char* w = "cvdvMeasureEach";
  if (!regIdxs || numRegs <= 0 || numRegs > kMargMaxOut || !probsOut) {
    set_error(c, kErrInvalidArg, "%s: need 1..%d registers and an output", w, kMargMaxOut);
    return;
  }
  for (int k = 0; k < numRegs; ++k)
    if (regIdxs[k] < 0 || regIdxs[k] >= c->numReg) {
      set_error(c, kErrInvalidArg, "%s: invalid register index %d", w, regIdxs[k]);
      return;
    }
  const std::vector<int> regs(regIdxs, regIdxs + numRegs);
  // qubit registers after a row program on the last register: the program writes
  // the row sums on its way out and the marginals come from them, not another pass
  const bool asked = request_row_sums(c, regs);
  const bool ok = ready(c, w);
  c->rowSums = nullptr;
  if (!ok) return;
  const int parts = asked ? c->rowSumParts : 0;
  c->rowSumParts = 0;
  arena_reset(c);
  // device order: the registers read by one pass of tiles first (several registers
  // above the tile, one block sum per tile serves them all), then the others
  std::vector<int> tiled, axis;
  long long tiledBins = 0;
  for (int k = 0; k < numRegs; ++k) {
    const long long b = 1ll << c->q[regs[k]];
    if (parts > 0 || (c->flw[regs[k]] >= kMargLogTile && tiled_ok(c, tiledBins + b))) {
      tiled.push_back(k);
      tiledBins += b;
    } else {
      axis.push_back(k);
    }
  }
  if (parts == 0 && tiled.size() < 2) {
    axis.insert(axis.begin(), tiled.begin(), tiled.end());
    tiled.clear();
  }
  std::vector<size_t> hostPos(numRegs);
  size_t total = 0;
  for (int k = 0; k < numRegs; ++k) {
    hostPos[k] = total;
    total += (size_t)1 << c->q[regs[k]];
  }
  double* dOut = (double*)arena_alloc(c, total * sizeof(double));
  if (!dOut) return;
  std::vector<HostPart> host;
  size_t at = 0;
  std::vector<std::vector<int>> outs;
  std::vector<int> first, rest;
  std::vector<size_t> restPos;
  for (int k : tiled) {
    first.push_back(regs[k]);
    outs.push_back({regs[k]});
    host.push_back({probsOut + hostPos[k], at, (size_t)1 << c->q[regs[k]]});
    at += host.back().count;
  }
  for (int k : axis) {
    rest.push_back(regs[k]);
    restPos.push_back(at);
    host.push_back({probsOut + hostPos[k], at, (size_t)1 << c->q[regs[k]]});
    at += host.back().count;
  }
  if (!first.empty() && !(parts > 0 ? marginals_from_rows(c, first, parts, dOut) : marginals_tiled(c, outs, dOut))) return;
  if (!rest.empty() && !marginals_axis(c, rest, restPos, dOut)) return;
  read_back(c, host, dOut, total, "marginal");
}

void cvdvGetFidelity(CVDVContext* ctx, void** devicePtrs, int numReg, double* fidOut) {
  if (!ctx) return;
  Context* c = C(ctx);
  if (fidOut) *fidOut = 0.0;
  if (!fidOut || !devicePtrs) {
    set_error(c, kErrInvalidArg, "cvdvGetFidelity: NULL argument");
    return;
  }
  if (numReg != c->numReg) {
    set_error(c, kErrInvalidArg, "cvdvGetFidelity: numReg mismatch (context %d, got %d)",
              c->numReg, numReg);
    return;
  }
  if (!ready(c, "cvdvGetFidelity")) return;
  arena_reset(c);
  size_t totalN = 0;
  for (int r = 0; r < numReg; ++r) totalN += (size_t)1 << c->q[r];
  double2* base = (double2*)arena_alloc(c, totalN * sizeof(double2));
  if (!base) return;
  if (!copy_register_arrays(c, devicePtrs, base, "cvdvGetFidelity copy")) return;
  std::vector<const double2*> arrs(numReg);
  size_t off = 0;
  for (int r = 0; r < numReg; ++r) {
    arrs[r] = base + off;
    off += (size_t)1 << c->q[r];
  }
  // outer product of all registers but the last (same helper as the initialiser)
  int R = c->numReg, qLast = c->q[R - 1];
  uint64_t nOuter = 1ull << (c->totalQbt - qLast);
  double2* outer = (double2*)arena_alloc(c, nOuter * sizeof(double2));
  if (!outer) return;
  if (!launch_outer(c, arrs.data(), outer)) return;
  double2 ip;
  bool ok = c->precision == kC128
                ? reduce(c, OpSep<double2>{(const double2*)c->state(), outer, arrs[R - 1], qLast}, c->size(), &ip)
                : reduce(c, OpSep<float2>{(const float2*)c->state(), outer, arrs[R - 1], qLast}, c->size(), &ip);
  if (ok) *fidOut = ip.x * ip.x + ip.y * ip.y;
}

double cvdvGetPhotonNumber(CVDVContext* ctx, int regIdx) {
  if (!ctx) return -1.0;
  Context* c = C(ctx);
  if (regIdx < 0 || regIdx >= c->numReg) {
    set_error(c, kErrInvalidArg, "cvdvGetPhotonNumber: invalid register index %d", regIdx);
    return -1.0;
  }
  if (!ready(c, "cvdvGetPhotonNumber")) return -1.0;
  arena_reset(c);
  const int N = 1 << c->q[regIdx];
  // <x^2> and <p^2> are the second moments of the register's marginal in each basis
  double* m = (double*)arena_alloc(c, (2 * (size_t)N + 2) * sizeof(double));
  if (!m || !marginals_axis(c, {regIdx}, {0}, m)) return -1.0;
  // |FtQ2P psi|^2 = |FFT(pre-twiddle * psi)|^2 / N, out of place: a row or column program
  // where the register has one (one pass into the second buffer, which is free
  // between flushes), else the tile passes into a scratch state
  Term tw{};
  tw.kind = kTermFtTw;
  tw.r = regIdx;
  tw.s = -1;
  tw.ctrlBit = -1;
  tw.sign = 1;
  Term sc{};
  sc.kind = kTermScalar;
  sc.ctrlBit = -1;
  sc.g0 = make_double2(1.0 / sqrt((double)N), 0.0);
  const int home = c->cur;
  void* own = c->buf[home];
  bool ok;
  if (row_eligible(c, regIdx) || col_program_ok(c, regIdx)) {
    const std::vector<HostRowOp> ops = {{kRowDiag, 0, {tw, sc}}, {kRowFft, 1, {}}};
    ok = launch_row_program(c, regIdx, ops);
    ok = ok && marginals_axis(c, {regIdx}, {(size_t)N}, m);  // of the buffer it wrote
    c->cur = home;
  } else {
    FactorList pre;
    std::vector<Term> left;
    if (!build_factor_list(c, {tw, sc}, &pre, &left)) return -1.0;
    char* scratch = (char*)big_scratch(c, (size_t)c->size() * c->elemBytes);
    if (!scratch || !launch_fft_into(c, regIdx, 1, pre, scratch, c->other())) return -1.0;
    c->buf[home] = scratch;  // the marginal of the transformed state
    ok = marginals_axis(c, {regIdx}, {(size_t)N}, m);
    c->buf[home] = own;
  }
  if (!ok) return -1.0;
  {
    LaunchScope _ls(ctx, kKReduce);
    k_second_moments<<<2, 256, 0, c->stream>>>(m, N, c->dx[regIdx], m + 2 * (size_t)N);
  }
  double v[2];
  if (!cuda_ok(c, cudaGetLastError(), "photon number launch") ||
      !read_back(c, {{v, 0, 2}}, m + 2 * (size_t)N, 2, "photon number"))
    return -1.0;
  return (v[0] + v[1] - 1.0) / 2.0;
}

void cvdvFidelityStatevectors(CVDVContext* ctx1, CVDVContext* ctx2, double* fidOut) {
  if (fidOut) *fidOut = 0.0;
  if (!ctx1 || !ctx2 || !fidOut) return;
  Context* a = C(ctx1);
  Context* b = C(ctx2);
  if (a->totalQbt != b->totalQbt || a->numReg == 0 || b->numReg == 0) {
    set_error(a, kErrInvalidArg, "cvdvFidelityStatevectors: total qubit count mismatch (%d vs %d)",
              a->totalQbt, b->totalQbt);
    return;
  }
  if (!ready(a, "cvdvFidelityStatevectors") || !ready(b, "cvdvFidelityStatevectors")) return;
  if (a != b && !stream_sync(b, "fidelity sync")) return;
  arena_reset(a);
  double2 ip;
  bool ok;
  uint64_t n = a->size();
  if (a->precision == kC128 && b->precision == kC128)
    ok = reduce(a, OpDot<double2, double2>{(const double2*)a->state(), (const double2*)b->state()}, n, &ip);
  else if (a->precision == kC128)
    ok = reduce(a, OpDot<double2, float2>{(const double2*)a->state(), (const float2*)b->state()}, n, &ip);
  else if (b->precision == kC128)
    ok = reduce(a, OpDot<float2, double2>{(const float2*)a->state(), (const double2*)b->state()}, n, &ip);
  else
    ok = reduce(a, OpDot<float2, float2>{(const float2*)a->state(), (const float2*)b->state()}, n, &ip);
  if (ok) *fidOut = ip.x * ip.x + ip.y * ip.y;
}

int cvdvGetLastError(CVDVContext* ctx, char* msg, int len) {
  if (!ctx) return global_error(msg, len);
  Context* c = C(ctx);
  if (msg && len > 0) {
    strncpy(msg, c->lastMsg.c_str(), (size_t)len - 1);
    msg[len - 1] = 0;
  }
  return c->lastErr;
}

void cvdvClearError(CVDVContext* ctx) {
  if (!ctx) return;
  C(ctx)->lastErr = kOk;
  C(ctx)->lastMsg.clear();
}

}  // extern "C"

// ====================================================================== marginal without allocation
// Some callers cannot let a library call cudaMalloc: an application whose
// device memory is owned by another allocator (a framework's caching pool
// that has reserved the GPU, so a plain cudaMalloc fails although the pool has
// room), a service that sizes its device memory once at start-up and must not
// grow it afterwards, or a loop that cannot afford the device-wide
// synchronisation that cudaMalloc and cudaFree may perform.  For them,
// cvdvMeasureMultipleNoAlloc computes the same joint marginal as
// cvdvMeasureMultiple on a state they own, writes it to an output they own,
// and keeps its per-block partial histograms in the fixed array below.
//
// The array is part of this library's device code: every GPU that loads the
// library holds it (kNoAllocBlocks x kNoAllocMaxBins doubles = 4.625 MiB) until
// the process exits.  Every call shares it and it keeps the last call's
// contents; nothing in it has to start at zero, because each block writes its
// whole histogram row before the final kernel reads it.  Calls whose kernels
// overlap on the GPU (different streams, no ordering between them) race on it.
namespace cvdv {

constexpr int kNoAllocBlocks = 148;
constexpr int kNoAllocMaxBins = 4096;  // 2^12: joint marginals of up to 12 qubits
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) double g_noAllocScratch[kNoAllocBlocks * kNoAllocMaxBins];

static std::mutex g_noAllocMu;
static double* g_noAllocPtr[kNoAllocMaxDevices];  // device address per device, set up on first use

// Device address of the scratch array on the current device.  The array's name
// in host code is only a handle for the runtime; the address the kernels use is
// looked up once per device, with that device current.
static double* no_alloc_scratch(int dev, bool report) {
  std::lock_guard<std::mutex> lk(g_noAllocMu);
  if (!g_noAllocPtr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noAllocScratch);
    if (e != cudaSuccess) {
      cudaGetLastError();
      if (report)
        set_error(nullptr, kErrCuda, "cvdvMeasureMultipleNoAlloc: scratch lookup on device %d: %s", dev,
                  cudaGetErrorString(e));
      return nullptr;
    }
    g_noAllocPtr[dev] = (double*)p;
  }
  return g_noAllocPtr[dev];
}

// Loads, on device dev (current), the part of this library's device code that
// holds the array and the two kernels the entry point launches, and records the
// array's address.  Under CUDA's lazy module loading (the default since 12.2)
// that code is loaded on its first use, which takes device memory (the array and
// the kernels' code); cvdvCreate / cvdvCreateEx call this for their device so a
// process that made a context makes its first cvdvMeasureMultipleNoAlloc call
// without that load.
static std::atomic<bool> g_noAllocLoaded[kNoAllocMaxDevices];

double* no_alloc_prepare(int dev, bool report) {
  if (dev < 0 || dev >= kNoAllocMaxDevices) return nullptr;
  double* p = no_alloc_scratch(dev, report);
  if (!p || g_noAllocLoaded[dev].load()) return p;
  cudaFuncAttributes fa{};
  cudaError_t e = cudaFuncGetAttributes(&fa, k_marg_smem<double2>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_marg_smem<float2>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_marg_final);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (report)
      set_error(nullptr, kErrCuda, "cvdvMeasureMultipleNoAlloc: loading its kernels on device %d: %s", dev,
                cudaGetErrorString(e));
    return nullptr;
  }
  g_noAllocLoaded[dev].store(true);
  return p;
}

static bool device_pointer_on(const void* p, int dev) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == dev;
}

}  // namespace cvdv

extern "C" int cvdvMeasureMultipleNoAlloc(const void* state, int precision, const int* numQubits,
                                          int numReg, const int* regIdxs, int numRegs, double* probsOut,
                                          void* stream) {
  const char* fn = "cvdvMeasureMultipleNoAlloc";
  if (!state || !probsOut || !numQubits || !regIdxs) {
    set_error(nullptr, kErrInvalidArg, "%s: null pointer argument", fn);
    return kErrInvalidArg;
  }
  if (precision != kC128 && precision != kC64) {
    set_error(nullptr, kErrInvalidArg, "%s: precision %d (0 = complex128, 1 = complex64)", fn, precision);
    return kErrInvalidArg;
  }
  if (numReg < 1 || numReg > kMaxRegs) {
    set_error(nullptr, kErrInvalidArg, "%s: numReg %d outside 1..%d", fn, numReg, kMaxRegs);
    return kErrInvalidArg;
  }
  int flw[kMaxRegs];
  int total = 0;
  for (int r = numReg - 1; r >= 0; --r) {
    if (numQubits[r] < 1 || numQubits[r] > kMaxTotalQubits) {
      set_error(nullptr, kErrInvalidArg, "%s: register %d has %d qubits", fn, r, numQubits[r]);
      return kErrInvalidArg;
    }
    flw[r] = total;
    total += numQubits[r];
  }
  if (total > kMaxTotalQubits) {
    set_error(nullptr, kErrInvalidArg, "%s: %d qubits in total exceed %d", fn, total, kMaxTotalQubits);
    return kErrInvalidArg;
  }
  if (numRegs < 1 || numRegs > 16 || numRegs > numReg) {
    set_error(nullptr, kErrInvalidArg, "%s: numRegs %d outside 1..min(16, numReg)", fn, numRegs);
    return kErrInvalidArg;
  }
  MargDesc D{};
  D.nSel = numRegs;
  long long bins = 1;
  for (int s = 0; s < numRegs; ++s) {
    int r = regIdxs[s];
    if (r < 0 || r >= numReg) {
      set_error(nullptr, kErrInvalidArg, "%s: register index %d outside 0..%d", fn, r, numReg - 1);
      return kErrInvalidArg;
    }
    for (int t = 0; t < s; ++t)
      if (regIdxs[t] == r) {
        set_error(nullptr, kErrInvalidArg, "%s: register %d selected twice", fn, r);
        return kErrInvalidArg;
      }
    bins <<= numQubits[r];  // at most 2^12 * 2^34, no overflow
    if (bins > kNoAllocMaxBins) break;
    D.shift[s] = flw[r];
    D.mask[s] = (1 << numQubits[r]) - 1;
    D.stride[s] = bins >> numQubits[r];  // first selected register fastest, as cvdvMeasureMultiple
  }
  if (bins > kNoAllocMaxBins) {
    set_error(nullptr, kErrInvalidArg,
              "%s: the selected registers span more than %d outcomes; this entry point holds at most "
              "%d (12 qubits) -- use cvdvMeasureMultiple for larger marginals",
              fn, kNoAllocMaxBins, kNoAllocMaxBins);
    return kErrInvalidArg;
  }
  D.outSize = bins;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
    cudaGetLastError();
    set_error(nullptr, kErrCuda, "%s: no usable current device", fn);
    return kErrCuda;
  }
  const size_t elem = precision == kC128 ? sizeof(double2) : sizeof(float2);
  if (((uintptr_t)state % elem) || ((uintptr_t)probsOut % sizeof(double)) ||
      !device_pointer_on(state, dev) || !device_pointer_on(probsOut, dev)) {
    set_error(nullptr, kErrInvalidArg,
              "%s: state and probsOut must be aligned device memory of the current device %d", fn, dev);
    return kErrInvalidArg;
  }
  double* scratch = no_alloc_prepare(dev, true);
  if (!scratch) return kErrCuda;
  cudaStream_t s = (cudaStream_t)stream;
  const uint64_t n = 1ull << total;
  uint64_t maxBlocks = (n + 255) / 256;
  int blocks = kNoAllocBlocks < maxBlocks ? kNoAllocBlocks : (int)maxBlocks;
  size_t smem = (size_t)bins * sizeof(double);
  // an error the caller's own earlier CUDA work left pending is theirs: it is
  // neither reported as this call's nor cleared
  const cudaError_t before = cudaPeekAtLastError();
  {
    LaunchScope _ls(nullptr, kKReduce);
    if (precision == kC128)
      k_marg_smem<double2><<<blocks, 256, smem, s>>>((const double2*)state, n, D, scratch);
    else
      k_marg_smem<float2><<<blocks, 256, smem, s>>>((const float2*)state, n, D, scratch);
  }
  {
    LaunchScope _ls(nullptr, kKReduce);
    launch_marg_final(scratch, blocks, bins, probsOut, s);
  }
  e = cudaPeekAtLastError();
  if (e != cudaSuccess && e != before) {
    cudaGetLastError();
    set_error(nullptr, kErrCuda, "%s: launch: %s", fn, cudaGetErrorString(e));
    return kErrCuda;
  }
  return kOk;
}
