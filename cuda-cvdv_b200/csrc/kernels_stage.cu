// Batched independent circuits: one launch per gate stage.
//
// Every instance of the batch has its own layout [1-qubit registers..., mode]
// and gate list; at stage s each instance applies its s-th gate.  The host turns
// those gates into tasks (CvdvBatchTask): a row program -- the mode's transforms,
// parity and diagonal phases, on a group of rows -- or a 2x2 gate on a qubit bit
// over a range of pairs.  The stage's 512-thread CTAs, one per task up to the caller's
// limit, walk its task list; the task decides the code path, so instances with different
// gates and mode sizes share one launch.
//
// Row programs keep each row in registers (8, 16 or 32 amplitudes per thread, the
// task's choice) and use the Stockham stages of the row kernels; diagonal phases are
// running products from a small phase polynomial (phase_run), or evaluated per element
// where it has a cubic term (phase_factor: FP64 argument with exact transform twiddles,
// reduced mod 2 pi, then sin/cos in the state's precision), so nothing has to be
// tabulated per instance.

#include <cmath>
#include <type_traits>

#include "../../include/cvdv.h"
#include "cvdv_internal.cuh"
#include "row_fft.cuh"
#include "turns.cuh"

namespace cvdv {

constexpr int kStageThreads = 512;

// Amplitudes per thread of a row task, 2^LOGE with LOGE = 3, 4 or 5 (radix-8, 16 or
// 32 Stockham stages; 512 2^LOGE / N rows per CTA), chosen per task (the
// autotuner's knob).  A row must fit the 512 threads (N / 2^LOGE <= 512) and the
// CTA's rows the shared memory (complex128: 2^LOGE <= 16).  By default 32 for complex64
// rows of 2^13 and 2^14 points, else 16, and less for stages that do not fill the chip
// (adaptive_loge in batch.py, with the times).
template <typename C> constexpr int stage_max_log() { return sizeof(C) == sizeof(float2) ? 14 : 13; }
template <typename C> constexpr int stage_max_loge() { return sizeof(C) == sizeof(float2) ? 5 : 4; }
template <typename C, int LOGN, int LOGE>
constexpr bool stage_shape_ok() {
  return LOGE >= 3 && LOGE <= stage_max_loge<C>() && LOGN >= LOGE && (LOGN - LOGE) <= 9;
}

// shared memory of the largest row group (512 threads x E amplitudes, padded) + twiddles;
// the radix-8 shape's rows (512 x 8 amplitudes, padded by 1/8) are smaller
template <typename C>
constexpr size_t stage_smem() {
  constexpr int L = stage_max_log<C>();
  constexpr int E = 1 << stage_max_loge<C>();
  return (size_t)(kStageThreads * E + kStageThreads * E / 16) * sizeof(C) + (64 + (1 << (L - 6))) * sizeof(double2);
}

// after it, each warp's constants of a quadratic phase (phase_run): E for each of its rows
constexpr int kStageQuads = 128;
constexpr size_t stage_quad_bytes() { return (size_t)(kStageThreads / 32) * kStageQuads * sizeof(double2); }

template <typename C> struct StageReal;
template <> struct StageReal<double2> { using t = double; };
template <> struct StageReal<float2> { using t = float; };

template <typename C>
__device__ __forceinline__ C phase_factor(const CvdvBatchPhase& P, int j, int N, double zs) {
  // exact multiple of theta_j = pi (N-1)(2j-N+1) / (2N): integer argument mod 4N
  const int M4 = 4 * N;
  int m = (int)(((long long)(N - 1) * (2 * j - N + 1)) % M4);
  m = (int)(((long long)m * P.tw) % M4);
  if (m < 0) m += M4;
  const double dx = sqrt(2.0 * M_PI / (double)N);
  const double x = ((double)j - 0.5 * (double)(N - 1)) * dx;
  double ph = M_PI * (double)m / (double)(2 * N) + P.g0 + zs * P.h0 +
              x * ((P.a1 + zs * P.b1) + x * ((P.a2 + zs * P.b2) + x * P.a3));
  ph -= 2.0 * M_PI * rint(ph * (0.5 / M_PI));
  using R = typename StageReal<C>::t;
  R s, c;
  if constexpr (sizeof(R) == sizeof(float)) {
    __sincosf((float)ph, &s, &c);  // |ph| <= pi after the FP64 reduction
  } else {
    sincos(ph, &s, &c);
  }
  const R sc = (R)P.scale;
  return mk(sc * c, sc * s);
}

// A phase without a cubic term on the points t + k TPR of a row.  With u = 2 j - N + 1 and
// dx^2 = 2 pi / N its turns are a quadratic in the integer u,
//   tw (N-1) u / (4N) + (g0 + z h0) / 2pi + (a1 + z b1) dx u / 4pi + (a2 + z b2) u^2 / (4N),
// so a thread needs its value at its first point and its step (a sincospi each), a
// running product, and the E constants exp(2 pi i q (2 TPR)^2 k^2) of the quadratic
// part, which the row's lanes in the warp evaluate one each into `kq`.  Evaluating the
// polynomial per point took about 25 FP64 operations, the conversions of its integers
// and a fast sine and cosine each, about as long as the transforms between the phases;
// this takes 8, and is exact to FP64 where the fast intrinsic was to 4e-7.
// 96 circuits of 50 gates: 3.42 -> 3.30 ms, error 9.3e-6 -> 4.1e-6.  In complex128 the
// products keep their low words (turns.cuh) and a run of 16 starts anew at the eighth point: a
// displacement on 2^11 points is off by 0.9e-15 (3.0e-15 with the phases evaluated per point).
template <typename C, int LOGN, int LOGE>
__device__ __forceinline__ void phase_run(C (&v)[1 << LOGE], const CvdvBatchPhase& P, int t, double zs, double2* kq) {
  constexpr int E = 1 << LOGE, N = 1 << LOGN, TPR = N >> LOGE, LANES = TPR < 32 ? TPR : 32;
  constexpr double inv4N = 1.0 / (4.0 * N);
  const int u0 = 2 * t - N + 1;
  constexpr LinTurns L = lin_turns(LOGN);
  constexpr double perTurn = 0.5 / M_PI, perTurnLo = -9.839338337591243e-18;  // 1 / (2 pi) in two words
  const TurnRate lin = turn_rate(P.a1 + zs * P.b1, L.hi, L.lo), q = {(P.a2 + zs * P.b2) * inv4N, 0.0};
  // tw (N-1) u / (4N) turns, in -1/2 .. 1/2
  const int w = (P.tw * (N - 1)) & (4 * N - 1);
  auto twiddle = [&](int u) {
    return (double)(((int)((long long)w * u + 2 * N) & (4 * N - 1)) - 2 * N) * inv4N;
  };
  // (a run of 8 repeats a sum's rounding too seldom to pay for the second word: small batches)
  constexpr bool C128 = sizeof(C) == sizeof(double2);
  using Turns = std::conditional_t<C128 && E >= 16, Turns2, Turns1<C128>>;
  Turns p0(twiddle(u0)), p1(twiddle(2 * TPR));
  p0.add(lin, (double)u0);
  p1.add(lin, 2.0 * TPR);
  p0.add(turn_rate(P.g0 + zs * P.h0, perTurn, perTurnLo), 1.0);
  const bool quad = P.a2 != 0.0 || P.b2 != 0.0;  // the same for every row of the task
  if (quad) {
    p0.add(q, (double)u0 * (double)u0);
    p1.add(q, 4.0 * TPR * (double)u0);
    __syncwarp();  // the last run's constants are read
    const int lane = t & (LANES - 1);
#pragma unroll
    for (int k = lane; k < E; k += LANES) {
      Turns pk;
      pk.add(q, 4.0 * TPR * TPR * (double)(k * k));
      kq[k] = pk.root();
    }
    __syncwarp();
  }
  double2 f = p0.root();
  f.x *= P.scale;
  f.y *= P.scale;
  const double2 st = p1.root();
  // in complex128 from the eighth point's factor anew: a step's rounding is repeated
  // 7 + 1 times at most instead of 15
  constexpr bool ANCHOR = E >= 16 && C128;
  double2 eighth = f;
  if constexpr (ANCHOR) eighth = dmul(f, p1.times(8.0).root());
#pragma unroll
  for (int k = 0; k < E; ++k) {
    v[k] = cmul(v[k], fromd<C>(quad ? dmul(f, kq[k]) : f));
    f = ANCHOR && k == 7 ? eighth : dmul(f, st);
  }
}

template <typename C, int LOGN, int LOGE>
__device__ __forceinline__ void stage_row_task(C* __restrict__ st, const CvdvBatchTask& T,
                                               const CvdvBatchProgram& Pg, unsigned char* smraw) {
  constexpr int E = 1 << LOGE, N = 1 << LOGN, TPR = N >> LOGE, R = kStageThreads / TPR;
  // the Stockham exchanges pad a row once per radix: every 8 points for radix-8
  // stages (LOGE 3), every 16 or 32 otherwise
  constexpr int RS = N + (N >> (LOGE == 3 ? 3 : 4));
  C* sm = reinterpret_cast<C*>(smraw);
  double2* lo = reinterpret_cast<double2*>(sm + (size_t)RS * R);
  double2* hi = lo + 64;
  const int tid = threadIdx.x, row = tid / TPR, t = tid % TPR;
  const bool valid = row < T.count;  // rows past the task's count only take part in the syncs
  const uint64_t rowIdx = (uint64_t)T.first + (valid ? row : 0);
  C* src = st + T.stateOffset + (rowIdx << LOGN);
  C* smrow = sm + row * RS;
  // the quadratic constants: E for each row's lanes of a warp
  double2* kqs = reinterpret_cast<double2*>(smraw + stage_smem<C>());
  double2* kq = kqs + (tid >> 5) * kStageQuads + (TPR < 32 ? ((tid & 31) / TPR) * E : 0);
  static_assert(TPR >= 32 || (32 / TPR) * E <= kStageQuads, "constants per warp");
  for (int i = tid; i < 64 + (N >> 6); i += kStageThreads) {
    const int e = i < 64 ? i : (i - 64) << 6;
    double s, c;
    sincospi(-2.0 * (double)e / (double)N, &s, &c);
    lo[i] = make_double2(c, s);
  }
  C v[E];
#pragma unroll
  for (int k = 0; k < E; ++k) v[k] = src[t + k * TPR];
  __syncthreads();
  int d = 0;
  for (int o = 0; o < Pg.nOps; ++o) {
    const int op = Pg.op[o];
    if (op == 0) {
      const CvdvBatchPhase P = Pg.phase[d++];
      const double zs = (P.ctrlBit >= 0 && (((rowIdx << LOGN) >> P.ctrlBit) & 1ull)) ? -1.0 : 1.0;
      if (P.a3 == 0.0) {
        phase_run<C, LOGN, LOGE>(v, P, t, zs, kq);
      } else {
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] = cmul(v[k], phase_factor<C>(P, t + k * TPR, N, zs));
      }
    } else if (op == 1 || op == 2) {
      // one transform body for both directions (keeps the kernel's code small):
      // the unnormalised inverse DFT is conj(DFT(conj(x)))
      if (op == 2) {
#pragma unroll
        for (int k = 0; k < E; ++k) v[k].y = -v[k].y;
      }
      rr_stages<C, 1, LOGN, 0, LOGE>(v, smrow, t, lo, hi);
      if (op == 2) {
#pragma unroll
        for (int k = 0; k < E; ++k) v[k].y = -v[k].y;
      }
    } else {  // parity: element j <- element N-1-j of the same row
#pragma unroll
      for (int k = 0; k < E; ++k) smrow[rpad<C>(N - 1 - (t + k * TPR))] = v[k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < E; ++k) v[k] = smrow[rpad<C>(t + k * TPR)];
      __syncthreads();
    }
  }
  if (valid) {
#pragma unroll
    for (int k = 0; k < E; ++k) src[t + k * TPR] = v[k];
  }
  __syncthreads();  // shared memory is reused by the CTA's next task
}

template <typename C, int LOGN>
__device__ __forceinline__ void stage_row_dispatch(C* __restrict__ st, const CvdvBatchTask& T,
                                                   const CvdvBatchProgram& Pg, unsigned char* smraw, int le) {
  // (the host checks every task's shape against stage_shape_ok before launching)
  if (le == 3) {
    if constexpr (stage_shape_ok<C, LOGN, 3>()) stage_row_task<C, LOGN, 3>(st, T, Pg, smraw);
  } else if (le == 4) {
    if constexpr (stage_shape_ok<C, LOGN, 4>()) stage_row_task<C, LOGN, 4>(st, T, Pg, smraw);
  } else {
    if constexpr (stage_shape_ok<C, LOGN, 5>()) stage_row_task<C, LOGN, 5>(st, T, Pg, smraw);
  }
}

template <typename C>
__device__ __forceinline__ void stage_pair_task(C* __restrict__ st, const CvdvBatchTask& T) {
  const C a00 = fromd<C>(make_double2(T.m[0], T.m[1])), a01 = fromd<C>(make_double2(T.m[2], T.m[3]));
  const C a10 = fromd<C>(make_double2(T.m[4], T.m[5])), a11 = fromd<C>(make_double2(T.m[6], T.m[7]));
  C* base = st + T.stateOffset;
  const uint64_t low = (1ull << T.bit) - 1;
  for (int p = threadIdx.x; p < T.count; p += kStageThreads) {
    const uint64_t lp = (uint64_t)T.first + p;
    const uint64_t i0 = ((lp & ~low) << 1) | (lp & low);
    const uint64_t i1 = i0 | (1ull << T.bit);
    const C x = base[i0], y = base[i1];
    base[i0] = cadd(cmul(a00, x), cmul(a01, y));
    base[i1] = cadd(cmul(a10, x), cmul(a11, y));
  }
}

template <typename C>
__global__ void __launch_bounds__(kStageThreads, 1)
    k_batch_stage(C* __restrict__ st, const CvdvBatchTask* __restrict__ tasks, int nTasks,
                  const CvdvBatchProgram* __restrict__ progs) {
  extern __shared__ __align__(16) unsigned char smraw[];
  for (int ti = blockIdx.x; ti < nTasks; ti += gridDim.x) {
    const CvdvBatchTask T = tasks[ti];
    if (T.kind == 1) {
      stage_pair_task<C>(st, T);
      continue;
    }
    const CvdvBatchProgram& Pg = progs[T.program];
    const int le = T.logE ? T.logE : ((sizeof(C) == sizeof(float2) && T.logRow >= 13) ? 5 : 4);
    switch (T.logRow) {
      case 8: stage_row_dispatch<C, 8>(st, T, Pg, smraw, le); break;
      case 9: stage_row_dispatch<C, 9>(st, T, Pg, smraw, le); break;
      case 10: stage_row_dispatch<C, 10>(st, T, Pg, smraw, le); break;
      case 11: stage_row_dispatch<C, 11>(st, T, Pg, smraw, le); break;
      case 12: stage_row_dispatch<C, 12>(st, T, Pg, smraw, le); break;
      case 13: stage_row_dispatch<C, 13>(st, T, Pg, smraw, le); break;
      default:
        if constexpr (stage_max_log<C>() >= 14) stage_row_dispatch<C, 14>(st, T, Pg, smraw, le);
        break;
    }
  }
}

}  // namespace cvdv

using namespace cvdv;

template <typename C>
static cudaError_t launch_stage(void* states, const CvdvBatchTask* tasks, int nTasks, const CvdvBatchProgram* programs,
                                int gridCtas, cudaStream_t s) {
  const size_t smem = stage_smem<C>() + stage_quad_bytes();
  // the shared-memory opt-in is set once per device (so later calls can be captured)
  static std::atomic<bool> optedIn[kMaxDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool known = dev >= 0 && dev < kMaxDevices;
  if (!known || !optedIn[dev].load()) {
    e = cudaFuncSetAttribute(k_batch_stage<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (known) optedIn[dev].store(true);
  }
  k_batch_stage<C><<<gridCtas, kStageThreads, smem, s>>>((C*)states, tasks, nTasks, programs);
  return cudaGetLastError();
}

extern "C" {

void cvdvBatchStructSizes(int* sizes) {
  if (!sizes) return;
  sizes[0] = (int)sizeof(CvdvBatchPhase);
  sizes[1] = (int)sizeof(CvdvBatchProgram);
  sizes[2] = (int)sizeof(CvdvBatchTask);
}

int cvdvBatchRunStage(void* states, int precision, const CvdvBatchTask* tasks, int nTasks,
                      const CvdvBatchProgram* programs, int gridCtas, void* stream) {
  const char* fn = "cvdvBatchRunStage";
  if (!states || !tasks || nTasks < 0 || gridCtas < 1 || (precision != kC128 && precision != kC64)) {
    set_error(nullptr, kErrInvalidArg, "%s: invalid arguments", fn);
    return kErrInvalidArg;
  }
  if (nTasks == 0) return kOk;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaSuccess;
  {
    LaunchScope _ls(nullptr, kKFft);
    e = precision == kC128 ? launch_stage<double2>(states, tasks, nTasks, programs, gridCtas, s)
                           : launch_stage<float2>(states, tasks, nTasks, programs, gridCtas, s);
  }
  if (e != cudaSuccess) {
    set_error(nullptr, kErrCuda, "%s: %s", fn, cudaGetErrorString(e));
    return kErrCuda;
  }
  return kOk;
}

}  // extern "C"
