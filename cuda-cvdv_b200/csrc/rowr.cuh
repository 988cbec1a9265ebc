// A row program as the kernels take it, and the register-resident row kernel k_rowr
// with its launcher, instantiated per precision and form in kernels_rowr_*.cu.
#pragma once

#include <cmath>
#include <type_traits>

#include "cvdv_internal.cuh"
#include "row_fft.cuh"
#include "turns.cuh"

namespace cvdv {

constexpr int kMaxRowE = 32;  // amplitudes a k_rowr thread holds, at most

struct RowOp {
  int kind;
  int dir;   // fft: +1 forward, -1 inverse
  int diag;  // diag: index into RowProgram::diag
};

struct RowDiag {
  const double2* tab;  // [2^nCtrl][N] combined factor of the row register, or null
  int permuted;        // tab stored as [seg][rank][m] for k = rank + C m (transposed layout)
  int nCtrl;
  int ctrlShift[2];    // flat-index bits selecting the table segment (row bits)
  int hasRowF, hasElemF;
  FactorList rowF;     // factors constant along a row
  FactorList elemF;    // per-element factors (bilinear terms with the row register)
  // Bilinear terms c x_row x_other (other register and control bit off the row)
  // taken out of elemF for k_rowr and k_rowq: along one row they are the linear phase
  // a (m - regC) regDx with a = sum c x_other (+-1 by the control bit).  The other
  // register is side 1 of each XXFactor.
  int nLin;
  double regC, regDx;
  XXFactor lin[kMaxXX];
  // A run whose register terms are linear phases (no table; k_rowq, and k_rowr outside
  // the shapes that keep tables): transform twiddles, the sum of their signs s giving
  // exp(i pi s (N-1)(2n-N+1)/(2N)) at point n, and terms c x_n (x_n = (n - regC) regDx),
  // each negated when its control bit (a row bit, or none: -1) is set
  int ftSign;
  int hasQuad;  // k_rowr, 32 amplitudes a thread: the run also has c2 x^2 (uncontrolled terms' sum)
  double c2;
  double2 quad[kMaxRowE];  // exp(2 pi i c2 TPR^2 k^2 / N) for the kernel's E amplitudes a thread
  int nPl;
  double plC[2];
  int plCtrl[2];
};

struct RowProgram {
  int logN;     // register length
  int logM;     // row elements held by one CTA
  int logRows;  // rows per CTA (cluster size 1 only)
  int nOps;
  int nDiag;
  int logTwN;
  int loadT;    // cluster rows: start transposed (1: from the natural layout, 2: from the blocked one)
  int storeBlocked;  // cluster rows ending transposed: write the blocked layout
  int rowMask;       // k_rowr: rows (columns) of the state less one, at most those of a CTA less one
  int logS;          // k_rowr on a strided register: log2 of the amplitudes below it (0: rows)
  const double2* tw;
  double* rowSums;        // non-null: per-warp partial sums of |psi|^2 of every row's result
  unsigned int* waitErr;  // set when a bounded wait on the cluster peers gives up
  RowOp ops[kMaxRowOps];
  RowDiag diag[kMaxRowDiags];
};

// ---------------------------------------------------------------- register-resident rows
// Rows that fit one CTA (up to 2^13 complex128 / 2^14 complex64 points) run in
// k_rowr: each thread keeps E = 16 (or 32) amplitudes of one row in registers
// for the whole program -- elements t + TPR v (v < E) of its row, TPR = M / E
// threads per row.  A Stockham stage of radix R gives thread t the butterflies
// j = t + b TPR (b < E/R); their inputs j + u M/R are exactly the thread's E
// elements (register b + (E/R) u), and the last stage's outputs land on the same
// positions.  So the global load, the store and every diagonal run between
// transforms work on registers in place; only the stages inside a transform
// exchange data, through one padded shared-memory row.  Row length, radices and
// strides are template constants, so every shared-memory address is a
// per-thread base plus an immediate offset.

// exp(i pi s (N-1)(2n-N+1)/(2N)) with the angle reduced exactly in integers, and
// its ratio between n + d and n, exp(i pi s (N-1) d / N)
__device__ __forceinline__ double2 ft_tw_at(long long n, long long N, int s) {
  long long m = ((N - 1) * (2 * n - N + 1) * s) % (4 * N);
  if (m < 0) m += 4 * N;
  double sn, c;
  sincospi((double)m / (double)(2 * N), &sn, &c);
  return make_double2(c, sn);
}
__device__ __forceinline__ double2 ft_tw_ratio(long long d, long long N, int s) {
  long long m = ((N - 1) * d * s) % (2 * N);
  if (m < 0) m += 2 * N;
  double sn, c;
  sincospi((double)m / (double)N, &sn, &c);
  return make_double2(c, sn);
}

// A diagonal run on the amplitudes t + k TPR (k < E) of a row.  Register terms of
// degree up to two, transform twiddles and bilinear terms need no table (the shapes that
// keep one all the same: launch_row_program): with
// u = 2 n - N + 1 and x_n = dx u / 2, dx^2 = 2 pi / N, they are
//   c2 x^2 = c2 u^2 / (4 N),  a x = a dx u / (4 pi),  twiddle = s (N-1) u / (4 N)
// turns.  From u0 = 2 t - N + 1 a thread's points are u0 + 2 TPR k, so the factor is
//   [value at u0] [step]^k [exp(2 pi i (4 c2 / 4 N) TPR^2 k^2)]:
// two sincospi on turns reduced mod 1 (three in complex128), a running product, and
// (c2 != 0) E constants in the kernel's parameters.  Runs with a controlled c x^2, a cubic or a
// qubit term keep a table, and so do quadratic runs on shapes other than rr_quads:
// the sincospi cost more than the loads with 8 or 16 amplitudes a thread (a 2^8-point
// register's rotation, displacement and squeeze on a 2^26 complex128 state: 2.38 ms
// against 1.54 with tables).
template <typename C, int LOGM, int LOGE, bool QUAD>
__device__ __forceinline__ void rr_diag(C (&v)[1 << LOGE], const RowDiag& D, uint64_t rowBase, int t) {
  constexpr int E = 1 << LOGE, N = 1 << LOGM, TPR = 1 << (LOGM - LOGE);
  const double2 rs = D.hasRowF ? eval_factor(D.rowF, rowBase) : make_double2(1.0, 0.0);
  // running factor of element t + k TPR: rs times the linear phase, advanced by st per k
  double2 f = rs, st = make_double2(1.0, 0.0);
  // In complex128 the product starts anew from every eighth element's, so a step's rounding
  // is repeated 7 + 3 times at most instead of 31 (32 amplitudes a thread): a transform of
  // random amplitudes on 2^13 points 1.6e-15 -> 0.7e-15, for a third sine and cosine a run
  // (rotation, displacement and squeeze on the columns of a 2^24 state 0.85 -> 0.88 ms).
  constexpr bool ANCHORS = E >= 16 && sizeof(C) == sizeof(double2);
  constexpr int kAnchor = 8;
  double2 anchor = rs, stA = make_double2(1.0, 0.0);
  const bool lin = D.nLin || D.nPl || D.ftSign || (QUAD && D.hasQuad);
  if (lin) {
    double a = 0.0;
    for (int l = 0; l < D.nLin; ++l) {
      const XXFactor& X = D.lin[l];
      const int j = (int)((rowBase >> X.shift1) & (uint64_t)X.mask1);
      double c = X.coeff * (((double)j - X.c1) * X.dx1);
      if (X.ctrlShift >= 0 && ((rowBase >> X.ctrlShift) & 1ull)) c = -c;
      a += c;
    }
    for (int k = 0; k < D.nPl; ++k)
      a += (D.plCtrl[k] >= 0 && ((rowBase >> D.plCtrl[k]) & 1ull)) ? -D.plC[k] : D.plC[k];
    constexpr LinTurns L = lin_turns(LOGM);
    const TurnRate lr = turn_rate(a, L.hi, L.lo);
    const int u0 = 2 * t - N + 1;
    // s (N-1) u mod 4N in integers: at most 3 2^28 for the runs of a program
    constexpr double inv4N = 1.0 / (4.0 * N);
    const int w = (D.ftSign * (N - 1)) & (4 * N - 1);
    auto twiddle = [&](int u) {  // s (N-1) u / (4N) turns, in -1/2 .. 1/2
      return (double)(((int)((long long)w * u + 2 * N) & (4 * N - 1)) - 2 * N) * inv4N;
    };
    using Turns = std::conditional_t<sizeof(C) == sizeof(double2), Turns2, Turns1<false>>;
    Turns p0(twiddle(u0)), p1(twiddle(2 * TPR));
    p0.add(lr, (double)u0);
    p1.add(lr, 2.0 * TPR);
    if (QUAD && D.hasQuad) {
      const TurnRate q = {D.c2 * inv4N, 0.0};
      p0.add(q, (double)u0 * (double)u0);
      p1.add(q, 4.0 * TPR * (double)u0);
    }
    f = dmul(rs, p0.root());
    st = p1.root();
    if constexpr (ANCHORS) {
      anchor = f;
      stA = p1.times(kAnchor).root();
    }
  }
  // on to the next element's factor, from the last anchor's every kAnchor elements
  auto next = [&](int k) {
    if (ANCHORS && (k + 1) % kAnchor == 0) f = anchor = dmul(anchor, stA);
    else f = dmul(f, st);
  };
  if (D.tab) {
    int seg = 0;
    for (int c = 0; c < D.nCtrl; ++c) seg |= (int)((rowBase >> D.ctrlShift[c]) & 1ull) << c;
    const double2* tp = D.tab + ((size_t)seg << LOGM) + t;
#pragma unroll
    for (int k0 = 0; k0 < E; k0 += 8) {
      double2 w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) w[k] = __ldg(tp + (k0 + k) * TPR);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (D.hasRowF || lin) w[k] = dmul(w[k], f);
        if (lin) next(k0 + k);
        v[k0 + k] = cmul(v[k0 + k], fromd<C>(w[k]));
      }
    }
  } else if (QUAD && D.hasQuad) {
#pragma unroll
    for (int k = 0; k < E; ++k) {
      v[k] = cmul(v[k], fromd<C>(dmul(f, D.quad[k])));
      next(k);
    }
  } else if (lin) {
#pragma unroll
    for (int k = 0; k < E; ++k) {
      v[k] = cmul(v[k], fromd<C>(f));
      next(k);
    }
  } else if (D.hasRowF) {
    const C c = fromd<C>(rs);
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = cmul(v[k], c);
  }
}

// ---- asynchronous copies
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// 16- or 8-byte asynchronous copy from global to shared memory
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Runs `f` where its `on` is set: the last transform of a program's tile.
template <typename F>
struct HookIf {
  bool on;
  F f;
  __device__ __forceinline__ void operator()() const {
    if (on) f();
  }
};

// 256-thread CTAs run two per SM; 512- and 1024-thread CTAs one
// Ask L2 to fetch [p, p + bytes) ahead of use: bulk prefetches of 16 KB, one per
// lane of the first warp (bytes a multiple of 16 KB, at most 32 x 16 KB).
__device__ __forceinline__ void l2_prefetch_tile(const void* p, uint32_t bytes) {
  const uint32_t chunk = 16384;
  const uint32_t i = threadIdx.x;
  if (i < bytes / chunk) {
    const char* a = static_cast<const char*>(p) + (size_t)i * chunk;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(chunk) : "memory");
  }
}

// Whether the shape's transforms run with one CTA exchange (rr_two).  Its results sit
// in runs of 32 / G points per warp: rows take it where such a run fills a sector
// (complex64 2^14-point rows store 16-byte pieces with it: 2.33 against 1.63 ms per
// 2^28 state), and shapes of 8 or 16 amplitudes a thread, which keep tables, read them
// in short pieces (2^8-point columns 2.23 against 1.54 ms, 2^12-point 3.11 against
// 2.76; only the 2^7-point shape gains, 1.84 against 2.41; in complex64 its second tree
// of twiddle powers would cost half as much error again, so it keeps the stages there).
template <typename C, int LOGM, int LOGE, int LOGR, bool COL>
constexpr bool rr_use_two() {
  using T = RrTwo<C, LOGM, LOGE, COL ? LOGR : 0>;
  return T::ok && ((LOGE == 5 && (COL || 32 / T::G * sizeof(C) >= 32)) || (LOGM == 7 && sizeof(C) == 16));
}
// Whether the shape's quadratic runs go without a table: with 32 amplitudes a thread
// the two sincospi of a run are worth the loads they save, above all after rr_two, whose
// thread numbering reads a table in short pieces ([13, 13] network, rows / columns:
// complex128 7.95 / 11.9 ms against 9.1 / 13.2 with tables, complex64 4.4 / 6.5 against
// 5.6 / 7.1).
template <typename C, int LOGM, int LOGE, int LOGR, bool COL>
constexpr bool rr_quads() {
  return LOGE == 5 && rr_use_two<C, LOGM, LOGE, LOGR, COL>();
}

template <typename C, int LOGM, int LOGE, int LOGR, bool COL>
constexpr int rr_line_slots() {
  using T = RrTwo<C, LOGM, LOGE, COL ? LOGR : 0>;
  if (rr_use_two<C, LOGM, LOGE, LOGR, COL>()) return T::LINE;
  return COL ? rr_col_slots(LOGM, LOGE, LOGR, (int)sizeof(C)) : rr_row_slots(LOGM, LOGE);
}
// whether a CTA has an SM to itself (persistent over its tiles)
template <typename C, int LOGM, int LOGR, int LOGE>
constexpr bool rr_one() {
  return LOGM - LOGE + LOGR > 8 || (sizeof(C) << (LOGM + LOGR)) >= (128u << 10);
}

// The sum of |psi|^2 (FP64) over the E amplitudes of each of a group of W lanes
// (W = 32, or the lanes of one row when a warp holds several), written by the
// group's first lane.
template <typename C, int E, int W>
__device__ __forceinline__ void row_sum_part(const C (&v)[E], double* out) {
  double a = 0.0;
#pragma unroll
  for (int k = 0; k < E; ++k) a += (double)v[k].x * (double)v[k].x + (double)v[k].y * (double)v[k].y;
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & (W - 1)) == 0) *out = a;
}

// Tiles of one CTA per SM (rr_one) run persistent: each CTA walks tiles blockIdx.x,
// + gridDim.x, ...  A row's next tile is asked into L2 before the current one is
// worked on, so its load finds the data on chip.  A strided tile's loads are 16- or
// 32-byte pieces that keep the load queue busy: once the current tile's last exchange
// is read, the line buffer is free and the next tile is copied into it asynchronously
// while the last runs and the stores go on.  Column programs of the complex128
// [13, 13] network: 13.5 against 14.8 ms without the copy; copying half of the tile
// earlier, into a buffer of its own, took 15.1 (the L1 cache it costs holds the
// tables), and the same copy for rows gained nothing (9.2 against 9.3 ms, complex64
// 2^14-point rows 1.71 against 1.67).  Smaller tiles run two CTAs per SM, which already
// overlap one CTA's loads with the other's work; they get one tile per CTA.
//
// With COL the "rows" are the columns of a strided register (P.logS amplitudes
// below it): column c is inner index c mod S and outer index c / S, and element m
// sits m S amplitudes after its first.  The CTA's 2^LOGR columns (at least two
// within 512 threads) are adjacent inner indices interleaved lane by lane, so a
// warp's load covers runs of 2^LOGR amplitudes; the rest of each sector is read
// from L2 by the CTAs of the neighbouring columns.
//
// A state of fewer rows than a CTA holds (nRows < 2^LOGR, both powers of two) runs
// as one tile whose surplus thread groups repeat its rows: they read the same
// input and write the same values.
template <typename C, int LOGM, int LOGR, int LOGE, bool COL, bool FULL>
__global__ void __launch_bounds__(1 << (LOGM - LOGE + LOGR), rr_one<C, LOGM, LOGR, LOGE>() ? 1 : 2)
    k_rowr(const C* __restrict__ in, C* __restrict__ out, uint64_t nTiles, const __grid_constant__ RowProgram P) {
  constexpr int E = 1 << LOGE, M = 1 << LOGM, TPR = M >> LOGE, NT = TPR << LOGR;
  constexpr int RS = rr_line_slots<C, LOGM, LOGE, LOGR, COL>();
  constexpr uint32_t TILE_BYTES = (uint32_t)sizeof(C) << (LOGM + LOGR);
  constexpr bool ONE = rr_one<C, LOGM, LOGR, LOGE>();
  constexpr int LOGI = COL ? LOGR : 0;
  constexpr bool TWO = rr_use_two<C, LOGM, LOGE, LOGR, COL>();
  constexpr bool PF = COL && ONE && TWO;  // the next tile is copied ahead
  // The first tile is loaded while the twiddles are fetched: in complex128, where it makes up
  // for the two-word phases (rotation, displacement and squeeze of 2^10-point columns of a 2^22
  // state 160 -> 152 us, of 2^13-point rows of a 2^24 state 723 -> 711); complex64 is slower
  // with it (2^10-point columns 116 -> 118).
  constexpr bool AHEAD = !PF && sizeof(C) == sizeof(double2);
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  C* tws = sm + (RS << LOGR);  // the twiddles
  const int tid = threadIdx.x;
  // column form: the CTA's 2^LOGR adjacent columns interleave lane by lane, so a
  // warp's load covers 32 / 2^LOGR points of every column in runs of 2^LOGR
  int row = COL ? (tid & ((1 << LOGR) - 1)) : tid >> (LOGM - LOGE);
  const int t = COL ? (tid >> LOGR) : tid & (TPR - 1);
  C* smrow = sm + row * RS;
  const int logS = COL ? P.logS : 0;
  if constexpr (LOGM <= 8) row &= P.rowMask;  // (longer rows: LOGR = 0 where rows are few)

  C v[E];
  if constexpr (AHEAD) {
    uint64_t base;
    if constexpr (COL) {
      const uint64_t c = ((uint64_t)blockIdx.x << LOGR) + (uint64_t)row;
      base = (c & ((1ull << logS) - 1)) + ((c >> logS) << (LOGM + logS));
    } else {
      base = ((uint64_t)blockIdx.x << (LOGM + LOGR)) + ((uint64_t)row << LOGM);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = in[base + ((uint64_t)(t + k * TPR) << logS)];
  }

  const int scM = P.logTwN - LOGM;
  const auto tw = [&] {
    if constexpr (FULL && TWO) {
      for (int e = tid; e < M; e += NT) tws[e] = fromd<C>(__ldg(P.tw + ((size_t)e << scM)));
      return FullTw<C>{tws};
    } else if constexpr (FULL) {
#pragma unroll 8
      for (int y = tid; y < M; y += NT)
        tws[y] = fromd<C>(__ldg(P.tw + ((size_t)stage_tw_exponent<LOGM, LOGE>(y) << scM)));
      return StageTw<C>{tws};
    } else {
      double2* lo = reinterpret_cast<double2*>(tws);  // w_M^e, e < 64, then w_M^(64 h), h < M / 64
      for (int i = tid; i < rr_tw_slots(LOGM); i += NT) {
        const int e = i < 64 ? i : (i - 64) << 6;
        if (e < M) lo[i] = __ldg(P.tw + ((size_t)e << scM));
      }
      return SplitTw{lo, lo + 64};
    }
  }();
  __syncthreads();
  // copies a tile's amplitudes into sm in thread order (sm[tid + k NT] becomes v[k])
  auto fetch = [&](uint64_t tile) {
    // a point's 2^LOGR adjacent columns are one run of up to 16 bytes, or several
    constexpr int RUN = (int)sizeof(C) << LOGR, CH = RUN < 16 ? RUN : 16, PER = RUN / CH;
    const uint64_t c = tile << LOGR;
    const char* src = reinterpret_cast<const char*>(in + (c & ((1ull << logS) - 1)) + ((c >> logS) << (LOGM + logS)));
    const uint32_t dst = smem_addr(sm);
    const int logStep = logS + (sizeof(C) == 16 ? 4 : 3);  // bytes between points, log2
#pragma unroll
    for (int i = 0; i < (int)(TILE_BYTES / CH / NT); ++i) {
      const int q = tid + i * NT;
      cp_async<CH>(dst + q * CH, src + ((uint64_t)(q / PER) << logStep) + (q % PER) * CH);
    }
    cp_async_commit();
  };
  int lastFft = -1;
  if constexpr (PF) {
    for (int o = 0; o < P.nOps; ++o)
      if (P.ops[o].kind != kRowDiag) lastFft = o;
    fetch(blockIdx.x);
  }
  // Without PF there is no barrier between tiles: after a transform's last exchange
  // (which ends in a barrier) a thread touches shared memory again only in the next
  // tile's first exchange, and every thread has left the old tile's exchanges by then.
  for (uint64_t tile = blockIdx.x; tile < nTiles; tile += gridDim.x) {
    const bool more = tile + gridDim.x < nTiles;
    uint64_t rowBase;
    if constexpr (COL) {
      const uint64_t c = (tile << LOGR) + (uint64_t)row;
      rowBase = (c & ((1ull << logS) - 1)) + ((c >> logS) << (LOGM + logS));
    } else {
      if (ONE && more) l2_prefetch_tile(in + ((tile + gridDim.x) << (LOGM + LOGR)), TILE_BYTES);
      rowBase = (tile << (LOGM + LOGR)) + ((uint64_t)row << LOGM);
    }
    int tau = t;  // v[k] is point tau + k TPR of the row
    if constexpr (PF) {
      cp_async_wait_all();
      __syncthreads();
#pragma unroll
      for (int k = 0; k < E; ++k) v[k] = sm[tid + k * NT];  // (the exchanges wait for all to be read)
    } else if (!AHEAD || tile != blockIdx.x) {
#pragma unroll
      for (int k = 0; k < E; ++k) v[k] = in[rowBase + ((uint64_t)(t + k * TPR) << logS)];
    }
    for (int o = 0; o < P.nOps; ++o) {
      const RowOp& op = P.ops[o];
      if (op.kind == kRowDiag) {
        rr_diag<C, LOGM, LOGE, rr_quads<C, LOGM, LOGE, LOGR, COL>()>(v, P.diag[op.diag], rowBase, tau);
      } else if constexpr (TWO) {
        auto next = [&] {
          if constexpr (PF) {
            __syncthreads();  // every group has read its last exchange
            fetch(tile + gridDim.x);
          }
        };
        const HookIf<decltype(next)> hook{PF && more && o == lastFft, next};
        if (op.dir > 0) rr_two<C, 1, LOGM, LOGE, LOGI>(v, smrow, t, tau, tw, hook);
        else rr_two<C, -1, LOGM, LOGE, LOGI>(v, smrow, t, tau, tw, hook);
      } else {
        if (op.dir > 0) rr_stages_tw<C, 1, LOGM, 0, LOGE>(v, smrow, t, tw, NoHook());
        else rr_stages_tw<C, -1, LOGM, 0, LOGE>(v, smrow, t, tw, NoHook());
      }
    }
    if constexpr (!COL) {
      // the row's |psi|^2 in TPR / 32 partials (one when a warp holds several rows)
      constexpr int W = TPR < 32 ? TPR : 32, PARTS = TPR < 32 ? 1 : TPR / 32;
      if (P.rowSums) row_sum_part<C, E, W>(v, P.rowSums + (rowBase >> LOGM) * PARTS + t / 32);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) out[rowBase + ((uint64_t)(tau + k * TPR) << logS)] = v[k];
  }
}

// largest row k_rowr takes (one CTA: 2^13 complex128 / 2^14 complex64 points)
inline int rowr_max_log(int precision) { return precision == kC128 ? 13 : 14; }

// log2 of the amplitudes a thread keeps of a row of 2^logM points.  Rows of 2^13 and 2^14
// points: 32 (256 / 512 threads; two exchanges in shared memory per transform instead of
// three: complex128 [13, 13] network rows 8.4 against 9.6 ms, columns 12.6 against 13.9).
// Otherwise 16, and up to 2^12 points 8 for tiny states and, in complex128, for small ones
// (below) and for rows shorter than 2^8 points.
constexpr int rowr_log_e(bool c128, int logM, bool small, bool tiny) {
  return logM >= 13 ? 5 : tiny || (c128 && (small || logM < 8)) ? 3 : 4;
}

template <typename C, int LOGM>
struct RrShape {
  static constexpr int LOGE = rowr_log_e(sizeof(C) == sizeof(double2), LOGM, false, false);
  static constexpr int LOGR = LOGM < 8 ? 7 - (LOGM - LOGE) : LOGM - LOGE < 8 ? 8 - (LOGM - LOGE) : 0;
};

// Rows of 2^8 .. 2^12 points of a state below 2^kRowrSmallLog amplitudes run one row
// per CTA (two at 2^8 points in complex64: a warp), at 8 amplitudes a thread in
// complex128: such a state does not fill the chip, so a program takes the latency of
// one CTA's chain, and more warps and CTAs shorten it.  A rotation, a displacement and a
// squeeze on 2^10-point rows of a complex128 state, small shape against full tiles: 26
// against 39 us at 2^18 amplitudes, 40 and 39 at 2^19, 56 and 52 at 2^20 (columns 28 / 39,
// 45 / 38, 70 / 48; complex64 rows 31 / 34, 31 / 33, 49 / 39).  States below a k_row tile
// (rowr_tiny) take 8 amplitudes a thread in both precisions, on twiddles rounded once: the
// radix-8 arithmetic of the tile passes (in complex64 the norm drifts by -3e-8 a transform of
// 2^12 points, by -4e-8 with radix-16 stages).
inline int row_log_tile(int precision) { return precision == kC128 ? 12 : 13; }  // of a k_row CTA
constexpr int kRowrSmallLog = 19;
inline bool rowr_small(Context* ctx) { return ctx->totalQbt < kRowrSmallLog; }
inline bool rowr_tiny(Context* ctx) { return ctx->totalQbt < row_log_tile(ctx->precision); }

// Whether shapes of 2^logM-point rows (columns) keep all twiddles, each rounded once: short
// registers and 2^8-point columns, where the table is 4 KB at most.  (Tiny states do at every
// length.)  A power tree multiplies the rounding of w by up to 15.  Relative error of a
// transform of random amplitudes, tree -> table: 2^8-point columns 6.6e-16 -> 2.2e-16 in
// complex128, 2.2e-7 -> 1.1e-7 in complex64; a 2^10-point state 4.5e-16 -> 2.3e-16 and
// 2.2e-7 -> 1.2e-7.  The other shapes keep the tree: their tables would take the shared
// memory of the rows.
constexpr bool rr_full(int logM, bool col) { return logM < 8 || (col && logM == 8); }

// The constants of the quadratic runs for a kernel of 2^logE amplitudes a thread:
// 4 c2 TPR^2 k^2 / (4 N) turns, reduced mod 1 before the 64-bit sine and cosine.
inline void fill_quads(RowProgram& P, int logM, int logE) {
  const double tpr2 = ldexp(1.0, 2 * (logM - logE)), N = ldexp(1.0, logM);
  for (int d = 0; d < P.nDiag; ++d) {
    RowDiag& D = P.diag[d];
    if (!D.hasQuad) continue;
    const double q = D.c2 / N;
    for (int k = 0; k < 1 << logE; ++k) {
      // (the last quarter turns are exact, so the angle keeps its digits)
      const double m = tpr2 * (double)(k * k), p = fma(q, m, -rint(q * m)), n = rint(4.0 * p);
      const double ang = 2.0 * CVDV_PI * (p - 0.25 * n), c = cos(ang), s = sin(ang);
      const int quarter = (int)n & 3;
      D.quad[k] = quarter == 0 ? make_double2(c, s) : quarter == 1 ? make_double2(-s, c)
                : quarter == 2 ? make_double2(-c, -s) : make_double2(s, -c);
    }
  }
}

template <typename C, int LOGM, int LOGR, int LOGE, bool COL, bool FULL>
static cudaError_t launch_rowr_s(Context* ctx, const void* in, void* out, const RowProgram& program) {
  RowProgram P = program;
  if constexpr (rr_quads<C, LOGM, LOGE, LOGR, COL>()) fill_quads(P, LOGM, LOGE);
  constexpr int NT = 1 << (LOGM - LOGE + LOGR);
  const size_t smem = (size_t)rr_line_slots<C, LOGM, LOGE, LOGR, COL>() * (1 << LOGR) * sizeof(C) +
                      (FULL ? sizeof(C) << LOGM : rr_tw_slots(LOGM) * sizeof(double2));
  auto kern = k_rowr<C, LOGM, LOGR, LOGE, COL, FULL>;
  // CTAs per SM of this instantiation: opted in and asked once per device
  static std::atomic<int> perDevice[kMaxDevices];
  const bool known = ctx->device >= 0 && ctx->device < kMaxDevices;
  int resident = known ? perDevice[ctx->device].load(std::memory_order_acquire) : 0;
  if (!resident) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, NT, smem);
    if (e != cudaSuccess || resident < 1) return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
    if (known) perDevice[ctx->device].store(resident, std::memory_order_release);
  }
  uint64_t nTiles = ctx->size() >> (LOGM + LOGR);
  if (nTiles < 1) nTiles = 1;
  uint64_t grid = rr_one<C, LOGM, LOGR, LOGE>() ? (uint64_t)ctx->numSMs * resident : nTiles;
  if (grid > nTiles) grid = nTiles;
  kern<<<(unsigned)grid, NT, smem, ctx->stream>>>((const C*)in, (C*)out, nTiles, P);
  return cudaGetLastError();
}

template <typename C, int LOGM, bool COL>
static cudaError_t launch_rowr_t(Context* ctx, const void* in, void* out, const RowProgram& P) {
  constexpr int LOGE = RrShape<C, LOGM>::LOGE, LOGR0 = RrShape<C, LOGM>::LOGR;
  // column form: at least two columns a CTA while it stays within 512 threads
  constexpr int LOGR = (COL && LOGR0 == 0 && (sizeof(C) << LOGM) < (128u << 10)) ? 1 : LOGR0;
  if constexpr (LOGM <= 12) {
    constexpr bool C128 = sizeof(C) == sizeof(double2);
    constexpr int SR = LOGM < 8 ? 8 - LOGM : 0;  // (a warp at 8 amplitudes a thread)
    if (rowr_tiny(ctx)) return launch_rowr_s<C, LOGM, SR, 3, COL, true>(ctx, in, out, P);
    constexpr bool TWO_ROWS = !C128 && LOGM == 8;  // two rows fill a warp
    if constexpr (LOGM >= 8)
      if (rowr_small(ctx)) return launch_rowr_s<C, LOGM, TWO_ROWS, C128 ? 3 : 4, COL, rr_full(LOGM, COL)>(ctx, in, out, P);
  }
  return launch_rowr_s<C, LOGM, LOGR, LOGE, COL, rr_full(LOGM, COL)>(ctx, in, out, P);
}

template <typename C, bool COL>
cudaError_t launch_rowr(Context* ctx, const void* in, void* out, const RowProgram& P, int q) {
  switch (q) {
    case 4: return launch_rowr_t<C, 4, COL>(ctx, in, out, P);
    case 5: return launch_rowr_t<C, 5, COL>(ctx, in, out, P);
    case 6: return launch_rowr_t<C, 6, COL>(ctx, in, out, P);
    case 7: return launch_rowr_t<C, 7, COL>(ctx, in, out, P);
    case 8: return launch_rowr_t<C, 8, COL>(ctx, in, out, P);
    case 9: return launch_rowr_t<C, 9, COL>(ctx, in, out, P);
    case 10: return launch_rowr_t<C, 10, COL>(ctx, in, out, P);
    case 11: return launch_rowr_t<C, 11, COL>(ctx, in, out, P);
    case 12: return launch_rowr_t<C, 12, COL>(ctx, in, out, P);
    case 13: return launch_rowr_t<C, 13, COL>(ctx, in, out, P);
    default:
      if constexpr (sizeof(C) == sizeof(float2)) return launch_rowr_t<C, 14, COL>(ctx, in, out, P);
      return cudaErrorInvalidValue;
  }
}

// the host's view of rr_quads for a 2^q-point register
inline bool rowr_quads(Context* ctx, int q, bool col) {
  if (ctx->precision == kC128) return q == 13 && (col ? rr_quads<double2, 13, 5, 0, true>() : rr_quads<double2, 13, 5, 0, false>());
  if (q == 13) return col ? rr_quads<float2, 13, 5, 1, true>() : rr_quads<float2, 13, 5, 0, false>();
  return q == 14 && (col ? rr_quads<float2, 14, 5, 0, true>() : rr_quads<float2, 14, 5, 0, false>());
}

extern template cudaError_t launch_rowr<double2, false>(Context*, const void*, void*, const RowProgram&, int);
extern template cudaError_t launch_rowr<double2, true>(Context*, const void*, void*, const RowProgram&, int);
extern template cudaError_t launch_rowr<float2, false>(Context*, const void*, void*, const RowProgram&, int);
extern template cudaError_t launch_rowr<float2, true>(Context*, const void*, void*, const RowProgram&, int);

}  // namespace cvdv
