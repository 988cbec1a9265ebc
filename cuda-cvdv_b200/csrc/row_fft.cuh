// Device building blocks of the register-resident row transforms, shared by
// the row-program kernels (kernels_row.cu) and the batched circuit kernels
// (kernels_batch.cu): radix-2/4/8/16 butterflies, two-level twiddle tables in
// shared memory, and Stockham stages on E amplitudes per thread.
#pragma once

#include "cvdv_internal.cuh"

namespace cvdv {

// shared-memory position of element e of a row: one padding slot every 16
// (the radix-16 stride), which keeps the strided butterfly accesses conflict-free
template <typename C, int LOGP = 4>
__device__ __forceinline__ int rpad(int e) {
  return e + (e >> LOGP);
}

// shared-memory elements of a padded row of 2^logM points (8 amplitudes a thread pad
// every 8), and twiddle entries (w^e, e < 64, then w^(64 h)) for it
__host__ __device__ constexpr int rr_row_slots(int logM, int logE) {
  return (1 << logM) + ((1 << logM) >> (logE == 3 ? 3 : 4));
}
// The same with room for 2^logR columns interleaved lane by lane: the W lanes that one
// phase of a 16- or 8-byte shared-memory access serves (W = 128 / bytes) are 2^logR
// columns x W / 2^logR consecutive points, so lines W / 2^logR elements apart modulo W
// put them on distinct banks; the padded length alone is a multiple of W, which put
// all columns' points on the same banks.
__host__ __device__ constexpr int rr_col_slots(int logM, int logE, int logR, int bytes) {
  const int W = 128 / bytes, step = (W >> logR) > 1 ? (W >> logR) : 1, len = rr_row_slots(logM, logE);
  return logR == 0 ? len : len + (step - len % W + W) % W;
}
__host__ __device__ constexpr int rr_tw_slots(int logM) { return 64 + (logM > 6 ? 1 << (logM - 6) : 1); }

// ---------------------------------------------------------------- butterflies
template <typename C, int DIR>
__device__ __forceinline__ C rot_mi(C a) {  // * (-DIR i)
  return DIR > 0 ? mk(a.y, -a.x) : mk(-a.y, a.x);
}

template <typename C, int DIR>
__device__ __forceinline__ void bf2(C& a, C& b) {
  C t = a;
  a = cadd(t, b);
  b = csub(t, b);
}

template <typename C, int DIR>
__device__ __forceinline__ void bf4(C& a0, C& a1, C& a2, C& a3) {
  C s02 = cadd(a0, a2), d02 = csub(a0, a2);
  C s13 = cadd(a1, a3), d13 = rot_mi<C, DIR>(csub(a1, a3));
  a0 = cadd(s02, s13);
  a2 = csub(s02, s13);
  a1 = cadd(d02, d13);
  a3 = csub(d02, d13);
}

// multiply by w8^K, w8 = exp(-DIR i pi / 4)
template <typename C, int DIR, int K>
__device__ __forceinline__ C w8mul(C o) {
  using T = decltype(o.x);
  const T h = (T)0.70710678118654752440;
  if constexpr (K == 0) return o;
  else if constexpr (K == 1)
    return DIR > 0 ? mk(h * (o.x + o.y), h * (o.y - o.x)) : mk(h * (o.x - o.y), h * (o.y + o.x));
  else if constexpr (K == 2) return rot_mi<C, DIR>(o);
  else
    return DIR > 0 ? mk(h * (o.y - o.x), -h * (o.x + o.y)) : mk(-h * (o.x + o.y), h * (o.x - o.y));
}

template <typename C, int DIR>
__device__ __forceinline__ void bf8(C* v) {
  C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  C o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  bf4<C, DIR>(e0, e1, e2, e3);
  bf4<C, DIR>(o0, o1, o2, o3);
  o1 = w8mul<C, DIR, 1>(o1);
  o2 = w8mul<C, DIR, 2>(o2);
  o3 = w8mul<C, DIR, 3>(o3);
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  v[1] = cadd(e1, o1);
  v[5] = csub(e1, o1);
  v[2] = cadd(e2, o2);
  v[6] = csub(e2, o2);
  v[3] = cadd(e3, o3);
  v[7] = csub(e3, o3);
}

// radix 16 = 4 x 4: y[k1 + 4 k2] = sum_n2 w4^{n2 k2} [ w16^{n2 k1} sum_n1 w4^{n1 k1} x[4 n1 + n2] ]
template <typename C, int DIR>
__device__ __forceinline__ void bf16(C* v) {
  using T = decltype(v[0].x);
  const T c1 = (T)0.92387953251128675613, s1 = (T)0.38268343236508977173;
  const T sg = DIR > 0 ? (T)-1 : (T)1;  // sign of the imaginary part of w16
  C a[16];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    C x0 = v[n2], x1 = v[4 + n2], x2 = v[8 + n2], x3 = v[12 + n2];
    bf4<C, DIR>(x0, x1, x2, x3);
    a[n2 * 4 + 0] = x0;
    a[n2 * 4 + 1] = x1;
    a[n2 * 4 + 2] = x2;
    a[n2 * 4 + 3] = x3;
  }
  auto mulw = [&](C x, T c, T s) { return mk(x.x * c - x.y * s, x.x * s + x.y * c); };
  a[5] = mulw(a[5], c1, sg * s1);     // w^1
  a[6] = w8mul<C, DIR, 1>(a[6]);      // w^2
  a[7] = mulw(a[7], s1, sg * c1);     // w^3
  a[9] = w8mul<C, DIR, 1>(a[9]);      // w^2
  a[10] = rot_mi<C, DIR>(a[10]);      // w^4
  a[11] = w8mul<C, DIR, 3>(a[11]);    // w^6
  a[13] = mulw(a[13], s1, sg * c1);   // w^3
  a[14] = w8mul<C, DIR, 3>(a[14]);    // w^6
  a[15] = mulw(a[15], -c1, -sg * s1); // w^9 = -w^1
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    C y0 = a[k1], y1 = a[4 + k1], y2 = a[8 + k1], y3 = a[12 + k1];
    bf4<C, DIR>(y0, y1, y2, y3);
    v[k1 + 0] = y0;
    v[k1 + 4] = y1;
    v[k1 + 8] = y2;
    v[k1 + 12] = y3;
  }
}

// radix 32 = 2 x 16: y[k] = E[k] + w32^k O[k], y[k + 16] = E[k] - w32^k O[k] with E, O
// the 16-point DFTs of the even and odd inputs (complex64 rows, 32 amplitudes a thread)
template <typename C, int DIR>
__device__ __forceinline__ void bf32(C* v) {
  using T = decltype(v[0].x);
  // cos(k pi / 16), k = 0..8
  constexpr double cs[9] = {1.0,
                            0.98078528040323044913,
                            0.92387953251128675613,
                            0.83146961230254523708,
                            0.70710678118654752440,
                            0.55557023301960222474,
                            0.38268343236508977173,
                            0.19509032201612826785,
                            0.0};
  C e[16], o[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    e[i] = v[2 * i];
    o[i] = v[2 * i + 1];
  }
  bf16<C, DIR>(e);
  bf16<C, DIR>(o);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    // w32^k = cos(k pi / 16) - DIR i sin(k pi / 16)
    const T c = (T)(k <= 8 ? cs[k] : -cs[16 - k]);
    const T sn = (T)(k <= 8 ? cs[8 - k] : cs[k - 8]);
    const T si = DIR > 0 ? -sn : sn;
    const C t = mk(o[k].x * c - o[k].y * si, o[k].x * si + o[k].y * c);
    v[k] = cadd(e[k], t);
    v[k + 16] = csub(e[k], t);
  }
}

template <typename C, int DIR, int RHO>
__device__ __forceinline__ void bfly(C* v) {
  if constexpr (RHO == 32) bf32<C, DIR>(v);
  else if constexpr (RHO == 16) bf16<C, DIR>(v);
  else if constexpr (RHO == 8) bf8<C, DIR>(v);
  else if constexpr (RHO == 4) bf4<C, DIR>(v[0], v[1], v[2], v[3]);
  else bf2<C, DIR>(v[0], v[1]);
}

// w_L^e = hi[e >> 6] * lo[e & 63] for e < L, forward convention exp(-2 pi i e / L);
// the conjugate for DIR < 0
template <typename C, int DIR>
__device__ __forceinline__ C tw2(const double2* lo, const double2* hi, int e) {
  double2 a = hi[e >> 6], b = lo[e & 63];
  double2 w = make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
  if (DIR < 0) w.y = -w.y;
  return fromd<C>(w);
}

// Where a transform's twiddles come from.  SplitTw: the split tables, one product and a
// tree of powers per butterfly.  FullTw: w_M^e for all e < M in shared memory, each
// rounded once.  StageTw: the same, in the order in which the stages read them: entry
// u ns + jm is w_(ns R)^(u jm) of the stage of radix R after ns points' worth of stages
// (1 <= u < R, jm < ns), so a warp reads consecutive entries (by e, a stage's strides are
// powers of two and most lanes' entries share a bank: a rotation, a displacement and a squeeze
// of a 2^11-point complex128 state take 49 us instead of 41, of a complex64 one of 2^12 58
// instead of 46).
struct SplitTw {
  static constexpr bool kByStage = false;
  const double2 *lo, *hi;
};
template <typename C>
struct FullTw {
  static constexpr bool kByStage = false;
  const C* w;
};
template <typename C>
struct StageTw {
  static constexpr bool kByStage = true;
  const C* w;
};
template <int DIR, typename C>
__device__ __forceinline__ C tw_dir(C w) {
  return DIR > 0 ? w : mk(w.x, -w.y);
}
// log2 of a full stage's radix, by the amplitudes a thread keeps
__host__ __device__ constexpr int rr_log_radix(int logE) { return logE >= 5 ? 5 : (logE == 3 ? 3 : 4); }
// exponent of w_M at entry y of a StageTw table (0 below the second stage's first entry)
template <int LOGM, int LOGE>
__device__ __forceinline__ int stage_tw_exponent(int y) {
  constexpr int LR = rr_log_radix(LOGE);
  int e = 0;
#pragma unroll
  for (int logNs = LR; logNs < LOGM; logNs += LR) {
    const int logR = LOGM - logNs < LR ? LOGM - logNs : LR;
    if (y >> logNs) e = ((y >> logNs) * (y & ((1 << logNs) - 1))) << (LOGM - logNs - logR);
  }
  return e;
}

// x[u] *= w_M^(e u) for u < RAD
template <typename C, int DIR, int RAD>
__device__ __forceinline__ void stage_powers(C (&x)[RAD], const SplitTw& T, int e) {
  // powers w^u as a tree (w^(u + 2^j) = w^u w^(2^j)); for radix 32 the upper
  // half is formed as it is applied, so only 17 powers are live at once
  constexpr int RT = RAD > 16 ? 16 : RAD;
  C w[RT + 1];
  w[1] = tw2<C, DIR>(T.lo, T.hi, e);
#pragma unroll
  for (int p = 1; p < RT / 2; p <<= 1) {
    w[2 * p] = cmul(w[p], w[p]);
#pragma unroll
    for (int u = 1; u < p; ++u) w[p + u] = cmul(w[p], w[u]);
  }
#pragma unroll
  for (int u = RT / 2 + 1; u < RT; ++u) w[u] = cmul(w[RT / 2], w[u - RT / 2]);
  if constexpr (RAD > 16) w[16] = cmul(w[8], w[8]);
#pragma unroll
  for (int u = 1; u < RT; ++u) x[u] = cmul(x[u], w[u]);
  if constexpr (RAD > 16) {
    x[16] = cmul(x[16], w[16]);
#pragma unroll
    for (int u = 17; u < RAD; ++u) x[u] = cmul(x[u], cmul(w[16], w[u - 16]));
  }
}
template <typename C, int DIR, int RAD>
__device__ __forceinline__ void stage_powers(C (&x)[RAD], const FullTw<C>& T, int e) {
#pragma unroll
  for (int u = 1; u < RAD; ++u) x[u] = cmul(x[u], tw_dir<DIR>(T.w[e * u]));
}

template <typename C, int DIR, int LOGM, int LOGRAD, int LOGNS, int LOGE, typename TW>
__device__ __forceinline__ void rr_butterflies(C (&v)[1 << LOGE], int t, const TW& tw) {
  constexpr int E = 1 << LOGE, RAD = 1 << LOGRAD, NB = E / RAD, TPR = 1 << (LOGM - LOGE);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    C x[RAD];
#pragma unroll
    for (int u = 0; u < RAD; ++u) x[u] = v[b + NB * u];
    if constexpr (LOGNS > 0) {
      const int jm = (t + b * TPR) & ((1 << LOGNS) - 1);
      // w_{ns R}^{jm u} = w_M^{(jm u) << (LOGM - LOGNS - LOGRAD)}
      if constexpr (TW::kByStage) {
#pragma unroll
        for (int u = 1; u < RAD; ++u) x[u] = cmul(x[u], tw_dir<DIR>(tw.w[(u << LOGNS) + jm]));
      } else {
        stage_powers<C, DIR, RAD>(x, tw, jm << (LOGM - LOGNS - LOGRAD));
      }
    }
    bfly<C, DIR, RAD>(x);
#pragma unroll
    for (int u = 0; u < RAD; ++u) v[b + NB * u] = x[u];
  }
}

// outputs of a stage to their autosorted positions, then the next stage's inputs
// (padding period 2^LOGP elements: 16 for radix-16 stages, 32 for radix-32 ones,
// so the first stage's writes at stride RAD stay free of bank conflicts)
template <typename C, int LOGM, int LOGRAD, int LOGNS, int LOGE, int LOGP = 4>
__device__ __forceinline__ void rr_exchange(C (&v)[1 << LOGE], C* smrow, int t) {
  constexpr int E = 1 << LOGE, RAD = 1 << LOGRAD, NB = E / RAD, TPR = 1 << (LOGM - LOGE);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = t + b * TPR;
    const int y = ((j >> LOGNS) << (LOGNS + LOGRAD)) + (j & ((1 << LOGNS) - 1));
#pragma unroll
    for (int u = 0; u < RAD; ++u) smrow[rpad<C, LOGP>(y + (u << LOGNS))] = v[b + NB * u];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < E; ++k) v[k] = smrow[rpad<C, LOGP>(t + k * TPR)];
  __syncthreads();
}

// The stages of one transform: radix 16 (radix 32 with 32 amplitudes a thread,
// radix 8 with 8), then the remaining radix.  The shared row holds at least
// M + M/16 elements (M + M/8 with 8 amplitudes a thread).
// AFTER: a callable run once the shared row is no longer needed (after the last
// exchange, before the last stage's butterflies)
struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};
template <typename C, int DIR, int LOGM, int S, int LOGE, typename TW, typename H>
__device__ __forceinline__ void rr_stages_tw(C (&v)[1 << LOGE], C* smrow, int t, const TW& tw, H after) {
  constexpr int LR = rr_log_radix(LOGE);
  constexpr int NF = LOGM / LR, REM = LOGM % LR;
  if constexpr (S < NF) {
    rr_butterflies<C, DIR, LOGM, LR, LR * S, LOGE>(v, t, tw);
    if constexpr (S + 1 < NF || REM) rr_exchange<C, LOGM, LR, LR * S, LOGE, LR>(v, smrow, t);
    if constexpr ((REM > 0 && S + 1 == NF) || (REM == 0 && S + 2 == NF)) after();
    rr_stages_tw<C, DIR, LOGM, S + 1, LOGE>(v, smrow, t, tw, after);
  } else if constexpr (REM > 0) {
    rr_butterflies<C, DIR, LOGM, REM, LR * NF, LOGE>(v, t, tw);
  }
}
template <typename C, int DIR, int LOGM, int S, int LOGE = 4, typename H = NoHook>
__device__ __forceinline__ void rr_stages(C (&v)[1 << LOGE], C* smrow, int t, const double2* lo,
                                          const double2* hi, H after = H()) {
  rr_stages_tw<C, DIR, LOGM, S, LOGE>(v, smrow, t, SplitTw{lo, hi}, after);
}

// ---------------------------------------------------------------- one CTA exchange
// x[u] *= w^u for u < RAD, w = w_L^e from the tables, the powers as a tree.  w^16 (and
// w^4 in complex128) come from the tables too: products of w alone multiply its error
// by u, up to 31 where radix 16 has 15.  Error of a three-layer network on [13, 6]
// against extended precision: complex128 2.5e-14 with w alone, 1.6e-14 with w^16, 1.1e-14
// with w^4 and w^16, as with the radix-16 stages (complex64 2.5e-6, 1.7e-6, 2.1e-6).  For radix 32
// the upper half is formed as it is applied, so only 17 powers are live at once.
template <typename C, int DIR, int RAD>
__device__ __forceinline__ void mul_powers(C (&x)[RAD], const FullTw<C>& T, int e) {
  stage_powers<C, DIR, RAD>(x, T, e);
}
template <typename C, int DIR, int RAD>
__device__ __forceinline__ void mul_powers(C (&x)[RAD], const SplitTw& T, int e) {
  constexpr int RT = RAD > 16 ? 16 : RAD;
  C w[RT + 1];
#pragma unroll
  for (int p = 1; p < RT; p <<= 1) {
    if (p == 1 || (p == 4 && sizeof(C) == 16)) w[p] = tw2<C, DIR>(T.lo, T.hi, e * p);
    else w[p] = cmul(w[p / 2], w[p / 2]);
#pragma unroll
    for (int u = 1; u < p; ++u) w[p + u] = cmul(w[p], w[u]);
  }
  if constexpr (RAD > 16) w[16] = tw2<C, DIR>(T.lo, T.hi, e * 16);
#pragma unroll
  for (int u = 1; u < RT; ++u) x[u] = cmul(x[u], w[u]);
  if constexpr (RAD > 16) {
    x[16] = cmul(x[16], w[16]);
#pragma unroll
    for (int u = 17; u < RAD; ++u) x[u] = cmul(x[u], cmul(w[16], w[u - 16]));
  }
}

// Shape of a transform of N = E M points (M = E G threads a row, E amplitudes each)
// with one exchange across the row's threads and one inside groups of G <= 32 of them:
//   A  thread tau holds x[tau + M j]; radix E over j, times w_N^{tau k1}: y_k1[tau]
//   1  y_k1 goes to region k1 of the shared line; group k1's thread g takes y_k1[g + G j]
//   B  radix E over j, times w_M^{g c}: z_c[g]
//   2  z_c[g] inside the region; thread g takes z_c for c = g + G i (i < E / G)
//   C  radix G over g: X[k1 + E (c + E d)]
// so thread (k1, g) ends with X[tau' + M k], tau' = k1 + E g: the layout it started
// from, under another thread number.  Only exchange 1 needs the CTA's barriers (one
// before it is written, one after); exchange 2 is the warp's own, and from one
// transform's exchange 1 to the next the warps run apart, so one warp's butterflies
// overlap another's exchange.  The Stockham stages (rr_stages) pass two CTA barriers
// per exchange, which kept all warps of a row in the same phase ([13, 13] network with
// 32 amplitudes a thread: complex128 rows 7.95 against 8.39 ms, columns 11.9 against
// 12.6; complex64 columns 6.5 against 7.4).
//
// 2^LOGI lines are interleaved lane by lane (columns); the paddings PAD and RR put the
// W lanes that one phase of a shared access serves on distinct banks: they are 2^LOGI
// lines x consecutive g x consecutive k1.
template <typename C, int LOGM, int LOGE, int LOGI>
struct RrTwo {
  static constexpr int LOGG = LOGM - 2 * LOGE;
  static constexpr bool ok = LOGG >= 0 && LOGG <= LOGE && LOGG + LOGI <= 5;
  static constexpr int E = 1 << LOGE, G = ok ? 1 << LOGG : 1, M = E * G, W = 128 / (int)sizeof(C), I = 1 << LOGI;
  static constexpr int PAD = G * I < W ? W / (G * I) : 1;
  static constexpr int RR0 = M + (PAD * G > E ? PAD * G : E);
  static constexpr int RR = RR0 + (G < W ? (G - RR0 % W + W) % W : 0);
  static constexpr int LINE0 = E * RR;
  static constexpr int LINE = LOGI == 0 ? LINE0 : LINE0 + ((W / I > 1 ? W / I : 1) - LINE0 % W + W) % W;
};

template <typename C, int DIR, int LOGM, int LOGE, int LOGI, typename TW, typename H = NoHook>
__device__ __forceinline__ void rr_two(C (&v)[1 << LOGE], C* line, int t, int& tau, const TW& tw, H after = H()) {
  using S = RrTwo<C, LOGM, LOGE, LOGI>;
  constexpr int E = S::E, G = S::G, EG = E / G;
  bfly<C, DIR, E>(v);
  mul_powers<C, DIR, E>(v, tw, tau);
  __syncthreads();  // the line is free: every group has read its last exchange
  {
    C* p = line + tau + S::PAD * (tau >> LOGE);
#pragma unroll
    for (int k = 0; k < E; ++k) p[k * S::RR] = v[k];
  }
  __syncthreads();
  const int k1 = t >> S::LOGG, g = t & (G - 1);
  C* reg = line + k1 * S::RR;
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = reg[g + G * j + S::PAD * ((G * j) >> LOGE)];
  bfly<C, DIR, E>(v);
  if constexpr (G > 1) {
    mul_powers<C, DIR, E>(v, tw, g << LOGE);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < E; ++c) reg[c * (G + 1) + g] = v[c];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < EG; ++i) {
      C a[G];
#pragma unroll
      for (int u = 0; u < G; ++u) a[u] = reg[(g + G * i) * (G + 1) + u];
      bfly<C, DIR, G>(a);
#pragma unroll
      for (int d = 0; d < G; ++d) v[i + EG * d] = a[d];
    }
  }
  tau = k1 + (g << LOGE);
  after();
}

}  // namespace cvdv
