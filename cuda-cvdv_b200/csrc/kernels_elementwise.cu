// Elementwise kernels: diagonal factor tables, fused diagonal runs, 2x2 qubit
// pairs, register permutations and the separable-product initialiser.
//
// Every kernel here is one coalesced read + write of the state (HBM-bound);
// the per-element work is a handful of FP64 multiplies against factor tables
// that stay resident in L1/L2.

#include <cudaTypedefs.h>

#include "cvdv_internal.cuh"
#include "turns.cuh"

namespace cvdv {

// ----------------------------------------------------------------- tables
// Tables of one launch, by value: J tables with T terms between them.  Each table
// gets a run of consecutive blocks from block0 on.
struct TableHead {
  double2* out;
  double dx;
  int logN, ctrl, permLogC;
  int nTerms, term0, block0;
};
template <int J, int T>
struct TableBatch {
  int nJobs;
  TableHead job[J];
  TableTerm term[T];
};

// Table entry (b, j) = prod over terms.  Terms of degree one and two and transform
// twiddles are summed in turns (turns.cuh) and take one sine and cosine;
// cubic terms are summed in radians, in the reference's order of operations (x = (idx -
// (dim-1)*0.5)*dx, kernelPhaseX3, src/cuda/kernels/gates.cuh:5-16,184-209).
//
// All tables of a flush are built by one launch: a table is 2^8 .. 2^15 entries, a
// launch of its own took about 3 us however short, and a circuit has several per
// mode gate (63 tables of a 60-gate circuit: 198 us in 63 launches).
constexpr int kTableThreads = 256;
template <int J, int T>
__global__ void __launch_bounds__(kTableThreads) k_build_tables(const __grid_constant__ TableBatch<J, T> B) {
  int lo = 0, hi = B.nJobs;  // the table whose run of blocks holds this block
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (B.job[mid].block0 <= (int)blockIdx.x) lo = mid;
    else hi = mid;
  }
  const TableHead& H = B.job[lo];
  const int e = ((int)blockIdx.x - H.block0) * kTableThreads + (int)threadIdx.x;
  const int N = 1 << H.logN;
  if (e >= N << H.ctrl) return;
  int j = e & (N - 1);
  const int b = e >> H.logN;
  if (H.permLogC) {
    const int logM = H.logN - H.permLogC;
    j = ((j & ((1 << logM) - 1)) << H.permLogC) + (j >> logM);
  }
  // twiddles and terms of degree one and two in turns, cubic terms in radians
  const int u = 2 * j - N + 1;
  const double inv4N = 0.25 / (double)N;
  const LinTurns L = lin_turns(H.logN);
  Turns1<true> p;
  double cubic = 0.0;
  bool anyTurns = false, anyCubic = false;
  double2 f = make_double2(1.0, 0.0);
  for (int t = H.term0; t < H.term0 + H.nTerms; ++t) {
    const TableTerm& D = B.term[t];
    if (D.kind == kTermPoly) {
      const bool neg = (D.ctrlMode == 1 && ((b >> D.ctrlLocal) & 1)) || (D.ctrlMode == 2 && ((j >> D.ctrlLocal) & 1));
      const double c = neg ? -D.coeff : D.coeff;
      if (D.power == 1) {
        p.add(turn_rate(c, L.hi, L.lo), (double)u);
        anyTurns = true;
      } else if (D.power == 2) {
        p.add({c * inv4N, 0.0}, (double)u * (double)u);
        anyTurns = true;
      } else {
        const double x = 0.5 * (double)u * H.dx;
        cubic += c * x * x * x;
        anyCubic = true;
      }
    } else if (D.kind == kTermFtTw) {
      const long long n = N;  // (N-1) u mod 4N, N a power of two
      const long long m = (((n - 1) * u + 2 * n) & (4 * n - 1)) - 2 * n;
      p.add({(double)D.sign * inv4N, 0.0}, (double)m);
      anyTurns = true;
    } else if (D.kind == kTermBit) {
      f = dmul(f, ((j >> D.bit) & 1) ? D.g1 : D.g0);
    }
  }
  if (anyTurns) f = dmul(p.root(), f);
  if (anyCubic) {
    double s, c;
    sincos(cubic, &s, &c);
    f = dmul(make_double2(c, s), f);
  }
  H.out[e] = f;
}

// Launch sizes: parameters of up to 4 KB for a few tables, and close to the 32764
// bytes a kernel may take for many; longer lists go in several launches.
template <int J, int T>
static bool launch_table_batch(Context* ctx, const std::vector<TableJob>& jobs, size_t first, size_t count) {
  static_assert(sizeof(TableBatch<J, T>) <= 32764, "kernel parameters");
  TableBatch<J, T> B;
  B.nJobs = (int)count;
  int nt = 0, blocks = 0;
  for (size_t k = 0; k < count; ++k) {
    const TableJob& D = jobs[first + k];
    TableHead& H = B.job[k];
    H.out = D.out;
    H.dx = D.dx;
    H.logN = D.logN;
    H.ctrl = D.ctrl;
    H.permLogC = D.permLogC;
    H.nTerms = (int)D.terms.size();
    H.term0 = nt;
    H.block0 = blocks;
    for (const TableTerm& t : D.terms) B.term[nt++] = t;
    blocks += (int)((((size_t)1 << (D.logN + D.ctrl)) + kTableThreads - 1) / kTableThreads);
  }
  {
    LaunchScope _ls(ctx, kKTable);
    k_build_tables<J, T><<<blocks, kTableThreads, 0, ctx->stream>>>(B);
  }
  return cuda_ok(ctx, cudaGetLastError(), "build_table launch");
}

bool launch_tables(Context* ctx, const std::vector<TableJob>& jobs) {
  constexpr int JS = 24, TS = 60, JL = 160, TL = 500;
  size_t i = 0;
  while (i < jobs.size()) {
    size_t n = 0, terms = 0, blocks = 0;
    for (; i + n < jobs.size() && n < (size_t)JL; ++n) {
      const size_t t = jobs[i + n].terms.size(), b = ((size_t)1 << (jobs[i + n].logN + jobs[i + n].ctrl)) / kTableThreads + 1;
      if (n > 0 && (terms + t > (size_t)TL || blocks + b > (size_t)1 << 30)) break;
      terms += t;
      blocks += b;
    }
    if (!(n <= (size_t)JS && terms <= (size_t)TS ? launch_table_batch<JS, TS>(ctx, jobs, i, n)
                                                 : launch_table_batch<JL, TL>(ctx, jobs, i, n)))
      return false;
    i += n;
  }
  return true;
}

// Table over register r with nExt external control bits (extBits, flat-index
// positions outside r): entry [seg][j], seg bit c = value of extBits[c].
bool launch_build_table_ext(Context* ctx, int r, int nExt, const int* extBits, const Term* terms,
                            int nTerms, double2* out, int permLogC) {
  TableJob job;
  job.out = out;
  job.dx = ctx->dx[r];
  job.logN = ctx->q[r];
  job.ctrl = nExt;
  job.permLogC = permLogC;
  job.terms.reserve(nTerms);
  const int lo = ctx->flw[r], hi = ctx->flw[r] + ctx->q[r];
  for (int t = 0; t < nTerms; ++t) {
    const Term& T = terms[t];
    TableTerm D{};
    D.kind = (signed char)T.kind;
    D.power = (signed char)T.power;
    D.sign = (signed char)T.sign;
    D.bit = (signed char)T.bit;
    D.coeff = T.coeff;
    D.g0 = T.g0;
    D.g1 = T.g1;
    if (T.kind == kTermPoly && T.ctrlBit >= 0) {
      if (T.ctrlBit >= lo && T.ctrlBit < hi) {
        D.ctrlMode = 2;
        D.ctrlLocal = (signed char)(T.ctrlBit - lo);
      } else {
        D.ctrlMode = 1;
        for (int c = 0; c < nExt; ++c)
          if (extBits[c] == T.ctrlBit) D.ctrlLocal = (signed char)c;
      }
    }
    job.terms.push_back(D);
  }
  if (ctx->plan) {
    ctx->plan->tables.push_back(std::move(job));
    return true;
  }
  return launch_tables(ctx, {std::move(job)});
}

bool launch_build_table(Context* ctx, int r, bool ctrl, const Term* terms, int nTerms,
                        double2* out) {
  int bit = -1;
  if (ctrl) {
    int lo = ctx->flw[r], hi = lo + ctx->q[r];
    for (int t = 0; t < nTerms; ++t)
      if (terms[t].kind == kTermPoly && terms[t].ctrlBit >= 0 &&
          !(terms[t].ctrlBit >= lo && terms[t].ctrlBit < hi))
        bit = terms[t].ctrlBit;
  }
  return launch_build_table_ext(ctx, r, ctrl ? 1 : 0, &bit, terms, nTerms, out,
                                r == ctx->permReg ? ctx->permLogC : 0);
}

// ----------------------------------------------------------------- diag run
// A thread takes V = 4 amplitudes i0 + 256 k with i0 a multiple of 1024 plus the
// thread index: its indices differ only in bits 8-9, which hold k.  A register
// field that misses those bits has the same index for all four, so its table
// entry is loaded once; a field that contains both (and reaches bit 8 or lower)
// advances by 2^(8 - shift) per k, so a bilinear term c x_r x_s whose sides are
// each fixed or advancing (and whose control, if any, is not bit 8 or 9) is
// linear in k: its value at k = 0 and the ratio between steps, two sincos,
// replace the four per-amplitude ones.  Other factors are evaluated per amplitude.
template <typename C>
__global__ void __launch_bounds__(256) k_diag(C* __restrict__ st, uint64_t n, FactorList F) {
  constexpr int V = 4;  // 256 threads x V amplitudes span bits 0..9
  // -1: the field holds one of bits 8, 9 only; 0: neither; else the step per k
  auto field = [](int shift, int mask) -> int {
    const int q = __popc(mask);
    if (shift >= 10 || shift + q <= 8) return 0;
    return (shift <= 8 && shift + q >= 10) ? (1 << (8 - shift)) : -1;
  };
  auto ctrl_fixed = [](int c) { return c < 8 || c > 9; };  // (-1: no control)
  const uint64_t stride = (uint64_t)gridDim.x * 256 * V;
  for (uint64_t base = (uint64_t)blockIdx.x * 256 * V + threadIdx.x; base < n; base += stride) {
    C v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const uint64_t i = base + (uint64_t)k * 256;
      if (i < n) v[k] = st[i];
    }
    double2 g[V];
#pragma unroll
    for (int k = 0; k < V; ++k) g[k] = F.hasScalar ? F.scalar : make_double2(1.0, 0.0);
#pragma unroll
    for (int t = 0; t < kMaxTab; ++t) {
      if (t >= F.nTab) break;
      const TabFactor& T = F.tab[t];
      if (field(T.shift, T.mask) == 0 && ctrl_fixed(T.ctrlShift)) {
        int j = (int)((base >> T.shift) & (uint64_t)T.mask);
        if (T.ctrlShift >= 0) j += (int)((base >> T.ctrlShift) & 1ull) * T.half;
        const double2 a = __ldg(T.ptr + j);
#pragma unroll
        for (int k = 0; k < V; ++k) g[k] = dmul(g[k], a);
      } else {
        double2 a[V];
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const uint64_t i = base + (uint64_t)k * 256;
          int j = (int)((i >> T.shift) & (uint64_t)T.mask);
          if (T.ctrlShift >= 0) j += (int)((i >> T.ctrlShift) & 1ull) * T.half;
          a[k] = __ldg(T.ptr + j);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) g[k] = dmul(g[k], a[k]);
      }
    }
#pragma unroll 1
    for (int x = 0; x < F.nXX; ++x) {
      const XXFactor& X = F.xx[x];
      const int s1 = field(X.shift1, X.mask1), s2 = field(X.shift2, X.mask2);
      if (s1 >= 0 && s2 >= 0 && ctrl_fixed(X.ctrlShift)) {
        const double x1 = ((double)((base >> X.shift1) & (uint64_t)X.mask1) - X.c1) * X.dx1;
        const double x2 = ((double)((base >> X.shift2) & (uint64_t)X.mask2) - X.c2) * X.dx2;
        double c = X.coeff;
        if (X.ctrlShift >= 0 && ((base >> X.ctrlShift) & 1ull)) c = -c;
        // (the two registers differ, so at most one side advances)
        const double d = s1 ? c * ((double)s1 * X.dx1) * x2 : s2 ? c * x1 * ((double)s2 * X.dx2) : 0.0;
        double sn, cs;
        sincos(c * x1 * x2, &sn, &cs);
        double2 e = make_double2(cs, sn), stp;
        sincos(d, &stp.y, &stp.x);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          g[k] = dmul(g[k], e);
          e = dmul(e, stp);
        }
      } else {
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const uint64_t i = base + (uint64_t)k * 256;
          const double x1 = ((double)((i >> X.shift1) & (uint64_t)X.mask1) - X.c1) * X.dx1;
          const double x2 = ((double)((i >> X.shift2) & (uint64_t)X.mask2) - X.c2) * X.dx2;
          double ph = X.coeff * x1 * x2;
          if (X.ctrlShift >= 0 && ((i >> X.ctrlShift) & 1ull)) ph = -ph;
          double sn, cs;
          sincos(ph, &sn, &cs);
          g[k] = dmul(g[k], make_double2(cs, sn));
        }
      }
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const uint64_t i = base + (uint64_t)k * 256;
      if (i < n) st[i] = cmul(v[k], fromd<C>(g[k]));
    }
  }
}

static int grid_for(uint64_t work, int threads, int perThread) {
  uint64_t b = (work + (uint64_t)threads * perThread - 1) / ((uint64_t)threads * perThread);
  uint64_t cap = 148ull * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

bool launch_diag(Context* ctx, const FactorList& F) {
  const uint64_t n = ctx->size();
  const int blocks = grid_for(n, 256, 4);
  void* st = ctx->state();
  return enqueue(ctx, kKDiag, "diag launch", [=] {
    if (ctx->precision == kC128) k_diag<double2><<<blocks, 256, 0, ctx->stream>>>((double2*)st, n, F);
    else k_diag<float2><<<blocks, 256, 0, ctx->stream>>>((float2*)st, n, F);
    return cudaGetLastError();
  });
}

// ----------------------------------------------------------------- pair (2x2)
// Pair indexing as qubitPairIndices (src/cuda/kernels/utils.cuh:79-84).
// Each thread takes kPairV pairs per iteration, all loads issued first.  The
// factor-free instance (the common case: neighbouring diagonal runs usually
// ride on a row program) is a separate, lean specialisation.
constexpr int kPairV = 4;

// MAXT: 0 = no factors; 2 = at most two tables and no bilinear terms (the
// usual neighbouring run: a qubit phase and one mode table); kMaxTab = general.
template <typename C, int MAXT>
__global__ void __launch_bounds__(256) k_pair(C* __restrict__ st, uint64_t npairs, int bit,
                                             double2 m00, double2 m01, double2 m10, double2 m11,
                                             const __grid_constant__ FactorList pre,
                                             const __grid_constant__ FactorList post) {
  constexpr int V = MAXT == 0 ? kPairV : (MAXT == 2 ? 2 : 1);
  constexpr bool XX = MAXT == kMaxTab;
  const uint64_t lowMask = (1ull << bit) - 1;
  const C a00 = fromd<C>(m00), a01 = fromd<C>(m01), a10 = fromd<C>(m10), a11 = fromd<C>(m11);
  const bool hasPre = MAXT > 0 && !factor_empty(pre), hasPost = MAXT > 0 && !factor_empty(post);
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x * V;
  for (uint64_t p0 = (uint64_t)blockIdx.x * blockDim.x * V + threadIdx.x; p0 < npairs;
       p0 += step) {
    C a[V], b[V];
    uint64_t i0[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      uint64_t p = p0 + (uint64_t)v * blockDim.x;
      i0[v] = ((p & ~lowMask) << 1) | (p & lowMask);
      if (p < npairs) {
        a[v] = st[i0[v]];
        b[v] = st[i0[v] | (1ull << bit)];
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      uint64_t p = p0 + (uint64_t)v * blockDim.x;
      if (p >= npairs) continue;
      uint64_t i1 = i0[v] | (1ull << bit);
      C x = a[v], y = b[v];
      if constexpr (MAXT > 0) {
        if (hasPre) {
          x = cmul(x, fromd<C>(eval_factor_t<(MAXT > 0 ? MAXT : 1), XX>(pre, i0[v])));
          y = cmul(y, fromd<C>(eval_factor_t<(MAXT > 0 ? MAXT : 1), XX>(pre, i1)));
        }
      }
      C nx = cadd(cmul(a00, x), cmul(a01, y));
      C ny = cadd(cmul(a10, x), cmul(a11, y));
      if constexpr (MAXT > 0) {
        if (hasPost) {
          nx = cmul(nx, fromd<C>(eval_factor_t<(MAXT > 0 ? MAXT : 1), XX>(post, i0[v])));
          ny = cmul(ny, fromd<C>(eval_factor_t<(MAXT > 0 ? MAXT : 1), XX>(post, i1)));
        }
      }
      st[i0[v]] = nx;
      st[i1] = ny;
    }
  }
}

template <typename C>
static void pair_launch(Context* ctx, C* st, uint64_t np, int bit, const double2 m[4],
                        const FactorList& pre, const FactorList& post) {
  bool none = factor_empty(pre) && factor_empty(post);
  bool small = pre.nTab <= 2 && post.nTab <= 2 && pre.nXX == 0 && post.nXX == 0;
  if (none)
    k_pair<C, 0><<<grid_for(np, 256, kPairV), 256, 0, ctx->stream>>>(st, np, bit, m[0], m[1], m[2],
                                                                      m[3], pre, post);
  else if (small)
    k_pair<C, 2><<<grid_for(np, 256, 2), 256, 0, ctx->stream>>>(st, np, bit, m[0], m[1], m[2],
                                                                m[3], pre, post);
  else
    k_pair<C, kMaxTab><<<grid_for(np, 256, 1), 256, 0, ctx->stream>>>(st, np, bit, m[0], m[1],
                                                                      m[2], m[3], pre, post);
}

struct PairMatrix {
  double2 m[4];
};

bool launch_pair(Context* ctx, int bit, const double2 m[4], const FactorList& pre,
                 const FactorList& post) {
  const uint64_t np = ctx->size() / 2;
  void* st = ctx->state();
  const PairMatrix M = {{m[0], m[1], m[2], m[3]}};
  return enqueue(ctx, kKPair, "pair launch", [=] {
    if (ctx->precision == kC128) pair_launch<double2>(ctx, (double2*)st, np, bit, M.m, pre, post);
    else pair_launch<float2>(ctx, (float2*)st, np, bit, M.m, pre, post);
    return cudaGetLastError();
  });
}

// ----------------------------------------------------------------- permutations
// Out-of-place gather out[i] = in[src(i)].  src is an involution:
//  parity       j_r -> N-1-j_r  (kernelParity, gates.cuh:113-131)
//  cond parity  the pair {j, N-1-j} is exchanged iff the control bit of the
//               element with the smaller local index is 1
//               (kernelConditionalParity, gates.cuh:134-158)
//  swap         (j_r1, j_r2) -> (j_r2, j_r1)   (kernelSwapRegisters, gates.cuh:161-182)
struct PermDesc {
  int kind;
  int shift1, q1, shift2;
  int ctrlBit;
};

__device__ __forceinline__ uint64_t perm_src(const PermDesc& P, uint64_t i) {
  uint64_t m1 = ((1ull << P.q1) - 1) << P.shift1;
  if (P.kind == kPermParity) return i ^ m1;
  if (P.kind == kPermCondParity) {
    uint64_t loc = (i & m1) >> P.shift1;
    uint64_t N = 1ull << P.q1;
    uint64_t small = loc < (N - 1 - loc) ? loc : (N - 1 - loc);
    uint64_t is = (i & ~m1) | (small << P.shift1);
    return ((is >> P.ctrlBit) & 1ull) ? (i ^ m1) : i;
  }
  uint64_t m2 = ((1ull << P.q1) - 1) << P.shift2;
  uint64_t a = (i & m1) >> P.shift1;
  uint64_t b = (i & m2) >> P.shift2;
  return (i & ~(m1 | m2)) | (b << P.shift1) | (a << P.shift2);
}

// Each thread issues its V gathers before evaluating any factor, so V loads are in
// flight per thread.
template <typename C>
__global__ void __launch_bounds__(256) k_perm(const C* __restrict__ in, C* __restrict__ out,
                                             uint64_t n, PermDesc P, FactorList pre,
                                             FactorList post) {
  constexpr int V = 4;
  const bool hasPre = !factor_empty(pre), hasPost = !factor_empty(post);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * V;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x * V + threadIdx.x; base < n; base += stride) {
    C v[V];
    uint64_t s[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const uint64_t i = base + (uint64_t)k * blockDim.x;
      s[k] = i < n ? perm_src(P, i) : 0;
      if (i < n) v[k] = in[s[k]];
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const uint64_t i = base + (uint64_t)k * blockDim.x;
      if (i >= n) continue;
      if (hasPre) v[k] = cmul(v[k], fromd<C>(eval_factor(pre, s[k])));
      if (hasPost) v[k] = cmul(v[k], fromd<C>(eval_factor(post, i)));
      out[i] = v[k];
    }
  }
}

bool launch_perm(Context* ctx, const Stage& st, const FactorList& pre, const FactorList& post) {
  PermDesc P{};
  P.kind = st.perm;
  P.shift1 = ctx->flw[st.reg];
  P.q1 = ctx->q[st.reg];
  P.shift2 = st.reg2 >= 0 ? ctx->flw[st.reg2] : 0;
  P.ctrlBit = st.bit;
  const uint64_t n = ctx->size();
  const int blocks = grid_for(n, 256, 4);
  const void* in = ctx->state();
  void* out = ctx->other();
  const bool ok = enqueue(ctx, kKPerm, "perm launch", [=] {
    if (ctx->precision == kC128)
      k_perm<double2><<<blocks, 256, 0, ctx->stream>>>((const double2*)in, (double2*)out, n, P, pre, post);
    else
      k_perm<float2><<<blocks, 256, 0, ctx->stream>>>((const float2*)in, (float2*)out, n, P, pre, post);
    return cudaGetLastError();
  });
  if (ok) ctx->cur ^= 1;
  return ok;
}

// ----------------------------------------------------------------- separable init
// psi[i] = prod_r phi_r[j_r(i)], last register fastest (cvdvInitFromSeparable,
// src/cuda/context.cu:75-115; no normalisation).  Two steps: the product over
// all registers but the last into a small "outer" table, then one complex
// multiply per amplitude.
struct InitDesc {
  int numReg;
  int qLast;
  const double2* arr[kMaxRegs];  // the register arrays
  int shift[kMaxRegs];  // flw of each register minus qLast (index into outer)
  int mask[kMaxRegs];
};

__global__ void k_init_outer(InitDesc D, double2* outer, uint64_t nOuter) {
  for (uint64_t h = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; h < nOuter;
       h += (uint64_t)gridDim.x * blockDim.x) {
    double2 p = make_double2(1.0, 0.0);
    for (int r = D.numReg - 2; r >= 0; --r) {
      int j = (int)((h >> D.shift[r]) & (uint64_t)D.mask[r]);
      p = dmul(p, D.arr[r][j]);
    }
    outer[h] = p;
  }
}

template <typename C>
__global__ void __launch_bounds__(256) k_init_product(C* __restrict__ st, uint64_t n, int qLast,
                                                     const double2* __restrict__ last,
                                                     const double2* __restrict__ outer) {
  const uint64_t lm = (1ull << qLast) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    double2 v = dmul(__ldg(last + (i & lm)), __ldg(outer + (i >> qLast)));
    st[i] = fromd<C>(v);
  }
}

// The register arrays of a separable state in one launch: dst holds them back to
// back (a copy call per register took 5-7 us of host time each).
struct GatherDesc {
  int numReg;
  const double2* src[kMaxRegs];
  unsigned end[kMaxRegs];  // first element after the register in dst
};
__global__ void __launch_bounds__(256) k_gather_arrays(const __grid_constant__ GatherDesc D, double2* __restrict__ dst) {
  const unsigned total = D.end[D.numReg - 1];
  for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
    int r = 0;
    while (i >= D.end[r]) ++r;
    dst[i] = D.src[r][i - (r ? D.end[r - 1] : 0)];
  }
}

// Whether [p, p + bytes) lies in one allocation, as a copy call checks before it reads.
// False where the driver cannot tell.
static bool in_one_allocation(const void* p, size_t bytes) {
  static const PFN_cuMemGetAddressRange_v3020 range = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &found) != cudaSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<PFN_cuMemGetAddressRange_v3020>(f);
  }();
  CUdeviceptr base = 0;
  size_t size = 0;
  if (!range || range(&base, &size, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS) return false;
  return bytes <= size - (size_t)((uintptr_t)p - (uintptr_t)base);
}

// Copies the register arrays (of any memory) to dst, back to back, on the context's
// stream.  Arrays in this device's memory, 16-byte aligned, whole, and of 2^16 elements at
// most in total (larger ones are the copy engine's) are gathered by one kernel; the
// others go by copy calls, which refuse an array that ends before its register.
bool copy_register_arrays(Context* ctx, void* const* arrays, double2* dst, const char* what) {
  const int R = ctx->numReg;
  GatherDesc D;
  D.numReg = R;
  size_t total = 0;
  bool gather = R > 1;
  for (int r = 0; r < R; ++r) {
    total += (size_t)1 << ctx->q[r];
    gather = gather && total <= (size_t)1 << 16 && ((uintptr_t)arrays[r] & 15) == 0;
    if (!gather) continue;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, arrays[r]) != cudaSuccess) {
      cudaGetLastError();
      gather = false;
    } else {
      gather = a.type == cudaMemoryTypeDevice && a.device == ctx->device &&
               in_one_allocation(arrays[r], sizeof(double2) << ctx->q[r]);
    }
    D.src[r] = (const double2*)arrays[r];
    D.end[r] = (unsigned)total;
  }
  if (gather) {
    {
      LaunchScope _ls(ctx, kKTable);  // (small inputs of a flush, like its tables)
      k_gather_arrays<<<grid_for(total, 256, 1), 256, 0, ctx->stream>>>(D, dst);
    }
    return cuda_ok(ctx, cudaGetLastError(), what);
  }
  size_t off = 0;
  for (int r = 0; r < R; ++r) {
    const size_t N = (size_t)1 << ctx->q[r];
    if (!cuda_ok(ctx, cudaMemcpyAsync(dst + off, arrays[r], N * sizeof(double2), cudaMemcpyDefault, ctx->stream), what))
      return false;
    off += N;
  }
  return true;
}

static InitDesc init_desc(Context* ctx, const double2* const* regArrays) {
  int R = ctx->numReg;
  int qLast = ctx->q[R - 1];
  InitDesc D{};
  D.numReg = R;
  D.qLast = qLast;
  for (int r = 0; r < R; ++r) {
    D.arr[r] = regArrays[r];
    D.shift[r] = ctx->flw[r] - qLast;
    D.mask[r] = (1 << ctx->q[r]) - 1;
  }
  return D;
}

bool launch_outer(Context* ctx, const double2* const* regArrays, double2* outer) {
  int R = ctx->numReg;
  const uint64_t nOuter = 1ull << (ctx->totalQbt - ctx->q[R - 1]);
  if (R >= 2) {
    const InitDesc D = init_desc(ctx, regArrays);
    return enqueue(ctx, kKInit, "outer launch", [=] {
      k_init_outer<<<grid_for(nOuter, 256, 1), 256, 0, ctx->stream>>>(D, outer, nOuter);
      return cudaGetLastError();
    });
  }
  static const double2 one = {1.0, 0.0};
  return enqueue(ctx, -1, "outer copy", [=] {
    return cudaMemcpyAsync(outer, &one, sizeof(one), cudaMemcpyHostToDevice, ctx->stream);
  });
}

bool launch_init_product(Context* ctx, const double2* const* regArrays) {
  // regArrays: device pointers to our own copies, one per register
  const int R = ctx->numReg, qLast = ctx->q[R - 1];
  const uint64_t nOuter = 1ull << (ctx->totalQbt - qLast);
  double2* outer = (double2*)arena_alloc(ctx, nOuter * sizeof(double2));
  if (!outer) return false;
  if (!launch_outer(ctx, regArrays, outer)) return false;
  const uint64_t n = ctx->size();
  const int blocks = grid_for(n, 256, 4);
  const double2* last = regArrays[R - 1];
  void* st = ctx->state();
  return enqueue(ctx, kKInit, "init launch", [=] {
    if (ctx->precision == kC128)
      k_init_product<double2><<<blocks, 256, 0, ctx->stream>>>((double2*)st, n, qLast, last, outer);
    else
      k_init_product<float2><<<blocks, 256, 0, ctx->stream>>>((float2*)st, n, qLast, last, outer);
    return cudaGetLastError();
  });
}

}  // namespace cvdv
