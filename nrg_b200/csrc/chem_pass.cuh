// The analytic-Jacobian integrators' inner loop as passes of a warp (device
// code): the method, step control and event counts of chem_bdf.cuh, arranged
// for the GPU.
//
// One thread integrates one cell.  The loop body is one pass: every live lane
// of the warp evaluates one right-hand side and makes one corrector solve,
// whichever state its BDF step is in (first step, a new attempt after the
// predictor, a further corrector iteration, the same prediction with a fresh
// Jacobian).  A lane that repeats an attempt or iterates once more does so
// while the other lanes go on with their own next step, so the warp runs as
// many passes as its slowest cell has right-hand sides; the routine-by-routine
// form makes every lane wait for each retry and iteration of any other.
// The routines of a pass have one call site each and are inlined there, so that
// no call spills the cell's registers in every pass; out of line are the
// step-size ratios of the order choice (four uses, pass_ratio) and the table
// walks of decks without generated code.
//
// What bounds it, and where the state lives: with the Nordsieck array in
// shared memory a cell took 1,408 B there, so an SM held 4 warps, one per
// scheduler, and the kernel waited on dependent FP64 and shared-memory
// latency (issue slots 22 % used, FP64 pipe 19 %).  Here the Nordsieck array
// (6 N doubles; above 8 species part of it spills to the L1 cache) is in
// registers with compile-time column numbers: columns
// above a cell's order hold zeros, so lanes of different order run the same
// predictor, update and interpolation code (adding, scaling or multiplying
// zeros changes no value).  Shared memory keeps what is indexed at run time
// (the LU factors, whose pivot row varies) and what is read once per right-hand
// side (the rate constants, equal reactions merged): 880 B a cell of KEROMNES, 8
// warps on an SM at 252 registers.  What bounds it now is instruction issue
// (40 % of the slots at two warps per scheduler, FP64 pipe 39 %) and instruction
// fetch: the loop is about 4,000 instructions, so the warps of a block go through
// it in lockstep (k_chem_pass).  2048 x 2048 flame 72.0 -> 28.6 ms, 512 x 512
// ignition field 79.7 -> 16.1 ms, 64 x 64 random cells 2.49 -> 1.10 ms; a flame of
// 512 x 384 cells with the larger mechanisms: TEREZA 21.6 -> 8.3 ms, KONNOV 42.3
// -> 21.1 ms, ACETYLENE 30.9 -> 25.9 ms.
#pragma once

#include "chem_bdf.cuh"
#include "tc_sm100.cuh"

namespace nrg {

// Whether U's columns are multiplied by their pivots' reciprocals (pass_solve):
// not for float factors, where it would round each of them once more.
template <typename LUT>
constexpr bool kScaledU = std::is_same<LUT, double>::value;

// Slots of rate constants a cell keeps: the distinct reactions of the generated
// code, all of them in table-driven kernels.
template <int R, int SPEC>
struct RateSlots {
  static constexpr int value = SpecOf<SPEC>::kR;
};
template <int R>
struct RateSlots<R, 0> {
  static constexpr int value = R;
};

// Shared-memory arrays of a warp's cells, [element][lane].  The LU storage doubles
// as the scratch of the cells' set-up (with float factors the scratch of a
// lane covers factors of other lanes, but of no other warp); TAB: the
// table-driven right-hand side also indexes z and zd at run time and keeps its
// own copies.
//
// TM: the rate constants live in tensor memory instead, lane = cell, four
// 32-bit columns per reaction (k_f, k_r), next to the 227 KB of shared memory
// and of the same size.  They are what a cell of a larger mechanism has most
// of, and the right-hand side reads them in order, sixteen columns at a time.
// (Tensor memory is read and written by whole warps at warp-uniform columns,
// so nothing that a lane indexes on its own can go there.)
template <int N, int R, typename LUT, bool TAB, bool TM = false>
struct PassStore {
  static_assert(!(TAB && TM), "the table walk indexes the rate constants in shared memory");
  static constexpr int BS = 32;
  static constexpr bool kTM = TM;
  static constexpr int kRates = R;
  static constexpr int kSlots = TM ? 0 : R;  // in shared memory
  static constexpr int kTmCols = 4 * R <= 128 ? 128 : 4 * R <= 256 ? 256 : 512;
  static_assert(!TM || 4 * R <= 512, "tensor memory columns");
  static constexpr int kKF = 0;
  static constexpr int kKR = kSlots;
  static constexpr int kS = 2 * kSlots;          // permutation scratch / z
  static constexpr int kZD = kS + N;             // TAB only
  static constexpr int kDoubles = kS + (TAB ? 2 : 1) * N;
  static constexpr int kBytesPerThread = kDoubles * 8 + N * N * (int)sizeof(LUT);
  using lut_t = LUT;
  double* d;
  LUT* f;
  uint32_t tm;  // TM: the warp's lanes of column 0
  __device__ __forceinline__ void bind(char* smem, int tid) {
    smem += (size_t)(tid / BS) * BS * kBytesPerThread;
    d = reinterpret_cast<double*>(smem) + tid % BS;
    f = reinterpret_cast<LUT*>(smem + (size_t)kDoubles * 8 * BS) + tid % BS;
  }
  __device__ __forceinline__ double& kf(int r) const { return d[(kKF + r) * BS]; }
  __device__ __forceinline__ double& kr(int r) const { return d[(kKR + r) * BS]; }
  __device__ __forceinline__ double& s(int k) const { return d[(kS + k) * BS]; }
  __device__ __forceinline__ LUT& a(int j, int i) const { return f[(j * N + i) * BS]; }  // A(i+1, j+1)
};

// The store as rate_constants_fast sees it: z, zd and the rate constants of
// the reactions beyond the RS slots in the LU storage, which the integration
// does not use yet.
template <class S, int N, int RS>
struct SetupView {
  static constexpr int BS = S::BS;
  S st;
  double* lu;  // the lane's first element of the LU storage, as doubles
  __device__ __forceinline__ double& kf(int r) { return r < RS ? st.kf(r) : lu[(2 * N + 2 * (r - RS)) * BS]; }
  __device__ __forceinline__ double& kr(int r) { return r < RS ? st.kr(r) : lu[(2 * N + 2 * (r - RS) + 1) * BS]; }
  __device__ __forceinline__ double& z(int k) { return lu[k * BS]; }
  __device__ __forceinline__ double& zd(int k) { return lu[(N + k) * BS]; }
};

// The store as the generated right-hand side and matrix see it: z and zd in
// registers.
template <class S, int N>
struct RegView {
  const S& st;
  const double (&zin)[N];
  double (&out)[N];
  __device__ __forceinline__ double kf(int r) const { return st.kf(r); }
  __device__ __forceinline__ double kr(int r) const { return st.kr(r); }
  __device__ __forceinline__ double z(int k) const { return zin[k]; }
  __device__ __forceinline__ double& zd(int k) const { return out[k]; }
};

// RegView with the rate constants from tensor memory: four reactions in
// registers, the next four on their way.  The generated code asks for k_f then
// k_r of reactions 0, 1, 2, ...
template <class S, int N>
struct TmView {
  const S& st;
  const double (&zin)[N];
  double (&out)[N];
  uint32_t cur[16], nxt[16];
  __device__ __forceinline__ void start() { tc::tmem_ld16(st.tm, nxt); }
  __device__ __forceinline__ double kf(int r) {
    if ((r & 3) == 0) {
      tc::tmem_ld_wait(nxt);
#pragma unroll
      for (int i = 0; i < 16; ++i) cur[i] = nxt[i];
      if (r + 4 < S::kRates) tc::tmem_ld16(st.tm + 4 * (r + 4), nxt);
    }
    return __hiloint2double((int)cur[4 * (r & 3) + 1], (int)cur[4 * (r & 3)]);
  }
  __device__ __forceinline__ double kr(int r) const {
    return __hiloint2double((int)cur[4 * (r & 3) + 3], (int)cur[4 * (r & 3) + 2]);
  }
  __device__ __forceinline__ double z(int k) const { return zin[k]; }
  __device__ __forceinline__ double& zd(int k) const { return out[k]; }
};

// The store as the generated columns see it.  The rate constants are read
// again for each column (volatile): kept from one column to the next they
// would take the registers the Nordsieck array needs.
template <class S, int N>
struct ColumnView {
  const S& st;
  const double (&zin)[N];
  __device__ __forceinline__ double rate(int q) const {
    if constexpr (S::kTM) {
      uint32_t v[2];
      tc::tmem_ld2(st.tm + 2 * q, v);
      return __hiloint2double((int)v[1], (int)v[0]);
    } else {
      return *(const volatile double*)&((q & 1) ? st.kr(q >> 1) : st.kf(q >> 1));
    }
  }
  __device__ __forceinline__ double kf(int r) const { return rate(2 * r); }
  __device__ __forceinline__ double kr(int r) const { return rate(2 * r + 1); }
  __device__ __forceinline__ double z(int k) const { return zin[k]; }
};

// The store as the table-driven right-hand side and matrix see it.
template <class S, int N>
struct TabView {
  using lut_t = typename S::lut_t;
  const S& st;
  __device__ __forceinline__ double& kf(int r) { return st.kf(r); }
  __device__ __forceinline__ double& kr(int r) { return st.kr(r); }
  __device__ __forceinline__ double& z(int k) { return st.s(k); }
  __device__ __forceinline__ double& zd(int k) { return st.d[(S::kZD + k) * S::BS]; }
  __device__ __forceinline__ lut_t& a(int j, int i) { return st.a(j, i); }
};

// The table walks are functions of their own: inlined they had the registers the
// Nordsieck array leaves, and took 1.4 to 1.6 times as long (KONNOV, ACETYLENE).
template <int N, class S>
__device__ __noinline__ void pass_walk_rhs(double* d) {
  S st;
  st.d = d;
  st.f = nullptr;
  TabView<S, N> v{st};
  rhs<N>(v, c_mech.RM);
}

template <int N, int R, int SPEC, class S>
__device__ __forceinline__ void pass_rhs(const S& st, const double (&y)[N], double (&out)[N]) {
  if constexpr (SPEC != 0) {
    static_assert(N == SpecOf<SPEC>::kN, "specialised code is for another mechanism size");
    if constexpr (S::kTM) {
      TmView<S, N> v{st, y, out};
      __syncwarp();
      v.start();
      SpecOf<SPEC>::rhs(v);
    } else {
      RegView<S, N> v{st, y, out};
      SpecOf<SPEC>::rhs(v);
    }
  } else {
    TabView<S, N> v{st};
#pragma unroll
    for (int k = 0; k < N; ++k) v.z(k) = y[k];
    pass_walk_rhs<N, S>(st.d);
#pragma unroll
    for (int k = 0; k < N; ++k) out[k] = v.zd(k);
  }
}

// Column J of the iteration matrix and its elimination (left-looking): the
// generated column in registers, its rows in the order the earlier pivots gave
// them, the earlier multipliers applied, then the pivot search, interchange
// and scaling of dgefa.  Every element takes the operations of the
// right-looking dgefa<RECIP> in the same order, but the matrix never exists
// in memory before it is factored: 64 stores and 28 loads of elements instead
// of a store, a load and 3 to 4 updates of each.
// commit: the lane keeps the factors (with rates in tensor memory the whole warp
// goes through the columns).
template <int N, int SPEC, int J, class V, class S>
__device__ __forceinline__ void pass_factor_columns(const V& view, const S& st, double factor, RowPerm<N>& perm,
                                                    bool& ok, bool commit) {
  using LUT = typename S::lut_t;
  LUT v[N];
  // one column at a time: without this the loads of later columns are moved up
  // and 250 bytes of registers per thread spill
  asm volatile("" ::: "memory");
  if constexpr (S::kTM) __syncwarp();
  SpecOf<SPEC>::template column<J>(view, factor, v);
  if constexpr (J > 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) st.s(i) = (double)v[i];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = (LUT)st.s(perm.get(i));
#pragma unroll
    for (int k = 0; k < J; ++k)
#pragma unroll
      for (int i = k + 1; i < N; ++i) v[i] = lu_axpy<LUT, true>(v[i], v[k], *(const volatile LUT*)&st.a(k, i));
  }
  if constexpr (J < N - 1) {
    int l = J;
    LUT dmax = fabs(v[J]), piv = v[J];
#pragma unroll
    for (int i = J + 1; i < N; ++i)
      if (fabs(v[i]) > dmax) {
        l = i;
        dmax = fabs(v[i]);
        piv = v[i];
      }
    ok = ok && piv != (LUT)0;
    if (l != J) {
#pragma unroll
      for (int i = J + 1; i < N; ++i)
        if (i == l) v[i] = v[J];
      v[J] = piv;
      if (commit) {
#pragma unroll
        for (int k = 0; k < J; ++k) {
          const LUT m = st.a(k, l);
          st.a(k, l) = st.a(k, J);
          st.a(k, J) = m;
        }
      }
      const int pk = perm.get(J);
      perm.set(J, perm.get(l));
      perm.set(l, pk);
    }
    const LUT t = (LUT)-1 / v[J];
    v[J] = -t;
#pragma unroll
    for (int i = J + 1; i < N; ++i) v[i] = t * v[i];
  } else {
    ok = ok && v[J] != (LUT)0;
    v[J] = (LUT)1 / v[J];
  }
  if constexpr (kScaledU<LUT>) {
#pragma unroll
    for (int i = 0; i < J; ++i) v[i] = v[i] * v[J];
  }
  if (commit) {
#pragma unroll
    for (int i = 0; i < N; ++i) st.a(J, i) = v[i];
  }
  if constexpr (J + 1 < N) pass_factor_columns<N, SPEC, J + 1>(view, st, factor, perm, ok, commit);
}

// dgefa<RECIP> on the LU storage as two loops over columns (rows above the pivot
// get a zero multiplier, which changes nothing): the operations of
// pass_factor_columns in a tenth of its code.  A zero of the pivot row, where
// the species' reactions do not meet, leaves its column as it is.
template <int N, class S>
__device__ __forceinline__ bool pass_lu_loop(const S& st, RowPerm<N>& perm) {
  using LUT = typename S::lut_t;
  constexpr int BS = S::BS;
  bool ok = true;
  perm.identity();
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    LUT* ck = &st.a(k, 0);
    LUT c[N], piv = (LUT)0, ckk = (LUT)0, dmax = (LUT)-1;
    int l = k;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      c[i] = ck[i * BS];
      if (i == k) ckk = c[i];
      if (i >= k && fabs(c[i]) > dmax) {
        l = i;
        dmax = fabs(c[i]);
        piv = c[i];
      }
    }
    ok = ok && piv != (LUT)0;
    const LUT t = (LUT)-1 / piv;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const LUT u = c[i];
      c[i] = t * (i > k && i == l ? ckk : c[i]);
      ck[i * BS] = i > k ? c[i] : i < k ? (kScaledU<LUT> ? -c[i] : u) : -t;
      c[i] = i > k ? c[i] : (LUT)0;
    }
    const int pk = perm.get(k);
    perm.set(k, perm.get(l));
    perm.set(l, pk);
    LUT* cj = &st.a(0, 0);
#pragma unroll 1
    for (int j = 0; j < N; ++j, cj += N * BS) {
      if (j == k) continue;
      const LUT tj = cj[l * BS];
      cj[l * BS] = cj[k * BS];
      cj[k * BS] = tj;
      if (j > k && tj != (LUT)0) {
        constexpr int H = N / 2;  // rows 1..H-1 only while some lie below the pivot
        if (k < H - 1) {
#pragma unroll
          for (int i = 1; i < H; ++i) cj[i * BS] = lu_axpy<LUT, true>(cj[i * BS], tj, c[i]);
        }
#pragma unroll
        for (int i = H; i < N; ++i) cj[i * BS] = lu_axpy<LUT, true>(cj[i * BS], tj, c[i]);
      }
    }
  }
  return ok;
}

template <int N, class S>
__device__ __noinline__ bool pass_walk_factor(double* d, typename S::lut_t* f, double factor, RowPerm<N>* perm) {
  S st;
  st.d = d;
  st.f = f;
  TabView<S, N> v{st};
  analytic_iteration_matrix<N>(v, factor, c_mech.RM);
  RowPerm<N> p;
  const bool ok = pass_lu_loop<N>(st, p);
  *perm = p;
  return ok;
}

// Factors of I + factor * J(y); false when singular.
template <int N, int R, int SPEC, class S>
__device__ __forceinline__ bool pass_factor(const S& st, const double (&y)[N], double factor, RowPerm<N>& perm,
                                            bool commit) {
  if constexpr (SPEC != 0) {
    ColumnView<S, N> v{st, y};
    perm.identity();
    bool ok = true;
    pass_factor_columns<N, SPEC, 0>(v, st, factor, perm, ok, commit);
    return ok;
  } else {
    TabView<S, N> v{st};
#pragma unroll
    for (int k = 0; k < N; ++k) v.z(k) = y[k];
    RowPerm<N> p;
    const bool ok = pass_walk_factor<N, S>(st.d, st.f, factor, &p);
    perm = p;
    return ok;
  }
}

// Pascal-triangle predictor (sgn = 1) and its inverse (sgn = -1) on columns
// 0..Q of the register Nordsieck array: the additions of ddpsc.f90 in its
// order (a fused multiply by +-1 rounds as the addition does).  top: column Q
// is part of this lane's history (else, its order being lower, it holds the
// correction kept for the order choice and counts as zero).
template <int N, int Q>
__device__ __forceinline__ void pass_pascal(double (&yh)[kMaxOrd + 1][N], double sgn, bool top) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    double v[Q + 1];
#pragma unroll
    for (int j = 0; j < Q; ++j) v[j] = yh[j][i];
    v[Q] = (Q < kMaxOrd || top) ? yh[Q][i] : 0.0;
#pragma unroll
    for (int j1 = 1; j1 <= Q; ++j1)
#pragma unroll
      for (int j2 = j1; j2 <= Q; ++j2) {
        const int j = Q - j2 + j1;  // 1-based column
        v[j - 1] = fma(sgn, v[j], v[j - 1]);
      }
#pragma unroll
    for (int j = 0; j < Q; ++j) yh[j][i] = v[j];
  }
}

// The weighted norms' squares of two vectors with the same weights
// max(|y|, YWT), as weighted_norm forms them.  An error norm that overflows
// passes no test: the attempt fails, and the cell's tries are counted.
template <int N>
__device__ __forceinline__ void pass_norms2(const double (&x0)[N], const double (&x1)[N], const double (&y)[N],
                                            const double (&ywt)[N], double* n0, double* n1) {
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double w = NRG_FMAX(fabs(y[i]), ywt[i]);
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(w));
    r = fma(r, fma(-w, r, 1.0), r);
    const double q0 = x0[i] * r, q1 = x1[i] * r;
    s0 = fma(q0, q0, s0);
    s1 = fma(q1, q1, s1);
  }
  *n0 = s0;
  *n1 = s1;
}

// sqrt(x), x >= 0, for the convergence test: the hardware approximation of
// 1 / sqrt(x) and two Newton steps (0 below 1e-290; infinity and NaN stay).
__device__ __forceinline__ double pass_sqrt(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = r * fma(-0.5 * x * r, r, 1.5);
  r = r * fma(-0.5 * x * r, r, 1.5);
  return x < 1e-290 ? 0.0 : (x < 1.7e308 ? x * r : x);
}

// 1 / x for x > 0 in the step-size control: the hardware approximation and two
// Newton steps (x clamped to where they hold).
__device__ __forceinline__ double pass_rcp(double x) {
  const double w = NRG_FMIN(x, 1e300);
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(w));
  r = fma(r, fma(-w, r, 1.0), r);
  return fma(r, fma(-w, r, 1.0), r);
}

// The rate constants of a warp's cells from the set-up scratch (pass_begin) into
// tensor memory; all lanes.
template <int N, class S>
__device__ __forceinline__ void pass_rates_to_tm(const S& st) {
  const int lane = threadIdx.x % S::BS;
  SetupView<S, N, 0> v{st, reinterpret_cast<double*>(st.f - lane) + lane};
  __syncwarp();
#pragma unroll 4
  for (int r = 0; r < S::kRates; ++r) {
    const double f = v.kf(r), b = v.kr(r);
    tc::tmem_st4(st.tm + 4 * r, (uint32_t)__double2loint(f), (uint32_t)__double2hiint(f), (uint32_t)__double2loint(b),
                 (uint32_t)__double2hiint(b));
  }
  tc::tmem_st_wait();
}

// x^p, 0 < p < 1, for the step-size choices: 2^(p log2 x) with the logarithm's
// fraction and the power in single precision (relative error about 1e-6, as
// ratio_pow) over the whole range of x >= 0; NaN and infinity pass through.
__device__ __forceinline__ double pass_pow(double x, float p) {
  const int hi = __double2hiint(x);
  const int e = (hi >> 20) - 1023;
  const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));  // 2^-e x, in [1, 2)
  const float l2 = p * ((float)e + __log2f((float)m));
  const float fl = floorf(l2);
  const double r = (double)exp2f(l2 - fl) * __hiloint2double((int)(1023.0f + fl) << 20, 0);
  return x < 1.7e308 ? r : x;
}

// Corrector solve: the row permutation through the cell's scratch, then the two
// sweeps without tests for zero multipliers (adding a zero product changes
// nothing).  The factors hold the pivots' reciprocals on the diagonal and, in
// double, U's columns multiplied by them, so that the backward sweep is a chain
// of one fused multiply-add per row instead of a multiply and one.
template <int N, class S>
__device__ __forceinline__ void pass_solve(const S& st, const RowPerm<N>& piv, double (&b)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) st.s(i) = b[i];
#pragma unroll
  for (int i = 0; i < N; ++i) b[i] = st.s(piv.get(i));
#pragma unroll
  for (int k = 0; k < N - 1; ++k)
#pragma unroll
    for (int i = k + 1; i < N; ++i) b[i] = b[i] + b[k] * (double)st.a(k, i);
  constexpr bool kScaled = kScaledU<typename S::lut_t>;
#pragma unroll
  for (int k = N - 1; k >= 0; --k) {
    if constexpr (!kScaled) b[k] = b[k] * (double)st.a(k, k);
#pragma unroll
    for (int i = 0; i < k; ++i) b[i] = b[i] - b[k] * (double)st.a(k, i);
  }
  if constexpr (kScaled) {
#pragma unroll
    for (int k = 0; k < N; ++k) b[k] = b[k] * (double)st.a(k, k);
  }
}

// The state a finished cell hands to cell_finish.
template <int N, int NF>
struct PassResult {
  static constexpr int kNF = NF;
  double y[N];
  double tout;
};

// Set-up of a cell (cell_begin's part before the integrator's scalars): the
// skip rule, third-body sums and rate constants; concentrations into y.
// False when the cell is passed through (its outputs already written).
template <int N, int R, int NF, class S>
__device__ __forceinline__ bool pass_begin(const S& st, const StepArgs& a, long cid, double (&y)[N]) {
  const double Tc = a.T[cid];
  if (!reference_cell_active(Tc, a.bc, cid)) {
    write_skipped_cell(a, cid, NF, Tc);
    return false;
  }
  const double rho = a.rho[cid];
  double conc[NF];
#pragma unroll
  for (int k = 0; k < NF; ++k) conc[k] = a.Y[k * a.ld + cid] * rho / c_mech.W[k];
  constexpr int RS = S::kSlots;  // none with rates in tensor memory: pass_rates_to_tm moves them there
  static_assert(2 * N + 2 * (R - RS) <= N * N * (int)sizeof(typename S::lut_t) / 8, "set-up scratch");
  const int lane = threadIdx.x % S::BS;
  SetupView<S, N, RS> v{st, reinterpret_cast<double*>(st.f - lane) + lane};
#pragma unroll 1
  for (int r = 0; r < R; ++r) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < NF; ++k) s = s + conc[k] * c_mech.eff_t[k][r];
    v.kr(r) = s;  // third-body sum, consumed by rate_constants_fast
  }
  rate_constants_fast<N, R>(v, Tc);
  for (int r = c_mech.RM; r < R; ++r) {
    const int m = c_mech.m_of[r];
    v.kf(m) += v.kf(r);
    v.kr(m) += v.kr(r);
  }
  // mechanism order to integrated order (the inert species drop out); the
  // index is a table read, so through the scratch unless nothing drops out
  if constexpr (NF == N) {
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = conc[k];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int k = c_mech.full_of[i];
      y[i] = conc[0];
#pragma unroll
      for (int q = 1; q < NF; ++q)
        if (q == k) y[i] = conc[q];
    }
  }
  return true;
}

// Step-size ratio 1 / max(lo, bias * e2^(p/2)) of a squared error ratio e2.
static __device__ __noinline__ double pass_ratio(double e2, float p, double bias, double lo) {
  return pass_rcp(NRG_FMAX(lo, bias * pass_pow(e2, 0.5f * p)));
}

// Lanes of the warp (LOCK: threads of the block) for which p holds.
template <bool LOCK>
__device__ __forceinline__ int pass_count(bool p) {
  if constexpr (LOCK) return __syncthreads_count(p);
  else return __popc(__ballot_sync(0xffffffffu, p));
}

// Integrates the lanes' cells (live: the lane has one; y: its concentrations
// in and out) to tout.  All lanes of the warp take part, LOCK: all threads of the
// block.  Returns the cell's CellStatus.
template <int N, int R, int NF, int SPEC, bool LOCK, class S>
__device__ __forceinline__ int pass_integrate(const S& st, const StepArgs& a, bool live, double tout, double (&y)[N],
                                              unsigned long long* cnt) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr double BIAS1 = 1.3, BIAS2 = 1.2, BIAS3 = 1.4, RCTEST = 0.3, RMFAIL = 2.0, RMNORM = 10.0, TRSHLD = 1.0;
  constexpr int MXFAIL = 3, MXITER = 3, MXTRY = 50, NDJSTP = 10;
  constexpr double kInvSqrtNF = 1.0 / ct_sqrt((double)NF);
  const double uround = c_mech.uround, ewt = c_mech.ewt;
  const double eps = a.eps > 0.0 ? a.eps : c_mech.eps;
  const double inv_eps2 = 1.0 / (eps * eps * (double)NF);  // of the squared, unscaled error norms
  // what the lane does in its next pass: the first right-hand side (DDNTL), a
  // new attempt, a further corrector iteration, the same prediction with a
  // fresh Jacobian, waiting for that Jacobian, taking a failed attempt back,
  // the last scaling before the interpolation to tout
  enum { kInit = 0, kPredict, kIterate, kRedo, kWait, kUndo, kFinish };
  double yh[kMaxOrd + 1][N], s1[N], ywt[N];
  RowPerm<N> piv;
  piv.identity();
  double t = 0.0, rc = 0.0, rmax = 10000.0, trend = 1.0, d1 = 0.0, rh = 0.0;
  double h = tout * (1.0 - 4.0 * uround);
  h = copysign(NRG_FMIN(fabs(h), c_mech.hmax), h);
  int nq = 1, nwait = 3, jtask = 0, nstep = 0, jstepl = 0, ntry = 0, nfail = 0, iter = 0, phase = kInit;
  int nfe = 0, nje = 0, nsolve = 0, status = kCellOk;
  int order = 0;  // pending change of the order, with the pending factor rh of the step
  bool scale = false, fresh = false, accepted = false;
  bool convrg = false, ier = false, evaljc = false, done = false;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    yh[0][i] = y[i];
    ywt[i] = NRG_FMAX(ewt, fabs(y[i]));
    s1[i] = 0.0;
#pragma unroll
    for (int j = 1; j <= kMaxOrd; ++j) yh[j][i] = 0.0;
  }
  // ddriv3.f90:1304-1316 (see cell_advance): a tolerance below the rounding
  // unit returns the state as it is
  bool run = live && !(eps < uround);
  if (run && a.mxstep == 0) {
    status = kCellMxstep;
    run = false;
  }

  for (;;) {
    const int nrun = pass_count<LOCK>(run);
    if (nrun == 0) break;
    // ---- the pending change of order and step (DDSCL)
    if (run && scale && (phase == kPredict || phase == kFinish)) {
      scale = false;
      if (!accepted && rh * h == 0.0) {
        status = kCellFatal;  // the step size vanished
        run = false;
      } else {
        if (order != 0) {
          // the column that leaves becomes zero, the one that joins is s1 el / (nq + 1)
          const int jt = order < 0 ? nq : nq + 1;
          const double e = order < 0 ? 0.0 : EL(nq + 1, nq) * pass_rcp((double)(nq + 1));
#pragma unroll
          for (int j = 2; j <= kMaxOrd; ++j)
            if (j == jt) {
#pragma unroll
              for (int i = 0; i < N; ++i) yh[j][i] = s1[i] * e;
            }
          rc = rc * EL(1, nq + order) * pass_rcp(EL(1, nq));
          nq += order;
          order = 0;
        }
        if (fresh) nwait = nq + 2;
        // |h| <= hmax = 1e-7 here: DDSCL's branch for |h| < 1
        const double ah = fabs(h);
        rh = NRG_FMIN(NRG_FMIN(ah * rh, ah * rmax), c_mech.hmax) * pass_rcp(ah);
        double r1 = 1.0;
#pragma unroll
        for (int j = 1; j <= kMaxOrd; ++j) {
          r1 = r1 * rh;
#pragma unroll
          for (int i = 0; i < N; ++i) yh[j][i] = yh[j][i] * r1;
        }
        h = h * rh;
        rc = rc * rh;
        if (accepted && fresh) rmax = RMNORM;
      }
    }
    if (phase == kFinish && run) {
      run = false;
      done = true;
    }

    // ---- a new attempt: DDPSC, and whether the Jacobian is due; or an attempt
    // taken back
    const bool undo = run && phase == kUndo;
    bool pred = run && phase == kPredict;
    if (pred) {
      ntry += 1;
      iter = 0;
      evaljc = (fabs(rc - 1.0) > RCTEST) || (nstep >= jstepl + NDJSTP);
      if (ntry > MXTRY) {
        status = kCellFatal;
        run = false;
        pred = false;
      }
    }
    const int qp = __reduce_max_sync(kAll, pred || undo ? nq : 0);
    if (pred || undo) {
      const double sgn = undo ? -1.0 : 1.0;
      if (qp <= 3) pass_pascal<N, 3>(yh, sgn, true);
      else if (qp == 4) pass_pascal<N, 4>(yh, sgn, true);
      else pass_pascal<N, 5>(yh, sgn, nq == kMaxOrd);
    }
    if (phase != kIterate) {
#pragma unroll
      for (int i = 0; i < N; ++i) s1[i] = 0.0;
    }

    // ---- iteration matrix and its factors (DDPST) where due.  They cost more
    // than the rest of a pass, so they are made when half of the live lanes
    // (of the warp, or of the block in lockstep) wait for theirs; a waiting
    // lane sits passes out.  The lanes' own sequences do not change.  Table
    // walks: two thirds (196,608 random cells, KONNOV: half 255 ms, two thirds
    // 244, all 319 before the walk read ahead; ACETYLENE 122.5 and 119.8 ms).
    const bool due = run && (pred || phase == kRedo || phase == kWait) && (evaljc || ier);
    const bool make = (SPEC == 0 ? 3 : 4) * pass_count<LOCK>(due) >= 2 * nrun;
    const bool need = due && make;
    if (due) phase = make ? kPredict : kWait;
    const double jac_factor = -(EL(1, nq) * h);
    RowPerm<N> made;
    bool factored = false;
    if constexpr (S::kTM) {
      if (__any_sync(kAll, need)) factored = pass_factor<N, R, SPEC>(st, yh[0], jac_factor, made, need);
    }
    if (need) {
      nje += 1;
      if constexpr (S::kTM) piv = made;
      else factored = pass_factor<N, R, SPEC>(st, yh[0], jac_factor, piv, true);
      ier = !factored;
      if (!ier) {
        convrg = false;
        rc = 1.0;
        jstepl = nstep;
      }
    }
    const bool singular = need && ier;
    const bool go = run && phase != kWait && !undo;
    const double el1 = EL(1, nq);
#pragma unroll
    for (int i = 0; i < N; ++i) y[i] = yh[0][i] + el1 * s1[i];

    // ---- right-hand side
    double s2[N];
    pass_rhs<N, R, SPEC>(st, y, s2);
    nfe += go ? 1 : 0;

    // ---- corrector solve and the norms of the corrections; the first right-hand
    // side and restarts (DDNTL) take the norm of dy/dt with weights max(1, YWT)
    const bool first = go && phase == kInit;
    bool fail = singular, conv = false;
    double ctest = 0.0, e2 = 0.0;  // e2: the squared ratio of the error estimate to eps
    if (go && !singular) {
      double x[N], d, unit = 1.0;
      if (first) {
        // the squares of rates above 1e134 (densities far beyond any gas) are kept
        // in range by a power of two
        bool big = false;
#pragma unroll
        for (int i = 0; i < N; ++i) big = big || (__double2hiint(s2[i]) & 0x7fffffff) >= (1023 + 448) << 20;
        unit = big ? 0x1p-448 : 1.0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          x[i] = s2[i] * unit;
          y[i] = 1.0;
        }
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = h * s2[i] - yh[1][i] - s1[i];
        pass_solve<N>(st, piv, x);
        nsolve += 1;
#pragma unroll
        for (int i = 0; i < N; ++i) s1[i] = s1[i] + x[i];
      }
      pass_norms2<N>(x, s1, y, ywt, &d, &e2);
      d = pass_sqrt(d) * kInvSqrtNF;
      if (first) {
        if (jtask == 0) rmax = 10000.0;
        if (jtask == 2) rmax = RMNORM;
        rc = 0.0;
        convrg = false;
        ier = false;
        trend = 1.0;
        nq = 1;
        nwait = 3;
        // d is in units of 1 / unit; an infinite one (infinite rates) leaves a step
        // whose attempts show it
        const double hd = NRG_FMAX(eps * pass_rcp(d) * unit, 1e-309);
        if (hd < fabs(h)) h = copysign(hd, h);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          yh[1][i] = h * s2[i];
#pragma unroll
          for (int j = 2; j <= kMaxOrd; ++j) yh[j][i] = 0.0;
        }
        if (h == 0.0) {
          status = kCellFatal;
          run = false;
        }
        phase = kPredict;
      } else {
        // convergence test (DDCOR)
        e2 = e2 * (c_mech.itq2[nq][1] * inv_eps2);
        if (iter > 0) trend = NRG_FMAX(0.9 * trend, d * pass_rcp(d1));
        d1 = d;
        ctest = NRG_FMIN(2.0 * trend, 1.0) * d;
        conv = ctest <= eps;
        if (conv) {
          convrg = true;
        } else {
          iter += 1;
          if (iter < MXITER) {
            phase = kIterate;
          } else if (convrg) {
            evaljc = true;
            iter = 0;
            phase = kRedo;
          } else {
            fail = true;
          }
        }
      }
    }
    const bool reject = conv && e2 > 1.0;
    const bool accept = conv && !reject;
    bool norms = reject;
    if (fail) {
      nwait = nq + 2;
      if (jtask == 1) rmax = RMFAIL;
      rh = iter == 0 ? 0.3 : 0.9 * pass_pow(eps * pass_rcp(ctest), 0.2f);
      scale = true;
      fresh = false;
      accepted = false;
      phase = kUndo;
    }
    if (reject) {
      nfail += 1;
      phase = kUndo;
      if (nfail < MXFAIL || nq == 1) {
        if (jtask == 1) rmax = RMFAIL;
      } else {
        nfail = 0;
        jtask = 2;
        norms = false;
      }
    }
    if (accept) {
      nstep += 1;
      t = t + h;
#pragma unroll
      for (int j = 0; j <= kMaxOrd; ++j) {
        const double e = EL(j + 1, nq);  // zero above the order
#pragma unroll
        for (int i = 0; i < N; ++i) yh[j][i] = yh[j][i] + e * s1[i];
      }
#pragma unroll
      for (int i = 0; i < N; ++i) y[i] = yh[0][i];
      ntry = 0;
      nfail = 0;
      phase = kPredict;
      if (jtask != 1) {
        rh = pass_ratio(e2, __fdividef(1.0f, (float)(nq + 1)), BIAS2, uround);
        scale = rh > TRSHLD;
        fresh = false;
        accepted = true;
        jtask = 1;
      } else if (nwait > 1) {
        nwait -= 1;
        if (nwait == 1 && nq < kMaxOrd) {
#pragma unroll
          for (int i = 0; i < N; ++i) yh[kMaxOrd][i] = s1[i];
        }
      } else {
        norms = true;
      }
    }

    // ---- order and step size (accepted step with a full history, or the
    // rejected attempt's smaller step); applied at the next attempt
    if (norms) {
      double v[N], u[N], dn, up;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        v[i] = yh[2][i];
#pragma unroll
        for (int j = 3; j <= kMaxOrd; ++j)
          if (j == nq) v[i] = yh[j][i];
        u[i] = s1[i] - yh[kMaxOrd][i];
      }
      pass_norms2<N>(v, u, y, ywt, &dn, &up);
      const float fq = (float)nq;
      const double lo = reject ? 1.0 : uround;
      const double r1 = pass_ratio(dn * (c_mech.itq2[nq][0] * inv_eps2), __fdividef(1.0f, fq), BIAS1, lo);
      const double r3 = pass_ratio(up * (c_mech.itq2[nq][2] * inv_eps2), __fdividef(1.0f, fq + 2.0f), BIAS3, uround);
      const double rh1 = nq > 1 ? r1 : 0.0;
      const double rh2 = pass_ratio(e2, __fdividef(1.0f, fq + 1.0f), BIAS2, uround);
      const double rh3 = !reject && nq < kMaxOrd ? r3 : 0.0;
      scale = true;
      fresh = true;
      accepted = accept;
      if (rh1 > rh2 && rh1 >= rh3) {
        rh = rh1;
        order = -1;
      } else if (reject || (rh2 >= rh1 && rh2 >= rh3)) {
        rh = rh2;
        order = 0;
      } else {
        rh = rh3;
        order = 1;
      }
      if (accept && rh <= TRSHLD) {
        scale = false;
        order = 0;
        nwait = nq + 2;
      }
    }

    // ---- after an accepted step: the end of the interval, or new weights
    if (accept) {
      if (!(t < tout)) {
        phase = kFinish;
        run = scale;
        done = !scale;
      } else {
        if (nstep == a.mxstep) {
          status = kCellMxstep;
          run = false;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) ywt[i] = NRG_FMAX(ewt, fabs(yh[0][i]));
      }
    }
    if (undo) phase = scale ? kPredict : kInit;  // no step choice pending: the restart of DDNTL
  }
#pragma unroll
  for (int i = 0; i < N; ++i) y[i] = yh[0][i];
  if (done) {  // DDNTP: interpolation to tout (the columns above the order are zero)
    const double r = (tout - t) / h;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      y[i] = nq == kMaxOrd ? yh[kMaxOrd][i] : 0.0;
#pragma unroll
      for (int j = kMaxOrd - 1; j >= 0; --j) y[i] = yh[j][i] + r * y[i];
    }
  }
  cnt[1] += nstep;
  cnt[2] += nfe;
  cnt[3] += nje;
  cnt[4] += nsolve;
  return status;
}

}  // namespace nrg
