// Field-aligned heat diffusion with the reference's own band solve (multifluid.f90:309-342,
// collisions.f90:162-199, diffusion.f90:24-152, PDEparabolic.f90:19-346).
//
// One (x1 column, species) per thread.  The thread walks its column along x1 and, for each
// row, forms the thermal conductivity (thermal_conduct), the diffusion coefficients
// (diffusion_prep) and the TRBDF2 / backward-Euler band row in registers, with the
// reference's operation order.  Each band system is then factored and solved exactly as
// the reference's gbsv call does it (PDEparabolic.f90:142,216,337 -> gbsv.in.f90:90 ->
// LAPACK dgbsv with kl = ku = 2: dgbtrf -> dgbtf2, then dgbtrs -> dtbsv), specialised to
// the tridiagonal matrices the reference stores in that band:
//
//   dgbtf2 step j (rows j and j+1 are the only pivot candidates: row j+2 holds a structural
//   zero in column j, so its multiplier is 0 and its updates add zeros):
//     current row j = (p, q) in columns (j, j+1); original row j+1 = (s, d, e | r).
//     IDAMAX picks row j+1 only when |s| > |p| (ties keep row j).
//     no interchange: U(j) = (p, q, 0), recip = 1/p, m = recip*s (DSCAL), DGER:
//                     p' = d - m*q, q' = e;            dgbtrs: y(j) = b, b' = r - m*b
//     interchange:    U(j) = (s, d, e), recip = 1/s, m = recip*p, DGER:
//                     p' = q - m*d, q' = 0 - m*e;      dgbtrs: y(j) = r, b' = b - m*r
//   dtbsv (upper, no transpose, non-unit, bandwidth kl+ku), columns from the last:
//     x(i) = ((y(i) - x(i+2)*U(i,i+2)) - x(i+1)*U(i,i+1)) / U(i,i)
//   (the products with the zero fill entries U(i,i+3), U(i,i+4) subtract zeros).
// Every division is an IEEE division (or the exact reciprocal-corrected one for grid
// divisors), nothing is contracted, so the solution equals, bit for bit, the reference
// arithmetic with reference-BLAS semantics for IDAMAX/DSWAP/DSCAL/DGER/DTBSV.  The only
// departure: T**2.5 is the correctly rounded value (pow25), where the reference calls the
// C library's pow, which is not correctly rounded for about 1 argument in 1200.
//
// The forward elimination runs while the rows are formed.  It keeps no factor row: a row's
// conduction factors and right-hand side go to a per-thread scratch (the warp's 32 threads
// interleaved, so every scratch access is one coalesced 256-byte line), and the elimination
// state (p, q, b) is checkpointed every LU_K rows.  The back substitution walks the chunks
// of LU_K rows from the last one, repeats a chunk's elimination from its checkpoint (the same
// operations on the same values, so the same bits), holds the chunk's factor rows in
// registers and substitutes.  Storing the factor rows instead (U(i,i), U(i,i+1), U(i,i+2),
// y(i) written and read back in both stages) moved 28 doubles per row and species, this
// 21.  The reciprocal of the pivot, which the elimination needs, also serves the
// substitution's exact quotient x/U(i,i).
//
// The body is written once for a column accessor, so the same code runs on the device
// (thread per column) and, compiled for the host, over every column on a CPU.
#pragma once

#ifdef __CUDACC__
#define GEMD_HD __host__ __device__ __forceinline__
#else
#define GEMD_HD inline
#include <cmath>
#include <cstring>
#endif

namespace gemd {

constexpr int NSP = 7;
constexpr double KB = 1.38064852e-23;     // phys_consts.in.f90:24
constexpr double ELCHRG = 1.60217662e-19;  // phys_consts.in.f90:25
constexpr double MINDENSDIV = 1.0e-5;      // phys_consts.in.f90:84

GEMD_HD double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

GEMD_HD unsigned hi_abs(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(x) & 0x7fffffffu;
#else
  unsigned long long u;
  std::memcpy(&u, &x, 8);
  return (unsigned)(u >> 32) & 0x7fffffffu;
#endif
}

GEMD_HD double sqrt_rn(double x) {
#ifdef __CUDA_ARCH__
  return sqrt(x);
#else
  return std::sqrt(x);
#endif
}

#ifdef __CUDA_ARCH__
__device__ __noinline__ double div_rn_slow(double a, double b) { return a / b; }
#else
inline double div_rn_slow(double a, double b) { return a / b; }
#endif

// a/b for a divisor with a precomputed correctly rounded reciprocal y = RN(1/b): q0 = RN(a*y),
// one exact remainder r = a - b*q0 and q = RN(q0 + r*y), which is the IEEE quotient RN(a/b)
// whenever |a| is in (2^-500, 2^500) and |y| in [2^-400, 2^400] (Markstein); a zero numerator
// gives the correctly signed zero; anything else takes the IEEE division.
GEMD_HD double qdiv(double a, double b, double y) {
  const double q0 = a * y;
  const double r = fma_rn(-q0, b, a);
  const double q1 = fma_rn(r, y, q0);
  const unsigned ha = hi_abs(a), hy = hi_abs(y);
  if ((ha - (523u << 20) < (1000u << 20)) & (hy - (623u << 20) < (800u << 20))) return q1;
  if (a == 0.0 && (hy - (623u << 20) < (800u << 20))) return q0;
  return div_rn_slow(a, b);
}

// qdiv for a divisor whose reciprocal comes from a grid table: gem_grid_create rejects grids
// with a tabulated reciprocal outside [2^-400, 2^400], so only the numerator is range-checked.
GEMD_HD double qdiv_t(double a, double b, double y) {
  const double q0 = a * y;
  const double r = fma_rn(-q0, b, a);
  const double q1 = fma_rn(r, y, q0);
  if (hi_abs(a) - (523u << 20) < (1000u << 20)) return q1;
  if (a == 0.0) return q0;
  return div_rn_slow(a, b);
}

// The same quotients without their fallback: ok is cleared when a needs it.  A group of
// quotients then shares one branch to a slow path that forms them all again with qdiv: a
// branch per quotient costs four or five instructions and splits the code the compiler can
// interleave.  The remainder is formed negated, r = b*q0 - a, so that a zero numerator's
// quotient keeps its sign; zeros still take the slow path, except in qtry_z.
GEMD_HD double qtry_t(double a, double b, double y, bool& ok) {
  const double q0 = a * y;
  const double r = fma_rn(q0, b, -a);
  ok = ok & (hi_abs(a) - (523u << 20) < (1000u << 20));
  return fma_rn(-r, y, q0);
}
GEMD_HD double qtry_z(double a, double b, double y, bool& ok) {
  const double q0 = a * y;
  const double r = fma_rn(q0, b, -a);
  ok = ok & ((hi_abs(a) - (523u << 20) < (1000u << 20)) | (a == 0.0));
  return fma_rn(-r, y, q0);
}
// y is not from a grid table
GEMD_HD double qtry(double a, double b, double y, bool& ok) {
  ok = ok & (hi_abs(y) - (623u << 20) < (800u << 20));
  return qtry_t(a, b, y, ok);
}

GEMD_HD double fmax_f(double a, double b) { return (a > b) ? a : b; }
GEMD_HD double fabs_f(double a) { return (a < 0.0) ? -a : a; }

// 1/sqrt(x) to about an ulp
GEMD_HD double rsqrt_approx(double x) {
#ifdef __CUDA_ARCH__
  return rsqrt(x);
#else
  return 1.0 / std::sqrt(x);
#endif
}

// x**2.5 as x*x*sqrt(x) in double-double (fma for the exact product errors), rounded once:
// the correctly rounded value except in vanishingly rare near-halfway cases.  The root is
// s + sl with s = x*r, r = 1/sqrt(x) to an ulp or two, and sl = (x - s*s)*r/2 its remainder,
// so it needs neither a correctly rounded square root nor a division.
GEMD_HD double pow25_pos(double x) {
  const double rh = rsqrt_approx(x);
  const double s = x * rh;
  const double es = fma_rn(-s, s, x);
  const double sl = es * (0.5 * rh);
  const double x2 = x * x;
  const double x2l = fma_rn(x, x, -x2);
  const double p = x2 * s;
  const double pl = fma_rn(x2, s, -p);
  return p + (pl + (x2 * sl + x2l * s));
}
GEMD_HD double pow25(double x) {
  if (x > 0.0) return pow25_pos(x);
#ifdef __CUDA_ARCH__
  return pow(x, 2.5);
#else
  return std::pow(x, 2.5);
#endif
}

// Per-column constants of one solve.
struct LuK {
  int n;          // lx1
  int s;          // species (6 = electrons)
  double dt;
  double tmin, tmax;  // Dirichlet values of rows 1 and lx1 (diffusion.f90:54-79)
  double c0;          // (gamma_s - 1)/kB
  double tcoef;       // ions: thermal_coeff(s) (collisions.f90:51-53)
};

// Correctly rounded 1/x (the reference's ONE / AB(KV+1,J) in DSCAL).
GEMD_HD double rcp_rn(double x) {
#ifdef __CUDA_ARCH__
  return __drcp_rn(x);
#else
  return 1.0 / x;
#endif
}

// The streaming inputs of one interior cell: state values and, for the electrons, the
// neutral densities and J1, these loaded two cells ahead of use (the metric factors, small
// tables that the warp's lanes share, are read when the coefficients are formed).
struct CellIn {
  double T, n, n1, n2, n3, j1;
};

// thermal_conduct + diffusion_prep of interior cell i (collisions.f90:162-199,
// diffusion.f90:24-52; A = E = 0): C = (gamma-1)/kB / max(n,1e-5) / (h1 h2 h3),
// D = lambda h2 h3 / h1, B = C beta / h1 (electrons; 0 for the ions).
struct Coef {
  double C, D, B;
};
struct Metric {
  double h1, h2, h3, yh1, ha1, yha1;
};
// any input; the fast form below takes what is in range
template <bool ELEC>
#ifdef __CUDACC__
__host__ __device__ __noinline__
#endif
Coef cell_coef_any(double c0, double tcoef, CellIn c, Metric m) {
  const double T = c.T;
  const double T25 = pow25(T);
  double lam, Bc = 0.0;
  if (!ELEC) {
    lam = tcoef * T25;
  } else {
    const double sq = sqrt_rn(T);
    const double X = c.n1 * 1.1e-16 * (1 + 5.7e-4 * T) + c.n2 * 2.82e-17 * sq * (1 - 1.21e-4 * T) +
                     c.n3 * 2.2e-16 * (1 + 3.6e-2 * sq);
    lam = ELCHRG * 100 * 7.7e5 * T25 / (1 + 3.22e4 * (T * T) / c.n * X);
    Bc = 5.0 / 2 * KB / ELCHRG * c.j1;  // beta (collisions.f90:197)
  }
  Coef f;
  f.C = qdiv_t(c0 / fmax_f(c.n, MINDENSDIV), m.ha1, m.yha1);
  f.D = qdiv_t(lam * m.h2 * m.h3, m.h1, m.yh1);
  f.B = ELEC ? qdiv_t(f.C * Bc, m.h1, m.yh1) : 0.0;
  return f;
}

template <bool UNIT, bool ELEC, class Acc>
GEMD_HD Coef cell_coef(const Acc& a, const LuK& k, int i, const CellIn& c) {
  Metric m{1.0, 1.0, 1.0, 1.0, 1.0, 1.0};
  if (!UNIT) a.metrics(i, m.h1, m.h2, m.h3, m.yh1, m.ha1, m.yha1);
  const double T = c.T;
  // the power and the densities' quotients need a positive, normal T
  bool ok = hi_abs(T) - (523u << 20) < (1000u << 20) && T > 0.0;
  const double T25 = pow25_pos(T);
  double lam, Bc = 0.0;
  if (!ELEC) {
    lam = k.tcoef * T25;
  } else {
    const double sq = sqrt_rn(T);
    const double X = c.n1 * 1.1e-16 * (1 + 5.7e-4 * T) + c.n2 * 2.82e-17 * sq * (1 - 1.21e-4 * T) +
                     c.n3 * 2.2e-16 * (1 + 3.6e-2 * sq);
    lam = ELCHRG * 100 * 7.7e5 * T25 / (1 + 3.22e4 * (T * T) / c.n * X);
    Bc = 5.0 / 2 * KB / ELCHRG * c.j1;
  }
  const double nd = fmax_f(c.n, MINDENSDIV);
  const double g = qtry(k.c0, nd, rcp_rn(nd), ok);
  Coef f;
  f.C = UNIT ? g : qtry_t(g, m.ha1, m.yha1, ok);
  f.D = UNIT ? lam : qtry_t(lam * m.h2 * m.h3, m.h1, m.yh1, ok);
  f.B = ELEC ? (UNIT ? f.C * Bc : qtry_z(f.C * Bc, m.h1, m.yh1, ok)) : 0.0;
  if (!ok) f = cell_coef_any<ELEC>(k.c0, k.tcoef, c, m);
  return f;
}

// The band rows (PDEparabolic.f90:66-136 TR, 150-210 BDF2, 250-319 backward Euler) from the
// per-row conduction factors q- = C Dh(i)/dx1i/dx1(i), q+ = C Dh(i+1)/dx1i/dx1(i+1) and the
// advection factor bq = B/(dx1(i+1)+dx1(i)).
enum Stage { ST_TR = 0, ST_BDF2 = 1, ST_BE = 2 };

struct BandRow {
  double s, d, e, r;  // sub-diagonal, diagonal, super-diagonal, right-hand side
};

// Per-row scratch slots: q-, q+, the right-hand side's input (the TR stage's T, replaced by
// the BDF2 right-hand side; the backward-Euler right-hand side), bq (electrons), and the
// elimination state at the first row of each chunk of LU_K rows.
constexpr int LU_QM = 0, LU_QP = 1, LU_RHS = 2, LU_BQ = 3, LU_CP = 4;
constexpr int LU_ROW = 8;  // scratch slots per row (an accessor may pack them)
// Rows per chunk of the back substitution.  Two rows (more checkpoints, less code) ran 7%
// slower at 384x192x192, and more than four do not fit the registers.
constexpr int LU_K = 4;

// conduction factors of row i (2 <= i < n) from C(i), B(i) and D(i-1), D(i), D(i+1)
struct RowFac {
  double qm, qp, bq;
};
struct RowDx {
  double dxi, ydxi, dx0, ydx0, dx1, ydx1, dxs, ydxs;  // of row i; dx0 = dx(i), dx1 = dx(i+1)
};
template <bool ELEC>
#ifdef __CUDACC__
__host__ __device__ __noinline__
#endif
RowFac row_factors_any(double C, double B, double Dhm, double Dhp, RowDx x) {
  RowFac f;
  f.qm = qdiv_t(qdiv_t(C * Dhm, x.dxi, x.ydxi), x.dx0, x.ydx0);
  f.qp = qdiv_t(qdiv_t(C * Dhp, x.dxi, x.ydxi), x.dx1, x.ydx1);
  f.bq = ELEC ? qdiv_t(B, x.dxs, x.ydxs) : 0.0;
  return f;
}
template <bool ELEC, class Acc>
GEMD_HD RowFac row_factors(const Acc& a, int i, double C, double B, double Dm, double Dc, double Dp) {
  const double Dhm = 0.5 * (Dm + Dc), Dhp = 0.5 * (Dc + Dp);  // PDEparabolic.f90:49
  const RowDx x{a.dxi(i), a.ydxi(i), a.dx(i), a.ydx(i), a.dx(i + 1), a.ydx(i + 1), ELEC ? a.dxs(i) : 1.0,
                ELEC ? a.ydxs(i) : 1.0};
  bool ok = true;
  RowFac f;
  f.qm = qtry_t(qtry_t(C * Dhm, x.dxi, x.ydxi, ok), x.dx0, x.ydx0, ok);
  f.qp = qtry_t(qtry_t(C * Dhp, x.dxi, x.ydxi, ok), x.dx1, x.ydx1, ok);
  f.bq = ELEC ? qtry_z(B, x.dxs, x.ydxs, ok) : 0.0;
  if (!ok) f = row_factors_any<ELEC>(C, B, Dhm, Dhp, x);
  return f;
}

// time constants of a stage
template <int STG>
struct StageDt {
  double h, y;  // the stage's step and its correctly rounded reciprocal
  GEMD_HD explicit StageDt(double dt) {
    h = STG == ST_TR ? dt / 2 : STG == ST_BDF2 ? dt / 3 : dt;
    y = 1 / h;
  }
};

// band row from the factors; TR right-hand side from T(i-1), T(i), T(i+1), else rhs as given
template <int STG>
GEMD_HD BandRow band_row(const StageDt<STG>& t, double qm, double qp, double bq, double Tm, double Tc, double Tp,
                         double rhs) {
  BandRow w;
  if (STG == ST_TR) {
    w.s = -(qm / 2) + bq / 2;
    w.d = t.y + qp / 2 + qm / 2;
    w.e = -(qp / 2) - bq / 2;
    const double Pd = qp / 2 + qm / 2;
    w.r = qdiv(Tc, t.h, t.y) - w.s * Tm - Pd * Tc - w.e * Tp;
  } else {
    w.s = -qm + bq;
    w.d = t.y + qp + qm;
    w.e = -qp - bq;
    w.r = rhs;
  }
  return w;
}

// BDF2 right-hand side of a row from T and the TR solution (PDEparabolic.f90:188-196)
#ifdef __CUDACC__
__host__ __device__ __noinline__
#else
inline
#endif
double bdf2_rhs_any(double h, double y, double T, double tr) {
  return -qdiv(1 / 3.0 * T, h, y) + qdiv(4 / 3.0 * tr, h, y);
}
GEMD_HD double bdf2_rhs(const StageDt<ST_BDF2>& t, double T, double tr) {
  bool ok = true;
  const double r = -qtry(1 / 3.0 * T, t.h, t.y, ok) + qtry_t(4 / 3.0 * tr, t.h, t.y, ok);
  return ok ? r : bdf2_rhs_any(t.h, t.y, T, tr);
}

struct LuState {
  double p, q, b;  // current (partially eliminated) row j and its right-hand side
};

struct LuU {
  double u0, rec, u1, u2, y;  // U(j,j) and its reciprocal, U(j,j+1), U(j,j+2), y(j)
};

// One dgbtf2/dgbtrs step with the original row j+1: returns U(j) and y(j).  Both outcomes of
// IDAMAX share one reciprocal through selects: the lanes of a warp interchange at
// different rows, and a branch would run both sides.
GEMD_HD LuU lu_step(LuState& st, const BandRow& w) {
  const bool sw = fabs_f(w.s) > fabs_f(st.p);  // IDAMAX takes row j+1: interchange (DSWAP)
  LuU u;
  u.u0 = sw ? w.s : st.p;
  const double o = sw ? st.p : w.s;
  u.u1 = sw ? w.d : st.q;
  u.u2 = sw ? w.e : 0.0;
  u.y = sw ? w.r : st.b;
  const double a = sw ? st.q : w.d;
  const double c = sw ? st.b : w.r;
  u.rec = rcp_rn(u.u0);
  const double m = u.rec * o;  // DSCAL(1/pivot)
  st.p = a - m * u.u1;
  st.b = c - m * u.y;
  st.q = sw ? 0.0 - m * w.e : w.e;
  return u;
}

// Forward pass of the first stage (TR half step, or the backward-Euler step): walks the cells
// 1..n, at cell i forming row i-1 and eliminating into it; returns the state at row n.
// io.tile(i0) makes the state values of cells i0 .. i0+LU_TILE-1 readable (all lanes).
constexpr int LU_TILE = 8;

// One chunk's scratch values: the factors of rows iq .. iq+LU_K-1 and slot LU_RHS of rows
// iv .. iv+LU_K-1.  io.request names the next chunk, io.take waits for it and reads it; rows
// past n are never used.
struct LuRows {
  double qm[LU_K], qp[LU_K], bq[LU_K], v[LU_K];
};

// plain element access (the host build); n: the column's rows
struct DirectIo {
  int iq = 1, iv = 1;
  GEMD_HD void tile(int) const {}
  template <bool ELEC>
  GEMD_HD void request(int q, int v) {
    iq = q;
    iv = v;
  }
  template <bool ELEC, class Acc>
  GEMD_HD LuRows take(const Acc& a, int n) const {
    LuRows w;
    for (int q = 0; q < LU_K; ++q) {
      const int i = iq + q < n - 1 ? iq + q : n - 1, j = iv + q < n ? iv + q : n;
      w.qm[q] = a.sld(i, LU_QM);
      w.qp[q] = a.sld(i, LU_QP);
      w.bq[q] = ELEC ? a.sld(i, LU_BQ) : 0.0;
      w.v[q] = a.sld(j, LU_RHS);
    }
    return w;
  }
};

template <bool UNIT, bool ELEC, int STG, class Acc, class Io>
GEMD_HD LuState lu_forward_first(const Acc& a, const LuK& k, Io& io) {
  const int n = k.n;
  const StageDt<STG> t(k.dt);
  LuState st{1.0, 0.0, k.tmin};  // row 1: identity, right-hand side Tsminx1
  double Cc = 0.0, Bc = 0.0, Dm = 0.0, Dc = 0.0, Tm = 0.0, Tc = 0.0;
  CellIn cA, cB;  // electrons: the neutral inputs of cells i, i+1
  auto aux = [&](int i, CellIn& c) {
    if (ELEC) a.neutrals(i < n ? i : n, c.n1, c.n2, c.n3, c.j1);
    else c.n1 = c.n2 = c.n3 = c.j1 = 0.0;
  };
  aux(1, cA);
  aux(2, cB);
  for (int i0 = 1; i0 <= n; i0 += LU_TILE) {
    io.tile(i0);
#ifdef __CUDA_ARCH__
#pragma unroll 1  // the passes' code competes for the instruction cache: unrolled twice, 17% slower
#endif
    for (int i = i0; i < i0 + LU_TILE && i <= n; ++i) {
      CellIn c = cA;
      cA = cB;
      aux(i + 2, cB);
      c.T = a.T(i);
      c.n = a.n(i);
      const Coef f = cell_coef<UNIT, ELEC>(a, k, i, c);
      if (i >= 3) {  // row r = i-1
        const int r = i - 1;
        const RowFac q = row_factors<ELEC>(a, r, Cc, Bc, Dm, Dc, f.D);
        const BandRow w = band_row<STG>(t, q.qm, q.qp, q.bq, Tm, Tc, c.T, STG == ST_BE ? qdiv(Tc, t.h, t.y) : 0.0);
        a.sst(r, LU_QM, q.qm);
        a.sst(r, LU_QP, q.qp);
        if (ELEC) a.sst(r, LU_BQ, q.bq);
        if (STG == ST_BE) a.sst(r, LU_RHS, w.r);
        if (r > 2 && (r - 2) % LU_K == 0) {  // the state before step j = r-1 starts a chunk
          a.sst(r - 1, LU_CP, st.p);
          a.sst(r - 1, LU_CP + 1, st.q);
          a.sst(r - 1, LU_CP + 2, st.b);
        }
        lu_step(st, w);
      }
      if (STG == ST_TR) a.sst(i, LU_RHS, c.T);
      Cc = f.C;
      Bc = f.B;
      Dm = Dc;
      Dc = f.D;
      Tm = Tc;
      Tc = c.T;
    }
  }
  const int j = n - 1;
  if (j > 1 && (j - 1) % LU_K == 0) {
    a.sst(j, LU_CP, st.p);
    a.sst(j, LU_CP + 1, st.q);
    a.sst(j, LU_CP + 2, st.b);
  }
  lu_step(st, BandRow{0.0, 1.0, 0.0, k.tmax});
  return st;
}

// Forward pass of the BDF2 stage from the stored q-, q+, bq and right-hand sides, requested a
// chunk ahead of use.
template <bool ELEC, class Acc, class Io>
GEMD_HD LuState lu_forward_bdf2(const Acc& a, const LuK& k, Io& io) {
  const int n = k.n;
  const StageDt<ST_BDF2> t(k.dt);
  LuState st{1.0, 0.0, k.tmin};
  io.template request<ELEC>(2, 2);
  for (int j0 = 1; j0 < n; j0 += LU_K) {  // steps j0 .. j0+LU_K-1, rows j+1
    const LuRows w = io.template take<ELEC>(a, n);
    if (j0 + LU_K < n) io.template request<ELEC>(j0 + LU_K + 1, j0 + LU_K + 1);
    if (j0 > 1) {
      a.sst(j0, LU_CP, st.p);
      a.sst(j0, LU_CP + 1, st.q);
      a.sst(j0, LU_CP + 2, st.b);
    }
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int q = 0; q < LU_K; ++q) {
      const int i = j0 + q + 1;
      if (i < n) lu_step(st, band_row<ST_BDF2>(t, w.qm[q], w.qp[q], w.bq[q], 0.0, 0.0, 0.0, w.v[q]));
      else if (i == n) lu_step(st, BandRow{0.0, 1.0, 0.0, k.tmax});
    }
  }
  return st;
}

// Back substitution of a stage from row n down to row 1 (dtbsv): per chunk of LU_K rows, the
// elimination repeated from the chunk's checkpoint, then
// x(i) = ((y(i) - x(i+2)*U(i,i+2)) - x(i+1)*U(i,i+1)) / U(i,i).  A chunk's inputs are requested
// while the chunk after it is processed.  The TR solution becomes the BDF2 right-hand side
// in the scratch; the other stages give it to OUT, which may need inputs (pre).
template <bool ELEC, int STG, class Acc, class Out, class Io>
GEMD_HD void lu_backward(const Acc& a, const LuK& k, const LuState& fin, const Out& out, Io& io) {
  const int n = k.n;
  const StageDt<STG> t(k.dt);
  const StageDt<ST_BDF2> t3(k.dt);
  auto state = [&](int j0) {
    if (j0 <= 1) return LuState{1.0, 0.0, k.tmin};
    return LuState{a.sld(j0, LU_CP), a.sld(j0, LU_CP + 1), a.sld(j0, LU_CP + 2)};
  };
  auto ask = [&](int j0) { io.template request<ELEC>(j0 + 1, STG == ST_TR ? j0 : j0 + 1); };
  int j0 = ((n - 2) / LU_K) * LU_K + 1;  // first step of the last chunk (steps 1 .. n-1)
  ask(j0);
  LuState next = state(j0);
  double x1 = qdiv(fin.b, fin.p, rcp_rn(fin.p)), x2 = 0.0;  // x(i+1), x(i+2)
  if (STG != ST_TR) out(n, x1, out.pre(n));
  double Ta = 0.0, Tb = 0.0;  // TR: T(j0+LU_K), T(j0+LU_K+1)
  if (STG == ST_TR) {
    Ta = a.sld(j0 + LU_K < n ? j0 + LU_K : n, LU_RHS);
    Tb = a.sld(j0 + LU_K + 1 < n ? j0 + LU_K + 1 : n, LU_RHS);
  }
  for (; j0 >= 1; j0 -= LU_K) {
    const LuRows w = io.template take<ELEC>(a, n);
    LuState st = next;
    if (j0 > 1) {
      ask(j0 - LU_K);
      next = state(j0 - LU_K);
    }
    LuU u[LU_K];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int q = 0; q < LU_K; ++q) {
      const int i = j0 + q + 1;  // row eliminated by step j = i-1; v: T(j0 ..) in TR, else the rhs
      const double Tc = q + 1 < LU_K ? w.v[q + 1 < LU_K ? q + 1 : 0] : Ta;
      const double Tp = q + 2 < LU_K ? w.v[q + 2 < LU_K ? q + 2 : 0] : (q + 2 == LU_K ? Ta : Tb);
      if (i < n) u[q] = lu_step(st, band_row<STG>(t, w.qm[q], w.qp[q], w.bq[q], w.v[q], Tc, Tp, w.v[q]));
      else u[q] = lu_step(st, BandRow{0.0, 1.0, 0.0, k.tmax});  // row n; past it unused
    }
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int q = LU_K - 1; q >= 0; --q) {
      const int j = j0 + q;
      if (j < n) {
        double x = u[q].y;
        if (j <= n - 2) x = x - x2 * u[q].u2;
        x = x - x1 * u[q].u1;
        x = qdiv(x, u[q].u0, u[q].rec);
        if (STG == ST_TR) a.sst(j, LU_RHS, bdf2_rhs(t3, w.v[q], x));
        else out(j, x, out.pre(j));
        x2 = x1;
        x1 = x;
      }
    }
    Ta = w.v[0];
    Tb = w.v[1];
  }
}

// The whole solve of one (column, species): TRBDF2 (solver 2) or backward Euler (solver 1).
// OUT receives the new temperature of each row (before the max(T,100) floor).
template <bool UNIT, bool ELEC, class Acc, class Out, class Io = DirectIo>
GEMD_HD void lu_column(const Acc& a, const LuK& k, int solver, const Out& out, Io io = Io{}) {
  if (solver == 2) {
    LuState st = lu_forward_first<UNIT, ELEC, ST_TR>(a, k, io);
    lu_backward<ELEC, ST_TR>(a, k, st, out, io);
    st = lu_forward_bdf2<ELEC>(a, k, io);
    lu_backward<ELEC, ST_BDF2>(a, k, st, out, io);
  } else {
    const LuState st = lu_forward_first<UNIT, ELEC, ST_BE>(a, k, io);
    lu_backward<ELEC, ST_BE>(a, k, st, out, io);
  }
}

}  // namespace gemd
