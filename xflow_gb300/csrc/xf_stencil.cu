// Operators (T3dLaplaceOperator, T3dVariableDivergentedOperator) and the
// masked matvec y |= A(x) (+/- s) of TRnRelease3dSpace::
// LocalReleaseAssignSpeedLinearCombination(op) (XSpace.cpp:3013-3217).
//
// Kernel layout (plane march): a thread owns one (j, k) column of the box and
// walks a chunk of i-planes, keeping x[i-1], x[i], x[i+1] in registers and
// prefetching plane i+2 while it computes plane i.  Consecutive threads own
// consecutive k, so every plane access is coalesced; the j+-1 / k+-1
// neighbours are re-reads of lines the neighbouring threads just fetched (L1/L2).
#include <atomic>
#include <type_traits>

#include "xf_control.cuh"
#include "xf_stencil.cuh"

template <>
StencilGrid<double> make_stencil_grid<double>(const xf_grid* g, const double* rho) {
  StencilGrid<double> s;
  s.kind = g->kind; s.brow_of = g->brow_of; s.brow_nrm = g->brow_nrm;
  s.hx = g->hx; s.hy = g->hy; s.hz = g->hz;
  s.cxm = g->cxm; s.cxp = g->cxp; s.cym = g->cym; s.cyp = g->cyp; s.czm = g->czm; s.czp = g->czp;
  s.rhx = g->rhx; s.rhy = g->rhy; s.rhz = g->rhz; s.rhhx = g->rhhx; s.rhhy = g->rhhy; s.rhhz = g->rhhz;
  s.rho = rho;
  s.n1 = g->n1; s.n2 = g->n2; s.n3 = g->n3; s.s1 = (int)g->s1; s.s2 = (int)g->s2;
  return s;
}
template <>
StencilGrid<float> make_stencil_grid<float>(const xf_grid* g, const float* rho) {
  StencilGrid<float> s;
  s.kind = g->kind; s.brow_of = g->brow_of; s.brow_nrm = g->brow_nrm;
  s.hx = g->fhx; s.hy = g->fhy; s.hz = g->fhz;
  s.cxm = g->fxm; s.cxp = g->fxp; s.cym = g->fym; s.cyp = g->fyp; s.czm = g->fzm; s.czp = g->fzp;
  s.rhx = g->frhx; s.rhy = g->frhy; s.rhz = g->frhz; s.rhhx = g->frhhx; s.rhhy = g->frhhy; s.rhhz = g->frhhz;
  s.rho = rho;
  s.n1 = g->n1; s.n2 = g->n2; s.n3 = g->n3; s.s1 = (int)g->s1; s.s2 = (int)g->s2;
  return s;
}

constexpr int MV_THREADS = 256;

// y |= A(x) + sign*s (negated when neg), written to y (T) and/or y32 (float);
// fused FP64 dots (w, v) -> slot_w and (v, v) -> slot_w+1; the last block to
// finish runs the solver control step `ctl`.
template <typename T>
struct MatvecArgs {
  StencilGrid<T> g;
  const T* __restrict__ x;
  T* __restrict__ y;
  float* __restrict__ y32;
  const T* __restrict__ s;
  const T* __restrict__ w;
  const double* __restrict__ diag;
  int sign, neg, zero_inactive, dot_w, dot_self;
  int slot_w, ctl, gate, chunk;
  const uint8_t* __restrict__ use;   // k_ad_fast: xf_op::adk, or adks
  const double* __restrict__ dinv;   // the same, scaled: the inverse diagonals
  DevScratch* S;
};

// Laplace Actual row on register-resident x[i-1], x[i], x[i+1].
template <typename T, bool USE_D>
__device__ __forceinline__ T march_lap(const StencilGrid<T>& g, const MatvecArgs<T>& a, int c, int i, uint8_t kb,
                                       T xm, T xc, T xp, T xjm, T xjp, T xkm, T xkp, T cym, T cyp, T czm, T czp) {
  const T cxm = g.cxm[i], cxp = g.cxp[i];
  if (USE_D) {
    // FP64: y = D x_c - sum_n c_n x_n  (one DMUL and six DFMA per row)
    const T kpx = (kb & K_PX) ? cxp : T(0), kmx = (kb & K_MX) ? cxm : T(0);
    const T kpy = (kb & K_PY) ? cyp : T(0), kmy = (kb & K_MY) ? cym : T(0);
    const T kpz = (kb & K_PZ) ? czp : T(0), kmz = (kb & K_MZ) ? czm : T(0);
    T acc = (T)a.diag[c] * xc;
    acc = fma(xneg(kpx), xp, acc);
    acc = fma(xneg(kmx), xm, acc);
    acc = fma(xneg(kpy), xjp, acc);
    acc = fma(xneg(kmy), xjm, acc);
    acc = fma(xneg(kpz), xkp, acc);
    acc = fma(xneg(kmz), xkm, acc);
    return acc;
  } else {
    // FP32: the reference's difference form, c * (x_n - x_c)
    const T tpx = (kb & K_PX) ? cxp * (xp - xc) : T(0);
    const T tmx = (kb & K_MX) ? cxm * (xc - xm) : T(0);
    const T tpy = (kb & K_PY) ? cyp * (xjp - xc) : T(0);
    const T tmy = (kb & K_MY) ? cym * (xc - xjm) : T(0);
    const T tpz = (kb & K_PZ) ? czp * (xkp - xc) : T(0);
    const T tmz = (kb & K_MZ) ? czm * (xc - xkm) : T(0);
    return -(((tpx - tmx) + (tpy - tmy)) + (tpz - tmz));
  }
}

// The fast rows are bound by the loads in flight (a plane's are behind the
// last plane's): four blocks an SM, at most 64 registers.
template <typename T, int OP, bool EXACT, bool USE_D>
__global__ void __launch_bounds__(MV_THREADS, EXACT ? 1 : 4) k_matvec(MatvecArgs<T> a) {
  __shared__ double sh[32];
  __shared__ bool last;
  // Solver kernels turn into no-ops once the solve is done (or, when gated,
  // while no true-residual replacement is pending).
  if (a.ctl != CTL_NONE && (a.S->iscalars[I_DONE] || (a.gate && !a.S->iscalars[I_NEEDREP]))) return;
  const StencilGrid<T>& g = a.g;
  const int P = g.n2 * g.n3;
  const int p = blockIdx.x * MV_THREADS + threadIdx.x;
  const int i0 = blockIdx.y * a.chunk;
  const int i1 = min(g.n1, i0 + a.chunk);
  DotAcc<T> dw, ds;
  if (p < P) {
    const int j = p / g.n3, k = p - j * g.n3;
    // side offsets clamped to stay inside the box (only used by interior rows)
    const int okm = k > 0 ? -1 : 0, okp = k < g.n3 - 1 ? 1 : 0;
    const int ojm = j > 0 ? -g.n3 : 0, ojp = j < g.n2 - 1 ? g.n3 : 0;
    const bool fast = (OP == XF_OP_LAPLACE) && !EXACT;
    T cym = 0, cyp = 0, czm = 0, czp = 0;
    if (fast) { cym = g.cym[j]; cyp = g.cyp[j]; czm = g.czm[k]; czp = g.czp[k]; }
    const T* __restrict__ x = a.x;
    int c = i0 * P + p;
    T xm = i0 > 0 ? x[c - P] : T(0);
    T xc = x[c];
    T xp = i0 + 1 < g.n1 ? x[c + P] : T(0);
    uint8_t kc = g.kind[c];
    for (int i = i0; i < i1; i++, c += P) {
      const T xpp = i + 2 < g.n1 ? x[c + 2 * P] : T(0);
      const uint8_t kn = i + 1 < g.n1 ? g.kind[c + P] : (uint8_t)0;
      const T xjm = x[c + ojm], xjp = x[c + ojp], xkm = x[c + okm], xkp = x[c + okp];
      const int row = row_of(kc);
      if (row == ROW_NONE) {
        if (a.zero_inactive) {
          if (a.y) a.y[c] = T(0);
          if (a.y32) a.y32[c] = 0.f;
        }
      } else {
        T v;
        if (fast && row == ROW_ACTUAL) v = march_lap<T, USE_D>(g, a, c, i, kc, xm, xc, xp, xjm, xjp, xkm, xkp, cym, cyp, czm, czp);
        else v = apply_row<T, OP, EXACT>(g, x, i, j, k, c, kc);
        if (a.sign > 0) v = v + a.s[c];
        else if (a.sign < 0) v = v - a.s[c];
        if (a.neg) v = xneg(v);
        if (a.dot_w) dw.add(a.w[c], v);
        if (a.dot_self) ds.add(v, v);
        if (a.y) a.y[c] = v;
        if (a.y32) a.y32[c] = (float)v;
      }
      xm = xc; xc = xp; xp = xpp; kc = kn;
    }
  }
  if (a.dot_w || a.dot_self || a.ctl != CTL_NONE) {
    double vals[2] = {dw.value(), ds.value()};
    if (publish_partials<2>(a.S, a.slot_w, vals, sh, &last)) {
      double tw = finish_partials(a.S, a.slot_w, sh);
      double ts = finish_partials(a.S, a.slot_w + 1, sh);
      if (threadIdx.x == 0) {
        if (a.dot_w) a.S->scalars[a.slot_w] = tw;
        if (a.dot_self) a.S->scalars[a.slot_w + 1] = ts;
        a.S->tickets[a.slot_w] = 0;
        control_step(a.S, a.ctl);
      }
    }
  }
}

// The advection fields of an XF_OP_ADVDIFF operator in a stencil grid.
template <typename T>
static void set_ad_fields(StencilGrid<T>& s, const xf_op* op) {
  constexpr bool D64 = std::is_same<T, double>::value;
  s.adv0 = D64 ? (const T*)op->adv64[0] : (const T*)op->adv32[0];
  s.adv1 = D64 ? (const T*)op->adv64[1] : (const T*)op->adv32[1];
  s.adv2 = D64 ? (const T*)op->adv64[2] : (const T*)op->adv32[2];
  s.ad_itau = (T)(1 / op->ad_tau);
  s.ad_D = (T)op->ad_D;
  s.adDf = !op->adD_set ? nullptr : D64 ? (const T*)op->adD64 : (const T*)op->adD32;
  s.ad_conv = (op->ad_flags & XF_ADV_CONVECTIVE) ? T(1) : T(0);
  s.ad_diff = (op->ad_flags & XF_ADV_DIFFUSIVE) ? T(1) : T(0);
  s.ad_upwind = (op->ad_flags & XF_ADV_UPWIND) ? 1 : 0;
  s.adc = (D64 && op->adc_valid) ? (const T*)op->adc64 : nullptr;
  s.adc_n = op->g->ncell;
}

// Per-axis factors of the fast coefficients, 5 arrays over the nodes m of an
// axis (the halves and the two flags folded in): conv 0.5/hx2, conv 0.5/h,
// diff 0.5 h/hxhxh, diff 0.5 hx2/hxhxh, diff 0.5 h_1/hxhxh with h_1 = h[m-1],
// h = h[m], hx2 = h_1 + h, hxhxh = h_1 h hx2 / 2 (the exact rows' quantities;
// nodes 0 and n-1, which carry no Actual row, get 0).
__global__ void k_ad_axis(const double* __restrict__ h, int n, double conv, double diff, double* __restrict__ t) {
  for (int m = threadIdx.x; m < n; m += blockDim.x) {
    double r2 = 0, rh = 0, dA = 0, dB = 0, dC = 0;
    if (m >= 1 && m <= n - 2) {
      const double h_1 = h[m - 1], hh = h[m], hx2 = h_1 + hh, hxhxh = h_1 * hh * hx2 / 2;
      r2 = conv * (0.5 / hx2);
      rh = conv * (0.5 / hh);
      dA = diff * (0.5 * hh / hxhxh);
      dB = diff * (0.5 * hx2 / hxhxh);
      dC = diff * (0.5 * h_1 / hxhxh);
    }
    t[m] = r2; t[n + m] = rh; t[2 * n + m] = dA; t[3 * n + m] = dB; t[4 * n + m] = dC;
  }
}

struct AdAxis { double r2, rh, dA, dB, dC; };
__device__ __forceinline__ AdAxis ad_axis(const double* __restrict__ t, int n, int m) {
  return {__ldg(t + m), __ldg(t + n + m), __ldg(t + 2 * n + m), __ldg(t + 3 * n + m), __ldg(t + 4 * n + m)};
}

// A and C of one direction from the axis factors (central or upwind), as the
// exact rows define them but with products for the divisions; B is added to
// the centre.  5 FP64 operations a direction (7 upwind): the FP64 pipe bounds
// the table's kernel.
template <bool UP>
__device__ __forceinline__ void ad_coef_fast(const AdAxis& t, double vd, double D, double& A, double& C, double& centre) {
  A = xneg(D) * t.dA;
  C = xneg(D) * t.dC;
  centre = fma(D, t.dB, centre);
  if (!UP) {
    A = fma(xneg(vd), t.r2, A);
    C = fma(vd, t.r2, C);
  } else if (vd < 0) {
    centre = fma(xneg(vd), t.rh, centre);
    C = fma(vd, t.rh, C);
  } else {
    A = fma(xneg(vd), t.rh, A);
    centre = fma(vd, t.rh, centre);
  }
}

// 1/d by two Newton-Raphson steps y <- y + y (1 - d y) from the hardware's
// approximation (2^-23 of it): 4 operations on the FP64 pipe where a division
// takes three times as many.  Within a rounding of 1/d, for the
// preconditioner; divided where the steps could leave the normal range.
__device__ __forceinline__ double ad_reciprocal(double d) {
  const int e = (__double2hiint(d) >> 20) & 0x7ff;
  if (e < 64 || e > 1982) return d != 0 ? 1.0 / d : 0.0;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  y = fma(y, fma(xneg(d), y, 1.0), y);
  return fma(y, fma(xneg(d), y, 1.0), y);
}

enum { AD_ROW = 64, AD_OBLIQUE = 128 };

// The border rows in the same seven-coefficient form (centre, x-, x+, y-,
// y+, z-, z+): a semi-sum row takes 1/2 of itself and of its neighbour
// against the normal (the last nonzero normal component decides, as the row
// does); a normal-difference row with an axis-aligned normal is
// n_a (f_c - f_{c-1}) / h (normal +) or n_a (f_{c+1} - f_c) / h (normal -),
// its 4-point face averages collapsing to single cells.  A normal-difference
// row with an oblique normal reaches beyond the seven points: NaN in the
// centre sends it to the general row.
__device__ __forceinline__ bool ad_nonzero(double v) { return (__double_as_longlong(v) << 1) != 0; }
struct AdBorder { int axis, nb; double q0, qn; };   // nb: the neighbour read (0 x- .. 5 z+), qn its coefficient
__device__ __forceinline__ AdBorder ad_border_coeffs(const StencilGrid<double>& g, int64_t c, int row, int i, int j,
                                                     int k) {
  const double* nrm = g.brow_nrm + 3 * g.brow_of[c];
  const double nx = nrm[0], ny = nrm[1], nz = nrm[2];
  const bool ux = ad_nonzero(nx), uy = ad_nonzero(ny), uz = ad_nonzero(nz);
  const int ax = uz ? 2 : uy ? 1 : ux ? 0 : -1;
  const double na = uz ? nz : uy ? ny : nx;
  AdBorder r = {ax, 0, 0.0, 0.0};
  if (ax < 0) return r;   // no normal: the row is 0
  const bool pos = __double_as_longlong(na) >= 0;
  r.nb = 2 * ax + (pos ? 0 : 1);
  if (row == ROW_PREDEF) {
    r.q0 = r.qn = 0.5;
  } else if (ux + uy + uz > 1) {
    r.q0 = __longlong_as_double(0x7ff8000000000000ll);
  } else {
    const int m = (ax == 0 ? i : ax == 1 ? j : k) - (pos ? 1 : 0);
    const double* h = ax == 0 ? g.hx : ax == 1 ? g.hy : g.hz;
    const double d = na / h[m];
    r.q0 = pos ? d : -d;
    r.qn = pos ? -d : d;
  }
  return r;
}

// A unit probe at the row's own cell: a border row evaluated on it is the
// row's diagonal coefficient.
struct UnitProbe {
  __device__ __forceinline__ double operator()(int a, int b, int d) const { return (a | b | d) == 0 ? 1.0 : 0.0; }
};

// The inverse diagonal of an oblique normal difference.
__device__ __noinline__ double ad_oblique_inverse(const StencilGrid<double>& g, int64_t c, int row, int i, int j, int k) {
  const double d = boundary_row_acc<double, false>(g, UnitProbe{}, i, j, k, (int)c, row);
  return d != 0 ? 1.0 / d : 0.0;
}

// A border row's part of the table: its coefficients, the neighbour it reads and its inverse diagonal.
__device__ __forceinline__ void ad_border_cell(const StencilGrid<double>& g, int64_t n, int64_t c, int row, int i, int j,
                                               int k, double* __restrict__ out, uint8_t* __restrict__ use,
                                               double* __restrict__ dinv) {
  const AdBorder b = ad_border_coeffs(g, c, row, i, j, k);
  const bool oblique = b.q0 != b.q0;
  const bool reads = !oblique && ad_nonzero(b.qn);
  out[c] = b.q0;
#pragma unroll
  for (int t = 0; t < 6; t++) out[(t + 1) * n + c] = t == b.nb && !oblique ? b.qn : 0.0;
  use[c] = AD_ROW | (oblique ? AD_OBLIQUE : 0) | (reads ? 1 << b.nb : 0);
  dinv[c] = oblique ? ad_oblique_inverse(g, c, row, i, j, k) : ad_reciprocal(b.q0);
}

// The FP64 coefficient table of the fast rows: for Actual rows a centre
// coefficient 1/tau + B_x + B_y + B_z and the six neighbour coefficients;
// border rows as ad_border_coeffs; with it the bytes of the neighbours a row
// reads and the inverse row diagonals (0 off the active set and where a
// diagonal is 0; border rows: the row on a unit probe).  A thread owns a
// (j, k) column and marches a chunk of planes with its y and z factors in
// registers.
constexpr int ADC_THREADS = 256, ADC_CHUNK = 8;
template <bool UP>
__global__ void __launch_bounds__(ADC_THREADS) k_ad_coeffs(StencilGrid<double> g, int64_t n,
                                                           const double* __restrict__ tx, const double* __restrict__ ty,
                                                           const double* __restrict__ tz, double* __restrict__ out,
                                                           uint8_t* __restrict__ use, double* __restrict__ dinv) {
  const int P = g.s1, p = blockIdx.x * ADC_THREADS + threadIdx.x;
  if (p >= P) return;
  const int j = p / g.n3, k = p - j * g.n3;
  const AdAxis fy = ad_axis(ty, g.n2, j), fz = ad_axis(tz, g.n3, k);
  const int i0 = blockIdx.y * ADC_CHUNK, i1 = min(g.n1, i0 + ADC_CHUNK);
  for (int i = i0; i < i1; i++) {
    const int64_t c = (int64_t)i * P + p;
    const int row = row_of(g.kind[c]);
    if (row == ROW_NONE) {
      use[c] = 0;
      dinv[c] = 0.0;
      continue;
    }
    if (row != ROW_ACTUAL) {
      ad_border_cell(g, n, c, row, i, j, k, out, use, dinv);
      continue;
    }
    const double D = g.adDf ? g.adDf[c] : g.ad_D;
    double A[3], C[3], q0 = g.ad_itau;
    ad_coef_fast<UP>(ad_axis(tx, g.n1, i), g.adv0[c], D, A[0], C[0], q0);
    ad_coef_fast<UP>(fy, g.adv1[c], D, A[1], C[1], q0);
    ad_coef_fast<UP>(fz, g.adv2[c], D, A[2], C[2], q0);
    out[c] = q0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      out[(1 + 2 * d) * n + c] = A[d];
      out[(2 + 2 * d) * n + c] = C[d];
    }
    use[c] = AD_ROW | 63;
    dinv[c] = ad_reciprocal(q0);
  }
}

// The fast FP64 advection-diffusion apply as a flat grid-stride kernel: a
// thread takes cell after cell (the row reads its seven coefficients and its
// neighbours directly, so the plane march buys nothing), at full occupancy.
// Border rows read the table too (their semi-sums and axis-aligned normal
// differences are seven-point rows), by the same instructions: the cell's byte
// says which neighbours its row reads, and the others are not read but taken
// as 0 with the coefficient 0.  (A branch for border rows ran both sides in a
// quarter of the warps, a k-row ending every 130 cells: 15 FP64 instructions a
// cell on average, where the row takes 7 and its dots 1 or 2.)  Only oblique
// normal differences take the general row.  Same dots and control step as
// k_matvec.  What bounds it: FP64 issue and, a little behind, the 81 bytes a
// cell.
constexpr int AD_THREADS = 256, AD_RESIDENT = 4;   // four blocks an SM, one wave
// The border rows, out of line: they are few, and inlined they would set the
// register budget of the whole loop.
__device__ __noinline__ double ad_border_row(const StencilGrid<double>& g, const double* __restrict__ x, int64_t c,
                                             int row) {
  const int64_t s1 = g.s1, s2 = g.s2;
  const int i = (int)(c / s1), j = (int)((c - (int64_t)i * s1) / s2), k = (int)(c % s2);
  return boundary_row<double, false>(g, x, i, j, k, (int)c, row);
}

// A D^-1's row of a cell that the scaled table does not hold: an oblique
// normal difference, or a row whose diagonal is 0 (D^-1 holds 0 there).
struct ScaledProbe {
  const double *x, *dinv;
  int64_t c, s1, s2;
  __device__ __forceinline__ double operator()(int a, int b, int d) const {
    const int64_t at = c + a * s1 + b * s2 + d;
    return dinv[at] * x[at];
  }
};
__device__ __noinline__ double ad_scaled_row(const StencilGrid<double>& g, const double* __restrict__ x,
                                             const double* __restrict__ dinv, int64_t c, uint32_t u) {
  const int row = row_of(g.kind[c]);
  const int64_t s1 = g.s1, s2 = g.s2, nn = g.adc_n;
  if (row == ROW_ACTUAL) {
    const int64_t off[6] = {-s1, s1, -s2, s2, -1, 1};
    double v = 0.0;
    for (int t = 0; t < 6; t++)
      if (u >> t & 1) v = fma(g.adc[t * nn + c], x[c + off[t]], v);
    return v;
  }
  const int i = (int)(c / s1), j = (int)((c - (int64_t)i * s1) / s2), k = (int)(c % s2);
  return boundary_row_acc<double, false>(g, ScaledProbe{x, dinv, c, s1, s2}, i, j, k, (int)c, row);
}

// SCALED: A D^-1 from the scaled table, its diagonal 1: a product and 8 bytes a
// cell less, and the solver keeps no preconditioned copies of its vectors.
template <bool SCALED>
__global__ void __launch_bounds__(AD_THREADS, AD_RESIDENT) k_ad_fast(MatvecArgs<double> a) {
  __shared__ double sh[32];
  __shared__ bool last;
  if (a.ctl != CTL_NONE && (a.S->iscalars[I_DONE] || (a.gate && !a.S->iscalars[I_NEEDREP]))) return;
  const StencilGrid<double>& g = a.g;
  const int64_t s1 = g.s1, s2 = g.s2, n = (int64_t)g.n1 * s1, nn = g.adc_n;
  const double* __restrict__ x = a.x;
  DotAcc<double> dw, ds;
  const int64_t step = (int64_t)gridDim.x * AD_THREADS;
  int64_t c = blockIdx.x * (int64_t)AD_THREADS + threadIdx.x;
  uint32_t next = c < n ? a.use[c] : 0;   // a cell's byte is loaded a cell ahead: the neighbours' loads wait for it
  for (; c < n; c += step) {
    const uint32_t u = next;
    if (c + step < n) next = a.use[c + step];
    if (u == 0) {
      if (a.zero_inactive) {
        if (a.y) a.y[c] = 0.0;
        if (a.y32) a.y32[c] = 0.f;
      }
      continue;
    }
    const double* __restrict__ q = g.adc + c;
    const double x1 = u & 1 ? x[c - s1] : 0.0, x2 = u & 2 ? x[c + s1] : 0.0, x3 = u & 4 ? x[c - s2] : 0.0;
    const double x4 = u & 8 ? x[c + s2] : 0.0, x5 = u & 16 ? x[c - 1] : 0.0, x6 = u & 32 ? x[c + 1] : 0.0;
    double v = SCALED ? x[c] : q[0] * x[c];
    if (!SCALED) q += nn;
    v = fma(q[0], x1, v);
    v = fma(q[nn], x2, v);
    v = fma(q[2 * nn], x3, v);
    v = fma(q[3 * nn], x4, v);
    v = fma(q[4 * nn], x5, v);
    v = fma(q[5 * nn], x6, v);
    if (u & AD_OBLIQUE) v = SCALED ? ad_scaled_row(g, x, a.dinv, c, u) : ad_border_row(g, x, c, row_of(g.kind[c]));
    if (a.sign > 0) v = v + a.s[c];
    else if (a.sign < 0) v = v - a.s[c];
    if (a.neg) v = xneg(v);
    if (a.dot_w) dw.add(a.w[c], v);
    if (a.dot_self) ds.add(v, v);
    if (a.y) a.y[c] = v;
    if (a.y32) a.y32[c] = (float)v;
  }
  if (a.dot_w || a.dot_self || a.ctl != CTL_NONE) {
    double vals[2] = {dw.value(), ds.value()};
    if (publish_partials<2>(a.S, a.slot_w, vals, sh, &last)) {
      double tw = finish_partials(a.S, a.slot_w, sh);
      double ts = finish_partials(a.S, a.slot_w + 1, sh);
      if (threadIdx.x == 0) {
        if (a.dot_w) a.S->scalars[a.slot_w] = tw;
        if (a.dot_self) a.S->scalars[a.slot_w + 1] = ts;
        a.S->tickets[a.slot_w] = 0;
        control_step(a.S, a.ctl);
      }
    }
  }
}

// Two consecutive cells a thread, 16-byte loads: half the load instructions,
// twice the bytes in flight a warp.  For grids of even rows (a pair lies in one
// row) and 16-byte aligned vectors; a neighbour that a row does not read is
// taken as 0 here too, though its pair was loaded for the other cell.  514 x
// 130 x 130: 168 -> 162 us a call (FP64 issue bounds both); the predictors of
// 64^3 2.48 -> 2.41 ms, the scalar of 256 x 64 x 64 1.60 -> 1.53.
constexpr int AD2_RESIDENT = 3;
template <bool SCALED>
__global__ void __launch_bounds__(AD_THREADS, AD2_RESIDENT) k_ad_fast2(MatvecArgs<double> a) {
  __shared__ double sh[32];
  __shared__ bool last;
  if (a.ctl != CTL_NONE && (a.S->iscalars[I_DONE] || (a.gate && !a.S->iscalars[I_NEEDREP]))) return;
  const StencilGrid<double>& g = a.g;
  const int64_t s1 = g.s1, s2 = g.s2, n = (int64_t)g.n1 * s1, nn = g.adc_n;
  const double* __restrict__ x = a.x;
  DotAcc<double> dw, ds;
  const int64_t step = (int64_t)gridDim.x * AD_THREADS * 2;
  int64_t c = 2 * (blockIdx.x * (int64_t)AD_THREADS + threadIdx.x);
  auto ld2 = [](const double* p) { return __ldg(reinterpret_cast<const double2*>(p)); };
  auto use2 = [&](int64_t at) { return (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(a.use + at)); };
  uint32_t next = c < n ? use2(c) : 0;   // the bytes are loaded a pair ahead: the neighbours' loads wait for them
  for (; c < n; c += step) {
    const uint32_t u = next, u0 = u & 255u, u1 = u >> 8, any = u0 | u1;
    if (c + step < n) next = use2(c + step);
    double2 v = make_double2(0.0, 0.0);
    if (u) {
      const double* __restrict__ q = g.adc + c;
      const double2 z = make_double2(0.0, 0.0);
      double2 x1 = any & 1 ? ld2(x + c - s1) : z, x2 = any & 2 ? ld2(x + c + s1) : z;
      double2 x3 = any & 4 ? ld2(x + c - s2) : z, x4 = any & 8 ? ld2(x + c + s2) : z;
      const double2 xc = ld2(x + c);
      double2 x5 = make_double2(u0 & 16 ? __ldg(x + c - 1) : 0.0, xc.x), x6 = make_double2(xc.y, u1 & 32 ? __ldg(x + c + 2) : 0.0);
      if ((u0 & u1 & 63u) != 63u) {   // border pairs
        if (!(u0 & 1)) x1.x = 0.0;
        if (!(u1 & 1)) x1.y = 0.0;
        if (!(u0 & 2)) x2.x = 0.0;
        if (!(u1 & 2)) x2.y = 0.0;
        if (!(u0 & 4)) x3.x = 0.0;
        if (!(u1 & 4)) x3.y = 0.0;
        if (!(u0 & 8)) x4.x = 0.0;
        if (!(u1 & 8)) x4.y = 0.0;
        if (!(u1 & 16)) x5.y = 0.0;
        if (!(u0 & 32)) x6.x = 0.0;
      }
      v = xc;
      if (!SCALED) {
        const double2 q0 = ld2(q);
        v.x *= q0.x;
        v.y *= q0.y;
        q += nn;
      }
      const double2 q1 = ld2(q), q2 = ld2(q + nn), q3 = ld2(q + 2 * nn), q4 = ld2(q + 3 * nn);
      const double2 q5 = ld2(q + 4 * nn), q6 = ld2(q + 5 * nn);
      v.x = fma(q1.x, x1.x, v.x);
      v.y = fma(q1.y, x1.y, v.y);
      v.x = fma(q2.x, x2.x, v.x);
      v.y = fma(q2.y, x2.y, v.y);
      v.x = fma(q3.x, x3.x, v.x);
      v.y = fma(q3.y, x3.y, v.y);
      v.x = fma(q4.x, x4.x, v.x);
      v.y = fma(q4.y, x4.y, v.y);
      v.x = fma(q5.x, x5.x, v.x);
      v.y = fma(q5.y, x5.y, v.y);
      v.x = fma(q6.x, x6.x, v.x);
      v.y = fma(q6.y, x6.y, v.y);
      if (any & AD_OBLIQUE) {
        if (u0 & AD_OBLIQUE) v.x = SCALED ? ad_scaled_row(g, x, a.dinv, c, u0) : ad_border_row(g, x, c, row_of(g.kind[c]));
        if (u1 & AD_OBLIQUE)
          v.y = SCALED ? ad_scaled_row(g, x, a.dinv, c + 1, u1) : ad_border_row(g, x, c + 1, row_of(g.kind[c + 1]));
      }
      if (a.sign) {
        const double2 s = ld2(a.s + c);
        v.x = a.sign > 0 ? v.x + s.x : v.x - s.x;
        v.y = a.sign > 0 ? v.y + s.y : v.y - s.y;
      }
      if (a.neg) v = make_double2(xneg(v.x), xneg(v.y));
      if (!u0) v.x = 0.0;   // no row: in no dot
      if (!u1) v.y = 0.0;
      if (a.dot_w) {
        const double2 w = ld2(a.w + c);
        if (u0) dw.add(w.x, v.x);
        if (u1) dw.add(w.y, v.y);
      }
      if (a.dot_self) {
        ds.add(v.x, v.x);
        ds.add(v.y, v.y);
      }
    }
    if (a.zero_inactive || (u0 && u1)) {
      if (a.y) *reinterpret_cast<double2*>(a.y + c) = v;
      if (a.y32) *reinterpret_cast<float2*>(a.y32 + c) = make_float2((float)v.x, (float)v.y);
    } else {
      if (u0) {
        if (a.y) a.y[c] = v.x;
        if (a.y32) a.y32[c] = (float)v.x;
      }
      if (u1) {
        if (a.y) a.y[c + 1] = v.y;
        if (a.y32) a.y32[c + 1] = (float)v.y;
      }
    }
  }
  if (a.dot_w || a.dot_self || a.ctl != CTL_NONE) {
    double vals[2] = {dw.value(), ds.value()};
    if (publish_partials<2>(a.S, a.slot_w, vals, sh, &last)) {
      double tw = finish_partials(a.S, a.slot_w, sh);
      double ts = finish_partials(a.S, a.slot_w + 1, sh);
      if (threadIdx.x == 0) {
        if (a.dot_w) a.S->scalars[a.slot_w] = tw;
        if (a.dot_self) a.S->scalars[a.slot_w + 1] = ts;
        a.S->tickets[a.slot_w] = 0;
        control_step(a.S, a.ctl);
      }
    }
  }
}

// The scaled table: each neighbour coefficient times the neighbour's inverse
// diagonal.  Bound by memory (6 planes in, 6 out: 0.15 ms for 514 x 130 x 130
// cells, against 69 us that each iteration gains).
__global__ void __launch_bounds__(AD_THREADS) k_ad_scale(const double* __restrict__ q, const uint8_t* __restrict__ use,
                                                         const double* __restrict__ dinv, int64_t n, int64_t s1,
                                                         int64_t s2, double* __restrict__ out,
                                                         uint8_t* __restrict__ uses) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t u = use[c];
    uses[c] = (uint8_t)(u && dinv[c] == 0.0 ? u | AD_OBLIQUE : u);
    if (u == 0) continue;
    const int64_t off[6] = {-s1, s1, -s2, s2, -1, 1};
#pragma unroll
    for (int t = 0; t < 6; t++) out[t * n + c] = u >> t & 1 ? q[(t + 1) * n + c] * dinv[c + off[t]] : 0.0;
  }
}
// x += D^-1 y on the active set.
__global__ void k_ad_unscale(double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ dinv,
                             const uint8_t* __restrict__ m, int64_t n) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
    if (m[c]) x[c] = fma(dinv[c], y[c], x[c]);
}

// The scaled table of a ready operator; false where it has none (no table) or
// no memory is left for it: the caller keeps to A and preconditioned copies.
bool xf_op_scaled(const xf_op* op) {
  if (op->kind != XF_OP_ADVDIFF || !op->adc_valid) return false;
  if (op->ads_valid) return true;
  const xf_grid* g = op->g;
  const int64_t n = g->ncell;
  if ((!op->ads64 && cudaMalloc(&op->ads64, 6 * n * 8) != cudaSuccess) ||
      (!op->adks && cudaMalloc(&op->adks, n) != cudaSuccess)) {
    cudaGetLastError();
    return false;
  }
  k_ad_scale<<<grid_blocks(g->ctx, n, AD_THREADS), AD_THREADS, 0, g->ctx->stream>>>(op->adc64, op->adk, op->adj64, n, g->s1,
                                                                                   g->s2, op->ads64, op->adks);
  op->ads_valid = 1;
  return true;
}
void xf_op_scaled_free(const xf_op* op) {
  cudaFree(op->ads64);
  cudaFree(op->adks);
  op->ads64 = nullptr;
  op->adks = nullptr;
  op->ads_valid = 0;
}
void xf_op_unscale(const xf_op* op, double* x, const double* y) {
  const xf_grid* g = op->g;
  k_ad_unscale<<<grid_blocks(g->ctx, g->ncell, 256), 256, 0, g->ctx->stream>>>(x, y, op->adj64, g->smask, g->ncell);
}

// The Laplace operator's inverse row diagonals (Actual: the fast row's
// diagonal; border rows: the row on a unit probe), 0 off the active set.
__global__ void k_lap_jacobi(StencilGrid<double> g, int64_t n, const double* __restrict__ diag,
                             double* __restrict__ dinv) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
    const int row = row_of(g.kind[c]);
    double d = 0;
    if (row == ROW_ACTUAL) {
      d = diag[c];
    } else if (row != ROW_NONE) {
      const int i = (int)(c / g.s1), j = (int)((c - (int64_t)i * g.s1) / g.s2), k = (int)(c % g.s2);
      d = boundary_row_acc<double, false>(g, UnitProbe{}, i, j, k, (int)c, row);
    }
    dinv[c] = d != 0 ? 1.0 / d : 0.0;
  }
}

// The inverse row diagonals of a Laplace or advection-diffusion operator
// (the latter refreshed by xf_op_ready), for Jacobi-preconditioned BiCGStab.
int xf_op_jacobi(const xf_op* op, const double** dinv) {
  xf_ctx* ctx = op->g->ctx;
  if (op->kind == XF_OP_ADVDIFF && op->adc_valid && op->adj64) {
    *dinv = op->adj64;
    return XF_OK;
  }
  if (op->kind != XF_OP_LAPLACE)
    return xf_fail(ctx, XF_ERR_UNSUPPORTED, "xf_solve: Jacobi BiCGStab takes a Laplace or advection-diffusion operator");
  const int64_t n = op->g->ncell;
  if (!op->lap_jac_valid) {
    if (!op->adj64 && cudaMalloc(&op->adj64, n * 8) != cudaSuccess) {
      cudaGetLastError();
      return xf_fail(ctx, XF_ERR_NOMEM, "xf_solve: allocation");
    }
    StencilGrid<double> s = make_stencil_grid<double>(op->g, nullptr);
    k_lap_jacobi<<<grid_blocks(ctx, n, 256), 256, 0, ctx->stream>>>(s, n, op->g->diag, op->adj64);
    XF_CUDA(ctx, cudaGetLastError());
    op->lap_jac_valid = 1;
  }
  *dinv = op->adj64;
  return XF_OK;
}

__global__ void k_d2f(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) b[c] = (float)a[c];
}

// The FP32 copies of the advection fields, made when the first FP32 row after
// a setter asks for them (a time step's solves are FP64).
void xf_op_ready32(const xf_op* op) {
  if (op->kind != XF_OP_ADVDIFF || op->adv32_valid) return;
  xf_ctx* ctx = op->g->ctx;
  const int64_t n = op->g->ncell;
  const int bl = grid_blocks(ctx, n, 256);
  for (int d = 0; d < 3; d++) k_d2f<<<bl, 256, 0, ctx->stream>>>(op->adv64[d], op->adv32[d], n);
  if (op->adD_set) k_d2f<<<bl, 256, 0, ctx->stream>>>(op->adD64, op->adD32, n);
  op->adv32_valid = 1;
}

template <typename T>
static void launch_matvec(const xf_op* op, const T* rho, const MvReq<T>& q) {
  const xf_grid* g = op->g;
  xf_ctx* ctx = g->ctx;
  if (std::is_same<T, float>::value) xf_op_ready32(op);
  MatvecArgs<T> a;
  a.g = make_stencil_grid<T>(g, rho);
  a.x = q.x; a.y = q.y; a.y32 = q.y32; a.s = q.s; a.w = q.w; a.diag = g->diag;
  a.sign = q.sign; a.neg = q.neg; a.zero_inactive = q.zero_inactive;
  a.dot_w = q.w != nullptr; a.dot_self = q.dot_self;
  a.slot_w = q.slot; a.ctl = q.ctl; a.gate = q.gate;
  a.S = ctx->scratch;
  const int P = g->n2 * g->n3;
  const int bx = (P + MV_THREADS - 1) / MV_THREADS;
  // plane chunk: 16 planes a block where that leaves four blocks an SM, down to
  // one plane for small boxes (35 x 31 x 29: 12 blocks of 16 planes took 65 us,
  // each plane's loads behind the last plane's); longer where the partial-sum
  // table would overflow
  int chunk = (int)((int64_t)bx * g->n1 / (4 * ctx->sm_count));
  chunk = chunk < 1 ? 1 : chunk > 16 ? 16 : chunk;
  while ((int64_t)bx * ((g->n1 + chunk - 1) / chunk) > RED_MAX_BLOCKS) chunk *= 2;
  a.chunk = chunk;
  dim3 grid(bx, (g->n1 + chunk - 1) / chunk);
  const bool use_d = std::is_same<T, double>::value && op->kind == XF_OP_LAPLACE && !q.exact;
  if (op->kind == XF_OP_ADVDIFF) {
    set_ad_fields<T>(a.g, op);
    if constexpr (std::is_same<T, double>::value) {
      if (!q.exact && a.g.adc) {
        a.use = q.scaled ? op->adks : op->adk;
        a.dinv = op->adj64;
        if (q.scaled) a.g.adc = op->ads64;
        // pairs where rows are even and every vector is 16-byte aligned, faster at every size there
        const uintptr_t at = (uintptr_t)a.x | (uintptr_t)a.y | (uintptr_t)a.s | (uintptr_t)a.w | (uintptr_t)a.g.adc;
        if (g->n3 % 2 == 0 && at % 16 == 0 && (uintptr_t)a.y32 % 8 == 0)
          (q.scaled ? k_ad_fast2<true> : k_ad_fast2<false>)<<<grid_blocks(ctx, g->ncell / 2, AD_THREADS, AD2_RESIDENT),
                                                              AD_THREADS, 0, ctx->stream>>>(a);
        else
          (q.scaled ? k_ad_fast<true> : k_ad_fast<false>)<<<grid_blocks(ctx, g->ncell, AD_THREADS, AD_RESIDENT),
                                                            AD_THREADS, 0, ctx->stream>>>(a);
        return;
      }
    }
    if (q.exact) k_matvec<T, XF_OP_ADVDIFF, true, false><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
    else k_matvec<T, XF_OP_ADVDIFF, false, false><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
    return;
  }
  if (op->kind == XF_OP_LAPLACE) {
    if (q.exact) k_matvec<T, XF_OP_LAPLACE, true, false><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
    else if (use_d) k_matvec<T, XF_OP_LAPLACE, false, true><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
    else k_matvec<T, XF_OP_LAPLACE, false, false><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
  } else {
    if (q.exact) k_matvec<T, XF_OP_VARDIV, true, false><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
    else k_matvec<T, XF_OP_VARDIV, false, false><<<grid, MV_THREADS, 0, ctx->stream>>>(a);
  }
}

void xf_pack_mv64(const xf_op* op, const MvReq<double>& q);
void xf_pack_free(PackData* P);

void xf_mv64(const xf_op* op, const MvReq<double>& q) {
  if (op->kind == XF_OP_PACK) xf_pack_mv64(op, q);
  else launch_matvec<double>(op, op->rho, q);
}
// (packed operators are FP64 only: the callers refuse FP32 with them)
void xf_mv32(const xf_op* op, const MvReq<float>& q) { launch_matvec<float>(op, op->rho32, q); }

// Used by the C-ABI helpers: plain apply with an optional dot into slot.
void xf_apply_f64(const xf_op* op, const double* x, double* y, const double* s, int sign, bool exact,
                  bool zero_inactive, const double* w, int slot) {
  MvReq<double> q;
  q.x = x; q.y = y; q.s = s; q.sign = sign; q.exact = exact; q.zero_inactive = zero_inactive; q.w = w; q.slot = slot;
  xf_mv64(op, q);
}
void xf_apply_f32(const xf_op* op, const float* x, float* y, const float* s, int sign, bool zero_inactive,
                  const float* w, int slot) {
  MvReq<float> q;
  q.x = x; q.y = y; q.s = s; q.sign = sign; q.zero_inactive = zero_inactive; q.w = w; q.slot = slot;
  xf_mv32(op, q);
}

// ---------------------------------------------------------------------------
extern "C" int xf_op_create(xf_grid* g, int kind, xf_op** out) {
  if (!g || !out || (kind != XF_OP_LAPLACE && kind != XF_OP_VARDIV && kind != XF_OP_ADVDIFF))
    return xf_fail(g ? g->ctx : nullptr, XF_ERR_ARG, "xf_op_create: bad arguments");
  *out = nullptr;
  int64_t bad = -1;
  int st = xf_grid_check(g, kind, &bad);
  if (st != XF_OK) {
    const int i = (int)(bad / g->s1), j = (int)((bad / g->s2) % g->n2), k = (int)(bad % g->n3);
    return xf_fail(g->ctx, XF_ERR_MASK,
                   "operator %d is not defined at cell (%d,%d,%d): the reference throws or reads outside its arrays there",
                   kind, i, j, k);
  }
  static std::atomic<unsigned long long> serials{0};
  xf_op* op = new xf_op();
  op->g = g; op->kind = kind; op->rho = nullptr; op->rho32 = nullptr; op->rho_set = 0;
  op->serial = ++serials;
  if (kind == XF_OP_VARDIV) {
    xf_ctx* ctx = g->ctx;
    if (cudaMalloc(&op->rho, g->ncell * 8) != cudaSuccess || cudaMalloc(&op->rho32, g->ncell * 4) != cudaSuccess) {
      cudaGetLastError();
      xf_op_destroy(op);
      return xf_fail(ctx, XF_ERR_NOMEM, "xf_op_create: density allocation failed");
    }
    // The reference dereferences a null density until withDensity is called
    // (XOperator.h:422); here the operator refuses to apply until it is set.
    cudaMemsetAsync(op->rho, 0, g->ncell * 8, ctx->stream);
    cudaMemsetAsync(op->rho32, 0, g->ncell * 4, ctx->stream);
  }
  *out = op;
  return XF_OK;
}

extern "C" int xf_op_destroy(xf_op* op) {
  if (!op) return XF_ERR_ARG;
  cudaSetDevice(op->g->ctx->device);
  cudaStreamSynchronize(op->g->ctx->stream);
  if (op->rho) cudaFree(op->rho);
  if (op->rho32) cudaFree(op->rho32);
  for (int d = 0; d < 3; d++) {
    if (op->adv64[d]) cudaFree(op->adv64[d]);
    if (op->adv32[d]) cudaFree(op->adv32[d]);
  }
  if (op->adD64) cudaFree(op->adD64);
  if (op->adD32) cudaFree(op->adD32);
  if (op->adc64) cudaFree(op->adc64);
  if (op->adj64) cudaFree(op->adj64);
  if (op->ads64) cudaFree(op->ads64);
  if (op->adks) cudaFree(op->adks);
  if (op->adk) cudaFree(op->adk);
  if (op->pack) xf_pack_free(op->pack);
  if (op->host_x) xf_vec_destroy(op->host_x);
  if (op->host_b) xf_vec_destroy(op->host_b);
  delete op;
  return XF_OK;
}

extern "C" int xf_op_set_density(xf_op* op, const double* host_rho) {
  if (!op || !host_rho) return XF_ERR_ARG;
  xf_ctx* ctx = op->g->ctx;
  if (op->kind != XF_OP_VARDIV) return xf_fail(ctx, XF_ERR_STATE, "xf_op_set_density: not a variable-density operator");
  const int64_t n = op->g->ncell;
  XF_CUDA(ctx, cudaMemcpyAsync(op->rho, host_rho, n * 8, cudaMemcpyHostToDevice, ctx->stream));
  k_d2f<<<grid_blocks(ctx, n, 256), 256, 0, ctx->stream>>>(op->rho, op->rho32, n);
  XF_CUDA(ctx, cudaGetLastError());
  XF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  op->rho_set = 1;
  return XF_OK;
}

extern "C" int xf_op_set_advection(xf_op* op, const xf_vec* u, const xf_vec* v, const xf_vec* w, double tau,
                                   double diff_coef, int flags) {
  if (!op) return XF_ERR_ARG;
  xf_ctx* ctx = op->g->ctx;
  if (op->kind != XF_OP_ADVDIFF) return xf_fail(ctx, XF_ERR_STATE, "xf_op_set_advection: not an advection-diffusion operator");
  if (!(tau != 0) || (flags & ~(XF_ADV_CONVECTIVE | XF_ADV_DIFFUSIVE | XF_ADV_UPWIND)))
    return xf_fail(ctx, XF_ERR_ARG, "xf_op_set_advection: tau must be nonzero and flags XF_ADV_*");
  const xf_vec* vel[3] = {u, v, w};
  for (int d = 0; d < 3; d++)
    if (vel[d] && (vel[d]->g != op->g || vel[d]->dtype != XF_F64))
      return xf_fail(ctx, XF_ERR_STATE, "xf_op_set_advection: velocities must be FP64 boxes of the operator's grid");
  XF_CUDA(ctx, cudaSetDevice(ctx->device));
  const int64_t n = op->g->ncell;
  op->adc_valid = 0;
  const int64_t nax = 5 * ((int64_t)op->g->n1 + op->g->n2 + op->g->n3);   // per-axis factors after the table
  if ((!op->adc64 && cudaMalloc(&op->adc64, (7 * n + nax) * 8) != cudaSuccess) ||
      (!op->adk && cudaMalloc(&op->adk, n) != cudaSuccess) ||
      (!op->adj64 && cudaMalloc(&op->adj64, n * 8) != cudaSuccess)) {
    cudaGetLastError();
    return xf_fail(ctx, XF_ERR_NOMEM, "xf_op_set_advection: allocation");
  }
  for (int d = 0; d < 3; d++) {
    if (!op->adv64[d] && (cudaMalloc(&op->adv64[d], n * 8) != cudaSuccess ||
                          cudaMalloc(&op->adv32[d], n * 4) != cudaSuccess)) {
      cudaGetLastError();
      return xf_fail(ctx, XF_ERR_NOMEM, "xf_op_set_advection: allocation");
    }
    if (vel[d]) XF_CUDA(ctx, cudaMemcpyAsync(op->adv64[d], vel[d]->data, n * 8, cudaMemcpyDeviceToDevice, ctx->stream));
    else XF_CUDA(ctx, cudaMemsetAsync(op->adv64[d], 0, n * 8, ctx->stream));
  }
  op->adv32_valid = 0;
  op->ad_tau = tau;
  op->ad_D = diff_coef;
  op->ad_flags = flags;
  op->adv_set = 1;
  return XF_OK;
}

extern "C" int xf_op_set_diffusion_field(xf_op* op, const xf_vec* d) {
  if (!op) return XF_ERR_ARG;
  xf_ctx* ctx = op->g->ctx;
  if (op->kind != XF_OP_ADVDIFF)
    return xf_fail(ctx, XF_ERR_STATE, "xf_op_set_diffusion_field: not an advection-diffusion operator");
  op->adc_valid = 0;
  if (!d) {
    op->adD_set = 0;
    return XF_OK;
  }
  if (d->g != op->g || d->dtype != XF_F64)
    return xf_fail(ctx, XF_ERR_STATE, "xf_op_set_diffusion_field: an FP64 box of the operator's grid expected");
  XF_CUDA(ctx, cudaSetDevice(ctx->device));
  const int64_t n = op->g->ncell;
  if (!op->adD64 && (cudaMalloc(&op->adD64, n * 8) != cudaSuccess || cudaMalloc(&op->adD32, n * 4) != cudaSuccess)) {
    cudaGetLastError();
    return xf_fail(ctx, XF_ERR_NOMEM, "xf_op_set_diffusion_field: allocation");
  }
  XF_CUDA(ctx, cudaMemcpyAsync(op->adD64, d->data, n * 8, cudaMemcpyDeviceToDevice, ctx->stream));
  op->adv32_valid = 0;
  op->adD_set = 1;
  return XF_OK;
}

int xf_op_ready(const xf_op* op) {
  if (op->kind == XF_OP_ADVDIFF && !op->adv_set)
    return xf_fail(op->g->ctx, XF_ERR_STATE, "advection-diffusion operator used before xf_op_set_advection");
  if (op->kind == XF_OP_ADVDIFF && !op->adc_valid && op->adc64) {   // refresh the coefficient table
    xf_ctx* ctx = op->g->ctx;
    XF_CUDA(ctx, cudaSetDevice(ctx->device));
    const xf_grid* g = op->g;
    StencilGrid<double> s = make_stencil_grid<double>(g, nullptr);
    op->adc_valid = 0;
    set_ad_fields<double>(s, op);
    const int64_t n = g->ncell;
    double* tx = op->adc64 + 7 * n;   // the axis factors sit after the table
    double* ty = tx + 5 * g->n1;
    double* tz = ty + 5 * g->n2;
    const double conv = s.ad_conv, diff = s.ad_diff;
    k_ad_axis<<<1, 256, 0, ctx->stream>>>(g->hx, g->n1, conv, diff, tx);
    k_ad_axis<<<1, 256, 0, ctx->stream>>>(g->hy, g->n2, conv, diff, ty);
    k_ad_axis<<<1, 256, 0, ctx->stream>>>(g->hz, g->n3, conv, diff, tz);
    const dim3 grid((unsigned)((g->s1 + ADC_THREADS - 1) / ADC_THREADS), (g->n1 + ADC_CHUNK - 1) / ADC_CHUNK);
    if (s.ad_upwind) k_ad_coeffs<true><<<grid, ADC_THREADS, 0, ctx->stream>>>(s, n, tx, ty, tz, op->adc64, op->adk, op->adj64);
    else k_ad_coeffs<false><<<grid, ADC_THREADS, 0, ctx->stream>>>(s, n, tx, ty, tz, op->adc64, op->adk, op->adj64);
    XF_CUDA(ctx, cudaGetLastError());
    op->adc_valid = 1;
    op->ads_valid = 0;
  }
  if (op->kind == XF_OP_VARDIV && !op->rho_set)
    return xf_fail(op->g->ctx, XF_ERR_STATE, "variable-density operator used before xf_op_set_density");
  return XF_OK;
}

static int check_vec(const xf_op* op, const xf_vec* v, const char* what) {
  if (!v) return xf_fail(op->g->ctx, XF_ERR_ARG, "%s: null vector", what);
  if (v->g != op->g) return xf_fail(op->g->ctx, XF_ERR_STATE, "%s: vector of another grid", what);
  return XF_OK;
}

extern "C" int xf_matvec(xf_op* op, const xf_vec* x, xf_vec* y, const xf_vec* s, int sign, int flags,
                         const xf_vec* opt_w, double* opt_dot) {
  if (!op) return XF_ERR_ARG;
  xf_ctx* ctx = op->g->ctx;
  int st;
  if ((st = check_vec(op, x, "xf_matvec x")) || (st = check_vec(op, y, "xf_matvec y"))) return st;
  if (sign != 0 && (st = check_vec(op, s, "xf_matvec s"))) return st;
  if (x == y) return xf_fail(ctx, XF_ERR_ARG, "xf_matvec: x and y must differ");
  if ((st = xf_op_ready(op))) return st;
  if (x->dtype != y->dtype || (sign != 0 && s->dtype != x->dtype))
    return xf_fail(ctx, XF_ERR_STATE, "xf_matvec: mixed dtypes");
  const bool exact = (flags & XF_EXACT) != 0;
  if (exact && x->dtype != XF_F64) return xf_fail(ctx, XF_ERR_UNSUPPORTED, "xf_matvec: XF_EXACT needs FP64 vectors");
  if (op->kind == XF_OP_PACK && x->dtype != XF_F64)
    return xf_fail(ctx, XF_ERR_UNSUPPORTED, "xf_matvec: packed operators are FP64");
  const xf_vec* w = opt_dot ? (opt_w ? opt_w : x) : nullptr;
  if (w && (st = check_vec(op, w, "xf_matvec w"))) return st;
  if (w && w->dtype != x->dtype) return xf_fail(ctx, XF_ERR_STATE, "xf_matvec: dot partner dtype");
  XF_CUDA(ctx, cudaSetDevice(ctx->device));
  const int slot = 0;
  if (x->dtype == XF_F64)
    xf_apply_f64(op, (const double*)x->data, (double*)y->data, s ? (const double*)s->data : nullptr, sign, exact,
                 (flags & XF_ZERO_INACTIVE) != 0, w ? (const double*)w->data : nullptr, slot);
  else
    xf_apply_f32(op, (const float*)x->data, (float*)y->data, s ? (const float*)s->data : nullptr, sign,
                 (flags & XF_ZERO_INACTIVE) != 0, w ? (const float*)w->data : nullptr, slot);
  XF_CUDA(ctx, cudaGetLastError());
  if (opt_dot) {
    XF_CUDA(ctx, cudaMemcpyAsync(ctx->host_scalars, &ctx->scratch->scalars[slot], 8, cudaMemcpyDeviceToHost, ctx->stream));
    XF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *opt_dot = ctx->host_scalars[0];
  }
  return XF_OK;
}
