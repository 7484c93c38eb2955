// Per-element passes of one tendency evaluation + stage update, shared by
// the single-instance kernels (swg_kernels.cu) and the batched persistent
// kernel (swg_batch.cu).  Each function handles one flat index i of its pass
// domain: (entity, level) with the level fastest.  Callers guarantee i is in
// range (pt_aux2: i < (V + C) K, vertices first).
#pragma once

#include "swg_internal.h"

#include <type_traits>

namespace swg {

// Shape of the kernels that run the fixed-point sums: blocks of two warps,
// and the minimum of resident blocks that bounds their registers.  The sums
// hold many operands, so few warps fit an SM; small blocks replace finished
// warps at once instead of waiting for a block of eight, whose warps load
// and compute in step.
constexpr int HTPB = 64;
constexpr int HEAVY_AUX2_BLOCKS = 20, HEAVY_EDGE_BLOCKS = 12,
              HEAVY_CELL_BLOCKS = 10;

// a + b and a b as multiply-adds with every operand in a register, which issue at
// 1.90 per SM per clock: 1.60 with an operand from the constant bank or a
// uniform register (kernel parameters, literals), and as additions and
// products by themselves.  a 1 + b and a b + (-0) are the sum and the product
// to the last bit; 1 and -0 come from memory.  For the passes that are FP64
// throughout, up to half of whose instructions are sums and products: k_edge1
// 228 -> 215 us at 256x256x64 and 20.4 -> 18.5 at 64x64x64, the RK4 step of
// 200x230 cells with one level 105 -> 98, the tangent-linear step of 96x80x32
// 795 -> 758.  In the passes with fixed-point sums the registers cost more
// (k_edge_final 499 -> 514 us).
static __device__ double2 fp64_units = {1.0, -0.0};
__device__ __forceinline__ double fma_reg(double a, double b, double c) {
  double r;
  asm("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(a), "d"(b), "d"(c));
  return r;
}
__device__ __forceinline__ double mul_reg(double a, double b) {
  return fma_reg(a, b, __ldg(&fp64_units).y);
}
__device__ __forceinline__ double add_reg(double a, double b) {
  return fma_reg(a, __ldg(&fp64_units).x, b);
}
// Forward-mode dual number (value, tangent): the pass functions instantiated
// with it are the exact tangent-linear model of the double instantiation
// (the value part computes each sum in FP64, where the double instantiation
// may take it in fixed point).
using ::fma; // keep the double overload visible beside the Dual ones
__device__ __forceinline__ Dual operator+(Dual a, Dual b) {
  return {add_reg(a.v, b.v), add_reg(a.d, b.d)};
}
__device__ __forceinline__ Dual operator+(Dual a, double b) { return {add_reg(a.v, b), a.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) {
  return {add_reg(a.v, -b.v), add_reg(a.d, -b.d)};
}
__device__ __forceinline__ Dual operator-(Dual a) { return {-a.v, -a.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) {
  return {mul_reg(a.v, b.v), fma(a.d, b.v, mul_reg(a.v, b.d))};
}
__device__ __forceinline__ Dual operator*(double a, Dual b) {
  return {mul_reg(a, b.v), mul_reg(a, b.d)};
}
__device__ __forceinline__ Dual operator*(Dual a, double b) { return b * a; }
__device__ __forceinline__ Dual &operator+=(Dual &a, Dual b) { a = a + b; return a; }
__device__ __forceinline__ Dual fma(double a, Dual b, Dual c) {
  return {::fma(a, b.v, c.v), ::fma(a, b.d, c.d)};
}
__device__ __forceinline__ Dual fma(Dual a, double b, Dual c) {
  return {::fma(a.v, b, c.v), ::fma(a.d, b, c.d)};
}
__device__ __forceinline__ Dual fma(Dual a, Dual b, Dual c) {
  return {::fma(a.v, b.v, c.v), ::fma(a.d, b.v, ::fma(a.v, b.d, c.d))};
}

// a b and a + b that the compiler may not fuse into multiply-adds: where a
// product is both used and summed, it could otherwise do so differently in
// the single-instance and the batched kernels, which must agree bit for bit
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ Dual mul_rn(double a, Dual b) { return a * b; }
__device__ __forceinline__ Dual add_rn(Dual a, Dual b) { return a + b; }

template <class A, class B>
__device__ __forceinline__ Dual mul_reg(A a, B b) { return a * b; }
template <class B>
__device__ __forceinline__ Dual add_reg(Dual a, B b) { return a + b; }

// 1/x: hardware estimate r refined by one third-order step: with the residual
// e = 1 - x r, 1/x = r / (1 - e) = r (1 + e + e^2 + ...), so r + r (e + e^2)
// has the relative error e^3 (the estimate's cubed) before its one rounding.
// Three FP64 instructions; two Newton steps take four.
// The estimate is the .ftz form: a subnormal input (|x| < 2^-1022) counts as
// zero (result infinite) and a result below 2^-1022 flushes to zero, so the
// function is for |x| in [2^-1022, 2^1022], far beyond any thickness.  On
// the GPU it is within 1 ulp of the correctly rounded 1.0 / x over 1e-6 ..
// 1e6 and random mantissas in [2^-40, 2^40] (tests/cpp/rcp_accuracy.cu).
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, __ldg(&fp64_units).x);
  return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ Dual rcp_nr(Dual x) {
  const double r = rcp_nr(x.v);
  return {r, -(r * r) * x.d};
}

// x / 2 and 2 x through the exponent field (exact, as the products are): an
// integer addition instead of an FP64 instruction.  Zeros, subnormals, the
// ends of the range, infinities and NaN take the product, out of line so that
// it is not issued with the predicate off.
static __device__ __noinline__ double times_rare(double x, double c) {
  return c * x;
}
__device__ __forceinline__ double half_of(double x) {
  const int hi = __double2hiint(x);
  if ((unsigned(hi) & 0x7ff00000u) - 0x00200000u > 0x7fc00000u)
    return times_rare(x, 0.5);
  return __hiloint2double(hi - 0x00100000, __double2loint(x));
}
__device__ __forceinline__ double twice(double x) {
  const int hi = __double2hiint(x);
  if ((unsigned(hi) & 0x7ff00000u) - 0x00100000u > 0x7fc00000u)
    return times_rare(x, 2.0);
  return __hiloint2double(hi + 0x00100000, __double2loint(x));
}
__device__ __forceinline__ Dual half_of(Dual x) { return 0.5 * x; }
__device__ __forceinline__ Dual twice(Dual x) { return 2.0 * x; }

using ::sqrt;
__device__ __forceinline__ Dual sqrt(Dual x) {
  const double s = ::sqrt(x.v);
  return {s, x.d * (0.5 / s)};
}

// The stage update in two parts, so that a pass can issue its loads with the
// others, ahead of the arithmetic: what mode `ep` reads of element i, and the
// update with the tendency x.
template <class T> struct EpiIn {
  T u{}, v{};
};
template <class T>
__device__ __forceinline__ void
epilogue_operands(const Epilogue &ep, const FieldIOT<T> &f, const T *&u,
                  const T *&v) {
  u = v = nullptr;
  switch (ep.mode) {
  case EPI_REPLACE: break;
  case EPI_INCREMENT: u = f.tend; break;
  case EPI_LSRK: u = f.tend, v = f.out; break;
  case EPI_LSRK_TEND: u = f.tend; break;
  case EPI_RK4_FIRST: v = f.old; break;
  case EPI_RK4_MID: u = f.acc, v = f.old; break;
  default: u = f.acc; break;
  }
}
template <class T>
__device__ __forceinline__ EpiIn<T> epilogue_in(const Epilogue &ep,
                                                const FieldIOT<T> &f,
                                                size_t i) {
  const T *u, *v;
  epilogue_operands(ep, f, u, v);
  EpiIn<T> r;
  if (u)
    r.u = u[i];
  if (v)
    r.v = v[i];
  return r;
}
template <class T>
__device__ __forceinline__ void epilogue(const Epilogue &ep,
                                         const FieldIOT<T> &f, size_t i, T x,
                                         const EpiIn<T> &in) {
  switch (ep.mode) {
  case EPI_REPLACE:
    f.tend[i] = x;
    break;
  case EPI_INCREMENT:
    f.tend[i] = in.u + x;
    break;
  case EPI_LSRK: {
    const T t = fma(ep.a, in.u, x);
    f.tend[i] = t;
    f.out[i] = fma(ep.dtb, t, in.v);
  } break;
  case EPI_LSRK_TEND:
    f.tend[i] = fma(ep.a, in.u, x);
    break;
  case EPI_RK4_FIRST:
    f.acc[i] = fma(ep.dtb, x, in.v);
    f.out[i] = fma(ep.dta, x, in.v);
    break;
  case EPI_RK4_MID:
    f.acc[i] = fma(ep.dtb, x, in.u);
    f.out[i] = fma(ep.dta, x, in.v);
    break;
  default: // EPI_RK4_LAST
    f.out[i] = fma(ep.dtb, x, in.u);
    break;
  }
}
// both at once, each mode loading what it needs
template <class T>
__device__ __forceinline__ void epilogue(const Epilogue &ep,
                                         const FieldIOT<T> &f, size_t i, T x) {
  switch (ep.mode) {
  case EPI_REPLACE:
    f.tend[i] = x;
    break;
  case EPI_INCREMENT:
    f.tend[i] += x;
    break;
  case EPI_LSRK: {
    const T t = fma(ep.a, f.tend[i], x);
    f.tend[i] = t;
    f.out[i] = fma(ep.dtb, t, f.out[i]);
  } break;
  case EPI_LSRK_TEND:
    f.tend[i] = fma(ep.a, f.tend[i], x);
    break;
  case EPI_RK4_FIRST: {
    const T s = f.old[i];
    f.acc[i] = fma(ep.dtb, x, s);
    f.out[i] = fma(ep.dta, x, s);
  } break;
  case EPI_RK4_MID:
    f.acc[i] = fma(ep.dtb, x, f.acc[i]);
    f.out[i] = fma(ep.dta, x, f.old[i]);
    break;
  default: // EPI_RK4_LAST
    f.out[i] = fma(ep.dtb, x, f.acc[i]);
    break;
  }
}

// ---- sums of doubles over an entity's neighbours, fixed-point
//
// One entity's terms from a table: N slots from `tab`, the field x.
template <int N>
__device__ __forceinline__ double raw_sum(const FxSlot *tab, const double *x,
                                          unsigned K, unsigned k, bool &slow) {
  Wt w[N];
  double v[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int4 t = __ldg(reinterpret_cast<const int4 *>(tab) + j);
    w[j] = {t.y, t.z, t.w};
    v[j] = x[unsigned(t.x) * K + k];
  }
  return fx_raw_sum(w, v, slow);
}
// the same in FP64, for terms the fixed-point sum leaves to it (out of line:
// see times_rare)
static __device__ __noinline__ double dot_f64(const double *coef,
                                              const int *idx, int n,
                                              const double *x, int K, int k) {
  double t = __ldg(coef) * x[size_t(__ldg(idx)) * K + k];
  for (int j = 1; j < n; ++j)
    t = fma(__ldg(coef + j), x[size_t(__ldg(idx + j)) * K + k], t);
  return t;
}
// sum_j coef_j x_(idx_j) over the N terms of entity c: RAW fixed-point from
// the table tab (1), in FP64 (0), or as the model's RAW_* bit BIT says (-1)
template <int N, int RAW, int BIT, class T>
__device__ __forceinline__ T entity_sum(const ModelView &p, const FxSlot *tab,
                                        const double *coef, const int *idx,
                                        int c, const T *x, int K, int k) {
  if constexpr (std::is_same<T, double>::value && RAW != 0) {
    if (RAW == 1 || (p.raw & BIT)) {
      bool slow = false;
      double t = raw_sum<N>(tab + N * c, x, unsigned(K), unsigned(k), slow);
      if (slow)
        t = dot_f64(coef + N * c, idx + N * c, N, x, K, k);
      return t;
    }
  }
  T t = mul_reg(__ldg(coef + N * c), x[size_t(__ldg(idx + N * c)) * K + k]);
#pragma unroll
  for (int j = 1; j < N; ++j)
    t = fma(__ldg(coef + N * c + j), x[size_t(__ldg(idx + N * c + j)) * K + k],
            t);
  return t;
}

// Vertex pass: relative vorticity and (rvort + f) / h_vertex.
template <class T, int RAW = -1>
__device__ __forceinline__ void
pt_vertex(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
          const T *__restrict__ h, const T *__restrict__ vn, unsigned i) {
  const int K = m.nlayers;
  const int v = int(i / unsigned(K)), k = int(i - unsigned(v) * unsigned(K));
  const T hv = entity_sum<3, RAW, RAW_VERTEX>(p, m.kvx, m.kvh, m.cv, v, h, K, k);
  const T z = entity_sum<3, RAW, RAW_VERTEX>(p, m.cvx, m.cvr, m.ev, v, vn, K, k);
  const T r = rcp_nr(hv);
  a.q[i] = mul_reg(add_reg(z, __ldg(p.f_vertex + v)), r);
  if (a.rhv)
    a.rhv[i] = r;
  if (p.vel_del2 | p.vel_del4)
    a.zeta[i] = z;
}

// Cell pass 1: velocity divergence (for the dissipation terms) and the
// normalised tracers tr / h.
template <class T, int RAW = -1>
__device__ __forceinline__ void
pt_cell1(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
         const T *__restrict__ h, const T *__restrict__ vn,
         const T *__restrict__ tr, unsigned i) {
  const int K = m.nlayers;
  const unsigned CK = unsigned(m.ncells) * unsigned(K);
  const int c = int(i / unsigned(K)), k = int(i - unsigned(c) * unsigned(K));
  if (p.do_vn && (p.vel_del2 | p.vel_del4)) {
    a.div[i] = entity_sum<MAXE, RAW, RAW_DIV>(p, m.cdx, m.ccd, m.ec, c, vn, K, k);
  }
  if (p.ntracers > 0) {
    const T r = rcp_nr(h[i]);
    if (a.rh)
      a.rh[i] = r;
    for (int l = 0; l < p.ntracers; ++l) {
      const size_t t = size_t(l) * CK + i;
      const T n = mul_reg(tr[t], r);
      a.ntr[t] = n;
      if constexpr (std::is_same<T, double>::value)
        if (a.nx)
          a.nx[t] = fx_word(n);
    }
  }
}

// What the PV sums read of edge element i: G = F Q, or the words of F and
// F Q where the sums are fixed-point.
template <class T>
__device__ __forceinline__ void store_pv(const AuxViewT<T> &a, unsigned i, T F,
                                         T Q) {
  if constexpr (std::is_same<T, double>::value)
    if (a.FGx) {
      reinterpret_cast<ulonglong2 *>(a.FGx)[i] =
          make_ulonglong2(fx_word<FX_PV_MINQ>(F),
                          fx_word<FX_PV_MINQ>(mul_reg(F, Q)));
      return;
    }
  a.G[i] = mul_reg(F, Q);
}

// Edge pass 1: mean thickness, thickness flux F = mean_h vn, vn^2, edge PV
// sum Q = q(v0) + q(v1), G = F Q, and the edge Laplacian of the velocity.
template <class T>
__device__ __forceinline__ void
pt_edge1(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
         const T *__restrict__ h, const T *__restrict__ vn, unsigned i) {
  const int K = m.nlayers;
  const int e = int(i / unsigned(K)), k = int(i - unsigned(e) * unsigned(K));
  const int c0 = __ldg(m.ce + 2 * e), c1 = __ldg(m.ce + 2 * e + 1);
  const T mh = half_of(add_reg(h[size_t(c0) * K + k], h[size_t(c1) * K + k]));
  const T u = vn[i];
  const T F = mul_reg(mh, u);
  a.F[i] = F;
  if (a.mh) // kept by every nonlinear model and in the adjoint's tape
    a.mh[i] = mh;
  if (p.do_vn) {
    const int v0 = __ldg(m.ve + 2 * e), v1 = __ldg(m.ve + 2 * e + 1);
    const T Q = add_reg(a.q[size_t(v0) * K + k], a.q[size_t(v1) * K + k]);
    a.Q[i] = Q;
    store_pv(a, i, F, Q);
    a.u2[i] = mul_reg(u, u);
    if (p.vel_del2 | p.vel_del4) {
      const T dd = add_reg(a.div[size_t(c1) * K + k], -a.div[size_t(c0) * K + k]);
      const T dz =
          add_reg(a.zeta[size_t(v1) * K + k], -a.zeta[size_t(v0) * K + k]);
      const double idc = __ldg(m.inv_dc + e);
      a.d2u[i] = fma(dd, idc, -mul_reg(dz, __ldg(m.inv_dv + e)));
      if (p.vel_del4 && m.dv4_differs)
        a.d2u4[i] = fma(dd, idc, -mul_reg(dz, __ldg(m.inv_dv4 + e)));
    }
  }
}

__device__ __forceinline__ void copy_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   unsigned(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
// What the fixed-point sums of the passes below leave to FP64: elements with
// a value or weight they cannot represent (NaN, infinities, magnitudes
// beyond their range).  Out of line, so that the passes keep neither their
// registers nor predicated-off FP64 instructions.  A run that has blown up
// gets here with every element, so the weights are formed once per cell, and a
// pass takes no sums whose shared operands say so already (Euler step, all
// NaN, 63x64x32, 7 tracers: 272 us with neither, 184 with both; FP64 alone
// 131, finite values 107).

// thickness-weighted Laplacians of the tracers at cell c
static __device__ __noinline__ void laplacians_f64(const MeshView &m,
                                                   const ModelView &p,
                                                   const AuxView &a, int c,
                                                   int k) {
  const int K = m.nlayers;
  const unsigned CK = unsigned(m.ncells) * unsigned(K);
  const size_t i = size_t(c) * K + k;
  double w[MAXE], M = 0;
  unsigned off[MAXE];
#pragma unroll
  for (int j = 0; j < MAXE; ++j) {
    w[j] = __ldg(m.ckq + 6 * c + j) *
           a.mh[size_t(__ldg(m.ec + 6 * c + j)) * K + k];
    M += w[j];
    off[j] = unsigned(__ldg(m.nbc + 6 * c + j)) * unsigned(K) + unsigned(k);
  }
#pragma unroll 1
  for (int l = 0; l < p.ntracers; ++l) {
    const double *n = a.ntr + size_t(l) * CK;
    double acc = 0;
#pragma unroll
    for (int j = 0; j < MAXE; ++j)
      acc = fma(w[j], n[off[j]], acc);
    const double L = fma(-M, n[i], acc);
    a.lap[size_t(l) * CK + i] = L;
    a.lx[size_t(l) * CK + i] = fx_word(L);
  }
}

// the PV flux Q_e sum_j w_j F_j + sum_j w_j F_j Q_j of edge e; S1 is taped
template <int NE>
static __device__ __noinline__ double pv_flux_f64(const MeshView &m,
                                                  const AuxView &a, int e,
                                                  int k) {
  const int K = m.nlayers;
  const size_t i = size_t(e) * K + k;
  double S1 = 0, S2 = 0;
#pragma unroll
  for (int j = 0; j < NE; ++j) {
    const size_t ij = size_t(__ldg(m.eoe + NE * e + j)) * K + k;
    const double w = __ldg(m.woe + NE * e + j);
    S1 = fma(w, a.F[ij], S1);
    S2 = fma(w, a.F[ij] * a.Q[ij], S2);
  }
  if (a.S1)
    a.S1[i] = S1;
  return fma(a.Q[i], S1, S2);
}

// Whether a tracer's sum over the words n (and with del4 L) of the neighbours
// is left to FP64: the decision of fx_sum, from the same weights.  Not an extra
// register of the tracer loop: there a mask of the tracers costs more than
// reading the words again here (k_cell_tracers with 8 tracers 630 -> 700 us at
// 256x256x64).
__device__ __forceinline__ bool
tracer_left(const fx_t *n, const fx_t *L, bool del4, const double (&w)[MAXE],
            const double (&r4)[MAXE], const unsigned (&off)[MAXE]) {
  fx_t x[MAXE], y[MAXE];
  unsigned f = 0, unused = 0;
#pragma unroll
  for (int j = 0; j < MAXE; ++j) {
    x[j] = n[off[j]];
    y[j] = del4 ? L[off[j]] : 0;
    f |= unsigned(x[j]) | unsigned(y[j]);
  }
  if (f & FX_FLAG)
    return true;
  int P = FX_ZERO_EXP;
#pragma unroll
  for (int j = 0; j < MAXE; ++j) {
    P = max(P, fx_exp(x[j], fx_weight<FX_TOP>(w[j], unused).e));
    if (del4)
      P = max(P, fx_exp(y[j], fx_weight<FX_TOP>(r4[j], unused).e));
  }
  return fx_left(P, FX_TOP, f) != 0;
}

// flux divergence, diffusion and hyperdiffusion at cell c, and the stage
// update, of every tracer (all) or of those that tracer_sums left here: the
// weights w are its own to the last bit
static __device__ __noinline__ void tracers_f64(const MeshView &m,
                                                const ModelView &p,
                                                const AuxView &a,
                                                const StageArgs &s, int c,
                                                int k, bool all) {
  const int K = m.nlayers;
  const size_t i = size_t(c) * K + k;
  const bool fold = p.tr_del2 && p.tr_del4 && p.r4f;
  double w[MAXE], r4[MAXE], wc = 0, rc = 0;
  unsigned off[MAXE];
#pragma unroll
  for (int j = 0; j < MAXE; ++j) {
    const size_t ie = size_t(__ldg(m.ec + 6 * c + j)) * K + k;
    off[j] = unsigned(__ldg(m.nbc + 6 * c + j)) * unsigned(K) + unsigned(k);
    w[j] = r4[j] = 0;
    if (!p.off_tr_hadv) {
      w[j] = mul_rn(__ldg(m.ccdh + 6 * c + j), a.F[ie]);
      wc += w[j];
    }
    if (p.tr_del2 && !fold) {
      const double b = mul_rn(__ldg(p.kd2 + 6 * c + j), a.mh[ie]);
      w[j] = add_rn(w[j], b);
      wc -= b;
    }
    if (p.tr_del4)
      r4[j] = __ldg(p.r4 + 6 * c + j);
  }
  if (p.tr_del4)
    rc = fold ? __ldg(p.r4f + c) : -__ldg(p.r4sum + c);
#pragma unroll 1
  for (int l = 0; l < p.ntracers; ++l) {
    const size_t base = size_t(l) * (unsigned(m.ncells) * unsigned(K));
    if (!all &&
        !tracer_left(a.nx + base, a.lx + base, p.tr_del4, w, r4, off))
      continue;
    const double *n = a.ntr + base, *L = a.lap + base;
    double acc = 0;
#pragma unroll
    for (int j = 0; j < MAXE; ++j)
      acc = fma(w[j], n[off[j]], acc);
    acc = fma(wc, n[i], acc);
    if (p.tr_del4) {
      acc = fma(rc, L[i], acc);
#pragma unroll
      for (int j = 0; j < MAXE; ++j)
        acc = fma(r4[j], L[off[j]], acc);
    }
    epilogue(s.ep, s.ftr, base + i, acc);
  }
}

// Second auxiliary pass: kinetic energy (cells), curl (vertices) and
// divergence (cells) of the edge Laplacian, and the thickness-weighted
// tracer Laplacian L (cells).  The first V*K threads take vertices, the
// rest cells.  TR4: no tracer Laplacian (0), with it in FP64 (1) or by
// fixed-point sums (2, the model keeps the words), in FP64 if at all (-2), or
// as the model says (-1).
template <class T, int TR4 = -1>
__device__ __forceinline__ void pt_aux2(const MeshView &m, const ModelView &p,
                                        const AuxViewT<T> &a, unsigned i) {
  const int K = m.nlayers;
  const unsigned VK = unsigned(m.nvertices) * unsigned(K);
  const unsigned CK = unsigned(m.ncells) * unsigned(K);
  const bool vel = p.do_vn && p.vel_del4;
  if (i < VK) {
    if (!vel)
      return;
    const int v = int(i / unsigned(K)), k = int(i - unsigned(v) * unsigned(K));
    a.z4[i] = entity_sum<3, 0, 0>(p, nullptr, m.cvr, m.ev, v, a.d2u4, K, k);
    return;
  }
  i -= VK;
  if (i >= CK)
    return;
  const int c = int(i / unsigned(K)), k = int(i - unsigned(c) * unsigned(K));
  const bool tr4 = TR4 < 0 ? p.ntracers > 0 && p.tr_del4 : TR4 != 0;
  if (p.do_vn) {
    // ke = sum_j dv dc / (4 area) vn_j^2
    a.ke[i] = entity_sum<MAXE, 0, 0>(p, nullptr, m.cke, m.ec, c, a.u2, K, k);
  }
  if (vel)
    a.d4[i] = entity_sum<MAXE, 0, 0>(p, nullptr, m.ccd, m.ec, c, a.d2u4, K, k);
  if (tr4) {
    // L = sum_j w_j (n_nb - n_c), w_j = ckq_j mean_h_j
    T w[MAXE], M;
    int nb[MAXE];
#pragma unroll
    for (int j = 0; j < MAXE; ++j) {
      w[j] = mul_rn(__ldg(m.ckq + 6 * c + j),
                    a.mh[size_t(__ldg(m.ec + 6 * c + j)) * K + k]);
      nb[j] = __ldg(m.nbc + 6 * c + j);
    }
    M = add_rn(w[0], w[1]);
#pragma unroll
    for (int j = 2; j < MAXE; ++j)
      M = add_rn(M, w[j]);
    constexpr bool FX =
        std::is_same<T, double>::value && (TR4 == 2 || TR4 == -1);
    const bool fx = FX && (TR4 == 2 || a.lx);
    if constexpr (FX) if (fx) {
      // one seven-term fixed-point sum per tracer
      unsigned bad = 0;
      Wt W[MAXE + 1];
      long long start = 0;
#pragma unroll
      for (int j = 0; j <= MAXE; ++j) {
        W[j] = fx_weight<FX_TOP>(j < MAXE ? w[j < MAXE ? j : 0] : -M, bad);
        start += W[j].hi;
      }
      start = fx_start(start);
      unsigned redo = bad;
      if (!bad) {
        unsigned off[MAXE + 1];
#pragma unroll
        for (int j = 0; j < MAXE; ++j)
          off[j] = unsigned(nb[j]) * unsigned(K) + unsigned(k);
        off[MAXE] = i;
#pragma unroll 1
        for (int l = 0; l < p.ntracers; ++l) {
          const size_t base = size_t(l) * CK;
          const fx_t *n = a.nx + base;
          fx_t x[MAXE + 1];
#pragma unroll
          for (int j = 0; j <= MAXE; ++j)
            x[j] = n[off[j]];
          const double L =
              fx_sum<MAXE + 1, FX_LEAVE>(W, x, start, FX_TOP, redo);
          a.lap[base + i] = L;
          a.lx[base + i] = fx_word(L);
        }
      }
      if (redo)
        laplacians_f64(m, p, a, c, k);
    }
    if (!fx) {
      for (int l = 0; l < p.ntracers; ++l) {
        const T *n = a.ntr + size_t(l) * CK;
        T acc = w[0] * n[size_t(nb[0]) * K + k];
#pragma unroll
        for (int j = 1; j < MAXE; ++j)
          acc = fma(w[j], n[size_t(nb[j]) * K + k], acc);
        a.lap[size_t(l) * CK + i] = fma(-M, n[i], acc);
      }
    }
  }
}

// Bottom drag -c_d sqrt(ke_0 + ke_1) vn / mean_h added to t on the lowest
// level (the term commented out at shallow_water_hierarchical.cpp:479-486),
// with the auxiliary state's mean thickness (h_drag_edge = h_mean).  Out of
// line: inlined, the short branch was if-converted, and every edge of every
// model without drag issued its FP64 instructions with the predicate off.
template <class T>
__device__ __noinline__ T drag_add(const MeshView &m, const ModelView &p,
                                   const AuxViewT<T> &a,
                                   const StageArgsT<T> &s, int c0, int c1,
                                   size_t i, int k, T t) {
  const int K = m.nlayers;
  const T hm = a.mh ? a.mh[i]
                    : 0.5 * (s.h[size_t(c0) * K + k] + s.h[size_t(c1) * K + k]);
  const T ks = a.ke[size_t(c0) * K + k] + a.ke[size_t(c1) * K + k];
  return t + (-p.drag_coeff * sqrt(ks)) * s.vn[i] * rcp_nr(hm);
}

// The del2 and del4 velocity dissipation of edge element i with a per-level
// edge mask (mask * coefficient).  Out of line: inlined, the compiler
// if-converted the masked and unmasked forms, and every edge of an unmasked
// model issued the masked form's multiplies with the predicate off.
template <class T>
__device__ __noinline__ T masked_dissipation(const MeshView &m,
                                             const ModelView &p,
                                             const AuxViewT<T> &a,
                                             const StageArgsT<T> &s, int c0,
                                             int c1, size_t i, int k,
                                             double idc, T t) {
  const int K = m.nlayers;
  const int e = int(i / unsigned(K));
  const double mk = m.mask[i];
  if (p.vel_del2)
    t = fma(__ldg(p.c2e + e) * mk, a.d2u[i], t);
  if (p.vel_del4) {
    const int v0 = __ldg(m.ve + 2 * e), v1 = __ldg(m.ve + 2 * e + 1);
    const T dd = a.d4[size_t(c1) * K + k] - a.d4[size_t(c0) * K + k];
    const T dz = a.z4[size_t(v1) * K + k] - a.z4[size_t(v0) * K + k];
    const T l = fma(dd, idc, -mul_reg(dz, __ldg(m.inv_dv + e)));
    t = fma(__ldg(p.c4e + e) * mk, l, t);
  }
  (void)s;
  return t;
}

// Operands of what the edge final pass adds to the PV flux of edge element i.
// LOAD: all loaded at construction (under the uniform term switches), for the
// fixed-point pass, which runs few warps: behind each switch they would be
// waited for one after another.  Otherwise loaded where they are used, with
// fewer registers.
template <class T, bool LOAD> struct EdgeIn {
  const MeshView &m;
  const ModelView &p;
  const AuxViewT<T> &a;
  const T *h;
  int e, k, c0, c1;
  size_t i;
  T d2u_{};
  T ke0{}, ke1{}, h0{}, h1{}, d0{}, d1{}, z0{}, z1{};
  double gidc_ = 0, c2_ = 0, c4i_ = 0, c4v_ = 0;

  __device__ __forceinline__ EdgeIn(const MeshView &m_, const ModelView &p_,
                                    const AuxViewT<T> &a_,
                                    const StageArgsT<T> &s, int e_, int k_,
                                    unsigned i_)
      : m(m_), p(p_), a(a_), h(s.h), e(e_), k(k_), c0(__ldg(m_.ce + 2 * e_)),
        c1(__ldg(m_.ce + 2 * e_ + 1)), i(i_) {
    if (!LOAD)
      return;
    gidc_ = __ldg(p.gidc + e);
    if (!p.off_ke)
      ke0 = a.ke[at(c0)], ke1 = a.ke[at(c1)];
    if (!p.off_ssh)
      h0 = h[at(c0)], h1 = h[at(c1)];
    if (!m.mask && p.vel_del2) {
      c2_ = __ldg(p.c2e + e);
      d2u_ = a.d2u[i];
    }
    if (!m.mask && p.vel_del4) {
      const int v0 = __ldg(m.ve + 2 * e), v1 = __ldg(m.ve + 2 * e + 1);
      c4i_ = __ldg(p.c4i + e);
      c4v_ = __ldg(p.c4v + e);
      d0 = a.d4[at(c0)], d1 = a.d4[at(c1)];
      z0 = a.z4[at(v0)];
      z1 = a.z4[at(v1)];
    }
  }
  __device__ __forceinline__ size_t at(int x) const {
    return size_t(x) * m.nlayers + k;
  }
  __device__ __forceinline__ T dke() const {
    return LOAD ? ke1 - ke0 : add_reg(a.ke[at(c1)], -a.ke[at(c0)]);
  }
  __device__ __forceinline__ T dh() const {
    return LOAD ? h1 - h0 : add_reg(h[at(c1)], -h[at(c0)]);
  }
  __device__ __forceinline__ T d2u() const { return LOAD ? d2u_ : a.d2u[i]; }
  __device__ __forceinline__ T dd() const {
    return LOAD ? d1 - d0 : add_reg(a.d4[at(c1)], -a.d4[at(c0)]);
  }
  __device__ __forceinline__ T dz() const {
    return LOAD ? z1 - z0
                : add_reg(a.z4[at(__ldg(m.ve + 2 * e + 1))],
                          -a.z4[at(__ldg(m.ve + 2 * e))]);
  }
  __device__ __forceinline__ double gidc() const {
    return LOAD ? gidc_ : __ldg(p.gidc + e);
  }
  __device__ __forceinline__ double c2() const {
    return LOAD ? c2_ : __ldg(p.c2e + e);
  }
  __device__ __forceinline__ double c4i() const {
    return LOAD ? c4i_ : __ldg(p.c4i + e);
  }
  __device__ __forceinline__ double c4v() const {
    return LOAD ? c4v_ : __ldg(p.c4v + e);
  }
};

// t plus the Bernoulli gradient, drag, del2 and del4 dissipation.
template <class T, bool LOAD>
__device__ __forceinline__ T edge_terms(const MeshView &m, const ModelView &p,
                                        const AuxViewT<T> &a,
                                        const StageArgsT<T> &s,
                                        const EdgeIn<T, LOAD> &r, T t) {
  const double idc = __ldg(m.inv_dc + r.e);
  // kinetic-energy and sea-surface-height gradients (the differences are
  // taken before scaling, as in the reference, so g h ~ 1e4 never rounds)
  if (!p.off_ke)
    t = fma(-idc, r.dke(), t);
  if (!p.off_ssh)
    t = fma(-r.gidc(), r.dh(), t);
  if (p.drag && r.k == p.drag_level)
    t = drag_add(m, p, a, s, r.c0, r.c1, r.i, r.k, t);
  if (m.mask) { // masked dissipation: out of line (see masked_dissipation)
    t = masked_dissipation(m, p, a, s, r.c0, r.c1, r.i, r.k, idc, t);
  } else {
    if (p.vel_del2)
      t = fma(r.c2(), r.d2u(), t);
    if (p.vel_del4) { // the coefficient folded into c4e/dc and -c4e/dv
      t = fma(r.c4i(), r.dd(), t);
      t = fma(r.c4v(), r.dz(), t);
    }
  }
  return t;
}

// The edge final pass of an edge whose PV sums need FP64 (see above).
template <int NE>
static __device__ __noinline__ void edge_final_f64(const MeshView &m,
                                                   const ModelView &p,
                                                   const AuxView &a,
                                                   const StageArgs &s, int e,
                                                   int k, unsigned i) {
  epilogue(s.ep, s.fvn, i,
           edge_terms(m, p, a, s, EdgeIn<double, false>(m, p, a, s, e, k, i),
                      p.off_pv ? 0.0 : pv_flux_f64<NE>(m, a, e, k)));
}

// The PV flux of edge element i by fixed-point sums: one over the words of F
// and one over those of F Q, with the edge's table of weights.
// EARLY: a flagged first word (a blown-up field) skips them; that keeps the
// words of both sums in registers at once, for which the batched kernel has
// none to spare (step of 12 members: 6.14 ms without, 6.49 with).
template <int NE, bool EARLY>
__device__ __forceinline__ void
edge_final_fixed(const MeshView &m, const ModelView &p, const AuxView &a,
                 const StageArgs &s, int e, int k, unsigned i) {
  const unsigned K = unsigned(m.nlayers);
  unsigned flag = 0;
  double S1 = 0, t = 0;
  const EdgeIn<double, true> er(m, p, a, s, e, k, i);
  const EpiIn<double> in = epilogue_in(s.ep, s.fvn, i);
  const double Q = p.off_pv ? 0.0 : a.Q[i];
  t = edge_terms(m, p, a, s, er, t);
  if (!p.off_pv) {
    const ulonglong2 *FG = reinterpret_cast<const ulonglong2 *>(a.FGx);
    const int4 *tab = reinterpret_cast<const int4 *>(m.fxe) + NE * e;
    Wt w[NE];
    fx_t x[NE], y[NE];
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int4 s4 = __ldg(tab + j);
      const ulonglong2 v = FG[unsigned(s4.x) * K + unsigned(k)];
      w[j] = {s4.y, s4.z, s4.w};
      x[j] = v.x;
      y[j] = v.y;
    }
    const long long start = __ldg(m.fxe0 + e);
    if (EARLY)
      flag = unsigned(x[0]) & FX_FLAG;
    if (!EARLY || !flag) {
      S1 = fx_sum<NE, FX_NONE>(w, x, start, FX_TOP, flag);
      const double S2 = fx_sum<NE, FX_NONE>(w, y, start, FX_TOP, flag);
      t = add_rn(fma(Q, S1, S2), t);
    }
  }
  if (flag) {
    edge_final_f64<NE>(m, p, a, s, e, k, i);
    return;
  }
  if (a.S1 && !p.off_pv)
    a.S1[i] = S1;
  epilogue(s.ep, s.fvn, i, t, in);
}

// Edge final pass: normal-velocity tendency (PV flux, Bernoulli gradient,
// del2 and del4 dissipation) and its stage update.  FX: PV sums in FP64 (0),
// fixed-point (1), or as the model keeps the words (-1).
template <int NE, class T, int FX = -1>
__device__ __forceinline__ void
pt_edge_final(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
              const StageArgsT<T> &s, unsigned i) {
  const int K = m.nlayers;
  const int e = int(i / unsigned(K)), k = int(i - unsigned(e) * unsigned(K));
  if constexpr (std::is_same<T, double>::value && FX != 0) {
    if (FX == 1 || a.FGx) {
      edge_final_fixed<NE, FX == 1>(m, p, a, s, e, k, i);
      return;
    }
  }
  // potential-vorticity flux: sum_j w_j F_j (Q_e + Q_j) / 4 with w/4 in woe
  T t{};
  if (!p.off_pv) {
    T S1, S2;
    {
      const int je = __ldg(m.eoe + NE * e);
      const double w = __ldg(m.woe + NE * e);
      S1 = mul_reg(w, a.F[size_t(je) * K + k]);
      S2 = mul_reg(w, a.G[size_t(je) * K + k]);
    }
#pragma unroll
    for (int j = 1; j < NE; ++j) {
      const int je = __ldg(m.eoe + NE * e + j);
      const double w = __ldg(m.woe + NE * e + j);
      S1 = fma(w, a.F[size_t(je) * K + k], S1);
      S2 = fma(w, a.G[size_t(je) * K + k], S2);
    }
    if (a.S1)
      a.S1[i] = S1;
    t = fma(a.Q[i], S1, S2);
  }
  epilogue(s.ep, s.fvn, i,
           edge_terms(m, p, a, s, EdgeIn<T, false>(m, p, a, s, e, k, i), t));
}

// The PV sum S1 = sum_j w_j F_j of edge element i alone, bit for bit the one
// the edge final pass tapes: for the adjoint, where only the auxiliary passes
// of a state have run.
template <int NE>
__device__ __forceinline__ void pt_pv_sum(const MeshView &m, const AuxView &a,
                                          unsigned i) {
  const unsigned K = unsigned(m.nlayers);
  const int e = int(i / K), k = int(i - unsigned(e) * K);
  unsigned flag = a.FGx ? 0 : FX_FLAG;
  double S1 = 0;
  if (!flag) {
    Wt w[NE];
    fx_t x[NE];
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int4 s4 = __ldg(reinterpret_cast<const int4 *>(m.fxe) + NE * e + j);
      const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(
          a.FGx)[unsigned(s4.x) * K + unsigned(k)];
      w[j] = {s4.y, s4.z, s4.w};
      x[j] = v.x;
      flag |= unsigned(v.y) & FX_FLAG; // of F Q: FP64 there takes both sums
    }
    S1 = fx_sum<NE, FX_NONE>(w, x, __ldg(m.fxe0 + e), FX_TOP, flag);
  }
  if (flag) {
    S1 = 0;
    for (int j = 0; j < NE; ++j)
      S1 = fma(__ldg(m.woe + NE * e + j),
               a.F[size_t(__ldg(m.eoe + NE * e + j)) * K + k], S1);
  }
  a.S1[i] = S1;
}

// ---- tracer part of the cell final pass, fixed-point sums
//
// A tracer's gathered words (6 normalised tracers and, with del4, 6
// Laplacians), its own values and the operands of its stage update.  ASYNC:
// copied into the thread's own shared-memory slots by cp.async one tracer
// ahead, so the gather of the next tracer is in flight, without holding
// registers, while the current one's sum runs.  Slots of a thread are
// `stride` words apart; TR_SLOTS words for each of the two stages.
constexpr int TR_SLOTS = 16;

template <bool D4>
__device__ __forceinline__ void
tracer_fetch(const AuxView &a, const StageArgs &s, int l, unsigned CK,
             const unsigned (&off)[MAXE + 1], fx_t *sm, unsigned stride) {
  const size_t base = size_t(l) * CK;
  const fx_t *n = a.nx + base;
  fx_t *d = sm + (l & 1) * (TR_SLOTS * stride);
#pragma unroll
  for (int j = 0; j < MAXE; ++j)
    copy_async8(d + j * stride, n + off[j]);
  copy_async8(d + 12 * stride, a.ntr + base + off[MAXE]);
  if (D4) {
    const fx_t *L = a.lx + base;
#pragma unroll
    for (int j = 0; j < MAXE; ++j)
      copy_async8(d + (6 + j) * stride, L + off[j]);
    copy_async8(d + 13 * stride, a.lap + base + off[MAXE]);
  }
  const double *u, *v;
  epilogue_operands(s.ep, s.ftr, u, v);
  if (u)
    copy_async8(d + 14 * stride, u + base + off[MAXE]);
  if (v)
    copy_async8(d + 15 * stride, v + base + off[MAXE]);
}

// The tracers of one cell-level from the weights w of the neighbours' and wc
// (rc) of the cell's own value (Laplacian).  One fixed-point sum over the
// neighbours of both stencils per tracer, the cell's own terms by FP64
// multiply-adds: per tracer 1 (conversion) + 2 (own terms) + 2 (update) FP64
// instructions instead of 16, and 12 integer terms, which takes the two
// kinds of pipe about equally long.
template <bool D4, bool ASYNC>
__device__ __forceinline__ void
tracer_sums(const MeshView &m, const ModelView &p, const AuxView &a,
            const StageArgs &s, int c, int k, unsigned CK,
            const double (&w)[MAXE], double wc, double rc,
            const unsigned (&off)[MAXE + 1], fx_t *sm, unsigned stride) {
  constexpr int N = D4 ? 2 * MAXE : MAXE;
  unsigned bad = 0;
  Wt W[N];
  long long start = 0;
#pragma unroll
  for (int j = 0; j < MAXE; ++j) {
    W[j] = fx_weight<FX_TOP>(w[j], bad);
    start += W[j].hi;
  }
  if (D4) {
#pragma unroll
    for (int j = 0; j < MAXE; ++j) {
      const int4 t = __ldg(reinterpret_cast<const int4 *>(p.r4x) + 6 * c + j);
      W[N - MAXE + j] = {t.y, t.z, t.w};
      start += W[N - MAXE + j].hi;
      bad |= t.w == FX_BAD_EXP ? FX_FLAG : 0u;
    }
  }
  start = fx_start(start);
  unsigned redo = bad;
  // with a bad weight no tracer has its sum here
#pragma unroll 1
  for (int l = bad ? p.ntracers : 0; l < p.ntracers; ++l) {
    const size_t base = size_t(l) * CK;
    fx_t x[N];
    double nc, Lc = 0;
    EpiIn<double> in;
    if (ASYNC) {
      if (l + 1 < p.ntracers)
        tracer_fetch<D4>(a, s, l + 1, CK, off, sm, stride);
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::
                       : "memory");
      const fx_t *d = sm + (l & 1) * (TR_SLOTS * stride);
#pragma unroll
      for (int j = 0; j < N; ++j)
        x[j] = d[j * stride];
      nc = __longlong_as_double((long long)d[12 * stride]);
      if (D4)
        Lc = __longlong_as_double((long long)d[13 * stride]);
      in.u = __longlong_as_double((long long)d[14 * stride]);
      in.v = __longlong_as_double((long long)d[15 * stride]);
    } else {
      const fx_t *n = a.nx + base, *L = a.lx + base;
#pragma unroll
      for (int j = 0; j < MAXE; ++j) {
        x[j] = n[off[j]];
        if (D4)
          x[N - MAXE + j] = L[off[j]];
      }
      nc = a.ntr[base + off[MAXE]];
      if (D4)
        Lc = a.lap[base + off[MAXE]];
      in = epilogue_in(s.ep, s.ftr, base + off[MAXE]);
    }
    unsigned flag = 0;
    double acc = fma(wc, nc, fx_sum<N, FX_LEAVE>(W, x, start, FX_TOP, flag));
    if (D4)
      acc = fma(rc, Lc, acc);
    redo |= flag;
    if (!flag)
      epilogue(s.ep, s.ftr, base + off[MAXE], acc, in);
  }
  if (redo) {
    // a bad weight left the first tracer's copies in flight: the thread's
    // next element (k_batch_heavy) copies to the same slots
    if (ASYNC)
      asm volatile("cp.async.wait_all;" ::: "memory");
    tracers_f64(m, p, a, s, c, k, bad != 0);
  }
}

// Cell final pass: thickness tendency and tracer tendencies (advection,
// del2, del4) with their stage updates.  MODE: tracers in FP64 (0), by
// fixed-point sums without (1) or with (2) del4, as the model keeps the words
// (-1).  ASYNC: sm is the thread's shared-memory slots.  PAIRS: FP64 tracers
// two at a time (the single-instance kernel; the batched kernels keep one at
// a time and their registers).
template <class T, int MODE = -1, bool ASYNC = false, bool PAIRS = false>
__device__ __forceinline__ void
pt_cell_final(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
              const StageArgsT<T> &s, unsigned i, fx_t *sm = nullptr,
              unsigned stride = 0) {
  constexpr bool FX = std::is_same<T, double>::value && MODE != 0;
  const int K = m.nlayers;
  const unsigned CK = unsigned(m.ncells) * unsigned(K);
  const int c = int(i / unsigned(K)), k = int(i - unsigned(c) * unsigned(K));
  const bool del4 = FX && MODE > 0 ? MODE == 2 : p.tr_del4;
  const bool fx = FX && (MODE > 0 || a.nx); // with tracers
  unsigned off[MAXE + 1];
#pragma unroll
  for (int j = 0; j < MAXE; ++j)
    off[j] = unsigned(__ldg(m.nbc + 6 * c + j)) * unsigned(K) + unsigned(k);
  off[MAXE] = i;
  if constexpr (FX && ASYNC) {
    if (p.ntracers > 0 && fx) {
      if (del4)
        tracer_fetch<true>(a, s, 0, CK, off, sm, stride);
      else
        tracer_fetch<false>(a, s, 0, CK, off, sm, stride);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // (the same bits either way; see mul_reg for where which is faster)
  auto mul = [](double x, T y) {
    if constexpr (FX)
      return mul_rn(x, y);
    else
      return mul_reg(x, y);
  };
  auto add = [](T x, T y) {
    if constexpr (FX)
      return add_rn(x, y);
    else
      return add_reg(x, y);
  };
  EpiIn<T> hin;
  if (p.do_h)
    hin = epilogue_in(s.ep, s.fh, i);
  // a_j = -F_j ccd_j / 2: half the flux divergence weight of edge j
  T w[MAXE], Sa{};
  int ej[MAXE];
#pragma unroll
  for (int j = 0; j < MAXE; ++j) {
    ej[j] = __ldg(m.ec + 6 * c + j);
    w[j] = T{};
  }
  if (!p.off_hadv || !p.off_tr_hadv) {
#pragma unroll
    for (int j = 0; j < MAXE; ++j)
      w[j] = mul(__ldg(m.ccdh + 6 * c + j), a.F[size_t(ej[j]) * K + k]);
    Sa = add(w[0], w[1]);
#pragma unroll
    for (int j = 2; j < MAXE; ++j)
      Sa = add(Sa, w[j]);
  }
  if (p.do_h) // -sum_j ccd_j F_j, or nothing with thickness advection off
    epilogue(s.ep, s.fh, i, p.off_hadv ? T{} : twice(Sa), hin);
  if (p.ntracers == 0)
    return;
  if (p.off_tr_hadv) { // tracer advection off: only diffusion weights
    Sa = T{};
#pragma unroll
    for (int j = 0; j < MAXE; ++j)
      w[j] = T{};
  }
  // advection + del2: sum_j a_j (n_c + n_j) + b_j (n_j - n_c); with a
  // uniform del2 scaling the del2 part is eddy_diff2 s L_c instead, taken
  // with the del4 stencil's centre weight (r4f)
  const bool fold = p.tr_del2 && del4 && p.r4f;
  T wc = Sa;
  if (p.tr_del2 && !fold) {
    T b[MAXE], Sb;
#pragma unroll
    for (int j = 0; j < MAXE; ++j) {
      b[j] = mul(__ldg(p.kd2 + 6 * c + j), a.mh[size_t(ej[j]) * K + k]);
      w[j] = add(w[j], b[j]);
    }
    Sb = add(b[0], b[1]);
#pragma unroll
    for (int j = 2; j < MAXE; ++j)
      Sb = add(Sb, b[j]);
    wc = add(Sa, -Sb);
  }
  // del4 centre weight: -sum r4, plus eddy_diff2 s when del2 is folded in
  const double rc = !del4 ? 0.0 : fold ? __ldg(p.r4f + c)
                                       : -__ldg(p.r4sum + c);
  if constexpr (FX) {
    if (fx) {
      if (del4)
        tracer_sums<true, ASYNC>(m, p, a, s, c, k, CK, w, wc, rc, off, sm,
                                 stride);
      else
        tracer_sums<false, ASYNC>(m, p, a, s, c, k, CK, w, wc, rc, off, sm,
                                  stride);
      return;
    }
  }
  // tracers in pairs: two independent FMA chains per thread keep more
  // loads and FP64 operations in flight (each tracer's operation sequence
  // is the same as alone, so the results are too)
  int l = 0;
  for (; PAIRS && l + 1 < p.ntracers; l += 2) {
    const size_t b0 = size_t(l) * CK, b1 = b0 + CK;
    const T *n0 = a.ntr + b0, *n1 = a.ntr + b1;
    T acc0 = mul_reg(wc, n0[i]), acc1 = mul_reg(wc, n1[i]);
#pragma unroll
    for (int j = 0; j < MAXE; ++j) {
      acc0 = fma(w[j], n0[off[j]], acc0);
      acc1 = fma(w[j], n1[off[j]], acc1);
    }
    if (del4) {
      const T *L0 = a.lap + b0, *L1 = a.lap + b1;
      acc0 = fma(rc, L0[i], acc0);
      acc1 = fma(rc, L1[i], acc1);
#pragma unroll
      for (int j = 0; j < MAXE; ++j) {
        const double r = __ldg(p.r4 + 6 * c + j);
        acc0 = fma(r, L0[off[j]], acc0);
        acc1 = fma(r, L1[off[j]], acc1);
      }
    }
    epilogue(s.ep, s.ftr, b0 + i, acc0);
    epilogue(s.ep, s.ftr, b1 + i, acc1);
  }
  for (; l < p.ntracers; ++l) {
    const size_t base = size_t(l) * CK;
    const T *n = a.ntr + base;
    T acc = wc * n[i];
#pragma unroll
    for (int j = 0; j < MAXE; ++j)
      acc = fma(w[j], n[off[j]], acc);
    if (del4) {
      const T *L = a.lap + base;
      acc = fma(rc, L[i], acc);
#pragma unroll
      for (int j = 0; j < MAXE; ++j)
        acc = fma(__ldg(p.r4 + 6 * c + j), L[off[j]], acc);
    }
    epilogue(s.ep, s.ftr, base + i, acc);
  }
}

// Pass domain sizes (threads) of pass `pass` for one instance.
// P_PV_SUM (pt_pv_sum) runs over P_EDGE_FINAL's domain.
enum Pass { P_VERTEX = 0, P_CELL1, P_EDGE1, P_AUX2, P_EDGE_FINAL,
            P_CELL_FINAL, NPASS, P_PV_SUM = NPASS };

// One member of a batched launch (swg_batch.cu, swg_ensemble.cu): its mesh,
// model, intermediates, stage arguments and the element count of each pass.
struct Member {
  MeshView m;
  ModelView p;
  AuxView a;
  StageArgs stage[5];
  unsigned units[NPASS]; // elements of each pass (0 = pass not needed)
  unsigned aux2_base;    // first element of the aux2 pass domain
};
// (swg_batch.cu) element counts of a model's passes
void batch_pass_units(const swg_model_s *md, unsigned units[NPASS],
                      unsigned &aux2_base);
// (swg_batch.cu) the passes a model runs with sums of words, as a bit set, and
// whether all or none of its sums of doubles are fixed-point (of a batch: in
// some member; both bits: the passes look at each member)
// and whether it has tracer Laplacians in FP64
constexpr unsigned HEAVY_RAW = 1u << 16, HEAVY_NO_RAW = 1u << 17,
                   HEAVY_LAP = 1u << 18;
unsigned batch_heavy_passes(const swg_model_s *md);
// (swg_batch.cu) passes [pass0, pass1] of stage `stage` over the nmem
// members of the device table `mem`, one 256-thread block per virtual block
// of 256 x items elements (items 1 or 2 per thread); prefix: [NPASS][nmem +
// 1] virtual-block offsets of the members for that block size (device) and
// prefix_h its host copy (grid sizes); heavy: the members' heavy passes.
int batch_launch_passes(const Member *mem, int nmem, const unsigned *prefix,
                        const unsigned *prefix_h, int ne, int items,
                        unsigned heavy, int pass0, int pass1, int stage,
                        cudaStream_t st);

// LinearShallowWaterModel (shallow_water_hierarchical.cpp:680-740):
// vn_t = f sum_j w_j vn_j - g (h_1 - h_0) / dc and h_t = -h0 div(vn), each
// with its stage update.
template <int NE, class T>
__device__ __forceinline__ void pt_lin_edge(const MeshView &m,
                                            const ModelView &p,
                                            const StageArgsT<T> &s,
                                            unsigned i) {
  const int K = m.nlayers;
  const int e = int(i / unsigned(K)), k = int(i - unsigned(e) * unsigned(K));
  T vt = __ldg(m.woe + NE * e) * s.vn[size_t(__ldg(m.eoe + NE * e)) * K + k];
#pragma unroll
  for (int j = 1; j < NE; ++j)
    vt = fma(__ldg(m.woe + NE * e + j),
             s.vn[size_t(__ldg(m.eoe + NE * e + j)) * K + k], vt);
  const int c0 = __ldg(m.ce + 2 * e), c1 = __ldg(m.ce + 2 * e + 1);
  const T t = fma(-__ldg(p.gidc + e),
                  s.h[size_t(c1) * K + k] - s.h[size_t(c0) * K + k],
                  p.f4 * vt);
  epilogue(s.ep, s.fvn, i, t);
}

template <class T>
__device__ __forceinline__ void pt_lin_cell(const MeshView &m,
                                            const ModelView &p,
                                            const StageArgsT<T> &s,
                                            unsigned i) {
  const int K = m.nlayers;
  const int c = int(i / unsigned(K)), k = int(i - unsigned(c) * unsigned(K));
  T d = __ldg(m.ccd + 6 * c) * s.vn[size_t(__ldg(m.ec + 6 * c)) * K + k];
#pragma unroll
  for (int j = 1; j < MAXE; ++j)
    d = fma(__ldg(m.ccd + 6 * c + j),
            s.vn[size_t(__ldg(m.ec + 6 * c + j)) * K + k], d);
  epilogue(s.ep, s.fh, i, -p.h0 * d);
}

} // namespace swg
