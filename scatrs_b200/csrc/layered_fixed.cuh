// The layered recursion for a number of layers known at compile time, with its derivative along one
// direction known at compile time (or none): the expressions of mie_device.cuh (Layered, LArg,
// layer_side, ratios_into) and layered_deriv.cuh, on values that carry a derivative only where the
// direction reaches them. With kDir < 0 it is the value recursion; kDir = l < kL the complex
// derivative along layer l's index, kDir = kL + l the derivative along the radius fraction f_l
// (x_l d/dx_l of the interface below the fixed outer surface).
//
// The general forms keep 15 layers' state in local memory, indexed at run time, and propagate
// derivatives that are zero (a direction reaches its own shell, its neighbours' lead terms and the
// log-derivatives above it). Here the loops unroll, the state of 2 to 4 layers is in registers and
// the zeros are not computed; the ratio arrays, independent downward recurrences, keep a derivative
// only where they have one.
#pragma once

#include "layered_deriv.cuh"

namespace sb {
namespace lfix {

template <bool D>
struct V {
  cplx v;
};
template <>
struct V<true> {
  cplx v, d;
};
template <bool D>
struct R {  // a real value
  double v;
};
template <>
struct R<true> {
  double v, d;
};
#define LF_FN __device__ __forceinline__
template <bool D>
LF_FN V<D> vv(cplx v) {
  V<D> r;
  r.v = v;
  if constexpr (D) r.d = rl(0.0);
  return r;
}
template <bool A, bool B>
LF_FN V<A || B> operator+(V<A> a, V<B> b) {
  V<A || B> r;
  r.v = a.v + b.v;
  if constexpr (A && B) r.d = a.d + b.d;
  else if constexpr (A) r.d = a.d;
  else if constexpr (B) r.d = b.d;
  return r;
}
template <bool A>
LF_FN V<A> operator-(V<A> a) {
  V<A> r;
  r.v = -a.v;
  if constexpr (A) r.d = -a.d;
  return r;
}
template <bool A, bool B>
LF_FN V<A || B> operator-(V<A> a, V<B> b) {
  V<A || B> r;
  r.v = a.v - b.v;
  if constexpr (A && B) r.d = a.d - b.d;
  else if constexpr (A) r.d = a.d;
  else if constexpr (B) r.d = -b.d;
  return r;
}
template <bool A, bool B>
LF_FN V<A || B> operator*(V<A> a, V<B> b) {
  V<A || B> r;
  r.v = a.v * b.v;
  if constexpr (A && B) r.d = a.d * b.v + a.v * b.d;
  else if constexpr (A) r.d = a.d * b.v;
  else if constexpr (B) r.d = a.v * b.d;
  return r;
}
template <bool A>
LF_FN V<A> operator*(V<A> a, cplx b) { return a * V<false>{b}; }
template <bool A>
LF_FN V<A> operator*(cplx a, V<A> b) { return V<false>{a} * b; }
template <bool A>
LF_FN V<A> operator+(V<A> a, cplx b) { return a + V<false>{b}; }
template <bool A>
LF_FN V<A> operator-(V<A> a, cplx b) { return a - V<false>{b}; }
// One copy of the reciprocal for the tens of them in an order.
static __device__ __noinline__ cplx cinv_call(cplx z) { return cinv(z); }
template <bool A>
LF_FN V<A> vinv(V<A> a) {
  V<A> r;
  r.v = cinv_call(a.v);
  if constexpr (A) r.d = -(a.d * r.v * r.v);
  return r;
}
template <bool A>
LF_FN V<A> vscl(V<A> a, double s) {
  V<A> r;
  r.v = scl(a.v, s);
  if constexpr (A) r.d = scl(a.d, s);
  return r;
}
template <bool A, bool B>
LF_FN V<A || B> vscl(V<A> a, R<B> s) {
  V<A || B> r;
  r.v = scl(a.v, s.v);
  if constexpr (A && B) r.d = scl(a.d, s.v) + scl(a.v, s.d);
  else if constexpr (A) r.d = scl(a.d, s.v);
  else if constexpr (B) r.d = scl(a.v, s.d);
  return r;
}
template <bool A>
LF_FN V<A> vsin(V<A> z) {
  V<A> r;
  r.v = csin(z.v);
  if constexpr (A) r.d = ccos(z.v) * z.d;
  return r;
}
template <bool A>
LF_FN V<A> vcos(V<A> z) {
  V<A> r;
  r.v = ccos(z.v);
  if constexpr (A) r.d = -(csin(z.v) * z.d);
  return r;
}
// e^(2 i z) - 1.
template <bool A>
LF_FN V<A> vexp_m1_2i(V<A> z) {
  V<A> r;
  r.v = cexp_m1(two_i(z.v));
  if constexpr (A) r.d = (r.v + rl(1.0)) * two_i(z.d);
  return r;
}
template <bool A>
LF_FN V<A> choose(bool c, V<A> a, V<A> b) {
  V<A> r;
  r.v = c ? a.v : b.v;
  if constexpr (A) r.d = c ? a.d : b.d;
  return r;
}
template <bool B, bool A>
LF_FN V<B> widen(V<A> a) {
  V<B> r;
  r.v = a.v;
  if constexpr (A && B) r.d = a.d;
  else if constexpr (B) r.d = rl(0.0);
  return r;
}

// Ratio arrays: value array a, and its derivative n_val arrays on.
template <int kVal>
struct Arrays {
  LayerArrays arr;
  template <bool D>
  LF_FN V<D> get(int a, int64_t k) const {
    V<D> r;
    r.v = arr.get(a, k);
    if constexpr (D) r.d = arr.get(a + kVal, k);
    return r;
  }
  template <bool D>
  LF_FN void put(int a, int64_t k, V<D> v) const {
    arr.put(a, k, v.v);
    if constexpr (D) arr.put(a + kVal, k, v.d);
  }
};

// u_k(m x), k = 1..n+1, into array a (ratios_into, ratios_d).
template <bool Dm, bool Dx, int kVal>
LF_FN void ratios(V<Dm> m, R<Dx> x, int64_t n, const Arrays<kVal>& A, int a) {
  constexpr bool D = Dm || Dx;
  const V<D> z = vscl(m, x);
  const int64_t top = n + 1;
  if (m.v.im == 0.0) {
    // The real form; z and its derivative are real here.
    const double inv_rho = 1.0 / z.v.re;
    double d_inv_rho = 0.0, u = 0.0, du = 0.0;
    if constexpr (D) d_inv_rho = -z.d.re * inv_rho * inv_rho;
    const int64_t start = start_index(top, fabs(z.v.re));
    for (int64_t k = start; k >= 1; --k) {
      const double c = inv_rho * (double)(2 * k + 1);
      double den = c - u, dden = 0.0;
      if constexpr (D) dden = d_inv_rho * (double)(2 * k + 1) - du;
      if (den == 0.0) {
        den = kEps * (fabs(c) + fabs(u));
        dden = 0.0;
      }
      u = 1.0 / den;
      if constexpr (D) du = -dden * u * u;
      if (k <= top) {
        V<D> v;
        v.v = rl(u);
        if constexpr (D) v.d = rl(du);
        A.put(a, k, v);
      }
    }
  } else {
    const V<D> inv_z = vinv(z);
    V<D> u = vv<D>(rl(0.0));
    const int64_t start = start_index(top, cabs_(z.v));
    for (int64_t k = start; k >= 1; --k) {
      const V<D> c = vscl(inv_z, (double)(2 * k + 1));
      V<D> den = c - u;
      if (den.v.re == 0.0 && den.v.im == 0.0)
        den = vv<D>(rl(step_eps(c.v, u.v)));
      u = vinv(den);
      if (k <= top) A.put(a, k, u);
    }
  }
}

// LArg (layered/kernel.rs:33-103).
template <bool D>
struct Arg {
  V<D> inv_z, pi, w, w_n;
  LF_FN void init(V<D> z, bool chi) {
    inv_z = vinv(z);
    if (chi) {
      const V<D> sz = vsin(z), cz = vcos(z);
      pi = sz * cz;
      w = inv_z + sz * vinv(cz);
    } else {
      pi = -vscl(vexp_m1_2i(z), 0.5);
      w = inv_z - mk(0.0, 1.0);
    }
    w_n = vv<D>(rl(0.0));
  }
  LF_FN void step(int64_t n, V<D> u_n) {
    w_n = w;
    pi = pi * u_n * w;
    w = vscl(inv_z, (double)(2 * n + 1)) - vinv(w);
  }
  LF_FN V<D> d1(int64_t n, V<D> u_next) const { return vscl(inv_z, (double)(n + 1)) - u_next; }
  LF_FN V<D> d3(int64_t n) const { return vscl(inv_z, (double)(n + 1)) - w; }
};

template <bool D>
struct SideV {
  bool direct;
  V<D> v;
};

// layer_side (layered/kernel.rs:158-183); the branch follows the values.
template <bool kOut, bool Dm, bool Dn, bool Dp, bool Dh, bool Dl, bool Du, bool Di, bool Do, bool Dq>
LF_FN SideV<kOut> side(V<Dm> mi, V<Dn> mo, SideV<Dp> prev, V<Dh> h, V<Dl> lead, V<Du> u_prev,
                       V<Di> u1, V<Di> d1i, V<Di> d3i, V<Do> d1o, V<Do> d3o, V<Do> pio, V<Dq> p,
                       cplx w, V<kOut>* h_out) {
  const auto mh = mi * h;
  constexpr bool G = Dm || Dn || Dp || Dh || Dl || Du || Di;
  const V<G> g1 = prev.direct ? widen<G>(mh - mo * d1i)
                              : widen<G>(lead - mi * u_prev + mo * u1 + mi * prev.v);
  const auto g2 = mh - mo * d3i;
  const auto inv_den = vinv(pio * g2 - p * g1);
  const V<kOut> delta = widen<kOut>(-(w * p * g1 * inv_den * vinv(pio)));
  const V<kOut> hd = widen<kOut>(d1o + delta);
  if (norm1(hd.v) * 4.0 >= fmax(norm1(d1o.v), norm1(delta.v))) {
    *h_out = hd;
    return {false, delta};
  }
  const V<kOut> hp = widen<kOut>(d3o - w * g2 * inv_den);
  *h_out = hp;
  return {true, hp};
}

// Where direction kDir of kL layers has derivatives: index m_l, interface x_l, shell l's arguments
// m_l x_{l-1} and m_l x_l, its lead term, and the log-derivative after it.
template <int kL, int kDir>
struct Flags {
  static constexpr bool m(int l) { return kDir == l; }
  static constexpr bool x(int l) { return kDir >= kL && l == kDir - kL; }
  static constexpr bool inner(int l) { return m(l) || x(l - 1); }
  static constexpr bool outer(int l) { return m(l) || x(l); }
  static constexpr bool p(int l) { return inner(l) || outer(l); }
  static constexpr bool lead(int l) { return m(l) || m(l - 1) || x(l - 1); }
  static constexpr bool h(int l) {
    return l == 0 ? outer(0) : h(l - 1) || p(l) || lead(l);
  }
};

// Shell l's state (l >= 1) on the shells below it.
template <int kL, int kDir, int l>
struct Shells : Shells<kL, kDir, l - 1> {
  using F = Flags<kL, kDir>;
  V<F::m(l)> m;
  Arg<F::inner(l)> in;
  Arg<F::outer(l)> out;
  V<F::p(l)> p;
  V<F::lead(l)> lead;
  R<F::x(l - 1)> x;  // the interface below
  bool chi;
};
template <int kL, int kDir>
struct Shells<kL, kDir, 0> {
  using F = Flags<kL, kDir>;
  V<F::m(0)> m;
  Arg<F::outer(0)> core;
};

// The recursion (Layered, LayeredD) for kL layers along kDir.
template <int kL, int kDir>
struct LayeredT {
  static constexpr bool kLayered = true;
  using F = Flags<kL, kDir>;
  static constexpr bool kH = F::h(kL - 1), kM = F::m(kL - 1);
  static constexpr int kVal = 2 * kL - 1;
  Arrays<kVal> arr;
  Shells<kL, kDir, kL - 1> st;

  static constexpr int a_outer(int l) { return l == kL - 1 ? 0 : 2 * l + 1; }
  static constexpr int a_inner(int l) { return 2 * l; }
  static constexpr int kCore = 1;

  template <bool D>
  static LF_FN V<D> index(cplx m) {
    V<D> r;
    r.v = m;
    if constexpr (D) r.d = rl(1.0);
    return r;
  }
  // The interface l < kL - 1, its derivative x (the particle's) along f_l; the outer surface is
  // fixed.
  template <int l>
  static LF_FN auto interface(const double* x) {
    R<F::x(l)> r;
    r.v = x[l];
    if constexpr (F::x(l)) r.d = x[kL - 1];
    return r;
  }

  template <int l>
  LF_FN void prepare_shell(int64_t n, const double* x, const cplx* ms) {
    if constexpr (l > 1) prepare_shell<l - 1>(n, x, ms);
    auto& s = static_cast<Shells<kL, kDir, l>&>(st);
    const auto m = index<F::m(l)>(ms[l]);
    const auto mb = index<F::m(l - 1)>(ms[l - 1]);
    const auto xi = interface<l - 1>(x);
    const auto xo = interface<l>(x);
    ratios(m, xi, n, arr, a_inner(l));
    if constexpr (l < kL - 1) ratios(m, xo, n, arr, a_outer(l));
    const bool c = ms[l].im * x[l] < 0.5;
    s.m = m;
    s.chi = c;
    s.x = xi;
    s.lead = widen<F::lead(l)>((m - mb) * (m + mb) * vinv(m * mb));
    const auto z1 = vscl(m, xi);
    const auto z2 = vscl(m, xo);
    s.in.init(z1, c);
    s.out.init(z2, c);
    if (c) {
      const auto c2 = vcos(z2);
      s.p = widen<F::p(l)>(vsin(z1) * vinv(vcos(z1)) * c2 * c2);
    } else {
      const double dx = x[l] - x[l - 1];
      const double ea = -(ms[l].im * dx * 2.0), eb = ms[l].re * dx * 2.0;
      double sb, cb;
      sincos(eb, &sb, &cb);
      const double ex = exp(ea);
      V<F::p(l)> e;
      e.v = scl(mk(cb, sb), ex);
      if constexpr (F::p(l)) {
        double xd = 0.0;
        if constexpr (F::x(l)) xd = xo.d;
        if constexpr (F::x(l - 1)) xd = -xi.d;
        const double mr = F::m(l) ? 1.0 : 0.0;  // dm = 1 along the index
        const double da = -(ms[l].im * xd) * 2.0, db = (mr * dx + ms[l].re * xd) * 2.0;
        e.d = scl(mk(-sb * db, cb * db), ex) + scl(mk(cb, sb), ex * da);
      }
      s.p = widen<F::p(l)>(-vscl(e * vexp_m1_2i(z1), 0.5));
    }
  }

  // The ratio arrays and the initial state; array 0's values come from mie_prepare where they
  // carry no derivative.
  LF_FN void prepare(int64_t n, const double* x, const cplx* ms) {
    if constexpr (kM) ratios(index<true>(ms[kL - 1]), R<false>{x[kL - 1]}, n, arr, 0);
    auto& s0 = static_cast<Shells<kL, kDir, 0>&>(st);
    s0.m = index<F::m(0)>(ms[0]);
    const auto x0 = interface<0>(x);
    ratios(s0.m, x0, n, arr, kCore);
    prepare_shell<kL - 1>(n, x, ms);
    s0.core.init(vscl(s0.m, x0), false);
  }

  template <int l>
  LF_FN void step_shell(int64_t k) {
    if constexpr (l > 1) step_shell<l - 1>(k);
    auto& s = static_cast<Shells<kL, kDir, l>&>(st);
    const auto u1 = arr.template get<F::inner(l)>(a_inner(l), k);
    s.in.step(k, u1);
    s.out.step(k, arr.template get<F::outer(l)>(a_outer(l), k));
    s.p = widen<F::p(l)>(s.p * u1 * vinv(s.in.w_n) * s.out.w_n * s.out.w_n);
  }
  template <int l, bool Dh, bool Ds>
  LF_FN void shell(int64_t k, V<Dh> ha, V<Dh> hb, SideV<Ds> a, SideV<Ds> b, SideV<kH>& sa,
                   SideV<kH>& sb) {
    const auto& s = static_cast<const Shells<kL, kDir, l>&>(st);
    const auto& below = static_cast<const Shells<kL, kDir, l - 1>&>(st);
    constexpr bool kPrev = F::outer(l - 1);
    const auto u_prev = arr.template get<kPrev>(l == 1 ? kCore : a_outer(l - 1), k + 1);
    const auto u1 = arr.template get<F::inner(l)>(a_inner(l), k + 1);
    const auto u2 = arr.template get<F::outer(l)>(a_outer(l), k + 1);
    const auto d1i = s.in.d1(k, u1);
    const auto d3i = s.in.d3(k);
    const auto d1o = s.out.d1(k, u2);
    const auto d3o = s.out.d3(k);
    const cplx w = s.chi ? rl(-1.0) : mk(0.0, 1.0);
    R<F::x(l - 1)> q;
    q.v = (double)(k + 1) / s.x.v;
    if constexpr (F::x(l - 1)) q.d = -(double)(k + 1) * s.x.d / (s.x.v * s.x.v);
    const auto ld = vscl(s.lead, q);
    constexpr bool kOut = F::h(l);
    V<kOut> na, nb;
    const SideV<kOut> a2 = side<kOut>(s.m, below.m, a, ha, ld, u_prev, u1, d1i, d3i, d1o, d3o,
                                      s.out.pi, s.p, w, &na);
    const SideV<kOut> b2 = side<kOut>(below.m, s.m, b, hb, V<false>{rl(0.0)}, u_prev, u1, d1i, d3i,
                                      d1o, d3o, s.out.pi, s.p, w, &nb);
    if constexpr (l == kL - 1) {
      sa = a2;
      sb = b2;
    } else {
      shell<l + 1>(k, na, nb, a2, b2, sa, sb);
    }
  }
  LF_FN void order(int64_t k, SideV<kH>& sa, SideV<kH>& sb) {
    step_shell<kL - 1>(k);
    const auto& s0 = static_cast<const Shells<kL, kDir, 0>&>(st);
    const auto h = s0.core.d1(k, arr.template get<F::outer(0)>(kCore, k + 1));
    const SideV<false> none{false, V<false>{rl(0.0)}};
    shell<1>(k, h, h, none, none, sa, sb);
  }
  // The value recursion's interface (mie_finish).
  LF_FN void order(int64_t k, Side& sa, Side& sb) {
    SideV<kH> a, b;
    order(k, a, b);
    sa = Side{a.direct, a.v.v};
    sb = Side{b.direct, b.v.v};
  }
};

// layered_finish_d on a typed recursion: the outer index carries a derivative along itself only.
template <class Emit, class Lay>
LF_FN double finish(double x, cplx m_v, int64_t n, const Scratch& s, ValueSums& vs, Emit emit,
                    Lay& layers, double abs_d[2]) {
  constexpr bool kM = Lay::kM, kH = Lay::kH;
  const double one = 1.0;
  const V<kM> m = Lay::template index<kM>(m_v);
  const V<kM> z = vscl(m, x);
  const int64_t n_s = upward_orders(x, n);
  const double inv_x = 1.0 / x;
  const V<kM> inv_z = vinv(z);
  const V<kM> inv_m = vinv(m);
  const V<kM> inv_m2 = inv_m * inv_m;
  const V<kM> m2_minus_1 = (m - rl(one)) * (m + rl(one));
  const V<kM> c_a = -(m2_minus_1 * inv_m2);
  const bool unit_m = m_v.re == 1.0 && m_v.im == 0.0;
  double sin_x, cos_x;
  sincos(x, &sin_x, &cos_x);
  double psi_prev = cos_x, psi = sin_x;
  double chi_prev = -sin_x, chi = cos_x;
  cplx t = rl(0.0), inv_xi = rl(0.0), r = rl(0.0);
  if (n_s == 0) {
    cplx xi0 = mk(sin_x, -cos_x);
    t = rl(sin_x) * cinv(xi0);
    inv_xi = mk(sin_x, cos_x);
    r = mk(0.0, one);
  }
  double asum = 0.0;
  abs_d[0] = abs_d[1] = 0.0;
  for (int64_t k = 1; k <= n; ++k) {
    const double k_x = (double)k * inv_x;
    const V<kM> u_z1 = layers.arr.template get<kM>(0, k + 1);
    const V<kM> d = vscl(inv_z, (double)(k + 1)) - u_z1;
    SideV<kH> sa, sb;
    layers.order(k, sa, sb);
    const V<kH> hh_a = sa.direct ? sa.v : widen<kH>(d + sa.v);
    const V<kH> hh_b = sb.direct ? sb.v : widen<kH>(d + sb.v);
    const V<kH> d_m = widen<kH>(hh_a * inv_m);
    const V<kH> md = widen<kH>(hh_b * m);
    const V<kH> big_a = d_m + rl(k_x);
    const V<kH> big_b = md + rl(k_x);
    V<kH> an, bn, inv_da, inv_db;
    if (k <= n_s) {
      const double c = (double)(2 * k - 1) * inv_x;
      const double psi_next = c * psi - psi_prev;
      psi_prev = psi;
      psi = psi_next;
      const double chi_next = c * chi - chi_prev;
      chi_prev = chi;
      chi = chi_next;
      const cplx xi = mk(psi, -chi);
      const cplx xi_prev = mk(psi_prev, -chi_prev);
      inv_da = vinv(big_a * xi - xi_prev);
      inv_db = vinv(big_b * xi - xi_prev);
      // The outer layer's own numerator (exactly 0 in value for m = 1, kernel.rs:412-435).
      V<kM> own_a = vscl(d * inv_m + rl(k_x), psi) - rl(psi_prev);
      V<kM> own_b = vscl(d * m + rl(k_x), psi) - rl(psi_prev);
      if (unit_m) {
        own_a.v = rl(0.0);
        own_b.v = rl(0.0);
      }
      an = sa.direct ? widen<kH>((vscl(big_a, psi) - rl(psi_prev)) * inv_da)
                     : widen<kH>((own_a + vscl(sa.v * inv_m, psi)) * inv_da);
      bn = sb.direct ? widen<kH>((vscl(big_b, psi) - rl(psi_prev)) * inv_db)
                     : widen<kH>((own_b + vscl(m * sb.v, psi)) * inv_db);
      if (k == n_s) {
        inv_xi = cinv(xi);
        t = rl(psi) * inv_xi;
        r = xi_prev * inv_xi;
      }
    } else {
      r = cinv(rl((double)(2 * k - 1) * inv_x) - r);
      t = scl(t * r, s.get_x(k));
      inv_xi = inv_xi * r;
      const cplx u_x1 = rl(s.get_x(k + 1));
      const cplx d_x = rl((double)(k + 1) * inv_x) - u_x1;
      const V<kH> num_a = sa.direct
                              ? d_m - d_x
                              : widen<kH>(vscl(c_a, (double)(k + 1) * inv_x) + u_x1 - u_z1 * inv_m +
                                          sa.v * inv_m);
      const V<kH> num_b = sb.direct ? md - d_x
                                    : widen<kH>((V<false>{u_x1} - m * u_z1) + m * sb.v);
      const V<kH> ia = vinv(big_a - r);
      const V<kH> ib = vinv(big_b - r);
      an = t * num_a * ia;
      bn = t * num_b * ib;
      inv_da = inv_xi * ia;
      inv_db = inv_xi * ib;
    }
    vs.add(k, an.v, bn.v);
    const double na = nsq(inv_da.v), nb = nsq(inv_db.v);
    const double weight = (double)(2 * k + 1);
    asum += weight * (-(d_m.v.im * na) - md.v.im * nb);
    // |g|^2 and Im f along the parameter, and along i times it (holomorphic f and g).
    const cplx pa = mk(inv_da.v.re, -inv_da.v.im) * inv_da.d;
    const cplx pb = mk(inv_db.v.re, -inv_db.v.im) * inv_db.d;
    abs_d[0] += weight * (-(d_m.d.im * na + d_m.v.im * 2.0 * pa.re) -
                          (md.d.im * nb + md.v.im * 2.0 * pb.re));
    abs_d[1] += weight * (-(d_m.d.re * na - d_m.v.im * 2.0 * pa.im) -
                          (md.d.re * nb - md.v.im * 2.0 * pb.im));
    emit(k, an.v, bn.v, an.d, bn.d);
  }
  return asum;
}

#undef LF_FN

}  // namespace lfix
}  // namespace sb
