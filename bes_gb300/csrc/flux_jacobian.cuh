// Derivatives of the Roe flux with respect to one side's conserved variables, by forward
// differentiation (the role of src/FluxJacobianWrapper.tpp:32-82) with the zeros known at compile
// time: the mask M of an SDual names the variables it can depend on, so that a density carries
// one derivative, a velocity two, the other side's state none.  Dual<5> carries and multiplies
// five for every quantity, and the compiler may not drop the products with zero; the derivatives
// that remain are formed by the same operations in the same order (FP64 Jacobians only: without the
// products with zero the compiler fuses other pairs of operations, a difference of rounding).
#pragma once
#include "physics.cuh"

namespace bes {

template <unsigned M, class S>
struct SDual {
  S v;
  S d[5];  // entry i only where bit i of M is set
};
#define BES_SD2 template <unsigned A, unsigned B, class S> BES_HD
#define BES_SD1 template <unsigned A, class S> BES_HD
BES_SD2 SDual<A | B, S> operator+(const SDual<A, S>& a, const SDual<B, S>& b) {
  SDual<A | B, S> r;
  r.v = a.v + b.v;
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if ((A & B) >> i & 1) r.d[i] = a.d[i] + b.d[i];
    else if (A >> i & 1) r.d[i] = a.d[i];
    else if (B >> i & 1) r.d[i] = b.d[i];
  return r;
}
BES_SD2 SDual<A | B, S> operator-(const SDual<A, S>& a, const SDual<B, S>& b) {
  SDual<A | B, S> r;
  r.v = a.v - b.v;
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if ((A & B) >> i & 1) r.d[i] = a.d[i] - b.d[i];
    else if (A >> i & 1) r.d[i] = a.d[i];
    else if (B >> i & 1) r.d[i] = -b.d[i];
  return r;
}
BES_SD2 SDual<A | B, S> operator*(const SDual<A, S>& a, const SDual<B, S>& b) {
  SDual<A | B, S> r;
  r.v = a.v * b.v;
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if ((A & B) >> i & 1) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    else if (A >> i & 1) r.d[i] = a.d[i] * b.v;
    else if (B >> i & 1) r.d[i] = a.v * b.d[i];
  return r;
}
// the value x with derivatives k times those of a
BES_SD1 SDual<A, S> scaled(S x, const SDual<A, S>& a, S k) {
  SDual<A, S> r;
  r.v = x;
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if (A >> i & 1) r.d[i] = a.d[i] * k;
  return r;
}
BES_SD1 SDual<A, S> operator*(const SDual<A, S>& a, S b) { return scaled(a.v * b, a, b); }
BES_SD1 SDual<A, S> operator*(S a, const SDual<A, S>& b) { return b * a; }
BES_SD1 SDual<A, S> operator+(const SDual<A, S>& a, S b) {
  SDual<A, S> r = a;
  r.v = a.v + b;
  return r;
}
BES_SD1 SDual<A, S> operator+(S a, const SDual<A, S>& b) { return b + a; }
BES_SD1 SDual<A, S> operator-(const SDual<A, S>& a) {
  SDual<A, S> r;
  r.v = -a.v;
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if (A >> i & 1) r.d[i] = -a.d[i];
  return r;
}
BES_SD1 SDual<A, S> operator-(const SDual<A, S>& a, S b) {
  SDual<A, S> r = a;
  r.v = a.v - b;
  return r;
}
BES_SD1 SDual<A, S> operator-(S a, const SDual<A, S>& b) {
  SDual<A, S> r = -b;
  r.v = a - b.v;
  return r;
}
BES_SD1 SDual<A, S> recip(const SDual<A, S>& a) {
  const S v = S(1) / a.v;
  return scaled(v, a, -v * v);
}
BES_SD1 SDual<A, S> bsqrt(const SDual<A, S>& a) {
  const S v = std::sqrt(a.v);
  return scaled(v, a, S(0.5) / v);
}
BES_SD1 SDual<A, S> babs(const SDual<A, S>& a) { return a.v < 0 ? -a : a; }
// the same number with room for every derivative
BES_SD1 SDual<31, S> widen(const SDual<A, S>& a) {
  SDual<31, S> r;
  r.v = a.v;
#pragma unroll
  for (int i = 0; i < 5; ++i) r.d[i] = (A >> i & 1) ? a.d[i] : S(0);
  return r;
}
#undef BES_SD1
#undef BES_SD2

// A side's state: of the side that is differentiated, or of the other one.
template <class S>
struct VarSide {
  SDual<1, S> rho, ir;
  SDual<2, S> m0;
  SDual<4, S> m1;
  SDual<8, S> m2;
  SDual<16, S> E;
  SDual<3, S> u0;
  SDual<5, S> u1;
  SDual<9, S> u2;
  SDual<31, S> p, H;
  SDual<15, S> vn;
};
template <class S>
struct FixedSide {
  S rho, ir, m0, m1, m2, E, u0, u1, u2, p, H, vn;
};
template <class S, class X>
BES_HD void finish_side(const GasConst& g, const double* n, X& s) {
  s.ir = recip(s.rho);
  s.u0 = s.m0 * s.ir;
  s.u1 = s.m1 * s.ir;
  s.u2 = s.m2 * s.ir;
  const auto k = s.m0 * s.m0 + s.m1 * s.m1 + s.m2 * s.m2;
  const auto e = s.E - k * (S(0.5) * s.ir);
  s.p = S(g.gm1) * e;
  s.H = (s.E + s.p) * s.ir;
  s.vn = s.u0 * S(n[0]) + s.u1 * S(n[1]) + s.u2 * S(n[2]);
}
template <class S>
BES_HD VarSide<S> var_side(const GasConst& g, const S* U, const double* n) {
  VarSide<S> s;
  s.rho.v = U[0];
  s.m0.v = U[1];
  s.m1.v = U[2];
  s.m2.v = U[3];
  s.E.v = U[4];
  s.rho.d[0] = s.m0.d[1] = s.m1.d[2] = s.m2.d[3] = s.E.d[4] = S(1);
  finish_side<S>(g, n, s);
  return s;
}
template <class S>
BES_HD FixedSide<S> fixed_side(const GasConst& g, const S* U, const double* n) {
  FixedSide<S> s;
  s.rho = U[0];
  s.m0 = U[1];
  s.m1 = U[2];
  s.m2 = U[3];
  s.E = U[4];
  finish_side<S>(g, n, s);
  return s;
}
template <unsigned M, class S>
BES_HD void put_row(const SDual<M, S>& f, S* row) {
#pragma unroll
  for (int i = 0; i < 5; ++i) row[i] = (M >> i & 1) ? f.d[i] : S(0);
}
// J = d F / d U of the differentiated side, row-major: the operations of roe_flux.
template <class S, class XL, class XR>
BES_HD void roe_derivative(const GasConst& g, const XL& L, const XR& R, const double* n, S* J) {
  const S n0 = S(n[0]), n1 = S(n[1]), n2 = S(n[2]);
  const auto sL = bsqrt(L.rho);
  const auto sR = bsqrt(R.rho);
  const auto iden = recip(sL + sR);
  const auto rho = sL * sR;
  const auto a0 = (L.u0 * sL + R.u0 * sR) * iden;
  const auto a1 = (L.u1 * sL + R.u1 * sR) * iden;
  const auto a2 = (L.u2 * sL + R.u2 * sR) * iden;
  const auto H = (L.H * sL + R.H * sR) * iden;
  const auto q2 = a0 * a0 + a1 * a1 + a2 * a2;
  const auto vn = a0 * n0 + a1 * n1 + a2 * n2;
  const auto c2 = S(g.gm1) * (H - S(0.5) * q2);
  const auto c = bsqrt(c2);
  const auto ic2 = recip(c2);
  const auto delta = babs(c * S(g.harten));
  SDual<31, S> l1 = babs(vn - c), l2 = widen(babs(vn)), l5 = babs(vn + c);
  if (l1.v <= delta.v || l2.v <= delta.v || l5.v <= delta.v) {
    const auto ih = S(0.5) * recip(delta);
    if (l1.v <= delta.v) l1 = (l1 * l1 + delta * delta) * ih;
    if (l2.v <= delta.v) l2 = (l2 * l2 + delta * delta) * ih;
    if (l5.v <= delta.v) l5 = (l5 * l5 + delta * delta) * ih;
  }
  const auto drho = R.rho - L.rho;
  const auto dp = R.p - L.p;
  const auto dvn = R.vn - L.vn;
  const auto d0 = R.u0 - L.u0;
  const auto d1 = R.u1 - L.u1;
  const auto d2 = R.u2 - L.u2;
  const auto rc = rho * c;
  const auto k1 = l1 * (dp - rc * dvn) * (S(0.5) * ic2);
  const auto k5 = l5 * (dp + rc * dvn) * (S(0.5) * ic2);
  const auto c1 = l2 * (drho - dp * ic2);
  const auto cc2 = l2 * rho;
  const auto t = d0 * a0 + d1 * a1 + d2 * a2;
  const auto k15 = k1 + k5;
  const auto k51 = k5 - k1;
  put_row(S(0.5) * (L.rho * L.vn + R.rho * R.vn - k15 - c1), J);
  put_row(S(0.5) * ((L.m0 * L.vn + L.p * n0) + (R.m0 * R.vn + R.p * n0) - k15 * a0 - k51 * c * n0 -
                    (c1 * a0 + cc2 * (d0 - dvn * n0))), J + 5);
  put_row(S(0.5) * ((L.m1 * L.vn + L.p * n1) + (R.m1 * R.vn + R.p * n1) - k15 * a1 - k51 * c * n1 -
                    (c1 * a1 + cc2 * (d1 - dvn * n1))), J + 10);
  put_row(S(0.5) * ((L.m2 * L.vn + L.p * n2) + (R.m2 * R.vn + R.p * n2) - k15 * a2 - k51 * c * n2 -
                    (c1 * a2 + cc2 * (d2 - dvn * n2))), J + 15);
  put_row(S(0.5) * (((L.E + L.p) * L.vn) + ((R.E + R.p) * R.vn) - k15 * H - k51 * c * vn -
                    (c1 * S(0.5) * q2 + cc2 * (t - dvn * vn))), J + 20);
}

}  // namespace bes
