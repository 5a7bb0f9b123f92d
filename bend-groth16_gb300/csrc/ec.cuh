// Short Weierstrass curves y^2 = x^3 + b (a = 0) over Fq (G1) and Fq2 (G2) on the device.
//
// Affine points use the wire convention of the reference: infinity is (0, 0), which is not
// on the curve (bend2/FORMAT.md:14-16, bend2/src/g1.bend:19-25).  Accumulators use
// extended Jacobian "XYZZ" coordinates (x = X/ZZ, y = Y/ZZZ, ZZ^3 = ZZZ^2), infinity is
// ZZ = 0.  Formulas are the Explicit-Formulas Database ones for XYZZ with a = 0:
//   madd-2008-s (XYZZ + affine, 8M + 2S), add-2008-s (XYZZ + XYZZ, 12M + 2S),
//   dbl-2008-s-1 (XYZZ, 6M + 3S), mdbl-2008-s (affine -> XYZZ double, 3M + 2S).
// The reference's Jacobian madd-2007-bl / add-2007-bl / dbl-2009-l (bend2/src/g1.bend:76-172)
// compute the same group law; only the projective representation differs, and every
// result leaving the device is normalised (affine, or Jacobian with Z = 1).
// Special cases (infinity, P == Q, P == -Q) are resolved by branches before the generic
// formula; they are rare on random inputs, so the branch is almost never divergent.
#pragma once
#include "fp.cuh"

namespace bg {

// Products used by the curve formulas: shared out-of-line bodies (fp_wide.cuh), so the loops of
// the reductions, the tables and the G2 accumulation stay small in the instruction cache.
BG_DEV Fq fmul(const Fq& a, const Fq& b) { return mul_ool(a, b); }
BG_DEV Fq fsqr(const Fq& a) { return sqr_ool(a); }
BG_DEV Fq fmul_sub(const Fq& a, const Fq& b, const Fq& c, const Fq& d) { return mul_sub_mul_ool(a, b, c, d); }
BG_DEV Fq2 fmul(const Fq2& a, const Fq2& b) { return fq2_mul_ool(a, b); }
BG_DEV Fq2 fsqr(const Fq2& a) {
  return {fmul(add(a.c0, a.c1), sub(a.c0, a.c1)), fmul(dbl(a.c0), a.c1)};
}
BG_DEV Fq2 fmul_sub(const Fq2& a, const Fq2& b, const Fq2& c, const Fq2& d) {
  return fq2_mul_sub_mul_ool(a, b, c, d);
}
// The mixed addition and the affine pair addition are the whole loop of the G1 accumulation: their
// Fq products are inlined (a call moves 24 registers): G1 MSM 2^20's accumulation 0.75 -> 0.70 ms
// and pair rounds 2.05 -> 1.91 ms.  Fq2 products stay calls (inlined, the G2 accumulation measured
// 1.89 -> 2.12 ms).
BG_DEV Fq imul(const Fq& a, const Fq& b) { return mul(a, b); }
BG_DEV Fq isqr(const Fq& a) { return sqr_wide(a); }
BG_DEV Fq imul_sub(const Fq& a, const Fq& b, const Fq& c, const Fq& d) { return mul_sub_mul(a, b, c, d); }
BG_DEV Fq2 imul(const Fq2& a, const Fq2& b) { return fmul(a, b); }
BG_DEV Fq2 isqr(const Fq2& a) { return fsqr(a); }
BG_DEV Fq2 imul_sub(const Fq2& a, const Fq2& b, const Fq2& c, const Fq2& d) { return fmul_sub(a, b, c, d); }

// 1/a (0 -> 0): Fermat in Fq; in Fq2 through the norm a0^2 + a1^2 (bend2/src/fq2.bend:46-50)
BG_DEV Fq field_inv_any(const Fq& a) { return inv(a); }
BG_DEV Fq2 field_inv_any(const Fq2& a) {
  const Fq ni = inv(add(fsqr(a.c0), fsqr(a.c1)));
  return {fmul(a.c0, ni), neg(fmul(a.c1, ni))};
}

// 1/a by division steps (fp.cuh): the latency-critical inversions of a batch
BG_DEV Fq field_inv_fast(const Fq& a) { return inv_divsteps(a); }
BG_DEV Fq2 field_inv_fast(const Fq2& a) {
  const Fq ni = inv_divsteps(add(fsqr(a.c0), fsqr(a.c1)));
  return {fmul(a.c0, ni), neg(fmul(a.c1, ni))};
}

template <class F>
struct Affine {
  F x, y;
};

template <class F>
struct XYZZ {
  F x, y, zz, zzz;
};

template <class F>
BG_DEV bool is_inf(const Affine<F>& p) { return is_zero(p.x) && is_zero(p.y); }

template <class F>
BG_DEV bool is_inf(const XYZZ<F>& p) { return is_zero(p.zz); }

template <class F>
BG_DEV XYZZ<F> xyzz_inf() {
  XYZZ<F> r;
  r.x = field_one<F>();
  r.y = field_one<F>();
  r.zz = field_zero<F>();
  r.zzz = field_zero<F>();
  return r;
}

template <class F>
BG_DEV XYZZ<F> xyzz_from_affine(const Affine<F>& p) {
  if (is_inf(p)) return xyzz_inf<F>();
  XYZZ<F> r;
  r.x = p.x;
  r.y = p.y;
  r.zz = field_one<F>();
  r.zzz = field_one<F>();
  return r;
}

template <class F>
BG_DEV Affine<F> affine_neg(const Affine<F>& p) {
  Affine<F> r;
  r.x = p.x;
  r.y = neg(p.y);  // neg(0) = 0 keeps the (0, 0) infinity encoding
  return r;
}

template <class F>
BG_DEV XYZZ<F> xyzz_neg(const XYZZ<F>& p) {
  XYZZ<F> r = p;
  r.y = neg(p.y);
  return r;
}

// 2P for affine P != infinity, y != 0 (mdbl-2008-s)
template <class F>
BG_DEV XYZZ<F> xyzz_dbl_affine(const Affine<F>& p) {
  const F u = dbl(p.y);
  const F v = fsqr(u);
  const F w = fmul(u, v);
  const F s = fmul(p.x, v);
  const F x2 = fsqr(p.x);
  const F m = add(dbl(x2), x2);
  XYZZ<F> r;
  r.x = sub(fsqr(m), dbl(s));
  r.y = fmul_sub(m, sub(s, r.x), w, p.y);
  r.zz = v;
  r.zzz = w;
  return r;
}

// 2P (dbl-2008-s-1)
template <class F>
BG_DEV XYZZ<F> xyzz_dbl(const XYZZ<F>& p) {
  if (is_inf(p)) return p;
  const F u = dbl(p.y);
  const F v = fsqr(u);
  const F w = fmul(u, v);
  const F s = fmul(p.x, v);
  const F x2 = fsqr(p.x);
  const F m = add(dbl(x2), x2);
  XYZZ<F> r;
  r.x = sub(fsqr(m), dbl(s));
  r.y = fmul_sub(m, sub(s, r.x), w, p.y);
  r.zz = fmul(v, p.zz);
  r.zzz = fmul(w, p.zzz);
  return r;
}

// P + Q for XYZZ P and affine Q (madd-2008-s)
template <class F>
BG_DEV XYZZ<F> xyzz_madd(const XYZZ<F>& p, const Affine<F>& q) {
  if (is_inf(q)) return p;
  if (is_inf(p)) return xyzz_from_affine(q);
  const F u2 = imul(p.zz, q.x);
  const F s2 = imul(p.zzz, q.y);
  const F pp_ = sub(u2, p.x);
  const F r_ = sub(s2, p.y);
  if (is_zero(pp_)) {
    if (is_zero(r_)) return xyzz_dbl_affine(q);
    return xyzz_inf<F>();
  }
  const F pp = isqr(pp_);
  const F ppp = imul(pp_, pp);
  const F qq = imul(p.x, pp);
  XYZZ<F> r;
  r.x = sub(sub(isqr(r_), ppp), dbl(qq));
  r.y = imul_sub(r_, sub(qq, r.x), p.y, ppp);
  r.zz = imul(p.zz, pp);
  r.zzz = imul(p.zzz, ppp);
  return r;
}

// P + Q for XYZZ P, Q (add-2008-s).  The products that read p and q come first, so neither
// input is live past them: (u1, s1, zz1 zz2, zzz1 zzz2) is p itself in other coordinates
// (x = u1 / (zz1 zz2), y = s1 / (zzz1 zzz2)), and the P = Q case doubles that.
template <class F>
BG_DEV XYZZ<F> xyzz_add(const XYZZ<F>& p, const XYZZ<F>& q) {
  if (is_inf(q)) return p;
  if (is_inf(p)) return q;
  const F u1 = fmul(p.x, q.zz);
  const F u2 = fmul(q.x, p.zz);
  const F s1 = fmul(p.y, q.zzz);
  const F s2 = fmul(q.y, p.zzz);
  const F zz12 = fmul(p.zz, q.zz);
  const F zzz12 = fmul(p.zzz, q.zzz);
  const F pp_ = sub(u2, u1);
  const F r_ = sub(s2, s1);
  if (is_zero(pp_)) {
    if (is_zero(r_)) return xyzz_dbl(XYZZ<F>{u1, s1, zz12, zzz12});
    return xyzz_inf<F>();
  }
  const F pp = fsqr(pp_);
  const F ppp = fmul(pp_, pp);
  const F qq = fmul(u1, pp);
  XYZZ<F> r;
  r.x = sub(sub(fsqr(r_), ppp), dbl(qq));
  r.y = fmul_sub(r_, sub(qq, r.x), s1, ppp);
  r.zz = fmul(zz12, pp);
  r.zzz = fmul(zzz12, ppp);
  return r;
}

// the same with its Fq products inlined, for an addition that is itself out of line
template <class F>
BG_DEV XYZZ<F> xyzz_add_inline(const XYZZ<F>& p, const XYZZ<F>& q) {
  if (is_inf(q)) return p;
  if (is_inf(p)) return q;
  const F u1 = imul(p.x, q.zz);
  const F u2 = imul(q.x, p.zz);
  const F s1 = imul(p.y, q.zzz);
  const F s2 = imul(q.y, p.zzz);
  const F zz12 = imul(p.zz, q.zz);
  const F zzz12 = imul(p.zzz, q.zzz);
  const F pp_ = sub(u2, u1);
  const F r_ = sub(s2, s1);
  if (is_zero(pp_)) {
    if (is_zero(r_)) return xyzz_dbl(XYZZ<F>{u1, s1, zz12, zzz12});
    return xyzz_inf<F>();
  }
  const F pp = isqr(pp_);
  const F ppp = imul(pp_, pp);
  const F qq = imul(u1, pp);
  XYZZ<F> r;
  r.x = sub(sub(isqr(r_), ppp), dbl(qq));
  r.y = imul_sub(r_, sub(qq, r.x), s1, ppp);
  r.zz = imul(zz12, pp);
  r.zzz = imul(zzz12, ppp);
  return r;
}

// ---------------------------------------------------------------- affine pair additions
// P + Q for affine P and Q whose denominator is inverted together with those of many other additions
// (Montgomery's simultaneous inversion): the chord slope and the new coordinates (two products and a
// square) plus three products of the shared inversion, against madd-2008-s's eight products and
// two squares.  The affine infinity is (0, 0) as everywhere on the device, and a missing point.
// a - b as some representative below 2^256 (a, b < p): for the second factor of a product
BG_DEV Fq sub_loose(const Fq& a, const Fq& b) {
  Fq r;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "n"(FqParams::P0), "n"(FqParams::P1), "n"(FqParams::P2), "n"(FqParams::P3), "n"(FqParams::P4),
        "n"(FqParams::P5), "n"(FqParams::P6), "n"(FqParams::P7));
  asm("sub.cc.u32  %0, %0, %8;\n\t"
      "subc.cc.u32 %1, %1, %9;\n\t"
      "subc.cc.u32 %2, %2, %10;\n\t"
      "subc.cc.u32 %3, %3, %11;\n\t"
      "subc.cc.u32 %4, %4, %12;\n\t"
      "subc.cc.u32 %5, %5, %13;\n\t"
      "subc.cc.u32 %6, %6, %14;\n\t"
      "subc.u32    %7, %7, %15;"
      : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]), "+r"(r.v[7])
      : "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return r;
}
// (an Fq2 product adds its factors' halves, which leaves no room)
BG_DEV Fq2 sub_loose(const Fq2& a, const Fq2& b) { return sub(a, b); }

BG_DEV Fq select(bool c, const Fq& a, const Fq& b) {
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = c ? a.v[i] : b.v[i];
  return r;
}
BG_DEV Fq2 select(bool c, const Fq2& a, const Fq2& b) { return {select(c, a.c0, b.c0), select(c, a.c1, b.c1)}; }

// The denominator's last step, for points of equal x (x_Q - x_P = 0, which cannot be a factor of the
// running product): 2 y for the tangent (P = Q), 1 where no addition is due -- Q = -P, two missing
// points, or one and a point of x = 0.  A missing point beside one of x != 0 gives that point's +-x,
// as good a factor as any.
template <class F>
BG_DEV F pair_equal_x(const F& yp, const F& yq) {
  return eq(yp, yq) && !is_zero(yp) ? dbl(yp) : field_one<F>();
}

// The denominator of P + Q as the forward pass took it, with the slope's numerator, and whether the
// sum is (0, 0); mp, mq: P or Q is missing.
template <class F>
BG_DEV bool pair_terms(const Affine<F>& p, const Affine<F>& q, bool mp, bool mq, F& d, F& num) {
  d = sub(q.x, p.x);
  num = sub_loose(q.y, p.y);
  bool none = mp && mq;  // no sum, or a sum at infinity
  if (is_zero(d)) {
    if (!none && eq(p.y, q.y) && !is_zero(p.y)) {
      d = dbl(p.y);
      const F x2 = fsqr(p.x);
      num = add(dbl(x2), x2);
    } else {
      d = field_one<F>();
      none = none || (!mp && !mq);
    }
  }
  return none;
}

// the sum, from pair_terms' numerator and the inverse of its denominator
template <class F>
BG_DEV Affine<F> pair_sum(const Affine<F>& p, const Affine<F>& q, bool mp, bool mq, bool none, const F& num,
                          const F& dinv) {
  const F l = imul(dinv, num);
  Affine<F> r;
  r.x = sub(sub(isqr(l), p.x), q.x);  // the tangent case has q.x = p.x
  r.y = sub(imul(l, sub_loose(p.x, r.x)), p.y);
  if (mp || mq || none) {
    r = mp ? q : p;
    if (none) {
      r.x = field_zero<F>();
      r.y = field_zero<F>();
    }
  }
  return r;
}

// ---------------------------------------------------------------- packed memory layout
// G1 affine: x[8] y[8] (64 B).  G2 affine: x.c0 x.c1 y.c0 y.c1 (128 B).
// XYZZ: x, y, zz, zzz (4 field elements).
BG_DEV void load_elem(Fq& r, const uint32_t* src) { r = load_fp<FqParams>(src); }
BG_DEV void load_elem(Fq2& r, const uint32_t* src) {
  r.c0 = load_fp<FqParams>(src);
  r.c1 = load_fp<FqParams>(src + 8);
}
BG_DEV void store_elem(uint32_t* dst, const Fq& x) { store_fp(dst, x); }
BG_DEV void store_elem(uint32_t* dst, const Fq2& x) {
  store_fp(dst, x.c0);
  store_fp(dst + 8, x.c1);
}

template <class F>
struct FieldWords;
template <>
struct FieldWords<Fq> {
  static constexpr int value = 8;
};
template <>
struct FieldWords<Fq2> {
  static constexpr int value = 16;
};

template <class F>
BG_DEV Affine<F> load_affine(const uint32_t* src) {
  constexpr int W = FieldWords<F>::value;
  Affine<F> p;
  load_elem(p.x, src);
  load_elem(p.y, src + W);
  return p;
}
template <class F>
BG_DEV void store_affine(uint32_t* dst, const Affine<F>& p) {
  constexpr int W = FieldWords<F>::value;
  store_elem(dst, p.x);
  store_elem(dst + W, p.y);
}
template <class F>
BG_DEV XYZZ<F> load_xyzz(const uint32_t* src) {
  constexpr int W = FieldWords<F>::value;
  XYZZ<F> p;
  load_elem(p.x, src);
  load_elem(p.y, src + W);
  load_elem(p.zz, src + 2 * W);
  load_elem(p.zzz, src + 3 * W);
  return p;
}
template <class F>
BG_DEV void store_xyzz(uint32_t* dst, const XYZZ<F>& p) {
  constexpr int W = FieldWords<F>::value;
  store_elem(dst, p.x);
  store_elem(dst + W, p.y);
  store_elem(dst + 2 * W, p.zz);
  store_elem(dst + 3 * W, p.zzz);
}

}  // namespace bg
