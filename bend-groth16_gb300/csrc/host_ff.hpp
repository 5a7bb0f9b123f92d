// Host-side BN254 arithmetic for the library's serial steps: the window combination of an
// MSM (a few hundred doublings), normalisation to affine, the Groth16 combine
// (bend2/src/groth16.bend:298-308), NTT twiddle / coset table seeds, and canonical
// conversion for printing.  4 x 64-bit little-endian limbs, Montgomery form with R = 2^256
// (the same integers the device holds as 8 x 32-bit limbs on a little-endian host).
#pragma once
#include <cstdint>
#include <cstring>

namespace bgh {

typedef unsigned __int128 u128;

struct Mod {
  uint64_t p[4];
  uint64_t n0;      // -p^-1 mod 2^64
  uint64_t one[4];  // R mod p
  uint64_t r2[4];   // R^2 mod p
};

// p from bend2/src/fq.bend:2 and bend2/src/fr.bend:2; compile-time constants, so every product
// below is built for its modulus
inline constexpr Mod FQ = {
    {0x3c208c16d87cfd47ull, 0x97816a916871ca8dull, 0xb85045b68181585dull, 0x30644e72e131a029ull},
    0x87d20782e4866389ull,
    {0xd35d438dc58f0d9dull, 0x0a78eb28f5c70b3dull, 0x666ea36f7879462cull, 0x0e0a77c19a07df2full},
    {0xf32cfc5b538afa89ull, 0xb5e71911d44501fbull, 0x47ab1eff0a417ff6ull, 0x06d89f71cab8351full}};
inline constexpr Mod FR = {
    {0x43e1f593f0000001ull, 0x2833e84879b97091ull, 0xb85045b68181585dull, 0x30644e72e131a029ull},
    0xc2e1f593efffffffull,
    {0xac96341c4ffffffbull, 0x36fc76959f60cd29ull, 0x666ea36f7879462eull, 0x0e0a77c19a07df2full},
    {0x1bb8e645ae216da7ull, 0x53fe3ab1e35c59e3ull, 0x8c49833d53bb8085ull, 0x0216d0b17f4e44a5ull}};

struct Fe {
  uint64_t v[4];
};

inline bool fe_is_zero(const Fe& a) { return (a.v[0] | a.v[1] | a.v[2] | a.v[3]) == 0; }
inline bool fe_eq(const Fe& a, const Fe& b) {
  return a.v[0] == b.v[0] && a.v[1] == b.v[1] && a.v[2] == b.v[2] && a.v[3] == b.v[3];
}
inline Fe fe_zero() { return Fe{{0, 0, 0, 0}}; }
inline Fe fe_one(const Mod& m) { return Fe{{m.one[0], m.one[1], m.one[2], m.one[3]}}; }
inline Fe fe_raw(uint64_t x) { return Fe{{x, 0, 0, 0}}; }

// a >= b as 256-bit integers
inline bool geq(const uint64_t* a, const uint64_t* b) {
  for (int i = 3; i >= 0; i--) {
    if (a[i] != b[i]) return a[i] > b[i];
  }
  return true;
}
inline uint64_t sub4(uint64_t* r, const uint64_t* a, const uint64_t* b) {
  u128 d = (u128)a[0] - b[0];
  r[0] = (uint64_t)d;
  d = (u128)a[1] - b[1] - ((uint64_t)(d >> 64) & 1);
  r[1] = (uint64_t)d;
  d = (u128)a[2] - b[2] - ((uint64_t)(d >> 64) & 1);
  r[2] = (uint64_t)d;
  d = (u128)a[3] - b[3] - ((uint64_t)(d >> 64) & 1);
  r[3] = (uint64_t)d;
  return (uint64_t)(d >> 64) & 1;
}
inline uint64_t add4(uint64_t* r, const uint64_t* a, const uint64_t* b) {
  u128 s = (u128)a[0] + b[0];
  r[0] = (uint64_t)s;
  s = (u128)a[1] + b[1] + (uint64_t)(s >> 64);
  r[1] = (uint64_t)s;
  s = (u128)a[2] + b[2] + (uint64_t)(s >> 64);
  r[2] = (uint64_t)s;
  s = (u128)a[3] + b[3] + (uint64_t)(s >> 64);
  r[3] = (uint64_t)s;
  return (uint64_t)(s >> 64);
}
// r = t - p when t >= p, else t (t < 2p), without a branch
inline Fe fe_cond_sub(const Mod& m, const uint64_t* t) {
  uint64_t d[4];
  const uint64_t keep = 0 - sub4(d, t, m.p);  // all ones when t < p
  Fe r;
  for (int i = 0; i < 4; i++) r.v[i] = d[i] ^ ((d[i] ^ t[i]) & keep);
  return r;
}

inline Fe fe_add(const Mod& m, const Fe& a, const Fe& b) {
  uint64_t t[4];
  add4(t, a.v, b.v);  // < 2p < 2^255, no carry out
  return fe_cond_sub(m, t);
}
inline Fe fe_sub(const Mod& m, const Fe& a, const Fe& b) {
  Fe r;
  const uint64_t mask = 0 - sub4(r.v, a.v, b.v);
  const uint64_t pm[4] = {m.p[0] & mask, m.p[1] & mask, m.p[2] & mask, m.p[3] & mask};
  add4(r.v, r.v, pm);
  return r;
}
inline Fe fe_neg(const Mod& m, const Fe& a) { return fe_sub(m, fe_zero(), a); }
inline Fe fe_dbl(const Mod& m, const Fe& a) { return fe_add(m, a, a); }

// Row b of a CIOS Montgomery product: t = (t + a b + q p) / 2^64 with the q that clears limb 0.
// For a < p < 2^254 the sum stays below 2p after every row, so four limbs hold it and the two
// carry words can be added without overflow.
inline __attribute__((always_inline)) void fe_mul_row(const Mod& m, uint64_t* t, const uint64_t* a, uint64_t b) {
  u128 s = (u128)a[0] * b + t[0];
  const uint64_t q = (uint64_t)s * m.n0;
  uint64_t c = (uint64_t)(s >> 64);
  u128 u = (u128)q * m.p[0] + (uint64_t)s;
  s = (u128)a[1] * b + t[1] + c;
  c = (uint64_t)(s >> 64);
  u = (u128)q * m.p[1] + (uint64_t)s + (uint64_t)(u >> 64);
  t[0] = (uint64_t)u;
  s = (u128)a[2] * b + t[2] + c;
  c = (uint64_t)(s >> 64);
  u = (u128)q * m.p[2] + (uint64_t)s + (uint64_t)(u >> 64);
  t[1] = (uint64_t)u;
  s = (u128)a[3] * b + t[3] + c;
  c = (uint64_t)(s >> 64);
  u = (u128)q * m.p[3] + (uint64_t)s + (uint64_t)(u >> 64);
  t[2] = (uint64_t)u;
  t[3] = (uint64_t)(u >> 64) + c;
}
// a b 2^-256 mod p for a < p and any 256-bit b
inline __attribute__((always_inline)) Fe fe_mul(const Mod& m, const Fe& a, const Fe& b) {
  uint64_t t[4] = {0, 0, 0, 0};
  fe_mul_row(m, t, a.v, b.v[0]);
  fe_mul_row(m, t, a.v, b.v[1]);
  fe_mul_row(m, t, a.v, b.v[2]);
  fe_mul_row(m, t, a.v, b.v[3]);
  return fe_cond_sub(m, t);
}
// t = a b (512 bits)
inline __attribute__((always_inline)) void fe_wide_row(uint64_t* t, const uint64_t* a, uint64_t b) {
  u128 s = (u128)a[0] * b + t[0];
  t[0] = (uint64_t)s;
  s = (u128)a[1] * b + t[1] + (uint64_t)(s >> 64);
  t[1] = (uint64_t)s;
  s = (u128)a[2] * b + t[2] + (uint64_t)(s >> 64);
  t[2] = (uint64_t)s;
  s = (u128)a[3] * b + t[3] + (uint64_t)(s >> 64);
  t[3] = (uint64_t)s;
  t[4] = (uint64_t)(s >> 64);
}
inline __attribute__((always_inline)) void fe_wide(uint64_t* t, const uint64_t* a, const uint64_t* b) {
  t[0] = t[1] = t[2] = t[3] = 0;
  fe_wide_row(t, a, b[0]);
  fe_wide_row(t + 1, a, b[1]);
  fe_wide_row(t + 2, a, b[2]);
  fe_wide_row(t + 3, a, b[3]);
}
// t -= u (512 bits), returns the borrow
inline __attribute__((always_inline)) uint64_t fe_wide_sub(uint64_t* t, const uint64_t* u) {
  uint64_t borrow = 0;
  for (int i = 0; i < 8; i++) {
    const u128 d = (u128)t[i] - u[i] - borrow;
    t[i] = (uint64_t)d;
    borrow = (uint64_t)(d >> 64) & 1;
  }
  return borrow;
}
// t 2^-256 mod p for t < p 2^256: the low half reduced alone (at most p) plus the high half
inline __attribute__((always_inline)) Fe fe_wide_redc(const Mod& m, const uint64_t* t) {
  uint64_t r[4] = {t[0], t[1], t[2], t[3]};
  for (int i = 0; i < 4; i++) {
    const uint64_t q = r[0] * m.n0;
    u128 u = (u128)q * m.p[0] + r[0];
    u = (u128)q * m.p[1] + r[1] + (uint64_t)(u >> 64);
    r[0] = (uint64_t)u;
    u = (u128)q * m.p[2] + r[2] + (uint64_t)(u >> 64);
    r[1] = (uint64_t)u;
    u = (u128)q * m.p[3] + r[3] + (uint64_t)(u >> 64);
    r[2] = (uint64_t)u;
    r[3] = (uint64_t)(u >> 64);
  }
  add4(r, r, t + 4);
  return fe_cond_sub(m, r);
}
inline Fe fe_sqr(const Mod& m, const Fe& a) { return fe_mul(m, a, a); }
// (any 256-bit a)
inline Fe fe_to_mont(const Mod& m, const Fe& a) {
  return fe_mul(m, Fe{{m.r2[0], m.r2[1], m.r2[2], m.r2[3]}}, a);
}
inline Fe fe_from_mont(const Mod& m, const Fe& a) { return fe_mul(m, fe_raw(1), a); }
// a mod p for any 256-bit a: what a caller's words become before the arithmetic here, whose first
// factors have to be below p
inline Fe fe_reduce(const Mod& m, Fe a) {
  while (geq(a.v, m.p)) sub4(a.v, a.v, m.p);  // at most five times
  return a;
}

inline Fe fe_pow(const Mod& m, const Fe& a, const uint64_t e[4]) {
  Fe r = fe_one(m);
  for (int i = 3; i >= 0; i--)
    for (int b = 63; b >= 0; b--) {
      r = fe_sqr(m, r);
      if ((e[i] >> b) & 1) r = fe_mul(m, r, a);
    }
  return r;
}
inline Fe fe_pow_u64(const Mod& m, const Fe& a, uint64_t e) {
  const uint64_t ee[4] = {e, 0, 0, 0};
  return fe_pow(m, a, ee);
}
// 1/a for a Montgomery element below p (0 -> 0): Bernstein and Yang's division steps, as the
// device's inversion (fp.cuh, which has the recurrence), 62 steps to a matrix and five signed 62-bit
// limbs.  2 us against the Fermat power's 8; a proof's host tail makes three, a standalone MSM's one.
namespace dsteps {
constexpr int64_t kMask = ((int64_t)1 << 62) - 1;
struct S62 {
  int64_t v[5];
};
inline S62 split(const uint64_t* w) {
  return {{(int64_t)(w[0] & kMask), (int64_t)((w[0] >> 62 | w[1] << 2) & kMask), (int64_t)((w[1] >> 60 | w[2] << 4) & kMask),
           (int64_t)((w[2] >> 58 | w[3] << 6) & kMask), (int64_t)(w[3] >> 56)}};
}
// (a run of even g is taken at once: the time depends on the input, as that of the additions does)
inline int64_t steps62(int64_t delta, uint64_t f, uint64_t g, int64_t* m) {
  int64_t u = 1, v = 0, q = 0, r = 1;
  for (int left = 62;;) {
    const int even = __builtin_ctzll(g | (uint64_t)1 << left);
    delta += even;
    g >>= even;
    u = (int64_t)((uint64_t)u << even);
    v = (int64_t)((uint64_t)v << even);
    left -= even;
    if (left == 0) break;
    const bool move = delta > 0;
    const uint64_t f0 = f;
    const int64_t u0 = u, v0 = v;
    f = move ? g : f;
    u = 2 * (move ? q : u);
    v = 2 * (move ? r : v);
    g = (g + (move ? 0 - f0 : f0)) >> 1;
    q += move ? -u0 : u0;
    r += move ? -v0 : v0;
    delta = 1 + (move ? -delta : delta);
    left--;
  }
  m[0] = u;
  m[1] = v;
  m[2] = q;
  m[3] = r;
  return delta;
}
// (a, b) = (m0 a + m1 b + k p, m2 a + m3 b + l p) / 2^62 with the k, l (n62 = -p^-1 mod 2^62) that make
// them whole, centred; without p (n62 = 0) for the pair that is divisible by itself
inline void apply(S62& a, S62& b, const int64_t* m, const S62& p, uint64_t n62) {
  typedef __int128 i128;
  i128 ca = (i128)m[0] * a.v[0] + (i128)m[1] * b.v[0], cb = (i128)m[2] * a.v[0] + (i128)m[3] * b.v[0];
  const int64_t k = (int64_t)(((uint64_t)ca * n62) << 2) >> 2, l = (int64_t)(((uint64_t)cb * n62) << 2) >> 2;
  ca = (ca + (i128)k * p.v[0]) >> 62;
  cb = (cb + (i128)l * p.v[0]) >> 62;
  for (int i = 1; i < 5; i++) {
    const int64_t ai = a.v[i], bi = b.v[i];
    ca += (i128)m[0] * ai + (i128)m[1] * bi + (i128)k * p.v[i];
    cb += (i128)m[2] * ai + (i128)m[3] * bi + (i128)l * p.v[i];
    a.v[i - 1] = (int64_t)ca & kMask;
    b.v[i - 1] = (int64_t)cb & kMask;
    ca >>= 62;
    cb >>= 62;
  }
  a.v[4] = (int64_t)ca;
  b.v[4] = (int64_t)cb;
}
}  // namespace dsteps
inline Fe fe_inv(const Mod& m, const Fe& a) {
  using dsteps::S62;
  const S62 p = dsteps::split(m.p);
  S62 f = p, g = dsteps::split(a.v), d = {{0, 0, 0, 0, 0}}, e = dsteps::split(m.r2);
  int64_t delta = 1, mat[4];
  for (int i = 0; i < 12; i++) {  // 744 steps, of which 735 suffice
    delta = dsteps::steps62(delta, (uint64_t)f.v[0] | (uint64_t)f.v[1] << 62, (uint64_t)g.v[0] | (uint64_t)g.v[1] << 62, mat);
    dsteps::apply(d, e, mat, p, m.n0 & (uint64_t)dsteps::kMask);
    dsteps::apply(f, g, mat, p, 0);
    if ((g.v[0] | g.v[1] | g.v[2] | g.v[3] | g.v[4]) == 0) break;
  }
  // f = +-1 and |d| <= (1/2 + 12/2) p: d f + 7 p lies in (0, 14 p), below 2^258
  const int64_t sign = f.v[4] >> 63;
  __int128 c = 0;
  uint64_t t[5];
  for (int i = 0; i < 5; i++) {
    c += (__int128)((d.v[i] ^ sign) - sign) + (__int128)7 * p.v[i];
    t[i] = (uint64_t)c & (uint64_t)dsteps::kMask;
    c >>= 62;
  }
  for (int k = 3; k >= 0; k--) {  // minus 8 p, 4 p, 2 p, p where they fit
    uint64_t s[5];
    __int128 bw = 0;
    for (int i = 0; i < 5; i++) {
      bw += (__int128)t[i] - ((__int128)p.v[i] << k);
      s[i] = (uint64_t)bw & (uint64_t)dsteps::kMask;
      bw >>= 62;
    }
    if (bw >= 0)
      for (int i = 0; i < 5; i++) t[i] = s[i];
  }
  return Fe{{t[0] | t[1] << 62, t[1] >> 2 | t[2] << 60, t[2] >> 4 | t[3] << 58, t[3] >> 6 | t[4] << 56}};
}

// ---------------------------------------------------------------- Fq2 = Fq[u]/(u^2+1)
struct Fe2 {
  Fe c0, c1;
};
inline bool fe_is_zero(const Fe2& a) { return fe_is_zero(a.c0) && fe_is_zero(a.c1); }
inline bool fe_eq(const Fe2& a, const Fe2& b) { return fe_eq(a.c0, b.c0) && fe_eq(a.c1, b.c1); }

// Field adaptors so curve code is generic over Fq and Fq2
struct FqOps {
  typedef Fe T;
  static T zero() { return fe_zero(); }
  static T one() { return fe_one(FQ); }
  static T add(const T& a, const T& b) { return fe_add(FQ, a, b); }
  static T sub(const T& a, const T& b) { return fe_sub(FQ, a, b); }
  static T neg(const T& a) { return fe_neg(FQ, a); }
  static T mul(const T& a, const T& b) { return fe_mul(FQ, a, b); }
  static T sqr(const T& a) { return fe_mul(FQ, a, a); }
  static T inv(const T& a) { return fe_inv(FQ, a); }
  static bool is_zero(const T& a) { return fe_is_zero(a); }
  static bool eq(const T& a, const T& b) { return fe_eq(a, b); }
  static constexpr int WORDS = 8;  // 32-bit words
};
struct Fq2Ops {
  typedef Fe2 T;
  static T zero() { return {fe_zero(), fe_zero()}; }
  static T one() { return {fe_one(FQ), fe_zero()}; }
  static T add(const T& a, const T& b) { return {fe_add(FQ, a.c0, b.c0), fe_add(FQ, a.c1, b.c1)}; }
  static T sub(const T& a, const T& b) { return {fe_sub(FQ, a.c0, b.c0), fe_sub(FQ, a.c1, b.c1)}; }
  static T neg(const T& a) { return {fe_neg(FQ, a.c0), fe_neg(FQ, a.c1)}; }
  // Karatsuba on unreduced sums with two reductions; c0 = a0 b0 - a1 b1 takes p 2^256 back when it
  // goes below zero
  static T mul(const T& a, const T& b) {
    uint64_t t0[8], t1[8], t2[8], sa[4], sb[4];
    fe_wide(t0, a.c0.v, b.c0.v);
    fe_wide(t1, a.c1.v, b.c1.v);
    add4(sa, a.c0.v, a.c1.v);
    add4(sb, b.c0.v, b.c1.v);
    fe_wide(t2, sa, sb);
    fe_wide_sub(t2, t0);
    fe_wide_sub(t2, t1);
    const uint64_t mask = 0 - fe_wide_sub(t0, t1);
    const uint64_t pm[4] = {FQ.p[0] & mask, FQ.p[1] & mask, FQ.p[2] & mask, FQ.p[3] & mask};
    add4(t0 + 4, t0 + 4, pm);
    return {fe_wide_redc(FQ, t0), fe_wide_redc(FQ, t2)};
  }
  static T sqr(const T& a) {
    return {fe_mul(FQ, fe_add(FQ, a.c0, a.c1), fe_sub(FQ, a.c0, a.c1)), fe_mul(FQ, fe_dbl(FQ, a.c0), a.c1)};
  }
  static T inv(const T& a) {
    Fe n = fe_add(FQ, fe_sqr(FQ, a.c0), fe_sqr(FQ, a.c1));
    Fe ni = fe_inv(FQ, n);
    return {fe_mul(FQ, a.c0, ni), fe_neg(FQ, fe_mul(FQ, a.c1, ni))};
  }
  static bool is_zero(const T& a) { return fe_is_zero(a); }
  static bool eq(const T& a, const T& b) { return fe_eq(a, b); }
  static constexpr int WORDS = 16;
};

// ---------------------------------------------------------------- curve points
template <class F>
struct Aff {
  typename F::T x, y;
  bool inf;
};
template <class F>
struct Xyzz {
  typename F::T x, y, zz, zzz;
};

template <class F>
Xyzz<F> xyzz_inf() {
  return {F::one(), F::one(), F::zero(), F::zero()};
}
template <class F>
bool xyzz_is_inf(const Xyzz<F>& p) {
  return F::is_zero(p.zz);
}
template <class F>
Xyzz<F> xyzz_from(const Aff<F>& a) {
  if (a.inf) return xyzz_inf<F>();
  return {a.x, a.y, F::one(), F::one()};
}
template <class F>
Xyzz<F> xyzz_dbl(const Xyzz<F>& p) {
  if (xyzz_is_inf(p)) return p;
  auto u = F::add(p.y, p.y);
  auto v = F::sqr(u);
  auto w = F::mul(u, v);
  auto s = F::mul(p.x, v);
  auto x2 = F::sqr(p.x);
  auto m = F::add(F::add(x2, x2), x2);
  Xyzz<F> r;
  r.x = F::sub(F::sqr(m), F::add(s, s));
  r.y = F::sub(F::mul(m, F::sub(s, r.x)), F::mul(w, p.y));
  r.zz = F::mul(v, p.zz);
  r.zzz = F::mul(w, p.zzz);
  return r;
}
template <class F>
Xyzz<F> xyzz_add(const Xyzz<F>& p, const Xyzz<F>& q) {
  if (xyzz_is_inf(q)) return p;
  if (xyzz_is_inf(p)) return q;
  auto u1 = F::mul(p.x, q.zz);
  auto u2 = F::mul(q.x, p.zz);
  auto s1 = F::mul(p.y, q.zzz);
  auto s2 = F::mul(q.y, p.zzz);
  auto pp_ = F::sub(u2, u1);
  auto r_ = F::sub(s2, s1);
  if (F::is_zero(pp_)) {
    if (F::is_zero(r_)) return xyzz_dbl(p);
    return xyzz_inf<F>();
  }
  auto pp = F::sqr(pp_);
  auto ppp = F::mul(pp_, pp);
  auto qq = F::mul(u1, pp);
  Xyzz<F> r;
  r.x = F::sub(F::sub(F::sqr(r_), ppp), F::add(qq, qq));
  r.y = F::sub(F::mul(r_, F::sub(qq, r.x)), F::mul(s1, ppp));
  r.zz = F::mul(F::mul(p.zz, q.zz), pp);
  r.zzz = F::mul(F::mul(p.zzz, q.zzz), ppp);
  return r;
}
// Jacobian points (x = X / Z^2, y = Y / Z^3) for the Horner chain of an MSM, most of whose steps are
// doublings: dbl-2009-l takes 2 products and 5 squares where the XYZZ doubling takes 6 and 3.
template <class F>
struct Jac {
  typename F::T x, y, z;
};
template <class F>
Jac<F> jac_inf() {
  return {F::one(), F::one(), F::zero()};
}
template <class F>
Jac<F> jac_dbl(const Jac<F>& p) {
  if (F::is_zero(p.z)) return p;
  const auto a = F::sqr(p.x), b = F::sqr(p.y), c = F::sqr(b);
  auto d = F::sub(F::sub(F::sqr(F::add(p.x, b)), a), c);
  d = F::add(d, d);
  const auto e = F::add(F::add(a, a), a);
  Jac<F> r;
  r.x = F::sub(F::sqr(e), F::add(d, d));
  auto c8 = F::add(c, c);
  c8 = F::add(c8, c8);
  c8 = F::add(c8, c8);
  r.y = F::sub(F::mul(e, F::sub(d, r.x)), c8);
  const auto yz = F::mul(p.y, p.z);
  r.z = F::add(yz, yz);
  return r;
}
// p + q for Jacobian p and XYZZ q (x = X / ZZ, y = Y / ZZZ): q with Z = ZZZ is (X ZZ^2, Y ZZZ^2, ZZZ)
template <class F>
Jac<F> jac_add(const Jac<F>& p, const Xyzz<F>& q) {
  if (F::is_zero(q.zz)) return p;
  const auto qz2 = F::sqr(q.zzz), qx = F::mul(q.x, F::sqr(q.zz)), qy = F::mul(q.y, qz2);
  if (F::is_zero(p.z)) return {qx, qy, q.zzz};
  const auto pz2 = F::sqr(p.z);
  const auto u1 = F::mul(p.x, qz2), u2 = F::mul(qx, pz2);
  const auto s1 = F::mul(p.y, F::mul(q.zzz, qz2)), s2 = F::mul(qy, F::mul(p.z, pz2));
  const auto h = F::sub(u2, u1), r_ = F::sub(s2, s1);
  if (F::is_zero(h)) return F::is_zero(r_) ? jac_dbl(p) : jac_inf<F>();
  const auto hh = F::sqr(h), hhh = F::mul(h, hh), v = F::mul(u1, hh);
  Jac<F> r;
  r.x = F::sub(F::sub(F::sqr(r_), hhh), F::add(v, v));
  r.y = F::sub(F::mul(r_, F::sub(v, r.x)), F::mul(s1, hhh));
  r.z = F::mul(F::mul(p.z, q.zzz), h);
  return r;
}
template <class F>
Xyzz<F> xyzz_from_jac(const Jac<F>& p) {
  const auto zz = F::sqr(p.z);
  return {p.x, p.y, zz, F::mul(zz, p.z)};
}
template <class F>
Xyzz<F> xyzz_neg(const Xyzz<F>& p) {
  Xyzz<F> r = p;
  r.y = F::neg(p.y);
  return r;
}
template <class F>
Aff<F> xyzz_to_affine(const Xyzz<F>& p) {
  Aff<F> a;
  if (xyzz_is_inf(p)) {
    a.x = F::zero();
    a.y = F::zero();
    a.inf = true;
    return a;
  }
  // x = X/ZZ, y = Y/ZZZ with one inversion: 1/(ZZ*ZZZ)
  auto t = F::inv(F::mul(p.zz, p.zzz));
  a.x = F::mul(p.x, F::mul(t, p.zzz));
  a.y = F::mul(p.y, F::mul(t, p.zz));
  a.inf = false;
  return a;
}
// k*P for a canonical scalar k (4 x 64 little-endian), 4-bit fixed window
template <class F>
Xyzz<F> xyzz_mul(const Xyzz<F>& p, const uint64_t k[4]) {
  Xyzz<F> tab[16];
  tab[0] = xyzz_inf<F>();
  for (int i = 1; i < 16; i++) tab[i] = xyzz_add(tab[i - 1], p);
  Xyzz<F> r = xyzz_inf<F>();
  for (int i = 63; i >= 0; i--) {
    for (int d = 0; d < 4; d++) r = xyzz_dbl(r);
    unsigned nib = (unsigned)(k[i / 16] >> (4 * (i % 16))) & 15u;
    if (nib) r = xyzz_add(r, tab[nib]);
  }
  return r;
}

// k*P for a 64-bit k, the same 4-bit fixed window
template <class F>
Xyzz<F> xyzz_mul64(const Xyzz<F>& p, uint64_t k) {
  Xyzz<F> tab[16];
  tab[0] = xyzz_inf<F>();
  for (int i = 1; i < 16; i++) tab[i] = xyzz_add(tab[i - 1], p);
  Xyzz<F> r = xyzz_inf<F>();
  for (int i = 15; i >= 0; i--) {
    for (int d = 0; d < 4; d++) r = xyzz_dbl(r);
    const unsigned nib = (unsigned)(k >> (4 * i)) & 15u;
    if (nib) r = xyzz_add(r, tab[nib]);
  }
  return r;
}

// ---------------------------------------------------------------- wire-format conversion
// FORMAT.md element: 16 words, each a 16-bit limb (bend2/FORMAT.md:7-8)
inline Fe fe_from_words16(const uint32_t* w) {
  Fe r;
  for (int i = 0; i < 4; i++) {
    r.v[i] = (uint64_t)(w[4 * i] & 0xffff) | ((uint64_t)(w[4 * i + 1] & 0xffff) << 16) |
             ((uint64_t)(w[4 * i + 2] & 0xffff) << 32) | ((uint64_t)(w[4 * i + 3] & 0xffff) << 48);
  }
  return r;
}
inline void fe_to_words16(uint32_t* w, const Fe& a) {
  for (int i = 0; i < 16; i++) w[i] = (uint32_t)(a.v[i / 4] >> (16 * (i % 4))) & 0xffffu;
}
inline Fe fe_from_words32(const uint32_t* w) {
  Fe r;
  for (int i = 0; i < 4; i++) r.v[i] = (uint64_t)w[2 * i] | ((uint64_t)w[2 * i + 1] << 32);
  return r;
}
inline void fe_to_words32(uint32_t* w, const Fe& a) {
  for (int i = 0; i < 8; i++) w[i] = (uint32_t)(a.v[i / 2] >> (32 * (i % 2)));
}

template <class F>
void elem_from_words32(typename F::T& r, const uint32_t* w);
template <>
inline void elem_from_words32<FqOps>(Fe& r, const uint32_t* w) {
  r = fe_from_words32(w);
}
template <>
inline void elem_from_words32<Fq2Ops>(Fe2& r, const uint32_t* w) {
  r.c0 = fe_from_words32(w);
  r.c1 = fe_from_words32(w + 8);
}
template <class F>
void elem_to_words32(uint32_t* w, const typename F::T& a);
template <>
inline void elem_to_words32<FqOps>(uint32_t* w, const Fe& a) {
  fe_to_words32(w, a);
}
template <>
inline void elem_to_words32<Fq2Ops>(uint32_t* w, const Fe2& a) {
  fe_to_words32(w, a.c0);
  fe_to_words32(w + 8, a.c1);
}
template <class F>
Xyzz<F> xyzz_from_words32(const uint32_t* w) {
  Xyzz<F> p;
  elem_from_words32<F>(p.x, w);
  elem_from_words32<F>(p.y, w + F::WORDS);
  elem_from_words32<F>(p.zz, w + 2 * F::WORDS);
  elem_from_words32<F>(p.zzz, w + 3 * F::WORDS);
  return p;
}
template <class F>
Aff<F> aff_from_words32(const uint32_t* w) {
  Aff<F> a;
  elem_from_words32<F>(a.x, w);
  elem_from_words32<F>(a.y, w + F::WORDS);
  a.inf = F::is_zero(a.x) && F::is_zero(a.y);
  return a;
}
// the same from a caller's words, whose coordinates may lie at or above p
inline void elem_reduce(Fe& a) { a = fe_reduce(FQ, a); }
inline void elem_reduce(Fe2& a) { a = {fe_reduce(FQ, a.c0), fe_reduce(FQ, a.c1)}; }
template <class F>
Aff<F> aff_from_input32(const uint32_t* w) {
  Aff<F> a = aff_from_words32<F>(w);
  elem_reduce(a.x);
  elem_reduce(a.y);
  return a;
}
// A proof's blinding scalars r, s and r s, canonical, from their 16-word Montgomery form (rs.bin: r,
// then s; words at or above the modulus are taken modulo it)
inline void blinding_scalars(const uint32_t* rs16, uint64_t r[4], uint64_t s[4], uint64_t rs[4]) {
  const Fe rm = fe_from_words16(rs16), sm = fe_from_words16(rs16 + 16);
  const Fe rc = fe_from_mont(FR, rm), sc = fe_from_mont(FR, sm);
  const Fe prod = fe_mul(FR, rc, sm);
  for (int i = 0; i < 4; i++) {
    r[i] = rc.v[i];
    s[i] = sc.v[i];
    rs[i] = prod.v[i];
  }
}
template <class F>
void aff_to_words32(uint32_t* w, const Aff<F>& a) {
  if (a.inf) {
    memset(w, 0, sizeof(uint32_t) * 2 * F::WORDS);
    return;
  }
  elem_to_words32<F>(w, a.x);
  elem_to_words32<F>(w + F::WORDS, a.y);
}

}  // namespace bgh
