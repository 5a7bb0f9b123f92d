// BN254 base field Fq and scalar field Fr on the device: 8 x 32-bit little-endian limbs,
// Montgomery form with R = 2^256 (the value stored for x is x*2^256 mod p).
//
// Reference: the Bend prover keeps the same Montgomery representation in 16 x 16-bit limbs
// (bend2/FORMAT.md:5-12; Fr.mul CIOS at bend2/src/fr.bend:269, Fq.mul at bend2/src/fq.bend:269,
// n0' at fr.bend:4 / fq.bend:4).  Here one limb is 32 bits and a product is 8 rows of operand
// scanning with the reduction interleaved (CIOS, Koc-Acar-Kaliski 1996), written as PTX carry
// chains of 64-bit multiply-adds (fp_wide.cuh).  Every carry chain lives inside a single asm
// statement so no compiler-generated instruction can sit between two .cc instructions.
//
// Invariants: inputs and outputs of add/sub/mul are fully reduced (< p).  Both moduli are
// below 2^254, so a row's running value stays below 2^288 (9 limbs) and the final
// result is below 2p; one conditional subtraction reduces it.
#pragma once
#include <cstdint>

#ifndef BG_DEV
#define BG_DEV __device__ __forceinline__
#endif

namespace bg {

// ---------------------------------------------------------------- moduli and constants
struct FqParams {
  static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t N0 = 0xe4866389u;  // -p^-1 mod 2^32
  // R mod p (Montgomery one)
  static constexpr uint32_t ONE0 = 0xc58f0d9du, ONE1 = 0xd35d438du, ONE2 = 0xf5c70b3du, ONE3 = 0x0a78eb28u,
                            ONE4 = 0x7879462cu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
  // R^2 mod p (turns the inverse of a Montgomery representative into a Montgomery inverse)
  static constexpr uint32_t R2_0 = 0x538afa89u, R2_1 = 0xf32cfc5bu, R2_2 = 0xd44501fbu, R2_3 = 0xb5e71911u,
                            R2_4 = 0x0a417ff6u, R2_5 = 0x47ab1effu, R2_6 = 0xcab8351fu, R2_7 = 0x06d89f71u;
};
struct FrParams {
  static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t N0 = 0xefffffffu;
  static constexpr uint32_t ONE0 = 0x4ffffffbu, ONE1 = 0xac96341cu, ONE2 = 0x9f60cd29u, ONE3 = 0x36fc7695u,
                            ONE4 = 0x7879462eu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
  static constexpr uint32_t R2_0 = 0xae216da7u, R2_1 = 0x1bb8e645u, R2_2 = 0xe35c59e3u, R2_3 = 0x53fe3ab1u,
                            R2_4 = 0x53bb8085u, R2_5 = 0x8c49833du, R2_6 = 0x7f4e44a5u, R2_7 = 0x0216d0b1u;
};

template <class P>
struct Fp {
  uint32_t v[8];
};
using Fq = Fp<FqParams>;
using Fr = Fp<FrParams>;

// ---------------------------------------------------------------- basic predicates
template <class P>
BG_DEV bool is_zero(const Fp<P>& a) {
  uint32_t o = a.v[0] | a.v[1] | a.v[2] | a.v[3] | a.v[4] | a.v[5] | a.v[6] | a.v[7];
  return o == 0;
}
template <class P>
BG_DEV bool eq(const Fp<P>& a, const Fp<P>& b) {
  uint32_t o = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) o |= a.v[i] ^ b.v[i];
  return o == 0;
}
template <class P>
BG_DEV Fp<P> fp_zero() {
  Fp<P> r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = 0;
  return r;
}
template <class P>
BG_DEV Fp<P> fp_one() {
  Fp<P> r;
  r.v[0] = P::ONE0; r.v[1] = P::ONE1; r.v[2] = P::ONE2; r.v[3] = P::ONE3;
  r.v[4] = P::ONE4; r.v[5] = P::ONE5; r.v[6] = P::ONE6; r.v[7] = P::ONE7;
  return r;
}

// ---------------------------------------------------------------- reduction helper
// r = t - p if t >= p else t   (t < 2p, 8 limbs)
template <class P>
BG_DEV void reduce_once(uint32_t* r, const uint32_t* t) {
  uint32_t d0, d1, d2, d3, d4, d5, d6, d7, bw;
  asm("sub.cc.u32  %0, %9,  %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3), "=r"(d4), "=r"(d5), "=r"(d6), "=r"(d7), "=r"(bw)
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
        "n"(P::P0), "n"(P::P1), "n"(P::P2), "n"(P::P3), "n"(P::P4), "n"(P::P5), "n"(P::P6), "n"(P::P7));
  // bw = 0xffffffff when t < p (borrow): keep t
  const bool keep = bw != 0;
  r[0] = keep ? t[0] : d0;
  r[1] = keep ? t[1] : d1;
  r[2] = keep ? t[2] : d2;
  r[3] = keep ? t[3] : d3;
  r[4] = keep ? t[4] : d4;
  r[5] = keep ? t[5] : d5;
  r[6] = keep ? t[6] : d6;
  r[7] = keep ? t[7] : d7;
}

// ---------------------------------------------------------------- add / sub / neg
template <class P>
BG_DEV Fp<P> add(const Fp<P>& a, const Fp<P>& b) {
  uint32_t t[8];
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  Fp<P> r;
  reduce_once<P>(r.v, t);
  return r;
}

template <class P>
BG_DEV Fp<P> sub(const Fp<P>& a, const Fp<P>& b) {
  uint32_t t[8], bw;
  asm("sub.cc.u32  %0, %9,  %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(bw)
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  // on borrow add p back (mask p by bw)
  Fp<P> r;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
        "r"(P::P0 & bw), "r"(P::P1 & bw), "r"(P::P2 & bw), "r"(P::P3 & bw), "r"(P::P4 & bw), "r"(P::P5 & bw),
        "r"(P::P6 & bw), "r"(P::P7 & bw));
  return r;
}

template <class P>
BG_DEV Fp<P> neg(const Fp<P>& a) {
  // p - a, and 0 stays 0
  return sub(fp_zero<P>(), a);
}

template <class P>
BG_DEV Fp<P> dbl(const Fp<P>& a) { return add(a, a); }

// ---------------------------------------------------------------- Montgomery product
// defined in fp_wide.cuh: a b R^-1 mod p for a < p and any 256-bit b; a R^-1 mod p (Montgomery ->
// canonical)
template <class P>
BG_DEV Fp<P> mul(const Fp<P>& a, const Fp<P>& b);
template <class P>
BG_DEV Fp<P> from_mont(const Fp<P>& a);

// squaring product (28 off-diagonal limb products doubled, then one reduction; fp_wide.cuh)
template <class P>
BG_DEV Fp<P> sqr_wide(const Fp<P>& a);
template <class P>
BG_DEV Fp<P> sqr(const Fp<P>& a) { return sqr_wide(a); }

// a^e for a 256-bit exponent given as 8 limbs (square-and-multiply, MSB first)
template <class P>
BG_DEV Fp<P> pow_limbs(const Fp<P>& a, const uint32_t* e) {
  Fp<P> r = fp_one<P>();
  for (int i = 7; i >= 0; i--) {
    for (int b = 31; b >= 0; b--) {
      r = sqr(r);
      if ((e[i] >> b) & 1u) r = mul(r, a);
    }
  }
  return r;
}

// 1/a = a^(p-2) (Fermat); inv(0) = 0 as in bend2/src/fq.bend:1991
template <class P>
BG_DEV Fp<P> inv(const Fp<P>& a) {
  const uint32_t e[8] = {P::P0 - 2u, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  return pow_limbs(a, e);
}

// ---------------------------------------------------------------- inversion by division steps
// 1/a for a Montgomery element a (0 -> 0): the division steps of Bernstein and Yang ("Fast
// constant-time gcd computation and modular inversion", CHES 2019),
//   (delta, f, g) -> (1 - delta, g, (g - f) / 2)                 if delta > 0 and g is odd
//                    (1 + delta, f, (g + (g mod 2) f) / 2)       otherwise
// from delta = 1, f = p, g = a, which end at g = 0 and f = +-1 after at most floor((49 254 + 57) / 17) =
// 735 steps (their Theorem 11.2 with f^2 + 4 g^2 <= 5 2^508).  30 steps at a time run on the low words of
// f and g alone and give a 2 x 2 matrix (entries at most 2^30), which is then applied
// to the whole f and g (exactly divisible by 2^30) and to d and e, which follow f and g modulo p:
// (u d + v e + m p) / 2^30 with the m, centred in +-2^29, that makes it whole, so d and e grow by
// at most p / 2 per matrix and need no reduction before the end.  e starts at R^2, so d ends as
// +-(a R)^-1 R^2, the Montgomery inverse.  The inversion is what a CTA of the batch-affine bucket
// accumulation waits for, so its latency counts: a step is the same few instructions for every input
// (no divergence between lanes that invert together; the sign s of f is a factor of three
// multiply-adds), and a matrix costs
// 90 multiply-adds; binary Euclid with its compares and shifts of whole numbers took about three
// times as long, the Fermat power is 320 dependent products.  Requires a < p (every stored element
// is).
namespace dsteps {
constexpr int32_t kMask = 0x3fffffff;  // 30-bit limbs, nine of them, the top one signed
// limb i of an 8-word number
BG_DEV int32_t limb30(const uint32_t* w, int i) {
  const int bit = 30 * i, l = bit >> 5, s = bit & 31;
  const uint32_t lo = w[l] >> s;
  const uint32_t hi = (s && l + 1 < 8) ? w[l + 1] << (32 - s) : 0u;
  return (int32_t)((lo | hi) & (uint32_t)kMask);
}
// 30 division steps on the low words of f and g.  With `mat` = (u v; q r), 2^i f_i = u f + v g and 2^i g_i =
// q f + r g after i steps for the f and g at entry: a step adds s f to g (s = 0 for an even g, -1 where it
// also moves g into f, else 1), so (q, r) take s (u, v), and f's row doubles where g is halved.
BG_DEV int32_t steps30(int32_t delta, uint32_t f, uint32_t g, int32_t* mat) {
  int32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 6
  for (int i = 0; i < 30; i++) {
    const int32_t odd = (int32_t)(g & 1u);
    const bool move = odd && delta > 0;
    const int32_t s = move ? -1 : odd;
    const uint32_t sum = g + (uint32_t)s * f;
    const int32_t q1 = q + s * u, r1 = r + s * v;
    delta = 1 + (move ? -delta : delta);
    f = move ? g : f;
    u = 2 * (move ? q : u);
    v = 2 * (move ? r : v);
    g = sum >> 1;
    q = q1;
    r = r1;
  }
  mat[0] = u;
  mat[1] = v;
  mat[2] = q;
  mat[3] = r;
  return delta;
}
BG_DEV void update_fg(int32_t* f, int32_t* g, const int32_t* m) {
  int64_t cf = (int64_t)m[0] * f[0] + (int64_t)m[1] * g[0];
  int64_t cg = (int64_t)m[2] * f[0] + (int64_t)m[3] * g[0];
  cf >>= 30;
  cg >>= 30;
#pragma unroll
  for (int i = 1; i < 9; i++) {
    const int32_t fi = f[i], gi = g[i];
    cf += (int64_t)m[0] * fi + (int64_t)m[1] * gi;
    cg += (int64_t)m[2] * fi + (int64_t)m[3] * gi;
    f[i - 1] = (int32_t)cf & kMask;
    g[i - 1] = (int32_t)cg & kMask;
    cf >>= 30;
    cg >>= 30;
  }
  f[8] = (int32_t)cf;
  g[8] = (int32_t)cg;
}
// x -> m with x + m p divisible by 2^30, -2^29 <= m < 2^29 (n30 = -p^-1 mod 2^30)
BG_DEV int32_t centre(int64_t x, uint32_t n30) {
  return (int32_t)(((uint32_t)x * n30) << 2) >> 2;
}
BG_DEV void update_de(int32_t* d, int32_t* e, const int32_t* m, const int32_t* p, uint32_t n30) {
  int64_t cd = (int64_t)m[0] * d[0] + (int64_t)m[1] * e[0];
  int64_t ce = (int64_t)m[2] * d[0] + (int64_t)m[3] * e[0];
  const int32_t md = centre(cd, n30), me = centre(ce, n30);
  cd += (int64_t)md * p[0];
  ce += (int64_t)me * p[0];
  cd >>= 30;
  ce >>= 30;
#pragma unroll
  for (int i = 1; i < 9; i++) {
    const int32_t di = d[i], ei = e[i];
    cd += (int64_t)m[0] * di + (int64_t)m[1] * ei + (int64_t)md * p[i];
    ce += (int64_t)m[2] * di + (int64_t)m[3] * ei + (int64_t)me * p[i];
    d[i - 1] = (int32_t)cd & kMask;
    e[i - 1] = (int32_t)ce & kMask;
    cd >>= 30;
    ce >>= 30;
  }
  d[8] = (int32_t)cd;
  e[8] = (int32_t)ce;
}
}  // namespace dsteps

template <class P>
BG_DEV Fp<P> inv_divsteps(const Fp<P>& a) {
  const uint32_t pw[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  const uint32_t r2[8] = {P::R2_0, P::R2_1, P::R2_2, P::R2_3, P::R2_4, P::R2_5, P::R2_6, P::R2_7};
  int32_t p[9], f[9], g[9], d[9], e[9], m[4];
#pragma unroll
  for (int i = 0; i < 9; i++) {
    p[i] = f[i] = dsteps::limb30(pw, i);
    g[i] = dsteps::limb30(a.v, i);
    d[i] = 0;
    e[i] = dsteps::limb30(r2, i);
  }
  int32_t delta = 1;
#pragma unroll 1
  for (int b = 0; b < 25; b++) {  // 750 steps
    delta = dsteps::steps30(delta, (uint32_t)(f[0] | (f[1] << 30)), (uint32_t)(g[0] | (g[1] << 30)), m);
    dsteps::update_de(d, e, m, p, P::N0 & 0x3fffffffu);
    dsteps::update_fg(f, g, m);
    int32_t left = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) left |= g[i];
    if (left == 0) break;
  }
  // f = +-1, d = +-1/a with |d| <= (1/2 + 25/2) p: make it d f, then add 13 p and subtract 16 p, 8 p,
  // 4 p, 2 p and p where they fit (a = 0 leaves d = 0)
  const int32_t sign = f[8] >> 31;
  int64_t c = 0;
  int32_t t[9];
#pragma unroll
  for (int i = 0; i < 9; i++) {
    c += (int64_t)((d[i] ^ sign) - sign) + (int64_t)13 * p[i];
    t[i] = (int32_t)c & dsteps::kMask;
    c >>= 30;  // ends at zero: the sum lies in [0, 26 p], below 2^259
  }
#pragma unroll
  for (int k = 4; k >= 0; k--) {
    int32_t s[9];
    int64_t bw = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) {
      bw += (int64_t)t[i] - ((int64_t)p[i] << k);
      s[i] = (int32_t)bw & dsteps::kMask;
      bw >>= 30;
    }
    if (bw >= 0) {
#pragma unroll
      for (int i = 0; i < 9; i++) t[i] = s[i];
    }
  }
  Fp<P> r;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    // word i spans 30-bit limbs l and l + 1 (and l + 2 never: 32 <= 60 - 28)
    const int bit = 32 * i, l = bit / 30, sft = bit % 30;
    uint32_t w = (uint32_t)t[l] >> sft;
    w |= (uint32_t)t[l + 1] << (30 - sft);
    if (60 - sft < 32 && l + 2 < 9) w |= (uint32_t)t[l + 2] << (60 - sft);
    r.v[i] = w;
  }
  return r;
}

// ---------------------------------------------------------------- Fq2 = Fq[u]/(u^2 + 1)
// bend2/src/fq2.bend:31-50: Karatsuba product (3M), complex square (2M)
struct Fq2 {
  Fq c0, c1;
};

BG_DEV bool is_zero(const Fq2& a) { return is_zero(a.c0) && is_zero(a.c1); }
BG_DEV bool eq(const Fq2& a, const Fq2& b) { return eq(a.c0, b.c0) && eq(a.c1, b.c1); }
BG_DEV Fq2 add(const Fq2& a, const Fq2& b) { return {add(a.c0, b.c0), add(a.c1, b.c1)}; }
BG_DEV Fq2 sub(const Fq2& a, const Fq2& b) { return {sub(a.c0, b.c0), sub(a.c1, b.c1)}; }
BG_DEV Fq2 neg(const Fq2& a) { return {neg(a.c0), neg(a.c1)}; }
BG_DEV Fq2 dbl(const Fq2& a) { return {dbl(a.c0), dbl(a.c1)}; }
BG_DEV Fq2 mul(const Fq2& a, const Fq2& b) {
  const Fq t0 = mul(a.c0, b.c0);
  const Fq t1 = mul(a.c1, b.c1);
  const Fq t2 = mul(add(a.c0, a.c1), add(b.c0, b.c1));
  return {sub(t0, t1), sub(sub(t2, t0), t1)};
}
BG_DEV Fq2 sqr(const Fq2& a) {
  return {mul(add(a.c0, a.c1), sub(a.c0, a.c1)), mul(dbl(a.c0), a.c1)};
}

template <class F>
BG_DEV F field_zero();
template <>
BG_DEV Fq field_zero<Fq>() { return fp_zero<FqParams>(); }
template <>
BG_DEV Fr field_zero<Fr>() { return fp_zero<FrParams>(); }
template <>
BG_DEV Fq2 field_zero<Fq2>() { return {fp_zero<FqParams>(), fp_zero<FqParams>()}; }

template <class F>
BG_DEV F field_one();
template <>
BG_DEV Fq field_one<Fq>() { return fp_one<FqParams>(); }
template <>
BG_DEV Fr field_one<Fr>() { return fp_one<FrParams>(); }
template <>
BG_DEV Fq2 field_one<Fq2>() { return {fp_one<FqParams>(), fp_zero<FqParams>()}; }

// ---------------------------------------------------------------- global memory helpers
// 128-bit loads/stores of packed elements (an element is 32 bytes, 32-byte aligned)
template <class P>
BG_DEV Fp<P> load_fp(const uint32_t* src) {
  const uint4 a = reinterpret_cast<const uint4*>(src)[0];
  const uint4 b = reinterpret_cast<const uint4*>(src)[1];
  Fp<P> r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}
template <class P>
BG_DEV void store_fp(uint32_t* dst, const Fp<P>& x) {
  reinterpret_cast<uint4*>(dst)[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  reinterpret_cast<uint4*>(dst)[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

}  // namespace bg

#include "fp_wide.cuh"
