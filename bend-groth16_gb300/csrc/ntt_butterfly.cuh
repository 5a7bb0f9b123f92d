// The butterflies of the NTT passes (ntt.cu) on loosely reduced values.
//
// Values inside a pass are kept loosely reduced (after Harvey, "Faster arithmetic for
// number-theoretic transforms", 2014): below 2r between DIF stages, below 4r between DIT ones, and
// only stores to memory reduce fully.  A twiddle product takes any factor below 5r and returns
// one below 2r without its final subtraction (mul_loose), a difference adds 2r instead of
// testing its sign: a butterfly is 26 instructions of 313 shorter.
#pragma once
#include "fp.cuh"

namespace bg {

// 2r
static constexpr uint32_t kTwoR[8] = {0xe0000002u, 0x87c3eb27u, 0xf372e122u, 0x5067d090u,
                                      0x0302b0bau, 0x70a08b6du, 0xc2634053u, 0x60c89ce5u};

BG_DEV Fr add_raw(const Fr& a, const Fr& b) {
  Fr r;
  raw_add8(r.v, a.v, b.v);
  return r;
}
// a - b + 2r
BG_DEV Fr sub_plus2(const Fr& a, const Fr& b) {
  Fr t;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(t.v[0]), "=r"(t.v[1]), "=r"(t.v[2]), "=r"(t.v[3]), "=r"(t.v[4]), "=r"(t.v[5]), "=r"(t.v[6]), "=r"(t.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "n"(kTwoR[0]), "n"(kTwoR[1]), "n"(kTwoR[2]), "n"(kTwoR[3]), "n"(kTwoR[4]), "n"(kTwoR[5]), "n"(kTwoR[6]),
        "n"(kTwoR[7]));
  asm("sub.cc.u32  %0, %0, %8;\n\t"
      "subc.cc.u32 %1, %1, %9;\n\t"
      "subc.cc.u32 %2, %2, %10;\n\t"
      "subc.cc.u32 %3, %3, %11;\n\t"
      "subc.cc.u32 %4, %4, %12;\n\t"
      "subc.cc.u32 %5, %5, %13;\n\t"
      "subc.cc.u32 %6, %6, %14;\n\t"
      "subc.u32    %7, %7, %15;"
      : "+r"(t.v[0]), "+r"(t.v[1]), "+r"(t.v[2]), "+r"(t.v[3]), "+r"(t.v[4]), "+r"(t.v[5]), "+r"(t.v[6]), "+r"(t.v[7])
      : "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return t;
}
// a below 4r -> below 2r
BG_DEV Fr reduce2(const Fr& a) {
  uint32_t d[8], bw;
  asm("sub.cc.u32  %0, %9,  %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(bw)
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "n"(kTwoR[0]), "n"(kTwoR[1]), "n"(kTwoR[2]), "n"(kTwoR[3]), "n"(kTwoR[4]), "n"(kTwoR[5]), "n"(kTwoR[6]),
        "n"(kTwoR[7]));
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = bw ? a.v[i] : d[i];
  return r;
}
// a below 2r -> below r
BG_DEV Fr reduce1(const Fr& a) {
  Fr r;
  reduce_once<FrParams>(r.v, a.v);
  return r;
}

// any 256-bit word -> below 2r: what a pass reads may be a caller's, at or above the modulus (2^256 <
// 6r).  One comparison for the others: NTT 2^20 201.1 -> 201.6 us, smaller ones level; in the first
// pass alone, by a flag, 202.3.
BG_DEV Fr below2(const Fr& a) {
  constexpr uint32_t top = kTwoR[7];
  return a.v[7] < top ? a : reduce2(reduce2(a));
}

// one butterfly: DIF (x0 + x1, (x0 - x1) w), values below 2r; DIT (x0 + x1 w, x0 - x1 w), values
// below 4r.  `unit`: w = 1, no product.
template <bool DIT>
BG_DEV void butterfly(Fr& x0, Fr& x1, const uint32_t* __restrict__ tw, size_t widx, bool unit) {
  if (DIT) {
    const Fr a = reduce2(x0);
    Fr b;
    if (unit) b = reduce2(x1);
    else b = mul_loose(load_fp<FrParams>(tw + 8 * widx), x1);
    x0 = add_raw(a, b);
    x1 = sub_plus2(a, b);
  } else {
    const Fr d = sub_plus2(x0, x1);
    x0 = reduce2(add_raw(x0, x1));
    if (unit) x1 = reduce2(d);
    else x1 = mul_loose(load_fp<FrParams>(tw + 8 * widx), d);
  }
}

}  // namespace bg
