// The field products, written for the 64-bit multiply-add, and lazy reduction.
//
// What bounds every kernel of the MSM and the NTT is the FMA-heavy pipe, and on it a 32 x 32 ->
// 64-bit multiply-add with carry in and out costs what its high half alone costs.  Measured on
// GB300 (cycles per warp and scheduler, independent chains): mad.lo 2.2, mad.hi 4.45; a product
// as a mad.lo in one carry chain and a mad.hi in another 6.4; the same two instructions next to
// each other on an aligned register pair (mad.lo.cc, madc.hi.cc), which the assembler can issue
// as one 64-bit multiply-add, 4.4.  So products are laid out by limb parity: the products of a
// multiplier with the even limbs of the other factor tile whole register pairs at even
// positions, those with the odd limbs tile pairs one limb higher, and each lands in its own
// accumulator (x at even positions, y one limb up), joined by one addition at the end.
// A Montgomery product at 16 warps per SM, in cycles per warp and scheduler (floor 528: 128
// multiply-adds of 4 and 8 mul.lo of 2): 550 inlined and 600 out of line, against 968 for the
// Karatsuba product and reduction in separate lo and hi chains that it replaced; a square 525
// against 741.
//
// Lazy reduction: when a formula needs a +- b c +- d e, the 16-limb products are combined and
// reduced once; the Fq2 Karatsuba product (three Fq products, two reductions instead of three)
// saves one of every six.  A square computes its 28 off-diagonal limb products once and doubles
// them.  Bounds: every value reduced here is below p R (R = 2^256), so the reduction returns a
// value below 2p that one conditional subtraction brings below p; combinations add 2 p^2 before
// subtracting, which keeps them non-negative and below 4 p^2 < p R (4p < 2^256 for the BN254
// base field).
//
// Each asm block is one carry chain.  The host test tests/device_emul.py executes these chains
// instruction by instruction on the CPU.
#pragma once
// included by fp.cuh (needs Fp, Fq, Fq2 and reduce_once)

namespace bg {

struct Wide {
  uint32_t v[16];
};

// t = a b (512 bits)
BG_DEV void wide_mul(Wide& t, const uint32_t* a, const uint32_t* b);
// t = a^2
BG_DEV void wide_sqr(Wide& t, const uint32_t* a);

// D[0..7] += M (X0 + X1 2^64 + X2 2^128 + X3 2^192), one chain of four 64-bit multiply-adds; K is
// the constraint of the X ("r" registers, "n" constants).  BG_MAC4 has no carry out (the caller
// knows the sum fits), BG_MAC4_TOP adds it to T, BG_MAC4_JOIN first does C += S and takes that
// carry into D[0].
#define BG_MAC4(D, K, X0, X1, X2, X3, M)                                                           \
  asm("mad.lo.cc.u32  %0, %9, %8, %0;\n\t"                                                         \
      "madc.hi.cc.u32 %1, %9, %8, %1;\n\t"                                                         \
      "madc.lo.cc.u32 %2, %10, %8, %2;\n\t"                                                        \
      "madc.hi.cc.u32 %3, %10, %8, %3;\n\t"                                                        \
      "madc.lo.cc.u32 %4, %11, %8, %4;\n\t"                                                        \
      "madc.hi.cc.u32 %5, %11, %8, %5;\n\t"                                                        \
      "madc.lo.cc.u32 %6, %12, %8, %6;\n\t"                                                        \
      "madc.hi.u32    %7, %12, %8, %7;"                                                            \
      : "+r"((D)[0]), "+r"((D)[1]), "+r"((D)[2]), "+r"((D)[3]),                                    \
        "+r"((D)[4]), "+r"((D)[5]), "+r"((D)[6]), "+r"((D)[7])                                     \
      : "r"(M), K(X0), K(X1), K(X2), K(X3))
#define BG_MAC4_TOP(D, T, K, X0, X1, X2, X3, M)                                                    \
  asm("mad.lo.cc.u32  %0, %10, %9, %0;\n\t"                                                        \
      "madc.hi.cc.u32 %1, %10, %9, %1;\n\t"                                                        \
      "madc.lo.cc.u32 %2, %11, %9, %2;\n\t"                                                        \
      "madc.hi.cc.u32 %3, %11, %9, %3;\n\t"                                                        \
      "madc.lo.cc.u32 %4, %12, %9, %4;\n\t"                                                        \
      "madc.hi.cc.u32 %5, %12, %9, %5;\n\t"                                                        \
      "madc.lo.cc.u32 %6, %13, %9, %6;\n\t"                                                        \
      "madc.hi.cc.u32 %7, %13, %9, %7;\n\t"                                                        \
      "addc.u32       %8, %8, 0;"                                                                  \
      : "+r"((D)[0]), "+r"((D)[1]), "+r"((D)[2]), "+r"((D)[3]),                                    \
        "+r"((D)[4]), "+r"((D)[5]), "+r"((D)[6]), "+r"((D)[7]), "+r"(T)                            \
      : "r"(M), K(X0), K(X1), K(X2), K(X3))
#define BG_MAC4_JOIN(D, C, S, K, X0, X1, X2, X3, M)                                                \
  asm("add.cc.u32     %8, %8, %14;\n\t"                                                            \
      "madc.lo.cc.u32 %0, %10, %9, %0;\n\t"                                                        \
      "madc.hi.cc.u32 %1, %10, %9, %1;\n\t"                                                        \
      "madc.lo.cc.u32 %2, %11, %9, %2;\n\t"                                                        \
      "madc.hi.cc.u32 %3, %11, %9, %3;\n\t"                                                        \
      "madc.lo.cc.u32 %4, %12, %9, %4;\n\t"                                                        \
      "madc.hi.cc.u32 %5, %12, %9, %5;\n\t"                                                        \
      "madc.lo.cc.u32 %6, %13, %9, %6;\n\t"                                                        \
      "madc.hi.u32    %7, %13, %9, %7;"                                                            \
      : "+r"((D)[0]), "+r"((D)[1]), "+r"((D)[2]), "+r"((D)[3]),                                    \
        "+r"((D)[4]), "+r"((D)[5]), "+r"((D)[6]), "+r"((D)[7]), "+r"(C)                            \
      : "r"(M), K(X0), K(X1), K(X2), K(X3), "r"(S))

// (hi, lo) = a b
BG_DEV void mul_pair(uint32_t* d, uint32_t a, uint32_t b) {
  const uint64_t t = (uint64_t)a * b;
  d[0] = (uint32_t)t;
  d[1] = (uint32_t)(t >> 32);
}

// t[1..15] += y[0..14]: the odd-position accumulator joined to the even one
BG_DEV void join_odd(uint32_t* t, const uint32_t* y) {
  asm("add.cc.u32 %0, %0, %15;\n\t"
      "addc.cc.u32 %1, %1, %16;\n\t"
      "addc.cc.u32 %2, %2, %17;\n\t"
      "addc.cc.u32 %3, %3, %18;\n\t"
      "addc.cc.u32 %4, %4, %19;\n\t"
      "addc.cc.u32 %5, %5, %20;\n\t"
      "addc.cc.u32 %6, %6, %21;\n\t"
      "addc.cc.u32 %7, %7, %22;\n\t"
      "addc.cc.u32 %8, %8, %23;\n\t"
      "addc.cc.u32 %9, %9, %24;\n\t"
      "addc.cc.u32 %10, %10, %25;\n\t"
      "addc.cc.u32 %11, %11, %26;\n\t"
      "addc.cc.u32 %12, %12, %27;\n\t"
      "addc.cc.u32 %13, %13, %28;\n\t"
      "addc.u32 %14, %14, %29;"
      : "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]), "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12]), "+r"(t[13]), "+r"(t[14]), "+r"(t[15])
      : "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]), "r"(y[8]), "r"(y[9]), "r"(y[10]), "r"(y[11]), "r"(y[12]), "r"(y[13]), "r"(y[14]));
}

// Rows 2k and 2k + 1 (multipliers b[2k], b[2k + 1]) share their windows: x[2k..2k+9] and
// y[2k..2k+8].  A window's top limbs are fresh when its first row gets there, so only the rows
// that come second at a limb have a carry out: x + 8 in row 2k, y + 8 in row 2k + 1.
BG_DEV void wide_mul(Wide& t, const uint32_t* a, const uint32_t* b) {
  uint32_t y[15];
  uint32_t* x = t.v;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    mul_pair(x + 2 * j, a[2 * j], b[0]);
    mul_pair(y + 2 * j, a[2 * j + 1], b[0]);
  }
  x[8] = x[9] = y[8] = 0;
  BG_MAC4(x + 2, "r", a[1], a[3], a[5], a[7], b[1]);
  BG_MAC4_TOP(y, y[8], "r", a[0], a[2], a[4], a[6], b[1]);
  x[10] = x[11] = y[9] = y[10] = 0;
  BG_MAC4_TOP(x + 2, x[10], "r", a[0], a[2], a[4], a[6], b[2]);
  BG_MAC4(y + 2, "r", a[1], a[3], a[5], a[7], b[2]);
  BG_MAC4(x + 4, "r", a[1], a[3], a[5], a[7], b[3]);
  BG_MAC4_TOP(y + 2, y[10], "r", a[0], a[2], a[4], a[6], b[3]);
  x[12] = x[13] = y[11] = y[12] = 0;
  BG_MAC4_TOP(x + 4, x[12], "r", a[0], a[2], a[4], a[6], b[4]);
  BG_MAC4(y + 4, "r", a[1], a[3], a[5], a[7], b[4]);
  BG_MAC4(x + 6, "r", a[1], a[3], a[5], a[7], b[5]);
  BG_MAC4_TOP(y + 4, y[12], "r", a[0], a[2], a[4], a[6], b[5]);
  x[14] = x[15] = y[13] = y[14] = 0;
  BG_MAC4_TOP(x + 6, x[14], "r", a[0], a[2], a[4], a[6], b[6]);
  BG_MAC4(y + 6, "r", a[1], a[3], a[5], a[7], b[6]);
  BG_MAC4(x + 8, "r", a[1], a[3], a[5], a[7], b[7]);
  BG_MAC4_TOP(y + 6, y[14], "r", a[0], a[2], a[4], a[6], b[7]);
  join_odd(x, y);
}

// t = a^2: the off-diagonal products once (a_i a_j with j - i even in x, odd in y), doubled, plus
// the diagonal
BG_DEV void wide_sqr(Wide& t, const uint32_t* a) {
  uint32_t y[15];
  uint32_t* x = t.v;
#pragma unroll
  for (int i = 0; i < 16; i++) x[i] = 0;
#pragma unroll
  for (int i = 0; i < 15; i++) y[i] = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) mul_pair(y + 2 * j, a[2 * j + 1], a[0]);
#pragma unroll
  for (int j = 0; j < 3; j++) mul_pair(x + 2 + 2 * j, a[2 * j + 2], a[0]);
  asm("mad.lo.cc.u32  %0, %8, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %7, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %7, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %7, %5;\n\t"
      "addc.u32       %6, %6, 0;"
      : "+r"(y[2]), "+r"(y[3]), "+r"(y[4]), "+r"(y[5]), "+r"(y[6]), "+r"(y[7]),
        "+r"(y[8])
      : "r"(a[1]), "r"(a[2]), "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %8, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %7, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %7, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %7, %5;\n\t"
      "addc.u32       %6, %6, 0;"
      : "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "+r"(x[8]), "+r"(x[9]),
        "+r"(x[10])
      : "r"(a[1]), "r"(a[3]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %8, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %7, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %7, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %7, %5;\n\t"
      "addc.u32       %6, %6, 0;"
      : "+r"(y[4]), "+r"(y[5]), "+r"(y[6]), "+r"(y[7]), "+r"(y[8]), "+r"(y[9]),
        "+r"(y[10])
      : "r"(a[2]), "r"(a[3]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %6, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %5, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %5, %3;\n\t"
      "addc.u32       %4, %4, 0;"
      : "+r"(x[6]), "+r"(x[7]), "+r"(x[8]), "+r"(x[9]), "+r"(x[10])
      : "r"(a[2]), "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %6, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %5, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %5, %3;\n\t"
      "addc.u32       %4, %4, 0;"
      : "+r"(y[6]), "+r"(y[7]), "+r"(y[8]), "+r"(y[9]), "+r"(y[10])
      : "r"(a[3]), "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %6, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %5, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %5, %3;\n\t"
      "addc.u32       %4, %4, 0;"
      : "+r"(x[8]), "+r"(x[9]), "+r"(x[10]), "+r"(x[11]), "+r"(x[12])
      : "r"(a[3]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %6, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %5, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %5, %3;\n\t"
      "addc.u32       %4, %4, 0;"
      : "+r"(y[8]), "+r"(y[9]), "+r"(y[10]), "+r"(y[11]), "+r"(y[12])
      : "r"(a[4]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %4, %3, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %3, %1;\n\t"
      "addc.u32       %2, %2, 0;"
      : "+r"(x[10]), "+r"(x[11]), "+r"(x[12])
      : "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %4, %3, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %3, %1;\n\t"
      "addc.u32       %2, %2, 0;"
      : "+r"(y[10]), "+r"(y[11]), "+r"(y[12])
      : "r"(a[5]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %4, %3, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %3, %1;\n\t"
      "addc.u32       %2, %2, 0;"
      : "+r"(x[12]), "+r"(x[13]), "+r"(x[14])
      : "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %4, %3, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %3, %1;\n\t"
      "addc.u32       %2, %2, 0;"
      : "+r"(y[12]), "+r"(y[13]), "+r"(y[14])
      : "r"(a[6]), "r"(a[7]));
  join_odd(x, y);
  asm("add.cc.u32     %0, %0, %0;\n\t"
      "addc.cc.u32    %1, %1, %1;\n\t"
      "addc.cc.u32    %2, %2, %2;\n\t"
      "addc.cc.u32    %3, %3, %3;\n\t"
      "addc.cc.u32    %4, %4, %4;\n\t"
      "addc.cc.u32    %5, %5, %5;\n\t"
      "addc.cc.u32    %6, %6, %6;\n\t"
      "addc.cc.u32    %7, %7, %7;\n\t"
      "addc.cc.u32    %8, %8, %8;\n\t"
      "addc.cc.u32    %9, %9, %9;\n\t"
      "addc.cc.u32    %10, %10, %10;\n\t"
      "addc.cc.u32    %11, %11, %11;\n\t"
      "addc.cc.u32    %12, %12, %12;\n\t"
      "addc.cc.u32    %13, %13, %13;\n\t"
      "addc.cc.u32    %14, %14, %14;\n\t"
      "addc.u32       %15, %15, %15;"
      : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]),
        "+r"(x[6]), "+r"(x[7]), "+r"(x[8]), "+r"(x[9]), "+r"(x[10]), "+r"(x[11]),
        "+r"(x[12]), "+r"(x[13]), "+r"(x[14]), "+r"(x[15])
      :);
  asm("mad.lo.cc.u32  %0, %16, %16, %0;\n\t"
      "madc.hi.cc.u32 %1, %16, %16, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %17, %2;\n\t"
      "madc.hi.cc.u32 %3, %17, %17, %3;\n\t"
      "madc.lo.cc.u32 %4, %18, %18, %4;\n\t"
      "madc.hi.cc.u32 %5, %18, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %19, %19, %6;\n\t"
      "madc.hi.cc.u32 %7, %19, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %20, %20, %8;\n\t"
      "madc.hi.cc.u32 %9, %20, %20, %9;\n\t"
      "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
      "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
      "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
      "madc.hi.u32    %15, %23, %23, %15;"
      : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]),
        "+r"(x[6]), "+r"(x[7]), "+r"(x[8]), "+r"(x[9]), "+r"(x[10]), "+r"(x[11]),
        "+r"(x[12]), "+r"(x[13]), "+r"(x[14]), "+r"(x[15])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]),
        "r"(a[6]), "r"(a[7]));
}

// One row of Montgomery's reduction on a nine-limb running value split by limb parity: e holds
// limbs 0..7, o limbs 1..8.  Adds m p with m = -e[0] / p mod 2^32, which clears limb 0.  The
// running value stays below 2^288 (callers' bounds), so o has no carry out and e's goes to limb 8.
template <class P>
BG_DEV void redc_row(uint32_t* e, uint32_t* o) {
  const uint32_t m = e[0] * P::N0;
  BG_MAC4(o, "n", P::P1, P::P3, P::P5, P::P7, m);
  BG_MAC4_TOP(e, o[7], "n", P::P0, P::P2, P::P4, P::P6, m);
}
// Dropping limb 0 swaps the roles: o's limbs are now 0..7, e's limbs 2..7 move to 1..6 (in place,
// register pairs keep their alignment), and e's limb 1 is the new limb 0's second part, returned
// for the caller to join.
BG_DEV uint32_t shift_row(uint32_t* e) {
  const uint32_t c = e[1];
#pragma unroll
  for (int i = 0; i < 6; i++) e[i] = e[i + 2];
  e[6] = e[7] = 0;
  return c;
}
// the running value after the last row (limb 0 of e is zero): r = limbs 1..8
BG_DEV void join_rows(uint32_t* r, const uint32_t* e, const uint32_t* o) {
  asm("add.cc.u32     %0, %8, %15;\n\t"
      "addc.cc.u32    %1, %9, %16;\n\t"
      "addc.cc.u32    %2, %10, %17;\n\t"
      "addc.cc.u32    %3, %11, %18;\n\t"
      "addc.cc.u32    %4, %12, %19;\n\t"
      "addc.cc.u32    %5, %13, %20;\n\t"
      "addc.cc.u32    %6, %14, %21;\n\t"
      "addc.u32       %7, %22, 0;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(o[0]), "r"(o[1]),
        "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]));
}

// Row b of a Montgomery product: the running value (o its even part after the last row) drops its
// cleared limb, takes a b and is reduced by a row.  For a < p it is below 2p before and after
// ((2p + 2^32 a + 2^32 p) / 2^32), whatever the limb b, so below 2^288 in between.
template <class P>
BG_DEV void mul_row(uint32_t* e, uint32_t* o, const uint32_t* a, uint32_t b) {
  const uint32_t c = shift_row(o);
  BG_MAC4_JOIN(o, e[0], c, "r", a[1], a[3], a[5], a[7], b);
  BG_MAC4_TOP(e, o[7], "r", a[0], a[2], a[4], a[6], b);
  redc_row<P>(e, o);
}

// a b R^-1 mod p, below p + a b / R, for a < p and any 256-bit b (below 2p for b < 5p): product and
// reduction interleaved row by row (the two accumulators take 16 registers instead of a 16-limb
// product's 31)
template <class P>
BG_DEV Fp<P> mul_loose(const Fp<P>& a, const Fp<P>& b) {
  uint32_t u[8], w[8];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    mul_pair(u + 2 * j, a.v[2 * j], b.v[0]);
    mul_pair(w + 2 * j, a.v[2 * j + 1], b.v[0]);
  }
  redc_row<P>(u, w);
  mul_row<P>(w, u, a.v, b.v[1]);
  mul_row<P>(u, w, a.v, b.v[2]);
  mul_row<P>(w, u, a.v, b.v[3]);
  mul_row<P>(u, w, a.v, b.v[4]);
  mul_row<P>(w, u, a.v, b.v[5]);
  mul_row<P>(u, w, a.v, b.v[6]);
  mul_row<P>(w, u, a.v, b.v[7]);
  Fp<P> r;
  join_rows(r.v, w, u);
  return r;
}
// the same, fully reduced
template <class P>
BG_DEV Fp<P> mul(const Fp<P>& a, const Fp<P>& b) {
  const Fp<P> t = mul_loose(a, b);
  Fp<P> r;
  reduce_once<P>(r.v, t.v);
  return r;
}

// Row of a reduction alone: as mul_row without the product
template <class P>
BG_DEV void redc_next(uint32_t* e, uint32_t* o) {
  const uint32_t c = shift_row(o);
  const uint32_t m = (e[0] + c) * P::N0;
  BG_MAC4_JOIN(o, e[0], c, "n", P::P1, P::P3, P::P5, P::P7, m);
  BG_MAC4_TOP(e, o[7], "n", P::P0, P::P2, P::P4, P::P6, m);
}

// (t + U p) / R for t < R, the U that makes it whole: at most p
template <class P>
BG_DEV void redc_low(uint32_t* r, const uint32_t* t) {
  uint32_t u[8], w[8];
#pragma unroll
  for (int i = 0; i < 8; i++) u[i] = t[i];
  const uint32_t m = u[0] * P::N0;
  mul_pair(w, P::P1, m);
  mul_pair(w + 2, P::P3, m);
  mul_pair(w + 4, P::P5, m);
  mul_pair(w + 6, P::P7, m);
  BG_MAC4_TOP(u, w[7], "n", P::P0, P::P2, P::P4, P::P6, m);
  redc_next<P>(w, u);
  redc_next<P>(u, w);
  redc_next<P>(w, u);
  redc_next<P>(u, w);
  redc_next<P>(w, u);
  redc_next<P>(u, w);
  redc_next<P>(w, u);
  join_rows(r, w, u);
}

// t += u (the caller keeps the sum below 2^512)
BG_DEV void wide_add(Wide& t, const Wide& u) {
  asm("add.cc.u32     %0, %0, %16;\n\t"
      "addc.cc.u32    %1, %1, %17;\n\t"
      "addc.cc.u32    %2, %2, %18;\n\t"
      "addc.cc.u32    %3, %3, %19;\n\t"
      "addc.cc.u32    %4, %4, %20;\n\t"
      "addc.cc.u32    %5, %5, %21;\n\t"
      "addc.cc.u32    %6, %6, %22;\n\t"
      "addc.cc.u32    %7, %7, %23;\n\t"
      "addc.cc.u32    %8, %8, %24;\n\t"
      "addc.cc.u32    %9, %9, %25;\n\t"
      "addc.cc.u32    %10, %10, %26;\n\t"
      "addc.cc.u32    %11, %11, %27;\n\t"
      "addc.cc.u32    %12, %12, %28;\n\t"
      "addc.cc.u32    %13, %13, %29;\n\t"
      "addc.cc.u32    %14, %14, %30;\n\t"
      "addc.u32       %15, %15, %31;"
      : "+r"(t.v[0]), "+r"(t.v[1]), "+r"(t.v[2]), "+r"(t.v[3]), "+r"(t.v[4]), "+r"(t.v[5]), "+r"(t.v[6]), "+r"(t.v[7]), "+r"(t.v[8]), "+r"(t.v[9]), "+r"(t.v[10]), "+r"(t.v[11]), "+r"(t.v[12]), "+r"(t.v[13]), "+r"(t.v[14]), "+r"(t.v[15])
      : "r"(u.v[0]), "r"(u.v[1]), "r"(u.v[2]), "r"(u.v[3]), "r"(u.v[4]), "r"(u.v[5]), "r"(u.v[6]), "r"(u.v[7]), "r"(u.v[8]), "r"(u.v[9]), "r"(u.v[10]), "r"(u.v[11]), "r"(u.v[12]), "r"(u.v[13]), "r"(u.v[14]), "r"(u.v[15]));
}

// t -= u (the caller keeps t >= u)
BG_DEV void wide_sub(Wide& t, const Wide& u) {
  asm("sub.cc.u32     %0, %0, %16;\n\t"
      "subc.cc.u32    %1, %1, %17;\n\t"
      "subc.cc.u32    %2, %2, %18;\n\t"
      "subc.cc.u32    %3, %3, %19;\n\t"
      "subc.cc.u32    %4, %4, %20;\n\t"
      "subc.cc.u32    %5, %5, %21;\n\t"
      "subc.cc.u32    %6, %6, %22;\n\t"
      "subc.cc.u32    %7, %7, %23;\n\t"
      "subc.cc.u32    %8, %8, %24;\n\t"
      "subc.cc.u32    %9, %9, %25;\n\t"
      "subc.cc.u32    %10, %10, %26;\n\t"
      "subc.cc.u32    %11, %11, %27;\n\t"
      "subc.cc.u32    %12, %12, %28;\n\t"
      "subc.cc.u32    %13, %13, %29;\n\t"
      "subc.cc.u32    %14, %14, %30;\n\t"
      "subc.u32       %15, %15, %31;"
      : "+r"(t.v[0]), "+r"(t.v[1]), "+r"(t.v[2]), "+r"(t.v[3]), "+r"(t.v[4]), "+r"(t.v[5]), "+r"(t.v[6]), "+r"(t.v[7]), "+r"(t.v[8]), "+r"(t.v[9]), "+r"(t.v[10]), "+r"(t.v[11]), "+r"(t.v[12]), "+r"(t.v[13]), "+r"(t.v[14]), "+r"(t.v[15])
      : "r"(u.v[0]), "r"(u.v[1]), "r"(u.v[2]), "r"(u.v[3]), "r"(u.v[4]), "r"(u.v[5]), "r"(u.v[6]), "r"(u.v[7]), "r"(u.v[8]), "r"(u.v[9]), "r"(u.v[10]), "r"(u.v[11]), "r"(u.v[12]), "r"(u.v[13]), "r"(u.v[14]), "r"(u.v[15]));
}

// t += 2 p^2 (Fq)
BG_DEV void wide_add_2p2(Wide& t) {
  asm("add.cc.u32     %0, %0, %16;\n\t"
      "addc.cc.u32    %1, %1, %17;\n\t"
      "addc.cc.u32    %2, %2, %18;\n\t"
      "addc.cc.u32    %3, %3, %19;\n\t"
      "addc.cc.u32    %4, %4, %20;\n\t"
      "addc.cc.u32    %5, %5, %21;\n\t"
      "addc.cc.u32    %6, %6, %22;\n\t"
      "addc.cc.u32    %7, %7, %23;\n\t"
      "addc.cc.u32    %8, %8, %24;\n\t"
      "addc.cc.u32    %9, %9, %25;\n\t"
      "addc.cc.u32    %10, %10, %26;\n\t"
      "addc.cc.u32    %11, %11, %27;\n\t"
      "addc.cc.u32    %12, %12, %28;\n\t"
      "addc.cc.u32    %13, %13, %29;\n\t"
      "addc.cc.u32    %14, %14, %30;\n\t"
      "addc.u32       %15, %15, %31;"
      : "+r"(t.v[0]), "+r"(t.v[1]), "+r"(t.v[2]), "+r"(t.v[3]), "+r"(t.v[4]), "+r"(t.v[5]), "+r"(t.v[6]), "+r"(t.v[7]), "+r"(t.v[8]), "+r"(t.v[9]), "+r"(t.v[10]), "+r"(t.v[11]), "+r"(t.v[12]), "+r"(t.v[13]), "+r"(t.v[14]), "+r"(t.v[15])
      : "n"(0x4ebad362u), "n"(0x76a8b144u), "n"(0x13d58202u), "n"(0x4c040e5au), "n"(0xdb2d95b9u), "n"(0x94a03138u), "n"(0xf4248590u), "n"(0x08d13d2au), "n"(0x698d671au), "n"(0x4ddbf4b8u), "n"(0x2c6eac0cu), "n"(0x60170aa2u), "n"(0x0691a439u), "n"(0xb334def8u), "n"(0xec797f38u), "n"(0x124b8970u));
}

// r = a + b as integers (a, b < p: the sum is below 2^255)
BG_DEV void raw_add8(uint32_t* r, const uint32_t* a, const uint32_t* b) {
  asm("add.cc.u32     %0, %8, %16;\n\t"
      "addc.cc.u32    %1, %9, %17;\n\t"
      "addc.cc.u32    %2, %10, %18;\n\t"
      "addc.cc.u32    %3, %11, %19;\n\t"
      "addc.cc.u32    %4, %12, %20;\n\t"
      "addc.cc.u32    %5, %13, %21;\n\t"
      "addc.cc.u32    %6, %14, %22;\n\t"
      "addc.u32       %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

// Montgomery reduction of t < p R: t R^-1 mod p.  The low half is reduced alone (at most p) and
// the high half (below p) added.
template <class P>
BG_DEV Fp<P> redc(const Wide& t) {
  uint32_t u[8];
  redc_low<P>(u, t.v);
  raw_add8(u, u, t.v + 8);
  Fp<P> r;
  reduce_once<P>(r.v, u);
  return r;
}

// x * 2^-256: Montgomery -> canonical
template <class P>
BG_DEV Fp<P> from_mont(const Fp<P>& a) {
  uint32_t u[8];
  redc_low<P>(u, a.v);
  Fp<P> r;
  reduce_once<P>(r.v, u);
  return r;
}

// a^2 with the squaring product
template <class P>
BG_DEV Fp<P> sqr_wide(const Fp<P>& a) {
  Wide t;
  wide_sqr(t, a.v);
  return redc<P>(t);
}

// a b - c d with one reduction (the difference of the products offset by 2 p^2)
BG_DEV Fq mul_sub_mul(const Fq& a, const Fq& b, const Fq& c, const Fq& d) {
  Wide t, u;
  wide_mul(t, a.v, b.v);
  wide_add_2p2(t);
  wide_mul(u, c.v, d.v);
  wide_sub(t, u);
  return redc<FqParams>(t);
}

// Out-of-line bodies for the curve formulas: one each for an Fq product, square and a b - c d,
// and an Fq2 product and a b - c d with the products and reductions inside inlined, so a formula
// of a dozen products stays small in the instruction cache.  Against bodies made of calls to a
// shared 512-bit product and a shared reduction: G2 MSM 2^18's accumulation 2.15 -> 1.89 ms and
// reduction 1.38 -> 1.17 ms, G1's (2^20) 0.85 -> 0.75 and 0.48 -> 0.44 ms, SquareChain(2^18)
// 7.58 -> 6.80 ms; an Fq2 body calling a shared reduction or a shared product alone measured
// 1.95-2.00 ms, an Fq2 addition with everything inlined 2.12 ms (instruction fetch).
static __device__ __noinline__ Fq mul_ool(Fq a, Fq b) { return mul(a, b); }
static __device__ __noinline__ Fq sqr_ool(Fq a) { return sqr_wide(a); }
static __device__ __noinline__ Fq mul_sub_mul_ool(Fq a, Fq b, Fq c, Fq d) { return mul_sub_mul(a, b, c, d); }

// Fq2 product (Karatsuba) with two reductions:
//   c0 = a0 b0 - a1 b1,  c1 = (a0 + a1)(b0 + b1) - a0 b0 - a1 b1 = a0 b1 + a1 b0
// with the sums a0 + a1, b0 + b1 kept unreduced (below 2p) so that c1 is exact
static __device__ __noinline__ Fq2 fq2_mul_ool(Fq2 a, Fq2 b) {
  Wide t0, t1, t2;
  wide_mul(t0, a.c0.v, b.c0.v);
  wide_mul(t1, a.c1.v, b.c1.v);
  Fq sa, sb;
  raw_add8(sa.v, a.c0.v, a.c1.v);
  raw_add8(sb.v, b.c0.v, b.c1.v);
  wide_mul(t2, sa.v, sb.v);
  wide_sub(t2, t0);
  wide_sub(t2, t1);
  wide_add_2p2(t0);
  wide_sub(t0, t1);
  return {redc<FqParams>(t0), redc<FqParams>(t2)};
}

// a b - c d in Fq2 with two reductions (both components offset by 2 p^2, below 4 p^2)
static __device__ __noinline__ Fq2 fq2_mul_sub_mul_ool(Fq2 a, Fq2 b, Fq2 c, Fq2 d) {
  Fq s0, s1;
  // a b: re = a0 b0 - a1 b1 + 2p^2, im = (a0 + a1)(b0 + b1) - a0 b0 - a1 b1 + 2p^2
  Wide re, im, w0, w1;
  wide_mul(re, a.c0.v, b.c0.v);
  wide_mul(w1, a.c1.v, b.c1.v);
  raw_add8(s0.v, a.c0.v, a.c1.v);
  raw_add8(s1.v, b.c0.v, b.c1.v);
  wide_mul(im, s0.v, s1.v);
  wide_sub(im, re);
  wide_sub(im, w1);
  wide_add_2p2(im);
  wide_add_2p2(re);
  wide_sub(re, w1);
  // - c d: re += c1 d1 - c0 d0, im += c0 d0 + c1 d1 - (c0 + c1)(d0 + d1)
  wide_mul(w0, c.c0.v, d.c0.v);
  wide_mul(w1, c.c1.v, d.c1.v);
  wide_add(re, w1);
  wide_sub(re, w0);
  wide_add(im, w0);
  wide_add(im, w1);
  raw_add8(s0.v, c.c0.v, c.c1.v);
  raw_add8(s1.v, d.c0.v, d.c1.v);
  wide_mul(w0, s0.v, s1.v);
  wide_sub(im, w0);
  return {redc<FqParams>(re), redc<FqParams>(im)};
}

#undef BG_MAC4
#undef BG_MAC4_TOP
#undef BG_MAC4_JOIN

}  // namespace bg
