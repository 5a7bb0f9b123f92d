// Radix-2 NTTs over BN254 Fr and the Groth16 QAP quotient h(x).
//
// Reference semantics: Ntt.fft / ifft / coset_fft (bend2/src/ntt.bend:431-438) over
// arkworks' Radix2EvaluationDomain (generator w = root^(2^(28-L)), ntt.bend:73-74), and
// Ntt.qap_h (ntt.bend:446-459) = ark-groth16 LibsnarkReduction:
//   h = coset_iNTT((coset_NTT(iNTT a) * coset_NTT(iNTT b) - coset_NTT(iNTT c)) / (g^d - 1)),
// with g = 5 (bend2/gen/ref_qap.py:59-72).  The reference runs log2(d) Stockham stages on a
// chunk tree with running-product twiddles (ntt.bend:1-18).
//
// Here a transform is a few passes over HBM/L2; each pass loads a tile of up to 1024
// elements into shared memory, runs up
// to 10 radix-2 stages there with twiddles from a resident table, and writes the tile back.
// 1024-element tiles (32 KiB) give a 2^19 transform 512 CTAs instead of 256 with 64 KiB tiles.
//   DIF (Gentleman-Sande): natural order in -> bit-reversed out (used for inverse transforms)
//   DIT (Cooley-Tukey):    bit-reversed in -> natural order out (forward transforms)
// so iNTT followed by a coset NTT needs no permutation: the coset factor g^j of coefficient j
// is applied in bit-reversed position, fused with n^-1 into the last DIF pass.  A transform that has
// to end in natural order writes its last pass to the bit-reversed places of another buffer.
#include <mutex>

#include "common.cuh"
#include "fp.cuh"
#include "host_ff.hpp"
#include "ntt.h"
#include "ntt_butterfly.cuh"

namespace bg {

constexpr int kNttThreads = 256;
constexpr int kNttTile = 1024;   // elements per CTA tile (32 KiB of shared memory)
constexpr int kContigMax = 10;   // stages in one pass, contiguous or strided (a 1024-element tile)

enum ScaleMode { SC_NONE = 0, SC_NATURAL = 1, SC_BITREV = 2, SC_CONST = 3 };

struct ScaleTab {
  const uint32_t* lo = nullptr;  // T(i) = lo[i & (2^bits-1)] * hi[i >> bits]
  const uint32_t* hi = nullptr;
  int bits = 0;
};

BG_DEV Fr scale_factor(int mode, size_t j, int L, const ScaleTab& t) {
  if (mode == SC_CONST) return load_fp<FrParams>(t.hi);
  size_t i = j;
  if (mode == SC_BITREV) i = __brevll((unsigned long long)j) >> (64 - L);
  const Fr a = load_fp<FrParams>(t.lo + 8 * (i & ((size_t(1) << t.bits) - 1)));
  const Fr b = load_fp<FrParams>(t.hi + 8 * (i >> t.bits));
  return mul(a, b);
}

// The tile in shared memory: element e's low and high 16 bytes at uint4 slot e of two arrays
// of E slots, so an element moves in two 128-bit accesses.
BG_DEV void tile_store(uint32_t* sm, int E, int e, const Fr& x) {
  uint4* lo = reinterpret_cast<uint4*>(sm);
  lo[e] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  lo[E + e] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}
BG_DEV Fr tile_load(const uint32_t* sm, int E, int e) {
  const uint4* lo = reinterpret_cast<const uint4*>(sm);
  const uint4 a = lo[e], b = lo[E + e];
  Fr x;
  x.v[0] = a.x; x.v[1] = a.y; x.v[2] = a.z; x.v[3] = a.w;
  x.v[4] = b.x; x.v[5] = b.y; x.v[6] = b.z; x.v[7] = b.w;
  return x;
}

// Up to three vectors transformed by one launch (the QAP's a, b and c), blockIdx.y picks one.
struct NttVecs {
  const uint32_t* src[3];
  uint32_t* dst[3];
};
// what a pass does on load besides its scaling: nothing, or the QAP's quotient on the coset,
// (src[0] src[1] - src[2]) zinv
enum LoadMode { LD_PLAIN = 0, LD_QUOTIENT = 1 };

// One pass: stages [s0, s0 + k) of a size-2^L transform.  A CTA owns G independent groups of
// 2^k elements; group element t of group (hi, lo) sits at hi*2^(s0+k) + t*2^s0 + lo, and goes back
// there or (rev) to the bit-reversed place.  Two stages at a time on four elements in registers
// (R4), so a tile crosses shared memory and its barrier once per two stages; the latency-bound
// passes of small domains take one stage at a time, with twice the threads.
//
// Bound by the FMA-heavy pipe (10 M products of a 2^20 transform: 138 us) and, a third of the time,
// by the latency of the twiddles (32 bytes from L2 per product of the strided pass).  Three
// 256-thread CTAs per SM (80 registers): 2^20 forward 200 us, against 216 with two (102 registers)
// and 208 with four (64, some spills); one stage at a time with full reductions, and the bit
// reversal as a pass of its own and a copy back, took 239.  The QAP takes the four-CTA form (OCC): a
// proof's accumulations take an SM's slots first, and smaller CTAs fit beside them (SquareChain(2^18)
// 6.72 -> 6.67 ms).
template <bool DIT, bool R4, int NT, int OCC>
__global__ void __launch_bounds__(NT, OCC) k_ntt_pass(NttVecs vecs, const uint32_t* __restrict__ tw, int L, int s0, int k,
                                                 int G, int pre_mode, int post_mode, ScaleTab sc, int load_mode,
                                                 const uint32_t* __restrict__ zinv, int rev) {
  extern __shared__ __align__(16) uint32_t sm[];
  const uint32_t* src = blockIdx.y == 0 ? vecs.src[0] : blockIdx.y == 1 ? vecs.src[1] : vecs.src[2];
  uint32_t* dst = blockIdx.y == 0 ? vecs.dst[0] : blockIdx.y == 1 ? vecs.dst[1] : vecs.dst[2];
  const int E = G << k;
  const uint32_t kmask = (1u << k) - 1u;
  const size_t lomask = (size_t(1) << s0) - 1;
  const size_t gid0 = (size_t)blockIdx.x * G;
  auto place = [&](int idx, int& e) -> size_t {
    int grp, t;
    if (s0 == 0) {
      grp = idx >> k;
      t = idx & kmask;
    } else {
      grp = idx % G;
      t = idx / G;
    }
    e = (grp << k) | t;
    const size_t gid = gid0 + grp;
    return (s0 == 0) ? ((gid << k) | (size_t)t)
                     : (((gid >> s0) << (s0 + k)) | ((size_t)t << s0) | (gid & lomask));
  };

  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    int e;
    const size_t j = place(idx, e);
    Fr x = load_fp<FrParams>(src + 8 * j);
    if (load_mode == LD_QUOTIENT) {
      const Fr y = load_fp<FrParams>(vecs.src[1] + 8 * j), z = load_fp<FrParams>(vecs.src[2] + 8 * j);
      x = mul(load_fp<FrParams>(zinv), sub(mul(x, y), z));
    }
    if (pre_mode != SC_NONE) x = mul(scale_factor(pre_mode, j, L, sc), x);
    else if (load_mode == LD_PLAIN) x = below2(x);
    tile_store(sm, E, e, x);
  }
  __syncthreads();

  // twiddle of the pair at stage r whose lower r bits are q, in group `lo`: w^(((q << s0) + lo) << (L - s - 1))
  if constexpr (R4) {
    const int quads = E >> 2;
    int done = 0;
    if (k & 1) {  // an odd stage by itself: the lowest for DIT, the highest for DIF
      const int r = DIT ? 0 : k - 1;
      const uint32_t rmask = (1u << r) - 1u;
      for (int b = threadIdx.x; b < (E >> 1); b += blockDim.x) {
        const int grp = b >> (k - 1);
        const uint32_t q = (uint32_t)b & ((1u << (k - 1)) - 1u);
        const int e1 = (grp << k) | (int)(((q >> r) << (r + 1)) | (q & rmask)), e2 = e1 | (1 << r);
        const size_t lo = (s0 == 0) ? 0 : ((gid0 + grp) & lomask);
        const size_t widx = ((((size_t)(q & rmask)) << s0) + lo) << (L - s0 - r - 1);
        Fr x0 = tile_load(sm, E, e1), x1 = tile_load(sm, E, e2);
        butterfly<DIT>(x0, x1, tw, widx, s0 == 0 && r == 0);
        tile_store(sm, E, e1, x0);
        tile_store(sm, E, e2, x1);
      }
      __syncthreads();
      done = 1;
    }
    for (; done < k; done += 2) {
      const int r = DIT ? done : k - 2 - done;  // the lower of the two stages
      const uint32_t rmask = (1u << r) - 1u;
      const bool unit = s0 == 0 && r == 0;
      for (int b = threadIdx.x; b < quads; b += blockDim.x) {
        const int grp = b >> (k - 2);
        const uint32_t q = (uint32_t)b & ((1u << (k - 2)) - 1u);
        const int e = (grp << k) | (int)(((q >> r) << (r + 2)) | (q & rmask));
        const int st = 1 << r;
        const size_t lo = (s0 == 0) ? 0 : ((gid0 + grp) & lomask);
        // lower stage: both pairs at w^(2 h); upper stage: w^h and w^(h + 2^(L-2))
        const size_t h = ((((size_t)(q & rmask)) << s0) + lo) << (L - s0 - r - 2), quarter = size_t(1) << (L - 2);
        Fr x0 = tile_load(sm, E, e), x1 = tile_load(sm, E, e + st), x2 = tile_load(sm, E, e + 2 * st),
           x3 = tile_load(sm, E, e + 3 * st);
        if (DIT) {
          butterfly<DIT>(x0, x1, tw, 2 * h, unit);
          butterfly<DIT>(x2, x3, tw, 2 * h, unit);
          butterfly<DIT>(x0, x2, tw, h, unit);
          butterfly<DIT>(x1, x3, tw, h + quarter, false);
        } else {
          butterfly<DIT>(x0, x2, tw, h, unit);
          butterfly<DIT>(x1, x3, tw, h + quarter, false);
          butterfly<DIT>(x0, x1, tw, 2 * h, unit);
          butterfly<DIT>(x2, x3, tw, 2 * h, unit);
        }
        tile_store(sm, E, e, x0);
        tile_store(sm, E, e + st, x1);
        tile_store(sm, E, e + 2 * st, x2);
        tile_store(sm, E, e + 3 * st, x3);
      }
      __syncthreads();
    }
  } else {
    const int half = E >> 1;
    for (int rr = 0; rr < k; rr++) {
      const int r = DIT ? rr : (k - 1 - rr);
      const uint32_t rmask = (1u << r) - 1u;
      for (int b = threadIdx.x; b < half; b += blockDim.x) {
        const int grp = b >> (k - 1);
        const uint32_t q = (uint32_t)b & ((1u << (k - 1)) - 1u);
        const int e1 = (grp << k) | (int)(((q >> r) << (r + 1)) | (q & rmask)), e2 = e1 | (1 << r);
        const size_t lo = (s0 == 0) ? 0 : ((gid0 + grp) & lomask);
        const size_t widx = ((((size_t)(q & rmask)) << s0) + lo) << (L - s0 - r - 1);
        Fr x0 = tile_load(sm, E, e1), x1 = tile_load(sm, E, e2);
        butterfly<DIT>(x0, x1, tw, widx, s0 == 0 && r == 0);
        tile_store(sm, E, e1, x0);
        tile_store(sm, E, e2, x1);
      }
      __syncthreads();
    }
  }

  for (int idx = threadIdx.x; idx < E; idx += blockDim.x) {
    int e;
    const size_t j = place(idx, e);
    Fr x = tile_load(sm, E, e);
    if (post_mode != SC_NONE) x = mul(scale_factor(post_mode, j, L, sc), x);
    else x = reduce1(DIT ? reduce2(x) : x);
    store_fp(dst + 8 * (rev && L ? (size_t)(__brevll((unsigned long long)j) >> (64 - L)) : j), x);
  }
}

// out[i] = lo[i & (2^bits - 1)] * hi[i >> bits]
__global__ void k_table_expand(uint32_t* __restrict__ out, const uint32_t* __restrict__ lo,
                               const uint32_t* __restrict__ hi, int bits, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Fr a = load_fp<FrParams>(lo + 8 * (i & ((size_t(1) << bits) - 1)));
  const Fr b = load_fp<FrParams>(hi + 8 * (i >> bits));
  store_fp(out + 8 * i, mul(a, b));
}

// ---------------------------------------------------------------- host side
using bgh::Fe;
using bgh::FR;

// 2-adic root of unity of order 2^28 (canonical; bend2/gen/gen_ntt.py:11)
static const Fe kRootCanonical{{0x9bd61b6e725b19f0ull, 0x402d111e41112ed4ull, 0x00e0a7eb8ef62abcull,
                                0x2a3c09f0a58a7e85ull}};

static Fe fr_mont_u64(uint64_t x) { return bgh::fe_to_mont(FR, bgh::fe_raw(x)); }

static Fe omega_mont(int L) {
  Fe w = bgh::fe_to_mont(FR, kRootCanonical);
  for (int i = L; i < 28; i++) w = bgh::fe_sqr(FR, w);
  return w;
}

static void upload_fes(Ctx& ctx, uint32_t* d, const std::vector<Fe>& v) {
  std::vector<uint32_t> words(v.size() * 8);
  for (size_t i = 0; i < v.size(); i++) bgh::fe_to_words32(words.data() + 8 * i, v[i]);
  BG_CUDA(cudaMemcpyAsync(d, words.data(), words.size() * 4, cudaMemcpyHostToDevice, ctx.stream));
  ctx.h2d_bytes += words.size() * 4;
  BG_CUDA(cudaStreamSynchronize(ctx.stream));
}

static std::vector<Fe> powers(const Fe& base, size_t n, const Fe& first) {
  std::vector<Fe> out(n);
  Fe x = first;
  for (size_t i = 0; i < n; i++) {
    out[i] = x;
    x = bgh::fe_mul(FR, x, base);
  }
  return out;
}

size_t ntt_table_bytes(int L) {
  const size_t half = L > 0 ? size_t(1) << (L - 1) : 1, lo = size_t(1) << ((L + 1) / 2), hi = (size_t(1) << L) / lo;
  const size_t nlo = std::min(half, size_t(1) << 10), nhi = (half + nlo - 1) / nlo;
  return 32 * (2 * half + nlo + nhi + 2 * lo + 4 * hi + 2);
}

NttTables& ntt_tables(Ctx& ctx, int L) {
  NttTables& slot = ctx.ntt_tabs[L];
  if (slot.ready) return slot;
  const size_t n = size_t(1) << L;
  const size_t half = n > 1 ? n / 2 : 1;
  const std::string tag = "ntt" + std::to_string(L);
  slot.tw_fwd = ctx.ws.get_t<uint32_t>(tag + ".tw_fwd", half * 8);
  slot.tw_inv = ctx.ws.get_t<uint32_t>(tag + ".tw_inv", half * 8);
  const Fe one = bgh::fe_one(FR);
  const Fe w = omega_mont(L);
  const Fe winv = bgh::fe_inv(FR, w);
  // twiddles: two-level expansion lo (2^10) x hi
  const int tb = 10;
  const size_t nlo = std::min(half, size_t(1) << tb);
  const size_t nhi = (half + nlo - 1) / nlo;
  uint32_t* tmp_lo = ctx.ws.get_t<uint32_t>(tag + ".tmp_lo", nlo * 8);
  uint32_t* tmp_hi = ctx.ws.get_t<uint32_t>(tag + ".tmp_hi", nhi * 8);
  const int lo_bits = (nlo == 1) ? 0 : tb;
  for (int dir = 0; dir < 2; dir++) {
    const Fe base = dir == 0 ? w : winv;
    Fe step = base;
    for (int i = 0; i < lo_bits; i++) step = bgh::fe_sqr(FR, step);
    upload_fes(ctx, tmp_lo, powers(base, nlo, one));
    upload_fes(ctx, tmp_hi, powers(step, nhi, one));
    k_table_expand<<<ceil_div(half, 256), 256, 0, ctx.stream>>>(dir == 0 ? slot.tw_fwd : slot.tw_inv, tmp_lo,
                                                                  tmp_hi, lo_bits, half);
    BG_CHECK_LAUNCH();
  }
  // coset tables: g^i, g^-i (lo), and n^-1 * g^(i 2^a), n^-1 * g^(-i 2^a) (hi), plain g^(i 2^a) for
  // the natural-order coset NTT
  const int a = (L + 1) / 2;
  const size_t clo = size_t(1) << a, chi = size_t(1) << (L - a);
  const Fe g = fr_mont_u64(5);
  const Fe ginv = bgh::fe_inv(FR, g);
  const Fe ninv = bgh::fe_inv(FR, fr_mont_u64(n));
  Fe ga = g, gia = ginv;
  for (int i = 0; i < a; i++) {
    ga = bgh::fe_sqr(FR, ga);
    gia = bgh::fe_sqr(FR, gia);
  }
  slot.coset_bits = a;
  slot.g_lo = ctx.ws.get_t<uint32_t>(tag + ".g_lo", clo * 8);
  slot.gi_lo = ctx.ws.get_t<uint32_t>(tag + ".gi_lo", clo * 8);
  slot.g_hi = ctx.ws.get_t<uint32_t>(tag + ".g_hi", chi * 8);
  slot.g_hi_ninv = ctx.ws.get_t<uint32_t>(tag + ".g_hi_ninv", chi * 8);
  slot.gi_hi_ninv = ctx.ws.get_t<uint32_t>(tag + ".gi_hi_ninv", chi * 8);
  slot.gi_hi_ninv_canon = ctx.ws.get_t<uint32_t>(tag + ".gi_hi_ninv_canon", chi * 8);
  slot.ninv = ctx.ws.get_t<uint32_t>(tag + ".ninv", 8);
  slot.zinv = ctx.ws.get_t<uint32_t>(tag + ".zinv", 8);
  upload_fes(ctx, slot.g_lo, powers(g, clo, one));
  upload_fes(ctx, slot.gi_lo, powers(ginv, clo, one));
  upload_fes(ctx, slot.g_hi, powers(ga, chi, one));
  upload_fes(ctx, slot.g_hi_ninv, powers(ga, chi, ninv));
  upload_fes(ctx, slot.gi_hi_ninv, powers(gia, chi, ninv));
  upload_fes(ctx, slot.gi_hi_ninv_canon, powers(gia, chi, bgh::fe_from_mont(FR, ninv)));
  upload_fes(ctx, slot.ninv, {ninv});
  // Z(g x) on the coset is the constant g^n - 1
  const Fe zc = bgh::fe_sub(FR, bgh::fe_pow_u64(FR, g, n), one);
  upload_fes(ctx, slot.zinv, {bgh::fe_inv(FR, zc)});
  slot.ready = true;
  return slot;
}

struct PassPlan {
  int s0, k, G;
  int nt = kNttThreads;  // threads per CTA
  bool r4 = true;        // two stages at a time
};

// Small domains (at most 2^kSmallMaxL elements, a small proof's QAP) are a chain of
// latency-bound transforms: they take 128-element tiles of 64 threads, one butterfly per thread
// per stage and at most 7 stages per pass, so a pass spreads over many SMs.  The 1024-element
// tiles give a 2^11 transform two passes of two CTAs each, every thread doing two butterflies
// per stage; one CTA of 1024 threads over the whole vector measured 60-70 us per transform,
// the SM's issue rate spread over 1024 butterflies a stage.
constexpr int kSmallMaxL = 14;
constexpr int kSmallTile = 128;
constexpr int kSmallThreads = 64;

static std::vector<PassPlan> plan_passes(int L) {
  const bool small = L <= kSmallMaxL;
  const int tile = small ? kSmallTile : kNttTile;
  const int kmax = small ? 7 : kContigMax;
  std::vector<PassPlan> out;
  auto add = [&](int s0, int k, int G) {
    PassPlan p{s0, k, G};
    p.nt = small ? std::max(32, (G << k) / 2) : kNttThreads;
    p.r4 = !small;
    out.push_back(p);
  };
  const int k0 = std::min(L, kmax);
  {
    int G = tile >> k0;
    const int groups = 1 << (L - k0);
    if (G > groups) G = groups;
    if (G < 1) G = 1;
    add(0, k0, G);
  }
  int rest = L - k0;
  int s0 = k0;
  const int npass = (rest + kmax - 1) / kmax;
  for (int p = 0; p < npass; p++) {
    const int k = (rest + (npass - p) - 1) / (npass - p);
    int G = tile >> k;
    const int lo_count = 1 << s0;
    if (G > lo_count) G = lo_count;
    add(s0, k, G);
    s0 += k;
    rest -= k;
  }
  return out;
}

// how a pass reads, scales and writes
struct PassIo {
  int pre = SC_NONE, post = SC_NONE;
  ScaleTab sc;
  int load = LD_PLAIN;
  const uint32_t* zinv = nullptr;
  bool rev = false;
  bool qap = false;
};

static void launch_pass(Ctx& ctx, cudaStream_t st, bool dit, const NttVecs& v, int nvec, const uint32_t* tw, int L,
                        const PassPlan& p, const PassIo& io) {
  const size_t n = size_t(1) << L;
  const int E = p.G << p.k;
  const dim3 grid((unsigned)(n / E), (unsigned)nvec);
  const size_t smem = (size_t)E * 32;
  KernelTimer kt(ctx, "ntt_pass", st);
  auto go = [&](auto kernel) {
    kernel<<<grid, p.nt, smem, st>>>(v, tw, L, p.s0, p.k, p.G, io.pre, io.post, io.sc, io.load, io.zinv, io.rev);
  };
  if (!p.r4) {
    if (dit) go(k_ntt_pass<true, false, kSmallThreads, 4>);
    else go(k_ntt_pass<false, false, kSmallThreads, 4>);
  } else if (io.qap) {
    if (dit) go(k_ntt_pass<true, true, kNttThreads, 4>);
    else go(k_ntt_pass<false, true, kNttThreads, 4>);
  } else {
    go(k_ntt_pass<false, true, kNttThreads, 3>);  // standalone transforms are DIF
  }
  BG_CHECK_LAUNCH();
}

// the opt-in to 32 KiB of dynamic shared memory holds for the device current when it is set:
// once per device, safely from several host threads (batch lanes, server threads)
void ntt_init_kernels() {
  constexpr int kMaxDevices = 64;
  static std::once_flag once[kMaxDevices];
  int dev = 0;
  BG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) throw Error(BG_E_ARG, "ntt: device index out of range");
  std::call_once(once[dev], [] {
    auto smem = [](auto* kernel) {
      BG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNttTile * 32));
    };
    smem(k_ntt_pass<true, true, kNttThreads, 4>);
    smem(k_ntt_pass<false, true, kNttThreads, 4>);
    smem(k_ntt_pass<false, true, kNttThreads, 3>);
  });
}

// DIF passes (natural order in, bit-reversed out): from v.src into v.dst by way of `mid` (v.dst
// itself, or where the last pass undoes the bit reversal into v.dst, whose elements then change
// places, another buffer).  `first` and `last` say how the outer passes read and write.
static void dif(Ctx& ctx, cudaStream_t st, const NttVecs& v, uint32_t* const* mid, int nvec, const uint32_t* tw, int L,
                const PassIo& first, const PassIo& last) {
  const auto plan = plan_passes(L);
  for (int i = (int)plan.size() - 1; i >= 0; i--) {
    const bool is_first = i == (int)plan.size() - 1, is_last = i == 0;
    NttVecs w = v;
    for (int k = 0; k < nvec; k++) {
      if (!is_first) w.src[k] = mid[k];
      if (!is_last) w.dst[k] = mid[k];
    }
    PassIo io;
    io.qap = last.qap;
    if (is_first) io = first;
    if (is_last) {
      if (is_first && first.pre != SC_NONE && last.post != SC_NONE)
        throw Error(BG_E_ARG, "ntt: pre and post scaling in a single-pass transform");
      io.post = last.post;
      io.rev = last.rev;
      if (last.post != SC_NONE) io.sc = last.sc;
    }
    launch_pass(ctx, st, false, w, nvec, tw, L, plan[i], io);
  }
}

static void dit(Ctx& ctx, cudaStream_t st, const NttVecs& v, int nvec, const uint32_t* tw, int L) {
  const auto plan = plan_passes(L);
  PassIo io;
  io.qap = true;
  for (size_t i = 0; i < plan.size(); i++) launch_pass(ctx, st, true, v, nvec, tw, L, plan[i], io);
}

void ntt_run(Ctx& ctx, cudaStream_t st, uint32_t* d_data, int L, int mode) {
  if (L == 0) return;
  ntt_init_kernels();
  NttTables& T = ntt_tables(ctx, L);
  const size_t n = size_t(1) << L;
  // the passes before the last leave their tiles in tmp; the last goes back in natural order
  uint32_t* tmp = ctx.ws.get_t<uint32_t>("ntt.tmp", n * 8);
  const NttVecs v{{d_data, d_data, d_data}, {d_data, d_data, d_data}};
  PassIo first, last;
  last.rev = true;
  const uint32_t* tw = T.tw_fwd;
  switch (mode) {
    case BG_NTT_FORWARD:
      break;
    case BG_NTT_INVERSE:
      tw = T.tw_inv;
      last.post = SC_CONST;
      last.sc.hi = T.ninv;
      break;
    case BG_NTT_COSET_FORWARD:
      first.pre = SC_NATURAL;
      first.sc = ScaleTab{T.g_lo, T.g_hi, T.coset_bits};
      break;
    case BG_NTT_COSET_INVERSE:
      tw = T.tw_inv;
      last.post = SC_BITREV;
      last.sc = ScaleTab{T.gi_lo, T.gi_hi_ninv, T.coset_bits};
      break;
    default:
      throw Error(BG_E_ARG, "ntt: unknown mode");
  }
  dif(ctx, st, v, &tmp, 1, tw, L, first, last);
}

// h from the three evaluation vectors (all natural order, packed Montgomery, n = 2^L each).
// a, b, c are overwritten; h receives n elements (h[n-1] = 0 for a satisfied R1CS), Montgomery or
// (canonical) as MSM scalars: the factor of the last scaling then comes from a table that is not in
// Montgomery form, which takes h's own factor R out.
void qap_h_run(Ctx& ctx, cudaStream_t st, uint32_t* d_a, uint32_t* d_b, uint32_t* d_c, uint32_t* d_h, int L,
               bool canonical) {
  ntt_init_kernels();
  NttTables& T = ntt_tables(ctx, L);
  // a, b and c are transformed by the same launches (grid y = 3): each pass fills three times
  // the CTAs, and a small proof's QAP is 6 launches instead of 16
  uint32_t* const abc[3] = {d_a, d_b, d_c};
  const NttVecs v{{d_a, d_b, d_c}, {d_a, d_b, d_c}};
  PassIo plain, to_coset;  // iNTT, then * n^-1 g^j
  plain.qap = to_coset.qap = true;
  to_coset.post = SC_BITREV;
  to_coset.sc = ScaleTab{T.g_lo, T.g_hi_ninv, T.coset_bits};
  dif(ctx, st, v, abc, 3, T.tw_inv, L, plain, to_coset);
  dit(ctx, st, v, 3, T.tw_fwd, L);  // NTT on the coset
  PassIo quotient, from_coset;      // (a b - c) / Z, then the coset iNTT
  quotient.qap = from_coset.qap = true;
  quotient.load = LD_QUOTIENT;
  quotient.zinv = T.zinv;
  from_coset.post = SC_BITREV;
  from_coset.sc = ScaleTab{T.gi_lo, canonical ? T.gi_hi_ninv_canon : T.gi_hi_ninv, T.coset_bits};
  from_coset.rev = true;
  const NttVecs q{{d_a, d_b, d_c}, {d_h, d_h, d_h}};
  dif(ctx, st, q, abc, 1, T.tw_inv, L, quotient, from_coset);
}

}  // namespace bg
