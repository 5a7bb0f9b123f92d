// Pippenger multi-scalar multiplication sum_i s_i * P_i over BN254 G1 (Fq) and G2 (Fq2).
//
// Reference semantics: Msm.g1 / Msm.g2 (bend2/src/msm.bend:297, :529) take n affine
// Montgomery points and n canonical scalars and return the sum as a Jacobian point; the
// caller normalises it (bend2/src/groth16.bend:281-295).  The reference runs unsigned c-bit
// windows (msm.bend:34-58), private per-leaf bucket arrays joined element-wise (:158-173),
// a running-sum reduction per window (:192-205) and a Horner window combine (:225-239).
//
// This implementation (one device, all phases on the device except the final Horner):
//   1. k_digits_hist  signed c-bit digits (|d| <= 2^(c-1)), one thread per scalar; a global
//                     histogram of (window, |d|-1) bucket keys
//   2. exclusive scan of the histogram -> bucket offsets
//   3. k_scatter      (point index | sign << 31) written into bucket order
//   4. k_bucket_acc   load-balanced slices of K entries per thread: XYZZ accumulator += +-P
//                     (mixed add); a bucket cut by slice boundaries leaves pieces, joined
//                     where the reduction reads it (k_bucket_heavy first joins the rare
//                     buckets of very many pieces)
//   5. k_window_reduce one CTA per window part: running sums over M buckets per thread and a tree
//                     that leaves sum_b (b+1) B_b as one sum per bit of the thread's index;
//                     k_window_join sums the parts of a window
//   6. host: one Horner over those bit positions -> affine.  Windows have balanced widths of at
//      most c bits (window_width).
// Window sums and the final point are exact group elements, so the affine result equals the
// reference's for the same inputs regardless of bucket order inside a window.
#include "common.cuh"
#include "ec.cuh"
#include "host_ff.hpp"
#include "host_pool.hpp"
#include "msm.h"
#include "msm_tune.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

namespace bg {

// ---------------------------------------------------------------- scan (exclusive, u32)
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// (inputs rounded up to multiples of pad + 1, pad + 1 a power of two)
__global__ void k_scan_tile(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                            uint32_t* __restrict__ tile_sums, size_t n, uint32_t pad) {
  __shared__ uint32_t warp_tot[kScanThreads / 32];
  const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    v[k] = (base + k < n) ? (in[base + k] + pad) & ~pad : 0u;
    sum += v[k];
  }
  // inclusive warp scan of per-thread sums
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint32_t t = lane < kScanThreads / 32 ? warp_tot[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = t;  // inclusive
  }
  __syncthreads();
  uint32_t excl = x - sum + (wid > 0 ? warp_tot[wid - 1] : 0u);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < n) out[base + k] = excl;
    excl += v[k];
  }
  if (threadIdx.x == kScanThreads - 1 && tile_sums) tile_sums[blockIdx.x] = excl;
}

__global__ void k_scan_add(uint32_t* __restrict__ out, const uint32_t* __restrict__ tile_off, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += tile_off[i / kScanTile];
}

// exclusive scan of n u32 (n >= 1); recursion depth log_2048(n)
void exclusive_scan(Workspace& ws, const std::string& tag, const uint32_t* d_in, uint32_t* d_out, size_t n,
                    cudaStream_t st, int depth, uint32_t pad) {
  const unsigned tiles = ceil_div(n, kScanTile);
  if (tiles == 1) {
    k_scan_tile<<<1, kScanThreads, 0, st>>>(d_in, d_out, nullptr, n, pad);
    BG_CHECK_LAUNCH();
    return;
  }
  uint32_t* sums = ws.get_t<uint32_t>(tag + ".scan_sums" + std::to_string(depth), tiles);
  uint32_t* offs = ws.get_t<uint32_t>(tag + ".scan_offs" + std::to_string(depth), tiles);
  k_scan_tile<<<tiles, kScanThreads, 0, st>>>(d_in, d_out, sums, n, pad);
  BG_CHECK_LAUNCH();
  exclusive_scan(ws, tag, sums, offs, tiles, st, depth + 1, 0);
  k_scan_add<<<ceil_div(n, 256), 256, 0, st>>>(d_out, offs, n);
  BG_CHECK_LAUNCH();
}

// ---------------------------------------------------------------- digits
BG_DEV uint32_t window_bits(const uint32_t* s, int bit, int c) {
  const int limb = bit >> 5, sh = bit & 31;
  if (limb >= 8) return 0u;
  uint64_t v = s[limb];
  if (limb + 1 < 8) v |= (uint64_t)s[limb + 1] << 32;
  return (uint32_t)(v >> sh) & ((1u << c) - 1u);
}

BG_DEV void load_scalar(uint32_t* s, const uint32_t* __restrict__ scalars, size_t i) {
  const uint4 a = reinterpret_cast<const uint4*>(scalars + 8 * i)[0];
  const uint4 b = reinterpret_cast<const uint4*>(scalars + 8 * i)[1];
  s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
  s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
}

// Window layout: W windows cover bits [0, 255) (254 scalar bits and room for the last carry)
// with balanced widths -- the first 255 mod W windows one bit wider -- so that no window is
// much narrower than the others (a narrow top window would pile its entries into a few huge
// buckets).  W = floor(254 / c) + 1 keeps every width at most c.
__host__ __device__ inline int window_width(int w, int W) { return 255 / W + (w < 255 % W ? 1 : 0); }
__host__ __device__ inline int window_offset(int w, int W) { return w * (255 / W) + (w < 255 % W ? w : 255 % W); }

// signed digit of window w of W: returns magnitude (0 = no bucket) and updates carry; *neg set
// when the digit is negative.  Digits lie in [-(2^(b-1) - 1), 2^(b-1)] for a window of b bits;
// scalars below 2^254 leave no carry out of the top window.
BG_DEV uint32_t signed_digit(const uint32_t* s, int w, int W, uint32_t& carry, bool& negd) {
  const int b = window_width(w, W);
  const uint32_t half = 1u << (b - 1);
  const uint32_t d = window_bits(s, window_offset(w, W), b) + carry;
  if (d > half) {
    carry = 1u;
    negd = true;
    return (1u << b) - d;
  }
  carry = 0u;
  negd = false;
  return d;
}

// Bucket key of window w's digit: w * key_stride + |d| - 1 (key_stride = 2^(c-1): one bucket
// set per window; 0: all windows share one set).  Point index stored with it:
// i + w * idx_stride (0: the point itself; n: row w of a table of 2^(o_w)-multiples).
__global__ void k_digits_hist(const uint32_t* __restrict__ scalars, size_t n, int c, int W, uint32_t key_stride,
                              uint32_t* __restrict__ counts, uint32_t* __restrict__ status) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[8];
  load_scalar(s, scalars, i);
  if (s[7] >> 30) {  // scalars must be below 2^254 (every canonical Fr element is)
    atomicOr(status, BG_DSTATUS_SCALAR_RANGE);
    return;
  }
  uint32_t carry = 0;
  for (int w = 0; w < W; w++) {
    bool ng;
    const uint32_t mag = signed_digit(s, w, W, carry, ng);
    if (mag) atomicAdd(&counts[(size_t)w * key_stride + mag - 1], 1u);
  }
}

__global__ void k_scatter(const uint32_t* __restrict__ scalars, size_t n, int c, int W, uint32_t key_stride,
                          uint32_t idx_stride, uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[8];
  load_scalar(s, scalars, i);
  if (s[7] >> 30) return;
  uint32_t carry = 0;
  for (int w = 0; w < W; w++) {
    bool ng;
    const uint32_t mag = signed_digit(s, w, W, carry, ng);
    if (mag) {
      const uint32_t slot = atomicAdd(&cursor[(size_t)w * key_stride + mag - 1], 1u);
      sorted[slot] = ((uint32_t)i + (uint32_t)w * idx_stride) | (ng ? 0x80000000u : 0u);
    }
  }
}

// The same two passes for fewer than 2^kRankLog2 scalars, which are bound by latency: the count an
// entry found is kept as its rank in its bucket (ranks[w n + i]), so the second pass needs no atomics
// and no copy of the offsets; eight windows' digits are recoded first, so that eight atomics or
// writes are in flight per thread instead of one round trip each; and blockIdx.y takes the windows
// in groups of `wg` (the lower windows are recoded again for the carry), so they run side by side.
// 1000 scalars in 43 windows: 51 -> 35 us; 65000: 73 -> 66 us; 2^18 level.  Larger vectors are bound
// by the L2's rate (about 190 G random accesses per second), where the ranks cost more than the
// second atomic: 2^20 scalars in 17 windows, 302 us above and 336 us here.
constexpr int kRankLog2 = 17;
constexpr int kDigitBatch = 8;

// digits of windows [w0, w0 + kDigitBatch) below w1: magnitude | sign << 31 (0: none)
BG_DEV void digit_batch(uint32_t* d, const uint32_t* s, int w0, int w1, int W, uint32_t& carry) {
#pragma unroll
  for (int j = 0; j < kDigitBatch; j++) {
    d[j] = 0;
    if (w0 + j < w1) {
      bool ng;
      const uint32_t mag = signed_digit(s, w0 + j, W, carry, ng);
      d[j] = mag ? (mag | (ng ? 0x80000000u : 0u)) : 0u;
    }
  }
}
// the carry into window w0
BG_DEV uint32_t digit_carry(const uint32_t* s, int w0, int W) {
  uint32_t carry = 0;
  for (int w = 0; w < w0; w++) {
    bool ng;
    signed_digit(s, w, W, carry, ng);
  }
  return carry;
}

__global__ void k_digits_rank(const uint32_t* __restrict__ scalars, size_t n, int W, int wg, uint32_t key_stride,
                              uint32_t* __restrict__ counts, uint32_t* __restrict__ ranks,
                              uint32_t* __restrict__ status) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[8];
  load_scalar(s, scalars, i);
  if (s[7] >> 30) {  // scalars must be below 2^254 (every canonical Fr element is)
    atomicOr(status, BG_DSTATUS_SCALAR_RANGE);
    return;
  }
  const int wb = (int)blockIdx.y * wg, w1 = wb + wg < W ? wb + wg : W;
  uint32_t carry = digit_carry(s, wb, W);
  for (int w0 = wb; w0 < w1; w0 += kDigitBatch) {
    uint32_t d[kDigitBatch], r[kDigitBatch];
    digit_batch(d, s, w0, w1, W, carry);
#pragma unroll
    for (int j = 0; j < kDigitBatch; j++)
      if (d[j]) r[j] = atomicAdd(&counts[(size_t)(w0 + j) * key_stride + (d[j] & 0x7fffffffu) - 1], 1u);
#pragma unroll
    for (int j = 0; j < kDigitBatch; j++)
      if (d[j]) ranks[(size_t)(w0 + j) * n + i] = r[j];
  }
}

__global__ void k_scatter_rank(const uint32_t* __restrict__ scalars, size_t n, int W, int wg, uint32_t key_stride,
                          uint32_t idx_stride, const uint32_t* __restrict__ offsets,
                          const uint32_t* __restrict__ ranks, uint32_t* __restrict__ sorted) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[8];
  load_scalar(s, scalars, i);
  if (s[7] >> 30) return;
  const int wb = (int)blockIdx.y * wg, w1 = wb + wg < W ? wb + wg : W;
  uint32_t carry = digit_carry(s, wb, W);
  for (int w0 = wb; w0 < w1; w0 += kDigitBatch) {
    uint32_t d[kDigitBatch], slot[kDigitBatch];
    digit_batch(d, s, w0, w1, W, carry);
#pragma unroll
    for (int j = 0; j < kDigitBatch; j++)
      if (d[j])
        slot[j] = offsets[(size_t)(w0 + j) * key_stride + (d[j] & 0x7fffffffu) - 1] + ranks[(size_t)(w0 + j) * n + i];
#pragma unroll
    for (int j = 0; j < kDigitBatch; j++)
      if (d[j]) sorted[slot[j]] = ((uint32_t)i + (uint32_t)(w0 + j) * idx_stride) | (d[j] & 0x80000000u);
  }
}

// Window table of a fixed point set: row w holds 2^(o_w) P_i, o_w the offset of window w
// (affine, row-major, n points per row); computed once per proving key, one thread per point
// (a window's width of doublings per row, one inversion per entry).
template <class F>
__global__ void __launch_bounds__(128) k_build_table(const uint32_t* __restrict__ pts, size_t n, int c, int W,
                                                     uint32_t* __restrict__ table) {
  constexpr int PW = 2 * FieldWords<F>::value;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Affine<F> p = load_affine<F>(pts + i * PW);
  store_affine(table + i * PW, p);
  XYZZ<F> q = xyzz_from_affine(p);
  for (int w = 1; w < W; w++) {
    for (int d = 0; d < window_width(w - 1, W); d++) q = xyzz_dbl(q);
    Affine<F> a;
    if (is_inf(q)) {
      a.x = field_zero<F>();
      a.y = field_zero<F>();
    } else {
      const F t = field_inv_any(fmul(q.zz, q.zzz));
      a.x = fmul(q.x, fmul(t, q.zzz));
      a.y = fmul(q.y, fmul(t, q.zz));
    }
    store_affine(table + ((size_t)w * n + i) * PW, a);
  }
}


// ---------------------------------------------------------------- buckets
// Segmented accumulation: the bucket-ordered entry list (T entries) is cut into slices of K
// entries, one per thread, so every thread runs exactly K mixed additions whatever the bucket
// sizes are (one thread per bucket would idle most lanes of a warp on Poisson-sized buckets).
// A run of entries that covers a whole bucket is written to that bucket; a run cut by a slice
// boundary becomes a piece: entry 2t of the piece list if the run started in an earlier slice,
// entry 2t+1 if the bucket starts in slice t and continues into a later one.  So a bucket with
// entries [o, o') cut into slices t0 = o / K .. t1 = (o' - 1) / K has its pieces at 2 t0 + 1
// and 2 u for t0 < u <= t1; the window reduction adds them where it reads the
// bucket, which costs the same additions as a separate join pass without its launch
// and its mostly idle lanes.  A bucket of more than `limit` + 1 pieces (piece_limit; a scalar value
// repeated thousands of times) is joined beforehand by k_bucket_heavy: the thread that owns its
// first piece lists it in heavy[1 + i] (heavy[0] counts, cleared before the accumulation).
// G2's accumulation stages the next entry's point in shared memory (cp.async) instead of
// registers, where a prefetched Fq2 point held 32 registers across the whole addition: 20 registers
// fewer (214 now) and 1% of the G2 accumulation.  The registers saved do
// not buy more warps: with 9, 10 or 12 per SM instead of 8 the accumulation of a 2^18 MSM measured
// 2.25-2.29 ms against 1.89.  G1 keeps its register
// prefetch (128 registers, four 128-thread CTAs per SM either way).
template <class F>
constexpr bool kAccStaged = FieldWords<F>::value == 16;
// CTA size of the accumulation
template <class F>
constexpr int kAccThreads = 128;

// 16-byte asynchronous copy global -> shared (cached in L2 only), and the wait for a thread's
// own copies
BG_DEV void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
BG_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
BG_DEV void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// the affine point held in 16-byte chunks c[0 .. 2 FW / 4)
BG_DEV Fq fp_of(const uint4& a, const uint4& b) {
  Fq r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}
template <class F>
BG_DEV Affine<F> affine_of_chunks(const uint4* c, size_t stride) {
  Affine<F> p;
  if constexpr (FieldWords<F>::value == 16) {
    p.x.c0 = fp_of(c[0], c[stride]);
    p.x.c1 = fp_of(c[2 * stride], c[3 * stride]);
    p.y.c0 = fp_of(c[4 * stride], c[5 * stride]);
    p.y.c1 = fp_of(c[6 * stride], c[7 * stride]);
  } else {
    p.x = fp_of(c[0], c[stride]);
    p.y = fp_of(c[2 * stride], c[3 * stride]);
  }
  return p;
}

template <class F>
__global__ void __launch_bounds__(kAccThreads<F>) k_bucket_acc(const uint32_t* __restrict__ points,
                                                               const uint32_t* __restrict__ offsets,
                                                               const uint32_t* __restrict__ sorted, uint32_t nbuckets,
                                                               uint32_t K, uint32_t limit,
                                                               uint32_t* __restrict__ buckets,
                                                               uint32_t* __restrict__ parts, uint32_t* __restrict__ heavy) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int PW = 4 * FW;
  const uint32_t total = offsets[nbuckets];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t beg64 = (uint64_t)t * K;
  if (beg64 >= total) return;
  const uint32_t beg = (uint32_t)beg64;
  const uint32_t end = (total - beg) < K ? total : beg + K;
  // bucket holding entry `beg`: the last b with offsets[b] <= beg
  uint32_t lo = 0, hi = nbuckets;  // offsets[lo] <= beg < offsets[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (offsets[mid] <= beg) lo = mid;
    else hi = mid;
  }
  // One flat loop of exactly (end - beg) mixed additions, so the lanes of a warp stay in
  // step; a bucket boundary only costs a short divergent flush.
  uint32_t b = lo;
  uint32_t bstart = offsets[b], bend = offsets[b + 1];
  XYZZ<F> acc = xyzz_inf<F>();
  // The next entry's point is gathered before this entry's addition, so the gather's latency
  // hides behind the arithmetic (1.5% of a G1 accumulation; four 128-thread CTAs per SM either
  // way): into registers for G1, into one of two shared-memory slots for G2 (the
  // slot read in this iteration is refilled two iterations later, after the addition that
  // consumed it).
  // sorted == nullptr: the entries are the points themselves (the output of the pair rounds)
  constexpr int CH = 2 * FW / 4;  // 16-byte chunks of an affine point
  constexpr int kSlots = kAccStaged<F> ? 2 : 1, kChunks = kAccStaged<F> ? CH : 1;
  __shared__ uint4 stage[kSlots][kChunks][kAccThreads<F>];
  auto gather = [&](uint32_t c, int slot) {
    if constexpr (kAccStaged<F>) {
      const uint4* src = reinterpret_cast<const uint4*>(points + (size_t)(c & 0x7fffffffu) * 2 * FW);
#pragma unroll
      for (int j = 0; j < CH; j++) cp_async16(&stage[slot][j][threadIdx.x], src + j);
      cp_async_commit();
    }
  };
  uint32_t code = sorted ? sorted[beg] : beg;
  Affine<F> p;
  if constexpr (kAccStaged<F>) gather(code, 0);
  else p = load_affine<F>(points + (size_t)(code & 0x7fffffffu) * 2 * FW);
  int slot = 0;
  for (uint32_t e = beg; e < end; e++) {
    uint32_t code_n = 0;
    Affine<F> pn;
    if constexpr (kAccStaged<F>) {
      cp_async_wait_all();
      p = affine_of_chunks<F>(&stage[slot][0][threadIdx.x], kAccThreads<F>);
      if (e + 1 < end) {
        code_n = sorted ? sorted[e + 1] : e + 1;
        gather(code_n, slot ^ 1);
      }
      slot ^= 1;
    } else if (e + 1 < end) {
      code_n = sorted ? sorted[e + 1] : e + 1;
      pn = load_affine<F>(points + (size_t)(code_n & 0x7fffffffu) * 2 * FW);
    }
    if (code >> 31) p = affine_neg(p);
    acc = xyzz_madd(acc, p);
    if constexpr (!kAccStaged<F>) p = pn;
    code = code_n;
    if (e + 1 == bend || e + 1 == end) {
      if (bstart < beg || bend > end) {
        const size_t slot = 2 * (size_t)t + (bstart < beg ? 0 : 1);
        store_xyzz(parts + slot * PW, acc);
        if (bstart >= beg && (bend - 1) / K - t > limit) heavy[1 + atomicAdd(heavy, 1u)] = b;
      } else {
        store_xyzz(buckets + (size_t)b * PW, acc);
      }
      acc = xyzz_inf<F>();
      if (e + 1 < end) {
        do {
          b++;
        } while (offsets[b + 1] <= e + 1);  // skip empty buckets
        bstart = offsets[b];
        bend = offsets[b + 1];
      }
    }
  }
}

// Heavy buckets: one CTA per bucket, a strided sum of its pieces per thread and a tree over the
// CTA; the sum goes to the bucket.  The grid is fixed; CTAs loop over however many the
// accumulation listed (none for uniformly spread scalars).
template <class F>
__global__ void __launch_bounds__(256) k_bucket_heavy(const uint32_t* __restrict__ offsets,
                                                      const uint32_t* __restrict__ parts, uint32_t K,
                                                      const uint32_t* __restrict__ heavy,
                                                      uint32_t* __restrict__ buckets) {
  constexpr int PW = 4 * FieldWords<F>::value;
  extern __shared__ uint32_t sm[];
  const uint32_t nh = heavy[0];
  for (uint32_t h = blockIdx.x; h < nh; h += gridDim.x) {
    const uint32_t b = heavy[1 + h];
    const uint32_t t0 = offsets[b] / K;
    const uint32_t np = (offsets[b + 1] - 1) / K - t0 + 1;
    XYZZ<F> acc = xyzz_inf<F>();
    for (uint32_t i = threadIdx.x; i < np; i += blockDim.x) {
      const size_t slot = i == 0 ? 2 * (size_t)t0 + 1 : 2 * ((size_t)t0 + i);
      acc = xyzz_add(acc, load_xyzz<F>(parts + slot * PW));
    }
    store_xyzz(sm + (size_t)threadIdx.x * PW, acc);
    __syncthreads();
    for (uint32_t d = blockDim.x >> 1; d >= 1; d >>= 1) {
      if (threadIdx.x < d) {
        acc = xyzz_add(acc, load_xyzz<F>(sm + (size_t)(threadIdx.x + d) * PW));
        store_xyzz(sm + (size_t)threadIdx.x * PW, acc);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) store_xyzz(buckets + (size_t)b * PW, acc);
    __syncthreads();
  }
}
// CTA size: a bucket with a large part of an MSM's entries (the top bit of scalars of 16 bits under 15-bit
// windows: 4000 pieces) is one CTA's strided sum, so a standalone G1 MSM takes as many threads as the
// shared memory that needs no opt-in holds; a proof's pass fits beside other kernels' CTAs.
template <class F>
constexpr uint32_t heavy_threads(bool in_proof) {
  return FieldWords<F>::value == 8 && !in_proof ? 256 : 128;
}
constexpr uint32_t kHeavyGrid = 152;

#include "msm_pairs.cuh"

// Entries per accumulation thread in a proof and for MSMs that fill the GPU, from a latency model in
// dependent mixed additions: a thread's K, or the whole accumulation at its throughput when that is
// longer (then 32, the fewest pieces), and the e / K pieces that a bucket of e entries leaves for the
// reduction.  A piece costs more the more buckets share the multiplier, and little in all, since the
// reductions run beside other accumulations.  Against one price per piece: SquareChain(2^12) 0.622 ->
// 0.608 ms, 2^15 1.44 -> 1.37, 2^16 2.28 -> 2.19.  K stays a power of two (12 and 24 too: one-shot 2^11
// 0.79 -> 0.86 ms, 2^13 1.14 -> 1.21).
template <class F>
uint32_t slice_entries(size_t max_entries, size_t nkeys) {
  constexpr bool g2 = FieldWords<F>::value == 16;
  const double e = (double)max_entries / (double)(nkeys ? nkeys : 1);
  const double least = (double)max_entries / (g2 ? 26000.0 : 47000.0);
  const double piece = std::min(g2 ? 1.4 : 3.0, std::max(1.0, (double)nkeys / (g2 ? 1000.0 : 2700.0)));
  uint32_t best = 32;
  double best_t = 1e300;
  for (uint32_t k = 4; k <= 32; k <<= 1) {
    const double t = std::max((double)k, least) + e / k * piece;
    if (t < best_t) {
      best_t = t;
      best = k;
    }
  }
  return best;
}

// Most positions a thread of a pair round takes: the CTA's batch that shares an inversion (18 us with
// its tree, which the CTA's neighbours on the SM start together).  G1 MSM 2^20's two rounds: 1.82 ms
// with at most 24 positions, 1.73 with 48, 1.71 with 128 (one wave of 115 and 57).
constexpr double kPairPer = 64;
// Threads of a kernel resident on the whole GPU at once (SMs x CTAs per SM x CTA size).
template <class K>
int resident_threads(K kernel, int threads, size_t smem) {
  int dev = 0, sms = 0, occ = 0;
  BG_CUDA(cudaGetDevice(&dev));
  BG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  BG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem));
  return sms * (occ > 0 ? occ : 1) * threads;
}
// of a pair round
template <class F>
double pair_slots() {
  static CachedInt slots;
  return slots.get([] { return resident_threads(k_pair_round<F, true>, kPairThreads<F>, pair_smem_bytes<F>()); });
}
// of the accumulation
template <class F>
double acc_slots() {
  static CachedInt slots;
  return slots.get([] { return resident_threads(k_bucket_acc<F>, kAccThreads<F>, 0); });
}

// Pieces after the first from which a bucket goes to k_bucket_heavy, whose tree costs its eight
// additions whatever the count.  The reduction adds a bucket's pieces one after another, M buckets
// per thread, and its shape counts on the e / K that a bucket of e = max_entries / nkeys entries
// leaves: three times that and four more are what evenly spread scalars never reach, 24 the most.
// With 24 alone, scalars of 8 bits put up to 20 pieces into each of the 255 lowest buckets where the
// shape counts on one: MSMs of 131072 such scalars took 1.29 ms in G1 and 3.39 in G2, 0.50 and 1.01 now.
inline uint32_t piece_limit(size_t max_entries, size_t nkeys, uint32_t K) {
  const size_t mean = max_entries / ((nkeys ? nkeys : 1) * K);
  return (uint32_t)std::min<size_t>(24, 4 + 3 * mean);
}

// Scratch of the bucket phase for at most max_entries entries (words): pieces and the heavy list.
struct BucketScratch {
  uint32_t K = 32;            // entries per accumulation thread
  uint32_t limit = 24;        // piece_limit
  uint32_t* parts = nullptr;  // 2 x slices XYZZ points
  uint32_t* heavy = nullptr;  // 1 + slices / limit + 1
};
inline size_t bucket_slices(size_t max_entries, uint32_t K) { return (max_entries + K - 1) / K; }

// Every slice costs the same K additions, so an accumulation grid of 1.6 waves takes as long
// as 2.  When the model's slices need more than one wave, K is rounded so that the grid is a
// whole number of waves (the nearest, at least one): 9% of the G2 accumulation of a 2^18
// MSM, whose slices fill 1.6 waves.  Slices then hold at least 3/4 of the model's K
// (rounding 1.5 waves up to 2 at worst); the model picks K = 32 for every MSM that needs more
// than a wave and at least 2^21 entries.
template <class F>
uint32_t whole_wave_slices(size_t max_entries, uint32_t K) {
  const double slots = acc_slots<F>();
  const double waves = std::ceil((double)max_entries / K) / slots;
  if (waves <= 1.0) return K;
  const double rounded = std::max(1.0, std::round(waves));
  return (uint32_t)std::ceil((double)max_entries / (rounded * slots));
}

// A standalone MSM's K where its slices do not fill the GPU.  The accumulation lasts as long as the SM
// with the most CTAs, K additions each at a price that depends on how many share it, so the good K are
// those whose grid just fits 1, 2, ... CTAs on every SM (G1 44236 points, 281 / 321 / 375 / 450 CTAs on
// 152 SMs: 532 / 602 / 571 / 554 us; G2 32768 points 256 / 307 CTAs: 1028 / 1162 us); a piece
// costs one addition where the buckets fit a warp per scheduler, several where many share the multiplier.
// With K of 4, 6, 8, 12, 16, 24 or 32 whatever the grid G2 32768 points measured 1140 us, here 989; G1
// 1000 points 241 and 240, where one price per piece and K of 4, 8, 16 or 32 measured 267.
template <class F>
uint32_t level_slices(size_t max_entries, size_t nkeys) {
  constexpr bool g2 = FieldWords<F>::value == 16;
  constexpr int kResident = g2 ? 2 : 4;  // CTAs per SM
  // an addition with 1 .. kResident CTAs on the SM, in those of one alone
  const double price[4] = {1.0, g2 ? 1.28 : 1.2, 1.7, 2.26};
  const double piece = std::min(g2 ? 8.0 : 4.5, std::max(1.0, (double)nkeys / (g2 ? 3300.0 : 600.0)));
  const double e = (double)max_entries / (double)(nkeys ? nkeys : 1);
  const double sms = std::max(1.0, acc_slots<F>() / (kResident * kAccThreads<F>));
  uint32_t best = 32;
  double best_t = 1e300;
  for (uint32_t k = 4; k <= 48; k++) {
    const double ctas = std::ceil(std::ceil((double)max_entries / k) / kAccThreads<F>);
    const double level = std::ceil(ctas / sms), waves = std::ceil(level / kResident);
    const double t = k * waves * price[(int)std::min<double>(level, kResident) - 1] + e / k * piece;
    if (t < best_t) {
      best_t = t;
      best = k;
    }
  }
  return best;
}

template <class F, class Get>
BucketScratch bucket_scratch(size_t max_entries, size_t nkeys, bool in_proof, Get get, uint32_t K = 0) {
  constexpr int PW = 4 * FieldWords<F>::value;
  BucketScratch b;
  if (!K && !in_proof && max_entries < (size_t(1) << 21)) K = level_slices<F>(max_entries, nkeys);
  b.K = K ? K : whole_wave_slices<F>(max_entries, slice_entries<F>(max_entries, nkeys));
  const size_t s = bucket_slices(max_entries, b.K);
  b.limit = piece_limit(max_entries, nkeys, b.K);
  b.parts = get("parts", 2 * s * PW);
  b.heavy = get("heavy", s / b.limit + 2);
  return b;
}

// Accumulation on `st`: buckets of single-slice runs are final, cut buckets leave pieces.
template <class F>
void bucket_accumulate(Ctx* prof, cudaStream_t st, const uint32_t* points, const uint32_t* offsets,
                       const uint32_t* sorted, uint32_t nkeys, size_t max_entries, uint32_t* buckets,
                       const BucketScratch& s) {
  constexpr int FW = FieldWords<F>::value;
  const size_t slices = bucket_slices(max_entries, s.K);
  BG_CUDA(cudaMemsetAsync(s.heavy, 0, sizeof(uint32_t), st));
  std::unique_ptr<KernelTimer> kt(prof ? new KernelTimer(*prof, FW == 8 ? "msm_bucket_acc_g1" : "msm_bucket_acc_g2", st)
                                       : nullptr);
  k_bucket_acc<F><<<ceil_div(slices, kAccThreads<F>), kAccThreads<F>, 0, st>>>(points, offsets, sorted, nkeys, s.K, s.limit, buckets, s.parts,
                                                         s.heavy);
  BG_CHECK_LAUNCH();
}

// Heavy buckets on `st` (a pass that exits at once when there are none).
template <class F>
void bucket_heavy(Ctx* prof, cudaStream_t st, const uint32_t* offsets, uint32_t* buckets, const BucketScratch& s,
                  bool in_proof) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int PW = 4 * FW;
  std::unique_ptr<KernelTimer> kt(prof ? new KernelTimer(*prof, FW == 8 ? "msm_heavy_g1" : "msm_heavy_g2", st)
                                       : nullptr);
  const uint32_t threads = heavy_threads<F>(in_proof);
  k_bucket_heavy<F><<<kHeavyGrid, threads, threads * PW * sizeof(uint32_t), st>>>(offsets, s.parts, s.K, s.heavy,
                                                                                  buckets);
  BG_CHECK_LAUNCH();
}

// Window reduction, one CTA per (window, part).  Part j of window w covers buckets
// [j RT M, (j+1) RT M); thread t folds M consecutive buckets into R_t = sum B and
// T_t = sum_k (k+1) B_{tM+k} (running sums).  The part's weighted sum
//   S_j = sum_{local b} (b+1) B_b = sum_t T_t + M sum_t t R_t
// is left split by the bits of t: sum_t t R_t = sum_b 2^b U_b with U_b the sum of the R_t whose t
// has bit b.  Halving R over t and t + d leaves in the columns [d, 2d) just the terms of U_log2(d),
// so one tree of log2(RT) levels sums R, T and, in the columns that it frees, every U_b; no level
// has more than RT additions and the host's Horner, which doubles through all those bit positions
// anyway, adds each U_b at its own.  k_window_join sums the parts of a window the same way.
//
// The points a thread owns lie in shared memory (word i of thread t's point at base[i * RT + t]): R
// and T.  One out-of-line body adds a point into another, its products inlined, so no point is live
// in registers across a call: fourteen calls per addition, registers across all of them, measured
// 207 us for the reductions of 16000 G1 points where this took 185.
//
// Bound by the latency of the chain of additions, two warps per scheduler at most.  The suffix scan
// of R that this tree replaced (all threads in each of log2(RT) steps, then M Suf_t by doublings and
// a second tree) was half of that chain: reductions of G1 MSMs of 16000 / 2^18 / 2^20 points 185 /
// 410 / 404 -> 94 / 334 / 326 us, of G2 MSMs of 65000 / 2^18 points 687 / 1172 -> 395 / 903 us;
// proofs SquareChain(2^10) 0.555 -> 0.525 ms, 2^14 1.15 -> 1.08, 2^15 1.63 -> 1.48, 2^17 3.98 ->
// 3.74, 2^20 20.5 -> 20.3 (a mixed batch of 16: 16.5 -> 16.7).
BG_DEV void elem_load(Fq& e, const uint32_t* src, uint32_t stride) {
#pragma unroll
  for (int l = 0; l < 8; l++) e.v[l] = src[l * stride];
}
BG_DEV void elem_load(Fq2& e, const uint32_t* src, uint32_t stride) {
  elem_load(e.c0, src, stride);
  elem_load(e.c1, src + 8 * stride, stride);
}
BG_DEV void elem_store(uint32_t* dst, uint32_t stride, const Fq& e) {
#pragma unroll
  for (int l = 0; l < 8; l++) dst[l * stride] = e.v[l];
}
BG_DEV void elem_store(uint32_t* dst, uint32_t stride, const Fq2& e) {
  elem_store(dst, stride, e.c0);
  elem_store(dst + 8 * stride, stride, e.c1);
}
template <class F>
BG_DEV void pt_load(XYZZ<F>& p, const uint32_t* src, uint32_t stride) {
  constexpr int FW = FieldWords<F>::value;
  elem_load(p.x, src, stride);
  elem_load(p.y, src + FW * stride, stride);
  elem_load(p.zz, src + 2 * FW * stride, stride);
  elem_load(p.zzz, src + 3 * FW * stride, stride);
}
template <class F>
BG_DEV void pt_store(uint32_t* dst, uint32_t stride, const XYZZ<F>& p) {
  constexpr int FW = FieldWords<F>::value;
  elem_store(dst, stride, p.x);
  elem_store(dst + FW * stride, stride, p.y);
  elem_store(dst + 2 * FW * stride, stride, p.zz);
  elem_store(dst + 3 * FW * stride, stride, p.zzz);
}
// dst (stride) += src: shared memory with stride sstride, or a contiguous point in global
// memory (sstride 1)
template <class F>
static __device__ __noinline__ void pt_add_into(uint32_t* dst, uint32_t stride, const uint32_t* src,
                                                uint32_t sstride) {
  XYZZ<F> p, q;
  pt_load(p, dst, stride);
  if (sstride == 1) q = load_xyzz<F>(src);
  else pt_load(q, src, sstride);
  pt_store(dst, stride, xyzz_add_inline(p, q));
}
// shared memory of k_window_reduce: R and T (one bucket per thread: T_t = R_t)
template <class F>
constexpr size_t reduce_sm_bytes(uint32_t RT, uint32_t M) {
  return (M == 1 ? 1 : 2) * (size_t)RT * 4 * FieldWords<F>::value * sizeof(uint32_t);
}
// The tree's level d: additions col += col + d for the first d columns of R, of T (with_t) and of
// each U_b split off so far (offset o).  Index i of them -> column of R, or of T (from RT up).
BG_DEV uint32_t tree_column(uint32_t i, uint32_t d, uint32_t RT, bool with_t) {
  const uint32_t q = i / d, k = i % d;
  if (q == 0) return k;
  if (with_t && q == 1) return RT + k;
  return ((2 * d) << (q - 1 - (with_t ? 1 : 0))) + k;
}
BG_DEV uint32_t tree_count(uint32_t d, uint32_t RT, bool with_t) {
  uint32_t arrays = with_t ? 2 : 1;
  for (uint32_t e = 2 * d; e < RT; e <<= 1) arrays++;
  return arrays * d;
}

// A part's points in `out`: T, U_0 .. U_(log2 RT - 1), and with several parts R last.
template <class F>
__global__ void __launch_bounds__(256)
    k_window_reduce(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ buckets,
                    const uint32_t* __restrict__ pieces, uint32_t K, uint32_t limit, uint32_t nb, uint32_t M,
                    uint32_t J, uint32_t* __restrict__ out) {
  constexpr int PW = 4 * FieldWords<F>::value;
  extern __shared__ uint32_t sm[];
  const uint32_t RT = blockDim.x;
  const uint32_t w = blockIdx.x / J, j = blockIdx.x % J, t = threadIdx.x;
  const size_t key0 = (size_t)w * nb + ((size_t)j * RT + t) * M;
  const bool with_t = M > 1;
  // point of column c: R below RT, T from RT up
  auto col = [&](uint32_t c) { return sm + (c < RT ? c : (size_t)PW * RT + (c - RT)); };
  uint32_t* R = sm + t;                     // running sum R_t
  uint32_t* T = sm + (size_t)PW * RT + t;   // weighted sum T_t
  pt_store(R, RT, xyzz_inf<F>());
  if (with_t) pt_store(T, RT, xyzz_inf<F>());
  for (int k = (int)M - 1; k >= 0; k--) {
    const size_t key = key0 + k;
    const uint32_t o0 = offsets[key], o1 = offsets[key + 1];
    if (o1 != o0) {
      const uint32_t t0 = o0 / K, t1 = (o1 - 1) / K;
      if (t0 == t1 || t1 - t0 > limit) {
        pt_add_into<F>(R, RT, buckets + key * PW, 1);
      } else {
        pt_add_into<F>(R, RT, pieces + (2 * (size_t)t0 + 1) * PW, 1);
        for (uint32_t u = t0 + 1; u <= t1; u++) pt_add_into<F>(R, RT, pieces + 2 * (size_t)u * PW, 1);
      }
    }
    if (with_t) pt_add_into<F>(T, RT, R, RT);
  }
  __syncthreads();
  for (uint32_t d = RT >> 1; d >= 1; d >>= 1) {
    if (t < tree_count(d, RT, with_t)) {
      const uint32_t c = tree_column(t, d, RT, with_t);
      pt_add_into<F>(col(c), RT, col(c + d), RT);
    }
    __syncthreads();
  }
  uint32_t lrt = 0;
  while ((1u << lrt) < RT) lrt++;
  const uint32_t np = lrt + 1 + (J > 1 ? 1 : 0);
  uint32_t* o = out + (size_t)blockIdx.x * np * PW;
  for (uint32_t i = t; i < np * PW; i += RT) {
    const uint32_t q = i / PW;
    const uint32_t c = q == 0 ? (with_t ? RT : 0u) : q <= lrt ? 1u << (q - 1) : 0u;
    o[i] = col(c)[(size_t)(i % PW) * RT];
  }
}

// Shape of the window reduction: RT threads x M buckets per thread x J parts per window, picked
// by a latency model.  A thread's dependent chain is M (2 + e / K) additions (each bucket
// costs its pieces, about 1 + e / K for e entries per bucket, plus the running-sum addition that
// a single bucket does without) and the tree's log2(RT), times the number of waves the sets x J
// CTAs need at the kernel's occupancy; the join of several parts adds a launch and its own levels.
constexpr double kCoopAddCost = 0.45, kCoopWarpCost = 0.1;
struct ReduceShape {
  uint32_t RT, M, J;
  double cost = 0;     // the model's latency, in dependent additions
  bool coop = false;   // k_window_reduce_coop: RT groups of 8 lanes
  bool scan = false;   // which weighs its one part's sums itself
};
inline int log2_of(uint32_t x) {
  int l = 0;
  while ((1u << l) < x) l++;
  return l;
}
template <class F>
int reduce_blocks_per_sm(uint32_t RT) {
  static CachedInt cache[9];
  return cache[log2_of(RT)].get([&] {
    int n = 0;
    BG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_window_reduce<F>, (int)RT, reduce_sm_bytes<F>(RT, 2)));
    return n > 0 ? n : 1;
  });
}
// dependent additions over a thread's own buckets
inline double reduce_chain(uint32_t M, double entries_per_slice) {
  return M * (1.0 + entries_per_slice) + (M > 1 ? M : 0);
}
// the join of J parts, in additions of the reduction's threads
constexpr double kJoinLaunchCost = 0.5;
// A set's points beside T cost the host an addition each.  From 64 additions on they go to the
// host pool, whose wake-up (about 45 us) is worth four additions here: for the small sets of a small
// MSM more than the levels saved, so that a part that covers its set weighs its sums itself (a
// suffix scan, log2(RT) levels more; MSMs of 1000 points G1 / G2 269 / 493 us, 305 / 556 by bits).
constexpr int kHostPoolPoints = 64;
constexpr double kHostPoolCost = 4.0;
inline bool reduce_scan(uint32_t RT, uint32_t M, uint32_t J, int sets) {
  return J == 1 && M == 1 && sets * log2_of(RT) >= kHostPoolPoints;
}
inline double host_cost(bool scan, uint32_t span, int sets) {
  return !scan && sets >= 4 && sets * log2_of(span) >= kHostPoolPoints ? kHostPoolCost : 0.0;
}
constexpr uint32_t kCoopMaxParts = 4096;  // of all sets: bounds the parts buffer (8 MB in G2)
// (k_window_join: 32 groups at most, the last point's tree the longest)
inline double join_cost(uint32_t J) {
  if (J == 1) return 0.0;
  double adds = 0;
  for (uint32_t d = J >> 1, arrays = 1; d >= 1; d >>= 1, arrays++) adds += (arrays * d + 31) / 32;
  return kJoinLaunchCost + kCoopAddCost * adds;
}
// Waves of CTAs times how far warps that share a scheduler slow each other's additions, two of them
// being the unit; small CTAs follow one another without a last empty wave.
inline double thread_waves(double ctas, int bps, uint32_t RT, int sm_count) {
  const double waves = ctas / ((double)sm_count * bps);
  const double resident = std::min<double>(bps, std::ceil(ctas / sm_count)) * RT / 128.0;
  return std::max(1.0, bps >= 4 ? waves : std::ceil(waves)) * (1.0 + 0.35 * std::max(0.0, resident - 2.0));
}

template <class F>
ReduceShape reduce_shape(uint32_t nb, int sets, size_t entries, uint32_t K, int sm_count, uint32_t min_rt,
                         uint32_t max_rt) {
  const double e = (double)entries / ((double)nb * sets);
  ReduceShape best{nb < 32 ? nb : 32, 1, 1};
  best.J = nb / best.RT;
  double best_cost = 1e300;
  for (uint32_t RT = nb < min_rt ? 32 : min_rt; RT <= max_rt; RT <<= 1) {
    for (uint32_t M = 1; M <= 16; M <<= 1) {
      if ((uint64_t)RT * M > nb) continue;
      const uint32_t J = nb / (RT * M);
      const double waves = thread_waves((double)J * sets, reduce_blocks_per_sm<F>(RT), RT, sm_count);
      const double cost = waves * (reduce_chain(M, e / K) + log2_of(RT)) + join_cost(J) +
                          host_cost(false, nb / M, sets);
      if (cost < best_cost) {
        best_cost = cost;
        best = {RT, M, J, cost, false};
      }
    }
  }
  best.cost = best_cost;
  return best;
}

// A hidden reduction's shape by work instead of latency: the one with the fewest warp-additions
// per bucket (the running sums, plus the tree that a CTA of RT threads adds on top, counted per
// warp as a warp issues them) whose latency by reduce_shape's model stays
// within `max_cost` dependent additions; {0, 0, 0} when none does.
template <class F>
ReduceShape reduce_shape_work(uint32_t nb, int sets, size_t entries, uint32_t K, int sm_count, uint32_t max_rt,
                              double max_cost) {
  const double e = (double)entries / ((double)nb * sets);
  ReduceShape best{0, 0, 0, 1e300, false};
  double best_work = 1e300;
  for (uint32_t RT = 32; RT <= max_rt; RT <<= 1) {
    for (uint32_t M = 1; M <= 16; M <<= 1) {
      if ((uint64_t)RT * M > nb) continue;
      const uint32_t J = nb / (RT * M);
      const double waves = thread_waves((double)J * sets, reduce_blocks_per_sm<F>(RT), RT, sm_count);
      const double cost = waves * (reduce_chain(M, e / K) + log2_of(RT)) + join_cost(J);
      if (cost > max_cost) continue;
      double tree = 0;
      for (uint32_t d = RT >> 1; d >= 1; d >>= 1)
        tree += std::ceil(d * (log2_of(RT / d) + (M > 1 ? 1 : 0)) / 32.0);
      const double work = (RT / 32.0 * reduce_chain(M, e / K) + tree) / ((double)RT * M);
      if (work < best_work - 1e-12) {
        best_work = work;
        best = {RT, M, J, cost, false};
      }
    }
  }
  return best;
}

#include "msm_coop.cuh"

// The cooperative form's shape by the same model: RT groups (of 8 lanes) per CTA, each addition
// about kCoopAddCost of a thread's addition (dependency depth 4.6 of 14 products, plus the
// group's exchanges) with one warp per scheduler and kCoopWarpCost more for each further one.
template <class F>
int reduce_coop_blocks_per_sm(uint32_t RT) {
  static CachedInt cache[6];
  return cache[log2_of(RT)].get([&] {
    int n = 0;
    BG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_window_reduce_coop<F>, (int)RT * kCoopLanes,
                                                          RT * coop_group_words<F>() * sizeof(uint32_t)));
    return n > 0 ? n : 1;
  });
}
template <class F>
ReduceShape reduce_shape_coop(uint32_t nb, int sets, size_t entries, uint32_t K, int sm_count) {
  const double e = (double)entries / ((double)nb * sets);
  ReduceShape best{0, 0, 0, 1e300, true};
  for (uint32_t RT = 4; RT <= 32; RT <<= 1) {
    for (uint32_t M = 1; M <= 16; M <<= 1) {
      if ((uint64_t)RT * M > nb) continue;
      const uint32_t J = nb / (RT * M);
      if (J > 1 && J * (uint32_t)sets > kCoopMaxParts) continue;
      const int bps = reduce_coop_blocks_per_sm<F>(RT);
      const double ctas = (double)J * sets;
      const double resident = std::min<double>(bps, std::ceil(ctas / sm_count)) * RT * kCoopLanes / 128.0;
      const double add = kCoopAddCost + kCoopWarpCost * std::max(0.0, resident - 1.0);
      const bool scan = reduce_scan(RT, M, J, sets);
      const double cost = std::max(1.0, ctas / ((double)sm_count * bps)) * add *
                              (reduce_chain(M, e / K) + log2_of(RT) * (scan ? 2 : 1)) +
                          join_cost(J) + host_cost(scan, nb / M, sets);
      if (cost < best.cost) best = {RT, M, J, cost, true, scan};
    }
  }
  return best;
}

// Points a bucket set leaves: T and a sum per bit above a thread's buckets.
inline size_t reduce_points(const ReduceShape& r) { return r.scan ? 1 : 1 + log2_of(r.RT) + log2_of(r.J); }
// Points of the parts buffer per bucket set: with several parts theirs (one more each) and the
// joined ones.
inline size_t reduce_part_points(const ReduceShape& r) {
  return r.J > 1 ? r.J * (size_t)(2 + log2_of(r.RT)) + reduce_points(r) : reduce_points(r);
}
// The reduction and, for several parts per window, their join; returns where the sets' points are.
template <class F>
uint32_t* window_reduce(cudaStream_t st, const ReduceShape& r, const uint32_t* offsets, const uint32_t* buckets,
                        const BucketScratch& bs, uint32_t nb, int sets, uint32_t* parts) {
  constexpr int PW = 4 * FieldWords<F>::value;
  if (r.coop)
    k_window_reduce_coop<F><<<sets * r.J, r.RT * kCoopLanes, r.RT * coop_group_words<F>() * sizeof(uint32_t), st>>>(
        offsets, buckets, bs.parts, bs.K, bs.limit, nb, r.M, r.J, r.scan, parts);
  else
    k_window_reduce<F><<<sets * r.J, r.RT, reduce_sm_bytes<F>(r.RT, r.M), st>>>(offsets, buckets, bs.parts, bs.K,
                                                                               bs.limit, nb, r.M, r.J, parts);
  BG_CHECK_LAUNCH();
  if (r.J == 1) return parts;
  const int np = 2 + log2_of(r.RT);
  uint32_t* joined = parts + (size_t)sets * r.J * np * PW;
  const uint32_t groups = std::min<uint32_t>(32, r.J / 2);
  k_window_join<F><<<sets * np, groups * kCoopLanes, groups * (size_t)kCoopTmp * FieldWords<F>::value * sizeof(uint32_t),
                     st>>>(parts, r.J, np, joined);
  BG_CHECK_LAUNCH();
  return joined;
}

// ---------------------------------------------------------------- host driver
static int floor_log2(size_t n) {
  int lg = 0;
  while ((size_t(1) << (lg + 1)) <= n) lg++;
  return lg;
}
static int tuned(const signed char (*tab)[kTuneMaxLog2 - kTuneMinLog2 + 1], size_t n, bool g2) {
  const int lg = floor_log2(n);
  return lg >= kTuneMinLog2 && lg <= kTuneMaxLog2 ? tab[g2 ? 1 : 0][lg - kTuneMinLog2] : 0;
}

int msm_pick_c(size_t n, bool g2) {
  if (const int t = tuned(kTuneSets, n, g2)) return t;
  int c = floor_log2(n) - 3;
  if (c < 3) c = 3;
  if (c > 16) c = 16;
  return c;
}

template <class F>
struct HostField;
template <>
struct HostField<Fq> {
  typedef bgh::FqOps T;
};
template <>
struct HostField<Fq2> {
  typedef bgh::Fq2Ops T;
};

// Sizes of a sort: windows, bucket keys, and entries as padded for as many of `rounds` pair rounds as the
// padding allows (a few empty slots per entry, and positions that fit 31 bits).
struct SortSizes {
  int W, sets, rounds;
  size_t nkeys, entries, padded;
};
static SortSizes sort_sizes(size_t n, int c, bool shared_set, int rounds) {
  SortSizes z;
  z.W = 254 / c + 1;
  z.sets = shared_set ? 1 : z.W;
  z.nkeys = (size_t)z.sets << (c - 1);
  z.entries = n * (size_t)z.W;
  auto padded_to = [&](int r) { return z.entries + z.nkeys * ((size_t(1) << r) - 1); };
  while (rounds > 0 && ((z.nkeys << rounds) > std::max(8 * z.entries, size_t(1) << 20) ||
                        padded_to(rounds) >= 0x80000000ull))
    rounds--;
  z.rounds = rounds;
  z.padded = padded_to(rounds);
  return z;
}
// one rank buffer for a context's sorts below 2^kRankLog2 scalars, else cursors by key
static bool sort_by_rank(size_t n) { return n < (size_t(1) << kRankLog2); }

void msm_sort(Ctx& ctx, cudaStream_t st, const std::string& tag, const uint32_t* d_scalars, size_t n, int c,
              bool shared_set, int rounds, MsmSort& out) {
  out = MsmSort();
  out.n = n;
  if (n == 0) return;
  if (n >= 0x80000000ull) throw Error(BG_E_ARG, "msm: n must be below 2^31");
  if (c < 2 || c > 24) throw Error(BG_E_ARG, "msm: window width out of range");
  const SortSizes z = sort_sizes(n, c, shared_set, rounds);
  if (z.entries >= 0x80000000ull) throw Error(BG_E_ARG, "msm: n x windows must be below 2^31");
  const int W = z.W;
  const uint32_t nb = 1u << (c - 1);
  const size_t nkeys = z.nkeys, padded = z.padded;
  const uint32_t key_stride = shared_set ? 0u : nb;
  const uint32_t idx_stride = shared_set ? (uint32_t)n : 0u;
  rounds = z.rounds;
  out.rounds = rounds;
  out.c = c;
  out.W = W;
  out.sets = z.sets;
  out.nb = nb;
  out.nkeys = nkeys;
  out.max_entries = padded;

  Workspace& ws = ctx.ws;
  uint32_t* counts = ws.get_t<uint32_t>(tag + ".counts", nkeys + 1);
  const bool by_rank = sort_by_rank(n);
  // one rank buffer: the context's sorts are ordered
  uint32_t* cursor = by_rank ? ws.get_t<uint32_t>("sort.ranks", n * (size_t)W)
                             : ws.get_t<uint32_t>(tag + ".cursor", nkeys + 1);
  const dim3 rgrid(ceil_div(n, 256), ceil_div((size_t)W, (size_t)kDigitBatch));
  out.offsets = ws.get_t<uint32_t>(tag + ".offsets", nkeys + 1);
  out.sorted = ws.get_t<uint32_t>(tag + ".sorted", padded);
  BG_CUDA(cudaMemsetAsync(counts, 0, (nkeys + 1) * sizeof(uint32_t), st));
  if (rounds) BG_CUDA(cudaMemsetAsync(out.sorted, 0xff, padded * sizeof(uint32_t), st));  // null entries
  {
    KernelTimer kt(ctx, "msm_digits", st);
    if (by_rank)
      k_digits_rank<<<rgrid, 256, 0, st>>>(d_scalars, n, W, kDigitBatch, key_stride, counts, cursor, ctx.d_status);
    else
      k_digits_hist<<<ceil_div(n, 256), 256, 0, st>>>(d_scalars, n, c, W, key_stride, counts, ctx.d_status);
    BG_CHECK_LAUNCH();
  }
  exclusive_scan(ws, tag, counts, out.offsets, nkeys + 1, st, 0, (1u << rounds) - 1u);
  if (!by_rank)
    BG_CUDA(cudaMemcpyAsync(cursor, out.offsets, (nkeys + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  {
    KernelTimer kt(ctx, "msm_scatter", st);
    if (by_rank)
      k_scatter_rank<<<rgrid, 256, 0, st>>>(d_scalars, n, W, kDigitBatch, key_stride, idx_stride, out.offsets, cursor,
                                            out.sorted);
    else
      k_scatter<<<ceil_div(n, 256), 256, 0, st>>>(d_scalars, n, c, W, key_stride, idx_stride, cursor, out.sorted);
    BG_CHECK_LAUNCH();
  }
  out.done = ctx.event(tag + ".sorted");
  BG_CUDA(cudaEventRecord(out.done, st));
}

template <class F>
void msm_accumulate(Ctx& ctx, cudaStream_t st, const std::string& tag, const uint32_t* d_points, const MsmSort& so,
                    MsmPlan& plan, cudaStream_t st_reduce, const MsmTable* table) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int PW = 4 * FW;
  if (so.n == 0) {
    plan.W = 0;
    return;
  }
  if (table && (table->n != so.n || table->c != so.c || so.sets != 1))
    throw Error(BG_E_ARG, "msm: window table and bucket order disagree");
  if (!table && so.sets == 1) throw Error(BG_E_ARG, "msm: a shared bucket set needs a window table");
  msm_init_kernels();
  if (table) d_points = table->d;
  plan.c = so.c;
  plan.W = so.sets;
  Workspace& ws = ctx.ws;
  if (so.done) BG_CUDA(cudaStreamWaitEvent(st, so.done, 0));
  Ctx* prof = (ctx.profile || ctx.timeline) ? &ctx : nullptr;

  // Batch-affine pair rounds, as many as the sort padded its buckets for, halve every bucket in
  // affine coordinates first (msm_pairs.cuh); the XYZZ accumulation, the heavy pass and the
  // reduction then read the last level's points directly, with its offsets.  Accumulations queued
  // on one stream share the levels' memory.
  const uint32_t* acc_points = d_points;
  const uint32_t* acc_sorted = so.sorted;
  const uint32_t* acc_offsets = so.offsets;
  size_t acc_entries = so.max_entries;
  const int rounds = so.rounds;
  if (rounds > 0) {
    constexpr int NT = kPairThreads<F>;
    const double pslots = pair_slots<F>();
    const size_t me = so.max_entries;
    const uint32_t nk = (uint32_t)so.nkeys;
    const std::string lv = plan.own_stream ? tag : "acc";
    uint32_t* lvl[2] = {ws.get_t<uint32_t>(lv + ".pairs0", (me >> 1) * 2 * FW), nullptr};
    if (rounds > 1) lvl[1] = ws.get_t<uint32_t>(lv + ".pairs1", (me >> 2) * 2 * FW);
    uint32_t* fin = ws.get_t<uint32_t>(tag + ".pair_offsets", so.nkeys + 1);
    KernelTimer kt(ctx, FW == 8 ? "msm_pair_g1" : "msm_pair_g2", st);
    for (int r = 0; r < rounds; r++) {
      const double outs = (double)(me >> (r + 1));
      const double waves = std::max(1.0, std::ceil(outs / (pslots * kPairPer)));
      const uint32_t per = (uint32_t)std::max(1.0, std::ceil(outs / (waves * pslots)));
      const unsigned grid = ceil_div(ceil_div((size_t)outs, per), NT);
      if (!grid) continue;
      if (r == 0)
        k_pair_round<F, true><<<grid, NT, pair_smem_bytes<F>(), st>>>(d_points, so.sorted, so.offsets, nk, 0, per,
                                                                      lvl[0], rounds, fin);
      else
        k_pair_round<F, false><<<grid, NT, pair_smem_bytes<F>(), st>>>(lvl[(r - 1) & 1], nullptr, so.offsets, nk, r,
                                                                       per, lvl[r & 1], rounds, nullptr);
      BG_CHECK_LAUNCH();
    }
    acc_points = lvl[(rounds - 1) & 1];
    acc_sorted = nullptr;
    acc_offsets = fin;
    acc_entries = me >> rounds;
  }
  plan.entries = acc_entries;
  uint32_t* buckets = ws.get_t<uint32_t>(tag + ".buckets", so.nkeys * PW);
  const BucketScratch bs = bucket_scratch<F>(acc_entries, so.nkeys, plan.in_proof, [&](const char* name, size_t words) {
    return ws.get_t<uint32_t>(tag + ".slice_" + name, words);
  });
  bucket_accumulate<F>(prof, st, acc_points, acc_offsets, acc_sorted, (uint32_t)so.nkeys, acc_entries, buckets, bs);

  cudaStream_t rs = st;
  if (st_reduce && st_reduce != st) {
    // the latency-bound heavy-bucket pass and reduction run on their own stream and overlap
    // whatever `st` does next (the next MSM's accumulation)
    cudaEvent_t ev = ctx.event(tag + ".acc_done");
    BG_CUDA(cudaEventRecord(ev, st));
    BG_CUDA(cudaStreamWaitEvent(st_reduce, ev, 0));
    rs = st_reduce;
  }
  bucket_heavy<F>(prof, rs, acc_offsets, buckets, bs, plan.in_proof);

  // A reduction hidden under a later accumulation runs in CTAs of 128 threads: 256 leave no room for
  // an accumulation CTA on their SM for their whole (latency-bound) life, and smaller ones spread
  // over more SMs (a mixed batch of 16 proofs 17.0 ms with 32 and 64 allowed, 16.7 without).
  ReduceShape rsh =
      reduce_shape<F>(so.nb, so.sets, acc_entries, bs.K, ctx.sm_count, plan.latency_critical ? 32u : 128u,
                      plan.latency_critical ? 256u : 128u);
  // A reduction meant to run under later accumulations that the latency model says outlasts them
  // (SquareChain(2^14)'s G2 MSM: 0.53 ms, 0.29 ms of accumulations left) is critical after all and
  // takes the critical shapes: 2^14 proofs 1.28 ms where it had to outlast them twice over, 1.09 ms
  // so and with half the time, other sizes level.  Latency of one dependent addition at a
  // reduction's occupancy: about 11 us (G1), 29 us (G2).
  bool critical = plan.latency_critical;
  const double add_us = FW == 16 ? 29.0 : 11.0;
  if (!critical && plan.hidden_us > 0 && rsh.cost * add_us > plan.hidden_us) critical = true;
  // A hidden G1 reduction takes the shape with the least work per bucket (longer chains, fewer tree
  // additions per bucket) whose modelled latency stays within a small part of its budget, which the
  // accumulations beside it stretch: a quarter / 6% / 3% of it measured 2^17 3.78 / 3.74 / 3.73 ms,
  // 2^18 6.60 / 6.55 / 6.53, 2^20 20.27 / 20.25 / 20.29.  G2 keeps the shortest chain (at 2^20 the
  // least work crowded the last accumulations).
  if (!critical && plan.hidden_us > 0 && FW == 8) {
    const ReduceShape wsh =
        reduce_shape_work<F>(so.nb, so.sets, acc_entries, bs.K, ctx.sm_count, 128u, 0.06 * plan.hidden_us / add_us);
    if (wsh.RT) rsh = wsh;
  }
  if (critical && !plan.latency_critical)
    rsh = reduce_shape<F>(so.nb, so.sets, acc_entries, bs.K, ctx.sm_count, 32u, 256u);
  // a reduction that ends a critical path may take the cooperative form (8 lanes per addition)
  if (critical && ctx.coop_reduce != 0) {
    const ReduceShape csh = reduce_shape_coop<F>(so.nb, so.sets, acc_entries, bs.K, ctx.sm_count);
    if (csh.RT && (ctx.coop_reduce > 0 || csh.cost < rsh.cost)) rsh = csh;
  }
  uint32_t* parts = ws.get_t<uint32_t>(tag + ".parts", so.sets * reduce_part_points(rsh) * PW);
  const size_t points = reduce_points(rsh);  // per bucket set
  {
    KernelTimer kt(ctx, FW == 8 ? "msm_reduce_g1" : "msm_reduce_g2", rs);
    plan.d_window_sums = window_reduce<F>(rs, rsh, acc_offsets, buckets, bs, so.nb, so.sets, parts);
  }
  plan.fetch_stream = rs;
  plan.bits = (int)points - 1;
  plan.shift = log2_of(rsh.M);
  plan.host_window_sums = ctx.host_cache.get_t<uint32_t>(tag + ".window_sums", so.sets * points * PW);
}

int msm_rounds_model(size_t n, int c, bool shared_set, bool g2) {
  const size_t W = 254 / c + 1;
  return pair_rounds_model(n, n * W, (shared_set ? 1 : W) << (c - 1), g2, shared_set);
}
int msm_rounds(const Ctx& ctx, size_t n, int c, bool shared_set, bool g2) {
  return ctx.pair_rounds_override >= 0 ? ctx.pair_rounds_override : msm_rounds_model(n, c, shared_set, g2);
}

// ---- the device bytes of the buffers above, for a proof's reservation.  Bounds where a choice depends on
// the GPU: slices at three quarters of the model's K (whole_wave_slices), the most parts a reduction's
// shape can have.
size_t msm_sort_bytes(size_t n, int c, bool shared_set, int rounds) {
  const SortSizes z = sort_sizes(n, c, shared_set, rounds);
  const size_t tiles = (z.nkeys + 1) / kScanTile + 1;
  const size_t keyed = (sort_by_rank(n) ? 2 : 3) * (z.nkeys + 1);  // counts, offsets, cursors
  return 4 * (keyed + z.padded + 2 * tiles + 2 * (tiles / kScanTile + 1));
}
size_t msm_rank_bytes(size_t n, int c) { return sort_by_rank(n) ? 4 * n * (size_t)(254 / c + 1) : 0; }
void msm_level_bytes(size_t n, int c, bool shared_set, int rounds, bool g2, size_t out[2]) {
  const SortSizes z = sort_sizes(n, c, shared_set, rounds);
  const size_t point = g2 ? 128 : 64;
  out[0] = z.rounds > 0 ? (z.padded >> 1) * point : 0;
  out[1] = z.rounds > 1 ? (z.padded >> 2) * point : 0;
}
size_t msm_bucket_bytes(size_t n, int c, bool shared_set, int rounds, bool g2) {
  const SortSizes z = sort_sizes(n, c, shared_set, rounds);
  const size_t entries = z.padded >> z.rounds, nb = size_t(1) << (c - 1), point = g2 ? 256 : 128;
  const uint32_t K = g2 ? slice_entries<Fq2>(entries, z.nkeys) : slice_entries<Fq>(entries, z.nkeys);
  const size_t slices = 4 * entries / (3 * K) + 1;
  size_t parts = 0;  // points per bucket set
  for (uint32_t RT = 4; RT <= 256 && RT <= std::max<size_t>(nb, 4); RT <<= 1) {
    ReduceShape r{RT, 1, (uint32_t)std::max<size_t>(1, nb / RT)};
    // fewer than 32 threads, or a scan, in the cooperative form alone
    if (RT < 32 && r.J > 1) r.J = std::min<uint32_t>(r.J, kCoopMaxParts / z.sets + 1);
    parts = std::max(parts, reduce_part_points(r));
  }
  return point * (z.nkeys + 2 * slices + z.sets * parts) + 4 * (slices / 4 + 2) +
         (z.rounds ? 4 * (z.nkeys + 1) : 0);
}

template <class F>
void msm_launch(Ctx& ctx, cudaStream_t st, const std::string& tag, const uint32_t* d_points,
                const uint32_t* d_scalars, size_t n, MsmPlan& plan, cudaStream_t st_reduce, const MsmTable* table) {
  if (table && table->n != n) throw Error(BG_E_ARG, "msm: window table built for another size");
  const int c = table ? table->c : (plan.c > 0 ? plan.c : msm_pick_c(n, FieldWords<F>::value == 16));
  MsmSort so;
  msm_sort(ctx, st, tag, d_scalars, n, c, table != nullptr,
           msm_rounds(ctx, n, c, table != nullptr, FieldWords<F>::value == 16), so);
  so.done = nullptr;  // same stream: already ordered
  msm_accumulate<F>(ctx, st, tag, d_points, so, plan, st_reduce, table);
}

int msm_pair_rounds_entries(size_t max_entries, size_t nkeys, bool g2) {
  return pair_rounds_model(0, max_entries, nkeys, g2, false);
}

int msm_pair_rounds(size_t n, bool g2) {
  if (n == 0) return 0;
  const int c = msm_pick_c(n, g2);
  const size_t W = 254 / c + 1;
  return pair_rounds_model(n, n * W, W << (c - 1), g2, false);
}

int msm_pick_c_proof(size_t n, bool g2) {
  if (const int t = tuned(kTuneProofSets, n, g2)) return t;
  return msm_pick_c(n, g2);
}

int msm_pick_c_table(size_t n, bool g2) {
  // one shared bucket set: wider windows (fewer additions) at the price of 2^(c-1) buckets
  if (const int t = tuned(kTuneTables, n, g2)) return t;
  const int lg = floor_log2(n);
  // the smallest proofs are bound by the chains of their reductions, whose length is the entries per
  // bucket: SquareChain(2^5) 0.388 ms at 6 bits, 0.330 at 8; 2^6 0.427 at 6, 0.344 at 9; 2^7 0.520 at 6,
  // 0.358 at 10 and 11; 2^8 0.377 at 10, 0.367 at 11; 2^9 0.424 at 10, 0.397 at 11; below 2^5 level
  if (lg <= 9) return std::min(11, std::max(7, lg + 3));
  return std::min(18, std::max(6, lg - 1));
}

template <class F>
void msm_build_table(cudaStream_t st, const uint32_t* d_points, size_t n, MsmTable& t, int c) {
  constexpr int PW = 2 * FieldWords<F>::value;
  if (c != 0 && (c < 2 || c > 22)) throw Error(BG_E_ARG, "msm table: window width out of range");
  t.n = n;
  t.c = c ? c : msm_pick_c_table(n, FieldWords<F>::value == 16);
  t.W = 254 / t.c + 1;
  if (n == 0) return;
  if (n * (size_t)t.W >= 0x80000000ull) throw Error(BG_E_ARG, "msm table: n x windows must be below 2^31");
  void* p = nullptr;
  const size_t bytes = n * (size_t)t.W * PW * sizeof(uint32_t);
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error(BG_E_OOM, "window table allocation of " + std::to_string(bytes) + " bytes failed");
  }
  t.d = static_cast<uint32_t*>(p);
  k_build_table<F><<<ceil_div(n, 128), 128, 0, st>>>(d_points, n, t.c, t.W, t.d);
  BG_CHECK_LAUNCH();
}

template void msm_build_table<Fq>(cudaStream_t, const uint32_t*, size_t, MsmTable&, int);
template void msm_build_table<Fq2>(cudaStream_t, const uint32_t*, size_t, MsmTable&, int);

template <class F>
void msm_fetch(Ctx& ctx, cudaStream_t st, MsmPlan& plan) {
  constexpr int PW = 4 * FieldWords<F>::value;
  if (plan.W == 0) return;
  if (plan.fetch_stream) st = plan.fetch_stream;
  BG_CUDA(cudaMemcpyAsync(plan.host_window_sums, plan.d_window_sums,
                          (size_t)plan.W * (plan.bits + 1) * PW * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  ctx.d2h_bytes += (uint64_t)plan.W * (plan.bits + 1) * PW * sizeof(uint32_t);
}

// Window w = T + 2^shift sum_b 2^b U_b, total = sum_w 2^(o_w) window_w: one Horner over the bit
// positions.  Positions from the window's width up hold no digit (a last bucket set of narrower
// windows leaves them at infinity).
template <class H>
bgh::Xyzz<H> msm_sum(const MsmPlan& plan) {
  constexpr int PW = 4 * H::WORDS;
  auto point = [&](int w, int i) {
    return bgh::xyzz_from_words32<H>(plan.host_window_sums + ((size_t)w * (plan.bits + 1) + i) * PW);
  };
  // acc 2^(positions) + the window's points below its `positions` lowest bits
  auto horner = [&](bgh::Jac<H> acc, int w, int positions) {
    for (int d = positions - 1; d >= 0; d--) {
      acc = bgh::jac_dbl(acc);
      if (d >= plan.shift && d < plan.shift + plan.bits) acc = bgh::jac_add(acc, point(w, 1 + d - plan.shift));
    }
    return bgh::jac_add(acc, point(w, 0));
  };
  const int top = plan.shift + plan.bits;
  bgh::Jac<H> acc = bgh::jac_inf<H>();
  // The windows' own sums run on the host pool where they take longer than its wake-up.
  if (plan.W >= 4 && plan.W * plan.bits >= kHostPoolPoints) {
    std::vector<bgh::Xyzz<H>> win(plan.W);
    HostPool::get().parallel_for(plan.W, [&](int w) {
      win[w] = bgh::xyzz_from_jac(horner(bgh::jac_inf<H>(), w, std::min(top, window_width(w, plan.W))));
    });
    for (int w = plan.W - 1; w >= 0; w--) {
      for (int d = window_width(w, plan.W); d > 0; d--) acc = bgh::jac_dbl(acc);
      acc = bgh::jac_add(acc, win[w]);
    }
  } else {
    for (int w = plan.W - 1; w >= 0; w--)
      acc = horner(acc, w, w == plan.W - 1 ? std::min(top, window_width(w, plan.W)) : window_width(w, plan.W));
  }
  return bgh::xyzz_from_jac(acc);
}

template <class F>
void msm_finish(const MsmPlan& plan, uint32_t* out_affine_words32) {
  typedef typename HostField<F>::T H;
  bgh::aff_to_words32<H>(out_affine_words32, bgh::xyzz_to_affine(msm_sum<H>(plan)));
}

// Kernel attributes (the opt-in to large dynamic shared memory) apply to the device that is
// current when they are set, so they are set once per device; batch lanes and server threads
// may get here at the same time, hence the per-device once flags.
constexpr int kInitMaxDevices = 64;
void msm_init_kernels() {
  static std::once_flag once[kInitMaxDevices];
  int dev = 0;
  BG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kInitMaxDevices) throw Error(BG_E_ARG, "msm: device index out of range");
  std::call_once(once[dev], [] {
    auto smem = [](auto* k, size_t bytes) {
      BG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    };
    smem(k_pair_round<Fq, true>, pair_smem_bytes<Fq>());
    smem(k_pair_round<Fq, false>, pair_smem_bytes<Fq>());
    smem(k_pair_round<Fq2, true>, pair_smem_bytes<Fq2>());
    smem(k_pair_round<Fq2, false>, pair_smem_bytes<Fq2>());
    smem(k_window_reduce<Fq>, reduce_sm_bytes<Fq>(256, 2));
    smem(k_window_reduce<Fq2>, reduce_sm_bytes<Fq2>(256, 2));
  });
}

template void msm_launch<Fq>(Ctx&, cudaStream_t, const std::string&, const uint32_t*, const uint32_t*, size_t,
                             MsmPlan&, cudaStream_t, const MsmTable*);
template void msm_accumulate<Fq>(Ctx&, cudaStream_t, const std::string&, const uint32_t*, const MsmSort&, MsmPlan&,
                                 cudaStream_t, const MsmTable*);
template void msm_accumulate<Fq2>(Ctx&, cudaStream_t, const std::string&, const uint32_t*, const MsmSort&, MsmPlan&,
                                  cudaStream_t, const MsmTable*);
template void msm_launch<Fq2>(Ctx&, cudaStream_t, const std::string&, const uint32_t*, const uint32_t*, size_t,
                              MsmPlan&, cudaStream_t, const MsmTable*);
template void msm_fetch<Fq>(Ctx&, cudaStream_t, MsmPlan&);
template void msm_fetch<Fq2>(Ctx&, cudaStream_t, MsmPlan&);
template bgh::Xyzz<bgh::FqOps> msm_sum<bgh::FqOps>(const MsmPlan&);
template bgh::Xyzz<bgh::Fq2Ops> msm_sum<bgh::Fq2Ops>(const MsmPlan&);
template void msm_finish<Fq>(const MsmPlan&, uint32_t*);
template void msm_finish<Fq2>(const MsmPlan&, uint32_t*);

}  // namespace bg

// ---------------------------------------------------------------- allocation-free G1 MSM
// bg_msm_g1_noalloc serves callers that must not allocate device memory at all: a host
// program that has handed the whole GPU to its own memory pool and forbids any further
// cudaMalloc, or a latency-critical loop in which the device-wide synchronisation that
// cudaMalloc/cudaFree imply is not acceptable.  It runs the same kernels as the other MSM
// entry points, but every scratch buffer is carved out of one fixed array that lives in the
// library's own device image, so the call allocates nothing (no cudaMalloc, cudaFree,
// pinned-host allocation or context).  The price is a hard size limit and shared state:
//   * at most kNoAllocMaxPoints points (larger requests fail with BG_E_ARG);
//   * every GPU that loads the library holds the kNoAllocScratchBytes array until the process
//     exits;
//   * all calls use the same array, which keeps the previous call's contents (the bucket
//     counters are cleared at the start of each call); calls that overlap on the GPU race, so
//     this entry point serialises calls made from one process and returns only when its work
//     is complete;
//   * the first call on a device looks up the array's device address on that device (the
//     device current at the call);
//   * every call ends with a synchronisation of its stream and copies to pageable host memory,
//     so it must not be called on a stream that is being captured.
namespace bg {
namespace {

constexpr size_t kNoAllocMaxPoints = size_t(1) << 14;
constexpr size_t kNoAllocScratchBytes = size_t(9) << 20;  // the worst case up to 2^14 points needs 6.6 MiB
constexpr size_t kNoAllocHostWords = 16384;               // window points copied back for the Horner
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocScratchBytes];
static uint32_t g_noalloc_host_parts[kNoAllocHostWords];
static uint32_t g_noalloc_host_status;
static void* g_noalloc_dev_ptr[kNoAllocMaxDevices];
static std::mutex g_noalloc_mu;

// device address of the scratch array on the current device (looked up once per device)
uint8_t* noalloc_scratch() {
  int dev = 0;
  BG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) throw Error(BG_E_ARG, "bg_msm_g1_noalloc: device index out of range");
  if (!g_noalloc_dev_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      throw Error(BG_E_DEVICE, std::string("bg_msm_g1_noalloc: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
    g_noalloc_dev_ptr[dev] = p;
  }
  return static_cast<uint8_t*>(g_noalloc_dev_ptr[dev]);
}

void msm_g1_noalloc(const uint32_t* d_points, const uint32_t* d_scalars, size_t n, cudaStream_t st,
                    uint32_t* out_aff32) {
  constexpr int PW = 32;  // packed words of a G1 XYZZ point
  if (n == 0) {
    memset(out_aff32, 0, 16 * sizeof(uint32_t));
    return;
  }
  if (n > kNoAllocMaxPoints)
    throw Error(BG_E_ARG, "bg_msm_g1_noalloc: " + std::to_string(n) + " points exceed the fixed maximum of " +
                              std::to_string(kNoAllocMaxPoints));
  uint8_t* base = noalloc_scratch();
  const int c = msm_pick_c(n);
  const int W = 254 / c + 1;
  const uint32_t nb = 1u << (c - 1);
  const size_t nkeys = (size_t)W * nb;
  const size_t max_entries = n * (size_t)W;
  int dev = 0, sms = 0;
  BG_CUDA(cudaGetDevice(&dev));
  BG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  msm_init_kernels();
  const ReduceShape rsh = reduce_shape<Fq>(nb, W, max_entries, 32, sms, 32u, 256u);
  const unsigned tiles = ceil_div(nkeys + 1, kScanTile);

  size_t off = 0;
  auto carve = [&](size_t words) {
    uint32_t* p = reinterpret_cast<uint32_t*>(base + off);
    off += (words * sizeof(uint32_t) + 255) & ~size_t(255);
    return p;
  };
  uint32_t* status = carve(1);
  uint32_t* counts = carve(nkeys + 1);
  uint32_t* offsets = carve(nkeys + 1);
  uint32_t* cursor = carve(nkeys + 1);
  uint32_t* tile_sums = carve(tiles);
  uint32_t* tile_offs = carve(tiles);
  uint32_t* sorted = carve(max_entries);
  uint32_t* buckets = carve(nkeys * PW);
  // 32-entry slices: the fixed array is sized for them
  const BucketScratch bs =
      bucket_scratch<Fq>(max_entries, nkeys, false, [&](const char*, size_t words) { return carve(words); }, 32);
  uint32_t* parts = carve(W * reduce_part_points(rsh) * PW);
  const size_t host_words = W * reduce_points(rsh) * PW;
  if (off > kNoAllocScratchBytes || host_words > kNoAllocHostWords || tiles > (unsigned)kScanTile)
    throw Error(BG_E_ARG, "bg_msm_g1_noalloc: scratch layout exceeds the fixed array");

  // what must start at zero: the status word and the bucket counters
  BG_CUDA(cudaMemsetAsync(status, 0, sizeof(uint32_t), st));
  BG_CUDA(cudaMemsetAsync(counts, 0, (nkeys + 1) * sizeof(uint32_t), st));
  k_digits_hist<<<ceil_div(n, 256), 256, 0, st>>>(d_scalars, n, c, W, nb, counts, status);
  BG_CHECK_LAUNCH();
  if (tiles == 1) {
    k_scan_tile<<<1, kScanThreads, 0, st>>>(counts, offsets, nullptr, nkeys + 1, 0);
    BG_CHECK_LAUNCH();
  } else {
    k_scan_tile<<<tiles, kScanThreads, 0, st>>>(counts, offsets, tile_sums, nkeys + 1, 0);
    BG_CHECK_LAUNCH();
    k_scan_tile<<<1, kScanThreads, 0, st>>>(tile_sums, tile_offs, nullptr, tiles, 0);
    BG_CHECK_LAUNCH();
    k_scan_add<<<ceil_div(nkeys + 1, 256), 256, 0, st>>>(offsets, tile_offs, nkeys + 1);
    BG_CHECK_LAUNCH();
  }
  BG_CUDA(cudaMemcpyAsync(cursor, offsets, (nkeys + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  k_scatter<<<ceil_div(n, 256), 256, 0, st>>>(d_scalars, n, c, W, nb, 0, cursor, sorted);
  BG_CHECK_LAUNCH();
  bucket_accumulate<Fq>(nullptr, st, d_points, offsets, sorted, (uint32_t)nkeys, max_entries, buckets, bs);
  bucket_heavy<Fq>(nullptr, st, offsets, buckets, bs, false);
  const uint32_t* sums = window_reduce<Fq>(st, rsh, offsets, buckets, bs, nb, W, parts);
  BG_CUDA(cudaMemcpyAsync(g_noalloc_host_parts, sums, host_words * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  BG_CUDA(cudaMemcpyAsync(&g_noalloc_host_status, status, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  BG_CUDA(cudaStreamSynchronize(st));
  if (g_noalloc_host_status & BG_DSTATUS_SCALAR_RANGE)
    throw Error(BG_E_ARG, "bg_msm_g1_noalloc: a scalar is not below 2^254 (not a canonical Fr)");
  MsmPlan plan;
  plan.c = c;
  plan.W = W;
  plan.bits = (int)reduce_points(rsh) - 1;
  plan.shift = log2_of(rsh.M);
  plan.host_window_sums = g_noalloc_host_parts;
  msm_finish<Fq>(plan, out_aff32);
}

}  // namespace
}  // namespace bg

extern "C" int bg_msm_g1_noalloc(const uint32_t* d_points, const uint32_t* d_scalars, size_t n, void* stream,
                                 uint32_t* out_aff32) {
  if (!out_aff32 || (n && (!d_points || !d_scalars))) {
    bg::set_noctx_error("bg_msm_g1_noalloc: invalid argument (a null pointer)");
    return BG_E_ARG;
  }
  // points and scalars are read in 16-byte vectors: refuse a pointer off that boundary here
  // rather than let the device fault on it
  if ((reinterpret_cast<uintptr_t>(d_points) | reinterpret_cast<uintptr_t>(d_scalars)) & 15u) {
    bg::set_noctx_error("bg_msm_g1_noalloc: invalid argument (a device pointer not 16-byte aligned)");
    return BG_E_ARG;
  }
  std::lock_guard<std::mutex> lock(bg::g_noalloc_mu);
  try {
    bg::msm_g1_noalloc(d_points, d_scalars, n, static_cast<cudaStream_t>(stream), out_aff32);
    return BG_OK;
  } catch (const bg::Error& e) {
    bg::set_noctx_error(e.what());
    if (e.status == BG_E_DEVICE) cudaGetLastError();
    return e.status;
  } catch (const std::bad_alloc&) {
    bg::set_noctx_error("bg_msm_g1_noalloc: host allocation failed");
    return BG_E_OOM;
  } catch (const std::exception& e) {
    bg::set_noctx_error(std::string("bg_msm_g1_noalloc: ") + e.what());
    return BG_E_DEVICE;
  }
}
