// Batch-affine pair rounds of the MSM bucket accumulation (included by msm.cu).
//
// The bucket phase of Msm.g1 / Msm.g2 (bend2/src/msm.bend:120-158 adds every point of a
// window into its bucket with a Jacobian mixed addition) may be preceded by rounds that halve
// every bucket: a round adds the points of each bucket in pairs, in affine coordinates, and
// writes the sums as the bucket's points for the next round.  The additions of a round are
// independent, so they share their field inversions: each thread multiplies its denominators
// into a running product, the CTA multiplies the threads' products in a tree in shared memory up to
// 32 nodes, a warp inverts those side by side (division steps, inv_divsteps), and the tree and the
// running products are walked back to give every addition 1 / d (Montgomery's simultaneous inversion).  An
// addition then costs 5 products and a square (3 of them for the shared inversion) against
// madd-2008-s's 8 products and 2 squares; the XYZZ accumulation that follows adds what the
// rounds left, and the window reduction is unchanged.
//
// Layout.  The sort pads every bucket to a multiple of 2^L entries (L its number of rounds) with
// null entries, so pair j of a round is the level's points 2 j and 2 j + 1, always of one bucket:
// no round looks a bucket up, levels r >= 1 are read and written in order, and level r's bucket
// offsets are the sort's shifted right by r.  Round 0 reads its points through the sort's entries
// (index | sign << 31) from the MSM's point set or window table.  A missing point (a null entry,
// a sum at infinity) is (0, 0) on every level, as an input at infinity is.
//
// Positions are dealt to the threads of a CTA in turn, so that neighbouring lanes read
// neighbouring entries, and every operand is staged in shared memory by cp.async a few positions
// ahead: the gathers of round 0 are 32 and 64-byte accesses all over the point set.

// a null entry of a padded bucket
constexpr uint32_t kNullEntry = 0xffffffffu;

// CTA size; four CTAs per SM in G1 (at most 122 registers; five at 96 measured 1.57 -> 1.95 ms for
// G1 MSM 2^20's two rounds), two in G2
template <class F>
constexpr int kPairThreads = 128;
// stages of the operand rings (power of two): x coordinates ahead in the forward pass, whole
// points and a running product in the backward pass
constexpr int kPairFwd = 4;
constexpr int kPairBwd = 2;

// 16-byte chunks per field element
template <class F>
constexpr int kPairCh = FieldWords<F>::value / 4;
// shared memory: the ring (the larger pass's), under which the product tree lies between the passes
template <class F>
constexpr size_t pair_ring_chunks() {
  constexpr int fwd = kPairFwd * 2 * kPairCh<F>, bwd = kPairBwd * 5 * kPairCh<F>;
  return (size_t)(fwd > bwd ? fwd : bwd) * kPairThreads<F>;
}
template <class F>
constexpr size_t pair_smem_bytes() {
  const size_t tree = 2 * (size_t)kPairThreads<F> * FieldWords<F>::value * 4;
  return pair_ring_chunks<F>() * 16 > tree ? pair_ring_chunks<F>() * 16 : tree;
}

template <class F>
BG_DEV F elem_of_chunks(const uint4* c, int stride) {
  if constexpr (FieldWords<F>::value == 16) {
    return {fp_of(c[0], c[stride]), fp_of(c[2 * stride], c[3 * stride])};
  } else {
    return fp_of(c[0], c[stride]);
  }
}
// 16 bytes global -> shared, or zeros
BG_DEV void cp_async16_or_zero(void* smem, const void* gmem, bool take) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  const int bytes = take ? 16 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
template <int N>
BG_DEV void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// One round: `per_thread` positions per thread.  dst's x field of each position first holds the
// thread's running product up to it (read back by the backward pass) and is then overwritten by
// the sum.  Round 0 also writes the offsets of the accumulation's level, offsets >> rounds.
template <class F, bool kFirst>
__global__ void __launch_bounds__(kPairThreads<F>, FieldWords<F>::value == 8 ? 4 : 2)
    k_pair_round(const uint32_t* __restrict__ src, const uint32_t* __restrict__ sorted,
                 const uint32_t* __restrict__ offsets, uint32_t nkeys, int level, uint32_t per_thread,
                 uint32_t* __restrict__ dst, int rounds, uint32_t* __restrict__ final_offsets) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int PW = 2 * FW;
  constexpr int NT = kPairThreads<F>;
  constexpr int CH = kPairCh<F>;
  constexpr int FD = kPairFwd;
  extern __shared__ __align__(16) uint32_t sm[];
  uint4* const ring = reinterpret_cast<uint4*>(sm) + threadIdx.x;  // chunk c of a stage at ring[c * NT]
  uint32_t* const tree = sm;
  const uint32_t tid = threadIdx.x;
  if (final_offsets) {
    for (size_t g = (size_t)blockIdx.x * NT + tid; g <= nkeys; g += (size_t)gridDim.x * NT)
      final_offsets[g] = offsets[g] >> rounds;
  }
  const uint32_t total = offsets[nkeys] >> (level + 1);
  const uint64_t base = (uint64_t)blockIdx.x * NT * per_thread + tid;
  if ((uint64_t)blockIdx.x * NT * per_thread >= total) return;
  // positions base, base + NT, ... below total
  const uint32_t cnt =
      base >= total ? 0u : (uint32_t)min((uint64_t)per_thread, (total - base + NT - 1) / (uint64_t)NT);

  auto entries = [&](uint32_t t) -> uint2 {
    if constexpr (kFirst) return *reinterpret_cast<const uint2*>(sorted + 2 * (base + (uint64_t)t * NT));
    else return make_uint2(0u, 0u);
  };
  auto stage_elem = [&](uint4* slot, const uint32_t* g, bool take) {
#pragma unroll
    for (int c = 0; c < CH; c++) cp_async16_or_zero(slot + c * NT, g + 4 * c, take);
  };
  // address of input point `k` (0 or 1) of position t
  auto point = [&](uint32_t t, uint2 e, int k) -> const uint32_t* {
    if constexpr (kFirst) {
      const uint32_t c = k ? e.y : e.x;
      return src + (size_t)(c == kNullEntry ? 0u : c & 0x7fffffffu) * PW;
    } else {
      return src + (2 * (size_t)(base + (uint64_t)t * NT) + k) * PW;
    }
  };

  // ---- forward: the running product of the denominators x_Q - x_P (1 where there is no addition)
  F acc = field_one<F>();
  {
    auto stage = [&](uint32_t t, uint2 e) {
      if (t < cnt) {
        uint4* s = ring + (size_t)(t & (FD - 1)) * 2 * CH * NT;
        stage_elem(s, point(t, e, 0), !kFirst || e.x != kNullEntry);
        stage_elem(s + CH * NT, point(t, e, 1), !kFirst || e.y != kNullEntry);
      }
      cp_async_commit();
    };
#pragma unroll
    for (int t = 0; t < FD - 1; t++) stage(t, (uint32_t)t < cnt ? entries(t) : make_uint2(0u, 0u));
    uint2 e = FD - 1 < cnt ? entries(FD - 1) : make_uint2(0u, 0u);
    for (uint32_t t = 0; t < cnt; t++) {
      stage(t + FD - 1, e);
      if (t + FD < cnt) e = entries(t + FD);
      cp_async_wait<FD - 1>();
      const uint4* s = ring + (size_t)(t & (FD - 1)) * 2 * CH * NT;
      const F xp = elem_of_chunks<F>(s, NT), xq = elem_of_chunks<F>(s + CH * NT, NT);
      F d = sub(xq, xp);
      if (is_zero(d)) {
        const uint2 en = entries(t);
        F yp = field_zero<F>(), yq = field_zero<F>();
        if (!kFirst || en.x != kNullEntry) load_elem(yp, point(t, en, 0) + FW);
        if (!kFirst || en.y != kNullEntry) load_elem(yq, point(t, en, 1) + FW);
        if (kFirst && (en.x >> 31)) yp = neg(yp);
        if (kFirst && (en.y >> 31)) yq = neg(yq);
        d = pair_equal_x(yp, yq);
      }
      acc = imul(acc, d);
      store_elem(dst + (base + (uint64_t)t * NT) * PW, acc);
    }
    cp_async_wait<0>();
  }

  // ---- the CTA's product tree (leaves NT..2NT-1, node i = node 2i * node 2i+1) up to the 32
  // nodes of one level, which a warp inverts side by side, and the tree walked back: leaf t ends
  // as 1 / (thread t's product)
  __syncthreads();
  store_elem(tree + (size_t)(NT + tid) * FW, acc);
  __syncthreads();
  for (uint32_t half = NT / 2; half >= 32; half >>= 1) {
    if (tid < half) {
      const uint32_t i = half + tid;
      F a, b;
      load_elem(a, tree + (size_t)(2 * i) * FW);
      load_elem(b, tree + (size_t)(2 * i + 1) * FW);
      store_elem(tree + (size_t)i * FW, fmul(a, b));
    }
    __syncthreads();
  }
  if (tid < 32) {
    F root;
    load_elem(root, tree + (size_t)(32 + tid) * FW);
    store_elem(tree + (size_t)(32 + tid) * FW, field_inv_fast(root));
  }
  __syncthreads();
  for (uint32_t half = 32; half < NT; half <<= 1) {
    if (tid < half) {
      const uint32_t i = half + tid;
      F iv, a, b;
      load_elem(iv, tree + (size_t)i * FW);
      load_elem(a, tree + (size_t)(2 * i) * FW);
      load_elem(b, tree + (size_t)(2 * i + 1) * FW);
      store_elem(tree + (size_t)(2 * i) * FW, fmul(iv, b));
      store_elem(tree + (size_t)(2 * i + 1) * FW, fmul(iv, a));
    }
    __syncthreads();
  }
  F inv;
  load_elem(inv, tree + (size_t)(NT + tid) * FW);
  __syncthreads();
  if (!cnt) return;

  // ---- backward: 1 / d_t = inv * (product up to t - 1), inv *= d_t, and the sums.  A slot holds
  // x_P, y_P, x_Q, y_Q and the product before the position.
  auto stage = [&](int64_t t, uint2 e) {
    if (t >= 0) {
      uint4* s = ring + (size_t)(t & (kPairBwd - 1)) * 5 * CH * NT;
      const uint32_t *p = point((uint32_t)t, e, 0), *q = point((uint32_t)t, e, 1);
      const bool tp = !kFirst || e.x != kNullEntry, tq = !kFirst || e.y != kNullEntry;
      stage_elem(s, p, tp);
      stage_elem(s + CH * NT, p + FW, tp);
      stage_elem(s + 2 * CH * NT, q, tq);
      stage_elem(s + 3 * CH * NT, q + FW, tq);
      if (t > 0) stage_elem(s + 4 * CH * NT, dst + (base + (uint64_t)(t - 1) * NT) * PW, true);
    }
    cp_async_commit();
  };
  uint2 e = entries(cnt - 1), e_n = cnt > 1 ? entries(cnt - 2) : make_uint2(0u, 0u);
  stage((int64_t)cnt - 1, e);
  for (uint32_t t = cnt; t-- > 0;) {
    const uint2 ec = e;
    stage((int64_t)t - 1, e_n);
    e = e_n;
    if (t > 1) e_n = entries(t - 2);
    cp_async_wait<1>();
    const uint64_t j = base + (uint64_t)t * NT;
    const uint4* s = ring + (size_t)(t & (kPairBwd - 1)) * 5 * CH * NT;
    Affine<F> p, q;
    p.x = elem_of_chunks<F>(s, NT);
    q.x = elem_of_chunks<F>(s + 2 * CH * NT, NT);
    p.y = elem_of_chunks<F>(s + CH * NT, NT);
    q.y = elem_of_chunks<F>(s + 3 * CH * NT, NT);
    const bool mp = is_inf(p), mq = is_inf(q);
    if constexpr (kFirst) {
      p.y = select(ec.x >> 31, neg(p.y), p.y);
      q.y = select(ec.y >> 31, neg(q.y), q.y);
    }
    F d, num;
    const bool none = pair_terms(p, q, mp, mq, d, num);
    F dinv = inv;
    if (t > 0) dinv = imul(inv, elem_of_chunks<F>(s + 4 * CH * NT, NT));
    inv = imul(inv, d);
    store_affine(dst + j * PW, pair_sum(p, q, mp, mq, none, num, dinv));
  }
}

// Rounds before the XYZZ accumulation.  A pair addition costs 3056 cycles of the multiply pipe per
// warp against madd-2008-s's 4784 and about 1500 instructions against 2120; a round adds its share
// of an inversion, a launch, and the gathers twice.  Measured on GB300, two rounds against none: G1
// MSM 2^20 (17.8 M entries, 64 per bucket) 2.42 ms of mixed additions -> 1.57 + 0.65 ms, the MSM
// 3.49 -> 3.19 ms (one round 3.33, three 3.3); SquareChain(2^20) 23.2 -> 20.75 ms, 2^19 12.2 ->
// 11.15 ms, 16 mixed proofs in a batch 17.2 -> 16.5 ms; SquareChain(2^18) level (6.65-6.77 ms either
// way), with tables of 2 M entries too 2^17 and the batch 2% slower: window tables of 2^18 points and
// up, of which a proof takes as many rounds as its reservation has room for (prove_round_cap).  The
// bucket sets of standalone MSMs hold fewer entries per bucket; of those only the largest G1 ones
// take rounds (G2: one round measured 3.20 -> 3.04 ms at 2^18 points and 4.33 -> 3.98 at 400,000;
// bg_msm_pair_rounds is documented to take none there).
inline int pair_rounds_model(size_t n, size_t max_entries, size_t nkeys, bool g2, bool shared_set) {
  if (shared_set) return n >= (size_t(1) << 18) && max_entries >= 3000000 && max_entries >= 24 * nkeys ? 2 : 0;
  if (g2 || max_entries < (size_t(1) << 23) || max_entries < 32 * nkeys) return 0;
  return 2;
}
