// What the prompt attention kernels share (attention_tc.cu over pages, mla_prefill.cu over expanded keys): the matrix-product and the
// softmax roles of a CTA that takes one or two tiles of 128 query rows through the same keys.
//
//   S_t = Q_t K^T      both operands from shared memory, 128 x 128 scores of 32 bits in tensor memory
//   P_t = 2^(S_t - m)  16-bit, written over the scores in tensor memory; O_t += P_t V reads it from there as its A operand
//
// A thread owns a query row (a lane of tensor memory): it reads all 128 scores of a key tile at once and keeps them in registers, so maximum,
// exponentials and row sum take one pass and no exchange.  With two tiles the tensor core works on one tile's products while the
// other tile's warpgroup is at its exponentials; with one tile per CTA the two warpgroups share it, one takes the even, the other the odd key
// tiles, and their results are merged at the end.  The products of a warpgroup are issued in the order P V of its key tile j, Q K of its
// tile j + 1 by one thread and run in that order, so a full S_t also says that O_t is complete: the rescaling of O needs no barrier of
// its own, and P may lie over S.
//
// CAP: scores are capped, c tanh(s / c).  SPLIT: the weights keep 16 more bits (P = hi + lo, two products): for paths whose weights are held
// in 32 bits elsewhere, at half as much tensor work again.  Results of capped prompts and decode steps are then as far from 64 bits as with
// 32-bit weights on the CUDA cores, to three digits (8 / 2 and 16 / 4 heads, 16 to 4100 tokens: bf16 0.00139 to 0.00170, fp16 0.00017 to 0.00021).
// Tensor memory: S_0, S_1 (128 columns each), O_0, O_1 (up to 128 each).
//
// Bound by the length of a turn (scores out of tensor memory, maximum, exponentials, weights back) and not by a unit: 32 / 8 heads, two prompts
// of 3800 tokens keep the tensor core busy for 44 % of the cycles, the special-function unit for 44 %, and instructions issue in 37 %;
// capped, 16 / 4 heads, eight prompts of 860 tokens 13, 9 and 32 % (instruction fetches and barriers are what warps wait for most).  Measured:
// the former 576 us with one tile of rows, scores read twice and weights through shared memory, 347 us so; the latter 2536 us on the CUDA
// cores, 182 us so.
#pragma once
#include "common.cuh"

namespace prompt {

// Query tiles (of all requests and heads) for each SM from which a CTA takes two of them: below, SMs would be left without any, and the two
// warpgroups of a CTA share one.  One prompt of 2000 tokens, 8 / 2 heads (125 tiles): 42 us shared, 57 us with one warpgroup at work; 2 x 1000,
// 16 / 4 heads (250): 40 against 49; from 300 tiles on two per CTA: 8 x 300, 16 / 4 heads (300) 34 us, 2 x 2000, 32 / 8 (1000) 124 us, where one
// tile of rows per CTA took 182.  The two forms add a row's keys in different orders, so batch-invariant mode (in_order) has one: always two
// tiles, the second one empty where a portion ends within the first.
constexpr int PAIR_MIN_TILES = 2;

constexpr int ROWS = 128, KEYS = 128;
constexpr int NUM_THREADS = 384;            // warp 0 TMA producer, 1 MMA issuer, 2 and 3 clear values, 4..7 and 8..11 softmax of the two tiles
// registers a thread: launched with 168; 384 x 168 = 128 x 72 + 256 x 216
constexpr int REGS_AUX = 72, REGS_SOFTMAX = 216;
template <int N> VB_DEVICE void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> VB_DEVICE void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr int BLK = 128 * 128;              // one [128 rows x 64 values] block of 16-bit values, 16 KB

// D[tmem] (+)= A[tmem] * B[smem desc]: A holds two 16-bit values of a row in a column
VB_DEVICE void warp_umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
VB_DEVICE void tma_load_3d(void* dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(smem_u32(dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
VB_DEVICE void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
VB_DEVICE void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
VB_DEVICE void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// KS stages of keys, VS of values.  edge: values of the first and the last key tile, where they are cleared before the product
template <int KS, int VS> struct Bars {
  uint64_t q_full, k_full[KS], k_empty[KS], v_full[VS], v_empty[VS], s_full[2], p_full[2], o_done[2], edge[2];
  VB_DEVICE void init() {
    mbar_init(&q_full, 1);
    for (int s = 0; s < KS; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < VS; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    for (int t = 0; t < 2; ++t) { mbar_init(&s_full[t], 1); mbar_init(&p_full[t], ROWS); mbar_init(&o_done[t], 1); mbar_init(&edge[t], 1); }
    mbar_fence_init();
  }
  // a producer that gave up: let its copies in flight land before the block gives up its memory
  VB_DEVICE void drain() {
    mbar_let_land(k_full, KS);
    mbar_let_land(v_full, VS);
    mbar_let_land(edge, 2);
  }
};

// A weight of 0 keeps neither an infinity nor a NaN out of a sum, but the slots of a key tile that no row sees (behind a sequence's end, in front
// of a window) may hold values of another request.  The products leave out the groups of 16 slots (an MMA's depth) that nobody sees; where
// a part of a group is seen, the rest of it is overwritten with zeros before the product.  In prompts such a tile's values arrive at a
// barrier of their own and two idle warps clear and pass them on (in the softmax warps: 549 → 594 us for 32 / 8 heads, 4 x 3800 tokens, by the
// registers); in decode steps the softmax warps do it last, where the product waits for the values as well.  us without and so: 32 / 8
// heads, 4 x 3800 tokens 553 and 534 (no clearing of shared memory at the start), decode 24 x 500 11.6 and 11.6, 64 x 280 16.7 and
// 17.9, 64 x 288 16.7 and 16.5, 64 x 1000 46.3 and 46.6.
// Tokens [lo, hi) of the tile are seen, of `keys`.
struct Seen {
  int lo, hi;
  VB_DEVICE Seen(int first, int begin, int end, int keys) : lo(max(begin - first, 0)), hi(min(end - first, keys)) {}
  VB_DEVICE bool cut() const { return ((lo | hi) & 15) != 0; }
  VB_DEVICE int k0() const { return lo >> 4; }
  VB_DEVICE int k1() const { return (hi + 15) >> 4; }
};
// Row r of blocks of 64 tokens per 128-byte swizzled row, `stride` bytes apart: tokens [lo, hi), all of one group of 16, become zeros.
VB_DEVICE void clear_group(unsigned char* blocks, int stride, int r, int lo, int hi) {
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int c = (lo >> 4) * 2 + e, a = lo - c * 8, b = hi - c * 8;        // 16 bytes: 8 tokens
    if (a >= 8 || b <= 0) continue;
    uint4* p = reinterpret_cast<uint4*>(blocks + (c >> 3) * stride + r * 128 + (((c & 7) ^ (r & 7)) << 4));
    if (a <= 0 && b >= 8) { *p = make_uint4(0, 0, 0, 0); continue; }
    uint4 v = *p;
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (2 * i >= a && 2 * i < b) w[i] &= 0xffff0000u;
      if (2 * i + 1 >= a && 2 * i + 1 < b) w[i] &= 0x0000ffffu;
    }
    *p = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
// what is not seen of the groups that are seen in part, in row r
VB_DEVICE void clear_cut(unsigned char* blocks, int stride, int r, const Seen& s) {
  if (s.lo & 15) clear_group(blocks, stride, r, s.lo & ~15, s.lo);
  if (s.hi & 15) clear_group(blocks, stride, r, s.hi, (s.hi + 15) & ~15);
}
VB_DEVICE void pass_on(uint64_t* v_full) {
  fence_proxy_async();
  asm volatile("bar.sync 2, 64;" ::: "memory");
  if ((threadIdx.x & 63) == 0) mbar_arrive(v_full);
}

// MMA issuer (one warp).  qk(t, stage) issues S_t, pv(t, stage, key tile, first) issues O_t.  n >= 1 key tiles, each for both of two query tiles
// (`pair`), or the even ones for t = 0 and the odd ones for t = 1.
template <int KS, int VS, class QK, class PV>
VB_DEVICE void mma_role(Bars<KS, VS>& b, int n, bool pair, int& budget, QK qk, PV pv) {
  mbar_wait_lim(&b.q_full, 0, budget);
  const int ahead = pair ? 1 : 2;                          // key tiles between a product Q K of a warpgroup and its next
  for (int j = 0; j < min(ahead, n); ++j) {
    mbar_wait_lim(&b.k_full[j % KS], 0, budget);           // (ahead <= KS)
    tc_fence_after();
    __syncwarp();
    {
      for (int t = pair ? 0 : j; t < (pair ? 2 : j + 1); ++t) { qk(t, j % KS); warp_umma_commit(&b.s_full[t]); }
      warp_umma_commit(&b.k_empty[j % KS]);
    }
    __syncwarp();
  }
  for (int j = 0; j < n; ++j) {
    const int vs = j % VS, nx = j + ahead, ks = nx % KS;
    mbar_wait_lim(&b.v_full[vs], (j / VS) & 1, budget);
    const int t0 = pair ? 0 : j & 1, t1 = pair ? 1 : t0;
    const int phase = (pair ? j : j >> 1) & 1;
    for (int t = t0; t <= t1; ++t) {
      mbar_wait_lim(&b.p_full[t], phase, budget);
      tc_fence_after();
      __syncwarp();
      {
        pv(t, vs, j, pair ? j == 0 : j < 2);
        if (t == t1) warp_umma_commit(&b.v_empty[vs]);
        if (nx >= n) warp_umma_commit(&b.o_done[t]);
      }
      __syncwarp();
      if (nx < n) {
        if (t == t0) { mbar_wait_lim(&b.k_full[ks], (nx / KS) & 1, budget); tc_fence_after(); }
        __syncwarp();
        {
          qk(t, ks);
          warp_umma_commit(&b.s_full[t]);
          if (t == t1) warp_umma_commit(&b.k_empty[ks]);
        }
        __syncwarp();
      }
    }
  }
}

// c2 tanh(x), |x| <= 1 in the whole warp (`small`): x times a polynomial of x^2 that interpolates tanh(x) / x at the Chebyshev points of
// [0, 1] (relative error 1.6e-7 in 32 bits); elsewhere by one exponential.
VB_DEVICE float cap_small(float x, float c2) {
  const float z = x * x;
  float r = 0.0010380251333117485f;
  r = fmaf(r, z, -0.0061943246982991695f);
  r = fmaf(r, z, 0.02027970738708973f);
  r = fmaf(r, z, -0.053451646119356155f);
  r = fmaf(r, z, 0.13325075805187225f);
  r = fmaf(r, z, -0.3333282768726349f);
  r = fmaf(r, z, 0.9999999403953552f);
  return r * (x * c2);
}
VB_DEVICE float cap_any(float x, float c2) {
  const float e = ex2(fabsf(x) * 2.8853900817779268f);          // e^(2 |x|), at worst infinite: 1 - 0
  return fabsf(x) <= 1.f ? cap_small(x, c2) : copysignf(1.f - 2.f / (e + 1.f), x) * c2;      // (no matter which of the two a warp takes)
}

struct Softmax {
  float scale_log2;            // plain scores
  float ku, c2;                // capped: scale / cap, cap log2(e)
};

// Softmax of one query tile: thread = row.  The row sees the keys [lo, hi) of its request (lo >= hi: none); `first`: the first key of the first
// of the warpgroup's n key tiles, which are `step` keys apart.  Leaves O_t complete; returns the row's reference maximum (powers of two) and
// its sum.
template <typename T, int OC, bool CAP, int KS, int VS>
VB_DEVICE void softmax_role(Bars<KS, VS>& b, int t, uint32_t t_s, uint32_t t_o, int n, int first, int step, int lo, int hi, const Softmax& sm, bool split,
                            int& budget, float& m_used, float& l_run) {
  m_used = -INFINITY;
  l_run = 0.f;
  for (int j = 0; j < n; ++j, first += step) {
    mbar_wait_lim(&b.s_full[t], j & 1, budget);
    __syncwarp();
    tc_fence_after();
    uint32_t v[4][32];
#pragma unroll
    for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, v[c]);
    tmem_ld_wait();
    const int l = lo - first, h = hi - first;                   // visible columns of this tile: [l, h)
    const bool full = __all_sync(0xffffffffu, l <= 0 && h >= KEYS) != 0;
    float mx = -INFINITY, far = 0.f;
    if (full) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          mx = fmaxf(mx, __uint_as_float(v[c][i]));
          if (CAP) far = fmaxf(far, fabsf(__uint_as_float(v[c][i])));
        }
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const bool in = c * 32 + i >= l && c * 32 + i < h;
          if (in) mx = fmaxf(mx, __uint_as_float(v[c][i]));
          if (CAP) {
            if (!in) v[c][i] = 0u;
            far = fmaxf(far, fabsf(__uint_as_float(v[c][i])));
          } else if (!in) {
            v[c][i] = 0xff800000u;                              // -inf: a weight of 0
          }
        }
    }
    bool small = true;
    if (CAP) {
      small = __all_sync(0xffffffffu, far * fabsf(sm.ku) <= 1.f) != 0;
      mx = mx == -INFINITY ? mx : cap_any(mx * sm.ku, sm.c2);
    } else {
      mx *= sm.scale_log2;
    }
    // keep the old reference maximum unless the new one is more than 2^8 above it
    float alpha = 1.f;
    bool rescale = false;
    if (mx > m_used + 8.f || (m_used == -INFINITY && mx > -INFINITY)) {
      rescale = m_used != -INFINITY;
      if (rescale) alpha = ex2(m_used - mx);
      m_used = mx;
    }
    const float m_ref = m_used == -INFINITY ? 0.f : m_used;
    if (__any_sync(0xffffffffu, rescale)) {                     // accesses to tensor memory are the whole warp's
      l_run *= alpha;
#pragma unroll
      for (int c = 0; c < OC; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32(t_o + c, o);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
        tmem_st_32x32(t_o + c, o);
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (CAP) {
        if (small) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[c][i] = __float_as_uint(cap_small(__uint_as_float(v[c][i]) * sm.ku, sm.c2));
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[c][i] = __float_as_uint(cap_any(__uint_as_float(v[c][i]) * sm.ku, sm.c2));
        }
      }
      auto weight = [&](int i) {
        const float x = __uint_as_float(v[c][i]);
        const float e = CAP ? ex2(x - m_ref) : ex2(fmaf(x, sm.scale_log2, -m_ref));
        return CAP && !full && (c * 32 + i < l || c * 32 + i >= h) ? 0.f : e;
      };
      uint32_t hi16[16];
      if (split) {
        uint32_t lo16[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = weight(i), p1 = weight(i + 1);
          sum += p0 + p1;
          hi16[i / 2] = pack2<T>(p0, p1);
          const float2 f = unpack2<T>(hi16[i / 2]);
          lo16[i / 2] = pack2<T>(p0 - f.x, p1 - f.y);
        }
        tmem_st_32x16(t_s + KEYS / 2 + c * 16, lo16);
      } else {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = weight(i), p1 = weight(i + 1);
          sum += p0 + p1;
          hi16[i / 2] = pack2<T>(p0, p1);
        }
      }
      tmem_st_32x16(t_s + c * 16, hi16);
    }
    l_run += sum;
    tmem_st_wait();
    tc_fence_before();
    mbar_arrive(&b.p_full[t]);
  }
  mbar_wait_lim(&b.o_done[t], 0, budget);
  __syncwarp();
  tc_fence_after();
}

// One query tile shared by both warpgroups: the second hands its row's maximum and sum over (`ml`, one per row) when its O is complete; the
// first waits for it and gets the factors of both O, those of the whole softmax.
VB_DEVICE void hand_over(float2* ml, int row, float m, float l) {
  ml[row] = make_float2(m, l);
  tc_fence_before();
  asm volatile("bar.sync 1, 256;" ::: "memory");
}
VB_DEVICE void take_over(const float2* ml, int row, float& m, float& l, float& f0, float& f1) {
  asm volatile("bar.sync 1, 256;" ::: "memory");
  tc_fence_after();
  const float2 o = ml[row];
  const float top = fmaxf(m, o.x);
  f0 = m == -INFINITY ? 0.f : ex2(m - top);
  f1 = o.x == -INFINITY ? 0.f : ex2(o.x - top);
  l = l * f0 + o.y * f1;
  m = top;
}
// columns c .. c + 31 of O, of a shared tile O_0 f0 + O_1 f1
VB_DEVICE void load_o(uint32_t t_o, int c, bool shared, float f0, float f1, uint32_t (&v)[32]) {
  tmem_ld_32x32(t_o + c, v);
  if (shared) {
    uint32_t u[32];
    tmem_ld_32x32(t_o + 128 + c, u);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * f0 + __uint_as_float(u[i]) * f1);
  } else {
    tmem_ld_wait();
  }
}

// O_t += P_t V: db(kk) is the descriptor of 16 keys of the values; groups k0 .. k1 - 1 of 16 keys
template <class DB> VB_DEVICE void issue_pv(uint32_t tmem_o, uint32_t tmem_p, uint32_t idesc, bool first, bool split, int k0, int k1, DB db) {
  if (k0 == 0 && k1 == KEYS / 16) {
#pragma unroll
    for (int kk = 0; kk < KEYS / 16; ++kk) warp_umma_f16_ta(tmem_o, tmem_p + kk * 8, db(kk), idesc, !first || kk != 0);
    if (split) {
#pragma unroll
      for (int kk = 0; kk < KEYS / 16; ++kk) warp_umma_f16_ta(tmem_o, tmem_p + KEYS / 2 + kk * 8, db(kk), idesc, 1);
    }
  } else {
#pragma unroll 1
    for (int kk = k0; kk < k1; ++kk) warp_umma_f16_ta(tmem_o, tmem_p + kk * 8, db(kk), idesc, !first || kk != k0);
    if (split) {
#pragma unroll 1
      for (int kk = k0; kk < k1; ++kk) warp_umma_f16_ta(tmem_o, tmem_p + KEYS / 2 + kk * 8, db(kk), idesc, 1);
    }
  }
}

}  // namespace prompt
