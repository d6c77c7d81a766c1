// Multi-head latent attention (MLA) decode: MQA over the paged latent cache, a tile of latents shared by sixteen heads and by both products.
//
//   cache row (one per token, all heads share it):  [ c_kv : R | k_rope : up to 64 ]  (bf16 / fp16)
//   S^T[tok, h] = Kc[tok, :] · Q[h, :]^T        rows of both from the tile as it came
//   O^T[d, h]  += Kc[tok, d]^T · P^T[tok, h]    the SAME bytes, turned on their way into registers
//
// A CTA takes one (request, sixteen heads, part of the tokens): eight warps and a TMA producer, tiles of 64 tokens (R = 512 with rope: nine blocks of
// [64 tokens x 64 dims], 72 KB) in a ring.  Tokens are the rows of m16n8k16 products, the heads their columns.  Scores: a warp takes 16 tokens and half
// of the dims, its queries stay in registers; the halves meet through shared memory.  Four warps turn scores into weights (one reference maximum
// per head and tile), all eight multiply them with 64 of the 512 dims each.  The parts of a request are a thread-block cluster and merge through
// distributed shared memory: no workspace, no second launch, the same order in every run.
//
// R is any multiple of 8 up to 512: NL blocks of 64 dims; TMA zero-fills the tail of the last one or brings what follows in the row, which meets
// zeros of Q and output dims that are not stored.
//
// What it costs is latency: 7 us of launch, lengths, page ids, first tile and stores, 1.4 us a tile (of them 0.85 the products, 72 KB would come in 0.7),
// 1.5 us for merging.  With tcgen05 (M = 128 for 64 tokens, N = 16) a tile took 36 + 16 products of 90 cycles and two round trips through tensor
// memory, 3.2 us, and a split a launch of 4 us.  us before (with the best of 1 to 8 splits) and now: see mla_decode_splits in ops/cuda.py.
//
// wide: the rows of short portions in steps that are not decode steps alone, whose weights were held in 32 bits on the CUDA cores.
//
// Reference kernels for the op: csrc/libtorch_stable/attention/mla/sm100_cutlass_mla_kernel.cu (+ cutlass_sm100_mla/),
// FlashMLA; algorithm: vllm/model_executor/layers/attention/mla_attention.py:1-200 (absorbed-weight decode).
#include "warp_mma.cuh"

namespace mla {

constexpr int DR = 64;                // block of the rope part, where there is one (TMA zero-fills a narrower one)
constexpr int TILE = 64, N = 16;      // tokens and heads
constexpr int KB_BYTES = TILE * 128;  // 8 KB: one block [64 tok x 64 dims]
constexpr int WARPS = 8, NUM_THREADS = WARPS * 32;       // two per scheduler, so that a thread may have 255 registers
constexpr int P_BYTES = N * 128;      // weights [16 heads x 64 tok]
constexpr int MAX_PARTS = 16;
// tile geometry of a latent of NL 64-dim blocks with (ROPE = 1) or without a rope block behind it
template <int NL, int ROPE> struct Geo {
  static constexpr int NKB = NL + ROPE;
  static constexpr int STAGE_BYTES = NKB * KB_BYTES;
  static constexpr int STAGES = NKB >= 7 ? 3 : (NKB >= 5 ? 4 : 6);
  static constexpr int MT = (NL + 1) / 2;          // 16-dim groups of a warp, WARPS apart
  static constexpr int ROW = NL * 64 + 4;          // floats between merged rows
  // A tile as rows of NKB 128-byte pieces, one box a page, instead of as blocks, a box each: asking for a box takes 130 cycles, of all threads, as
  // they wait for the one that asks (nine of them a third of a tile's time).  The swizzle goes by the number of the piece, so the pieces of
  // eight tokens lie on different banks where NKB is odd; and rows must end with a block, or the last one would read on.
  static constexpr bool ROWS = NL == 8 && ROPE == 1;
};

struct Params {
  const void* q_nope; const void* q_pe;
  const int* block_table;
  const int* seq_lens;
  void* out;            // [B, H, R]
  float* lse_out;       // optional [B, H] (natural log)
  int64_t qn_b, qn_h, qr_b, qr_h;
  int64_t out_stride;   // elements between batch rows of out
  int bt_stride;
  int H, BS, parts, split_tiles, R, rope;
  int window;           // > 0: a query sees its last `window` keys
  int wide;             // weights keep 16 more bits: P = hi + lo, two products (rows of mixed steps, whose weights are held in 32 bits)
  int* error;           // raised when a wait ran into its limit
  float scale_log2;
};

VB_DEVICE void tma_load_3d_hint(void* dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
               " [%0], [%1, {%3, %4, %5}], [%2], %6;"
               ::"r"(smem_u32(dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "l"(policy) : "memory");
}
template <int ID, int THREADS> VB_DEVICE void bar_sync() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory"); }
VB_DEVICE void heads_sync(int kh) { if (kh) bar_sync<4, 128>(); else bar_sync<3, 128>(); }     // the groups of tokens of eight heads

template <typename T, int NL, int ROPE, bool WIDE, bool ROWS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
mla_decode_kernel(const __grid_constant__ CUtensorMap tmap_kv, const Params p) {
  using G_ = Geo<NL, ROPE>;
  constexpr int NKB = G_::NKB, STAGE_BYTES = G_::STAGE_BYTES, STAGES = G_::STAGES, MT = G_::MT, ROW = G_::ROW;
  constexpr int KH = NKB * 2;                 // 16-dim steps of a half of the dims
  static_assert(N * ROW * 4 <= STAGES * STAGE_BYTES, "merged rows fit the ring");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* p_smem = ring + STAGES * STAGE_BYTES;                      // [2 parts][16 heads x 64 tok]
  float* half = reinterpret_cast<float*>(p_smem + 2 * P_BYTES);             // [4 token groups][from a half][32 lanes x 4]
  __shared__ __align__(8) uint64_t full[STAGES];
  __shared__ __align__(16) float wmax[2][4][N], alpha_s[2][N], sums[4][N], top_s[N], sum_s[N];
  __shared__ int moved_s[2][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = blockIdx.x % p.parts, b = blockIdx.x / p.parts, h0 = blockIdx.y * N;
  int budget = MBAR_BUDGET;                   // failed polls left (mbar_wait_lim)
  pdl_trigger();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_kv);
    for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();
  const int kv_end = p.seq_lens[b], kv_begin = p.window > 0 ? max(0, kv_end - p.window) : 0;
  int tile_lo = kv_begin / TILE, tile_hi = (kv_end + TILE - 1) / TILE;
  const bool whole = p.parts == 1 || tile_hi - tile_lo <= p.split_tiles;       // merging takes as long as a tile
  if (whole) {
    if (part > 0) return;
  } else {
    const int per = (tile_hi - tile_lo + p.parts - 1) / p.parts;
    tile_lo += part * per;
    tile_hi = min(tile_hi, tile_lo + per);
  }
  const int n_tiles = max(tile_hi - tile_lo, 0), G = min(N, p.H - h0);

  // warp 0 asks for tile j; 32 page ids at a time
  const int BS = p.BS, ppt = BS >= TILE ? 1 : TILE / BS, rows = BS >= TILE ? TILE : BS;
  int box = -1;                               // row of a box in the cache
  auto fetch = [&](int j) {
    const int i0 = j * ppt;
    if ((i0 & 31) == 0) {
      const int tok = tile_lo * TILE + (i0 + lane) * rows;
      box = tok < kv_end && i0 + lane < n_tiles * ppt ? p.block_table[(int64_t)b * p.bt_stride + tok / BS] * BS + tok % BS : -1;
    }
    int row[4], n_valid = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      row[u] = __shfl_sync(0xffffffffu, box, (i0 + u) & 31);
      if (u >= ppt) row[u] = -1;
      n_valid += row[u] >= 0;
    }
    if (lane == 0) {
      const int s = j % STAGES;
      mbar_expect_tx(&full[s], (uint32_t)n_valid * rows * 128 * NKB);
      unsigned char* to = ring + s * STAGE_BYTES;
      if constexpr (ROWS) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (row[u] >= 0) tma_load_3d_hint(to + u * rows * (NKB * 128), &tmap_kv, 0, 0, row[u], &full[s], L2_EVICT_FIRST);
      } else {
        for (int kb = 0; kb < NKB; ++kb)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (row[u] >= 0)
              tma_load_2d_hint(to + kb * KB_BYTES + u * rows * 128, &tmap_kv, kb == NL ? p.R : kb * 64, row[u], &full[s], L2_EVICT_FIRST);
      }
    }
    __syncwarp();
  };
  if (warp == 0)
    for (int j = 0; j < STAGES && j < n_tiles; ++j) fetch(j);

  // a lane's share: of scores the tokens r0, r0 + 8 and the heads c0, c0 + 1 of a group of eight; of results the dims r0, r0 + 8 and the same heads
  const int r0 = lane >> 2, c0 = (lane & 3) * 2, mi = lane >> 3, l7 = lane & 7;
  const int tg = warp & 3, kh = warp >> 2;             // group of tokens; half of the dims, and of the heads from there on
  float o[MT][2][4], m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][nt][j] = 0.f;
  if (n_tiles > 0) {
    uint32_t q[KH][2][2];
    const T* qn = reinterpret_cast<const T*>(p.q_nope) + (int64_t)b * p.qn_b;
    const T* qr = reinterpret_cast<const T*>(p.q_pe) + (int64_t)b * p.qr_b;
#pragma unroll
    for (int i = 0; i < KH; ++i) {
      const int ks = kh * KH + i;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int head = h0 + nt * 8 + r0, d = ks * 16 + j * 8 + c0;
          uint32_t v = 0;
          if (head < p.H) {
            if (!ROPE || ks < NL * 4) { if (d < p.R) v = *reinterpret_cast<const uint32_t*>(qn + (int64_t)head * p.qn_h + d); }
            else if (d - NL * 64 < p.rope) v = *reinterpret_cast<const uint32_t*>(qr + (int64_t)head * p.qr_h + d - NL * 64);
          }
          q[i][nt][j] = v;
        }
    }
    const uint32_t ring_u = smem_u32(ring), p_u = smem_u32(p_smem);
    // the lane's row in the 8 x 8 matrices of a load: token l7 of a group of eight, sixteen bytes `chunk` of block kb
    constexpr uint32_t TOK = ROWS ? NKB * 128 : 128, BLOCK = ROWS ? 128 : KB_BYTES;
    const uint32_t k_row = (uint32_t)(tg * 16 + (mi & 1) * 8 + l7) * TOK, v_row = (uint32_t)((mi >> 1) * 8 + l7) * TOK;
    auto piece = [&](int kb, int chunk) { return kb * BLOCK + (uint32_t)((chunk ^ (ROWS ? (l7 + kb) & 7 : l7)) << 4); };
    static_assert(!ROWS || NKB % 8 == 1, "the swizzle of token t, block kb is that of piece t NKB + kb");
    float sc[2][4];
    // (on the way out: the sums of the chains, and half of them to the other half)
    auto pass_on = [&](float (&sd)[2][4]) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[nt][i] += sd[nt][i];
      float4* to = reinterpret_cast<float4*>(half + (tg * 2 + kh) * 128) + lane;
      *to = kh ? make_float4(sc[0][0], sc[0][1], sc[0][2], sc[0][3]) : make_float4(sc[1][0], sc[1][1], sc[1][2], sc[1][3]);
    };
    // scores of a tile over the warp's half of the dims; those of the other half's heads go to it
    auto scores = [&](int j) {
      const int s = j % STAGES;
      mbar_wait_lim(&full[s], (j / STAGES) & 1, budget);
      __syncwarp();
      const uint32_t st = ring_u + s * STAGE_BYTES + k_row;
      float sd[2][4];                                            // two chains for either group of heads
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[nt][i] = sd[nt][i] = 0.f;
#pragma unroll
      for (int i = 0; i < KH; ++i) {
        const int ks = kh * KH + i;
        uint32_t ka[4];
        ldsm4(ka, st + piece(ks >> 2, (ks & 3) * 2 + (mi >> 1)));
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma16816<T>(i & 1 ? sd[nt] : sc[nt], ka, q[i][nt][0], q[i][nt][1]);
      }
      pass_on(sd);
    };
    // the same beside the results of the tile before, whose tokens are all seen: a load and two products of either in turn, loads one step ahead
    auto scores_and_results = [&](int j) {
      const int s = j % STAGES;
      mbar_wait_lim(&full[s], (j / STAGES) & 1, budget);
      __syncwarp();
      const uint32_t st = ring_u + s * STAGE_BYTES + k_row, sv = ring_u + (j - 1) % STAGES * STAGE_BYTES + v_row;
      const uint32_t pa = p_u + ((mi >> 1) * 8 + l7) * 128;
      uint32_t ph[4][4], pl[WIDE ? 4 : 1][4], ka[2][4], va[2][4];
      auto load_k = [&](int i) {
        const int ks = kh * KH + i;
        ldsm4(ka[i & 1], st + piece(ks >> 2, (ks & 3) * 2 + (mi >> 1)));
      };
      auto load_v = [&](int i) {                                 // 16 tokens of step i / MT
        const int mt = warp + i % MT * WARPS;
        if (NL % 2 == 0 || mt < NL * 4) ldsm4_t(va[i & 1], sv + i / MT * 16 * TOK + piece(mt >> 2, (mt & 3) * 2 + (mi & 1)));
      };
      load_k(0);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        ldsm4(ph[ks], pa + (((ks * 2 + (mi & 1)) ^ l7) << 4));
        if (WIDE) ldsm4(pl[ks], pa + P_BYTES + (((ks * 2 + (mi & 1)) ^ l7) << 4));
      }
      load_v(0);
      float sd[2][4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[nt][i] = sd[nt][i] = 0.f;
      constexpr int MOST = KH > 4 * MT ? KH : 4 * MT;
#pragma unroll
      for (int i = 0; i < MOST; ++i) {
        if (i + 1 < KH) load_k(i + 1);
        if (i + 1 < 4 * MT) load_v(i + 1);
        if (i < KH)
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma16816<T>(i & 1 ? sd[nt] : sc[nt], ka[i & 1], q[i][nt][0], q[i][nt][1]);
        if (i < 4 * MT && (NL % 2 == 0 || warp + i % MT * WARPS < NL * 4))
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            mma16816<T>(o[i % MT][nt], va[i & 1], ph[i / MT][nt * 2], ph[i / MT][nt * 2 + 1]);
            if (WIDE) mma16816<T>(o[i % MT][nt], va[i & 1], pl[WIDE ? i / MT : 0][nt * 2], pl[WIDE ? i / MT : 0][nt * 2 + 1]);
          }
      }
      pass_on(sd);
    };
    scores(0);
    for (int j = 0; j < n_tiles; ++j) {
      const int s = j % STAGES, buf = j & 1;
      const int tok0 = (tile_lo + j) * TILE, tok = tok0 + tg * 16;
      bar_sync<1, NUM_THREADS>();              // the halves of the scores are there, and everything has been read of the tile before
      if (warp == 0 && j > 0 && j - 1 + STAGES < n_tiles) fetch(j - 1 + STAGES);
      // ---- weights of the warp's 16 tokens and eight heads (8 kh ..)
      {
        const float4 x4 = *(reinterpret_cast<const float4*>(half + (tg * 2 + (kh ^ 1)) * 128) + lane);
        const float other[4] = {x4.x, x4.y, x4.z, x4.w};
        const bool in[2] = {tok + r0 >= kv_begin && tok + r0 < kv_end, tok + 8 + r0 >= kv_begin && tok + 8 + r0 < kv_end};
        float x[4], mx[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = in[i >> 1] ? ((kh ? sc[1][i] : sc[0][i]) + other[i]) * p.scale_log2 : -INFINITY;
#pragma unroll
        for (int u = 0; u < 2; ++u) mx[u] = fmaxf(x[u], x[2 + u]);
#pragma unroll
        for (int y = 4; y < 32; y <<= 1)
#pragma unroll
          for (int u = 0; u < 2; ++u) mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], y));
        if (r0 == 0) *reinterpret_cast<float2*>(&wmax[buf][tg][kh * 8 + c0]) = make_float2(mx[0], mx[1]);
        heads_sync(kh);
        float2 w[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) w[g] = *reinterpret_cast<const float2*>(&wmax[buf][g][kh * 8 + c0]);
        const float all[2] = {fmaxf(fmaxf(w[0].x, w[1].x), fmaxf(w[2].x, w[3].x)), fmaxf(fmaxf(w[0].y, w[1].y), fmaxf(w[2].y, w[3].y))};
        float alpha[2], ref[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float was = m_run[u];
          // the old reference stays unless the new maximum is more than 2^8 above it
          const bool up = all[u] > was + 8.f || (was == -INFINITY && all[u] > -INFINITY);
          m_run[u] = up ? all[u] : was;
          ref[u] = m_run[u] == -INFINITY ? 0.f : m_run[u];
          alpha[u] = was == -INFINITY ? 1.f : ex2(was - ref[u]);           // (1 where it stays)
          l_run[u] *= alpha[u];
        }
        if (tg == 0 && r0 == 0) *reinterpret_cast<float2*>(&alpha_s[buf][kh * 8 + c0]) = make_float2(alpha[0], alpha[1]);
        const bool moved = __any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f);
        if (tg == 0 && lane == 0) moved_s[buf][kh] = moved;
        unsigned char* pr = p_smem + (kh * 8 + r0) * 128 + c0 * 2;       // after turning: head r0, tokens c0, c0 + 1
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float a = ex2(x[2 * t] - ref[0]), c = ex2(x[2 * t + 1] - ref[1]);
          l_run[0] += a; l_run[1] += c;
          const uint32_t hi = pack2<T>(a, c);
          const int at = ((tg * 2 + t) ^ r0) << 4;
          *reinterpret_cast<uint32_t*>(pr + at) = turn8(hi);
          if (WIDE) {
            const float2 back = unpack2<T>(hi);
            *reinterpret_cast<uint32_t*>(pr + P_BYTES + at) = turn8(pack2<T>(a - back.x, c - back.y));
          }
        }
      }
      bar_sync<2, NUM_THREADS>();
      // ---- results
      if (moved_s[buf][0] | moved_s[buf][1]) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float2 a = *reinterpret_cast<const float2*>(&alpha_s[buf][nt * 8 + c0]);
#pragma unroll
          for (int i = 0; i < MT; ++i) { o[i][nt][0] *= a.x; o[i][nt][1] *= a.y; o[i][nt][2] *= a.x; o[i][nt][3] *= a.y; }
        }
      }
      if (j + 1 < n_tiles && tok0 >= kv_begin && tok0 + TILE <= kv_end) {
        scores_and_results(j + 1);
        continue;
      }
      if (j + 1 < n_tiles) scores(j + 1);
      const uint32_t st = ring_u + s * STAGE_BYTES + v_row, pa = p_u + ((mi >> 1) * 8 + l7) * 128;
#pragma unroll 1
      for (int ks = 0; ks < 4; ++ks) {
        const int t = tok0 + ks * 16;
        if (t >= kv_end || t + 16 <= kv_begin) continue;
        // slots that are not the sequence's may hold what a weight of 0 does not cancel (attention_prompt.cuh)
        const uint32_t k0 = keep2(t + c0, kv_begin, kv_end), k1 = keep2(t + 8 + c0, kv_begin, kv_end);
        uint32_t ph[4], pl[4], va[MT][4];                        // heads 0-7: tokens 0-7, 8-15; heads 8-15
        ldsm4(ph, pa + (((ks * 2 + (mi & 1)) ^ l7) << 4));
        if (WIDE) ldsm4(pl, pa + P_BYTES + (((ks * 2 + (mi & 1)) ^ l7) << 4));
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const int mt = warp + i * WARPS;
          if (NL % 2 == 0 || mt < NL * 4) ldsm4_t(va[i], st + ks * 16 * TOK + piece(mt >> 2, (mt & 3) * 2 + (mi & 1)));
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          if (NL % 2 && warp + i * WARPS >= NL * 4) continue;
          va[i][0] &= k0; va[i][1] &= k0; va[i][2] &= k1; va[i][3] &= k1;
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            mma16816<T>(o[i][nt], va[i], ph[nt * 2], ph[nt * 2 + 1]);
            if (WIDE) mma16816<T>(o[i][nt], va[i], pl[nt * 2], pl[nt * 2 + 1]);
          }
        }
      }
    }
  }
  if (budget < 0 && threadIdx.x == 0)          // let the copies in flight land before the block gives up its memory
    for (int n = 0; n < 4096 * STAGES; ++n) mbar_try_wait(&full[n % STAGES], n / STAGES & 1);
  // ===== the warps' dims side by side, then the parts
  __syncthreads();                             // every tile has come and been read: the ring is free
  float* merged = reinterpret_cast<float*>(ring);
  {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const int mt = warp + i * WARPS;
          if (NL % 2 && mt >= NL * 4) continue;
          float* row = merged + (nt * 8 + c0 + u) * ROW + mt * 16 + r0;
          row[0] = o[i][nt][u]; row[8] = o[i][nt][2 + u];
        }
        if (nt == 0) {
          float l = l_run[u];
#pragma unroll
          for (int x = 4; x < 32; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
          if (r0 == 0) { sums[tg][kh * 8 + c0 + u] = l; if (tg == 0) top_s[kh * 8 + c0 + u] = m_run[u]; }
        }
      }
  }
  __syncthreads();
  if (threadIdx.x < N) sum_s[threadIdx.x] = sums[0][threadIdx.x] + sums[1][threadIdx.x] + sums[2][threadIdx.x] + sums[3][threadIdx.x];
  T* out = reinterpret_cast<T*>(p.out) + (int64_t)b * p.out_stride;
  auto finish = [&](int g, int d, float2 acc, float m, float l) {
    const float inv = l > 0.f ? 1.f / l : 0.f;
    *reinterpret_cast<uint32_t*>(out + (int64_t)(h0 + g) * p.R + d) = pack2<T>(acc.x * inv, acc.y * inv);
    if (p.lse_out && d == 0) p.lse_out[(int64_t)b * p.H + h0 + g] = l > 0.f ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
  };
  if (whole) {
    __syncthreads();
    for (int i = threadIdx.x; i < G * NL * 32; i += NUM_THREADS) {
      const int g = i / (NL * 32), d = i % (NL * 32) * 2;
      if (d < p.R) finish(g, d, *reinterpret_cast<const float2*>(merged + g * ROW + d), top_s[g], sum_s[g]);
    }
  } else {
    cluster_sync();
    // 64 dims of a head go to one warp at a time: a lane reads the maximum and the sum of a part
    const uint32_t rows = smem_u32(merged), tops = smem_u32(top_s), ls = smem_u32(sum_s);
    for (int i = part * WARPS + warp; i < G * NL; i += p.parts * WARPS) {
      const int g = i / NL, d = i % NL * 64 + lane * 2, from = lane < p.parts ? lane : 0;
      float2 v[MAX_PARTS];
#pragma unroll
      for (int x = 0; x < MAX_PARTS; ++x) v[x] = x < p.parts ? ld_dsmem_f32x2(dsmem_addr(rows + (g * ROW + d) * 4, x)) : make_float2(0.f, 0.f);
      const float pm = lane < p.parts ? ld_dsmem_f32(dsmem_addr(tops + g * 4, from)) : -INFINITY;
      const float pl = lane < p.parts ? ld_dsmem_f32(dsmem_addr(ls + g * 4, from)) : 0.f;
      const float m = warp_max(pm), f = m == -INFINITY ? 0.f : ex2(pm - m), l = warp_sum(f * pl);
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int x = 0; x < MAX_PARTS; ++x) {
        const float fx = __shfl_sync(0xffffffffu, f, x);
        acc.x += fx * v[x].x; acc.y += fx * v[x].y;
      }
      if (d < p.R) finish(g, d, acc, m, l);
    }
    cluster_sync();                            // the others may still read this CTA's rows
  }
  if (budget < 0 && p.error) *p.error = 1;
}

constexpr int MISC_BYTES = 2 * P_BYTES + 4 * 2 * 128 * 4 + 1024;

template <typename T, int NL, int ROPE, bool WIDE, bool ROWS>
static int launch_one(const CUtensorMap& tkv, const Params& p, int B, cudaStream_t st) {
  const int smem = Geo<NL, ROPE>::STAGES * Geo<NL, ROPE>::STAGE_BYTES + MISC_BYTES;
  auto k = mla_decode_kernel<T, NL, ROPE, WIDE, ROWS>;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -20;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return -21;
    set = true;
  }
  return (int)vb_launch_parts(k, dim3(p.parts * B, (p.H + N - 1) / N), dim3(NUM_THREADS), (size_t)smem, st, p.parts, tkv, p);
}

template <typename T, int NL, int ROPE>
static int launch(const CUtensorMap& tkv, const Params& p, int B, bool rows, cudaStream_t st) {
  constexpr bool ROWS = Geo<NL, ROPE>::ROWS;
  if (ROWS && !rows) return p.wide ? launch_one<T, NL, ROPE, true, false>(tkv, p, B, st) : launch_one<T, NL, ROPE, false, false>(tkv, p, B, st);
  return p.wide ? launch_one<T, NL, ROPE, true, ROWS>(tkv, p, B, st) : launch_one<T, NL, ROPE, false, ROWS>(tkv, p, B, st);
}

}  // namespace mla

// clusters of `parts` CTAs that run at a time (of the widest latents)
EXPORT int vb_mla_clusters(int parts) {
  using namespace mla;
  auto k = mla_decode_kernel<__nv_bfloat16, 8, 1, false, true>;
  const int smem = Geo<8, 1>::STAGES * Geo<8, 1>::STAGE_BYTES + MISC_BYTES;
  if (parts < 1 || parts > MAX_PARTS || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return -1;
  return vb_max_clusters(k, dim3(NUM_THREADS), (size_t)smem, parts);
}

// q_nope: [B, H, R] (absorbed W_UK), q_pe: [B, H, rope] or null, cache: [num_blocks, BS, R + rope]; out: [B, H, R].
// bf16 covers every R (a multiple of 8 up to 512) and rope part (none, or a multiple of 8 up to 64); fp16 R = 512 with 64 only.
// window > 0: row b sees keys seq_lens[b] - window .. seq_lens[b] - 1.  parts: token ranges per row, a cluster (1 to 16); rows of split_tiles
// tiles or fewer stay whole.
// `error` (device int, may be null) becomes 1 when a wait inside the kernel ran into its limit.
EXPORT int vb_mla_decode3(const void* q_nope, const void* q_pe, const void* cache, int64_t num_blocks, const int* block_table,
                         const int* seq_lens, void* out, float* lse_out, int* error, int B,
                         int H, int R, int rope, int BS, int64_t qn_stride_b, int64_t qn_stride_h, int64_t qr_stride_b,
                         int64_t qr_stride_h, int64_t out_stride, int bt_stride, int parts, int split_tiles, int window, int wide, float scale, int dtype,
                         cudaStream_t st) {
  using namespace mla;
  if (B == 0) return 0;
  if (dtype == DT_F32 || R < 8 || R > 512 || R % 8) return -1;
  if (rope < 0 || rope > DR || rope % 8 || (dtype != DT_BF16 && (rope != DR || R != 512))) return -2;
  if (BS != 16 && BS != 32 && BS != 64 && BS != 128) return -4;
  if (parts < 1 || parts > MAX_PARTS) return -5;
  // queries are read and results written two values at a time
  if ((qn_stride_b | qn_stride_h | out_stride) & 1 || (rope && (qr_stride_b | qr_stride_h) & 1)) return -6;
  if (((reinterpret_cast<uintptr_t>(q_nope) | reinterpret_cast<uintptr_t>(q_pe) | reinterpret_cast<uintptr_t>(out)) & 3) || (rope && !q_pe)) return -7;
  auto enc = get_encode();
  if (!enc) return -10;
  const bool bf16 = dtype == DT_BF16;
  const int DK = R + rope;
  Params p;
  p.q_nope = q_nope; p.q_pe = q_pe; p.block_table = block_table; p.seq_lens = seq_lens; p.out = out; p.lse_out = lse_out; p.error = error;
  p.qn_b = qn_stride_b; p.qn_h = qn_stride_h; p.qr_b = qr_stride_b; p.qr_h = qr_stride_h; p.out_stride = out_stride; p.bt_stride = bt_stride;
  p.H = H; p.BS = BS; p.parts = parts; p.split_tiles = split_tiles; p.R = R; p.rope = rope; p.window = window; p.wide = wide;
  p.scale_log2 = scale * 1.4426950408889634f;
  CUtensorMap tkv;
  bool rows;
  {
    const cuuint32_t tokens = BS >= TILE ? TILE : BS;
    rows = R == 512 && rope == DR;             // Geo::ROWS
    cuuint64_t d3[3] = {64, (cuuint64_t)DK / 64, (cuuint64_t)num_blocks * BS}, s3[2] = {128, (cuuint64_t)DK * 2};
    cuuint32_t b3[3] = {64, (cuuint32_t)(DK / 64), tokens}, e3[3] = {1, 1, 1};
    cuuint64_t d2[2] = {(cuuint64_t)DK, (cuuint64_t)num_blocks * BS}, s2[1] = {(cuuint64_t)DK * 2};
    cuuint32_t b2[2] = {64, tokens}, e2[2] = {1, 1};
    const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    if (enc(&tkv, dt, rows ? 3 : 2, const_cast<void*>(cache), rows ? d3 : d2, rows ? s3 : s2, rows ? b3 : b2, rows ? e3 : e2,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -13;
  }
#define GO(TT, NL, RP) return launch<TT, NL, RP>(tkv, p, B, rows, st)
  const int nl = (R + 63) / 64;
#define WIDTHS(RP)                                                                                            \
  do {                                                                                                        \
    if (nl <= 1) GO(__nv_bfloat16, 1, RP);                                                                    \
    else if (nl == 2) GO(__nv_bfloat16, 2, RP);                                                               \
    else if (nl == 3) GO(__nv_bfloat16, 3, RP);                                                               \
    else if (nl == 4) GO(__nv_bfloat16, 4, RP);                                                               \
    else if (nl <= 6) GO(__nv_bfloat16, 6, RP);                                                               \
    else GO(__nv_bfloat16, 8, RP);                                                                            \
  } while (0)
  if (!bf16) GO(__half, 8, 1);
  else if (rope) WIDTHS(1);
  else WIDTHS(0);
#undef WIDTHS
#undef GO
}
