// Paged attention on the 5th-gen tensor cores, head_dim 128, 64-token pages: prompts, mixed batches, and decode steps that the kernel of
// attention_tc_decode.cu does not take.
//
// Reference back-ends for this op: FlashInfer TRT-LLM-gen cubins / FA4 CuTe-DSL (v1/attention/backends/
// flashinfer.py:2239,2457).  This is our own kernel, designed around a cache layout chosen for tcgen05:
//   K page  [64 tokens, 128 dims]  (dims contiguous)      → K-major B operand of  S = Q·K^T
//   V page  [128 dims, 64 tokens]  (tokens contiguous)    → K-major B operand of  O = P·V
// so every operand is a plain 128B-swizzled K-major tile that one TMA box load drops into shared memory
// (page-table driven: the block id of each page becomes the TMA row coordinate), with no transposes.
//
// CTA = one (request, kv head) x one or two tiles of 128 query rows (rows = q tokens x GQA group; decode uses G rows) x a KV
// range (split-KV for decode); warps: 0 TMA producer, 1 MMA issuer + TMEM owner, 2 and 3 clear values, 4..7 and 8..11 softmax and epilogue of the two tiles
// (attention_prompt.cuh).
#include "attention_prompt.cuh"

namespace fmha {

using prompt::BLK;
using prompt::tma_load_3d;
constexpr int D = 128;
constexpr int BS = 64;              // tokens per page
constexpr int TILE_N = prompt::KEYS;   // kv tokens per iteration (2 pages)
constexpr int TILE_M = prompt::ROWS;   // query rows per tile
constexpr int NUM_THREADS = prompt::NUM_THREADS;
constexpr int KV_STAGES = 2;
constexpr int MAX_TILES_SMEM = 1024;  // 2 block ids per tile cached in smem (covers 128k tokens)

constexpr int Q_BYTES = 2 * BLK;                   // 32 KB per tile (2 k-blocks of [128 x 64])
constexpr int K_BYTES = 2 * BLK;                   // 32 KB per stage (2 k-blocks of [128 tokens x 64])
constexpr int V_BYTES = 2 * BLK;                   // 32 KB per stage (2 pages of [128 dims x 64 tokens])
typedef prompt::Bars<KV_STAGES, KV_STAGES> Bars;

struct Params {
  const int* block_table;
  const int* seq_lens;
  const int* qsl;          // null → decode (1 token per request)
  void* out;               // [T, Hq, D]
  float* part_out;         // [T, Hq, S, D]
  float* part_lse;         // [T, Hq, S]  (log2 units)
  float* lse_out;          // optional [T, Hq] natural log
  int64_t out_stride;
  int bt_stride;
  int Hq, Hkv, G, TQ, num_splits;
  int tiles;               // query tiles per CTA: 1 or 2
  int in_order;            // a row's keys are added in their order, whatever else is in the batch
  int window, causal;
  prompt::Softmax sm;
  int flat_B;              // > 0: grid.x enumerates the (request, query tile) pairs of `flat_B` requests (device-side
                           //      schedule from qsl: the launch geometry depends only on the bucket, not on the lengths)
  int chunk;               // > 0: a query sees the keys of its own chunk of positions only
  const float* sinks;      // optional [Hq] logits in the softmax denominator that have no key
  float out_scale;         // factor of the output
  int* error;
};

template <typename T, bool CAP>
__global__ void __launch_bounds__(NUM_THREADS, 1)
fmha_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
            const __grid_constant__ CUtensorMap tmap_v, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* q_smem = smem;                             // 2 tiles
  unsigned char* k_smem = q_smem + 2 * Q_BYTES;             // KV_STAGES x K_BYTES
  unsigned char* v_smem = k_smem + KV_STAGES * K_BYTES;     // KV_STAGES x V_BYTES
  Bars& bars = *reinterpret_cast<Bars*>(v_smem + KV_STAGES * V_BYTES);
  float2* ml = reinterpret_cast<float2*>(&bars + 1);        // [TILE_M]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ml + TILE_M);
  int* blk_ids = reinterpret_cast<int*>(tmem_slot + 2);   // [2 * MAX_TILES_SMEM]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int budget = MBAR_BUDGET;                        // failed polls left (mbar_wait_lim)
  const int TC = p.TQ * p.tiles;                   // query tokens per CTA
  int b = blockIdx.z;
  const int h = blockIdx.y;
  int split = 0, qt = 0;
  pdl_trigger();
  pdl_wait();
  if (p.flat_B > 0) {
    // flat tile index → (request, tile): every warp walks the per-request tile counts 32 requests at a time (redundantly:
    // no shared memory or barrier before the early exit)
    int target = blockIdx.x, found_b = -1;
    for (int base = 0; base < p.flat_B && found_b < 0; base += 32) {
      const int r = base + lane;
      int nt = 0;
      if (r < p.flat_B) nt = (p.qsl[r + 1] - p.qsl[r] + TC - 1) / TC;
      int inc = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, target < inc);
      if (hit) {
        const int l = __ffs(hit) - 1;
        const int before = __shfl_sync(0xffffffffu, inc - nt, l);
        found_b = base + l;
        qt = target - before;
      } else {
        target -= __shfl_sync(0xffffffffu, inc, 31);
      }
    }
    if (found_b < 0) return;                       // more CTAs than tiles (bucket padding)
    b = found_b;
  } else if (p.qsl) {
    qt = (int)gridDim.x - 1 - (int)blockIdx.x;     // the latest tiles have the most keys: first
  } else {
    split = blockIdx.x;
  }
  const int seq_len = p.seq_lens[b];
  const int q0 = p.qsl ? p.qsl[b] : b;
  const int q_len = p.qsl ? p.qsl[b + 1] - q0 : 1;
  const int tok0 = qt * TC;
  if (tok0 >= q_len) return;                       // uniform across the CTA
  const int n_tok = min(TC, q_len - tok0);
  const int tiles = n_tok > p.TQ || p.in_order ? 2 : 1;
  const int pos0 = seq_len - q_len + tok0;
  const int pos_last = pos0 + n_tok - 1;
  const int kv_end = p.causal ? pos_last + 1 : seq_len;
  int kv_begin = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
  if (p.chunk > 0) kv_begin = max(kv_begin, pos0 / p.chunk * p.chunk);
  int tile_lo = kv_begin / TILE_N, tile_hi = (kv_end + TILE_N - 1) / TILE_N;
  {
    const int total = tile_hi - tile_lo;
    const int per = (total + p.num_splits - 1) / p.num_splits;
    tile_lo += split * per;
    tile_hi = min(tile_hi, tile_lo + per);
  }
  const int n_tiles = max(tile_hi - tile_lo, 0);
  const int n_pages_total = (kv_end + BS - 1) / BS;   // pages that hold valid tokens

  if (n_tiles == 0) {
    // nothing to attend to (can happen for empty splits): emit a neutral partial
    if (p.num_splits > 1 && (int)threadIdx.x < p.G * n_tok) {
      const int64_t pi = ((int64_t)(q0 + tok0 + threadIdx.x / p.G) * p.Hq + (h * p.G + threadIdx.x % p.G)) * p.num_splits + split;
      for (int d = 0; d < D; ++d) p.part_out[pi * D + d] = 0.f;
      p.part_lse[pi] = -INFINITY;
    }
    return;
  }

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
    bars.init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  for (int i = threadIdx.x; i < 2 * n_tiles && i < 2 * MAX_TILES_SMEM; i += NUM_THREADS) {
    const int page = tile_lo * 2 + i;
    blk_ids[i] = page < n_pages_total ? p.block_table[(int64_t)b * p.bt_stride + page] : -1;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto seen = [&](int j) { return prompt::Seen((tile_lo + j) * TILE_N, kv_begin, kv_end, TILE_N); };   // cut: the first or the last key tile

  if (warp < 4) {
    prompt::regs_dec<prompt::REGS_AUX>();
    if (warp == 0 && lane == 0) {
      // ===== TMA producer
      mbar_expect_tx(&bars.q_full, tiles * 2 * p.G * p.TQ * 64 * 2);   // TMA always delivers the full box
      for (int t = 0; t < tiles; ++t) {
        tma_load_3d(q_smem + t * Q_BYTES, &tmap_q, 0, h * p.G, q0 + tok0 + t * p.TQ, &bars.q_full);
        tma_load_3d(q_smem + t * Q_BYTES + BLK, &tmap_q, 64, h * p.G, q0 + tok0 + t * p.TQ, &bars.q_full);
      }
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % KV_STAGES;
        const uint32_t par = ((j / KV_STAGES) & 1) ^ 1;
        int blk[2];
        for (int u = 0; u < 2; ++u) {
          const int page = (tile_lo + j) * 2 + u;
          blk[u] = j < MAX_TILES_SMEM ? blk_ids[2 * j + u] : page < n_pages_total ? p.block_table[(int64_t)b * p.bt_stride + page] : -1;
        }
        const int n_valid = (blk[0] >= 0) + (blk[1] >= 0);
        unsigned char* ks = k_smem + s * K_BYTES;
        unsigned char* vs = v_smem + s * V_BYTES;
        mbar_wait_lim(&bars.k_empty[s], par, budget);
        if (budget < 0) break;
        mbar_expect_tx(&bars.k_full[s], n_valid * BS * D * 2);
        for (int u = 0; u < 2; ++u) {
          if (blk[u] < 0) continue;
          const int chunk = (blk[u] * 2 + 0) * p.Hkv + h;       // K chunk index
          // K view: [chunks*BS rows, D cols]; k-block kb lands at kb*16KB + u*8KB
          tma_load_2d(ks + 0 * BLK + u * (BS * 128), &tmap_k, 0, chunk * BS, &bars.k_full[s]);
          tma_load_2d(ks + 1 * BLK + u * (BS * 128), &tmap_k, 64, chunk * BS, &bars.k_full[s]);
        }
        mbar_wait_lim(&bars.v_empty[s], par, budget);
        if (budget < 0) break;
        uint64_t* v_bar = seen(j).cut() ? &bars.edge[j != 0] : &bars.v_full[s];
        mbar_expect_tx(v_bar, n_valid * BS * D * 2);
        for (int u = 0; u < 2; ++u) {
          if (blk[u] < 0) continue;
          const int chunk = (blk[u] * 2 + 1) * p.Hkv + h;       // V chunk index
          // V view: [chunks*D rows, BS cols]; page u is k-block u of the PV product: [128 dims x 64 tokens]
          tma_load_2d(vs + u * BLK, &tmap_v, 0, chunk * D, v_bar);
        }
      }
      if (budget < 0) bars.drain();
    } else if (warp == 1) {
    // ===== MMA issuer
    const uint32_t idesc = umma_idesc_f16(TILE_M, TILE_N, DTypeOf<T>::v == DT_BF16);
    const uint64_t d_q = umma_desc_sw128(q_smem), d_k = umma_desc_sw128(k_smem), d_v = umma_desc_sw128(v_smem);
    prompt::mma_role(
        bars, n_tiles, tiles == 2, budget,
        [&](int t, int s) {
          const int qt = tiles == 2 ? t : 0;
#pragma unroll
          for (int kb = 0; kb < 2; ++kb)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              warp_umma_f16(tmem_base + t * 128, d_q + (uint64_t)((qt * Q_BYTES + kb * BLK + k * 32) >> 4),
                       d_k + (uint64_t)((s * K_BYTES + kb * BLK + k * 32) >> 4), idesc, (kb | k) != 0);
        },
        [&](int t, int s, int j, bool first) {
          const prompt::Seen k = seen(j);
          prompt::issue_pv(tmem_base + 256 + t * 128, tmem_base + t * 128, idesc, first, CAP, k.k0(), k.k1(),
                           [&](int kk) { return d_v + (uint64_t)((s * V_BYTES + (kk / 4) * BLK + (kk & 3) * 32) >> 4); });
        });
    } else if (warp >= 2) {
      // ===== zeros into the values' slots that no row sees
      for (int e = 0; e < 2; ++e) {
        const int j = e ? n_tiles - 1 : 0, s = j % KV_STAGES;
        if ((e && n_tiles == 1) || !seen(j).cut()) continue;
        mbar_wait_lim(&bars.edge[e], 0, budget);
        for (int r = threadIdx.x & 63; r < 128; r += 64) prompt::clear_cut(v_smem + s * V_BYTES, BLK, r, seen(j));
        prompt::pass_on(&bars.v_full[s]);
      }
    }
  } else {
    prompt::regs_inc<prompt::REGS_SOFTMAX>();
    // ===== softmax / correction / epilogue: thread = query row = TMEM lane
    const int t = (warp >> 2) - 1, qd = warp & 3;
    const bool shared = tiles == 1 && n_tiles > 1;   // both warpgroups at one tile
    const int r = qd * 32 + lane;
    const uint32_t t_lane = (uint32_t)(qd * 32) << 16, t_o = tmem_base + 256 + (tiles == 2 ? t : 0) * 128 + t_lane;
    const int tq = (tiles == 2 ? t : 0) * p.TQ + r / p.G, g = r % p.G;
    const bool row_valid = tq < n_tok && r < p.G * p.TQ;
    const int qpos = row_valid ? pos0 + tq : -1;
    const int row_lo = max(max(p.window > 0 ? qpos - p.window + 1 : 0, p.chunk > 0 ? max(qpos, 0) / p.chunk * p.chunk : 0), kv_begin);
    const int row_hi = row_valid ? min(kv_end, p.causal ? qpos + 1 : kv_end) : -1;
    const int n_mine = tiles == 2 ? n_tiles : (n_tiles + 1 - t) / 2;
    float m_used, l_run, f0 = 1.f, f1 = 0.f;
    if (n_mine > 0)
      prompt::softmax_role<T, D, CAP>(bars, t, tmem_base + t * 128 + t_lane, tmem_base + 256 + t * 128 + t_lane, n_mine,
                                      (tile_lo + (tiles == 2 ? 0 : t)) * TILE_N, tiles == 2 ? TILE_N : 2 * TILE_N, row_lo, row_hi, p.sm, CAP, budget,
                                      m_used, l_run);
    if (shared && t == 1) prompt::hand_over(ml, r, m_used, l_run);
    if (tiles == 2 || t == 0) {
    if (shared) prompt::take_over(ml, r, m_used, l_run, f0, f1);
    // ---- epilogue
    const int64_t tok = q0 + tok0 + tq;
    const int hq = h * p.G + g;
    float inv = l_run > 0.f ? 1.f / l_run : 0.f;
    if (p.num_splits == 1) {
      if (p.sinks && row_valid) {                    // the sink joins the denominator once, behind the last key
        const float sink = p.sinks[hq] * 1.4426950408889634f;
        const float top = fmaxf(m_used, sink), f = ex2(m_used - top);
        l_run = l_run * f + ex2(sink - top);
        m_used = top;
        inv = f / l_run;
      }
      inv *= p.out_scale;
      T* orow = reinterpret_cast<T*>(p.out) + tok * p.out_stride + (int64_t)hq * D;
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        prompt::load_o(t_o, c, shared, f0, f1, v);
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 o;
            o.x = pack2<T>(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv);
            o.y = pack2<T>(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
            o.z = pack2<T>(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv);
            o.w = pack2<T>(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c + i) = o;
          }
        }
      }
      if (row_valid && p.lse_out)
        p.lse_out[tok * p.Hq + hq] = l_run > 0.f ? (m_used + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
    } else {
      const int64_t pi = (tok * p.Hq + hq) * p.num_splits + split;
      float* orow = p.part_out + pi * D;
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        prompt::load_o(t_o, c, shared, f0, f1, v);
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(orow + c + i) =
                make_float4(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv,
                            __uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
        }
      }
      if (row_valid) p.part_lse[pi] = l_run > 0.f ? m_used + log2f(l_run) : -INFINITY;
    }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
  if (budget < 0 && p.error) *p.error = 1;
}

template <typename T, int DD>
__global__ void __launch_bounds__(DD) split_reduce(const float* __restrict__ part_out, const float* __restrict__ part_lse,
                                                   T* __restrict__ out, float* __restrict__ lse_out, int Hq, int S,
                                                   int64_t out_stride, const float* __restrict__ sinks, float out_scale) {
  const int tok = blockIdx.x, hq = blockIdx.y, d = threadIdx.x;
  const int64_t base = ((int64_t)tok * Hq + hq) * S;
  const float sink = sinks ? sinks[hq] * 1.4426950408889634f : -INFINITY;
  float m = sink;
  for (int s = 0; s < S; ++s) m = fmaxf(m, part_lse[base + s]);
  const float m_use = (m == -INFINITY) ? 0.f : m;
  float den = sinks ? ex2(sink - m_use) : 0.f, o = 0.f;
  for (int s = 0; s < S; ++s) {
    const float wgt = ex2(part_lse[base + s] - m_use);
    den += wgt;
    o += wgt * part_out[(base + s) * DD + d];
  }
  out[(int64_t)tok * out_stride + (int64_t)hq * DD + d] = from_f32<T>(den > 0.f ? o / den * out_scale : 0.f);
  if (lse_out && d == 0) lse_out[(int64_t)tok * Hq + hq] = den > 0.f ? (m + log2f(den)) * 0.6931471805599453f : -INFINITY;
}

template <typename T, bool CAP>
static int launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const Params& p, dim3 grid, cudaStream_t st) {
  const int smem = 2 * Q_BYTES + KV_STAGES * (K_BYTES + V_BYTES) + (int)sizeof(Bars) + TILE_M * 8 + 16 + 2 * MAX_TILES_SMEM * 4 + 1024;
  auto k = fmha_kernel<T, CAP>;
  static bool a = false;
  if (!a) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); a = true; }
  vb_launch(k, grid, dim3(NUM_THREADS), (size_t)smem, st, tq, tk, tv, p);
  return (int)cudaGetLastError();
}

}  // namespace fmha

// kv_cache: [nb, 2, Hkv, BS*D] with K pages [BS, D] and V pages stored transposed [D, BS].
// flat != 0 (varlen only): the grid is sized from (T_total, B) alone — T_total / TQ + B tiles bound every split of
// T_total tokens over B requests — so one captured launch serves any mixed batch of that bucket.
// in_order != 0: a row's result does not depend on the size of the batch or on where its portion begins.
EXPORT int vb_fmha_tc4(const void* q, const void* kv_cache, int64_t num_blocks, const int* block_table,
                       const int* seq_lens, const int* qsl, void* out, float* part_out, float* part_lse,
                       float* lse_out, int* error, int B, int T_total, int max_q_len, int Hq, int Hkv, int64_t q_stride,
                       int64_t out_stride, int bt_stride, int num_splits, int window, float scale, float soft_cap, int causal,
                       int flat, int chunk, const float* sinks, float out_scale, int in_order, int num_sms, int dtype, cudaStream_t st) {
  using namespace fmha;
  if (B == 0) return 0;
  if (dtype == DT_F32) return -1;
  const int G = Hq / Hkv;
  if (G > 128 || 128 % G != 0) return -4;
  auto enc = get_encode();
  if (!enc) return -10;
  const bool bf16 = dtype == DT_BF16;
  const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  Params p;
  p.block_table = block_table; p.seq_lens = seq_lens; p.qsl = qsl; p.out = out; p.part_out = part_out;
  p.part_lse = part_lse; p.lse_out = lse_out; p.out_stride = out_stride; p.bt_stride = bt_stride; p.Hq = Hq;
  p.Hkv = Hkv; p.G = G; p.TQ = qsl ? TILE_M / G : 1; p.num_splits = qsl ? 1 : num_splits; p.window = window;
  p.causal = causal; p.sm.scale_log2 = scale * 1.4426950408889634f;
  p.sm.ku = soft_cap > 0.f ? scale / soft_cap : 0.f; p.sm.c2 = soft_cap * 1.4426950408889634f;
  p.flat_B = (flat && qsl) ? B : 0;
  p.chunk = chunk; p.sinks = sinks; p.out_scale = out_scale; p.error = error;
  p.in_order = in_order && qsl;
  p.tiles = p.in_order || (qsl && (int64_t)T_total * Hq / TILE_M >= prompt::PAIR_MIN_TILES * num_sms) ? 2 : 1;
  CUtensorMap tq, tk, tv;
  {  // q: [T, Hq, D] with token stride q_stride; box {64, G, TQ}
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)Hq, (cuuint64_t)T_total};
    cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)q_stride * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)p.TQ};
    cuuint32_t es[3] = {1, 1, 1};
    if (enc(&tq, dt, 3, const_cast<void*>(q), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -11;
  }
  {  // K view: [nb*2*Hkv*BS, D], box {64 cols, 64 rows}
    cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)num_blocks * 2 * Hkv * BS};
    cuuint64_t strides[1] = {(cuuint64_t)D * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)BS};
    cuuint32_t es[2] = {1, 1};
    if (enc(&tk, dt, 2, const_cast<void*>(kv_cache), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -12;
  }
  {  // V view: [nb*2*Hkv*D, BS], box {64 cols (tokens), 128 rows (dims)}
    cuuint64_t dims[2] = {(cuuint64_t)BS, (cuuint64_t)num_blocks * 2 * Hkv * D};
    cuuint64_t strides[1] = {(cuuint64_t)BS * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)D};
    cuuint32_t es[2] = {1, 1};
    if (enc(&tv, dt, 2, const_cast<void*>(kv_cache), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -13;
  }
  const int TC = p.TQ * p.tiles;
  dim3 grid = qsl ? dim3((max_q_len + TC - 1) / TC, Hkv, B) : dim3(p.num_splits, Hkv, B);
  if (p.flat_B) grid = dim3(T_total / TC + B, Hkv, 1);
  int rc = bf16 ? (soft_cap > 0.f ? launch<__nv_bfloat16, true>(tq, tk, tv, p, grid, st) : launch<__nv_bfloat16, false>(tq, tk, tv, p, grid, st))
                : (soft_cap > 0.f ? launch<__half, true>(tq, tk, tv, p, grid, st) : launch<__half, false>(tq, tk, tv, p, grid, st));
  if (rc) return rc;
  if (!qsl && p.num_splits > 1) {
    if (bf16) split_reduce<__nv_bfloat16, D><<<dim3(B, Hq), D, 0, st>>>(part_out, part_lse, (__nv_bfloat16*)out, lse_out, Hq, p.num_splits, out_stride, sinks, out_scale);
    else split_reduce<__half, D><<<dim3(B, Hq), D, 0, st>>>(part_out, part_lse, (__half*)out, lse_out, Hq, p.num_splits, out_stride, sinks, out_scale);
  }
  return (int)cudaGetLastError();
}
