// Latent-attention prefill on tcgen05: causal multi-head attention of a step's prompt portions over keys and values that
// were expanded from the latent cache (K = W_uk c, V = W_uv c, two GEMMs over the portion's whole context).
//
// Expanding costs one GEMM per layer but a score then takes `dim` multiplications instead of the latent width, and a
// value row `vdim`: for prompts that is several times fewer FLOPs than attending in the latent space (mla_decode.cu),
// which in turn never writes K / V and so is the better form for a handful of query tokens.
//
//   Q [T, H, dim]  K [KV, h, dim]  V [KV, h, vdim]   plain row-major GEMM outputs — no pages, no transposed copy:
//   S = Q · K^T    both operands K-major (dims contiguous), 128 x 128 tile, dim in 64-wide k-blocks
//   O += P · V     V is read as an MN-major B operand: a 128-byte swizzle row holds 64 dims of ONE token
// dim and vdim are multiples of 8 up to 128; TMA zero-fills the tail of a 64-wide block, so odd widths cost nothing else.
// A rotated part of the score (up to 64 wide, one key part for all heads) is one more k-block: its queries are columns of the query
// heads, its keys columns of the gathered cache rows, so nothing is copied together.  With a window, the request's key rows start at
// the first one that its portion sees.
//
// CTA = (request, head, one or two tiles of 128 query tokens), heaviest (latest) query tiles first.  Warps: 0 TMA producer, 1 MMA
// issuer + TMEM owner, 4..7 and 8..11 softmax and epilogue of the two tiles (attention_prompt.cuh).  Two stages of keys; two of values where
// they fit beside two query tiles (not with a rotated part behind 128 unrotated dimensions: one, whose load hides behind the second tile).
// Measured: 16 heads of 128 + 64, eight prompts of 860 tokens, weights in two parts: 105 us (attending in the latent space on the CUDA cores,
// in 32 bits: 15.8 ms).
#include "attention_prompt.cuh"

namespace mlap {

using prompt::BLK;
using prompt::tma_load_3d;
constexpr int TM = prompt::ROWS, TN = prompt::KEYS;
constexpr int NUM_THREADS = prompt::NUM_THREADS;
constexpr int KS = 2;

struct Params {
  const int* q_start;      // [B] first row of the request's portion in q / out
  const int* q_len;        // [B] rows of the portion
  const int* seq_len;      // [B] keys of the request (the portion is its tail)
  const int* kv_start;     // [B] first key row of the request in K / V
  void* out;               // [T, H, vdim]
  int64_t out_st, out_sh;
  int h0;                  // first head of this launch in q / out (K and V hold the launch's heads only)
  int vdim;
  int window;              // > 0: a query sees its last `window` keys
  int tiles;               // query tiles per CTA: 1 or 2
  int in_order;            // a row's keys are added in their order, whatever else is in the batch
  int split;               // weights keep 16 more bits
  prompt::Softmax sm;
  int* error;
};

// MN-major SW128 operand: 128-byte rows of 64 N-values (dims) of one K-value (token), 8 tokens per 1024-byte atom (SBO),
// the next 64 dims one block further (LBO)
VB_DEVICE uint64_t desc_mn(const void* smem_tile) {
  const uint32_t addr = smem_u32(smem_tile);
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((BLK >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// NN blocks of unrotated and NR of rotated dimensions; VS stages of values
template <typename T, int NN, int NR, int NV, int VS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
mla_prefill_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_qr,
                   const __grid_constant__ CUtensorMap tmap_kr, const Params p) {
  constexpr int NQ = NN + NR;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* q_smem = smem;                             // 2 x NQ blocks
  unsigned char* k_smem = q_smem + 2 * NQ * BLK;            // KS x NQ blocks
  unsigned char* v_smem = k_smem + KS * NQ * BLK;           // VS x NV blocks
  typedef prompt::Bars<KS, VS> Bars;
  Bars& bars = *reinterpret_cast<Bars*>(v_smem + VS * NV * BLK);
  float2* ml = reinterpret_cast<float2*>(&bars + 1);        // [TM]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ml + TM);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int budget = MBAR_BUDGET;                    // failed polls left (mbar_wait_lim)
  const int b = blockIdx.z, h = blockIdx.y;
  pdl_trigger();
  pdl_wait();
  const int q_len = p.q_len[b];
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int tok0 = qt * TM * p.tiles;
  if (tok0 >= q_len) return;                                // uniform over the CTA
  const int n_tok = min(TM * p.tiles, q_len - tok0);
  const int tiles = n_tok > TM || p.in_order ? 2 : 1;
  const int q0 = p.q_start[b] + tok0;
  const int kv0 = p.kv_start[b];
  const int pos0 = p.seq_len[b] - q_len + tok0;             // position of the first tile's first query
  const int kv_end = pos0 + n_tok;                          // keys any query of the CTA can see
  const int tile_lo = p.window > 0 ? max(0, pos0 - p.window + 1) / TN : 0;
  const int n_tiles = (kv_end + TN - 1) / TN - tile_lo;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
    bars.init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    prompt::regs_dec<prompt::REGS_AUX>();
    if (warp == 0 && lane == 0) {
      // ===== TMA producer.  Boxes are always whole: rows past the buffer read as zeros, rows of the next request are
      // masked by the softmax (finite values times a weight of 0).
      mbar_expect_tx(&bars.q_full, tiles * NQ * BLK);
      for (int t = 0; t < tiles; ++t) {
        unsigned char* qs = q_smem + t * NQ * BLK;
#pragma unroll
        for (int i = 0; i < NN; ++i) tma_load_3d(qs + i * BLK, &tmap_q, i * 64, p.h0 + h, q0 + t * TM, &bars.q_full);
        if (NR) tma_load_3d(qs + NN * BLK, &tmap_qr, 0, p.h0 + h, q0 + t * TM, &bars.q_full);
      }
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % KS, vs = j % VS;
        const int row = kv0 + (tile_lo + j) * TN;
        mbar_wait_lim(&bars.k_empty[s], ((j / KS) & 1) ^ 1, budget);
        if (budget < 0) break;
        mbar_expect_tx(&bars.k_full[s], NQ * BLK);
#pragma unroll
        for (int i = 0; i < NN; ++i) tma_load_3d(k_smem + (s * NQ + i) * BLK, &tmap_k, i * 64, h, row, &bars.k_full[s]);
        if (NR) tma_load_3d(k_smem + (s * NQ + NN) * BLK, &tmap_kr, 0, 0, row, &bars.k_full[s]);
        mbar_wait_lim(&bars.v_empty[vs], ((j / VS) & 1) ^ 1, budget);
        if (budget < 0) break;
        mbar_expect_tx(&bars.v_full[vs], NV * BLK);
#pragma unroll
        for (int i = 0; i < NV; ++i) tma_load_3d(v_smem + (vs * NV + i) * BLK, &tmap_v, i * 64, h, row, &bars.v_full[vs]);
      }
      if (budget < 0) bars.drain();
    } else if (warp == 1) {
      // ===== MMA issuer
      const bool bf16 = DTypeOf<T>::v == DT_BF16;
      const uint32_t idesc_s = umma_idesc_f16(TM, TN, bf16);
      const uint32_t idesc_o = umma_idesc_f16(TM, NV * 64, bf16) | (1u << 16);      // bit 16: B operand is MN-major
      const uint64_t d_q = umma_desc_sw128(q_smem), d_k = umma_desc_sw128(k_smem), d_v = desc_mn(v_smem);
      const bool split = p.split != 0;
      prompt::mma_role(
          bars, n_tiles, tiles == 2, budget,
          [&](int t, int s) {
            const int qt = tiles == 2 ? t : 0;
#pragma unroll
            for (int kb = 0; kb < NQ; ++kb)
#pragma unroll
              for (int k = 0; k < 4; ++k)
                warp_umma_f16(tmem_base + t * 128, d_q + (uint64_t)(((qt * NQ + kb) * BLK + k * 32) >> 4),
                         d_k + (uint64_t)(((s * NQ + kb) * BLK + k * 32) >> 4), idesc_s, (kb | k) != 0);
          },
          [&](int t, int s, int, bool first) {              // 16 keys per MMA: 16 rows of 128 bytes of V
            prompt::issue_pv(tmem_base + 256 + t * 128, tmem_base + t * 128, idesc_o, first, split, 0, TN / 16,
                             [&](int kk) { return d_v + (uint64_t)((s * NV * BLK + kk * 2048) >> 4); });
          });
    }
  } else {
    prompt::regs_inc<prompt::REGS_SOFTMAX>();
    // ===== softmax / rescale / epilogue: thread = query row = TMEM lane
    const int t = (warp >> 2) - 1, qd = warp & 3, row = qd * 32 + lane;
    const bool shared = tiles == 1 && n_tiles > 1;          // both warpgroups at one tile
    const int r = (tiles == 2 ? t : 0) * TM + row;
    const uint32_t t_lane = (uint32_t)(qd * 32) << 16, t_o = tmem_base + 256 + (tiles == 2 ? t : 0) * 128 + t_lane;
    const bool row_valid = r < n_tok;
    const int hi = row_valid ? pos0 + r + 1 : -1;
    const int lo = p.window > 0 ? max(hi - p.window, 0) : 0;
    const int n_mine = tiles == 2 ? n_tiles : (n_tiles + 1 - t) / 2;
    float m_used, l_run, f0 = 1.f, f1 = 0.f;
    if (n_mine > 0)
      prompt::softmax_role<T, NV * 64, false>(bars, t, tmem_base + t * 128 + t_lane, tmem_base + 256 + t * 128 + t_lane, n_mine,
                                              (tile_lo + (tiles == 2 ? 0 : t)) * TN, tiles == 2 ? TN : 2 * TN, lo, hi, p.sm, p.split != 0, budget, m_used,
                                              l_run);
    if (shared && t == 1) prompt::hand_over(ml, row, m_used, l_run);
    if (tiles == 2 || t == 0) {
      if (shared) prompt::take_over(ml, row, m_used, l_run, f0, f1);
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      T* orow = reinterpret_cast<T*>(p.out) + (int64_t)(q0 + r) * p.out_st + (int64_t)(p.h0 + h) * p.out_sh;
#pragma unroll
      for (int c = 0; c < NV * 64; c += 32) {
        uint32_t v[32];
        prompt::load_o(t_o, c, shared, f0, f1, v);
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            if (c + i >= p.vdim) break;
            uint4 o;
            o.x = pack2<T>(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv);
            o.y = pack2<T>(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
            o.z = pack2<T>(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv);
            o.w = pack2<T>(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c + i) = o;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
  if (budget < 0 && p.error) *p.error = 1;
}

// [rows, heads, width] with row stride `rs` and head stride `hs` elements; box = 128 rows of 64 values of one head
static int tmap(CUtensorMap* m, const void* ptr, int width, int heads, int64_t rows, int64_t rs, int64_t hs, bool bf16) {
  auto enc = get_encode();
  if (!enc) return -10;
  cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)heads, (cuuint64_t)rows};
  cuuint64_t strides[2] = {(cuuint64_t)hs * 2, (cuuint64_t)rs * 2};
  cuuint32_t box[3] = {64, 1, 128};
  cuuint32_t es[3] = {1, 1, 1};
  return enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(ptr), dims,
             strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -11;
}

struct Maps { CUtensorMap q, k, v, qr, kr; };

template <typename T, int NN, int NR, int NV>
static int launch(const Maps& m, const Params& p, dim3 grid, cudaStream_t st) {
  constexpr int NQ = NN + NR;
  constexpr int VS = (2 + KS) * NQ + 2 * NV <= 14 ? 2 : 1;                    // what fits into shared memory
  const int smem = ((2 + KS) * NQ + VS * NV) * BLK + (int)sizeof(prompt::Bars<KS, VS>) + TM * 8 + 16 + 1024;
  auto k = mla_prefill_kernel<T, NN, NR, NV, VS>;
  static bool a = false;
  if (!a) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); a = true; }
  vb_launch(k, grid, dim3(NUM_THREADS), (size_t)smem, st, m.q, m.k, m.v, m.qr, m.kr, p);
  return (int)cudaGetLastError();
}

}  // namespace mlap

// q [T, H, dim + rot] and out [T, H, vdim] (row strides q_st / out_st); k [KV, hl, dim], v [KV, hl, vdim] (row and head strides free) hold
// the heads h0 .. h0 + hl - 1; k_pe [KV, rot] (row stride kr_st; rot = 0: none) is the rotated key part of all heads.  Request b owns query rows
// q_start[b] .. + q_len[b] and key rows kv_start[b] .. + seq_len[b], of which its portion is the tail.
EXPORT int vb_mla_prefill3(const void* q, const void* k, const void* v, const void* k_pe, void* out, const int* q_start, const int* q_len,
                          const int* seq_len, const int* kv_start, int* error, int B, int T_, int64_t KV, int H, int h0, int hl,
                          int dim, int rot, int vdim, int64_t q_st, int64_t k_st, int64_t k_sh, int64_t v_st, int64_t v_sh, int64_t kr_st,
                          int64_t out_st, int max_q, int window, float scale, int split, int in_order, int num_sms,
                          int dtype, cudaStream_t st) {
  using namespace mlap;
  if (B == 0 || T_ == 0 || max_q <= 0) return 0;
  if (dtype == DT_F32 || dim < 8 || dim > 128 || dim % 8 || vdim < 8 || vdim > 128 || vdim % 8 || rot < 0 || rot > 64 || rot % 8) return -1;
  if (q_st % 8 || k_st % 8 || v_st % 8 || k_sh % 8 || v_sh % 8 || out_st % 8 || h0 < 0 || h0 + hl > H || (rot && (!k_pe || kr_st % 8))) return -2;
  const bool bf16 = dtype == DT_BF16;
  Maps m;
  int rc;
  if ((rc = tmap(&m.q, q, dim, H, T_, q_st, dim + rot, bf16))) return rc;
  if ((rc = tmap(&m.k, k, dim, hl, KV, k_st, k_sh, bf16))) return rc;
  if ((rc = tmap(&m.v, v, vdim, hl, KV, v_st, v_sh, bf16))) return rc;
  m.qr = m.q; m.kr = m.k;
  if (rot) {
    if ((rc = tmap(&m.qr, reinterpret_cast<const char*>(q) + (int64_t)dim * 2, rot, H, T_, q_st, dim + rot, bf16))) return rc;
    if ((rc = tmap(&m.kr, k_pe, rot, 1, KV, kr_st, kr_st, bf16))) return rc;
  }
  Params p;
  p.q_start = q_start; p.q_len = q_len; p.seq_len = seq_len; p.kv_start = kv_start; p.out = out; p.out_st = out_st;
  p.out_sh = vdim; p.h0 = h0; p.vdim = vdim; p.window = window; p.sm.scale_log2 = scale * 1.4426950408889634f; p.sm.ku = p.sm.c2 = 0.f; p.split = split; p.error = error;
  p.in_order = in_order;
  p.tiles = in_order || (int64_t)(T_ / TM) * hl >= prompt::PAIR_MIN_TILES * num_sms ? 2 : 1;
  const dim3 grid((max_q + TM * p.tiles - 1) / (TM * p.tiles), hl, B);
  const int nq = (dim + 63) / 64, nv = (vdim + 63) / 64;
#define GV(TT, N, R) (nv == 1 ? launch<TT, N, R, 1>(m, p, grid, st) : launch<TT, N, R, 2>(m, p, grid, st))
#define GO(TT) (rot ? (nq == 1 ? GV(TT, 1, 1) : GV(TT, 2, 1)) : (nq == 1 ? GV(TT, 1, 0) : GV(TT, 2, 0)))
  return bf16 ? GO(__nv_bfloat16) : GO(__half);
#undef GO
#undef GV
}
