// Grouped GEMM of prompt-sized expert batches on tcgen05:  Y[r, :] = X[r, :] · W[e(r)]^T  for rows sorted by expert; gated:
// Y[r, n] = act(X[r, :] · W[e, n]^T) * (X[r, :] · W[e, I + n]^T), the activation in 32 bits between the accumulator and the one rounding.
//
// The swap-AB kernel of gemm_tc.cu (weights on the MMA's M axis, 16..128 tokens on N) is made for decode steps, where the weight stream is the
// cost; with hundreds of rows per expert it is bound by its 128 x 128 tiles' operand traffic and its transposed 2-byte stores.  Here a CTA
// takes tiles of 128 rows x 256 columns (two accumulators of 256 columns fill tensor memory), rows are stored 16 bytes at a time, and the epilogue of a
// tile runs while the next tile's products do.  Persistent: every CTA walks the (expert, rows, 256 columns) tiles with a stride of the grid, columns
// first, so that neighbours share rows.
// Bound by the operands' way from L2: 48 KB per 64-deep step of a tile were 59 bytes per cycle and SM and kept the tensor core busy for 64 % of the cycles.
// PAIR: two CTAs take 256 rows (cta_group::2), each brings its 128 and half of the columns, 32 KB per step.  The price is the rows that fill up an
// expert's last 256; both measured at vb_gemm_grouped.
// Warps: 0 TMA producer, 1 MMA issuer (pairs: of the first CTA), 2..5 epilogue (thread = row).
#include "act.cuh"
#include "pair_mma.cuh"
#include "cluster.cuh"

namespace gg {

constexpr int TM = 128, TN = 256, BK = 64;
constexpr int NUM_THREADS = 192;
constexpr int A_BYTES = TM * BK * 2, HALF = TN / 2 * BK * 2;       // a CTA's rows, half of the columns
constexpr int MAX_E = 512;

struct Params {
  void* y;                 // [R, N] or, gated, [R, I]
  const int* offs;         // [E + 1]
  int E, N, K;             // N: rows of an expert's weight (gated: 2 I)
  int cols;                // output columns: N or I
  int col_tiles;           // of 256, gated: of 128
  int second;              // weight rows between the two halves of a tile: 128 or I
  int act;
  int* error;
};

template <bool PAIR> constexpr int stages() { return PAIR ? 6 : 4; }
template <bool PAIR> constexpr int stage_bytes() { return A_BYTES + (PAIR ? HALF : 2 * HALF); }

template <typename T, bool GATED, bool PAIR>
__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const Params p) {
  constexpr int STAGES = stages<PAIR>(), STAGE = stage_bytes<PAIR>(), PM = PAIR ? 2 * TM : TM;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);          // (a pair's first CTA's counts the bytes of both)
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;       // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2] (a pair's first CTA's: the epilogue warps of both)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* first = reinterpret_cast<int*>(tmem_slot + 2);          // [E + 1] row tiles before each expert
  int* offs = first + MAX_E + 1;                               // [E + 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = PAIR ? (int)cluster_ctarank() : 0;
  const int start = PAIR ? blockIdx.x / 2 : blockIdx.x, step = PAIR ? gridDim.x / 2 : gridDim.x;
  int budget = MBAR_BUDGET;                  // failed polls left (mbar_wait_lim)

  pdl_trigger();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_x); tma_prefetch_desc(&tmap_w);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], PAIR ? 8 : 4); }
    mbar_fence_init();
  }
  if (warp == 1) { if constexpr (PAIR) tmem2_alloc(tmem_slot, 512); else tmem_alloc(tmem_slot, 512); }
  pdl_wait();
  if (warp == 2) {
    int before = 0;
    for (int base = 0; base < p.E; base += 32) {
      const int e = base + lane;
      const int lo = e <= p.E ? p.offs[e] : 0, hi = e < p.E ? p.offs[e + 1] : lo;
      int n = (hi - lo + PM - 1) / PM, inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (e < p.E) { first[e] = before + inc - n; offs[e] = lo; if (e == p.E - 1) { first[p.E] = before + inc; offs[p.E] = hi; } }
      before += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int tiles = first[p.E] * p.col_tiles, nkb = (p.K + BK - 1) / BK;
  // tile → this CTA's first row, its rows (none or fewer, maybe), expert, column tile
  auto find = [&](int t, int& row, int& rows, int& e, int& n) {
    const int m = t / p.col_tiles;
    n = t - m * p.col_tiles;
    int lo = 0, hi = p.E;                    // the last expert whose first tile is <= m has it
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first[mid] <= m) lo = mid; else hi = mid;
    }
    e = lo;
    row = offs[e] + (m - first[e]) * PM + rank * TM;
    rows = min(TM, offs[e + 1] - row);
  };

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int t = start; t < tiles && budget >= 0; t += step) {
        int row, rows, e, n;
        find(t, row, rows, e, n);
        const int w0 = e * p.N + n * (GATED ? TN / 2 : TN) + rank * p.second;
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int s = it % STAGES;
          mbar_wait_lim(&empty[s], ((it / STAGES) & 1) ^ 1, budget);
          if (budget < 0) break;
          unsigned char* a = smem + s * STAGE;
          if constexpr (PAIR) {
            if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE);
            const uint32_t bar = dsmem_addr(smem_u32(&full[s]), 0);
            tma2_load_2d(a, &tmap_x, kb * BK, row, bar);
            tma2_load_2d(a + A_BYTES, &tmap_w, kb * BK, w0, bar);
          } else {
            mbar_expect_tx(&full[s], STAGE);
            tma_load_2d(a, &tmap_x, kb * BK, row, &full[s]);
            tma_load_2d(a + A_BYTES, &tmap_w, kb * BK, w0, &full[s]);
            tma_load_2d(a + A_BYTES + HALF, &tmap_w, kb * BK, w0 + p.second, &full[s]);
          }
        }
      }
      if (budget < 0 && rank == 0)           // let the copies in flight land before the block (the pair) gives up its memory
        mbar_let_land(full, STAGES);
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(PM, TN, DTypeOf<T>::v == DT_BF16);
    const uint64_t d0 = umma_desc_sw128(smem);
    int it = 0, i = 0;
    for (int t = rank == 0 ? start : tiles; t < tiles; t += step, ++i) {
      const int buf = i & 1;
      wait_cluster_lim(&acc_empty[buf], ((i >> 1) & 1) ^ 1, budget);
      tc_fence_after();
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int s = it % STAGES;
        mbar_wait_lim(&full[s], (it / STAGES) & 1, budget);
        tc_fence_after();
        __syncwarp();
        {
          const uint64_t da = d0 + (uint64_t)((s * STAGE) >> 4), db = da + (uint64_t)(A_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            if constexpr (PAIR) umma2_f16(tmem_base + buf * TN, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0);
            else warp_umma_f16(tmem_base + buf * TN, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0);
          }
          if constexpr (PAIR) umma2_commit(&empty[s]); else warp_umma_commit(&empty[s]);
          if (kb == nkb - 1) { if constexpr (PAIR) umma2_commit(&acc_full[buf]); else warp_umma_commit(&acc_full[buf]); }
        }
        __syncwarp();
      }
    }
  } else {
    const int q = warp & 3, r = q * 32 + lane;
    T* y = reinterpret_cast<T*>(p.y);
    const uint32_t drained = PAIR ? dsmem_addr(smem_u32(acc_empty), 0) : 0;
    int i = 0;
    for (int t = start; t < tiles; t += step, ++i) {
      int row, rows, e, n;
      find(t, row, rows, e, n);
      const int buf = i & 1, c0 = n * (GATED ? TN / 2 : TN);
      const uint32_t acc = tmem_base + buf * TN + ((uint32_t)(q * 32) << 16);
      mbar_wait_lim(&acc_full[buf], (i >> 1) & 1, budget);
      __syncwarp();
      tc_fence_after();
      T* out = y + (int64_t)(row + r) * p.cols + c0;
      const bool mine = r < rows;
#pragma unroll 1
      for (int c = 0; c < (GATED ? TN / 2 : TN); c += 32) {
        uint32_t v[32], u[32];
        tmem_ld_32x32(acc + c, v);
        if (GATED) tmem_ld_32x32(acc + TN / 2 + c, u);
        tmem_ld_wait();
        if (GATED) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float g = __uint_as_float(v[j]);
            const float a = p.act == ACT_SILU ? act_fn<ACT_SILU>(g) : p.act == ACT_GELU ? act_fn<ACT_GELU>(g) : act_fn<ACT_GELU_TANH>(g);
            v[j] = __float_as_uint(a * __uint_as_float(u[j]));
          }
        }
        if (mine) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (c0 + c + j >= p.cols) break;                   // cols is a multiple of 8
            uint4 o;
            o.x = pack2<T>(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
            o.y = pack2<T>(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
            o.z = pack2<T>(__uint_as_float(v[j + 4]), __uint_as_float(v[j + 5]));
            o.w = pack2<T>(__uint_as_float(v[j + 6]), __uint_as_float(v[j + 7]));
            *reinterpret_cast<uint4*>(out + c + j) = o;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { if constexpr (PAIR) arrive_cluster(drained + buf * 8); else mbar_arrive(&acc_empty[buf]); }
    }
  }
  __syncwarp();
  tc_fence_before();
  if constexpr (PAIR) cluster_sync();        // nobody leaves while the other CTA may still arrive on its barriers or bring its rows
  else __syncthreads();
  if (warp == 1) { if constexpr (PAIR) tmem2_dealloc(tmem_base, 512); else tmem_dealloc(tmem_base, 512); }
  if (budget < 0 && p.error) *p.error = 1;
}

// row-major [rows, cols], box = 128 rows of 64 values
static int tmap(CUtensorMap* m, const void* ptr, int64_t rows, int cols, bool bf16) {
  auto enc = get_encode();
  if (!enc) return -10;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {BK, 128};
  cuuint32_t es[2] = {1, 1};
  return enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -11;
}

template <typename T, bool GATED, bool PAIR>
static int launch(const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int ctas, cudaStream_t st) {
  const int smem = stages<PAIR>() * (stage_bytes<PAIR>() + 16) + 4 * 8 + 8 + 2 * (MAX_E + 1) * 4 + 1024;
  auto k = grouped_kernel<T, GATED, PAIR>;
  static bool a = false;
  if (!a) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); a = true; }
  vb_launch_parts(k, dim3(ctas), dim3(NUM_THREADS), (size_t)smem, st, PAIR ? 2u : 1u, tx, tw, p);
  return (int)cudaGetLastError();
}

}  // namespace gg

// x [R, K] rows sorted by expert (offs[e] .. offs[e + 1]), w [E, N, K]; act < 0: y [R, N]; act 0 silu, 1 gelu, 2 gelu by tanh: w's rows are
// N / 2 gates and N / 2 ups, y [R, N / 2].  K and y's columns are multiples of 8.
EXPORT int vb_gemm_grouped(const void* x, const void* w, void* y, const int* offs, int* error, int R, int N, int K, int E, int act, int num_sms,
                           int dtype, cudaStream_t st) {
  using namespace gg;
  if (R == 0) return 0;
  const bool gated = act >= 0;
  const int cols = gated ? N / 2 : N;
  if (dtype == DT_F32 || K % 8 || cols % 8 || (gated && (N % 2 || act > 2)) || E < 1 || E > MAX_E) return -1;
  const bool bf16 = dtype == DT_BF16;
  CUtensorMap tx, tw;
  int rc;
  if ((rc = tmap(&tx, x, R, K, bf16)) || (rc = tmap(&tw, w, (int64_t)E * N, K, bf16))) return rc;
  Params p;
  p.y = y; p.offs = offs; p.E = E; p.N = N; p.K = K; p.cols = cols; p.act = act; p.error = error;
  const int width = gated ? TN / 2 : TN;
  p.col_tiles = (cols + width - 1) / width;
  p.second = gated ? cols : TN / 2;
  // Pairs where their tiles of 256 rows, at 0.88 of the time of two of 128, take an expert of average size less time.  us of the gated product with 2048 x
  // 768 and its second one, 32 experts, 128 and 256 rows: 75 rows each 66 + 25 and 66 + 27, 131 rows 75 + 29 and 66 + 30, 1293 rows 232 + 144 and
  // 222 + 133; 8 experts of 2048 x 2048, 1725 rows 202 + 103 and 183 + 93 (1.26 PFLOP/s); 128 of 768, 87 rows 167 + 78 and 188 + 96, 356 rows
  // 322 + 184 and 335 + 196, 431 rows 383 + 227 and 341 + 203.
  const int64_t avg = ((int64_t)R + E - 1) / E;
  const bool pair = num_sms >= 2 && (avg + 255) / 256 * 256 * 88 < (avg + 127) / 128 * 128 * 100;
  const int rows = pair ? 2 * TM : TM;
  const int64_t most = (int64_t)(R / rows + (E < R ? E : R)) * p.col_tiles;      // tiles there can be
  if (most > INT32_MAX / 2) return -6;
  const int ctas = pair ? 2 * (most < num_sms / 2 ? (int)most : num_sms / 2) : most < num_sms ? (int)most : num_sms;
  DISPATCH_HALF(dtype, TT, {
    if (pair) return gated ? launch<TT, true, true>(tx, tw, p, ctas, st) : launch<TT, false, true>(tx, tw, p, ctas, st);
    return gated ? launch<TT, true, false>(tx, tw, p, ctas, st) : launch<TT, false, false>(tx, tw, p, ctas, st);
  });
}
