// Grouped GEMM of decode steps:  Y[r, :] = X[r, :] · W[e(r)]^T  for a few rows per expert, sorted by expert; gated: Y[r, n] = act(X[r, :] · W[e, n]^T) *
// (X[r, :] · W[e, I + n]^T), the activation in 32 bits between the accumulator and the one rounding, or (`rounded`) between numbers that are rounded first:
// bit for bit what the product by tiles (gemm_tc.cu) and the activation behind it (norm_act.cu) give, so that neither a batch's size nor the choice of the
// kernel shows in a token's hidden row.
//
// Bound by the weights, which are read once.  gemm_tc.cu gives every tile of 128 weight rows a CTA, two to an SM: each begins with a look for its
// expert's rows and a first wait for memory and ends with a drain in which its half of the SM loads nothing.  Here a CTA stays on its SM
// and its ring of 160 KB and more runs through all its tiles: the tile to come is on its way while this one is multiplied and stored (two
// accumulators).  Tile i of the (expert, 128 rows) list belongs to CTA i mod grid.  Where nearly every expert has rows (`ahead`) the list is of all experts, so that a CTA
// knows its first tile before the router has chosen and asks for its weights ahead of the kernels before this one (a ring for an expert without rows is
// dropped); else it is of those with rows, which share the CTAs evenly.
// A gated tile is 64 gates and the 64 ups that belong to them.
// us of both products of gated experts, tiles → this → bytes at the rate of a copy: 144 rows of 2048 into 32 x 768 59 → 51 → 47; 32 rows into 8 x 2048
// 42 → 36 → 31; 128 rows of 1024 into 16 x 512 19 → 15 → 8 (start and end of two kernels); 512 rows into 128 x 768 192 → 179 → 184.  Rounding first
// costs nothing (51 either way).
// Warps: 0 TMA producer, 1 MMA issuer, 2..5 epilogue (thread = weight row).
#include "act.cuh"

namespace ge {

constexpr int TM = 128, BK = 64, A_BYTES = TM * BK * 2;
constexpr int NUM_THREADS = 192, MAX_E = 512, XCH = 32;      // XCH: tokens whose gates and ups change hands at a time

struct Params {
  void* y;                 // [R, N] or, gated, [R, I]
  const int* offs;         // [E + 1]
  int E, N, K;             // N: rows of an expert's weight (gated: 2 I)
  int tiles;               // per expert: of 128 rows, gated: of 64 + 64
  int second;              // weight rows between the two halves of a tile: 64 or I
  int act, rounded;
  int ahead;
  // sums (not gated): acc[token of row r, :] += weight of r * product, in 32 bits; a row's (token, slot) pair is row_pair[r]
  float* acc;
  const int* row_pair;
  const float* pair_w;
  int k, H;
  int* error;
};

VB_DEVICE void epilogue_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int BN> constexpr int stages() { return BN == 16 ? 10 : BN == 32 ? 9 : BN == 64 ? 8 : 6; }
template <int BN> constexpr int stage_bytes() { return A_BYTES + BN * BK * 2; }

template <typename T, int BN, bool GATED>
__global__ void __launch_bounds__(NUM_THREADS, 1)
experts_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const Params p) {
  constexpr int STAGES = stages<BN>(), STAGE = stage_bytes<BN>();
  constexpr uint32_t COLS = BN == 16 ? 32 : 2 * BN;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* xch = reinterpret_cast<float*>(smem + STAGES * STAGE);          // [XCH][128], gated
  uint64_t* full = reinterpret_cast<uint64_t*>(xch + (GATED ? XCH * TM : 0));
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;       // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* offs = reinterpret_cast<int*>(tmem_slot + 2);                     // [E + 1]
  int* list = offs + MAX_E + 1;                                          // [E] experts with rows, and how many
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int budget = MBAR_BUDGET;                  // failed polls left (mbar_wait_lim)
  const int nkb = (p.K + BK - 1) / BK, pre = p.ahead ? min(nkb, STAGES) : 0;      // (no CTA without a tile then)

  pdl_trigger();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w); tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 128); }
    mbar_fence_init();
  }
  auto weights = [&](int s, int kb, int e, int a) {
    unsigned char* dst = smem + s * STAGE;
    const int w0 = e * p.N + a * (GATED ? TM / 2 : TM);
    mbar_expect_tx(&full[s], STAGE);
    tma_load_2d_hint(dst, &tmap_w, kb * BK, w0, &full[s], L2_EVICT_FIRST);
    tma_load_2d_hint(dst + A_BYTES / 2, &tmap_w, kb * BK, w0 + p.second, &full[s], L2_EVICT_FIRST);
  };
  auto rows_of = [&](int s, int kb, int row) { tma_load_2d_hint(smem + s * STAGE + A_BYTES, &tmap_x, kb * BK, row, &full[s], L2_EVICT_LAST); };
  if (warp == 0 && lane == 0)
    for (int kb = 0; kb < pre; ++kb) weights(kb, kb, blockIdx.x / p.tiles, blockIdx.x % p.tiles);
  if (warp == 1) tmem_alloc(tmem_slot, COLS);
  pdl_wait();
  if (warp == 2) {
    int n = 0;
    for (int base = 0; base <= p.E; base += 32) {
      const int e = base + lane;
      const int lo = e <= p.E ? p.offs[e] : 0, hi = e < p.E ? p.offs[e + 1] : lo;
      const bool has = p.ahead ? e < p.E : hi > lo;
      const unsigned all = __ballot_sync(0xffffffffu, has);
      if (e <= p.E) offs[e] = lo;
      if (has) list[n + __popc(all & ((1u << lane) - 1u))] = e;
      n += __popc(all);
    }
    if (lane == 0) list[MAX_E] = n;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int total = list[MAX_E] * p.tiles;
  const bool drop = pre && offs[blockIdx.x / p.tiles] == offs[blockIdx.x / p.tiles + 1];

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      if (drop)
        for (; it < pre; ++it) rows_of(it, 0, 0);
      for (int t = blockIdx.x; t < total && budget >= 0; t += gridDim.x) {
        const int at = t / p.tiles, e = list[at], a = t - at * p.tiles, end = offs[e + 1];
        for (int row = offs[e]; row < end && budget >= 0; row += BN)
          for (int kb = 0; kb < nkb; ++kb, ++it) {
            const int s = it % STAGES;
            if (it >= pre) {
              mbar_wait_lim(&empty[s], ((it / STAGES) & 1) ^ 1, budget);
              if (budget < 0) break;
              weights(s, kb, e, a);
            }
            rows_of(s, kb, row);
          }
      }
      if (budget < 0)                        // let the copies in flight land before the block gives up its memory
        mbar_let_land(full, STAGES);
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(TM, BN, DTypeOf<T>::v == DT_BF16);
    const uint64_t d0 = umma_desc_sw128(smem);
    int it = 0, i = 0;
    if (drop)
      for (; it < pre; ++it) {
        mbar_wait_lim(&full[it], 0, budget);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[it]);
      }
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      const int e = list[t / p.tiles], end = offs[e + 1];
      for (int row = offs[e]; row < end; row += BN, ++i) {
        const int buf = i & 1;
        mbar_wait_lim(&acc_empty[buf], ((i >> 1) & 1) ^ 1, budget);
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int s = it % STAGES;
          mbar_wait_lim(&full[s], (it / STAGES) & 1, budget);
          tc_fence_after();
          __syncwarp();
          const uint64_t da = d0 + (uint64_t)((s * STAGE) >> 4), db = da + (uint64_t)(A_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) warp_umma_f16(tmem_base + buf * BN, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0);
          warp_umma_commit(&empty[s]);
          if (kb == nkb - 1) warp_umma_commit(&acc_full[buf]);
          __syncwarp();
        }
      }
    }
  } else {
    constexpr int CH = BN < 32 ? BN : 32;
    const int q = warp & 3, r = q * 32 + lane, et = threadIdx.x - 64;
    T* y = reinterpret_cast<T*>(p.y);
    int i = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      const int at = t / p.tiles, e = list[at], a = t - at * p.tiles, end = offs[e + 1];
      for (int row = offs[e]; row < end; row += BN, ++i) {
        const int buf = i & 1, rows = min(BN, end - row);
        const uint32_t acc = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
        mbar_wait_lim(&acc_full[buf], (i >> 1) & 1, budget);
        __syncwarp();
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < rows; c += CH) {
          float v[CH];
          {
            uint32_t u[CH];
            if constexpr (CH == 32) tmem_ld_32x32(acc + c, u);
            else tmem_ld_32x16(acc + c, u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < CH; ++j) v[j] = __uint_as_float(u[j]);
          }
          if constexpr (GATED) {
#pragma unroll
            for (int j = 0; j < CH; ++j) xch[j * TM + r] = v[j];
            epilogue_sync();
            const int n = et & 63, col = a * (TM / 2) + n;
            if (col < p.second)
              for (int j = et >> 6; j < min(CH, rows - c); j += 2) {
                float g = xch[j * TM + n], up = xch[j * TM + 64 + n];
                if (p.rounded) { g = to_f32(from_f32<T>(g)); up = to_f32(from_f32<T>(up)); }
                const float x = p.act == ACT_SILU ? act_fn<ACT_SILU>(g) : p.act == ACT_GELU ? act_fn<ACT_GELU>(g) : act_fn<ACT_GELU_TANH>(g);
                y[(int64_t)(row + c + j) * p.second + col] = from_f32<T>(x * up);
              }
            epilogue_sync();
          } else {
            const int n = a * TM + r;
            if (n < p.N) {
#pragma unroll
              for (int j = 0; j < CH; ++j)
                if (c + j < rows) {
                  if (p.acc) {
                    const int pair = p.row_pair[row + c + j];
                    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(p.acc + (int64_t)(pair / p.k) * p.H + n), "f"(v[j] * p.pair_w[pair]) : "memory");
                  } else {
                    y[(int64_t)(row + c + j) * p.N + n] = from_f32<T>(v[j]);
                  }
                }
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&acc_empty[buf]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, COLS);
  if (budget < 0 && p.error) *p.error = 1;
}

// row-major [rows, cols], box = some rows of 64 values
static int tmap(CUtensorMap* m, const void* ptr, int64_t rows, int cols, int box_rows, bool bf16) {
  auto enc = get_encode();
  if (!enc) return -10;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  return enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -11;
}

template <typename T, int BN, bool GATED>
static int launch(const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int ctas, cudaStream_t st) {
  const int smem = stages<BN>() * (stage_bytes<BN>() + 16) + (GATED ? XCH * TM * 4 : 0) + 4 * 8 + 8 + 2 * (MAX_E + 1) * 4 + 1024;
  auto k = experts_kernel<T, BN, GATED>;
  static bool a = false;
  if (!a) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); a = true; }
  vb_launch(k, dim3(ctas), dim3(NUM_THREADS), (size_t)smem, st, tw, tx, p);
  return (int)cudaGetLastError();
}

}  // namespace ge

// x [R, K] rows sorted by expert (offs[e] .. offs[e + 1]), w [E, N, K]; act < 0: y [R, N], or sums into acc where given; act 0 silu, 1 gelu, 2 gelu by
// tanh: w's rows are N / 2 gates and N / 2 ups (N / 2 a multiple of 64), y [R, N / 2]; rounded: gates and ups are rounded first.  bn: 16, 32, 64 or 128 rows of an expert at a time.
EXPORT int vb_gemm_experts(const void* x, const void* w, void* y, const int* offs, int* error, int R, int N, int K, int E, int bn, int act, int rounded, int ahead,
                           float* acc, const int* row_pair, const float* pair_w, int k, int H, int num_sms, int dtype, cudaStream_t st) {
  using namespace ge;
  if (R == 0) return 0;
  const bool gated = act >= 0;
  if (dtype == DT_F32 || K % 8 || K < 1 || N < 1 || (gated && (N % 128 || act > 2 || acc)) || E < 1 || E > MAX_E || (acc && (!row_pair || !pair_w || k < 1))) return -1;
  const bool bf16 = dtype == DT_BF16;
  CUtensorMap tw, tx;
  int rc;
  if ((rc = tmap(&tw, w, (int64_t)E * N, K, TM / 2, bf16)) || (rc = tmap(&tx, x, R, K, bn, bf16))) return rc;
  Params p;
  p.y = y; p.offs = offs; p.E = E; p.N = N; p.K = K; p.act = act; p.rounded = rounded; p.ahead = ahead; p.error = error;
  p.acc = acc; p.row_pair = row_pair; p.pair_w = pair_w; p.k = k; p.H = H;
  p.tiles = gated ? N / 128 : (N + TM - 1) / TM;
  p.second = gated ? N / 2 : TM / 2;
  if ((int64_t)E * p.tiles > INT32_MAX / 2) return -6;
  const int ctas = E * p.tiles < num_sms ? E * p.tiles : num_sms;
#define GO(BNV) DISPATCH_HALF(dtype, TT, return gated ? launch<TT, BNV, true>(tw, tx, p, ctas, st) : launch<TT, BNV, false>(tw, tx, p, ctas, st))
  switch (bn) {
    case 16: GO(16); break;
    case 32: GO(32); break;
    case 64: GO(64); break;
    case 128: GO(128); break;
    default: return -2;
  }
#undef GO
  return -2;
}
