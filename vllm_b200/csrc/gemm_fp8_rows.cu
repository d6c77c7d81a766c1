// Block-scaled fp8 GEMM of prompts:  Y[M, N] = sum_kb ws[n / 128, kb] xs[kb, m] (Xq[m, kb] · Wq[n, kb]),  tcgen05 kind::f8f6f4.
//
// The tile kernel of gemm_fp8.cu gives a CTA 128 x 128 outputs: one warpgroup promotes each 128-deep block's products into its registers,
// which takes longer than the block's products, and nothing runs beside a tile's fill, last promotion and stores.  Here a tile is 128
// tokens x 256 features: the tensor core is at a block for 512 cycles, in which two warpgroups promote 128 columns each of the block before
// (two blocks of 256 columns fill tensor memory), and 48 KB of operands feed twice the products.  Persistent, so the next tile's copies
// and its first two blocks run beside a tile's stores.  Tiles are taken down M in bands of BAND row tiles, so that a wave's operands stay in L2.
// Bound by the promotion's way out of tensor memory: 0.55 to 0.6 us per 128-deep block on a CTA alone as on all, the products take 0.27; with 32
// columns fetched at a time 0.65, whether or not the next were on their way, scales staged ahead made no difference.
// Measured against the tile kernel: 1000 x 28672 x 4096 199 → 139 us, 1000 x 4096 x 14336 109 → 70, 512 x 6144 x 4096 40 → 28, 8192 x 4096 x
// 14336 915 → 457 (2.1 PFLOP/s).
// Warps: 0 TMA producer, 1 MMA issuer, 4..7 and 8..11 promotion and stores of columns 0..127 and 128..255 (thread = token).
#include "attention_prompt.cuh"

namespace g8r {

constexpr int TM = 128, TN = 256, BK = 128, STAGES = 4, BAND = 16;
constexpr int NUM_THREADS = 384;
constexpr int REGS_AUX = 24, REGS_SUM = 240;    // 128 x 24 + 256 x 240 of the 384 x 168 registers at launch
constexpr int A_BYTES = TM * BK, B_BYTES = TN * BK, STAGE = A_BYTES + B_BYTES;

struct Params {
  void* y;                 // [M, N]
  const void* bias;        // [N] or null
  const float* xs;         // [blocks, xs_stride]: tokens next to each other
  const float* ws;         // [ceil(N / 128), blocks]
  int64_t xs_stride;
  int M, N, blocks, m_tiles, n_tiles;
  int* error;
};

VB_DEVICE uint64_t pack(uint32_t lo, uint32_t hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r; }
VB_DEVICE uint64_t pair(float x) { return pack(__float_as_uint(x), __float_as_uint(x)); }
VB_DEVICE uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r;
}

template <typename T>
__global__ void __launch_bounds__(NUM_THREADS, 1)
fp8_rows_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;       // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int budget = MBAR_BUDGET;                  // failed polls left (mbar_wait_lim)
  pdl_trigger();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_x); tma_prefetch_desc(&tmap_w);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 8); }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem_base = *tmem_slot;
  const int tiles = p.m_tiles * p.n_tiles;
  auto place = [&](int t, int& m0, int& n0) {
    const int band = t / (BAND * p.n_tiles), height = min(BAND, p.m_tiles - band * BAND), i = t - band * BAND * p.n_tiles;
    m0 = (band * BAND + i % height) * TM; n0 = i / height * TN;
  };

  if (warp < 4) {
    prompt::regs_dec<REGS_AUX>();
    if (warp == 0 && lane == 0) {
      int it = 0;
      for (int t = blockIdx.x; t < tiles && budget >= 0; t += gridDim.x) {
        int m0, n0;
        place(t, m0, n0);
        for (int kb = 0; kb < p.blocks; ++kb, ++it) {
          const int s = it % STAGES;
          mbar_wait_lim(&empty[s], ((it / STAGES) & 1) ^ 1, budget);
          if (budget < 0) break;
          unsigned char* a = smem + s * STAGE;
          mbar_expect_tx(&full[s], STAGE);
          tma_load_2d(a, &tmap_x, kb * BK, m0, &full[s]);
          tma_load_2d(a + A_BYTES, &tmap_w, kb * BK, n0, &full[s]);
          tma_load_2d(a + A_BYTES + B_BYTES / 2, &tmap_w, kb * BK, n0 + TN / 2, &full[s]);
        }
      }
      if (budget < 0)                        // let the copies in flight land before the block gives up its memory
        mbar_let_land(full, STAGES);
    } else if (warp == 1) {
      const uint32_t idesc = umma_idesc_f8(TM, TN);
      const uint64_t d0 = umma_desc_sw128(smem);
      int it = 0;
      for (int t = blockIdx.x; t < tiles; t += gridDim.x)
        for (int kb = 0; kb < p.blocks; ++kb, ++it) {
          const int s = it % STAGES, buf = it & 1;
          mbar_wait_lim(&acc_empty[buf], ((it >> 1) & 1) ^ 1, budget);
          mbar_wait_lim(&full[s], (it / STAGES) & 1, budget);
          tc_fence_after();
          __syncwarp();
          {
            const uint64_t da = d0 + (uint64_t)((s * STAGE) >> 4), db = da + (uint64_t)(A_BYTES >> 4);
#pragma unroll
            for (int k = 0; k < BK / 32; ++k) warp_umma_f8(tmem_base + buf * TN, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, k != 0);
            warp_umma_commit(&empty[s]);
            warp_umma_commit(&acc_full[buf]);
          }
          __syncwarp();
        }
    }
  } else {
    prompt::regs_inc<REGS_SUM>();
    const int half = (warp >> 2) - 1, q = warp & 3, r = q * 32 + lane;
    const uint32_t t_row = tmem_base + half * (TN / 2) + ((uint32_t)(q * 32) << 16);
    T* y = reinterpret_cast<T*>(p.y);
    int it = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      int m, n0;
      place(t, m, n0);
      m += r; n0 += half * (TN / 2);
      const bool rows = m < p.M, cols = n0 < p.N;
      const float* xp = p.xs + (rows ? m : 0);
      const float* wp = p.ws + (int64_t)(cols ? n0 / 128 : 0) * p.blocks;
      uint64_t acc[64];                      // pairs of neighbouring columns
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = 0;
      float xn = xp[0], wn = wp[0];
      for (int kb = 0; kb < p.blocks; ++kb, ++it) {
        const uint32_t t_buf = t_row + (it & 1) * TN;
        const uint64_t s = pair(xn * wn);
        if (kb + 1 < p.blocks) { xn = xp[(int64_t)(kb + 1) * p.xs_stride]; wn = wp[kb + 1]; }
        mbar_wait_lim(&acc_full[it & 1], (it >> 1) & 1, budget);
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 128; c += 64) {  // 64 columns on their way at a time
          uint32_t v[64];
          tmem_ld_32x32(t_buf + c, *reinterpret_cast<uint32_t (*)[32]>(v));
          tmem_ld_32x32(t_buf + c + 32, *reinterpret_cast<uint32_t (*)[32]>(v + 32));
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 64; ++j) asm volatile("" : "+r"(v[j]));      // no use moves in front of the wait
          if (c == 64) {                     // all of it is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[it & 1]);
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[c / 2 + j] = fma2(pack(v[2 * j], v[2 * j + 1]), s, acc[c / 2 + j]);
        }
      }
      if (rows && cols) {
        T* out = y + (int64_t)m * p.N + n0;
        const T* b = p.bias ? reinterpret_cast<const T*>(p.bias) + n0 : nullptr;
#pragma unroll
        for (int j = 0; j < 128; j += 8) {
          if (n0 + j >= p.N) break;          // N is a multiple of 8
          float o[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = __uint_as_float((uint32_t)(acc[(j + e) / 2] >> (e % 2 * 32))) + (b ? to_f32(b[j + e]) : 0.f);
          uint4 v;
          v.x = pack2<T>(o[0], o[1]); v.y = pack2<T>(o[2], o[3]); v.z = pack2<T>(o[4], o[5]); v.w = pack2<T>(o[6], o[7]);
          *reinterpret_cast<uint4*>(out + j) = v;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
  if (budget < 0 && p.error) *p.error = 1;
}

// row-major bytes [rows, cols], box = 128 rows of 128 bytes
static int tmap(CUtensorMap* m, const void* ptr, int64_t rows, int cols) {
  auto enc = get_encode();
  if (!enc) return -10;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols};
  cuuint32_t box[2] = {BK, 128};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -11;
}

template <typename T>
static int launch(const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int ctas, cudaStream_t st) {
  const int smem = STAGES * STAGE + (2 * STAGES + 4) * 8 + 16 + 1024;
  auto k = fp8_rows_kernel<T>;
  static bool a = false;
  if (!a) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); a = true; }
  vb_launch(k, dim3(ctas), dim3(NUM_THREADS), (size_t)smem, st, tx, tw, p);
  return (int)cudaGetLastError();
}

}  // namespace g8r

// xq [M, K], wq [N, K] e4m3 contiguous, xs [ceil(K / 128), xs_stride], ws [ceil(N / 128), ceil(K / 128)]; K a multiple of 16, N of 8
EXPORT int vb_gemm_fp8_rows(const void* xq, const float* xs, int64_t xs_stride, const void* wq, const float* ws, const void* bias, void* y, int* error,
                            int M, int N, int K, int num_sms, int dtype, cudaStream_t st) {
  using namespace g8r;
  if (M == 0) return 0;
  if (dtype == DT_F32 || K % 16 || N % 8 || K < 1) return -1;
  CUtensorMap tx, tw;
  int rc;
  if ((rc = tmap(&tx, xq, M, K)) || (rc = tmap(&tw, wq, N, K))) return rc;
  Params p;
  p.y = y; p.bias = bias; p.xs = xs; p.ws = ws; p.xs_stride = xs_stride; p.M = M; p.N = N; p.blocks = (K + BK - 1) / BK;
  p.m_tiles = (M + TM - 1) / TM; p.n_tiles = (N + TN - 1) / TN; p.error = error;
  const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;
  if (tiles > INT32_MAX / 2) return -6;
  const int ctas = tiles < num_sms ? (int)tiles : num_sms;
  return dtype == DT_BF16 ? launch<__nv_bfloat16>(tx, tw, p, ctas, st) : launch<__half>(tx, tw, p, ctas, st);
}
