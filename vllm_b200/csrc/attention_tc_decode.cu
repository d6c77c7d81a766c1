// Decode attention (one query row per request and head) over the tensor-core cache layout: K pages [64 tokens x 128], V pages stored transposed
// [128 x 64 tokens].
//
// A CTA takes one (request, kv head, part of the keys): one or two teams of four warps and a TMA producer, pages of 64 tokens in a ring.  The tokens
// are the rows of m16n8k16 products and the (at most 16) query rows of the kv head their columns, eight or sixteen.  A warp works for itself: of a
// page it takes 16 tokens through S^T = K Q^T, an own running maximum, P = 2^(S - m), turned in registers from the first product's result to
// the second one's operand, O^T += V^T P^T.  No barrier, no shared memory and no other warp between a page's arrival and its end; the warps'
// results are merged once, and those of a request's parts, a thread-block cluster, through distributed shared memory: no workspace, no second
// launch, the same order of additions in every run.
//
// What it costs is latency (launch, lengths, block table, first page, merging: 3 us), the bytes on their way (a page takes 1.6 us to come) and
// then bytes.  The warp-level products need no tensor memory: with tcgen05 (M = 128 over the tokens, N = 16) a tile of 128 tokens went through two
// round trips there and two barriers between the roles, and a split cost a launch of 2 us more.  Both measured: decode_parts and
// decode_form in ops/cuda.py.
//
// Reference for the op: FlashInfer trtllm_batch_decode_with_kv_cache (v1/attention/backends/flashinfer.py:2457).
// The weights keep 16 more bits in a second product, P = hi + lo: 2 % of the time, and the error against 64 bits is that of the result's own
// rounding (bf16, 33 to 2000 tokens: 0.00165; with 16-bit weights 0.0017 to 0.0022, as before).  CAP: capped scores.
#include "attention_prompt.cuh"

namespace fmha_dec {

constexpr int D = 128, BS = 64;
constexpr int K_BYTES = BS * D * 2;      // 16 KB: dims 0-63 and 64-127 of [64 tokens x 64]
constexpr int STAGE_BYTES = 2 * K_BYTES; // V behind it: [128 dims x 64 tokens]
constexpr int ROW_BYTES = (D + 4) * 4;   // a merged row: 128 values, maximum, sum; not a multiple of 128 bytes
constexpr int MAX_PARTS = 16;

// TEAMS teams of four warps take the pages in turn, STAGES pages are on their way or in use, CTAS CTAs share an SM
template <int TEAMS_, int STAGES_, int CTAS_> struct Form {
  static constexpr int TEAMS = TEAMS_, STAGES = STAGES_, CTAS = CTAS_, WARPS = 4 * TEAMS, NUM_THREADS = (WARPS + 1) * 32;
  // Barriers go by page, not by stage: an odd number of stages passes from one team to the other, and a team that has not seen the phase before
  // would take it for the one that it waits for.  Of an even number each barrier has one team.
  static constexpr int BARS = TEAMS * STAGES;
};

using Few = Form<2, 6, 1>;
using Some = Form<2, 3, 2>;
using Many = Form<1, 2, 3>;

struct Params {
  const void* q;
  const int* block_table;
  const int* seq_lens;
  void* out;
  float* lse_out;
  int* error;              // raised when a wait ran into its limit
  int64_t q_stride, out_stride;
  int bt_stride;
  int Hq, Hkv, G, parts, split_pages, window;
  float scale_log2;
  float ku, c2;            // capped scores: scale / cap, cap log2(e)
  int chunk;               // > 0: the query sees the keys of its own chunk of positions only
  const float* sinks;      // optional [Hq] logits in the softmax denominator that have no key
  float out_scale;         // factor of the output
};

VB_DEVICE void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <typename T> VB_DEVICE void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> VB_DEVICE void mma16816<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> VB_DEVICE void mma16816<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// an 8 x 8 matrix of 16-bit values, two to a lane, with rows and columns exchanged
VB_DEVICE uint32_t turn8(uint32_t x) { uint32_t r; asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x)); return r; }
VB_DEVICE float ld_dsmem_f32(uint32_t addr) { float v; asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr)); return v; }

// NT: groups of eight query rows
template <typename T, int NT, bool CAP, typename F>
__global__ void __launch_bounds__(F::NUM_THREADS, NT == 1 ? F::CTAS : 1)
fmha_decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const Params p) {
  constexpr int STAGES = F::STAGES, TEAMS = F::TEAMS, WARPS = F::WARPS, NUM_THREADS = F::NUM_THREADS, BARS = F::BARS;
  static_assert(WARPS * NT * 8 * ROW_BYTES <= STAGES * STAGE_BYTES, "warps' results fit the ring");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* merged = ring + STAGES * STAGE_BYTES;          // G rows of ROW_BYTES, read by the cluster
  __shared__ __align__(8) uint64_t full[BARS], empty[BARS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = blockIdx.x % p.parts, b = blockIdx.x / p.parts, h = blockIdx.y;
  int budget = MBAR_BUDGET;
  pdl_trigger();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
    for (int i = 0; i < BARS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], WARPS / TEAMS); }
    mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();   // q, the new K/V rows and seq_lens come from the preceding kernels
  const int kv_end = p.seq_lens[b];
  int kv_begin = p.window > 0 ? max(0, kv_end - p.window) : 0;
  if (p.chunk > 0) kv_begin = max(kv_begin, (kv_end - 1) / p.chunk * p.chunk);
  int page_lo = kv_begin / BS, page_hi = (kv_end + BS - 1) / BS;
  // few pages are left to one CTA, as merging parts takes more than 1 us
  const bool whole = p.parts == 1 || (page_hi - page_lo) * p.parts <= p.split_pages;
  if (whole) {
    if (part > 0) return;
  } else {
    const int per = (page_hi - page_lo + p.parts - 1) / p.parts;
    page_lo += part * per;
    page_hi = min(page_hi, page_lo + per);
  }

  if (warp == WARPS) {
    // ===== producer: 32 block ids at a time, a page's three boxes by one lane
    const int* bt = p.block_table + (int64_t)b * p.bt_stride;
    for (int first = page_lo; first < page_hi && budget >= 0; first += 32) {
      const int mine = first + lane < page_hi ? bt[first + lane] : 0;
      const int m = min(32, page_hi - first);
      for (int i = 0; i < m; ++i) {
        const int blk = __shfl_sync(0xffffffffu, mine, i);
        if (lane == 0 && budget >= 0) {
          const int n = first - page_lo + i, was = n - STAGES;      // the page that the stage held before
          if (was >= 0) mbar_wait_lim(&empty[was % BARS], (was / BARS) & 1, budget);
          if (budget >= 0) {
            unsigned char* to = ring + n % STAGES * STAGE_BYTES;
            uint64_t* bar = &full[n % BARS];
            const int key = (blk * 2 * p.Hkv + h), val = ((blk * 2 + 1) * p.Hkv + h);
            mbar_expect_tx(bar, STAGE_BYTES);
            tma_load_2d_hint(to, &tmap_k, 0, key * BS, bar, L2_EVICT_FIRST);
            tma_load_2d_hint(to + K_BYTES / 2, &tmap_k, 64, key * BS, bar, L2_EVICT_FIRST);
            tma_load_2d_hint(to + K_BYTES, &tmap_v, 0, val * D, bar, L2_EVICT_FIRST);
          }
        }
      }
      budget = __shfl_sync(0xffffffffu, budget, 0);
    }
    if (budget < 0 && lane == 0)              // let the copies in flight land before the block gives up its memory
      for (int n = 0; n < 4096 * BARS; ++n) mbar_try_wait(&full[n % BARS], n / BARS & 1);
  }
  // a lane's share: of scores the tokens r0, r0 + 8 and the rows c0, c0 + 1 of a group; of results the dims r0, r0 + 8 and the same rows
  float o[D / 16][NT][4], m_run[NT][2], l_run[NT][2];
  const int r0 = lane >> 2, c0 = (lane & 3) * 2;
  if (warp < WARPS) {
    uint32_t q[D / 16][NT][2];
    const T* qp = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride + (int64_t)h * p.G * D;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int i = 0; i < D / 16; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][nt][j] = 0.f;
#pragma unroll
      for (int u = 0; u < 2; ++u) { m_run[nt][u] = -INFINITY; l_run[nt][u] = 0.f; }
      const int r = nt * 8 + r0;
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j) q[k][nt][j] = r < p.G ? *reinterpret_cast<const uint32_t*>(qp + r * D + k * 16 + j * 8 + c0) : 0u;
    }
    // addresses of the lane's row in the 8 x 8 matrices of a load: two groups of eight tokens (dims of V) by two halves of 16 dims (tokens)
    const int mi = lane >> 3, l7 = lane & 7, w = warp & 3, team = warp >> 2;
    const uint32_t k_row = (uint32_t)((w * 16 + (mi & 1) * 8 + l7) * 128);
    const uint32_t v_at = (uint32_t)(K_BYTES + ((mi & 1) * 8 + l7) * 128 + (((w * 2 + (mi >> 1)) ^ l7) << 4));
    const uint32_t ring_u = smem_u32(ring);
    for (int page = page_lo + team; page < page_hi; page += TEAMS) {
      const int n = page - page_lo;
      mbar_wait_lim(&full[n % BARS], (n / BARS) & 1, budget);
      const int tok = page * BS + w * 16;                     // first of the warp's tokens
      const bool alive = __all_sync(0xffffffffu, budget >= 0);
      if (tok < kv_end && tok + 16 > kv_begin && alive) {
        const uint32_t st = ring_u + n % STAGES * STAGE_BYTES;
        float sc[NT][4], sd[NT][4];                           // even and odd steps: two chains
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) sc[nt][i] = sd[nt][i] = 0.f;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          uint32_t ka[4];
          ldsm4(ka, st + (k >> 2) * (K_BYTES / 2) + k_row + ((((k & 3) * 2 + (mi >> 1)) ^ l7) << 4));
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma16816<T>(k & 1 ? sd[nt] : sc[nt], ka, q[k][nt][0], q[k][nt][1]);
        }
        const bool cut = tok < kv_begin || tok + 16 > kv_end;
        const bool in[2] = {!cut || (tok + r0 >= kv_begin && tok + r0 < kv_end), !cut || (tok + 8 + r0 >= kv_begin && tok + 8 + r0 < kv_end)};
        uint32_t ph[NT][2], pl[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float mx[2], alpha[2];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float x = sc[nt][i] + sd[nt][i];
            sc[nt][i] = in[i >> 1] ? (CAP ? prompt::cap_any(x * p.ku, p.c2) : x * p.scale_log2) : -INFINITY;
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) mx[u] = fmaxf(sc[nt][u], sc[nt][2 + u]);
#pragma unroll
          for (int x = 4; x < 32; x <<= 1)
#pragma unroll
            for (int u = 0; u < 2; ++u) mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], x));
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float was = m_run[nt][u];
            // the old reference stays unless the new maximum is more than 2^8 above it
            const bool up = mx[u] > was + 8.f || (was == -INFINITY && mx[u] > -INFINITY);
            alpha[u] = up && was != -INFINITY ? ex2(was - mx[u]) : 1.f;
            m_run[nt][u] = up ? mx[u] : was;
          }
          if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
            for (int i = 0; i < D / 16; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) o[i][nt][j] *= alpha[j & 1];
            l_run[nt][0] *= alpha[0]; l_run[nt][1] *= alpha[1];
          }
          const float ref[2] = {m_run[nt][0] == -INFINITY ? 0.f : m_run[nt][0], m_run[nt][1] == -INFINITY ? 0.f : m_run[nt][1]};
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const float x = ex2(sc[nt][2 * t] - ref[0]), y = ex2(sc[nt][2 * t + 1] - ref[1]);
            l_run[nt][0] += x; l_run[nt][1] += y;
            const uint32_t hi = pack2<T>(x, y);
            ph[nt][t] = turn8(hi);
            const float2 back = unpack2<T>(hi);
            pl[nt][t] = turn8(pack2<T>(x - back.x, y - back.y));
          }
        }
        uint32_t keep[2] = {0xffffffffu, 0xffffffffu};        // of tokens c0, c0 + 1 of either group of eight
        if (cut) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int t = tok + j * 8 + c0;
            keep[j] = (t >= kv_begin && t < kv_end ? 0xffffu : 0u) | (t + 1 >= kv_begin && t + 1 < kv_end ? 0xffff0000u : 0u);
          }
        }
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
          uint32_t va[4];
          ldsm4(va, st + v_at + i * (16 * 128));
          if (cut) {           // slots that are not the sequence's may hold what a weight of 0 does not cancel (attention_prompt.cuh)
            va[0] &= keep[0]; va[1] &= keep[0]; va[2] &= keep[1]; va[3] &= keep[1];
          }
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            mma16816<T>(o[i][nt], va, ph[nt][0], ph[nt][1]);
            mma16816<T>(o[i][nt], va, pl[nt][0], pl[nt][1]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[n % BARS]);
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) l_run[nt][u] += __shfl_xor_sync(0xffffffffu, l_run[nt][u], x);
  }
  // ===== the warps' results, then the parts': rows of 128 unscaled values, maximum, sum
  __syncthreads();                             // every page has been read: the ring is free
  if (warp < WARPS) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = nt * 8 + c0 + u;
        if (r < p.G) {
          float* row = reinterpret_cast<float*>(ring + (warp * NT * 8 + r) * ROW_BYTES);
#pragma unroll
          for (int i = 0; i < D / 16; ++i) { row[i * 16 + r0] = o[i][nt][u]; row[i * 16 + 8 + r0] = o[i][nt][2 + u]; }
          if (r0 == 0) { row[D] = m_run[nt][u]; row[D + 1] = l_run[nt][u]; }
        }
      }
  }
  __syncthreads();
  auto finish = [&](int g, int d, float acc, float m, float l) {
    const int hq = h * p.G + g;
    float top = m, f = 1.f, den = l;           // the sink joins the denominator once, behind the last key
    if (p.sinks) {
      const float sink = p.sinks[hq] * 1.4426950408889634f;
      top = fmaxf(top, sink);
      f = m == -INFINITY ? 0.f : ex2(m - top);
      den = l * f + ex2(sink - top);
    }
    reinterpret_cast<T*>(p.out)[(int64_t)b * p.out_stride + (int64_t)hq * D + d] = from_f32<T>(den > 0.f ? acc * (f / den) * p.out_scale : 0.f);
    if (p.lse_out && d == 0) p.lse_out[(int64_t)b * p.Hq + hq] = den > 0.f ? (top + log2f(den)) * 0.6931471805599453f : -INFINITY;
  };
  for (int i = threadIdx.x; i < p.G * D; i += NUM_THREADS) {
    const int g = i / D, d = i % D;
    const float* row = reinterpret_cast<const float*>(ring + g * ROW_BYTES);
    constexpr int STEP = NT * 8 * ROW_BYTES / 4;              // between the warps' rows
    float m = -INFINITY, acc = 0.f, l = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) m = fmaxf(m, row[w * STEP + D]);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float f = m == -INFINITY ? 0.f : ex2(row[w * STEP + D] - m);
      acc += f * row[w * STEP + d];
      l += f * row[w * STEP + D + 1];
    }
    if (whole) finish(g, d, acc, m, l);
    else {
      float* to = reinterpret_cast<float*>(merged + g * ROW_BYTES);
      to[d] = acc;
      if (d == 0) { to[D] = m; to[D + 1] = l; }
    }
  }
  if (!whole) {
    cluster_sync();
    // a row's values go to one warp at a time: a lane reads the maximum and the sum of a part
    const uint32_t rows = smem_u32(merged);
    for (int i = part * (WARPS + 1) + warp; i < p.G * (D / 32); i += p.parts * (WARPS + 1)) {
      const int g = i / (D / 32), d = i % (D / 32) * 32 + lane;
      const uint32_t there = dsmem_addr(rows + g * ROW_BYTES, lane < p.parts ? lane : 0);
      float v[MAX_PARTS];
#pragma unroll
      for (int s = 0; s < MAX_PARTS; ++s) v[s] = s < p.parts ? ld_dsmem_f32(dsmem_addr(rows + g * ROW_BYTES + d * 4, s)) : 0.f;
      const float pm = lane < p.parts ? ld_dsmem_f32(there + D * 4) : -INFINITY, pl = lane < p.parts ? ld_dsmem_f32(there + (D + 1) * 4) : 0.f;
      const float m = warp_max(pm), f = m == -INFINITY ? 0.f : ex2(pm - m), l = warp_sum(f * pl);
      float acc = 0.f;
#pragma unroll
      for (int s = 0; s < MAX_PARTS; ++s) acc += __shfl_sync(0xffffffffu, f, s) * v[s];
      finish(g, d, acc, m, l);
    }
    cluster_sync();                            // the others may still read this CTA's rows
  }
  if (budget < 0 && p.error) *p.error = 1;
}

template <typename T, int NT, bool CAP, typename F>
static int launch(const CUtensorMap& tk, const CUtensorMap& tv, const Params& p, int B, cudaStream_t st) {
  const int smem = F::STAGES * STAGE_BYTES + p.G * ROW_BYTES + 1024;
  auto k = fmha_decode_kernel<T, NT, CAP, F>;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, F::STAGES * STAGE_BYTES + 16 * ROW_BYTES + 1024) != cudaSuccess) return -20;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return -21;
    set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.parts * B, p.Hkv); cfg.blockDim = dim3(F::NUM_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.parts > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = p.parts; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (vb_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr; cfg.numAttrs = n;
  return (int)cudaLaunchKernelEx(&cfg, k, tk, tv, p);
}

}  // namespace fmha_dec

// q [B, Hq, 128] (rows start on 4 bytes), out [B, Hq, 128]; parts: key ranges per (request, kv head), a cluster of CTAs (1 to 16).
// `error` (device int, may be null) becomes 1 when a wait inside the kernel ran into its limit.
EXPORT int vb_fmha_tc_decode3(const void* q, const void* kv_cache, int64_t num_blocks, const int* block_table, const int* seq_lens, void* out,
                              float* lse_out, int* error, int B, int Hq, int Hkv, int64_t q_stride, int64_t out_stride, int bt_stride, int parts, int split_pages, int form,
                              int window, float scale, float soft_cap, int chunk, const float* sinks, float out_scale, int dtype, cudaStream_t st) {
  using namespace fmha_dec;
  if (B == 0) return 0;
  if (dtype == DT_F32) return -1;
  const int G = Hq / Hkv;
  if (G < 1 || G > 16 || Hq % Hkv) return -4;
  if (parts < 1 || parts > MAX_PARTS || form < 0 || form > 2) return -5;
  if (q_stride % 2 || (reinterpret_cast<uintptr_t>(q) & 3)) return -6;
  auto enc = get_encode();
  if (!enc) return -10;
  const bool bf16 = dtype == DT_BF16;
  const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  Params p;
  p.q = q; p.block_table = block_table; p.seq_lens = seq_lens; p.out = out; p.lse_out = lse_out; p.error = error;
  p.q_stride = q_stride; p.out_stride = out_stride; p.bt_stride = bt_stride; p.Hq = Hq; p.Hkv = Hkv; p.G = G;
  p.parts = parts; p.split_pages = split_pages; p.window = window; p.scale_log2 = scale * 1.4426950408889634f;
  p.chunk = chunk; p.sinks = sinks; p.out_scale = out_scale;
  p.ku = soft_cap > 0.f ? scale / soft_cap : 0.f; p.c2 = soft_cap * 1.4426950408889634f;
  CUtensorMap tk, tv;
  auto pages = [&](CUtensorMap* m, int width, int rows) {
    cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)num_blocks * 2 * Hkv * rows};
    cuuint64_t strides[1] = {(cuuint64_t)width * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)rows}, es[2] = {1, 1};
    return enc(m, dt, 2, const_cast<void*>(kv_cache), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  if (pages(&tk, D, BS) != CUDA_SUCCESS) return -12;
  if (pages(&tv, BS, D) != CUDA_SUCCESS) return -13;
  const bool cap = soft_cap > 0.f;
#define VB_NT(T, F) (G <= 8 ? (cap ? launch<T, 1, true, F>(tk, tv, p, B, st) : launch<T, 1, false, F>(tk, tv, p, B, st)) \
                           : (cap ? launch<T, 2, true, F>(tk, tv, p, B, st) : launch<T, 2, false, F>(tk, tv, p, B, st)))
#define VB_GO(T) (form == 0 ? VB_NT(T, Few) : form == 1 ? VB_NT(T, Some) : VB_NT(T, Many))
  return bf16 ? VB_GO(__nv_bfloat16) : VB_GO(__half);
#undef VB_NT
#undef VB_GO
}
