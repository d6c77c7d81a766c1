// Mixture-of-experts routing / dispatch / combine kernels (decode-sized batches stay entirely on the device:
// no host sync, CUDA-graph capturable).  The expert GEMMs themselves are the grouped mode of gemm_tc.cu.
//
// Reference counterparts: csrc/moe/topk_softmax_kernels.cu, moe_align_sum_kernels.cu, moe_permute_unpermute_op.cu
// (here: routing probabilities + top-k in one warp per token; counting sort of (token, slot) pairs by expert with
// an inverse map; weighted un-permute that sums a token's k expert outputs in a fixed order → deterministic).
#include "cluster.cuh"

namespace moe {


// one warp per token: softmax over E <= 32 EL logits, pick the k largest, optionally renormalise.  A maximum is one instruction on the numbers' bits (they
// are not negative).  us for 24 and 6900 tokens that choose 6 of 32: 1.5 and 3.4 (4.1 and 11.4 with room for 512 experts and exchanged pairs).
template <typename T, int EL>
__global__ void topk_softmax_kernel(const T* __restrict__ logits, float* __restrict__ out_w, int* __restrict__ out_ids,
                                    int n_tokens, int E, int k, int renorm, float scale) {
  pdl_trigger();
  pdl_wait();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n_tokens) return;
  const T* row = logits + (size_t)warp * E;
  float v[EL];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < EL; ++i) {
    const int e = lane + i * 32;
    v[i] = e < E ? to_f32(row[e]) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < EL; ++i) {
    const int e = lane + i * 32;
    v[i] = e < E ? __expf(v[i] - mx) : 0.f;
    sum += v[i];
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
  uint32_t key[EL];                                             // 0: picked, NaN, or no expert
#pragma unroll
  for (int i = 0; i < EL; ++i) key[i] = lane + i * 32 < E && v[i] >= 0.f ? __float_as_uint(v[i]) + 1 : 0;
  float picked_sum = 0.f;
  float my_w = 0.f; int my_id = 0;
  for (int j = 0; j < k; ++j) {
    uint32_t best = 0;
    int bi = 0;
#pragma unroll
    for (int i = 0; i < EL; ++i)
      if (key[i] > best) { best = key[i]; bi = lane + i * 32; }  // lowest index wins ties inside a lane
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    const int e = (int)__reduce_min_sync(0xffffffffu, best == top ? (unsigned)bi : 0x7fffffffu);
    const float w = top ? __uint_as_float(top - 1) * inv : __uint_as_float(0x7fc00000u);   // nothing but NaN left: expert 0
#pragma unroll
    for (int i = 0; i < EL; ++i)
      if (lane + i * 32 == e) key[i] = 0;                       // remove the winner
    if (lane == j) { my_w = w; my_id = e; }
    picked_sum += w;
  }
  if (lane < k) {
    out_w[(size_t)warp * k + lane] = (renorm ? my_w / picked_sum : my_w) * scale;
    out_ids[(size_t)warp * k + lane] = my_id;
  }
}

// Router with sigmoid or softmax scores, a selection bias and group-limited choice; one CTA per token, fp32 throughout.
//   logits: given ([T, E] fp32, or as x where there is no w), or computed here from x [T, H] and w [E, H] (one warp per expert, decode batches)
//   choice score = score + bias;  a group (one of n_group contiguous runs) is ranked by the sum of its two best choice
//   scores (group_top2) or by its best;  the k best experts of the `keep` best groups are taken, the lowest
//   index winning ties;  weight = score WITHOUT the bias (optionally renormalised) * scale
template <typename TX, typename TW>
__global__ void __launch_bounds__(512)
grouped_topk_kernel(const float* __restrict__ logits, const TX* __restrict__ x, const TW* __restrict__ w, int H,
                    const float* __restrict__ bias, float* __restrict__ out_w, int* __restrict__ out_ids, int E, int k,
                    int n_group, int keep, int group_top2, int softmax, int renorm, float scale) {
  extern __shared__ float smf[];
  float* score = smf;               // [E]
  float* choice = score + E;        // [E]
  float* gs = choice + E;           // [n_group]
  float* xs = gs + n_group;         // [H] when the logits are computed here
  __shared__ float red[32];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  if (logits) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) score[e] = logits[(int64_t)t * E + e];
  } else if (!w) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) score[e] = to_f32(x[(int64_t)t * E + e]);
  } else {
    const TX* xr = x + (int64_t)t * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) xs[i] = to_f32(xr[i]);
    __syncthreads();
    constexpr int V = Vec16<TW>::N;
    const bool vec = H % V == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    constexpr int EB = 4;                       // experts of a warp in flight together
    for (int e0 = warp * EB; e0 < E; e0 += n_warps * EB) {
      float a[EB] = {};
      if (vec) {
        for (int i = lane * V; i < H; i += 32 * V) {
          Vec16<TW> wv[EB];
#pragma unroll
          for (int u = 0; u < EB; ++u) wv[u] = ld16(w + (int64_t)min(e0 + u, E - 1) * H + i);
#pragma unroll
          for (int j = 0; j < V; ++j) {
            const float xv = xs[i + j];
#pragma unroll
            for (int u = 0; u < EB; ++u) a[u] += xv * to_f32(wv[u].e[j]);
          }
        }
      } else {
        for (int i = lane; i < H; i += 32)
#pragma unroll
          for (int u = 0; u < EB; ++u) a[u] += xs[i] * to_f32(w[(int64_t)min(e0 + u, E - 1) * H + i]);
      }
#pragma unroll
      for (int u = 0; u < EB; ++u) {
        a[u] = warp_sum(a[u]);
        if (lane == 0 && e0 + u < E) score[e0 + u] = a[u];
      }
    }
  }
  __syncthreads();
  if (softmax) {
    float mx = -INFINITY;
    for (int e = threadIdx.x; e < E; e += blockDim.x) mx = fmaxf(mx, score[e]);
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = warp_max(lane < n_warps ? red[lane] : -INFINITY);
    __syncthreads();
    float sum = 0.f;
    for (int e = threadIdx.x; e < E; e += blockDim.x) { score[e] = expf(score[e] - mx); sum += score[e]; }
    const float inv = 1.f / block_sum(sum, red);
    for (int e = threadIdx.x; e < E; e += blockDim.x) score[e] *= inv;
  } else {
    for (int e = threadIdx.x; e < E; e += blockDim.x) score[e] = 1.f / (1.f + expf(-score[e]));
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) choice[e] = score[e] + (bias ? bias[e] : 0.f);
  __syncthreads();
  if (warp) return;                 // the choice is one warp's work
  auto argmax = [&](const float* v, int n) -> int {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = lane; i < n; i += 32)
      if (v[i] > best) { best = v[i]; bi = i; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    return bi;                      // 0x7fffffff: nothing above -inf is left
  };
  if (n_group > 1) {
    const int gsz = E / n_group;
    for (int g = lane; g < n_group; g += 32) {
      float a = -INFINITY, b = -INFINITY;
      for (int i = 0; i < gsz; ++i) {
        const float c = choice[g * gsz + i];
        if (c > a) { b = a; a = c; } else if (c > b) { b = c; }
      }
      gs[g] = group_top2 && gsz > 1 ? a + b : a;
    }
    __syncwarp();
    // drop the worst groups: what the keep-th best leaves behind.  A taken group is marked by -inf.
    for (int n = 0; n < keep; ++n) {
      const int g = argmax(gs, n_group);
      __syncwarp();
      if (lane == 0 && g < n_group) gs[g] = -INFINITY;
      __syncwarp();
    }
    for (int e = lane; e < E; e += 32)
      if (gs[e / gsz] != -INFINITY) choice[e] = -INFINITY;
    __syncwarp();
  }
  float wsum = 0.f, mine = 0.f;
  for (int j = 0; j < k; ++j) {
    int e = argmax(choice, E);
    if (e >= E) e = 0;              // fewer than k candidates: cannot happen for a valid configuration
    const float s = score[e];
    wsum += s;
    __syncwarp();
    if (lane == 0) {
      choice[e] = -INFINITY;
      out_ids[(int64_t)t * k + j] = e;
      if (!renorm) out_w[(int64_t)t * k + j] = s * scale;
    }
    if (lane == (j & 31)) mine = s;
    if (renorm && ((j & 31) == 31 || j == k - 1) && lane <= (j & 31)) out_w[(int64_t)t * k + (j & ~31) + lane] = mine;
    __syncwarp();
  }
  if (renorm)
    for (int j = lane; j < k; j += 32) out_w[(int64_t)t * k + j] *= scale / (wsum + 1e-20f);
}

// The same, to the bit, for given logits of up to 32 EL experts: a warp per token, its experts in registers, a maximum in one instruction (of keys that order as the
// numbers do); a CTA per token spent its time on barriers and on two-step exchanges.  us, before and so: 24 tokens, 6 of 32 in 4 groups 5.1 and 2.6, 6900
// tokens 21 and 6.2; 8 of 256 in 8 groups 7.1 and 7.9, 6900 tokens 39 and 20.
VB_DEVICE uint32_t order_key(float x) {            // NaN and what is left out order as -inf: 0x007fffff
  const uint32_t b = __float_as_uint(x + 0.f);
  return x != x ? 0x007fffffu : (b >> 31) ? ~b : b | 0x80000000u;
}
constexpr uint32_t NONE_KEY = 0x007fffffu;
template <typename TL, int EL>
__global__ void __launch_bounds__(128)
grouped_topk_warp_kernel(const TL* __restrict__ logits, const float* __restrict__ bias, float* __restrict__ out_w, int* __restrict__ out_ids, int n_tokens,
                         int E, int k, int n_group, int keep, int group_top2, int softmax, int renorm, float scale) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= n_tokens) return;
  constexpr unsigned ALL = 0xffffffffu;
  float score[EL];
  uint32_t choice[EL];
#pragma unroll
  for (int i = 0; i < EL; ++i) score[i] = lane + 32 * i < E ? to_f32(logits[(int64_t)t * E + lane + 32 * i]) : -INFINITY;
  if (softmax) {
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < EL; ++i) mx = fmaxf(mx, score[i]);
    mx = warp_max(mx);
#pragma unroll
    for (int i = 0; i < EL; ++i) score[i] = lane + 32 * i < E ? expf(score[i] - mx) : 0.f;
    // the sum in the order of the block's warps (64 threads up to 128 experts, 256 beyond) and of its sum over them: the same bits
    float part[EL];
#pragma unroll
    for (int i = 0; i < EL; ++i) part[i] = EL == 4 && i < 2 ? score[i] + score[i + 2] : score[i];
    constexpr int PARTS = EL == 4 ? 2 : EL;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) part[i] = warp_sum(part[i]);
#pragma unroll
    for (int o = PARTS / 2; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < o; ++i) part[i] += part[i + o];
    const float inv = 1.f / part[0];
#pragma unroll
    for (int i = 0; i < EL; ++i) score[i] *= inv;
  } else {
#pragma unroll
    for (int i = 0; i < EL; ++i) score[i] = 1.f / (1.f + expf(-score[i]));
  }
  int group[EL];
#pragma unroll
  for (int i = 0; i < EL; ++i) {
    const int e = lane + 32 * i;
    choice[i] = e < E ? order_key(score[i] + (bias ? bias[e] : 0.f)) : NONE_KEY;
    group[i] = e < E ? e / (E / n_group) : -1;
  }
  // the largest key among the lanes' and the first place that has it
  auto first = [&](uint32_t key, int place, uint32_t& top) {
    top = __reduce_max_sync(ALL, key);
    return (int)__reduce_min_sync(ALL, key == top ? (unsigned)place : 0x7fffffffu);
  };
  auto own = [&](int g, int but, uint32_t& key, int& place) {      // of this lane's in group g (-1: all), without one
    key = NONE_KEY; place = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < EL; ++i) {
      const int e = lane + 32 * i;
      if (choice[i] > key && e != but && (g < 0 || group[i] == g)) { key = choice[i]; place = e; }
    }
  };
  auto number = [](uint32_t key) { return __uint_as_float((key >> 31) ? key & 0x7fffffffu : ~key); };
  uint32_t key, top;
  int place;
  if (n_group > 1) {
    const bool two = group_top2 && E / n_group > 1;
    uint32_t mine = NONE_KEY;                      // of group `lane`
    bool low = false;                              // its score is -inf: such a group is neither chosen nor left out, as in the block
    for (int g = 0; g < n_group; ++g) {
      own(g, -1, key, place);
      const int p = first(key, place, top);
      float s = number(top);
      if (two) {
        own(g, p, key, place);
        s += number(__reduce_max_sync(ALL, key));
      }
      if (lane == g) { mine = order_key(s); low = s == -INFINITY; }
    }
    unsigned kept = 0;
    for (int n = 0; n < keep; ++n) {
      const int g = first(lane < n_group && !((kept >> lane) & 1u) ? mine : NONE_KEY, lane, top);
      if (top != NONE_KEY) kept |= 1u << g;
    }
    kept |= __ballot_sync(ALL, low);
#pragma unroll
    for (int i = 0; i < EL; ++i)
      if (group[i] >= 0 && !((kept >> group[i]) & 1u)) choice[i] = NONE_KEY;
  }
  float wsum = 0.f, my_w = 0.f;
  int my_id = 0;
  for (int j = 0; j < k; ++j) {
    own(-1, -1, key, place);
    int e = first(key, place, top);
    if (top == NONE_KEY) e = 0;                    // fewer than k candidates: cannot happen for a valid configuration
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < EL; ++i)
      if (i == e >> 5) { s = score[i]; if ((e & 31) == lane) choice[i] = NONE_KEY; }
    s = __shfl_sync(ALL, s, e & 31);
    wsum += s;
    if (lane == j) { my_w = s; my_id = e; }
  }
  if (lane < k) {
    out_w[(int64_t)t * k + lane] = my_w * (renorm ? scale / (wsum + 1e-20f) : scale);
    out_ids[(int64_t)t * k + lane] = my_id;
  }
}

// Grouped GEMM on the CUDA cores for what the tcgen05 kernel (gemm_tc.cu) does not take — fp32, or rows that are not
// 16-byte multiples:  y[r, n] = act(sum_k x[tok(r), k] * w[e(r), n, k]), rows sorted by expert.  64 x 64 tiles; grid.y
// enumerates (expert, row tile) pairs, found from `offs` on the device.
constexpr int GT = 64, GK = 16;
template <typename T>
__global__ void __launch_bounds__(256)
grouped_simt_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, const int* __restrict__ offs,
                    const int* __restrict__ row_tok, int N, int K, int E, int act) {
  __shared__ float as[GK][GT + 4], bs[GK][GT + 4];
  pdl_trigger();
  pdl_wait();
  int tile = blockIdx.y, e = 0, lo = 0, hi = 0;
  for (; e < E; ++e) {
    lo = offs[e]; hi = offs[e + 1];
    const int nt = (hi - lo + GT - 1) / GT;
    if (tile < nt) break;
    tile -= nt;
  }
  if (e == E) return;
  const int r0 = lo + tile * GT, n0 = blockIdx.x * GT;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += GK) {
    for (int i = threadIdx.x; i < GT * GK; i += 256) {
      const int r = i / GK, kk = i % GK, row = r0 + r, n = n0 + r, kc = k0 + kk;
      as[kk][r] = (row < hi && kc < K) ? to_f32(x[(int64_t)(row_tok ? row_tok[row] : row) * K + kc]) : 0.f;
      bs[kk][r] = (n < N && kc < K) ? to_f32(w[((int64_t)e * N + n) * K + kc]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = as[kk][ty * 4 + i]; b[i] = bs[kk][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = r0 + ty * 4 + i, n = n0 + tx * 4 + j;
      float v = acc[i][j];
      if (act == 2) { v = fmaxf(v, 0.f); v *= v; }
      if (row < hi && n < N) y[(int64_t)row * N + n] = from_f32<T>(v);
    }
}

// counting sort of R = T*k (token, slot) pairs by (mapped) expert id.  One CTA.
//   ids[i]  : global expert of pair i;  emap (optional): global → local expert or -1 (not on this rank)
//   sorted_tok[p] : token of the pair placed at sorted position p;  inv[i] : sorted position of pair i (or -1)
//   offs[e] : first sorted position of local expert e;  offs[E] = number of valid pairs
__global__ void align_kernel(const int* __restrict__ ids, const int* __restrict__ emap, int* __restrict__ sorted_tok,
                             int* __restrict__ inv, int* __restrict__ offs, int R, int k, int E,
                             int* __restrict__ sorted_pair) {
  extern __shared__ int sm[];
  int* cnt = sm;            // [E]
  int* start = sm + E;      // [E + 1]
  pdl_trigger();
  pdl_wait();
  for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < R; i += blockDim.x) {
    int e = ids[i];
    if (emap) e = emap[e];
    if (e >= 0) atomicAdd(&cnt[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) { start[e] = acc; offs[e] = acc; acc += cnt[e]; cnt[e] = 0; }
    start[E] = acc; offs[E] = acc;
  }
  __syncthreads();
  // placement: the order of pairs inside one expert's segment is arbitrary (atomic cursor) — every row of the
  // grouped GEMM is computed independently and the combine step goes through `inv`, so results do not depend on it
  for (int i = threadIdx.x; i < R; i += blockDim.x) {
    int e = ids[i];
    if (emap) e = emap[e];
    if (e < 0) { inv[i] = -1; continue; }
    const int p = start[e] + atomicAdd(&cnt[e], 1);
    sorted_tok[p] = i / k;
    if (sorted_pair) sorted_pair[p] = i;
    inv[i] = p;
  }
  // sorted positions past the valid pairs (padding rows of the activation buffer) point at token 0
  for (int p = start[E] + threadIdx.x; p < R; p += blockDim.x) { sorted_tok[p] = 0; if (sorted_pair) sorted_pair[p] = 0; }
}

// The same for prompts, over a cluster: each CTA counts a share of the pairs, kept in registers, adds up what the CTAs before it have of every expert and
// places its own.  One CTA spent its time on the counters' atomics: 41400 pairs, 32 experts 6.9 us (28 in one CTA).
constexpr int ALIGN_CTAS = 8, ALIGN_THREADS = 1024, ALIGN_KEEP = 8;
__global__ void __launch_bounds__(ALIGN_THREADS) align_cluster_kernel(const int* __restrict__ ids, const int* __restrict__ emap, int* __restrict__ sorted_tok,
                                                                      int* __restrict__ inv, int* __restrict__ offs, int R, int k, int E,
                                                                      int* __restrict__ sorted_pair) {
  extern __shared__ int sm[];
  int* cnt = sm;            // [E] of this CTA; then its cursor
  int* next = sm + E;       // [E]
  __shared__ int tot[32];
  __shared__ int valid;
  pdl_trigger();
  pdl_wait();
  const int rank = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = (R + ALIGN_CTAS - 1) / ALIGN_CTAS, lo = min(R, rank * per), hi = min(R, lo + per);
  auto expert = [&](int i) { int e = ids[i]; return emap ? emap[e] : e; };
  for (int e = threadIdx.x; e < E; e += ALIGN_THREADS) cnt[e] = 0;
  __syncthreads();
  int keep[ALIGN_KEEP];
#pragma unroll
  for (int u = 0; u < ALIGN_KEEP; ++u) {
    const int i = lo + u * ALIGN_THREADS + (int)threadIdx.x;
    keep[u] = i < hi ? expert(i) : -1;
    if (keep[u] >= 0) atomicAdd(&cnt[keep[u]], 1);
  }
  for (int i = lo + ALIGN_KEEP * ALIGN_THREADS + (int)threadIdx.x; i < hi; i += ALIGN_THREADS) {
    const int e = expert(i);
    if (e >= 0) atomicAdd(&cnt[e], 1);
  }
  cluster_sync();
  // experts in runs of 1024: how many pairs all CTAs have of each, and how many the ones before this
  int base = 0;
  for (int e0 = 0; e0 < E; e0 += ALIGN_THREADS) {
    const int e = e0 + (int)threadIdx.x;
    int all = 0, before = 0;
    if (e < E) {
#pragma unroll
      for (int r = 0; r < ALIGN_CTAS; ++r) {
        const int c = __float_as_int(ld_dsmem_f32(dsmem_addr(smem_u32(&cnt[e]), r)));
        all += c;
        if (r < rank) before += c;
      }
    }
    int inc = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
    if (lane == 31) tot[w] = inc;
    __syncthreads();
    int t = tot[lane], ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, ti, o); if (lane >= o) ti += v; }
    const int first = base + __shfl_sync(0xffffffffu, ti - t, w) + inc - all;
    if (e < E) {
      next[e] = first + before;
      if (rank == 0) offs[e] = first;
    }
    base += __shfl_sync(0xffffffffu, ti, 31);
    __syncthreads();
  }
  if (threadIdx.x == 0) { valid = base; if (rank == 0) offs[E] = base; }
  __syncthreads();
  auto put = [&](int i, int e) {
    if (e < 0) { inv[i] = -1; return; }
    const int p = atomicAdd(&next[e], 1);
    sorted_tok[p] = i / k;
    if (sorted_pair) sorted_pair[p] = i;
    inv[i] = p;
  };
#pragma unroll
  for (int u = 0; u < ALIGN_KEEP; ++u) {
    const int i = lo + u * ALIGN_THREADS + (int)threadIdx.x;
    if (i < hi) put(i, keep[u]);
  }
  for (int i = lo + ALIGN_KEEP * ALIGN_THREADS + (int)threadIdx.x; i < hi; i += ALIGN_THREADS) put(i, expert(i));
  for (int p = valid + rank * ALIGN_THREADS + (int)threadIdx.x; p < R; p += ALIGN_CTAS * ALIGN_THREADS) { sorted_tok[p] = 0; if (sorted_pair) sorted_pair[p] = 0; }
  cluster_sync();           // the others read this CTA's counts until their placement
}

// Tail of the fused MoE combine: acc (fp32, every rank holds the complete sum after the multimem.red epilogue of the
// w2 grouped GEMM) + residual → new residual, RMSNorm → out; acc is zeroed for its next use.  One CTA per token.
template <typename T, bool GEMMA>
__global__ void __launch_bounds__(1024) moe_finish_kernel(float* __restrict__ acc, T* __restrict__ residual,
                                                           const T* __restrict__ w, T* __restrict__ out, int H, float eps) {
  __shared__ float red[32];
  pdl_trigger();
  pdl_wait();
  const int64_t row = blockIdx.x;
  float* a = acc + row * H;
  T* r = residual ? residual + row * H : nullptr;
  constexpr int MAXV4 = 8;                     // float4 per thread kept in registers (H <= 1024 * 8 * 4)
  float4 v[MAXV4];
  float ss = 0.f;
  const int nv = H / 4;
#pragma unroll
  for (int i = 0; i < MAXV4; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nv) {
      v[i] = *reinterpret_cast<const float4*>(a + vi * 4);
      *reinterpret_cast<float4*>(a + vi * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r) {
        const uint2 rv = *reinterpret_cast<const uint2*>(r + vi * 4);
        const float2 r0 = unpack2<T>(rv.x), r1 = unpack2<T>(rv.y);
        // the stream is kept in T: round the sum through T like the unfused path
        v[i].x = to_f32(from_f32<T>(v[i].x)) + r0.x; v[i].y = to_f32(from_f32<T>(v[i].y)) + r0.y;
        v[i].z = to_f32(from_f32<T>(v[i].z)) + r1.x; v[i].w = to_f32(from_f32<T>(v[i].w)) + r1.y;
        uint2 o;
        o.x = pack2<T>(v[i].x, v[i].y); o.y = pack2<T>(v[i].z, v[i].w);
        *reinterpret_cast<uint2*>(r + vi * 4) = o;
        const float2 q0 = unpack2<T>(o.x), q1 = unpack2<T>(o.y);
        v[i] = make_float4(q0.x, q0.y, q1.x, q1.y);
      }
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
  }
  if (w == nullptr) {                          // no norm: out = combined (+ residual) in T
#pragma unroll
    for (int i = 0; i < MAXV4; ++i) {
      const int vi = threadIdx.x + i * blockDim.x;
      if (vi < nv) {
        uint2 o;
        o.x = pack2<T>(v[i].x, v[i].y); o.y = pack2<T>(v[i].z, v[i].w);
        *reinterpret_cast<uint2*>(out + row * H + vi * 4) = o;
      }
    }
    return;
  }
  ss = block_sum(ss, red);
  const float inv = rsqrtf(ss / (float)H + eps);
#pragma unroll
  for (int i = 0; i < MAXV4; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nv) {
      const uint2 wv = *reinterpret_cast<const uint2*>(w + vi * 4);
      float2 w0 = unpack2<T>(wv.x), w1 = unpack2<T>(wv.y);
      if (GEMMA) { w0.x += 1.f; w0.y += 1.f; w1.x += 1.f; w1.y += 1.f; }
      uint2 o;
      o.x = pack2<T>(v[i].x * inv * w0.x, v[i].y * inv * w0.y);
      o.y = pack2<T>(v[i].z * inv * w1.x, v[i].w * inv * w1.y);
      *reinterpret_cast<uint2*>(out + row * H + vi * 4) = o;
    }
  }
}

// out[t, :] = sum_j w[t, j] * y[inv[t*k + j], :]   (pairs not computed on this rank contribute 0)
template <typename T>
__global__ void combine_kernel(const T* __restrict__ y, const int* __restrict__ inv, const float* __restrict__ w,
                               T* __restrict__ out, int H, int k) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  for (int g = threadIdx.x; g < H / 8; g += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int j = 0; j < k; ++j) {
      const int p = inv[t * k + j];
      if (p < 0) continue;
      const float wj = w[t * k + j];
      const Vec16<T> v = ld16(y + (size_t)p * H + g * 8);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += wj * to_f32(v.e[e]);
    }
    Vec16<T> o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.e[e] = from_f32<T>(acc[e]);
    st16(out + (size_t)t * H + g * 8, o);
  }
}

// Tail of a sparse block, one CTA per token:  r += sum_j w[t, j] y[inv[t k + j], :] + sigmoid(gate[t]) extra[t, :];  out = norm(r) * nw
// (extra: a shared expert's output, or null; gate null: 1).  32-bit until r is rounded; a combine, a gating product, two additions and a
// norm were six launches and as many passes over [T, H].
template <typename T, bool GEMMA, int MAXV>
__global__ void __launch_bounds__(1024) combine_norm_kernel(const T* __restrict__ y, const int* __restrict__ inv, const float* __restrict__ w, int k,
                                                            const T* __restrict__ extra, const T* __restrict__ gate, T* __restrict__ residual,
                                                            const T* __restrict__ nw, T* __restrict__ out, int H, float eps) {
  __shared__ float red[32];
  pdl_trigger();
  pdl_wait();
  const int64_t t = blockIdx.x;
  const int nvec = H / 8;
  const float g = extra && gate ? 1.f / (1.f + expf(-to_f32(gate[t]))) : 1.f;
  Vec16<T> r[MAXV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi >= nvec) continue;
    r[i] = ld16(residual + t * H + vi * 8);
    float acc[8];
    if (extra) {
      const Vec16<T> e = ld16(extra + t * H + vi * 8);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = g * to_f32(e.e[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    }
    for (int u0 = 0; u0 < k; u0 += 4) {          // four rows on their way at a time
      int p[4];
      float wu[4];
      Vec16<T> v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        p[u] = u0 + u < k ? inv[t * k + u0 + u] : -1;
        if (p[u] >= 0) { wu[u] = w[t * k + u0 + u]; v[u] = ld16(y + (size_t)p[u] * H + vi * 8); }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (p[u] < 0) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += wu[u] * to_f32(v[u].e[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      r[i].e[j] = from_f32<T>(to_f32(r[i].e[j]) + acc[j]);
      const float f = to_f32(r[i].e[j]);
      ss += f * f;
    }
  }
  const float s = rsqrtf(block_sum(ss, red) / (float)H + eps);
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi >= nvec) continue;
    st16(residual + t * H + vi * 8, r[i]);
    const Vec16<T> n = ld16(nw + vi * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) r[i].e[j] = from_f32<T>(to_f32(r[i].e[j]) * s * (to_f32(n.e[j]) + (GEMMA ? 1.f : 0.f)));
    st16(out + t * H + vi * 8, r[i]);
  }
}

// xs[p, :] = x[sorted_tok[p], :]
template <typename T>
__global__ void gather_kernel(const T* __restrict__ x, const int* __restrict__ sorted_tok, T* __restrict__ xs, int H) {
  pdl_trigger();
  pdl_wait();
  const int p = blockIdx.x;
  const T* src = x + (size_t)sorted_tok[p] * H;
  for (int g = threadIdx.x; g < H / 8; g += blockDim.x) st16(xs + (size_t)p * H + g * 8, ld16(src + g * 8));
}

// The same from the tokens' side, one CTA each: a row is read once and written where its k pairs went (inv).  Places that no pair has are left alone.
// 6900 rows of 2048, k = 6: 32 us, 6.1 TB/s (45 by places: a CTA per place, k reads of a row); 1365 rows 5.8 and 9.1
template <typename T>
__global__ void __launch_bounds__(256) spread_kernel(const T* __restrict__ x, const int* __restrict__ inv, T* __restrict__ xs, int H, int k) {
  pdl_trigger();
  pdl_wait();
  const int64_t t = blockIdx.x;
  for (int g = threadIdx.x; g < H / 8; g += blockDim.x) {
    const Vec16<T> v = ld16(x + t * H + g * 8);
    for (int j = 0; j < k; ++j) {
      const int p = inv[t * k + j];
      if (p >= 0) st16(xs + (size_t)p * H + g * 8, v);
    }
  }
}

}  // namespace moe

EXPORT int vb_moe_spread(const void* x, const int* inv, void* xs, int T_, int H, int k, int dtype, cudaStream_t st) {
  if (T_ == 0) return 0;
  if (dtype == DT_F32 || H % 8 || k < 1) return -1;
  DISPATCH_HALF(dtype, T, vb_launch(moe::spread_kernel<T>, dim3(T_), dim3(256), 0, st, (const T*)x, inv, (T*)xs, H, k));
  return (int)cudaGetLastError();
}

EXPORT int vb_moe_topk_softmax(const void* logits, float* out_w, int* out_ids, int n_tokens, int E, int k, int renorm,
                               float scale, int dtype, cudaStream_t st) {
  if (E > 512 || k > 32) return -1;
  const int threads = 128, warps_per_block = threads / 32;
  dim3 grid((n_tokens + warps_per_block - 1) / warps_per_block);
  DISPATCH_DTYPE(dtype, T, {
    auto* kernel = E <= 32 ? moe::topk_softmax_kernel<T, 1> : E <= 64 ? moe::topk_softmax_kernel<T, 2> : E <= 128 ? moe::topk_softmax_kernel<T, 4>
                 : E <= 256 ? moe::topk_softmax_kernel<T, 8> : moe::topk_softmax_kernel<T, 16>;
    vb_launch(kernel, grid, dim3(threads), 0, st, (const T*)logits, out_w, out_ids, n_tokens, E, k, renorm, scale);
  });
  return (int)cudaGetLastError();
}

// x / w null: `logits` are given; w alone null: x holds them.  dtypes: x fp32 or the model dtype (x_f32), w the model dtype.
EXPORT int vb_moe_grouped_topk(const float* logits, const void* x, int x_f32, const void* w, int H, const float* bias,
                               float* out_w, int* out_ids, int n_tokens, int E, int k, int n_group, int keep, int group_top2,
                               int softmax, int renorm, float scale, int dtype, cudaStream_t st) {
  if (n_tokens == 0) return 0;
  if (E < 1 || E > 4096 || k < 1 || k > E || n_group < 1 || E % n_group || keep < 1 || keep > n_group) return -1;
  if (!logits && !x) return -1;
  const bool given = logits || !w;
  if (given && (E <= 128 || (E <= 256 && n_tokens >= 1024)) && n_group <= 32 && k <= 32) {          // eight experts to a lane: where there are warps enough
    const dim3 grid((n_tokens + 3) / 4);
#define GW(TL, EL) vb_launch(moe::grouped_topk_warp_kernel<TL, EL>, grid, dim3(128), 0, st, reinterpret_cast<const TL*>(logits ? (const void*)logits : x), bias, out_w, out_ids, n_tokens, E, k, n_group, keep, group_top2, softmax, renorm, scale)
#define GE(TL) do { if (E <= 32) GW(TL, 1); else if (E <= 64) GW(TL, 2); else if (E <= 128) GW(TL, 4); else GW(TL, 8); } while (0)
    if (logits) GE(float);
    else DISPATCH_DTYPE(dtype, T, GE(T));
#undef GE
#undef GW
    return (int)cudaGetLastError();
  }
  const size_t smem = (size_t)(2 * E + n_group + (given ? 0 : H)) * sizeof(float);
  if (smem > 48 * 1024) return -3;
  const int thr = given ? (E > 128 ? 256 : 64) : (E > 32 ? 512 : 256);
#define GO(TX, TW) vb_launch(moe::grouped_topk_kernel<TX, TW>, dim3(n_tokens), dim3(thr), smem, st, logits, (const TX*)x, (const TW*)w, H, bias, out_w, out_ids, E, k, n_group, keep, group_top2, softmax, renorm, scale)
  DISPATCH_DTYPE(dtype, T, {
    if (x_f32) GO(float, T); else GO(T, T);
  });
#undef GO
  return (int)cudaGetLastError();
}

// x [*, K] read through row_tok (null: x is already in sorted order), w [E, N, K], y [R, N]; act: 0 none, 2 squared ReLU
EXPORT int vb_moe_grouped_simt(const void* x, const void* w, void* y, const int* offs, const int* row_tok, int R, int N, int K,
                               int E, int act, int dtype, cudaStream_t st) {
  if (R == 0) return 0;
  if (act != 0 && act != 2) return -1;
  const dim3 grid((N + moe::GT - 1) / moe::GT, R / moe::GT + (E < R ? E : R));
  DISPATCH_DTYPE(dtype, T, {
    vb_launch(moe::grouped_simt_kernel<T>, grid, dim3(256), 0, st, (const T*)x, (const T*)w, (T*)y, offs, row_tok, N, K, E, act);
  });
  return (int)cudaGetLastError();
}

EXPORT int vb_moe_align2(const int* ids, const int* emap, int* sorted_tok, int* inv, int* offs, int R, int k, int E,
                         int* sorted_pair, cudaStream_t st) {
  if (E > 4096) return -1;
  if (R > 4096) {           // us for 4200, 8190 and 41400 pairs of 32 experts, one CTA of 1024 threads and eight: 5.0 and 3.7, 7.1 and 4.2, 28 and 6.9
    vb_launch_parts(moe::align_cluster_kernel, dim3(moe::ALIGN_CTAS), dim3(moe::ALIGN_THREADS), (size_t)2 * E * sizeof(int), st, (unsigned)moe::ALIGN_CTAS, ids, emap,
                    sorted_tok, inv, offs, R, k, E, sorted_pair);
    return (int)cudaGetLastError();
  }
  vb_launch(moe::align_kernel, dim3(1), dim3(256), (size_t)(2 * E + 1) * sizeof(int), st, ids, emap, sorted_tok, inv, offs,
            R, k, E, sorted_pair);
  return (int)cudaGetLastError();
}
EXPORT int vb_moe_align(const int* ids, const int* emap, int* sorted_tok, int* inv, int* offs, int R, int k, int E,
                        cudaStream_t st) {
  return vb_moe_align2(ids, emap, sorted_tok, inv, offs, R, k, E, nullptr, st);
}

// out = RMSNorm(acc + residual) (norm_w may be null: out = acc (+ residual)); residual updated in place; acc zeroed
EXPORT int vb_moe_finish(float* acc, void* residual, const void* norm_w, void* out, int T_, int H, float eps, int gemma,
                         int dtype, cudaStream_t st) {
  if (T_ == 0) return 0;
  if (dtype == DT_F32 || H % 4 || H > 1024 * 8 * 4) return -1;
  int thr = ((H / 4 + 7) / 8 + 31) / 32 * 32;
  thr = thr < 64 ? 64 : (thr > 1024 ? 1024 : thr);
  DISPATCH_HALF(dtype, T, {
    if (gemma) vb_launch(moe::moe_finish_kernel<T, true>, dim3(T_), dim3(thr), 0, st, acc, (T*)residual, (const T*)norm_w, (T*)out, H, eps);
    else vb_launch(moe::moe_finish_kernel<T, false>, dim3(T_), dim3(thr), 0, st, acc, (T*)residual, (const T*)norm_w, (T*)out, H, eps);
  });
  return (int)cudaGetLastError();
}

EXPORT int vb_moe_combine(const void* y, const int* inv, const float* w, void* out, int T_, int H, int k, int dtype,
                          cudaStream_t st) {
  if (H % 8) return -1;
  DISPATCH_HALF(dtype, T, {
    vb_launch(moe::combine_kernel<T>, dim3(T_), dim3(128), 0, st, (const T*)y, inv, w, (T*)out, H, k);
  });
  return (int)cudaGetLastError();
}

EXPORT int vb_moe_gather(const void* x, const int* sorted_tok, void* xs, int R, int H, int dtype, cudaStream_t st) {
  if (H % 8) return -1;
  DISPATCH_HALF(dtype, T, {
    vb_launch(moe::gather_kernel<T>, dim3(R), dim3(128), 0, st, (const T*)x, sorted_tok, (T*)xs, H);
  });
  return (int)cudaGetLastError();
}

// all of [T, H] contiguous (y [R, H]); H a multiple of 8 up to 32768; flags as vb_rms_norm's
EXPORT int vb_moe_combine_norm(const void* y, const int* inv, const float* w, int k, const void* extra, const void* gate, void* residual,
                               const void* nw, void* out, int T_, int H, float eps, int flags, int dtype, cudaStream_t st) {
  if (T_ == 0) return 0;
  if (dtype == DT_F32 || H % 8 || H / 8 > 4096 || k < 1) return -1;
  const int nvec = H / 8, quarter = ((nvec + 3) / 4 + 31) / 32 * 32;   // vectors of a row, threads with four each
  int thr = (nvec + 31) / 32 * 32;
  if (T_ >= 1024 && nvec >= 256 && !(flags & 2)) thr = quarter < 128 ? 128 : quarter;      // as norm_threads
  if (thr > 1024) thr = 1024;
#define GO(G) vb_launch(thr >= nvec ? moe::combine_norm_kernel<T, G, 1> : moe::combine_norm_kernel<T, G, 4>, dim3(T_), dim3(thr), 0, st, (const T*)y, inv, w, k, (const T*)extra, (const T*)gate, (T*)residual, (const T*)nw, (T*)out, H, eps)
  DISPATCH_HALF(dtype, T, { if (flags & 1) GO(true); else GO(false); });
#undef GO
  return (int)cudaGetLastError();
}
