// Sampling kernels: row argmax, fused temperature + Gumbel-max sampling, top-k/top-p/min-p
// threshold filtering, repetition / presence / frequency penalties.
//
// Reference: v1/sample/ops/topk_topp_sampler.py (FlashInfer sampling kernels or Triton),
// worker/gpu/sample/gumbel.py:182 (Triton Gumbel sampler), csrc sampler.cu (penalties).
// One CTA per row; logits are read once with 16-byte loads straight from the LM-head output
// dtype (no fp32 staging copy); the noise is a counter-based hash of (seed, step, token) so
// the result is independent of launch geometry and reproducible per request seed.
#include "cluster.cuh"

namespace {

VB_DEVICE uint32_t hash3(uint64_t seed, uint32_t step, uint32_t idx) {
  // 2 rounds of a 64-bit mix (splitmix64 finaliser) over (seed, step, idx)
  uint64_t z = seed + 0x9E3779B97F4A7C15ull * ((uint64_t)step << 32 | idx);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return (uint32_t)(z >> 32);
}
VB_DEVICE float gumbel(uint64_t seed, uint32_t step, uint32_t idx) {
  const float u = ((float)(hash3(seed, step, idx) >> 8) + 0.5f) * (1.0f / 16777216.0f);  // (0,1)
  return -__logf(-__logf(u));
}

struct ArgMax { float v; int i; };
VB_DEVICE ArgMax better(ArgMax a, ArgMax b) { return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a; }

template <typename T, bool SAMPLE>
__global__ void __launch_bounds__(1024) sample_kernel(const T* __restrict__ logits, int64_t row_stride, int V,
                                                       const float* __restrict__ temperature,
                                                       const int64_t* __restrict__ seeds, const int* __restrict__ step_ptr,
                                                       int64_t* __restrict__ out, int idx_off, float4* __restrict__ cand) {
  constexpr int N = Vec16<T>::N;
  __shared__ float sv[32];
  __shared__ int si[32];
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x;
  const T* lr = logits + (int64_t)row * row_stride;
  float temp = 0.f;
  uint64_t seed = 0;
  uint32_t step = 0;
  if (SAMPLE) {
    temp = temperature[row];
    seed = (uint64_t)seeds[row];
    step = (uint32_t)step_ptr[row];
  }
  const bool noisy = SAMPLE && temp >= 1e-5f;
  const float inv_t = noisy ? 1.f / temp : 1.f;
  ArgMax best{-INFINITY, 0x7fffffff};
  const int nvec = V / N;
  for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
    Vec16<T> v = ld16(lr + vi * N);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      float x = to_f32(v.e[j]);
      const int idx = idx_off + vi * N + j;        // global vocabulary id: the noise is indexed by it (TP-invariant)
      if (noisy) x = x * inv_t + gumbel(seed, step, (uint32_t)idx);
      best = better(best, ArgMax{x, idx});
    }
  }
  for (int i = nvec * N + threadIdx.x; i < V; i += blockDim.x) {
    float x = to_f32(lr[i]);
    const int idx = idx_off + i;
    if (noisy) x = x * inv_t + gumbel(seed, step, (uint32_t)idx);
    best = better(best, ArgMax{x, idx});
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { sv[w] = best.v; si[w] = best.i; }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    best = lane < nw ? ArgMax{sv[lane], si[lane]} : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = better(best, other);
    }
    if (lane == 0) {
      if (cand) cand[row] = make_float4(best.v, __int_as_float(best.i), 0.f, 0.f);   // this rank's candidate
      else out[row] = best.i == 0x7fffffff ? 0 : best.i;
    }
  }
}

// final pick over the per-rank candidates gathered as [B, W] x (value, index): same tie-break as the single-GPU kernel
__global__ void select_candidate_kernel(const float4* __restrict__ cands, int W, int64_t* __restrict__ out, int B) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= B) return;
  ArgMax best{-INFINITY, 0x7fffffff};
  for (int r = 0; r < W; ++r) {
    const float4 c = cands[(size_t)row * W + r];
    best = better(best, ArgMax{c.x, __float_as_int(c.y)});
  }
  out[row] = best.i == 0x7fffffff ? 0 : best.i;
}

// Log-probabilities of a row's sampled token and of its k likeliest: out [B, 2 k + 3] holds the k + 1 ids (the sampled one first), their log
// softmax (fp32 bits) and the sampled token's rank (tokens that are likelier, plus one).  One CTA per row; the row is read three times,
// the last two from L1 / L2.  The k likeliest are taken one by one: every thread keeps the best of its own elements, and only the one
// whose element was taken looks for its next (ties: the lowest index first).  A dozen library launches (log softmax, gather, compare and
// sum, four-pass radix top-k, concatenations) took 45 us for 24 rows of 32000.
template <typename T>
__global__ void __launch_bounds__(1024) logprobs_kernel(const T* __restrict__ logits, int64_t row_stride, int V, const int64_t* __restrict__ sampled,
                                                         int k, int* __restrict__ out) {
  constexpr int N = Vec16<T>::N;
  __shared__ float sv[32];
  __shared__ int si[32];
  __shared__ float red[32];
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const T* lr = logits + (int64_t)row * row_stride;
  const int nvec = V / N, tail = nvec * N;
  auto each = [&](auto f) {
    for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
      const Vec16<T> v = ld16(lr + vi * N);
#pragma unroll
      for (int j = 0; j < N; ++j) f(to_f32(v.e[j]), vi * N + j);
    }
    for (int i = tail + threadIdx.x; i < V; i += blockDim.x) f(to_f32(lr[i]), i);
  };
  ArgMax best{-INFINITY, 0x7fffffff};
  each([&](float x, int i) { best = better(best, ArgMax{x, i}); });
  auto top = [&]() {                       // best of the block, in every thread
    ArgMax b = best;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = better(b, ArgMax{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)});
    __syncthreads();
    if (lane == 0) { sv[w] = b.v; si[w] = b.i; }
    __syncthreads();
    b = lane < nw ? ArgMax{sv[lane], si[lane]} : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = better(b, ArgMax{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)});
    return b;
  };
  ArgMax t = top();
  const float mx = t.v;
  float sum = 0.f;
  each([&](float x, int) { sum += expf(x - mx); });
  const float lsum = logf(block_sum(sum, red));
  const int64_t pick = sampled[row];
  const int sidx = (int)(pick < 0 ? 0 : pick >= V ? V - 1 : pick);
  const float slp = (to_f32(lr[sidx]) - mx) - lsum;
  float above = 0.f;
  each([&](float x, int) { above += (x - mx) - lsum > slp ? 1.f : 0.f; });       // counts below 2^24 are exact
  above = block_sum(above, red);
  int* o = out + (int64_t)row * (2 * k + 3);
  if (threadIdx.x == 0) {
    o[0] = (int)pick;
    o[k + 1] = __float_as_int(slp);
    o[2 * k + 2] = (int)above + 1;
  }
  for (int r = 0; r < k; ++r) {
    if (threadIdx.x == 0) {
      o[1 + r] = t.i == 0x7fffffff ? 0 : t.i;
      o[k + 2 + r] = __float_as_int((t.v - mx) - lsum);
    }
    if (r + 1 == k) break;
    if (best.i == t.i) {                   // the owner of the taken element: its next one in order
      const ArgMax old = t;
      best = ArgMax{-INFINITY, 0x7fffffff};
      each([&](float x, int i) { if (x < old.v || (x == old.v && i > old.i)) best = better(best, ArgMax{x, i}); });
    }
    t = top();
  }
}

// The same for vocabularies of up to 8 x 32 x THREADS tokens: a row is a cluster's, 32 x THREADS values of it a CTA's, 32 a thread's, which holds
// them in registers for all passes.  The k likeliest are among the values that reach the k-th of the maxima of 2 k groups and more: hardly more than k
// of them, which the CTAs list and the first one ranks by comparing each with each.  Where the lists are too short for that (equal values, or the likeliest
// next to each other in a few groups), a CTA lists what is above the bound and the first k that are equal; with too many above it the bound is the
// largest of the CTAs' own k-th maxima of 256 groups.  Where the lists are still too short, a warp takes its k likeliest one by one, the CTA merges its
// warps' lists, the first CTA those of the cluster.  What bounds it is the chain of exchanges, not the 1.5 MB of 24 such rows: us for k = 5, here and with
// a CTA per row, 1 row of 32000 6.9 and 15.2, 24 rows 7.5 and 15.7, 24 rows of 102400 18 and 36, of 256000 32 and 89; for k = 64, 1 row of 32000
// 11 and 136.  Rows of one value and ascending ones: 24 of 32000 13 and 17, 17 and 16.
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS) logprobs_cluster_kernel(const T* __restrict__ logits, int64_t row_stride, int V,
                                                                   const int64_t* __restrict__ sampled, int k, int* __restrict__ out, int parts) {
  constexpr int N = Vec16<T>::N, NV = 32 / N, WARPS = THREADS / 32, LIST = 512, ALL = 1024;
  extern __shared__ float lp_smem[];                 // [WARPS + 1][k] values, then places: of the warps, then of the CTA
  float* lv = lp_smem;
  int* li = reinterpret_cast<int*>(lp_smem + (WARPS + 1) * k);
  __shared__ float red[32];
  __shared__ float part[2];                          // of the CTA: maximum, sum of exponentials
  __shared__ float groups[128];                      // maxima of the CTA's groups
  __shared__ __align__(16) float row_groups[256];    // of the row's
  __shared__ int count[3];                           // of the CTA: tokens above the sampled one, listed values, values above the bound
  __shared__ int tot[32];                            // of the warps: values equal to the bound
  __shared__ __align__(8) float2 list[LIST], all[ALL];               // (value, place)
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x / parts, rank = blockIdx.x % parts, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T* lr = logits + (int64_t)row * row_stride;
  const int base = rank * THREADS * 32;
  float v[32];                                       // place of v[j N + u]: at(j, u); behind the end -inf
  auto at = [&](int j, int u) { return base + (j * THREADS + (int)threadIdx.x) * N + u; };
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    if (at(j, N - 1) < V) {
      const Vec16<T> x = ld16(lr + at(j, 0));
#pragma unroll
      for (int u = 0; u < N; ++u) v[j * N + u] = to_f32(x.e[u]);
    } else {
#pragma unroll
      for (int u = 0; u < N; ++u) v[j * N + u] = at(j, u) < V ? to_f32(lr[at(j, u)]) : -INFINITY;
    }
  }
  const int64_t pick = sampled[row];
  const int sidx = (int)(pick < 0 ? 0 : pick >= V ? V - 1 : pick);
  const float picked = to_f32(lr[sidx]);
  if (threadIdx.x < 3) count[threadIdx.x] = 0;
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 32; ++j) mx = fmaxf(mx, v[j]);
  int size = 32;                                     // threads of a group: a warp, or fewer where those are not twice the k that are looked for
  while (parts * THREADS < 2 * k * size) size >>= 1;
  float gm = mx;
  for (int o = size >> 1; o > 0; o >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
  const int ng = THREADS / size;
  if (threadIdx.x % size == 0) groups[threadIdx.x / size] = gm;
  mx = warp_max(gm);
  if (lane == 0) red[w] = mx;
  __syncthreads();
  mx = warp_max(lane < WARPS ? red[lane] : -INFINITY);
  float sum = 0.f;
  if (mx != -INFINITY) {
#pragma unroll
    for (int j = 0; j < 32; ++j) sum += expf(v[j] - mx);             // 0 behind the end
  }
  __syncthreads();
  sum = block_sum(sum, red);
  if (threadIdx.x == 0) { part[0] = mx; part[1] = sum; }
  cluster_sync();
  const float pm = lane < parts ? ld_dsmem_f32(dsmem_addr(smem_u32(&part[0]), lane)) : -INFINITY;
  const float ps = lane < parts ? ld_dsmem_f32(dsmem_addr(smem_u32(&part[1]), lane)) : 0.f;
  if (k > 0) {                                       // the k-th of the maxima: no fewer than k values reach it (with fewer numbers among them, all do)
    if (threadIdx.x == 0) red[0] = -INFINITY;
    for (int i = threadIdx.x; i < parts * ng; i += THREADS) row_groups[i] = ld_dsmem_f32(dsmem_addr(smem_u32(&groups[i % ng]), i / ng));
    __syncthreads();
    for (int i = threadIdx.x; i < parts * ng; i += THREADS) {
      const float x = row_groups[i];
      int r = 0;
      for (int q = 0; q < parts * ng; ++q) r += row_groups[q] > x || (row_groups[q] == x && q < i) ? 1 : 0;
      if (r == k - 1 && x == x) red[0] = x;
    }
    __syncthreads();
  }
  float bound = red[0];
  mx = warp_max(pm);
  const float lsum = logf(warp_sum(pm == -INFINITY ? 0.f : ps * expf(pm - mx)));
  const float slp = (picked - mx) - lsum;
  int above = 0;
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const float x = v[j * N + u];
      above += (x - mx) - lsum > slp ? 1 : 0;        // (nothing behind the end: -inf or NaN on the left)
      if (k > 0 && x >= bound && at(j, u) < V) {
        const int n = atomicAdd(&count[1], 1);
        if (n < LIST) list[n] = make_float2(x, __int_as_float(at(j, u)));
      }
    }
  above = __reduce_add_sync(0xffffffffu, above);
  if (lane == 0 && above) atomicAdd(&count[0], above);
  cluster_sync();
  int* o = out + (int64_t)row * (2 * k + 3);
  const int c0 = lane < parts ? __float_as_int(ld_dsmem_f32(dsmem_addr(smem_u32(&count[0]), lane))) : 0;
  int c1 = lane < parts ? __float_as_int(ld_dsmem_f32(dsmem_addr(smem_u32(&count[1]), lane))) : 0;
  if (rank == 0 && threadIdx.x == 0) {
    o[0] = (int)pick;
    o[k + 1] = __float_as_int(slp);
  }
  above = __reduce_add_sync(0xffffffffu, c0);
  if (rank == 0 && threadIdx.x == 0) o[2 * k + 2] = above + 1;
  if (k == 0) { cluster_sync(); return; }
  int n = __reduce_add_sync(0xffffffffu, c1);
  auto fit = [&]() { return !__any_sync(0xffffffffu, c1 > LIST) && n <= ALL; };                // the same in all threads of the cluster
  if (!fit()) {
    constexpr int SHARE = THREADS / 256;             // threads of a group, each compares with a share of the groups
    float fm = -INFINITY;
    int more = 0;                                    // above the bound
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      fm = fmaxf(fm, v[j]);
      more += v[j] > bound ? 1 : 0;
    }
    more = __reduce_add_sync(0xffffffffu, more);
    if (lane == 0 && more) atomicAdd(&count[2], more);
#pragma unroll
    for (int o = SHARE >> 1; o > 0; o >>= 1) fm = fmaxf(fm, __shfl_xor_sync(0xffffffffu, fm, o));
    const int mine_g = threadIdx.x / SHARE, first_g = threadIdx.x % SHARE * (256 / SHARE);
    if (threadIdx.x % SHARE == 0) row_groups[mine_g] = fm;
    if (threadIdx.x == 0) part[0] = -INFINITY;
    cluster_sync();                                  // (everybody has read the counts, too)
    if (threadIdx.x == 0) count[1] = 0;
    const int c2 = lane < parts ? __float_as_int(ld_dsmem_f32(dsmem_addr(smem_u32(&count[2]), lane))) + k : 0;
    if (__any_sync(0xffffffffu, c2 > LIST) || __reduce_add_sync(0xffffffffu, c2) > ALL) {
      int before = 0;
      for (int q = first_g; q < first_g + 256 / SHARE; q += 4) {
        const float4 y = *reinterpret_cast<const float4*>(row_groups + q);
        before += (y.x > fm || (y.x == fm && q < mine_g)) + (y.y > fm || (y.y == fm && q + 1 < mine_g)) + (y.z > fm || (y.z == fm && q + 2 < mine_g)) +
                  (y.w > fm || (y.w == fm && q + 3 < mine_g));
      }
#pragma unroll
      for (int o = SHARE >> 1; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
      if (before == k - 1 && fm == fm && threadIdx.x % SHARE == 0) part[0] = fm;
      cluster_sync();
      bound = fmaxf(bound, warp_max(lane < parts ? ld_dsmem_f32(dsmem_addr(smem_u32(&part[0]), lane)) : -INFINITY));
    } else {
      __syncthreads();                               // the count is 0 before anybody lists
    }
    int equal = 0;                                   // to the bound, of the CTA so far: in the order of their places
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      int mine = 0;
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const float x = v[j * N + u];
        if (x > bound) {
          const int m = atomicAdd(&count[1], 1);
          if (m < LIST) list[m] = make_float2(x, __int_as_float(at(j, u)));
        }
        mine += x == bound && at(j, u) < V ? 1 : 0;
      }
      if (equal >= k) continue;
      int inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += y; }
      if (lane == 31) tot[w] = inc;
      __syncthreads();
      const int t = lane < WARPS ? tot[lane] : 0;
      int r = equal + inc - mine + __reduce_add_sync(0xffffffffu, lane < w ? t : 0);
      equal += __reduce_add_sync(0xffffffffu, t);
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (v[j * N + u] == bound && at(j, u) < V && r++ < k) {
          const int m = atomicAdd(&count[1], 1);
          if (m < LIST) list[m] = make_float2(bound, __int_as_float(at(j, u)));
        }
      __syncthreads();
    }
    cluster_sync();
    c1 = lane < parts ? __float_as_int(ld_dsmem_f32(dsmem_addr(smem_u32(&count[1]), lane))) : 0;
    n = __reduce_add_sync(0xffffffffu, c1);
  }
  if (fit()) {
    if (rank == 0) {
      for (int q = w; q < parts; q += WARPS) {       // a warp copies a CTA's list
        const int first = __reduce_add_sync(0xffffffffu, lane < q ? c1 : 0), len = __shfl_sync(0xffffffffu, c1, q);
        for (int i = lane; i < len; i += 32) all[first + i] = ld_dsmem_f32x2(dsmem_addr(smem_u32(&list[i]), q));
      }
      __syncthreads();
      for (int r = n + threadIdx.x; r < k; r += THREADS) {           // (fewer numbers than k: the rest is NaN)
        o[1 + r] = 0;
        o[k + 2 + r] = __float_as_int((-INFINITY - mx) - lsum);
      }
      for (int i = threadIdx.x; i < n; i += THREADS) {
        const ArgMax me{all[i].x, __float_as_int(all[i].y)};
        int r = 0;
        for (int q = 0; q < n; ++q) r += all[q].x > me.v || (all[q].x == me.v && __float_as_int(all[q].y) < me.i) ? 1 : 0;
        if (r < k) {
          o[1 + r] = me.i;
          o[k + 2 + r] = __float_as_int((me.v - mx) - lsum);
        }
      }
    }
    cluster_sync();                                  // the first CTA reads the others' lists until here
    return;
  }
  // the likeliest of the thread's behind (value, place) in order
  auto next = [&](float old, int old_i) {
    ArgMax b{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const float x = v[j * N + u];
        const int i = at(j, u);
        if (i < V && (x < old || (x == old && i > old_i))) b = better(b, ArgMax{x, i});
      }
    return b;
  };
  auto warp_best = [&](ArgMax b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = better(b, ArgMax{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)});
    return b;
  };
  ArgMax best = next(INFINITY, -1);
  for (int r = 0; r < k; ++r) {                      // the warp's k likeliest
    const ArgMax t = warp_best(best);
    if (lane == 0) { lv[w * k + r] = t.v; li[w * k + r] = t.i; }
    if (t.i == 0x7fffffff) {                         // (no more than there are)
      for (int q = r + 1 + lane; q < k; q += 32) { lv[w * k + q] = -INFINITY; li[w * k + q] = 0x7fffffff; }
      break;
    }
    if (best.i == t.i) best = next(t.v, t.i);
  }
  // the k likeliest of n sorted lists, a list per lane
  auto merge = [&](int n, auto value, auto place, auto put) {
    int mine = 0;
    ArgMax head = lane < n ? ArgMax{value(lane, 0), place(lane, 0)} : ArgMax{-INFINITY, 0x7fffffff};
    for (int r = 0; r < k; ++r) {
      const ArgMax t = warp_best(head);
      if (lane == 0) put(r, t);
      if (t.i != 0x7fffffff && head.i == t.i) {
        ++mine;
        head = mine < k ? ArgMax{value(lane, mine), place(lane, mine)} : ArgMax{-INFINITY, 0x7fffffff};
      }
    }
  };
  __syncthreads();
  if (w == 0)
    merge(WARPS, [&](int l, int r) { return lv[l * k + r]; }, [&](int l, int r) { return li[l * k + r]; },
          [&](int r, ArgMax t) { lv[WARPS * k + r] = t.v; li[WARPS * k + r] = t.i; });
  cluster_sync();
  if (rank == 0 && w == 0)
    merge(parts, [&](int l, int r) { return ld_dsmem_f32(dsmem_addr(smem_u32(lv + WARPS * k + r), l)); },
          [&](int l, int r) { return __float_as_int(ld_dsmem_f32(dsmem_addr(smem_u32(li + WARPS * k + r), l))); },
          [&](int r, ArgMax t) {
            o[1 + r] = t.i == 0x7fffffff ? 0 : t.i;
            o[k + 2 + r] = __float_as_int((t.v - mx) - lsum);
          });
  cluster_sync();
}

// In-place top-k / top-p / min-p masking of fp32 logits (already divided by temperature).
// Per row: find the k-th largest value and the top-p probability threshold with a bisection on
// the value axis (each pass is one streaming read from L2/SMEM-resident row), then mask.
__global__ void __launch_bounds__(1024) topk_topp_kernel(float* __restrict__ logits, int V,
                                                          const int* __restrict__ top_k,
                                                          const float* __restrict__ top_p,
                                                          const float* __restrict__ min_p) {
  __shared__ float red[32];
  __shared__ float bc;
  const int row = blockIdx.x;
  float* lr = logits + (int64_t)row * V;
  const int k = top_k ? top_k[row] : 0;
  const float pth = top_p ? top_p[row] : 1.f;
  const float mp = min_p ? min_p[row] : 0.f;
  // row max / min
  float mx = -INFINITY, mn = INFINITY;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float x = lr[i];
    mx = fmaxf(mx, x);
    if (x > -INFINITY) mn = fminf(mn, x);
  }
  mx = warp_max(mx);
  mn = -warp_max(-mn);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) red[w] = mx;
  __syncthreads();
  if (w == 0) { float r = lane < nw ? red[lane] : -INFINITY; r = warp_max(r); if (lane == 0) bc = r; }
  __syncthreads();
  mx = bc;
  __syncthreads();
  if (lane == 0) red[w] = -mn;
  __syncthreads();
  if (w == 0) { float r = lane < nw ? red[lane] : -INFINITY; r = warp_max(r); if (lane == 0) bc = -r; }
  __syncthreads();
  mn = bc;
  __syncthreads();
  // Exact selection by bisection over the order-preserving integer image of the floats (32 passes build the
  // answer bit by bit): no sort, no scratch memory, ties at the boundary are kept like the sort-based reference.
  auto key_of = [](float x) -> uint32_t { const uint32_t u = __float_as_uint(x); return (u & 0x80000000u) ? ~u : (u | 0x80000000u); };
  auto val_of = [](uint32_t k) -> float { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); };
  float cut = -INFINITY;  // keep x >= cut
  if (k > 0 && k < V) {
    // k-th largest key = max { c : count(key >= c) >= k }
    uint32_t prefix = 0;
    for (int bit = 31; bit >= 0; --bit) {
      const uint32_t cand = prefix | (1u << bit);
      float cnt = 0.f;
      for (int i = threadIdx.x; i < V; i += blockDim.x) cnt += key_of(lr[i]) >= cand ? 1.f : 0.f;
      cnt = block_sum(cnt, red);
      if (cnt >= (float)k) prefix = cand;
    }
    cut = val_of(prefix);
  }
  if (pth < 1.f || mp > 0.f) {
    float z = 0.f;
    for (int i = threadIdx.x; i < V; i += blockDim.x) { const float x = lr[i]; if (x >= cut) z += __expf(x - mx); }
    z = block_sum(z, red);
    if (mp > 0.f) cut = fmaxf(cut, mx + __logf(mp));  // p_i >= min_p * p_max
    if (pth < 1.f) {
      // nucleus: an element is dropped iff the probability mass of everything <= it is <= 1 - top_p.
      // smallest kept key = max { c : mass(key < c) <= (1 - top_p) * Z }
      const float thr = (1.f - pth) * z;
      const uint32_t kcut = key_of(cut);
      uint32_t prefix = 0;
      for (int bit = 31; bit >= 0; --bit) {
        const uint32_t cand = prefix | (1u << bit);
        float mass = 0.f;
        for (int i = threadIdx.x; i < V; i += blockDim.x) {
          const float x = lr[i];
          const uint32_t kx = key_of(x);
          if (kx >= kcut && kx < cand) mass += __expf(x - mx);
        }
        mass = block_sum(mass, red);
        if (mass <= thr) prefix = cand;
      }
      // never drop the arg-max (mass rounding): the largest element always survives
      cut = fmaxf(cut, fminf(val_of(prefix), mx));
    }
  }
  for (int i = threadIdx.x; i < V; i += blockDim.x)
    if (lr[i] < cut) lr[i] = -INFINITY;
}

// logits[b, v] adjusted by repetition / frequency / presence penalties given token histories.
__global__ void penalties_kernel(float* __restrict__ logits, int V, const int* __restrict__ prompt_mask_bits,
                                 const int* __restrict__ out_counts, const float* __restrict__ presence,
                                 const float* __restrict__ frequency, const float* __restrict__ repetition) {
  const int row = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V) return;
  const int cnt = out_counts[(int64_t)row * V + i];
  const bool in_prompt = prompt_mask_bits ? (prompt_mask_bits[(int64_t)row * ((V + 31) / 32) + (i >> 5)] >> (i & 31)) & 1 : false;
  float x = logits[(int64_t)row * V + i];
  if (in_prompt || cnt > 0) {
    const float rp = repetition[row];
    x = x > 0.f ? x / rp : x * rp;
  }
  x -= frequency[row] * (float)cnt;
  if (cnt > 0) x -= presence[row];
  logits[(int64_t)row * V + i] = x;
}

// per-row log-softmax statistics: out_lse[row] = logsumexp(logits[row])
template <typename T>
__global__ void __launch_bounds__(1024) row_lse_kernel(const T* __restrict__ logits, int64_t row_stride, int V,
                                                        float* __restrict__ out_lse) {
  __shared__ float red[32];
  __shared__ float bc;
  const int row = blockIdx.x;
  const T* lr = logits + (int64_t)row * row_stride;
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, to_f32(lr[i]));
  mx = warp_max(mx);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) red[w] = mx;
  __syncthreads();
  if (w == 0) { float r = lane < nw ? red[lane] : -INFINITY; r = warp_max(r); if (lane == 0) bc = r; }
  __syncthreads();
  mx = bc;
  __syncthreads();
  float s = 0.f;
  for (int i = threadIdx.x; i < V; i += blockDim.x) s += __expf(to_f32(lr[i]) - mx);
  s = block_sum(s, red);
  if (threadIdx.x == 0) out_lse[row] = mx + __logf(s);
}

}  // namespace

EXPORT int vb_argmax(const void* logits, int64_t row_stride, int B, int V, int64_t* out, int dtype, cudaStream_t st) {
  if (B == 0) return 0;
  DISPATCH_DTYPE(dtype, TT, {
    sample_kernel<TT, false><<<B, 1024, 0, st>>>((const TT*)logits, row_stride, V, nullptr, nullptr, nullptr, out, 0, nullptr);
  });
  return (int)cudaGetLastError();
}

EXPORT int vb_fused_sample(const void* logits, int64_t row_stride, int B, int V, const float* temperature,
                           const int64_t* seeds, const int* step, int64_t* out, int dtype, cudaStream_t st) {
  if (B == 0) return 0;
  DISPATCH_DTYPE(dtype, TT, {
    vb_launch(sample_kernel<TT, true>, B, 1024, 0, st, (const TT*)logits, row_stride, V, temperature, seeds, step, out, 0, (float4*)nullptr);
  });
  return (int)cudaGetLastError();
}

// TP vocab shards: every rank samples over ITS shard (global ids = idx_off + local id, V = valid local rows) and emits one
// (value, id) candidate per row; after a 16-byte-per-row all-gather vb_select_candidate picks the winner — the 2 MiB of
// logits per rank that the full all-gather moved never leave the GPU.
EXPORT int vb_fused_sample_cand(const void* logits, int64_t row_stride, int B, int V, const float* temperature,
                                const int64_t* seeds, const int* step, int idx_off, void* cand, int dtype, cudaStream_t st) {
  if (B == 0) return 0;
  DISPATCH_DTYPE(dtype, TT, {
    vb_launch(sample_kernel<TT, true>, B, 1024, 0, st, (const TT*)logits, row_stride, V, temperature, seeds, step,
              (int64_t*)nullptr, idx_off, (float4*)cand);
  });
  return (int)cudaGetLastError();
}
EXPORT int vb_select_candidate(const void* cands, int W, int64_t* out, int B, cudaStream_t st) {
  if (B == 0) return 0;
  vb_launch(select_candidate_kernel, dim3((B + 127) / 128), dim3(128), 0, st, (const float4*)cands, W, out, B);
  return (int)cudaGetLastError();
}

EXPORT int vb_topk_topp(float* logits, int B, int V, const int* top_k, const float* top_p, const float* min_p,
                        cudaStream_t st) {
  if (B == 0) return 0;
  topk_topp_kernel<<<B, 1024, 0, st>>>(logits, V, top_k, top_p, min_p);
  return (int)cudaGetLastError();
}

EXPORT int vb_penalties(float* logits, int B, int V, const int* prompt_mask_bits, const int* out_counts,
                        const float* presence, const float* frequency, const float* repetition, cudaStream_t st) {
  if (B == 0) return 0;
  penalties_kernel<<<dim3((V + 255) / 256, B), 256, 0, st>>>(logits, V, prompt_mask_bits, out_counts, presence,
                                                              frequency, repetition);
  return (int)cudaGetLastError();
}

EXPORT int vb_row_lse(const void* logits, int64_t row_stride, int B, int V, float* out, int dtype, cudaStream_t st) {
  if (B == 0) return 0;
  DISPATCH_DTYPE(dtype, TT, {
    row_lse_kernel<TT><<<B, 1024, 0, st>>>((const TT*)logits, row_stride, V, out);
  });
  return (int)cudaGetLastError();
}

// k <= V; rows 16-byte aligned (row_stride a multiple of 16 bytes).  alone: a CTA per row whatever B and k are, as the two forms add in different orders
static int logprobs(const void* logits, int64_t row_stride, int B, int V, const int64_t* sampled, int k, int* out, bool alone, int dtype, cudaStream_t st) {
  if (B == 0) return 0;
  if (k < 0 || k > V) return -1;
  // Clusters for up to 7.5 M values: beyond that there are rows enough for all SMs, and a CTA per row has less to exchange, while k is small (its
  // cost grows with k).  us for k = 5, clusters and CTAs: 128 rows of 32000 15 and 24, 256 29 and 24, 512 56 and 44; 64 rows of 102400 44 and 50, 128 79 and 58.
  if (!alone && B <= INT32_MAX / 8 && V <= 8 * 32 * 1024 && k <= 64 && (k > 8 || (int64_t)B * V <= 7500000)) {
    // the smallest CTAs of which eight hold a row
    const int threads = V <= 8 * 32 * 256 ? 256 : V <= 8 * 32 * 512 ? 512 : 1024, parts = (V + threads * 32 - 1) / (threads * 32);
    const size_t smem = (size_t)2 * (threads / 32 + 1) * k * 4;
    DISPATCH_DTYPE(dtype, T, {
      auto* kernel = threads == 256 ? logprobs_cluster_kernel<T, 256> : threads == 512 ? logprobs_cluster_kernel<T, 512> : logprobs_cluster_kernel<T, 1024>;
      vb_launch_parts(kernel, dim3(B * parts), dim3(threads), smem, st, parts, reinterpret_cast<const T*>(logits), row_stride, V, sampled, k, out, parts);
    });
    return (int)cudaGetLastError();
  }
  DISPATCH_DTYPE(dtype, T, vb_launch(logprobs_kernel<T>, dim3(B), dim3(1024), 0, st, reinterpret_cast<const T*>(logits), row_stride, V, sampled, k, out));
  return (int)cudaGetLastError();
}
EXPORT int vb_logprobs(const void* logits, int64_t row_stride, int B, int V, const int64_t* sampled, int k, int* out, int dtype, cudaStream_t st) {
  return logprobs(logits, row_stride, B, V, sampled, k, out, false, dtype, st);
}
EXPORT int vb_logprobs_alone(const void* logits, int64_t row_stride, int B, int V, const int64_t* sampled, int k, int* out, int dtype, cudaStream_t st) {
  return logprobs(logits, row_stride, B, V, sampled, k, out, true, dtype, st);
}
