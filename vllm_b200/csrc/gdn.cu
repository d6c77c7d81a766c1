// Gated delta rule over the paged recurrent states (Qwen3-Next, OLMo-hybrid), prompts and decode steps alike.  Per value head, state S [dk, dv]:
//
//   S *= a;  d = (v - S^T k) b;  S += k d^T;  o = S^T q        q, k l2-normalised, q times dk^-1/2
//   a = exp(-exp(A_log) softplus(x_a + dt_bias)),  b = sigmoid(x_b) beta_scale
//
// all in 32 bits on the CUDA cores, the recurrence itself: a token costs two dot products of the OLD state (o = a S^T q + d (k . q)) and one
// rank-1 update, a chain that no other token of the request can start before it ends, so its latency is the cost (8 prompts of 860 tokens:
// instructions issue in 42 % of the cycles, most stalls are for the instruction before; DRAM at 4 %).
//
// CTA = four warps of one (request, head); a warp owns 4 CW columns of S, a lane 4 NI rows (rg) x CW columns (cg) of them in registers, as
// pairs of rows for packed products.  The decay is kept aside (S = A S', A the running product, folded in before it gets small) instead of
// being multiplied through.  The 2 CW sums of a column group are reduced over the eight row groups by halving what a lane keeps at
// each exchange (7 shuffles for CW = 4 instead of 24).  q, k and v rows of sixteen tokens at a time are copied to shared memory ahead of
// their use; norms, k . q and the gates of a token are evaluated once per CTA.
//
// Measured against a warp per column with strided loads and two full reductions: 8 heads of 128 x 256, 8 prompts of 860 tokens 3408 → 456 us,
// one of 4000 5747 → 1459 us, 24 decode steps 65 → 19 us; 32 heads of 128 x 128, 8 prompts 5910 → 851 us, 64 decode steps 310 → 52 us.  (With v
// read from global memory token by token and eight tokens at a time, 560, 2313, 20, 1096 and 56 us: the loads of v were on the chain.)
#include "common.cuh"

namespace gdn {

constexpr int WARPS = 4, CHUNK = 16;

struct Params {
  const float* q; const float* k; const float* v;    // heads of a token next to each other, rows `stride` apart
  const void* ba;          // [T, 2 nv] raw: per key head r write strengths, then r decays (r = nv / nk)
  const float* A_log; const float* dt_bias;
  const float* g; const float* beta;                 // or, where ba is null, [T, nv] log decays and write strengths; q, k normalised
  float* o;                // [T, nv dv]
  float* state;            // rows of state_stride floats, [nv, dk, dv] at state_off
  const int* qsl; const int* seq_lens; const int* rows;
  int64_t q_stride, v_stride, ba_stride, state_stride, state_off, rows_stride;
  int nk, nv, dv;
  float q_scale, beta_scale, eps;
};

VB_DEVICE uint64_t pk(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
VB_DEVICE void upk(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
VB_DEVICE uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r;
}
VB_DEVICE uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
VB_DEVICE void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// VEC: columns, rows of qkv and states are 16-byte aligned in groups of CW (dv a multiple of 4)
template <typename T, int NI, int CW, bool VEC>
__global__ void __launch_bounds__(WARPS * 32) gdn_kernel(const Params p) {
  constexpr int DK = 32 * NI, LC = 4 * CW;                     // columns of a warp
  constexpr int BC = WARPS * LC;                               // columns of the CTA
  extern __shared__ __align__(16) float gdn_smem[];
  float (*kq)[CHUNK][2][DK] = reinterpret_cast<float (*)[CHUNK][2][DK]>(gdn_smem);                 // [2 buffers]
  float (*vs)[CHUNK][BC] = reinterpret_cast<float (*)[CHUNK][BC]>(gdn_smem + 2 * CHUNK * 2 * DK);  // [2 buffers]
  __shared__ float4 scal[2][CHUNK];                            // a, b, 1 / |k|, dk^-1/2 / |q|
  __shared__ float kdot_s[2][CHUNK];                           // k . q, normalised
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 2, cg = lane & 3;
  const int blocks = (p.dv + WARPS * LC - 1) / (WARPS * LC);
  const int h = blockIdx.x / blocks, r = blockIdx.y;
  const int bcol0 = (blockIdx.x % blocks) * BC, col0 = bcol0 + warp * LC + cg * CW;
  const int t0 = p.qsl[r], n = p.qsl[r + 1] - t0;
  if (n <= 0) return;
  const int per = p.nv / p.nk, kh = h / per;
  const float* qp = p.q + (int64_t)t0 * p.q_stride + kh * DK;
  const float* kp = p.k + (int64_t)t0 * p.q_stride + kh * DK;
  const float* vp = p.v + (int64_t)t0 * p.v_stride + (int64_t)h * p.dv;
  const T* ba = reinterpret_cast<const T*>(p.ba) + (int64_t)t0 * p.ba_stride + kh * 2 * per + (h - kh * per);
  const float decay_rate = p.ba ? -expf(p.A_log[h]) : 0.f, dt_bias = p.ba ? p.dt_bias[h] : 0.f;
  const bool has_init = p.seq_lens[r] > n;
  float* st = p.state + (int64_t)p.rows[r * p.rows_stride] * p.state_stride + p.state_off + (int64_t)h * DK * p.dv;

  // tokens c .. c + CHUNK - 1: q and k rows to shared memory
  auto stage = [&](int c) {
    const int buf = (c / CHUNK) & 1, m = min(CHUNK, n - c);
    for (int i = threadIdx.x; i < m * 2 * (DK / 4); i += WARPS * 32) {
      const int t = i / (2 * (DK / 4)), w = i % (2 * (DK / 4)), part = w / (DK / 4), x = (w % (DK / 4)) * 4;     // part 0: k, 1: q
      cp16(&kq[buf][t][part][x], (part ? qp : kp) + (int64_t)(c + t) * p.q_stride + x);
    }
    const int left = min(BC, p.dv - bcol0);                    // columns that exist
    if constexpr (VEC) {
      for (int i = threadIdx.x; i < m * (BC / 4); i += WARPS * 32) {
        const int t = i / (BC / 4), x = (i % (BC / 4)) * 4;
        if (x < left) cp16(&vs[buf][t][x], vp + (int64_t)(c + t) * p.v_stride + bcol0 + x);
      }
    } else {
      for (int i = threadIdx.x; i < m * BC; i += WARPS * 32) {
        const int t = i / BC, x = i % BC;
        if (x < left) vs[buf][t][x] = vp[(int64_t)(c + t) * p.v_stride + bcol0 + x];
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // eight threads per token: its norms and k . q; the raw gates were loaded a chunk before
  constexpr int PT = WARPS * 32 / CHUNK;
  const int st_t = threadIdx.x / PT, st_l = threadIdx.x % PT;
  float raw_b = 0.f, raw_a = 0.f;
  auto raw = [&](int c) {
    if (st_l == 0 && c + st_t < n) {
      if (p.ba) {
        raw_b = to_f32(ba[(int64_t)(c + st_t) * p.ba_stride]);
        raw_a = to_f32(ba[(int64_t)(c + st_t) * p.ba_stride + per]);
      } else {
        raw_b = p.beta[(int64_t)(t0 + c + st_t) * p.nv + h];
        raw_a = p.g[(int64_t)(t0 + c + st_t) * p.nv + h];
      }
    }
  };
  raw(0);
  stage(0);

  uint64_t S[CW][2 * NI];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float x[2][CW];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float* src = st + (int64_t)(32 * i + rg * 4 + 2 * j + u) * p.dv + col0;
        if constexpr (VEC) {
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (has_init && col0 < p.dv) {
            if constexpr (CW == 4) f = *reinterpret_cast<const float4*>(src);
            else { const float2 g = *reinterpret_cast<const float2*>(src); f.x = g.x; f.y = g.y; }
          }
          x[u][0] = f.x; x[u][1] = f.y;
          if constexpr (CW == 4) { x[u][2] = f.z; x[u][3] = f.w; }
        } else {
#pragma unroll
          for (int c = 0; c < CW; ++c) x[u][c] = has_init && col0 + c < p.dv ? src[c] : 0.f;
        }
      }
#pragma unroll
      for (int c = 0; c < CW; ++c) S[c][2 * i + j] = pk(x[0][c], x[1][c]);
    }

  // what a lane holds after the reduction: of column own (of its group) the product with k (lower half of the warp) or with q
  const int own = CW == 4 ? rg & 3 : (rg >> 1) & 1, my_col = col0 + own;
  const bool has_q = rg >= 4;
  float A = 1.f;
  for (int c = 0; c < n; c += CHUNK) {
    const int buf = (c / CHUNK) & 1, m = min(CHUNK, n - c);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (c + CHUNK < n) stage(c + CHUNK);
    {
      float kk = 0.f, qq = 0.f, kd = 0.f;
      if (st_t < m) {
#pragma unroll
        for (int i = 0; i < DK / PT; ++i) {
          const float a = kq[buf][st_t][0][st_l + PT * i], b = kq[buf][st_t][1][st_l + PT * i];
          kk += a * a; qq += b * b; kd += a * b;
        }
      }
#pragma unroll
      for (int o = PT / 2; o > 0; o >>= 1) {
        kk += __shfl_xor_sync(0xffffffffu, kk, o);
        qq += __shfl_xor_sync(0xffffffffu, qq, o);
        kd += __shfl_xor_sync(0xffffffffu, kd, o);
      }
      if (st_l == 0 && st_t < m) {
        float ik = 1.f, iq = 1.f, a = raw_a, b = raw_b;
        if (p.ba) {
          const float x = raw_a + dt_bias, soft = x > 20.f ? x : log1pf(expf(x));
          ik = 1.f / sqrtf(kk + p.eps); iq = p.q_scale / sqrtf(qq + p.eps);
          a = decay_rate * soft; b = p.beta_scale / (1.f + expf(-raw_b));
        }
        scal[buf][st_t] = make_float4(expf(a), b, ik, iq);
        kdot_s[buf][st_t] = kd * ik * iq;
      }
      raw(c + CHUNK);
    }
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < m; ++t) {
      const float4 s = scal[buf][t];
      const float kdot = kdot_s[buf][t], v = my_col < p.dv ? vs[buf][t][my_col - bcol0] : 0.f;
      A *= s.x;
      uint64_t kv[2 * NI], a1[CW], a2[CW];
#pragma unroll
      for (int i = 0; i < CW; ++i) a1[i] = a2[i] = 0ull;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const float4 k4 = *reinterpret_cast<const float4*>(&kq[buf][t][0][32 * i + rg * 4]);
        const float4 q4 = *reinterpret_cast<const float4*>(&kq[buf][t][1][32 * i + rg * 4]);
        kv[2 * i] = pk(k4.x, k4.y); kv[2 * i + 1] = pk(k4.z, k4.w);
        const uint64_t q0 = pk(q4.x, q4.y), q1 = pk(q4.z, q4.w);
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          a1[j] = fma2(S[j][2 * i], kv[2 * i], a1[j]);
          a2[j] = fma2(S[j][2 * i], q0, a2[j]);
          a1[j] = fma2(S[j][2 * i + 1], kv[2 * i + 1], a1[j]);
          a2[j] = fma2(S[j][2 * i + 1], q1, a2[j]);
        }
      }
      float dot[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        float k0, k1, q0, q1;
        upk(a1[j], k0, k1); upk(a2[j], q0, q1);
        k0 += k1; q0 += q1;
        const float away = __shfl_xor_sync(0xffffffffu, has_q ? k0 : q0, 16);
        dot[j] = (has_q ? q0 : k0) + away;
      }
      float mine;
      if constexpr (CW == 4) {
        const bool up = rg & 2;
        const float b0 = __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 8), b1 = __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 8);
        const float e0 = (up ? dot[2] : dot[0]) + b0, e1 = (up ? dot[3] : dot[1]) + b1;
        const bool odd = rg & 1;
        mine = (odd ? e1 : e0) + __shfl_xor_sync(0xffffffffu, odd ? e0 : e1, 4);
      } else {
        const bool up = rg & 2;
        mine = (up ? dot[1] : dot[0]) + __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[1], 8);
        mine += __shfl_xor_sync(0xffffffffu, mine, 4);
      }
      mine *= A;
      // lower half: d of the own column; upper half: S^T q of it
      const float d = (v - mine * s.z) * s.y;
      const float other = __shfl_xor_sync(0xffffffffu, d, 16);
      if (has_q && my_col < p.dv && (CW == 4 || !(rg & 1))) p.o[(int64_t)(t0 + c + t) * p.nv * p.dv + (int64_t)h * p.dv + my_col] = mine * s.w + other * kdot;
      float dc[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) dc[j] = __shfl_sync(0xffffffffu, d, (CW == 4 ? j * 4 : j * 8) + cg);
      if (A < 1.52587890625e-05f) {                            // 2^-16: fold the decay in (0 included)
        const uint64_t aa = pk(A, A);
#pragma unroll
        for (int j = 0; j < CW; ++j)
#pragma unroll
          for (int i = 0; i < 2 * NI; ++i) S[j][i] = mul2(S[j][i], aa);
        A = 1.f;
      }
      const float f = __fdividef(s.z, A);
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        const uint64_t dd = pk(dc[j] * f, dc[j] * f);
#pragma unroll
        for (int i = 0; i < 2 * NI; ++i) S[j][i] = fma2(kv[i], dd, S[j][i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float x[2][CW];
#pragma unroll
      for (int c = 0; c < CW; ++c) {
        upk(S[c][2 * i + j], x[0][c], x[1][c]);
        x[0][c] *= A; x[1][c] *= A;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float* dst = st + (int64_t)(32 * i + rg * 4 + 2 * j + u) * p.dv + col0;
        if constexpr (VEC) {
          if (col0 < p.dv) {
            if constexpr (CW == 4) *reinterpret_cast<float4*>(dst) = make_float4(x[u][0], x[u][1], x[u][2], x[u][3]);
            else *reinterpret_cast<float2*>(dst) = make_float2(x[u][0], x[u][1]);
          }
        } else {
#pragma unroll
          for (int c = 0; c < CW; ++c) if (col0 + c < p.dv) dst[c] = x[u][c];
        }
      }
    }
}

template <typename T, int NI, int CW>
static int launch(const Params& p, bool vec, int num_reqs, cudaStream_t st) {
  const int blocks = (p.dv + WARPS * 4 * CW - 1) / (WARPS * 4 * CW);
  const dim3 grid(p.nv * blocks, num_reqs);
  const size_t smem = (size_t)2 * CHUNK * (2 * 32 * NI + WARPS * 4 * CW) * sizeof(float);
  auto k = vec ? gdn_kernel<T, NI, CW, true> : gdn_kernel<T, NI, CW, false>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -5;
  vb_launch(k, grid, dim3(WARPS * 32), smem, st, p);
  return (int)cudaGetLastError();
}

}  // namespace gdn

// dk is a multiple of 32 up to 256; rows of q and k start on 16 bytes.  ba or, with normalised q and k (nk = nv), g and beta.
EXPORT int vb_gated_delta(const float* q, const float* k, int64_t q_stride, const float* v, int64_t v_stride, const void* ba, int64_t ba_stride,
                          const float* A_log, const float* dt_bias, const float* g, const float* beta, float* o, float* state,
                          int64_t state_stride, int64_t state_off, const int* qsl, const int* seq_lens, const int* rows, int64_t rows_stride,
                          int num_reqs, int nk, int nv, int dk, int dv, float q_scale, float beta_scale, float eps, int dtype, cudaStream_t st) {
  using namespace gdn;
  if (num_reqs == 0) return 0;
  if (dk % 32 || dk < 32 || dk > 256 || nk < 1 || nv % nk || dv < 1 || q_stride % 4 || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k)) & 15) ||
      (ba ? !A_log || !dt_bias : !g || !beta || nk != nv))
    return -1;
  Params p;
  p.q = q; p.k = k; p.v = v; p.ba = ba; p.A_log = A_log; p.dt_bias = dt_bias; p.g = g; p.beta = beta; p.o = o; p.state = state; p.qsl = qsl;
  p.seq_lens = seq_lens; p.rows = rows; p.q_stride = q_stride; p.v_stride = v_stride; p.ba_stride = ba_stride; p.state_stride = state_stride;
  p.state_off = state_off; p.rows_stride = rows_stride; p.nk = nk; p.nv = nv; p.dv = dv; p.q_scale = q_scale; p.beta_scale = beta_scale; p.eps = eps;
  const bool vec = dv % 4 == 0 && v_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(v) & 15) == 0 && state_stride % 4 == 0 && state_off % 4 == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0;
#define GO(NI, CW) launch<T, NI, CW>(p, vec, num_reqs, st)
  DISPATCH_DTYPE(dtype, T, {
    switch (dk / 32) {
      case 1: return GO(1, 4);
      case 2: return GO(2, 4);
      case 3: return GO(3, 4);
      case 4: return GO(4, 4);
      case 5: return GO(5, 2);
      case 6: return GO(6, 2);
      case 7: return GO(7, 2);
      default: return GO(8, 2);
    }
  });
#undef GO
  return -1;
}
