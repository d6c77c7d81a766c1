// GPU-side input preparation for the model runner: the per-token step inputs are expanded ON THE DEVICE from
// per-request state that already lives there, so the host ships O(requests) scalars per step instead of O(tokens)
// arrays and O(requests x blocks) block tables.
//
// Reference: vllm/v1/worker/gpu/input_batch.py:253-697 (Triton kernels prepare_prefill_inputs / prepare_pos_seq_lens /
// combine_sampled_and_draft_tokens), block_table.py:228-330 (_gather_block_tables / _compute_slot_mappings),
// buffer_utils.py:114-310 (staged writes).  Ours: three small sm_100a kernels over persistent device tensors
//   token_table [max_reqs, max_len] int32   every request's prompt + generated ids (sampled ids are appended on the
//                                           device by `publish`, never round-tripping through the host)
//   block_rows  [groups][max_reqs, max_blocks] int32   row-ordered block tables, patched by staged row changes
// A step is one host-to-device copy of a packed buffer and one fused expansion for all KV groups; where requests came, left or took pages, `row_update` runs
// before it, once for rows that moved (again for each that waits for another's old place) and once for what is new.  Above eight groups each is
// launched for eight at a time.
//   (req row, num_computed, num_scheduled) x nb  →  input_ids[T], positions[T], query_start_loc[nb+1], seq_lens[nb],
//                                                    slot_mapping[g][T], block_table[g][nb, nblk]
// and, behind the forward pass, `publish`, which writes the step's results to the host as well.
#include "common.cuh"

namespace {

constexpr int MAX_GROUPS = 8;      // KV groups of one launch

struct Prep {
  const int* rows; const int* num_computed; const int* num_sched;
  const int* token_table;
  int* input_ids; int64_t* positions; int* qsl; int* seq_lens; int64_t* last;
  const int64_t* pos_delta;
  const int* block_rows[MAX_GROUPS];
  int64_t* slot_mapping[MAX_GROUPS];
  int* block_table[MAX_GROUPS];
  int64_t tt_stride, br_stride, bt_stride;
  int nb, nblk, block_size, write_tokens, pad_t;
};

// One CTA per scheduled request and KV group (group 0 writes what the groups share).  qsl (exclusive prefix sum of num_sched) is computed by
// every CTA for its own request with a short loop (nb <= a few thousand) — no second launch, no host-side cumsum.
// Latency is all it costs (3 us for 64 rows); a launch per group was another 3 us and 25 us of host time each.
__global__ void __launch_bounds__(256) prep_step_kernel(const __grid_constant__ Prep p) {
  __shared__ int s_off;
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x, nb = p.nb, pad_t = p.pad_t;
  const bool write_tokens = p.write_tokens && blockIdx.y == 0;
  int64_t* slot_mapping = p.slot_mapping[blockIdx.y];
  int* bt = p.block_table[blockIdx.y] + (int64_t)b * p.bt_stride;
  // exclusive prefix of num_sched[0..min(b, nb))
  int part = 0;
  for (int i = threadIdx.x; i < min(b, nb); i += blockDim.x) part += p.num_sched[i];
  __shared__ int red[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) red[w] = part;
  __syncthreads();
  if (w == 0) {
    int v = lane < (int)(blockDim.x >> 5) ? red[lane] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) s_off = v;
  }
  __syncthreads();
  const int off = s_off;
  if (b >= nb && pad_t > 0) {
    // mixed-batch bucket: padding REQUESTS are empty (query length 0 — the flat attention schedule skips them, their
    // "last token" index resolves to the batch's last real token), padding TOKENS [T, pad_t) sit at position 0 and
    // write to no cache slot; the extra CTA b == gridDim.x - 1 fills the token padding
    if (threadIdx.x == 0 && b < (int)gridDim.x - 1) {
      if (write_tokens) { p.qsl[b + 1] = off; p.seq_lens[b] = 1; }
      bt[0] = 0;
    }
    if (b == (int)gridDim.x - 1)
      for (int i = off + threadIdx.x; i < pad_t; i += blockDim.x) {
        if (write_tokens) { p.input_ids[i] = 0; p.positions[i] = 0; }
        slot_mapping[i] = -1;
      }
    return;
  }
  if (b >= nb) {
    // padding slot of a decode bucket: one token at position 0 that writes to no cache slot and attends over one
    // token of the null block (same convention as the host path, worker/model_runner.py `_h2d`)
    if (threadIdx.x == 0) {
      const int idx = off + (b - nb);
      if (write_tokens) {
        p.input_ids[idx] = 0;
        p.positions[idx] = 0;
        p.qsl[b + 1] = idx + 1;
        p.seq_lens[b] = 1;
      }
      slot_mapping[idx] = -1;
      bt[0] = 0;
    }
    return;
  }
  const int row = p.rows[b], nc = p.num_computed[b], ns = p.num_sched[b];
  if (threadIdx.x == 0 && write_tokens) {
    p.qsl[b] = off;
    if (b == nb - 1) p.qsl[nb] = off + ns;
    p.seq_lens[b] = nc + ns;
    if (p.last) p.last[b] = off + ns - 1;
  }
  const int* toks = p.token_table + (int64_t)row * p.tt_stride;
  const int* blks = p.block_rows[blockIdx.y] + (int64_t)row * p.br_stride;
  const int64_t delta = p.pos_delta ? p.pos_delta[b] : 0;       // M-RoPE: rotary position runs behind the sequence index
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    const int pos = nc + i;
    if (write_tokens) {
      p.input_ids[off + i] = toks[pos];
      p.positions[off + i] = (int64_t)pos + delta;
    }
    slot_mapping[off + i] = (int64_t)blks[pos / p.block_size] * p.block_size + pos % p.block_size;
  }
  for (int i = threadIdx.x; i < p.nblk; i += blockDim.x) bt[i] = blks[i];
}

struct Tables {                    // rows of `stride` ints: the requests' tokens, their blocks per KV group
  int* at[MAX_GROUPS + 1];
  int64_t stride[MAX_GROUPS + 1];
};

// staged row changes: entry e puts cnt[e] ints into row row[e] of table tbl[e] (null: the first) from start[e] on.  They come from
// ids[off[e] ..] or (moved) from the beginning of row off[e] of the same table.  One launch for all tables and rows of a step.
__global__ void __launch_bounds__(128) row_update_kernel(const __grid_constant__ Tables t, const int* __restrict__ tbl, const int* __restrict__ row,
                                                          const int* __restrict__ start, const int* __restrict__ cnt,
                                                          const int* __restrict__ off, const int* ids, int moved) {
  pdl_trigger();
  pdl_wait();
  const int e = blockIdx.x, g = tbl ? tbl[e] : 0, n = cnt[e];
  int* dst = t.at[g] + (int64_t)row[e] * t.stride[g] + start[e];
  const int* src = moved ? t.at[g] + (int64_t)off[e] * t.stride[g] : ids + off[e];
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

// token_table[row[b], pos[b]] = sampled[b]  (the ids a step produced become the next step's inputs without a D2H/H2D); the ids and the
// packed log-probabilities also go straight to pinned host memory, where a reader finds them after the event behind this launch.  Two
// device-to-host copies and an index copy instead took 17 us after the last kernel of a step.
__global__ void __launch_bounds__(256) publish_kernel(int* __restrict__ token_table, int64_t tt_stride, const int* __restrict__ rows,
                                                       const int* __restrict__ pos, const int64_t* __restrict__ sampled, int nb,
                                                       int64_t* __restrict__ host_ids, const int* __restrict__ lp, int* __restrict__ host_lp,
                                                       int64_t n_lp) {
  pdl_trigger();
  pdl_wait();
  const int64_t at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, all = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b = at; b < nb; b += all) {
    if (pos[b] >= 0) token_table[(int64_t)rows[b] * tt_stride + pos[b]] = (int)sampled[b];
    if (host_ids) host_ids[b] = sampled[b];
  }
  for (int64_t i = at; i < n_lp; i += all) host_lp[i] = lp[i];
}

}  // namespace

// pad_b >= nb: entries [nb, pad_b) are graph-bucket padding; pad_t > 0: mixed-batch bucket of pad_t tokens / pad_b requests (empty padding
// requests + padding tokens).  Groups differ in block_rows, slot_mapping and block_table only; write_tokens: the first writes the rest.
// last: optional, where a request's last scheduled token is.
EXPORT int vb_prep_step4(const int* rows, const int* num_computed, const int* num_sched, int nb, int pad_b, int pad_t, const int* token_table,
                         int64_t tt_stride, int groups, const int* const* block_rows, int64_t br_stride, int* input_ids, int64_t* positions,
                         int* qsl, int* seq_lens, int64_t* last, int64_t* const* slot_mapping, int* const* block_table, int64_t bt_stride,
                         int nblk, int block_size, const int64_t* pos_delta, int write_tokens, cudaStream_t st) {
  if (pad_b <= 0) return 0;
  for (int g0 = 0; g0 < groups; g0 += MAX_GROUPS) {
    const int n = groups - g0 < MAX_GROUPS ? groups - g0 : MAX_GROUPS;
    Prep p = {};
    p.rows = rows; p.num_computed = num_computed; p.num_sched = num_sched; p.token_table = token_table; p.input_ids = input_ids;
    p.positions = positions; p.qsl = qsl; p.seq_lens = seq_lens; p.last = last; p.pos_delta = pos_delta; p.tt_stride = tt_stride;
    p.br_stride = br_stride; p.bt_stride = bt_stride; p.nb = nb; p.nblk = nblk; p.block_size = block_size;
    p.write_tokens = write_tokens && g0 == 0; p.pad_t = pad_t;
    for (int g = 0; g < n; ++g) {
      p.block_rows[g] = block_rows[g0 + g]; p.slot_mapping[g] = slot_mapping[g0 + g]; p.block_table[g] = block_table[g0 + g];
    }
    vb_launch(prep_step_kernel, dim3(pad_t > 0 ? pad_b + 1 : pad_b, n), dim3(256), 0, st, p);
  }
  return (int)cudaGetLastError();
}

// tables [n_tables]; tbl may be null (all entries in the first)
EXPORT int vb_row_update(int* const* tables, const int64_t* strides, int n_tables, const int* tbl, const int* row, const int* start,
                         const int* cnt, const int* off, const int* ids, int n, int moved, cudaStream_t st) {
  if (n == 0) return 0;
  if (n_tables < 1 || n_tables > MAX_GROUPS + 1) return -1;
  Tables t = {};
  for (int i = 0; i < n_tables; ++i) { t.at[i] = tables[i]; t.stride[i] = strides[i]; }
  vb_launch(row_update_kernel, dim3(n), dim3(128), 0, st, t, tbl, row, start, cnt, off, ids, moved);
  return (int)cudaGetLastError();
}

// host_ids, host_lp (n_lp ints from lp): pinned host memory, both optional
EXPORT int vb_publish(int* token_table, int64_t tt_stride, const int* rows, const int* pos, const int64_t* sampled, int nb, int64_t* host_ids,
                      const int* lp, int* host_lp, int64_t n_lp, cudaStream_t st) {
  if (nb == 0) return 0;
  const int64_t most = n_lp > nb ? n_lp : nb;
  vb_launch(publish_kernel, dim3((unsigned)(most > 256 * 64 ? 64 : (most + 255) / 256)), dim3(256), 0, st, token_table, tt_stride, rows, pos, sampled,
            nb, host_ids, lp, host_lp, n_lp);
  return (int)cudaGetLastError();
}
