// Paged causal attention in float32 for rows of several queries (prompts and portions of them), head sizes 64 and 128.
//
// The general kernel (attention_plain.cu) takes a block per token and head and reads every key and value once for each of them from
// L2.  Here a block takes 32 queries of a row and one head and walks the visible keys in tiles of 64 (boundaries at multiples of 64 of
// the key's position), which all its queries share in shared memory: 4 x 4 scores a thread, the softmax's maxima and sums by shuffles
// over the sixteen lanes of a query, 4 queries x hd / 16 columns of the output a thread.  Scores, softmax, P and all sums are float32
// (FFMA; P is not rounded).  A masked key's weight is exactly zero and its value is not looked at, so the order of a token's sums depends on its position and its first
// visible key alone.  Rows with fewer than `least` queries are left alone: attention_f32_short forms the same sums for a query at a time.
//
// The next tile's keys are on their way while P . V is formed, its values while the scores are.  What bounds it: the loads from shared
// memory (8 reads of 16 bytes for 64 products), with one or two blocks an SM.  16 heads of 128 over 8: 301 queries 48 us (the general kernel
// 443), 1,024 queries 209 (4,335); 8 queries behind 512 tokens 60 (82), behind 2,048 202 (292).
#include "common.cuh"
#include "mma_utils.cuh"
using namespace arle;

namespace {

constexpr int kQ = 32, kKeys = 64, kThreads = 128;

template <int HD>
__global__ void __launch_bounds__(kThreads) attention_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out,
                                                                 const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                                                                 const int* __restrict__ q_indptr, const int* __restrict__ kv_lens,
                                                                 const int* __restrict__ block_table, int bt_stride, int nq, int nkv,
                                                                 int page_size, float scale, int window, HeadTail<float> tail, int least) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int PITCH = HD + 4, PP = kKeys + 4, CH = HD / 4, NC = HD / 64;      // NC: groups of four output columns a thread holds
  __shared__ int place[2][kKeys];                          // a tile's keys: their rows of the caches, -1: none
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                                          // [32][PITCH], times the scale
  float* ks = qs + kQ * PITCH;                             // [64][PITCH]
  float* vs = ks + kKeys * PITCH;                          // [64][PITCH]
  float* ps = vs + kKeys * PITCH;                          // [32][PP]
  const int r = blockIdx.z, h = blockIdx.y;
  const int t0 = q_indptr[r], qlen = q_indptr[r + 1] - t0;
  const int m0 = (gridDim.x - 1 - blockIdx.x) * kQ;        // the last queries, which see the most keys, first
  if (qlen < least || m0 >= qlen) return;
  const int rows = min(kQ, qlen - m0), pos0 = kv_lens[r] - qlen + m0, kvh = h / (nq / nkv);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int* bt = block_table + (size_t)r * bt_stride;
  for (int idx = tid; idx < kQ * CH; idx += kThreads) {
    const int i = idx / CH, e = idx % CH * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < rows) x = *reinterpret_cast<const float4*>(q + (size_t)(t0 + m0 + i) * q_stride + (size_t)h * HD + e);
    *reinterpret_cast<float4*>(qs + i * PITCH + e) = make_float4(x.x * scale, x.y * scale, x.z * scale, x.w * scale);
  }
  float acc[4][NC * 4], m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < NC * 4; ++c) acc[i][c] = 0.f;
  }
  const int lo = first_visible_key(pos0, window, 0), last = pos0 + rows - 1;
  auto find = [&](int b, int j0) {
    const int j = j0 + tid;
    if (tid < kKeys) place[b][tid] = j >= lo && j <= last ? (bt[j / page_size] * nkv + kvh) * page_size + j % page_size : -1;
  };
  auto load = [&](float* dst, const float* cache, int b) {
#pragma unroll
    for (int it = 0; it < kKeys * CH / kThreads; ++it) {
      const int idx = tid + it * kThreads, jj = idx / CH, e = idx % CH * 4;
      const int row = place[b][jj];
      cp_async16(smem_u32(dst + jj * PITCH + e), cache + (row >= 0 ? (size_t)row * HD + e : 0), row >= 0 ? 16 : 0);
    }
    cp_commit();
  };
  const int j_first = lo / kKeys * kKeys;
  find(0, j_first);
  __syncthreads();
  load(ks, k_cache, 0);
  int b = 0;
  for (int j0 = j_first; j0 <= last; j0 += kKeys, b ^= 1) {
    load(vs, v_cache, b);
    if (j0 + kKeys <= last) find(b ^ 1, j0 + kKeys);
    cp_wait<1>();                                          // the keys are here
    __syncthreads();
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int e = 0; e < HD; e += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty * 4 + i) * PITCH + e);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * PITCH + e);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
          s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
          s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
          s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = pos0 + ty * 4 + i, first = window > 0 ? p - window + 1 : 0;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = j0 + tx + 16 * j;
        if (key > p || key < first) s[i][j] = -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[i], mx);
      const float base = mn == -INFINITY ? 0.f : mn;       // no key of the query yet
      const float f = expf(m[i] - base);                   // m = -inf: 0
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float pj = expf(s[i][j] - base);
        sum += pj;
        ps[(ty * 4 + i) * PP + tx + 16 * j] = pj;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[i] = fmaf(l[i], f, sum);
      m[i] = mn;
#pragma unroll
      for (int c = 0; c < NC * 4; ++c) acc[i][c] *= f;
    }
    __syncthreads();                                       // P is there and the keys are used up
    if (j0 + kKeys <= last) load(ks, k_cache, b ^ 1); else cp_commit();
    cp_wait<1>();                                          // the values are here; the next keys are on their way
    // A masked key's weight is zero, and zero times infinity is not: where some query does not see some key of the tile, the threads look
    // at the values they fetched, and a tile with an infinity or a NaN is added up key by key.
    const bool whole = j0 + kKeys - 1 <= pos0 && (window <= 0 || j0 >= last - window + 1);
    bool odd = false;
    if (!whole) {
#pragma unroll
      for (int it = 0; it < kKeys * CH / kThreads; ++it) {
        const int idx = tid + it * kThreads;
        const float4 x = *reinterpret_cast<const float4*>(vs + idx / CH * PITCH + idx % CH * 4);
        odd |= !(fabsf(x.x) < INFINITY && fabsf(x.y) < INFINITY && fabsf(x.z) < INFINITY && fabsf(x.w) < INFINITY);
      }
    }
    if (__syncthreads_or(odd)) {
#pragma unroll 1
      for (int j = 0; j < kKeys; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int p = pos0 + ty * 4 + i;
          if (j0 + j > p || (window > 0 && j0 + j < p - window + 1)) continue;
          const float w = ps[(ty * 4 + i) * PP + j];
#pragma unroll
          for (int c = 0; c < NC * 4; ++c) acc[i][c] = fmaf(w, vs[j * PITCH + (c >> 2) * 64 + tx * 4 + (c & 3)], acc[i][c]);
        }
    } else {
#pragma unroll 4
    for (int j = 0; j < kKeys; j += 4) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(ps + (ty * 4 + i) * PP + j);
#pragma unroll
      for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const float4 b = *reinterpret_cast<const float4*>(vs + (j + g) * PITCH + c * 64 + tx * 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float p = g == 0 ? a[i].x : g == 1 ? a[i].y : g == 2 ? a[i].z : a[i].w;
            acc[i][4 * c] = fmaf(p, b.x, acc[i][4 * c]);
            acc[i][4 * c + 1] = fmaf(p, b.y, acc[i][4 * c + 1]);
            acc[i][4 * c + 2] = fmaf(p, b.z, acc[i][4 * c + 2]);
            acc[i][4 * c + 3] = fmaf(p, b.w, acc[i][4 * c + 3]);
          }
        }
    }
    }
    __syncthreads();                                       // the values are used up
  }
  cp_wait<0>();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (ty * 4 + i >= rows) break;
    const int t = t0 + m0 + ty * 4 + i;
    float den = l[i], f = 1.0f;
    if (tail.sinks) {                                      // the sink's term may be larger than every score
      const float sink = tail.sinks[h], mm = fmaxf(m[i], sink);
      f = expf(m[i] - mm);
      den = fmaf(l[i], f, expf(sink - mm));
    }
    const float g = tail.gate_of(t, h);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      float4 o;
      o.x = acc[i][4 * c] * f / den * g;
      o.y = acc[i][4 * c + 1] * f / den * g;
      o.z = acc[i][4 * c + 2] * f / den * g;
      o.w = acc[i][4 * c + 3] * f / den * g;
      *reinterpret_cast<float4*>(out + ((size_t)t * nq + h) * HD + c * 64 + tx * 4) = o;
    }
  }
}

// Rows of fewer than `shorter_than` queries (0: every row): a block takes a query and a head and forms the very sums above, so a token has
// the same bits in a row of one query and in a row of many.  Half of the threads score 128 keys, a key each, while the other half adds up
// the values of the 128 before, a column each; one warp has the softmax of the two tiles in between.  Bound by the latency of those two
// chains of loads; the keys and values of a head are read once per query.  16 heads of 128 over 8, one query behind 512 tokens 27.7 us (the
// general kernel, which sums in another order, 79.8), behind 2,048 82.7 (283); 64 queries behind 2,048 each 367 (1,149).
constexpr int kStep = 2 * kKeys, kShortThreads = 2 * kStep;

template <int HD>
__global__ void __launch_bounds__(kShortThreads) attention_f32_short_kernel(
    const float* __restrict__ q, int q_stride, float* __restrict__ out, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
    const int* __restrict__ q_indptr, const int* __restrict__ positions, const int* __restrict__ row_of_token, const int* __restrict__ block_table,
    int bt_stride, int nq, int nkv, int page_size, float scale, int window, HeadTail<float> tail, int shorter_than) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) float qs[HD];
  __shared__ float ss[2][kStep], ps[2][kStep];             // scores and weights of a step
  __shared__ int place[2][kStep];                          // its keys' rows of the caches, -1: none
  __shared__ float factor[2][2], ending[2];                // what the sums shrink by in front of a tile; the maximum and the sum at the end
  const int t = blockIdx.x, h = blockIdx.y;
  const int row = row_of_token[t];
  if (shorter_than > 0 && q_indptr[row + 1] - q_indptr[row] >= shorter_than) return;
  const int pos = positions[t], kvh = h / (nq / nkv), lo = first_visible_key(pos, window, 0), j_first = lo / kKeys * kKeys;
  const int* bt = block_table + (size_t)row * bt_stride;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < HD; e += kShortThreads) qs[e] = q[(size_t)t * q_stride + (size_t)h * HD + e] * scale;
  __syncthreads();
  const int steps = (pos - j_first) / kStep + 1;
  auto score = [&](int st) {                               // the first half of the threads
    const int j = j_first + st * kStep + tid;
    int at = -1;
    float d = -INFINITY;
    if (j >= lo && j <= pos) {
      at = (bt[j / page_size] * nkv + kvh) * page_size + j % page_size;
      const float4* kp = reinterpret_cast<const float4*>(k_cache + (size_t)at * HD);
      d = 0.f;
#pragma unroll 16
      for (int e = 0; e < HD / 4; ++e) {
        const float4 b = kp[e], a = *reinterpret_cast<const float4*>(qs + 4 * e);
        d = fmaf(a.x, b.x, d);
        d = fmaf(a.y, b.y, d);
        d = fmaf(a.z, b.z, d);
        d = fmaf(a.w, b.w, d);
      }
    }
    place[st & 1][tid] = at;
    ss[st & 1][tid] = d;
  };
  float m = -INFINITY, l = 0.f;                            // the first warp's
  auto weigh = [&](int st) {                               // the first warp: sixteen lanes a tile
    const float* sc = ss[st & 1] + (lane >> 4) * kKeys + (lane & 15);
    float s[4], mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = sc[16 * j];
      mx = fmaxf(mx, s[j]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float mn0 = fmaxf(m, __shfl_sync(0xffffffffu, mx, 0)), mn1 = fmaxf(mn0, __shfl_sync(0xffffffffu, mx, 16));
    const float base0 = mn0 == -INFINITY ? 0.f : mn0, base1 = mn1 == -INFINITY ? 0.f : mn1;
    const float f0 = expf(m - base0), f1 = expf(mn0 - base1);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float pj = expf(s[j] - (lane < 16 ? base0 : base1));
      sum += pj;
      ps[st & 1][(lane >> 4) * kKeys + (lane & 15) + 16 * j] = pj;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float sum0 = __shfl_sync(0xffffffffu, sum, 0), sum1 = __shfl_sync(0xffffffffu, sum, 16);
    l = fmaf(l, f0, sum0);
    m = mn0;
    const bool second = j_first + st * kStep + kKeys <= pos;      // the step's second tile has keys
    if (second) {
      l = fmaf(l, f1, sum1);
      m = mn1;
    }
    if (lane == 0) {
      factor[st & 1][0] = f0;
      factor[st & 1][1] = second ? f1 : 1.f;
      ending[0] = m;
      ending[1] = l;
    }
  };
  float acc = 0.f;
  const int d = tid - kStep;
  if (tid < kStep) score(0);
  __syncthreads();
  if (tid < 32) weigh(0);
  __syncthreads();
  for (int st = 0; st < steps; ++st) {
    if (tid < kStep) {
      if (st + 1 < steps) score(st + 1);
    } else if (d < HD) {
      const int j0 = j_first + st * kStep;
#pragma unroll
      for (int tile = 0; tile < 2; ++tile) {
        const int from = max(lo - j0, tile * kKeys), to = min(pos - j0 + 1, (tile + 1) * kKeys);
        acc *= factor[st & 1][tile];
        int j = from;
        for (; j + 16 <= to; j += 16) {
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = v_cache[(size_t)place[st & 1][j + i] * HD + d];
#pragma unroll
          for (int i = 0; i < 16; ++i) acc = fmaf(ps[st & 1][j + i], v[i], acc);
        }
        for (; j < to; ++j) acc = fmaf(ps[st & 1][j], v_cache[(size_t)place[st & 1][j] * HD + d], acc);
      }
    }
    __syncthreads();
    if (st + 1 < steps && tid < 32) weigh(st + 1);
    __syncthreads();
  }
  if (d < 0 || d >= HD) return;
  float den = ending[1], f = 1.0f;
  if (tail.sinks) {
    const float sink = tail.sinks[h], mm = fmaxf(ending[0], sink);
    f = expf(ending[0] - mm);
    den = fmaf(ending[1], f, expf(sink - mm));
  }
  out[((size_t)t * nq + h) * HD + d] = acc * f / den * tail.gate_of(t, h);
}

template <int HD>
int launch(const float* q, int q_stride, float* out, const float* k_cache, const float* v_cache, const int* q_indptr, const int* kv_lens,
           const int* block_table, int bt_stride, int nq, int nkv, int page_size, float scale, int window, HeadTail<float> tail, int rows,
           int max_q_len, int least, cudaStream_t s) {
  constexpr size_t smem = ((size_t)(kQ + 2 * kKeys) * (HD + 4) + kQ * (kKeys + 4)) * sizeof(float);
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)attention_f32_kernel<HD>, smem);
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(attention_f32_kernel<HD>, dim3((max_q_len + kQ - 1) / kQ, nq, rows), dim3(kThreads), smem, s, 1, q, q_stride, out, k_cache, v_cache,
                q_indptr, kv_lens, block_table, bt_stride, nq, nkv, page_size, scale, window, tail, least);
  return launch_status();
}

}  // namespace

// q float32 [T, q_stride], caches float32 [pages, nkv, page_size, hd], out float32 [T, nq * hd]; rows of `least` queries and more.
ARLE_API int arle_attention_f32(const float* q, int q_stride, float* out, const float* k_cache, const float* v_cache, const int* q_indptr,
                                const int* kv_lens, const int* block_table, int bt_stride, int nq, int nkv, int hd, int page_size, float scale,
                                int window, const float* sinks, const float* gate, int gate_stride, int rows, int max_q_len, int least,
                                cudaStream_t s) {
  if (rows <= 0 || max_q_len <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || nq % nkv || page_size <= 0) return ARLE_E_BADARG;
  if ((hd != 64 && hd != 128) || q_stride % 4 || nq > 65535 || rows > 65535 ||
      (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15))
    return ARLE_E_UNSUPPORTED;
  const HeadTail<float> tail{sinks, gate, gate_stride};
  if (hd == 64)
    return launch<64>(q, q_stride, out, k_cache, v_cache, q_indptr, kv_lens, block_table, bt_stride, nq, nkv, page_size, scale, window, tail, rows,
                      max_q_len, least, s);
  return launch<128>(q, q_stride, out, k_cache, v_cache, q_indptr, kv_lens, block_table, bt_stride, nq, nkv, page_size, scale, window, tail, rows,
                     max_q_len, least, s);
}

// The rows of fewer than `shorter_than` queries (0: all rows), with the sums of arle_attention_f32 and the same arrays.
ARLE_API int arle_attention_f32_short(const float* q, int q_stride, float* out, const float* k_cache, const float* v_cache, const int* q_indptr,
                                      const int* positions, const int* row_of_token, const int* block_table, int bt_stride, int nq, int nkv, int hd,
                                      int page_size, float scale, int window, const float* sinks, const float* gate, int gate_stride,
                                      int num_tokens, int shorter_than, cudaStream_t s) {
  if (num_tokens <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || nq % nkv || page_size <= 0) return ARLE_E_BADARG;
  if ((hd != 64 && hd != 128) || nq > 65535 || (((uintptr_t)k_cache) & 15)) return ARLE_E_UNSUPPORTED;
  auto kernel = hd == 64 ? attention_f32_short_kernel<64> : attention_f32_short_kernel<128>;
  launch_kernel(kernel, dim3(num_tokens, nq), dim3(kShortThreads), 0, s, 1, q, q_stride, out, k_cache, v_cache, q_indptr, positions, row_of_token,
                block_table, bt_stride, nq, nkv, page_size, scale, window, HeadTail<float>{sinks, gate, gate_stride}, shorter_than);
  return launch_status();
}
