// The gated delta rule over long rows, in chunks of 64 tokens on the tensor cores:
//
//     S <- g_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t          (S: 128 x vdim, float32; k_t, q_t unit vectors)
//
// The scan in delta_rule.cu runs a token after the other.  With S_0 the memory before a chunk, D_ij = g_(j+1) .. g_i and D_i = g_1 .. g_i, the
// same u of a chunk solve a triangular system,
//     (I + A) u = beta (v - D_i S_0^T k_i),   A_ij = beta_i D_ij (k_i . k_j) for j < i,
//     o_i = D_i S_0^T q_i + sum_(j <= i) D_ij (q_i . k_j) u_j,        S_n = D_n S_0 + sum_j D_nj k_j u_j^T,
// and everything but S_0 is known before: delta_chunks forms T = (I + A)^-1 beta and P_ij = D_ij (q_i . k_j) of all chunks and heads side by
// side, and delta_tc goes through a row's chunks with small matrix products, S in registers (mma.sync accumulators).
//
// Precision: q and k are bfloat16 as the convolution leaves them, so their products are exact; their lengths enter as factors.  What is
// float32 (S_0, T, P, u) is cut into three bfloat16 numbers that together hold its 24 bits: three products with a bfloat16 matrix, the six
// largest with one another.  The decays come from sums of log2 g in float64, a decay of zero counts as 2^-300.  The triangular system is
// inverted in float32: tiles of 16 by forward substitution, the others from them.  Factors that meet in one number (decays, lengths, beta) are
// multiplied in float64 and rounded once: in float32 they cost a quarter of the digits that the scan keeps.  Against float64, with inputs as the
// layer makes them, rows of 64 to 2,048 tokens: outputs off by 0.98e-7 to 1.15e-7 of their norm (the scan: 1.07e-7 to 1.53e-7), memories by
// 0.90e-7 to 1.03e-7 (0.87e-7 to 1.73e-7).
//
// delta_tc: a block has a head and 16 G columns of v for a whole row, four warps 16 columns; the groups share the chunk's q and k and nothing
// else, so one group's barriers pass under another's products.  A warp forms the rows of a tile of 16 tokens and holds 32 rows of S.
// A row's own length decides whether it comes here; a token's sums have one order for its place in its row.
//
// What bounds it: a block's chain of chunks, some 4 us each with one group and 6 with two (four phases with a barrier between them, the tensor
// cores' legacy path about half of the time); delta_chunks takes some 20 us of a step of 2,000 tokens.  Rows of 819, 701 and 479 tokens, 32 heads
// of 128 x 128: 216 us (the scan 530); one row of 2,048 216 (650), with 8 heads 135 (510); 300 tokens, 8 heads 34 (79).  For keys of 128 alone, the size
// of the layers that run prompts; others are scanned.
#include "common.cuh"
#include "chunk_parts.cuh"
using namespace arle;

ARLE_API int arle_delta_scan(const void* q, const void* k, const void* v, int dtype, int q_stride, int k_stride, int v_stride, const float* beta,
                             const float* decay, float* state, long slot_stride, const int* q_indptr, const int* state_slots, float* out,
                             int num_tokens, int R, int H, int kq_heads, int dim, int vdim, float q_scale, float unit_eps, int longest,
                             cudaStream_t s);

namespace {

constexpr int kDim = 128, kQP = kDim + 8;
constexpr int kTiles = 10;                                 // tiles on and below the diagonal of a chunk
constexpr int kScalars = 256;                              // a chunk's numbers: [64] D_i / |k_i|, [64] q_scale D_i / |q_i|, [64] D_nj / |k_j|, D_n
constexpr size_t kChunkWords = 2 * kTiles * kTileWords + kScalars;   // of one head: T, P, numbers

struct ChunkSmem {
  __nv_bfloat16 q[kC][kQP], k[kC][kQP];
  float A[kC][kC + 4], T[kC][kC + 4];
  float W[3][16][17];                                      // products on their way into a tile of T
  double cum[kC];
  double iq[kC], ik[kC];                                   // q_scale / |q|, 1 / |k|
  float beta[kC];
};

// 256 threads a chunk and head.
__global__ void __launch_bounds__(256, 3) delta_chunks_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, long q_stride,
                                                           long k_stride, const float* __restrict__ beta, const float* __restrict__ decay,
                                                           const int* __restrict__ q_indptr, int rows, int longest, int H, int kq_heads,
                                                           float q_scale, float unit_eps, uint32_t* __restrict__ chunks) {
  pdl_launch_dependents();
  pdl_wait();
  int r, chunk;
  if (!chunk_of(blockIdx.x, q_indptr, rows, longest, r, chunk)) return;
  extern __shared__ __align__(16) unsigned char raw[];
  ChunkSmem& sm = *reinterpret_cast<ChunkSmem*>(raw);
  const int h = blockIdx.y, g = h / (H / kq_heads), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = q_indptr[r] + chunk * kC, n = min(kC, q_indptr[r + 1] - t0);
  uint32_t* to = chunks + ((size_t)blockIdx.x * H + h) * kChunkWords;
#pragma unroll
  for (int it = 0; it < kC * (kDim / 8) / 256; ++it) {
    const int idx = tid + it * 256, j = idx / (kDim / 8), e = idx % (kDim / 8) * 8;
    const bool ok = j < n;
    cp_async16(smem_u32(&sm.q[j][e]), ok ? q + (size_t)(t0 + j) * q_stride + (size_t)g * kDim + e : q, ok ? 16 : 0);
    cp_async16(smem_u32(&sm.k[j][e]), ok ? k + (size_t)(t0 + j) * k_stride + (size_t)g * kDim + e : k, ok ? 16 : 0);
  }
  cp_commit();
  if (warp == 0) {
    double x[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * lane + i;
      const float a = j < n ? decay[(size_t)(t0 + j) * H + h] : 1.f;
      sm.beta[j] = j < n ? beta[(size_t)(t0 + j) * H + h] : 0.f;
      x[i] = a == a ? (double)fmaxf(log2f(a), -300.f) : (double)a;
    }
    double sum = x[0] + x[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    double first = __shfl_up_sync(0xffffffffu, sum, 1);
    first = (lane ? first : 0.0) + x[0];
    sm.cum[2 * lane] = first;
    sm.cum[2 * lane + 1] = sum;
  }
  cp_wait<0>();
  __syncthreads();
  {                                                        // lengths: four threads a token
    const int j = tid >> 2, part = tid & 3;
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int e = 0; e < 32; e += 8) {
      float a[8], b[8];
      load_vec<__nv_bfloat16, 8>(&sm.q[j][part * 32 + e], a);
      load_vec<__nv_bfloat16, 8>(&sm.k[j][part * 32 + e], b);
#pragma unroll
      for (int i = 0; i < 8; ++i) sq = fmaf(a[i], a[i], sq), sk = fmaf(b[i], b[i], sk);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      sk += __shfl_xor_sync(0xffffffffu, sk, o);
    }
    if (part == 0) {                                       // behind the row's end zeros: with a unit_eps of zero the factors would be infinities
      sm.iq[j] = j < n ? q_scale / sqrt((double)sq + unit_eps) : 0.0;
      sm.ik[j] = j < n ? 1.0 / sqrt((double)sk + unit_eps) : 0.0;
    }
  }
  __syncthreads();
  {                                                        // k . k (four warps) and q . k
    const bool is_q = warp >= 4;
    const int rt = is_q ? 7 - warp : warp;                 // a scheduler's two warps have five tiles together
    const __nv_bfloat16* a = is_q ? &sm.q[0][0] : &sm.k[0][0];
    float sc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
#pragma unroll 4
    for (int kk = 0; kk < kDim / 16; ++kk) {
      uint32_t qa[4];
      ldsm_x4(smem_u32(a + (rt * 16 + (lane & 15)) * kQP + kk * 16 + (lane >> 4) * 8), qa[0], qa[1], qa[2], qa[3]);
#pragma unroll
      for (int jt = 0; jt < 4; ++jt) {
        if (jt > rt) break;
        uint32_t b0, b1, b2, b3;
        ldsm_x4(smem_u32(&sm.k[jt * 16 + (lane >> 4) * 8 + (lane & 7)][kk * 16 + ((lane >> 3) & 1) * 8]), b0, b1, b2, b3);
        mma_add(sc[2 * jt], qa, b0, b1);
        mma_add(sc[2 * jt + 1], qa, b2, b3);
      }
    }
    const int i0 = rt * 16 + (lane >> 2);
    const double cu[2] = {sm.cum[i0], sm.cum[i0 + 8]};
    const double fr[2] = {is_q ? sm.iq[i0] : sm.beta[i0] * sm.ik[i0], is_q ? sm.iq[i0 + 8] : sm.beta[i0 + 8] * sm.ik[i0 + 8]};
#pragma unroll
    for (int jt = 0; jt < 4; ++jt) {
      if (jt > rt) break;
      float w[8];
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int j = jt * 16 + hh * 8 + 2 * (lane & 3) + (i & 1), row = i0 + (i >> 1) * 8;
          const bool seen = is_q ? j <= row : j < row;
          w[hh * 4 + i] = seen ? (float)(sc[2 * jt + hh][i] * (fr[i >> 1] * (sm.ik[j] * exp2(cu[i >> 1] - sm.cum[j])))) : 0.f;
        }
      if (is_q) {
        split_tile(w, to + (kTiles + rt * (rt + 1) / 2 + jt) * kTileWords, lane);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) sm.A[i0 + ((i >> 1) & 1) * 8][jt * 16 + (i >> 2) * 8 + 2 * (lane & 3) + (i & 1)] = w[i];
      }
    }
  }
  if (tid < kC) {
    const double c = sm.cum[tid];
    const double d = exp2(c);
    float* s = reinterpret_cast<float*>(to + 2 * kTiles * kTileWords);
    s[tid] = (float)(d * sm.ik[tid]);
    s[kC + tid] = (float)(d * sm.iq[tid]);
    s[2 * kC + tid] = (float)(exp2(sm.cum[kC - 1] - c) * sm.ik[tid]);
    if (tid == kC - 1) s[3 * kC] = (float)d;
  }
  __syncthreads();
  if (tid < kC) {                                          // the tiles on the diagonal: a thread has a column
    const int b = tid & ~15, c = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s = 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) s = fmaf(sm.A[b + i][b + m], x[m], s);
      x[i] = i < c ? 0.f : (i == c ? 1.f : -s);
      sm.T[b + i][b + c] = x[i];
    }
  }
  const int er = tid >> 4, ec = tid & 15;
#pragma unroll
  for (int d = 1; d < 4; ++d) {                            // the tiles d below it: T_ij = -T_ii sum_(j <= k < i) A_ik T_kj
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4 - d; ++j) {
      float s = 0.f;
#pragma unroll
      for (int kt = j; kt < j + d; ++kt)
#pragma unroll
        for (int m = 0; m < 16; ++m) s = fmaf(sm.A[(j + d) * 16 + er][kt * 16 + m], sm.T[kt * 16 + m][j * 16 + ec], s);
      sm.W[j][er][ec] = s;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4 - d; ++j) {
      float s = 0.f;
#pragma unroll
      for (int m = 0; m < 16; ++m)
        if (m <= er) s = fmaf(sm.T[(j + d) * 16 + er][(j + d) * 16 + m], sm.W[j][m][ec], s);
      sm.T[(j + d) * 16 + er][j * 16 + ec] = -s;
    }
  }
  __syncthreads();
  for (int tile = warp; tile < kTiles; tile += 8) {
    const int rt = tile >= 6 ? 3 : tile >= 3 ? 2 : tile >= 1 ? 1 : 0, jt = tile - rt * (rt + 1) / 2;
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = rt * 16 + (lane >> 2) + ((i >> 1) & 1) * 8, j = jt * 16 + (i >> 2) * 8 + 2 * (lane & 3) + (i & 1);
      w[i] = j <= row ? sm.T[row][j] * sm.beta[j] : 0.f;
    }
    split_tile(w, to + tile * kTileWords, lane);
  }
}

template <int G>
struct Layout {
  static constexpr int VT = 16 * G, VP = VT + 8;           // pitches: eight rows of a matrix load fall on different banks
  static constexpr size_t QK = (size_t)kC * kQP, V = (size_t)kC * VP;
  static constexpr size_t BUF = 2 * QK + V + 2 * kScalars; // a chunk's q, k, v and numbers, in bfloat16's
  static constexpr size_t SS = (size_t)kDim * VP;          // one of the three parts
  static constexpr size_t SMEM = (2 * BUF + 3 * SS + 9 * V) * 2;
};

// acc (+ rest) += the tiles of 16 x 16 (three parts, in memory) of a row of tiles times the rows of x (three parts [part][64][VP] in shared
// memory, the warp's 16 columns); tiles 0 .. last.
template <int VP>
__device__ __forceinline__ void tiles_times(const uint4 (&w)[4][3], int last, uint32_t x, size_t part, int lane, float (&acc)[2][4], float (&rest)[2][4]) {
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    if (kt > last) break;
    uint32_t b[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
      ldsm_x4_t(x + (uint32_t)(i * part + (kt * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8) * 2, b[i][0], b[i][1], b[i][2], b[i][3]);
#pragma unroll
    for (int s = 2; s >= 0; --s)                           // small products first
#pragma unroll
      for (int i = 0; i <= s; ++i) {
        const uint32_t a[4] = {w[kt][i].x, w[kt][i].y, w[kt][i].z, w[kt][i].w};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          if (s) mma_bf16(rest[nt], a, b[s - i][2 * nt], b[s - i][2 * nt + 1]);
          else mma_add(acc[nt], a, b[0][2 * nt], b[0][2 * nt + 1]);
        }
      }
  }
}

// The same for a tile on the diagonal, one product at a time and only those that a row sees: a weight of zero does not silence an infinity.
template <int VP>
__device__ __forceinline__ void seen_alone(const uint32_t* tile, const __nv_bfloat16* x, size_t part, int lane, float (&acc)[2][4]) {
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int nt = v >> 2, i = v & 3, row = (lane >> 2) + (i >> 1) * 8, c = nt * 8 + 2 * (lane & 3) + (i & 1);
    float s = 0.f;
#pragma unroll 1
    for (int j = 0; j <= row; ++j) {
      const int at = ((row & 7) * 4 + ((j & 7) >> 1)) * 4 + (row >> 3) + 2 * (j >> 3);
      float w = 0.f, y = 0.f;
      for (int p = 2; p >= 0; --p) {
        const uint32_t two = tile[p * 128 + at];
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&two);
        w += j & 1 ? __high2float(b) : __low2float(b);
        y += __bfloat162float(x[p * part + j * VP + c]);
      }
      s = fmaf(w, y, s);
    }
    acc[nt][i] += s;
  }
}

template <int G>
__global__ void __launch_bounds__(128 * G, 1) delta_tc_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                              const __nv_bfloat16* __restrict__ v, long q_stride, long k_stride, long v_stride,
                                                              const uint32_t* __restrict__ chunks, float* __restrict__ state, long slot_stride,
                                                              const int* __restrict__ q_indptr, const int* __restrict__ state_slots,
                                                              float* __restrict__ out, int H, int kq_heads, int vdim, int longest) {
  pdl_launch_dependents();
  pdl_wait();
  typedef Layout<G> L;
  constexpr int VP = L::VP, VT = L::VT, NTH = 128 * G;
  extern __shared__ __align__(16) unsigned char raw[];
  __nv_bfloat16* bufs = reinterpret_cast<__nv_bfloat16*>(raw);
  const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * VT;
  const int beg = q_indptr[r], end = q_indptr[r + 1];
  if (end - beg <= longest) return;
  const int g = h / (H / kq_heads), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = warp >> 2, wq = warp & 3;
  const int gid = lane >> 2, t4 = lane & 3;
  const int rt = grp & 1 ? 3 - wq : wq;                    // a scheduler's warps take early and late rows
  __nv_bfloat16* ss = bufs + 2 * L::BUF + grp * 16;        // [3][128][VP], the group's columns
  __nv_bfloat16* rs = ss + 3 * L::SS;                      // [3][64][VP] v - D S_0^T k
  __nv_bfloat16* us = rs + 3 * L::V;                       // [3][64][VP] u
  __nv_bfloat16* ws = us + 3 * L::V;                       // [3][64][VP] D_nj u_j / |k_j|
  auto group_sync = [&]() { asm volatile("bar.sync %0, 128;\n" ::"r"(grp + 1) : "memory"); };
  int before = 0;                                          // chunks of the rows in front
  for (int r0 = lane; r0 < r; r0 += 32) before += row_chunks(q_indptr[r0 + 1] - q_indptr[r0], longest);
  before = __reduce_add_sync(0xffffffffu, before);
  const int um = wq * 32;
  float* sp = state + (size_t)state_slots[r] * slot_stride + (size_t)h * vdim * kDim;
  float S[2][2][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = um + m * 16 + gid + (i >> 1) * 8, c = c0 + grp * 16 + nn * 8 + 2 * t4 + (i & 1);
        S[m][nn][i] = c < vdim ? sp[(size_t)c * kDim + d] : 0.f;
      }
  auto of_chunk = [&](int chunk) { return chunks + ((size_t)(before + chunk) * H + h) * kChunkWords; };
  auto load = [&](int chunk, __nv_bfloat16* buf) {
    const int t0 = beg + chunk * kC, n = min(kC, end - t0);
    constexpr int CH = kDim / 8;
#pragma unroll
    for (int it = 0; it < kC * CH / NTH; ++it) {
      const int idx = tid + it * NTH, j = idx / CH, e = idx % CH * 8;
      const bool ok = j < n;
      cp_async16(smem_u32(buf + j * kQP + e), ok ? q + (size_t)(t0 + j) * q_stride + (size_t)g * kDim + e : q, ok ? 16 : 0);
      cp_async16(smem_u32(buf + L::QK + j * kQP + e), ok ? k + (size_t)(t0 + j) * k_stride + (size_t)g * kDim + e : k, ok ? 16 : 0);
    }
    for (int idx = tid; idx < kC * (VT / 8); idx += NTH) {
      const int j = idx / (VT / 8), c = idx % (VT / 8) * 8;
      const bool ok = j < n && c0 + c < vdim;
      cp_async16(smem_u32(buf + 2 * L::QK + j * VP + c), ok ? v + (size_t)(t0 + j) * v_stride + (size_t)h * vdim + c0 + c : v, ok ? 16 : 0);
    }
    if (tid < kScalars / 4) cp_async16(smem_u32(buf + 2 * L::QK + L::V + tid * 8), of_chunk(chunk) + 2 * kTiles * kTileWords + tid * 4, 16);
    cp_commit();
  };
  auto fetch_tiles = [&](const uint32_t* from, uint4 (&w)[4][3]) {      // the warp's row of tiles
#pragma unroll
    for (int kt = 0; kt < 4; ++kt)
      if (kt <= rt)
#pragma unroll
        for (int i = 0; i < 3; ++i)
          w[kt][i] = __ldg(reinterpret_cast<const uint4*>(from + (rt * (rt + 1) / 2 + kt) * kTileWords + (i * 32 + lane) * 4));
  };
  const int nchunks = (end - beg + kC - 1) / kC;
  load(0, bufs);
  for (int ch = 0; ch < nchunks; ++ch) {
    const int t0 = beg + ch * kC, n = min(kC, end - t0);
    const __nv_bfloat16* qs = bufs + (ch & 1) * L::BUF;
    const __nv_bfloat16* ks = qs + L::QK;
    const __nv_bfloat16* vs = ks + L::QK + grp * 16;
    const float* num = reinterpret_cast<const float*>(qs + 2 * L::QK + L::V);
    cp_wait<0>();
    __syncthreads();                                       // the chunk is here, and the one before is used up
    if (ch + 1 < nchunks) load(ch + 1, bufs + ((ch + 1) & 1) * L::BUF);
    const uint32_t* tiles = of_chunk(ch);
    uint4 w[4][3];
    fetch_tiles(tiles, w);
#pragma unroll
    for (int m = 0; m < 2; ++m)                            // S_0 in three parts
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t s3[3];
          split3(S[m][nn][2 * half], S[m][nn][2 * half + 1], s3[0], s3[1], s3[2]);
          const size_t at = (size_t)(um + m * 16 + gid + half * 8) * VP + nn * 8 + 2 * t4;
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(ss + i * L::SS + at) = s3[i];
        }
    group_sync();
    const int i0 = rt * 16 + gid;
    // three parts of the warp's 16 x 16 numbers x
    auto store3 = [&](__nv_bfloat16* to, const float (&x)[2][4]) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t s3[3];
          split3(x[nt][2 * half], x[nt][2 * half + 1], s3[0], s3[1], s3[2]);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(to + i * L::V + (size_t)(i0 + half * 8) * VP + nt * 8 + 2 * t4) = s3[i];
        }
    };
    float o[2][4];
    {
      float kS[2][4], k_rest[2][4], q_rest[2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[0][i] = o[1][i] = kS[0][i] = kS[1][i] = 0.f;
        k_rest[0][i] = k_rest[1][i] = q_rest[0][i] = q_rest[1][i] = 0.f;
      }
#pragma unroll 4
      for (int kk = 0; kk < kDim / 16; ++kk) {
        uint32_t qa[4], ka[4];
        const uint32_t at = (uint32_t)((rt * 16 + (lane & 15)) * kQP + kk * 16 + (lane >> 4) * 8) * 2;
        ldsm_x4(smem_u32(qs) + at, qa[0], qa[1], qa[2], qa[3]);
        ldsm_x4(smem_u32(ks) + at, ka[0], ka[1], ka[2], ka[3]);
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(smem_u32(ss + i * L::SS + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8), b0, b1, b2, b3);
          if (i > 0) {
            mma_bf16(k_rest[0], ka, b0, b1);
            mma_bf16(k_rest[1], ka, b2, b3);
            mma_bf16(q_rest[0], qa, b0, b1);
            mma_bf16(q_rest[1], qa, b2, b3);
          } else {
            mma_add(kS[0], ka, b0, b1);
            mma_add(kS[1], ka, b2, b3);
            mma_add(o[0], qa, b0, b1);
            mma_add(o[1], qa, b2, b3);
          }
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int row = i0 + half * 8;
          const float e = num[row], f = num[kC + row];
          const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(vs + row * VP + nt * 8 + 2 * t4);
          kS[nt][2 * half] = __low2float(x) - e * (kS[nt][2 * half] + k_rest[nt][2 * half]);
          kS[nt][2 * half + 1] = __high2float(x) - e * (kS[nt][2 * half + 1] + k_rest[nt][2 * half + 1]);
          o[nt][2 * half] = (o[nt][2 * half] + q_rest[nt][2 * half]) * f;
          o[nt][2 * half + 1] = (o[nt][2 * half + 1] + q_rest[nt][2 * half + 1]) * f;
        }
      store3(rs, kS);
    }
    group_sync();                                          // v - D S_0^T k is there; S_0's parts are used up
    {
      float u[2][4], rest[2][4];
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int i = 0; i < 4; ++i) u[0][i] = u[1][i] = rest[0][i] = rest[1][i] = 0.f;
        tiles_times<VP>(w, rt - pass, smem_u32(rs), L::V, lane, u, rest);
        float odd = 0.f;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            u[nt][i] += rest[nt][i];
            odd = fmaf(u[nt][i], 0.f, odd);
          }
        if (pass) seen_alone<VP>(tiles + (rt * (rt + 1) / 2 + rt) * kTileWords, rs + rt * 16 * VP, L::V, lane, u);
        else if (!__any_sync(0xffffffffu, odd != odd)) break;
      }
      fetch_tiles(tiles + kTiles * kTileWords, w);
      store3(us, u);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) u[nt][i] *= num[2 * kC + i0 + (i >> 1) * 8];
      store3(ws, u);
    }
    group_sync();                                          // u is there
    {
      float sum[2][4], rest[2][4];
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[nt][i] = rest[nt][i] = 0.f;
        tiles_times<VP>(w, rt - pass, smem_u32(us), L::V, lane, sum, rest);
        float odd = 0.f;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            sum[nt][i] = o[nt][i] + (sum[nt][i] + rest[nt][i]);
            odd = fmaf(sum[nt][i], 0.f, odd);
          }
        if (pass) seen_alone<VP>(tiles + (kTiles + rt * (rt + 1) / 2 + rt) * kTileWords, us + rt * 16 * VP, L::V, lane, sum);
        else if (!__any_sync(0xffffffffu, odd != odd)) break;
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int i = i0 + half * 8, c = c0 + grp * 16 + nt * 8 + 2 * t4;
          if (i < n && c < vdim)                           // vdim is even: both or none
            *reinterpret_cast<float2*>(out + ((size_t)(t0 + i) * H + h) * vdim + c) = make_float2(sum[nt][2 * half], sum[nt][2 * half + 1]);
        }
    }
    const float whole = num[3 * kC];
    float more[2][2][4], rest[2][2][4];                    // the chunk's own sums, so that S is rounded once a chunk
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) more[m][nn][i] = rest[m][nn][i] = 0.f;
#pragma unroll
    for (int kk = 0; kk < kC / 16; ++kk) {
      uint32_t ka[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
        ldsm_x4_t(smem_u32(ks + (kk * 16 + (lane >> 4) * 8 + (lane & 7)) * kQP + um + m * 16 + ((lane >> 3) & 1) * 8), ka[m][0], ka[m][1], ka[m][2],
                  ka[m][3]);
#pragma unroll
      for (int i = 2; i >= 0; --i) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4_t(smem_u32(ws + i * L::V + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8), b0, b1, b2, b3);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          if (i > 0) {
            mma_bf16(rest[m][0], ka[m], b0, b1);
            mma_bf16(rest[m][1], ka[m], b2, b3);
          } else {
            mma_add(more[m][0], ka[m], b0, b1);
            mma_add(more[m][1], ka[m], b2, b3);
          }
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[m][nn][i] = fmaf(S[m][nn][i], whole, more[m][nn][i] + rest[m][nn][i]);
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = um + m * 16 + gid + (i >> 1) * 8, c = c0 + grp * 16 + nn * 8 + 2 * t4 + (i & 1);
        if (c < vdim) sp[(size_t)c * kDim + d] = S[m][nn][i];
      }
}

template <int G>
int launch(const void* q, const void* k, const void* v, long q_stride, long k_stride, long v_stride, const uint32_t* chunks, float* state,
           long slot_stride, const int* q_indptr, const int* state_slots, float* out, int R, int H, int kq_heads, int vdim, int longest,
           cudaStream_t s) {
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)delta_tc_kernel<G>, Layout<G>::SMEM);
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(delta_tc_kernel<G>, dim3((vdim + 16 * G - 1) / (16 * G), H, R), dim3(128 * G), Layout<G>::SMEM, s, 1, (const __nv_bfloat16*)q,
                (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, q_stride, k_stride, v_stride, chunks, state, slot_stride, q_indptr, state_slots,
                out, H, kq_heads, vdim, longest);
  return launch_status();
}

int most_chunks(int num_tokens, int R, int longest) {      // of rows of more than `longest` tokens
  const int rows = num_tokens / (longest + 1);
  return num_tokens / kC + (rows < R ? rows : R);
}

}  // namespace

// Rows of more than `longest` tokens; the others go to arle_delta_scan.  long_rows, long_tokens: how many such rows there are and their tokens
// together, where the host knows them (long_rows below zero: it does not); what is launched goes by the rows that run there.  q, k bfloat16
// [T, kq_heads*128], v bfloat16 [T, H*vdim] (row strides multiples of 8, 16-byte aligned), beta, decay float32 [T, H]; state: float32, a slot
// every slot_stride numbers, [H][vdim][128] at its start; out float32 [T, H, vdim], 8-byte aligned; vdim a multiple of 8; scratch: 7,936 float32
// numbers for each head and chunk, 16-byte aligned, for as many chunks as such rows can have (num_tokens / 64 + min(R, num_tokens / (longest +
// 1)), whole numbers).
ARLE_API int arle_delta_tc(const void* q, const void* k, const void* v, int q_stride, int k_stride, int v_stride, const float* beta,
                           const float* decay, float* state, long slot_stride, const int* q_indptr, const int* state_slots, float* out,
                           float* scratch, int num_tokens, int R, int H, int kq_heads, int vdim, float q_scale, float unit_eps, int longest,
                           int long_rows, int long_tokens, cudaStream_t s) {
  if (R <= 0 || num_tokens <= 0) return 0;
  if (H <= 0 || kq_heads <= 0 || H % kq_heads || vdim <= 0 || longest < 0 || !scratch) return ARLE_E_BADARG;
  if (vdim % 8 || q_stride % 8 || k_stride % 8 || v_stride % 8 || H > 65535 || R > 65535 ||
      (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch) & 15) || ((uintptr_t)out & 7))
    return ARLE_E_UNSUPPORTED;
  const bool known = long_rows >= 0;
  const int slots = known && long_rows == 0 ? 0 : most_chunks(num_tokens, R, longest);
  if (slots == 0 || !known || long_rows < R) {
    // the scan's form goes by the tokens of the rows that it runs (63 of one token beside one of 128, 32 heads: 125 us, 159 in the form for prompts)
    const int short_tokens = known ? num_tokens - long_tokens + long_rows : num_tokens;
    const int e = arle_delta_scan(q, k, v, 1, q_stride, k_stride, v_stride, beta, decay, state, slot_stride, q_indptr, state_slots, out,
                                  short_tokens, R, H, kq_heads, kDim, vdim, q_scale, unit_eps, longest, s);
    if (e || slots == 0) return e;
  }
  uint32_t* chunks = reinterpret_cast<uint32_t*>(scratch);
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)delta_chunks_kernel, sizeof(ChunkSmem));
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(delta_chunks_kernel, dim3(slots, H), dim3(256), sizeof(ChunkSmem), s, 1, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k,
                (long)q_stride, (long)k_stride, beta, decay, q_indptr, R, longest, H, kq_heads, q_scale, unit_eps, chunks);
  // Groups of 16 columns by themselves while every block that has a row to run finds an SM (8 heads of 128, one row of 2,048: 134 us, 171 with two
  // to a block, 265 with four), two to a block beyond (32 heads: 309, 208 and 299; rows of 819, 701 and 479 tokens 298, 210 and 202).  The same bits.
  // Rows that are scanned don't count (8 heads, one row of 2,048 beside 8 decoded tokens: 143 us, 177 when they did).
  const int most = num_tokens / (longest + 1), rows = known ? long_rows : most < R ? most : R;
  if ((long)((vdim + 15) / 16) * H * rows <= 148)
    return launch<1>(q, k, v, q_stride, k_stride, v_stride, chunks, state, slot_stride, q_indptr, state_slots, out, R, H, kq_heads, vdim, longest, s);
  return launch<2>(q, k, v, q_stride, k_stride, v_stride, chunks, state, slot_stride, q_indptr, state_slots, out, R, H, kq_heads, vdim, longest, s);
}
