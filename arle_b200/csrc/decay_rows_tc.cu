// The recurrence of decay_tc.cu in two launches, for memories of 128 x vdim without a column of ones: what does not need the memory is formed for
// all chunks and heads side by side (decay_tiles: the weighted scores D_ij b_j (q_i . k_j), cut into three bfloat16 numbers, and the chunk's
// decays), and the chain of a row's chunks (decay_rows_tc) is left with S_0^T q, the weighted scores times v and the update.  Every sum has the
// order it has there: the same bits, so that a step may take either.  (Beside an infinity or a NaN in v, whose tile is added up value by value, the
// columns of the same warp differ in the last bits: 16 here, up to 32 there.)
//
// decay_rows_tc: a block has a head and 16 G columns of v for a whole row, four warps 16 columns; the groups share the chunk's q and k and
// nothing else.  A warp forms the rows of a tile of 16 tokens and holds 32 rows of S.  A chunk has one barrier for the block and one for the group.
// What bounds it: a block's chain of chunks, some 5 us each with four groups (the one launch: 9) and 2.2 with one; decay_tiles takes some 15 us of
// 2,048 tokens, 35 with 128 heads.  One row of 2,048 tokens: 128 heads of 128 x 64 in 8 groups 197 us (decay_tc 294), 32 heads 81 (215); three rows of
// 600 to 748 207 (300) and 78 (104); 300 tokens, 32 heads 26.5 (35.6).  For heads of 128 alone, the size of the Mamba-2 layers that run prompts; other
// sizes and a column of ones stay with the one launch.
#include "common.cuh"
#include "chunk_parts.cuh"
using namespace arle;

namespace {

constexpr int kDim = 128, kQP = kDim + 8, kTiles = 10, kNumbers = 256;      // numbers: [64] q_scale D_i, [64] D_nj b_j, D_n
constexpr size_t kChunkWords = kTiles * kTileWords + kNumbers;              // of one head
constexpr int kMostHeads = 4;                                               // heads of one q and k that a block of decay_tiles takes

struct TilesSmem {
  __nv_bfloat16 q[kC][kQP], k[kC][kQP];
  double cum[kMostHeads][kC];                                               // log2 of a_1 .. a_i
  float b[kMostHeads][kC];
};

__global__ void __launch_bounds__(128) decay_tiles_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, long q_stride,
                                                          long k_stride, const float* __restrict__ a, const float* __restrict__ b,
                                                          const int* __restrict__ q_indptr, int rows, int longest, int H, int kq_heads, int heads,
                                                          float q_scale, uint32_t* __restrict__ chunks) {
  pdl_launch_dependents();
  pdl_wait();
  int r, chunk;
  if (!chunk_of(blockIdx.x, q_indptr, rows, longest, r, chunk)) return;
  extern __shared__ __align__(16) unsigned char raw[];
  TilesSmem& sm = *reinterpret_cast<TilesSmem*>(raw);
  const int h0 = blockIdx.y * heads, g = h0 / (H / kq_heads), tid = threadIdx.x, lane = tid & 31, rt = tid >> 5;
  const int t0 = q_indptr[r] + chunk * kC, n = min(kC, q_indptr[r + 1] - t0);
  uint32_t* to = chunks + ((size_t)blockIdx.x * H + h0) * kChunkWords;
#pragma unroll
  for (int it = 0; it < kC * (kDim / 8) / 128; ++it) {
    const int idx = tid + it * 128, j = idx / (kDim / 8), e = idx % (kDim / 8) * 8;
    const bool ok = j < n;
    cp_async16(smem_u32(&sm.q[j][e]), ok ? q + (size_t)(t0 + j) * q_stride + (size_t)g * kDim + e : q, ok ? 16 : 0);
    cp_async16(smem_u32(&sm.k[j][e]), ok ? k + (size_t)(t0 + j) * k_stride + (size_t)g * kDim + e : k, ok ? 16 : 0);
  }
  cp_commit();
  if (rt < heads) {                                                         // a warp has a head's decays, two tokens a lane
    float la[2], lb[2];
    double x[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * lane + i;
      la[i] = j < n ? a[(size_t)(t0 + j) * H + h0 + rt] : 1.f;
      lb[i] = j < n ? b[(size_t)(t0 + j) * H + h0 + rt] : 0.f;
      x[i] = la[i] == la[i] ? (double)fmaxf(log2f(la[i]), -300.f) : (double)la[i];
    }
    double sum = x[0] + x[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const double total = __shfl_sync(0xffffffffu, sum, 31);
    double first = __shfl_up_sync(0xffffffffu, sum, 1);
    first = (lane ? first : 0.0) + x[0];
    const double c[2] = {first, sum};
    float* num = reinterpret_cast<float*>(to + rt * kChunkWords + kTiles * kTileWords);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * lane + i;
      sm.cum[rt][j] = c[i];
      sm.b[rt][j] = lb[i];
      num[j] = q_scale * exp2f((float)c[i]);
      num[kC + j] = lb[i] * exp2f((float)(total - c[i]));
    }
    if (lane == 31) num[2 * kC] = exp2f((float)sum);
  }
  cp_wait<0>();
  __syncthreads();
  float sc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
#pragma unroll 4
  for (int kk = 0; kk < kDim / 16; ++kk) {
    uint32_t qa[4];
    ldsm_x4(smem_u32(&sm.q[rt * 16 + (lane & 15)][kk * 16 + (lane >> 4) * 8]), qa[0], qa[1], qa[2], qa[3]);
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
#pragma unroll 1
  for (int hh = 0; hh < heads; ++hh) {
    const double cu[2] = {sm.cum[hh][i0], sm.cum[hh][i0 + 8]};
#pragma unroll
    for (int jt = 0; jt < 4; ++jt) {
      if (jt > rt) break;
      float w[8];
#pragma unroll
      for (int half = 0; half < 2; ++half) {                                // the tile's two groups of 8 keys
        const int j = jt * 16 + half * 8 + 2 * (lane & 3);
        const double cj[2] = {sm.cum[hh][j], sm.cum[hh][j + 1]};
        const float fb[2] = {sm.b[hh][j] * q_scale, sm.b[hh][j + 1] * q_scale};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = i0 + (i >> 1) * 8;
          w[half * 4 + i] = j + (i & 1) <= row ? sc[2 * jt + half][i] * (fb[i & 1] * exp2f((float)(cu[i >> 1] - cj[i & 1]))) : 0.f;
        }
      }
      split_tile(w, to + hh * kChunkWords + (rt * (rt + 1) / 2 + jt) * kTileWords, lane);
    }
  }
}

template <int G>
struct Layout {
  static constexpr int VT = 16 * G, VP = VT + 8;           // pitches: eight rows of a matrix load fall on different banks
  static constexpr size_t QK = (size_t)kC * kQP, V = (size_t)kC * VP;
  static constexpr size_t BUF = 2 * QK + V + 2 * kNumbers; // a chunk's q, k, v and numbers, in bfloat16's
  static constexpr size_t SS = (size_t)kDim * VP;          // one of the three parts
  static constexpr size_t SMEM = (2 * BUF + 3 * SS + 3 * V) * 2;
};

template <int G>
__global__ void __launch_bounds__(128 * G, 1) decay_rows_tc_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                                   const __nv_bfloat16* __restrict__ v, long q_stride, long k_stride, long v_stride,
                                                                   const uint32_t* __restrict__ chunks, float* __restrict__ state,
                                                                   long slot_stride, const int* __restrict__ q_indptr,
                                                                   const int* __restrict__ state_slots, float* __restrict__ out, int H, int kq_heads,
                                                                   int vdim, int longest) {
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
  __nv_bfloat16* ss = bufs + 2 * L::BUF + grp * 16;        // [3][128][VP] S_0, the group's columns
  __nv_bfloat16* wv = ss + 3 * L::SS;                      // [3][64][VP] D_nj b_j v_j
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
    if (tid < kNumbers / 4) cp_async16(smem_u32(buf + 2 * L::QK + L::V + tid * 8), of_chunk(chunk) + kTiles * kTileWords + tid * 4, 16);
    cp_commit();
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
    uint4 w[4][3];                                         // the weighted scores of the warp's row of tiles
#pragma unroll
    for (int kt = 0; kt < 4; ++kt)
      if (kt <= rt)
#pragma unroll
        for (int i = 0; i < 3; ++i)
          w[kt][i] = __ldg(reinterpret_cast<const uint4*>(of_chunk(ch) + (rt * (rt + 1) / 2 + kt) * kTileWords + (i * 32 + lane) * 4));
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
#pragma unroll
    for (int it = 0; it < 4; ++it) {                       // the weighted values
      const int idx = (wq * 32 + lane) + it * 128, j = idx >> 3, c = (idx & 7) * 2;
      const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(vs + j * VP + c);
      const float f = num[kC + j];
      uint32_t s3[3];
      split3(__low2float(x) * f, __high2float(x) * f, s3[0], s3[1], s3[2]);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(wv + i * L::V + j * VP + c) = s3[i];
    }
    asm volatile("bar.sync %0, 128;\n" ::"r"(grp + 1) : "memory");
    const int i0 = rt * 16 + gid;
    if (rt * 16 < n) {
      float o[2][4], rest[2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[0][i] = o[1][i] = rest[0][i] = rest[1][i] = 0.f;
#pragma unroll 4
      for (int kk = 0; kk < kDim / 16; ++kk) {
        uint32_t qa[4];
        ldsm_x4(smem_u32(qs + (rt * 16 + (lane & 15)) * kQP + kk * 16 + (lane >> 4) * 8), qa[0], qa[1], qa[2], qa[3]);
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(smem_u32(ss + i * L::SS + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8), b0, b1, b2, b3);
          if (i > 0) {
            mma_bf16(rest[0], qa, b0, b1);
            mma_bf16(rest[1], qa, b2, b3);
          } else {
            mma_add(o[0], qa, b0, b1);
            mma_add(o[1], qa, b2, b3);
          }
        }
      }
      const float f[2] = {num[i0], num[i0 + 8]};
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[nt][i] = (o[nt][i] + rest[nt][i]) * f[i >> 1];
      // In the rows' own tile a value that comes after a row meets a weight of zero, which an infinity or a NaN survives.  So a warp that
      // finds one among its sums forms them again, with that tile's products added up value by value.
      float sum[2][4];
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[nt][i] = o[nt][i], rest[nt][i] = 0.f;
#pragma unroll
        for (int jt = 0; jt < 4; ++jt) {
          if (jt > rt - pass) break;
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(smem_u32(vs + (jt * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8), b0, b1, b2, b3);
#pragma unroll
          for (int i = 2; i >= 0; --i) {
            const uint32_t pa[4] = {w[jt][i].x, w[jt][i].y, w[jt][i].z, w[jt][i].w};
            if (i > 0) {
              mma_bf16(rest[0], pa, b0, b1);
              mma_bf16(rest[1], pa, b2, b3);
            } else {
              mma_add(sum[0], pa, b0, b1);
              mma_add(sum[1], pa, b2, b3);
            }
          }
        }
        float odd = 0.f;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            sum[nt][i] += rest[nt][i];
            odd = fmaf(sum[nt][i], 0.f, odd);
          }
        if (pass) {
          uint32_t own[3][4];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const uint4 x = __ldg(reinterpret_cast<const uint4*>(of_chunk(ch) + (rt * (rt + 1) / 2 + rt) * kTileWords + (i * 32 + lane) * 4));
            own[i][0] = x.x, own[i][1] = x.y, own[i][2] = x.z, own[i][3] = x.w;
          }
          add_seen<VP>(own, vs + rt * 16 * VP + 2 * t4, lane, sum[0], sum[1]);
        } else if (!__any_sync(0xffffffffu, odd != odd)) {
          break;
        }
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
    const float whole = num[2 * kC];
    float rest[2][2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[m][nn][i] *= whole, rest[m][nn][i] = 0.f;
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
        ldsm_x4_t(smem_u32(wv + i * L::V + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8), b0, b1, b2, b3);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          if (i > 0) {
            mma_bf16(rest[m][0], ka[m], b0, b1);
            mma_bf16(rest[m][1], ka[m], b2, b3);
          } else {
            mma_add(S[m][0], ka[m], b0, b1);
            mma_add(S[m][1], ka[m], b2, b3);
          }
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[m][nn][i] += rest[m][nn][i];
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
  const cudaError_t raised = limit.raise((const void*)decay_rows_tc_kernel<G>, Layout<G>::SMEM);
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(decay_rows_tc_kernel<G>, dim3((vdim + 16 * G - 1) / (16 * G), H, R), dim3(128 * G), Layout<G>::SMEM, s, 1, (const __nv_bfloat16*)q,
                (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, q_stride, k_stride, v_stride, chunks, state, slot_stride, q_indptr, state_slots,
                out, H, kq_heads, vdim, longest);
  return launch_status();
}

}  // namespace

// What arle_decay_tc does with dim 128 and vcols == vdim (vdim a multiple of 8), out on 8-byte boundaries.  num_chunks: of 64 tokens, of the
// long_rows rows of more than `longest` tokens; scratch: 4,096 float32 numbers for each of them and each head, 16-byte aligned.
ARLE_API int arle_decay_rows_tc(const void* q, const void* k, const void* v, int q_stride, int k_stride, int v_stride, const float* a, const float* b,
                                float* state, long slot_stride, const int* q_indptr, const int* state_slots, float* out, float* scratch,
                                int num_chunks, int long_rows, int R, int H, int kq_heads, int vdim, float q_scale, int longest, cudaStream_t s) {
  if (R <= 0 || num_chunks <= 0) return 0;
  if (H <= 0 || kq_heads <= 0 || H % kq_heads || vdim <= 0 || longest < 0 || !scratch) return ARLE_E_BADARG;
  if (vdim % 8 || q_stride % 8 || k_stride % 8 || v_stride % 8 || H > 65535 || R > 65535 ||
      (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch) & 15) || ((uintptr_t)out & 7))
    return ARLE_E_UNSUPPORTED;
  static_assert(kChunkWords == 4096, "the scratch of a chunk and head");
  uint32_t* chunks = reinterpret_cast<uint32_t*>(scratch);
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)decay_tiles_kernel, sizeof(TilesSmem));
  if (raised != cudaSuccess) return (int)raised;
  const int heads = H / kq_heads % kMostHeads == 0 ? kMostHeads : 1;
  launch_kernel(decay_tiles_kernel, dim3(num_chunks, H / heads), dim3(128), sizeof(TilesSmem), s, 1, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k,
                (long)q_stride, (long)k_stride, a, b, q_indptr, R, longest, H, kq_heads, heads, q_scale, chunks);
  // one group a block while two of them an SM hold all columns of the rows that run here (32 heads of 64 columns, 2,048 tokens: 81 us, with four
  // groups 179), four beyond (128 heads: 226 with one or two groups, 197)
  if ((long)((vdim + 15) / 16) * H * long_rows <= 296)
    return launch<1>(q, k, v, q_stride, k_stride, v_stride, chunks, state, slot_stride, q_indptr, state_slots, out, R, H, kq_heads, vdim, longest, s);
  return launch<4>(q, k, v, q_stride, k_stride, v_stride, chunks, state, slot_stride, q_indptr, state_slots, out, R, H, kq_heads, vdim, longest, s);
}
