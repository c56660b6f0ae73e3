// Matrix memories with a scalar decay per token and head over long rows, in chunks of 64 tokens on the tensor cores:
//
//     S_t = a_t S_(t-1) + b_t k_t v_t^T,        o_t = S_t^T (q_scale q_t)        (S: dim x vcols, float32; a_t in [0, 1], b_t per head)
//
// The scan in recurrent.cu runs a token after the other: a chain of 2,048 steps that leaves the machine idle.  With S_0 the memory
// before a chunk and D_ij = a_(j+1) .. a_i the same sums are three small matrix products a chunk,
//     o_i = D_i S_0^T q_i + sum_(j <= i) D_ij b_j (q_i . k_j) v_j,        S_n = D_n S_0 + sum_j D_nj b_j k_j v_j^T     (D_i = a_1 .. a_i),
// and the chain has a step a chunk.  A block owns a head and VT columns of v for a whole row: S stays in registers (mma.sync
// accumulators), so nothing is written between chunks but the outputs; the next chunk's q, k and v are on their way meanwhile.
//
// Precision: q, k and v are bfloat16, so q . k is a sum of exact products with float32 accumulation.  What is float32 beside them (S_0,
// the weighted scores, the weighted values) is cut into three bfloat16 numbers that together hold its 24 bits, and takes three
// products.  D comes from sums of log2 a in float64: a token that forgets nearly everything would otherwise cost the pairs behind it
// their digits.  A decay of zero counts as 2^-300.
//
// Per chunk, eight warps: scores 16 rows x 64 (two warps each, half the columns of v), read-out of S_0 from its three parts in
// shared memory, weighted scores times v, and the update, where a warp holds 16 (or 32) rows of S.
// With 128 keys and no column of ones, most steps with rows of three chunks and all with four take decay_rows_tc.cu, which has the same bits.
// Rows of up to `longest` tokens are left alone (the scan runs them).  A token's sums have one order for its place in its row, whatever
// else is in the step; where a prompt is cut shows in the last bits.
//
// Against float64 over 64 to 2,048 tokens the outputs are off by 1.0e-7 to 1.3e-7 of their norm (the scan: 1.0e-7 to 1.3e-7), the memories
// by 0.8e-7 to 1.0e-7 (0.6e-7 to 1.1e-7).
//
// What bounds it: the chain of chunks of a block (some 9 us each: the tensor cores' legacy path, a third of the time, then the matrix
// loads and the barriers between the phases), with one block an SM.  A scheduler has two warps; one takes an early tile of rows and the other a
// late one, which sees more keys.  One row of 2,048 tokens: 128 heads of 128 x 64 in 8 groups 294 us (315 with two early or two late ones, the
// scan 1,162), 8 heads of 256 x 513 304 us (325; 1,740 to 1,937 as the scan's mean of both).
#include "common.cuh"
#include "chunk_parts.cuh"
using namespace arle;

namespace {

constexpr int kThreads = 256;

template <int DIM, int VT>
struct Layout {
  static constexpr int QP = DIM + 8, VP = VT + 8;                    // pitches: eight rows of a matrix load fall on different banks
  static constexpr size_t QK = (size_t)kC * QP, V = (size_t)kC * VP; // numbers of one buffer
  static constexpr size_t BUF = 2 * QK + V;
  static constexpr size_t SS = (size_t)DIM * VP, WV = V;             // one of the three parts
  static constexpr size_t SMEM = (2 * BUF + 3 * SS + 3 * WV) * 2 + kC * 8 + 2 * kC * 4;
};

template <int DIM, int VT>
__global__ void __launch_bounds__(kThreads, 1) decay_tc_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, long q_stride, long k_stride,
    long v_stride, const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ state, long slot_stride,
    const int* __restrict__ q_indptr, const int* __restrict__ state_slots, float* __restrict__ out, int H, int kq_heads, int vdim, int vcols,
    float q_scale, int longest) {
  pdl_launch_dependents();
  pdl_wait();
  typedef Layout<DIM, VT> L;
  constexpr int QP = L::QP, VP = L::VP;
  constexpr int NT = VT / 16;                              // tiles of 8 columns of a warp's half of the outputs
  constexpr bool SPLIT_N = DIM == 64;                      // the update: four tiles of 16 rows, two warps each with half the columns
  constexpr int MT = DIM >= 128 ? DIM / 128 : 1, UN = SPLIT_N ? VT / 16 : VT / 8;
  extern __shared__ __align__(16) unsigned char raw[];
  __nv_bfloat16* bufs = reinterpret_cast<__nv_bfloat16*>(raw);
  __nv_bfloat16* ss = bufs + 2 * L::BUF;                   // [3][DIM][VP]
  __nv_bfloat16* wv = ss + 3 * L::SS;                      // [3][64][VP]
  double* cum = reinterpret_cast<double*>(wv + 3 * L::WV); // [64] log2 of a_1 .. a_i
  float* bs = reinterpret_cast<float*>(cum + kC);          // [64]
  float* ws = bs + kC;                                     // [64] D_nj b_j
  const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * VT;
  const int beg = q_indptr[r], end = q_indptr[r + 1];
  if (end - beg <= longest) return;
  const int g = h / (H / kq_heads);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, t4 = lane & 3;
  const int rt = warp < 4 ? warp : 7 - warp, n_half = (warp >> 2) * (VT / 2);      // a scheduler's two warps take early and late rows
  const int um = (SPLIT_N ? (warp & 3) : warp * MT) * 16, un = SPLIT_N ? n_half : 0;
  float* sp = state + (size_t)state_slots[r] * slot_stride + (size_t)h * vcols * DIM;

  float S[MT][UN][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < UN; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = um + m * 16 + gid + (i >> 1) * 8, c = c0 + un + n * 8 + 2 * t4 + (i & 1);
        S[m][n][i] = c < vcols ? sp[(size_t)c * DIM + d] : 0.f;
      }

  auto load = [&](int t0, __nv_bfloat16* buf) {
    const int n = min(kC, end - t0);
    constexpr int CH = DIM / 8;
#pragma unroll
    for (int it = 0; it < kC * CH / kThreads; ++it) {
      const int idx = tid + it * kThreads, j = idx / CH, e = idx % CH * 8;
      const bool ok = j < n;
      cp_async16(smem_u32(buf + j * QP + e), ok ? q + (size_t)(t0 + j) * q_stride + (size_t)g * DIM + e : q, ok ? 16 : 0);
      cp_async16(smem_u32(buf + L::QK + j * QP + e), ok ? k + (size_t)(t0 + j) * k_stride + (size_t)g * DIM + e : k, ok ? 16 : 0);
    }
    __nv_bfloat16* vb = buf + 2 * L::QK;
    if (c0 < vdim) {
      for (int idx = tid; idx < kC * (VT / 8); idx += kThreads) {
        const int j = idx / (VT / 8), c = idx % (VT / 8) * 8;
        const bool ok = j < n && c0 + c < vdim;
        cp_async16(smem_u32(vb + j * VP + c), ok ? v + (size_t)(t0 + j) * v_stride + (size_t)h * vdim + c0 + c : v, ok ? 16 : 0);
      }
    } else {                                               // the column of ones
      for (int idx = tid; idx < kC * VT; idx += kThreads) {
        const int j = idx / VT, c = idx % VT;
        vb[j * VP + c] = __float2bfloat16_rn(j < n && c0 + c == vdim ? 1.f : 0.f);
      }
    }
    cp_commit();
  };
  // the first warp's decays and factors of a chunk (two tokens a lane), asked for a chunk ahead
  float la[2], lb[2];
  auto gates = [&](int t0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = t0 + 2 * lane + i;
      la[i] = t < end ? a[(size_t)t * H + h] : 1.f;
      lb[i] = t < end ? b[(size_t)t * H + h] : 0.f;
    }
  };
  load(beg, bufs);
  if (warp == 0) gates(beg);
  int p = 0;
  for (int t0 = beg; t0 < end; t0 += kC, p ^= 1) {
    const int n = min(kC, end - t0);
    __nv_bfloat16* qs = bufs + p * L::BUF;
    __nv_bfloat16* ks = qs + L::QK;
    __nv_bfloat16* vs = ks + L::QK;
    cp_wait<0>();
    __syncthreads();                                       // the chunk is here, and the one before is used up
    if (t0 + kC < end) load(t0 + kC, bufs + (p ^ 1) * L::BUF);
    if (warp == 0) {
      double x[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        x[i] = la[i] == la[i] ? (double)fmaxf(log2f(la[i]), -300.f) : (double)la[i];
      }
      double sum = x[0] + x[1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += y;
      }
      const double total = __shfl_sync(0xffffffffu, sum, 31);
      double first = __shfl_up_sync(0xffffffffu, sum, 1);  // of the tokens before this lane's: a NaN among the decays stays behind them
      first = (lane ? first : 0.0) + x[0];
      cum[2 * lane] = first;
      cum[2 * lane + 1] = sum;
      bs[2 * lane] = lb[0];
      bs[2 * lane + 1] = lb[1];
      ws[2 * lane] = lb[0] * exp2f((float)(total - first));
      ws[2 * lane + 1] = lb[1] * exp2f((float)(total - sum));
      if (t0 + kC < end) gates(t0 + kC);
    }
    // S_0 in three parts
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nn = 0; nn < UN; ++nn)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t s3[3];
          split3(S[m][nn][2 * half], S[m][nn][2 * half + 1], s3[0], s3[1], s3[2]);
          const size_t at = (size_t)(um + m * 16 + gid + half * 8) * VP + un + nn * 8 + 2 * t4;
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(ss + i * L::SS + at) = s3[i];
        }
    __syncthreads();                                       // the parts, the decays and the factors are there
    for (int idx = tid; idx < kC * (VT / 2); idx += kThreads) {
      const int j = idx / (VT / 2), c = idx % (VT / 2) * 2;
      const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(vs + j * VP + c);
      uint32_t s3[3];
      split3(__low2float(x) * ws[j], __high2float(x) * ws[j], s3[0], s3[1], s3[2]);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(wv + i * L::WV + j * VP + c) = s3[i];
    }
    // In the rows' own tile a value that comes after a row meets a weight of zero, which an infinity or a NaN survives.  So a warp that
    // finds one among its sums forms them again, with that tile's products added up value by value.
    const bool rows_here = rt * 16 < n;
#pragma unroll 1
    for (int pass = 0; rows_here && pass < 2; ++pass) {
      uint32_t own[3][4];                                  // second time: the weights of the rows' own tile
      float sc[8][4], o[NT][4], rest[NT][4];               // rest: from the middle and last parts
#pragma unroll
      for (int i = 0; i < 8; ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
#pragma unroll
      for (int i = 0; i < NT; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = rest[i][0] = rest[i][1] = rest[i][2] = rest[i][3] = 0.f;
#pragma unroll 4
      for (int kk = 0; kk < DIM / 16; ++kk) {
        uint32_t qa[4];
        ldsm_x4(smem_u32(qs + (rt * 16 + (lane & 15)) * QP + kk * 16 + (lane >> 4) * 8), qa[0], qa[1], qa[2], qa[3]);
#pragma unroll
        for (int jt = 0; jt < 4; ++jt) {
          if (jt > rt) break;                              // keys behind the rows' places
          uint32_t b0, b1, b2, b3;
          ldsm_x4(smem_u32(ks + (jt * 16 + (lane >> 4) * 8 + (lane & 7)) * QP + kk * 16 + ((lane >> 3) & 1) * 8), b0, b1, b2, b3);
          mma_add(sc[2 * jt], qa, b0, b1);
          mma_add(sc[2 * jt + 1], qa, b2, b3);
        }
#pragma unroll
        for (int i = 2; i >= 0; --i)
#pragma unroll
          for (int nt = 0; nt < NT; nt += 2) {
            uint32_t b0, b1, b2, b3;
            ldsm_x4_t(smem_u32(ss + i * L::SS + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + n_half + nt * 8 + (lane >> 4) * 8), b0,
                      b1, b2, b3);
            if (i > 0) {
              mma_bf16(rest[nt], qa, b0, b1);
              mma_bf16(rest[nt + 1], qa, b2, b3);
            } else {
              mma_add(o[nt], qa, b0, b1);
              mma_add(o[nt + 1], qa, b2, b3);
            }
          }
      }
      const int i0 = rt * 16 + gid;
      const double cu[2] = {cum[i0], cum[i0 + 8]};
      const float f0 = q_scale * exp2f((float)cu[0]), f1 = q_scale * exp2f((float)cu[1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o[nt][i] = (o[nt][i] + rest[nt][i]) * (i < 2 ? f0 : f1);
          rest[nt][i] = 0.f;
        }
      }
#pragma unroll
      for (int jt = 0; jt < 4; ++jt) {
        if (jt > rt) break;
        uint32_t pa[3][4];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {                   // the tile's two groups of 8 keys
          const int j = jt * 16 + hh * 8 + 2 * t4;
          const double cj[2] = {cum[j], cum[j + 1]};
          const float fb[2] = {bs[j] * q_scale, bs[j + 1] * q_scale};
          float w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = i0 + (i >> 1) * 8;
            w[i] = j + (i & 1) <= row ? sc[2 * jt + hh][i] * (fb[i & 1] * exp2f((float)(cu[i >> 1] - cj[i & 1]))) : 0.f;
          }
          split3(w[0], w[1], pa[0][2 * hh], pa[1][2 * hh], pa[2][2 * hh]);
          split3(w[2], w[3], pa[0][2 * hh + 1], pa[1][2 * hh + 1], pa[2][2 * hh + 1]);
        }
        if (pass && jt == rt) {
#pragma unroll
          for (int i = 0; i < 12; ++i) own[i / 4][i % 4] = pa[i / 4][i % 4];
          break;
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt += 2) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(smem_u32(vs + (jt * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + n_half + nt * 8 + (lane >> 4) * 8), b0, b1, b2, b3);
#pragma unroll
          for (int i = 2; i > 0; --i) {
            mma_bf16(rest[nt], pa[i], b0, b1);
            mma_bf16(rest[nt + 1], pa[i], b2, b3);
          }
          mma_add(o[nt], pa[0], b0, b1);
          mma_add(o[nt + 1], pa[0], b2, b3);
        }
      }
      float odd = 0.f;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o[nt][i] += rest[nt][i];
          odd = fmaf(o[nt][i], 0.f, odd);
        }
      if (pass == 0 && __any_sync(0xffffffffu, odd != odd)) continue;
      if (pass)
#pragma unroll
        for (int nt = 0; nt < NT; nt += 2) add_seen<VP>(own, vs + rt * 16 * VP + n_half + nt * 8 + 2 * t4, lane, o[nt], o[nt + 1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int i = i0 + half * 8, c = c0 + n_half + nt * 8 + 2 * t4;
          if (i >= n) continue;
          float* op = out + ((size_t)(t0 + i) * H + h) * vcols + c;
          if (c < vcols) op[0] = o[nt][2 * half];
          if (c + 1 < vcols) op[1] = o[nt][2 * half + 1];
        }
      break;
    }
    __syncthreads();                                       // the weighted values are there, S_0's parts are used up
    const float whole = exp2f((float)cum[kC - 1]);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int nn = 0; nn < UN; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[m][nn][i] *= whole;
    uint32_t ka[kC / 16][MT][4];
#pragma unroll
    for (int kk = 0; kk < kC / 16; ++kk)
#pragma unroll
      for (int m = 0; m < MT; ++m)
        ldsm_x4_t(smem_u32(ks + (kk * 16 + (lane >> 4) * 8 + (lane & 7)) * QP + um + m * 16 + ((lane >> 3) & 1) * 8), ka[kk][m][0], ka[kk][m][1],
                  ka[kk][m][2], ka[kk][m][3]);
#pragma unroll
    for (int nn = 0; nn < UN; nn += 2) {
      float rest[MT][2][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) rest[m][0][i] = rest[m][1][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < kC / 16; ++kk)
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(smem_u32(wv + i * L::WV + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + un + nn * 8 + (lane >> 4) * 8), b0, b1, b2,
                    b3);
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            if (i > 0) {
              mma_bf16(rest[m][0], ka[kk][m], b0, b1);
              mma_bf16(rest[m][1], ka[kk][m], b2, b3);
            } else {
              mma_add(S[m][nn], ka[kk][m], b0, b1);
              mma_add(S[m][nn + 1], ka[kk][m], b2, b3);
            }
          }
        }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          S[m][nn][i] += rest[m][0][i];
          S[m][nn + 1][i] += rest[m][1][i];
        }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int nn = 0; nn < UN; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = um + m * 16 + gid + (i >> 1) * 8, c = c0 + un + nn * 8 + 2 * t4 + (i & 1);
        if (c < vcols) sp[(size_t)c * DIM + d] = S[m][nn][i];
      }
}

template <int DIM, int VT>
int launch(const void* q, const void* k, const void* v, long q_stride, long k_stride, long v_stride, const float* a, const float* b, float* state,
           long slot_stride, const int* q_indptr, const int* state_slots, float* out, int R, int H, int kq_heads, int vdim, int vcols,
           float q_scale, int longest, cudaStream_t s) {
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)decay_tc_kernel<DIM, VT>, Layout<DIM, VT>::SMEM);
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(decay_tc_kernel<DIM, VT>, dim3((vcols + VT - 1) / VT, H, R), dim3(kThreads), Layout<DIM, VT>::SMEM, s, 1, (const __nv_bfloat16*)q,
                (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, q_stride, k_stride, v_stride, a, b, state, slot_stride, q_indptr, state_slots, out,
                H, kq_heads, vdim, vcols, q_scale, longest);
  return launch_status();
}

}  // namespace

// q, k bfloat16 [T, kq_heads*dim], v bfloat16 [T, H*vdim] (row strides multiples of 8, 16-byte aligned), a, b float32 [T, H]; state: float32,
// a slot every slot_stride numbers, [H][vcols][dim] at its start; vcols vdim, or vdim + 1 (a column of ones beside v; vdim then a
// multiple of 64); out float32 [T, H, vcols].  dim 64, 128 or 256, vdim a multiple of 8.
ARLE_API int arle_decay_tc(const void* q, const void* k, const void* v, int q_stride, int k_stride, int v_stride, const float* a, const float* b,
                           float* state, long slot_stride, const int* q_indptr, const int* state_slots, float* out, int R, int H, int kq_heads,
                           int dim, int vdim, int vcols, float q_scale, int longest, cudaStream_t s) {
  if (R <= 0) return 0;
  if (H <= 0 || kq_heads <= 0 || H % kq_heads || vdim <= 0 || (vcols != vdim && vcols != vdim + 1) || longest < 0) return ARLE_E_BADARG;
  if (vdim % 8 || (vcols != vdim && vdim % 64) || q_stride % 8 || k_stride % 8 || v_stride % 8 || H > 65535 || R > 65535 ||
      (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15))
    return ARLE_E_UNSUPPORTED;
#define ARLE_DECAY_TC(D, VT)                                                                                                                \
  return launch<D, VT>(q, k, v, q_stride, k_stride, v_stride, a, b, state, slot_stride, q_indptr, state_slots, out, R, H, kq_heads, vdim, vcols, \
                       q_scale, longest, s)
  // 64 columns a block share the scores; 32 where the blocks of 64 would leave half of the SMs idle
  const bool narrow = (long long)((vcols + 63) / 64) * H * R <= 74;
  if (dim == 64) {
    if (narrow) ARLE_DECAY_TC(64, 32);
    ARLE_DECAY_TC(64, 64);
  }
  if (dim == 128) {
    if (narrow) ARLE_DECAY_TC(128, 32);
    ARLE_DECAY_TC(128, 64);
  }
  if (dim == 256) ARLE_DECAY_TC(256, 32);
#undef ARLE_DECAY_TC
  return ARLE_E_UNSUPPORTED;
}
