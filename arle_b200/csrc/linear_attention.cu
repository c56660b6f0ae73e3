// Gated linear attention: a recurrent mixer with a matrix state per head,
//
//     S_t = diag(alpha_t) S_(t-1) + k_t v_t^T          S: [dim, vdim], float32, one per (request, head)
//     o_t = S_t^T q_t
//
// with a decay alpha_t in (0, 1) per key channel.  Three kernels:
//
//  * gla_decay: alpha[t, c] = sigmoid(z)^(1/tau), z = b[c] + sum_r low[t, r] * w2[c, r], the second
//    half of a low-rank gate (low = W_a1 x comes from the packed input projection).  Evaluated as
//    exp(-softplus(-z) / tau) in float32; a block takes sixteen tokens and 256 channels, r ascending.
//    A second form has tanh between the two matrices and another decay: alpha = exp(-exp(z)), z = b[c] + sum_r
//    tanh(low[t, r]) * w2[c, r].
//  * gla_scan: the recurrence over this step's tokens of every request row, from the state that the
//    request's slot holds, which is left updated.  Float32 throughout; q, k, v are read in the
//    activation type.  One block of 128 threads per (columns of vdim, head, row); a thread keeps four
//    consecutive key channels of each of four columns of S in registers (up to 32 consecutive lanes share a
//    column; the state is stored [vdim][dim], so a column's lanes read one contiguous run), the step's
//    q, k, alpha and v are staged in shared memory a chunk of tokens at a time, and o_t[j] is the sum
//    over the column's lanes.  What bounds it is a warp's instructions: a scheduler of the SM has one warp of a single prompt.  So
//    two channels are one packed instruction (fma.rn.f32x2), and the sums of eight tokens and four columns are added over the 32 lanes
//    together, 31 exchanges instead of 48.  The next chunk's loads are pinned in front
//    of the work that hides them (plain ones were moved behind it), and where there are few blocks four warps more bring them.  16 heads of
//    128 x 128, 2,048 tokens: 190 us (213 where the same warps bring them, 444 with single
//    numbers and a token's sums by themselves, 269 before the loads were pinned).  The order of every sum depends on (dim, vdim) only: a token's result
//    does not depend on how the prompt was cut or on what else is in the batch.
//    With a bonus u (one number per head and key channel) the read-out comes before the update and sees the current
//    token through u instead: o_t = (S_(t-1) + diag(u) k_t v_t^T)^T q_t.
//  * gla_out: per head, o / sqrt(mean(o^2) + eps) * weight (shared by the heads, or one of all heads' size), times silu(gate) (or sigmoid(gate)),
//    times a constant, rounded once into the activation type (a row of a wider buffer may be given).
#include <initializer_list>

#include "common.cuh"
#include "scan_utils.cuh"
using namespace arle;

constexpr int kScanThreads = 128;
constexpr int kScanCpt = 4;                      // columns of the state a thread keeps
constexpr int kDecayTokens = 16;                 // tokens a block of the decay kernel takes
constexpr int kDecayBatch = 16;                  // weights a thread asks for before it uses the first

// w2t is the second matrix of the gate transposed, [rank][channels]: consecutive threads read consecutive floats.
// Bound by instructions: a block's numbers of `low` stand in shared memory with the sixteen tokens of a channel of the rank side by side,
// so that four 16-byte reads feed sixteen sums, two tokens to a packed FMA (the roundings of single ones), and softplus has no branch whose
// two sides a warp would run both; three blocks an SM (one or two: 37 us; four spill at this batch of weights, 35).  2,048 tokens, 2,048
// channels, rank 64: 33 us (45 with a token's sum a read of its own and a branch in softplus); 300 tokens, 1,024 channels, rank 16: 6.3 (8.5).
template <typename T, bool DOUBLE_EXP>
__global__ void __launch_bounds__(256, 3) gla_decay_kernel(const T* __restrict__ low, int low_stride, const float* __restrict__ w2t,
                                                        const float* __restrict__ bias, float inv_tau, float* __restrict__ alpha,
                                                        int num_tokens, int channels, int rank) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float lo_s[];  // [rank][kDecayTokens]
  const int t0 = blockIdx.x * kDecayTokens;
  const int n = min(kDecayTokens, num_tokens - t0);
  for (int i = threadIdx.x; i < kDecayTokens * rank; i += blockDim.x) {
    const int tt = i / rank, r = i - tt * rank;
    const float v = tt < n ? to_f32(low[(size_t)(t0 + tt) * low_stride + r]) : 0.f;
    lo_s[r * kDecayTokens + tt] = DOUBLE_EXP ? tanhf(v) : v;
  }
  __syncthreads();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  f32x2 z[kDecayTokens / 2];                     // tokens 2i and 2i + 1
#pragma unroll
  for (int i = 0; i < kDecayTokens / 2; ++i) z[i] = 0;
  for (int r0 = 0; r0 < rank; r0 += kDecayBatch) {
    float w[kDecayBatch];
#pragma unroll
    for (int i = 0; i < kDecayBatch; ++i) w[i] = r0 + i < rank ? w2t[(size_t)(r0 + i) * channels + c] : 0.f;
#pragma unroll
    for (int i = 0; i < kDecayBatch; ++i) {
      if (r0 + i >= rank) break;
      const ulonglong2* lo = reinterpret_cast<const ulonglong2*>(lo_s + (r0 + i) * kDecayTokens);
      const f32x2 w2 = pair2(w[i], w[i]);
#pragma unroll
      for (int g = 0; g < kDecayTokens / 4; ++g) {
        const ulonglong2 x = lo[g];
        z[2 * g] = fma2(x.x, w2, z[2 * g]);
        z[2 * g + 1] = fma2(x.y, w2, z[2 * g + 1]);
      }
    }
  }
  const float b = bias ? bias[c] : 0.f;
#pragma unroll
  for (int tt = 0; tt < kDecayTokens; ++tt) {
    if (tt >= n) break;
    const float zt = (tt & 1 ? high2(z[tt / 2]) : low2(z[tt / 2])) + b;
    if (DOUBLE_EXP) {
      alpha[(size_t)(t0 + tt) * channels + c] = expf(-expf(zt));
      continue;
    }
    const float sp = fmaxf(-zt, 0.f) + log1pf(expf(-fabsf(zt)));     // softplus(-z) = log(1 + e^-z), the stable way
    alpha[(size_t)(t0 + tt) * channels + c] = expf(-sp * inv_tau);
  }
}

// Four elements as they lie in memory (converted only when they are staged: a conversion right after its load would
// make every load wait for the one before it).
__device__ __forceinline__ float4 load_raw4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ uint2 load_raw4(const __nv_bfloat16* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ float4 widen4(float4 u) { return u; }
__device__ __forceinline__ float4 widen4(uint2 u) {
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
template <typename T, bool VEC> struct Raw4 { using type = float4; };
template <> struct Raw4<__nv_bfloat16, true> { using type = uint2; };

// DPT: consecutive key channels that a thread keeps of each of its kScanCpt columns of the state (4 up to 128
// channels, then 8, 16).  LPC: lanes that share a column (a power of two; LPC * DPT >= dim).  VEC: four channels
// at a time can be fetched with one aligned load.  A chunk of CHUNK tokens is staged in shared memory; while it is
// worked on, the next chunk's q, k, alpha and v are already on their way into registers.  Every number of q, k and
// alpha that a thread reads from shared memory serves four columns: with one column a thread the kernel was bound by
// shared-memory bandwidth.
// BONUS: the read-out before the update, with the current token weighted by u.
// LONG: some row has eight tokens or more; with 32 lanes a column these run in groups of eight.  The form for shorter rows, decoded tokens
// above all, is bound by memory: single numbers instead of pairs, which leaves room for few_blocks() blocks an SM (the most that no form
// spills for), and loads that the compiler may place.  64 requests, 16 heads of 128 x 128: 30.9 us (31.1 with pairs), 64 heads 129.5
// (132).  The same cap on prompts of small heads spilled: 512 tokens, bfloat16, 16 heads of 4 258 us with it and 76 without.
template <typename T, int DPT, int LPC, bool VEC, bool BONUS>
constexpr int few_blocks() {
  if (DPT > 8) return BONUS ? 2 : 3;
  if (DPT > 4) return 4;
  if (LPC == 1) return 3;
  return VEC && !BONUS && LPC >= 4 ? 5 : 4;
}
// SPLIT (32 lanes of four channels a column): four warps more, which bring the chunks, so that the four that hold the memory do nothing else.  Chunks
// of eight tokens go through a ring of kRing places, two more are under way in the loaders' registers.
constexpr int kRing = 3;
__device__ __forceinline__ void named_sync(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(2 * kScanThreads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(2 * kScanThreads) : "memory");
}

template <typename T, int DPT, int LPC, bool VEC, bool BONUS, bool LONG, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 2 * kScanThreads : kScanThreads, SPLIT ? 2 : LONG ? 1 : few_blocks<T, DPT, LPC, VEC, BONUS>()) gla_scan_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, int in_stride,
    const float* __restrict__ alpha, const float* __restrict__ bonus, float* __restrict__ state, long slot_stride, const int* __restrict__ q_indptr,
    const int* __restrict__ state_slots, float* __restrict__ out, int heads, int dim, int vdim, float q_scale) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int CPT = kScanCpt;
  constexpr int COLS = kScanThreads / LPC * CPT; // columns a block takes
  constexpr int DSPAN = DPT * LPC;               // dim rounded up; channels past dim hold zeros
  constexpr int PAD = DPT == 4 ? 4 : DPT + 4;    // floats a thread's channels take in shared memory: 16-byte rows, spread over the banks
  constexpr int DPAD = PAD * LPC;
  // float32 rows with a bonus, decoded: at 16 tokens a chunk the numbers under way spill at four blocks an SM
  constexpr int CHUNK = SPLIT ? 8 : DSPAN >= 512 ? 4 : (DSPAN >= 256 || (!LONG && BONUS && sizeof(T) == 4) ? 8 : 16);
  constexpr int QUADS = CHUNK * DSPAN / 4;       // groups of four channels in a chunk
  constexpr int QPT = (QUADS + kScanThreads - 1) / kScanThreads;
  constexpr int VPT = (CHUNK * COLS + kScanThreads - 1) / kScanThreads;
  constexpr int PLACES = SPLIT ? kRing : 1;
  __shared__ __align__(16) float qs[PLACES * CHUNK * DPAD], ks[PLACES * CHUNK * DPAD], as[PLACES * CHUNK * DPAD];
  constexpr int VD = LONG && LPC >= 4 ? 2 : 1;           // v's numbers stand twice side by side (a factor of both halves of a pair), where there is room
  __shared__ __align__(16) float vs[PLACES * CHUNK * COLS * VD];
  const int r = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * COLS;
  const int tid = threadIdx.x & (kScanThreads - 1);    // among the loaders, or among those that hold the memory
  const int l = tid & (LPC - 1), jl = tid / LPC;
  const int jb = j0 + jl * CPT;                  // this thread's first column
  const int t_begin = q_indptr[r], t_end = q_indptr[r + 1];
  // the state of a head is kept as [vdim][dim]: a thread's channels of a column are contiguous
  float* S_g = state + (size_t)state_slots[r] * slot_stride + ((size_t)h * vdim) * dim + l * DPT;
  const bool vec_state = (dim & 3) == 0 && (slot_stride & 3) == 0 && ((uintptr_t)state & 15) == 0;
  f32x2 u2[BONUS ? DPT / 2 : 1];
  if constexpr (BONUS) {
#pragma unroll
    for (int i = 0; i < DPT / 2; ++i) {
      const int c = l * DPT + 2 * i;
      u2[i] = pair2(c < dim ? bonus[(size_t)h * dim + c] : 0.f, c + 1 < dim ? bonus[(size_t)h * dim + c + 1] : 0.f);
    }
  }
  f32x2 S[CPT][DPT / 2];                         // channels 2i and 2i + 1 of a column
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc) {
    const bool col_ok = jb + cc < vdim && !(SPLIT && threadIdx.x >= kScanThreads);
    const float* sp = S_g + (size_t)(col_ok ? jb + cc : 0) * dim;
#pragma unroll
    for (int i = 0; i < DPT; i += 4) {
      const int c = l * DPT + i;
      if (vec_state) {
        ulonglong2 x = make_ulonglong2(0, 0);    // as pairs: packing them here would wait for every load
        if (col_ok && c < dim) x = *reinterpret_cast<const ulonglong2*>(sp + i);
        S[cc][i / 2] = x.x, S[cc][i / 2 + 1] = x.y;
      } else {
#pragma unroll
        for (int e = 0; e < 4; e += 2)
          S[cc][(i + e) / 2] = pair2((col_ok && c + e < dim) ? sp[i + e] : 0.f, (col_ok && c + e + 1 < dim) ? sp[i + e + 1] : 0.f);
      }
    }
  }
  const size_t hq = (size_t)h * dim, hv = (size_t)h * vdim;
  const size_t a_stride = (size_t)heads * dim;
  using RawT = typename Raw4<T, VEC>::type;
  struct Raw {
    RawT q[QPT], k[QPT];
    float4 a[QPT];
    T v[VPT];
  };

  // The chunk's numbers into registers; nothing waits on them yet.  Loads are unconditional (a place outside the
  // chunk reads the row's first token instead and is zeroed when staged), so that they are all under way at once.
  auto fetch = [&](Raw& raw, int t0, int n) {
    RawT (&rq)[QPT] = raw.q, (&rk)[QPT] = raw.k;
    float4 (&ra)[QPT] = raw.a;
    T (&rv)[VPT] = raw.v;
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const int idx = tid + u * kScanThreads;
      const int tt = idx / (DSPAN / 4), c = (idx - tt * (DSPAN / 4)) * 4;
      const bool ok = idx < QUADS && tt < n && c < dim;
      const size_t row = ok ? (size_t)(t0 + tt) : (size_t)t_begin;
      const int cs = ok ? c : 0;
      if constexpr (VEC) {
        if constexpr (LONG) {
          rq[u] = load_now(q + row * in_stride + hq + cs, RawT());
          rk[u] = load_now(k + row * in_stride + hq + cs, RawT());
          ra[u] = load_now(alpha + row * a_stride + hq + cs, float4());
        } else {
          rq[u] = load_raw4(q + row * in_stride + hq + cs);
          rk[u] = load_raw4(k + row * in_stride + hq + cs);
          ra[u] = load_raw4(alpha + row * a_stride + hq + cs);
        }
      } else {
        float4 fq = make_float4(0.f, 0.f, 0.f, 0.f), fk = fq, fa = fq;
        float* pq = &fq.x; float* pk = &fk.x; float* pa = &fa.x;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (cs + e < dim) {
            pq[e] = to_f32(q[row * in_stride + hq + cs + e]);
            pk[e] = to_f32(k[row * in_stride + hq + cs + e]);
            pa[e] = alpha[row * a_stride + hq + cs + e];
          }
        *reinterpret_cast<float4*>(&rq[u]) = fq;
        *reinterpret_cast<float4*>(&rk[u]) = fk;
        ra[u] = fa;
      }
    }
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int idx = tid + u * kScanThreads;
      const int tt = idx / COLS, c = idx - tt * COLS;
      const bool ok = idx < CHUNK * COLS && tt < n && j0 + c < vdim;
      const T* vp = v + (ok ? (size_t)(t0 + tt) : (size_t)t_begin) * in_stride + hv + (ok ? j0 + c : 0);
      if constexpr (LONG) rv[u] = load_now(vp, T());
      else rv[u] = *vp;
    }
  };
  auto stage = [&](const Raw& raw, int n, int place) {   // registers to shared memory, widened, q scaled on the way
    const RawT (&rq)[QPT] = raw.q, (&rk)[QPT] = raw.k;
    const float4 (&ra)[QPT] = raw.a;
    const T (&rv)[VPT] = raw.v;
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const int idx = tid + u * kScanThreads;
      const int tt = idx / (DSPAN / 4), c = (idx - tt * (DSPAN / 4)) * 4;
      const int at = (place * CHUNK + tt) * DPAD + (c / DPT) * PAD + (c % DPT);
      if (idx >= QUADS) continue;
      const bool ok = tt < n && c < dim;
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 fq = widen4(rq[u]), fk = widen4(rk[u]);
      *reinterpret_cast<float4*>(qs + at) = ok ? make_float4(fq.x * q_scale, fq.y * q_scale, fq.z * q_scale, fq.w * q_scale) : z;
      *reinterpret_cast<float4*>(ks + at) = ok ? fk : z;
      *reinterpret_cast<float4*>(as + at) = ok ? ra[u] : z;
    }
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      const int idx = tid + u * kScanThreads;
      const int tt = idx / COLS, c = idx - tt * COLS;
      if (idx < CHUNK * COLS) {
        const float x = (tt < n && j0 + c < vdim) ? to_f32(rv[u]) : 0.f;
        if (VD == 2) *reinterpret_cast<float2*>(vs + VD * (place * CHUNK * COLS + idx)) = make_float2(x, x);
        else vs[place * CHUNK * COLS + idx] = x;
      }
    }
  };

  Raw raw;
  if constexpr (SPLIT) {
    // Barriers 1 .. kRing: a place is full; kRing + 1 .. 2 kRing: it has been read (waited for, and arrived at, where a later chunk needs it).
    const int chunks = (t_end - t_begin + CHUNK - 1) / CHUNK;
    if (threadIdx.x >= kScanThreads) {
      Raw other;
      auto get = [&](Raw& to, int c) {
        if (c < chunks) fetch(to, t_begin + c * CHUNK, min(CHUNK, t_end - t_begin - c * CHUNK));
      };
      auto put = [&](Raw& from, int c) {
        if (c >= chunks) return;
        const int place = c % kRing;
        if (c >= kRing) named_sync(kRing + 1 + place);
        stage(from, min(CHUNK, t_end - t_begin - c * CHUNK), place);
        named_arrive(1 + place);
        get(from, c + 2);
      };
      get(raw, 0);
      get(other, 1);
      for (int c = 0; c < chunks; c += 2) {
        put(raw, c);
        put(other, c + 1);
      }
      return;
    }
  } else if (t_begin < t_end) {
    fetch(raw, t_begin, min(CHUNK, t_end - t_begin));
  }
  int place = 0;
  for (int t0 = t_begin; t0 < t_end; t0 += CHUNK) {
    const int n = min(CHUNK, t_end - t0);
    if constexpr (SPLIT) {
      named_sync(1 + place);
    } else {
      __syncthreads();                           // the chunk before has been read by everyone
      stage(raw, n, 0);
      __syncthreads();
      if (t0 + CHUNK < t_end) fetch(raw, t0 + CHUNK, min(CHUNK, t_end - t0 - CHUNK));
    }
    const float *qp = qs + place * CHUNK * DPAD, *kp = ks + place * CHUNK * DPAD, *ap = as + place * CHUNK * DPAD;
    const float* vp = vs + place * CHUNK * COLS * VD;
    // one token: the memory's step and the thread's part of its columns' sums
    auto token = [&](int tt, float (&o)[CPT]) {
      if constexpr (!LONG) {                     // single numbers: the same roundings in fewer registers
        const float4 v4 = *reinterpret_cast<const float4*>(vp + tt * COLS + jl * CPT);
        const float vj[CPT] = {v4.x, v4.y, v4.z, v4.w};
        const float4* qt = reinterpret_cast<const float4*>(qp + tt * DPAD + l * PAD);
        const float4* kt = reinterpret_cast<const float4*>(kp + tt * DPAD + l * PAD);
        const float4* at = reinterpret_cast<const float4*>(ap + tt * DPAD + l * PAD);
        float lo[CPT], hi[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) lo[cc] = hi[cc] = 0.f;
#pragma unroll
        for (int i = 0; i < DPT / 4; ++i) {
          const float4 a4 = at[i], k4 = kt[i], q4 = qt[i];
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) {
            const float s0 = low2(S[cc][2 * i]), s1 = high2(S[cc][2 * i]), s2 = low2(S[cc][2 * i + 1]), s3 = high2(S[cc][2 * i + 1]);
            const float x0 = k4.x * vj[cc], x1 = k4.y * vj[cc], x2 = k4.z * vj[cc], x3 = k4.w * vj[cc];
            const float n0 = fmaf(a4.x, s0, x0), n1 = fmaf(a4.y, s1, x1), n2 = fmaf(a4.z, s2, x2), n3 = fmaf(a4.w, s3, x3);
            S[cc][2 * i] = pair2(n0, n1), S[cc][2 * i + 1] = pair2(n2, n3);
            if constexpr (BONUS) {
              lo[cc] = fmaf(fmaf(low2(u2[2 * i + 1]), x2, s2), q4.z, fmaf(fmaf(low2(u2[2 * i]), x0, s0), q4.x, lo[cc]));
              hi[cc] = fmaf(fmaf(high2(u2[2 * i + 1]), x3, s3), q4.w, fmaf(fmaf(high2(u2[2 * i]), x1, s1), q4.y, hi[cc]));
            } else {
              lo[cc] = fmaf(n2, q4.z, fmaf(n0, q4.x, lo[cc]));
              hi[cc] = fmaf(n3, q4.w, fmaf(n1, q4.y, hi[cc]));
            }
          }
        }
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) o[cc] = lo[cc] + hi[cc];
        return;
      }
      f32x2 vj[CPT];
      if constexpr (VD == 2) {
        const ulonglong2 va = *reinterpret_cast<const ulonglong2*>(vp + (tt * COLS + jl * CPT) * 2);
        const ulonglong2 vb = *reinterpret_cast<const ulonglong2*>(vp + (tt * COLS + jl * CPT) * 2 + 4);
        vj[0] = va.x, vj[1] = va.y, vj[2] = vb.x, vj[3] = vb.y;
      } else {
        const float4 v4 = *reinterpret_cast<const float4*>(vp + tt * COLS + jl * CPT);
        vj[0] = pair2(v4.x, v4.x), vj[1] = pair2(v4.y, v4.y), vj[2] = pair2(v4.z, v4.z), vj[3] = pair2(v4.w, v4.w);
      }
      const ulonglong2* qt = reinterpret_cast<const ulonglong2*>(qp + tt * DPAD + l * PAD);
      const ulonglong2* kt = reinterpret_cast<const ulonglong2*>(kp + tt * DPAD + l * PAD);
      const ulonglong2* at = reinterpret_cast<const ulonglong2*>(ap + tt * DPAD + l * PAD);
      f32x2 o2[CPT];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) o2[cc] = 0;
#pragma unroll
      for (int i = 0; i < DPT / 4; ++i) {
        const ulonglong2 a4 = at[i], k4 = kt[i], q4 = qt[i];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          const f32x2 kv0 = mul2(k4.x, vj[cc]), kv1 = mul2(k4.y, vj[cc]);
          if constexpr (BONUS) {
            o2[cc] = fma2(fma2(u2[2 * i], kv0, S[cc][2 * i]), q4.x, o2[cc]);
            o2[cc] = fma2(fma2(u2[2 * i + 1], kv1, S[cc][2 * i + 1]), q4.y, o2[cc]);
          }
          S[cc][2 * i] = fma2(a4.x, S[cc][2 * i], kv0);
          S[cc][2 * i + 1] = fma2(a4.y, S[cc][2 * i + 1], kv1);
          if constexpr (!BONUS) {
            o2[cc] = fma2(S[cc][2 * i], q4.x, o2[cc]);
            o2[cc] = fma2(S[cc][2 * i + 1], q4.y, o2[cc]);
          }
        }
      }
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) o[cc] = low2(o2[cc]) + high2(o2[cc]);
    };
    int first = 0;
    if constexpr (LONG && LPC == 32 && CHUNK % 8 == 0) {
      // Eight tokens at a time: their 32 sums over 32 lanes in 31 exchanges, after which lane l holds token l / 4's sum of column
      // l % 4.  A sum's additions are those of a token by itself (lanes 16 apart, then 8, 4, 2, 1).
      for (; first + 8 <= n; first += 8) {
        float x[32];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          float o[CPT];
          token(first + g, o);
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) x[g * CPT + cc] = o[cc];
        }
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
          const bool up = (l & w) != 0;
#pragma unroll
          for (int i = 0; i < w; ++i) {
            const float got = __shfl_xor_sync(0xffffffffu, up ? x[i] : x[i + w], w);
            x[i] = (up ? x[i + w] : x[i]) + got;
          }
        }
        if (jb + (l & 3) < vdim) out[(size_t)(t0 + first + (l >> 2)) * heads * vdim + hv + jb + (l & 3)] = x[0];
      }
    }
    constexpr int kUnroll = LPC < 32 ? 4 : 1;    // 32 lanes: at most seven tokens come here; fewer: all (f32 heads of 64, 512 tokens: 91 -> 86 us)
#pragma unroll kUnroll
    for (int tt = first; tt < n; ++tt) {
      float o[CPT];
      token(tt, o);
      // the four columns' sums over the LPC lanes: two exchanges halve what a lane holds, then a butterfly
      int mine = 0;                              // the column whose sum this lane ends up with
      float b;
      if (LPC >= 4) {
        const bool up = (l & (LPC / 2)) != 0, up2 = (l & (LPC / 4)) != 0;
        const float r0 = __shfl_xor_sync(0xffffffffu, up ? o[0] : o[2], LPC / 2);
        const float r1 = __shfl_xor_sync(0xffffffffu, up ? o[1] : o[3], LPC / 2);
        const float a0 = (up ? o[2] : o[0]) + r0, a1 = (up ? o[3] : o[1]) + r1;
        const float r2 = __shfl_xor_sync(0xffffffffu, up2 ? a0 : a1, LPC / 4);
        b = (up2 ? a1 : a0) + r2;
        mine = (up ? 2 : 0) + (up2 ? 1 : 0);
#pragma unroll
        for (int w = LPC / 8; w > 0; w >>= 1) b += __shfl_xor_sync(0xffffffffu, b, w);
        if ((l & (LPC / 4 - 1)) == 0 && jb + mine < vdim) out[(size_t)(t0 + tt) * heads * vdim + hv + jb + mine] = b;
      } else {
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          float x = o[cc];
#pragma unroll
          for (int w = LPC >> 1; w > 0; w >>= 1) x += __shfl_xor_sync(0xffffffffu, x, w);
          if (l == 0 && jb + cc < vdim) out[(size_t)(t0 + tt) * heads * vdim + hv + jb + cc] = x;
        }
      }
    }
    if constexpr (SPLIT) {
      if (t0 + kRing * CHUNK < t_end) named_arrive(kRing + 1 + place);
      place = place + 1 == kRing ? 0 : place + 1;
    }
  }
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc) {
    const bool col_ok = jb + cc < vdim;
    float* sp = S_g + (size_t)(col_ok ? jb + cc : 0) * dim;
#pragma unroll
    for (int i = 0; i < DPT; i += 4) {
      const int c = l * DPT + i;
      if (vec_state) {
        if (col_ok && c < dim)
          *reinterpret_cast<ulonglong2*>(sp + i) = make_ulonglong2(S[cc][i / 2], S[cc][i / 2 + 1]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (col_ok && c + e < dim) sp[i + e] = e & 1 ? high2(S[cc][(i + e) / 2]) : low2(S[cc][(i + e) / 2]);
      }
    }
  }
}

__device__ __forceinline__ void store4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, float a, float b, float c, float d) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// VEC4: four numbers a lane and access.  ONE: a head fits in one round of them (vdim up to 128): its gate and weights are asked for beside it and
// nothing is read twice.  Bound by instructions (exponentials, divisions, the warp's sum): 1,999 tokens of
// 32 heads of 128 22.8 us (24.9 in two rounds with a division of 64-bit numbers), 2,048 of 16 12.6 (14.7).
template <typename T, bool VEC4, bool ONE>
__global__ void gla_out_kernel(const float* __restrict__ o, const T* __restrict__ gate, int gate_stride,
                               const float* __restrict__ weight, float eps, float scale, T* __restrict__ out,
                               int out_stride, int heads, int vdim, long long units, int sigmoid_gate, int weight_stride) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= units) return;
  // a division of 64-bit numbers costs as much as the head's sum
  const long long t = (units >> 32) ? unit / heads : (long long)((unsigned)unit / (unsigned)heads);
  const int h = (int)(unit - t * heads);
  const float* src = o + ((size_t)t * heads + h) * vdim;
  if (weight) weight += (size_t)h * weight_stride;
  float ss = 0.f;
  if constexpr (ONE) {
    const int e = lane * 4;
    const bool on = e < vdim;
    const T* gp = gate + (size_t)t * gate_stride + (size_t)h * vdim;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), w = make_float4(1.f, 1.f, 1.f, 1.f), g = x;
    if (on) {
      x = *reinterpret_cast<const float4*>(src + e);
      if (gate) g = widen4(load_raw4(gp + e));
      if (weight) w = *reinterpret_cast<const float4*>(weight + e);
    }
    ss = warp_sum((x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w));
    const float inv = 1.0f / sqrtf(ss / (float)vdim + eps);
    if (!on) return;
    float y[4] = {x.x * inv, x.y * inv, x.z * inv, x.w * inv};
    if (weight) y[0] *= w.x, y[1] *= w.y, y[2] *= w.z, y[3] *= w.w;
    if (gate) {
      const float gs[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] *= (sigmoid_gate ? 1.0f : gs[i]) / (1.0f + expf(-gs[i]));
    }
    store4(out + (size_t)t * out_stride + (size_t)h * vdim + e, y[0] * scale, y[1] * scale, y[2] * scale, y[3] * scale);
  } else if constexpr (VEC4) {                   // vdim a multiple of 4, rows on 16-byte (8-byte for bfloat16) boundaries
    const T* gp = gate ? gate + (size_t)t * gate_stride + (size_t)h * vdim : nullptr;
    T* op = out + (size_t)t * out_stride + (size_t)h * vdim;
    for (int e = lane * 4; e < vdim; e += 128) {
      const float4 x = *reinterpret_cast<const float4*>(src + e);
      ss += (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w);
    }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)vdim + eps);
    for (int e = lane * 4; e < vdim; e += 128) {
      const float4 x = *reinterpret_cast<const float4*>(src + e);
      float y[4] = {x.x * inv, x.y * inv, x.z * inv, x.w * inv};
      if (weight) {
        const float4 w = *reinterpret_cast<const float4*>(weight + e);
        y[0] *= w.x, y[1] *= w.y, y[2] *= w.z, y[3] *= w.w;
      }
      if (gp) {
        const float4 g = widen4(load_raw4(gp + e));
        if (sigmoid_gate) {
          y[0] *= 1.0f / (1.0f + expf(-g.x)), y[1] *= 1.0f / (1.0f + expf(-g.y));
          y[2] *= 1.0f / (1.0f + expf(-g.z)), y[3] *= 1.0f / (1.0f + expf(-g.w));
        } else {
          y[0] *= g.x / (1.0f + expf(-g.x)), y[1] *= g.y / (1.0f + expf(-g.y));
          y[2] *= g.z / (1.0f + expf(-g.z)), y[3] *= g.w / (1.0f + expf(-g.w));
        }
      }
      store4(op + e, y[0] * scale, y[1] * scale, y[2] * scale, y[3] * scale);
    }
  } else {
    for (int e = lane; e < vdim; e += 32) ss += src[e] * src[e];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)vdim + eps);
    for (int e = lane; e < vdim; e += 32) {
      float y = src[e] * inv;
      if (weight) y *= weight[e];
      if (gate) {
        const float g = to_f32(gate[(size_t)t * gate_stride + (size_t)h * vdim + e]);
        y *= (sigmoid_gate ? 1.0f : g) / (1.0f + expf(-g));
      }
      out[(size_t)t * out_stride + (size_t)h * vdim + e] = from_f32<T>(y * scale);
    }
  }
}

ARLE_API int arle_gla_decay(const void* low, int dtype, int low_stride, const float* w2t, const float* bias, float tau,
                            float* alpha, int num_tokens, int channels, int rank, int double_exp, cudaStream_t s) {
  if (num_tokens <= 0) return 0;
  if (channels <= 0 || rank <= 0 || !(tau > 0.f) || rank > 1024) return ARLE_E_BADARG;
  const int threads = 256;
  dim3 grid((num_tokens + kDecayTokens - 1) / kDecayTokens, (channels + threads - 1) / threads);
  if (grid.y > 65535) return ARLE_E_UNSUPPORTED;
  const size_t smem = (size_t)kDecayTokens * rank * sizeof(float);
  if (smem > 40 * 1024) {
    for (auto k : {(const void*)gla_decay_kernel<float, false>, (const void*)gla_decay_kernel<float, true>,
                   (const void*)gla_decay_kernel<__nv_bfloat16, false>, (const void*)gla_decay_kernel<__nv_bfloat16, true>}) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return (int)e;
    }
  }
  if (dtype == 0)
    launch_kernel(double_exp ? gla_decay_kernel<float, true> : gla_decay_kernel<float, false>, grid, dim3(threads), smem, s, 1, (const float*)low,
                  low_stride, w2t, bias, 1.0f / tau, alpha, num_tokens, channels, rank);
  else if (dtype == 1)
    launch_kernel(double_exp ? gla_decay_kernel<__nv_bfloat16, true> : gla_decay_kernel<__nv_bfloat16, false>, grid, dim3(threads), smem, s, 1,
                  (const __nv_bfloat16*)low, low_stride, w2t, bias, 1.0f / tau, alpha, num_tokens, channels, rank);
  else
    return ARLE_E_BADARG;
  return launch_status();
}

namespace {

// Loaders beside the memory's warps, while no SM has more than two such blocks.  Without them bringing the chunks and the barriers around that are
// 60 of 213 us.  16 heads of 128 x 128, us, without and with: one row of 2,048 tokens (128 blocks) 213.5 and 189.8, of 512 57.9 and 51.8, 32 heads,
// 1,024 tokens (256 blocks) 153.7 and 149.8; but three rows of 600 to 748 (384 blocks, three an SM without) 156.1 and 169.4, 16 rows of 13 25.1
// and 29.1.
inline bool takes_loaders(dim3 grid) { return (long long)grid.x * grid.y * grid.z <= 296; }

template <typename T, int DPT, int LPC>
int scan_launch(const void* q, const void* k, const void* v, int in_stride, const float* alpha, const float* bonus, float* state, long slot_stride, const int* q_indptr,
                const int* state_slots, float* out, int rows, int heads, int dim, int vdim, float q_scale, int max_q_len, cudaStream_t s) {
  constexpr int COLS = kScanThreads / LPC * kScanCpt;
  dim3 grid((vdim + COLS - 1) / COLS, heads, rows);
  const size_t eb = sizeof(T) * 4;               // bytes of four elements of q or k
  const bool vec = dim % 4 == 0 && in_stride % 4 == 0 && ((uintptr_t)q % eb) == 0 && ((uintptr_t)k % eb) == 0 &&
                   ((uintptr_t)alpha % 16) == 0;
  auto run = [&](auto kernel, int threads) {
    launch_kernel(kernel, grid, dim3(threads), 0, s, 1, (const T*)q, (const T*)k, (const T*)v, in_stride, alpha, bonus, state, slot_stride, q_indptr,
                  state_slots, out, heads, dim, vdim, q_scale);
    return launch_status();
  };
#define ARLE_FORM(LONG, SPLIT)                                                                                                    \
  return bonus ? (vec ? run(gla_scan_kernel<T, DPT, LPC, true, true, LONG, SPLIT>, SPLIT ? 2 * kScanThreads : kScanThreads)       \
                      : run(gla_scan_kernel<T, DPT, LPC, false, true, LONG, SPLIT>, SPLIT ? 2 * kScanThreads : kScanThreads))     \
               : (vec ? run(gla_scan_kernel<T, DPT, LPC, true, false, LONG, SPLIT>, SPLIT ? 2 * kScanThreads : kScanThreads)      \
                      : run(gla_scan_kernel<T, DPT, LPC, false, false, LONG, SPLIT>, SPLIT ? 2 * kScanThreads : kScanThreads))
  if (max_q_len < 8) ARLE_FORM(false, false);
  if constexpr (LPC == 32 && DPT == 4) {
    if (takes_loaders(grid)) ARLE_FORM(true, true);
  }
  ARLE_FORM(true, false);
#undef ARLE_FORM
}

// The split of the key channels among threads depends on dim alone, so the order of a token's sums does too: four
// channels a thread up to 128 channels (as many lanes as that takes, a power of two), then 8 and 16 on 32 lanes.
template <typename T>
int scan_dispatch(const void* q, const void* k, const void* v, int in_stride, const float* alpha, const float* bonus, float* state,
                  long slot_stride, const int* q_indptr, const int* state_slots, float* out, int rows, int heads, int dim, int vdim, float q_scale,
                  int max_q_len, cudaStream_t s) {
#define ARLE_SCAN(D, L) \
  return scan_launch<T, D, L>(q, k, v, in_stride, alpha, bonus, state, slot_stride, q_indptr, state_slots, out, rows, heads, dim, vdim, q_scale, max_q_len, s)
  if (dim <= 4) ARLE_SCAN(4, 1);
  if (dim <= 8) ARLE_SCAN(4, 2);
  if (dim <= 16) ARLE_SCAN(4, 4);
  if (dim <= 32) ARLE_SCAN(4, 8);
  if (dim <= 64) ARLE_SCAN(4, 16);
  if (dim <= 128) ARLE_SCAN(4, 32);
  if (dim <= 256) ARLE_SCAN(8, 32);
  if (dim <= 512) ARLE_SCAN(16, 32);
#undef ARLE_SCAN
  return ARLE_E_UNSUPPORTED;
}

}  // namespace

ARLE_API int arle_gla_scan(const void* q, const void* k, const void* v, int dtype, int in_stride, const float* alpha, const float* bonus,
                           float* state, long slot_stride, const int* q_indptr, const int* state_slots, float* out, int rows, int heads,
                           int dim, int vdim, float q_scale, int max_q_len, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (heads <= 0 || dim <= 0 || vdim <= 0 || max_q_len <= 0 || slot_stride < (long)heads * vdim * dim) return ARLE_E_BADARG;
  if (dim > 512 || heads > 65535 || rows > 65535) return ARLE_E_UNSUPPORTED;
  if (dtype == 0)
    return scan_dispatch<float>(q, k, v, in_stride, alpha, bonus, state, slot_stride, q_indptr, state_slots, out, rows, heads, dim, vdim, q_scale, max_q_len, s);
  if (dtype == 1)
    return scan_dispatch<__nv_bfloat16>(q, k, v, in_stride, alpha, bonus, state, slot_stride, q_indptr, state_slots, out, rows, heads, dim, vdim, q_scale, max_q_len, s);
  return ARLE_E_BADARG;
}

ARLE_API int arle_gla_out(const float* o, const void* gate, int dtype, int gate_stride, const float* weight, float eps,
                          float scale, void* out, int out_stride, int num_tokens, int heads, int vdim, int sigmoid_gate, int weight_stride, cudaStream_t s) {
  if (num_tokens <= 0) return 0;
  if (heads <= 0 || vdim <= 0) return ARLE_E_BADARG;
  const long long units = (long long)num_tokens * heads;
  const int warps = 8;
  const long long blocks = (units + warps - 1) / warps;
  if (blocks > 0x7fffffffLL) return ARLE_E_UNSUPPORTED;
  const size_t eb = dtype == 0 ? 16 : 8;         // bytes of four elements of gate and out
  const bool vec = vdim % 4 == 0 && gate_stride % 4 == 0 && out_stride % 4 == 0 && ((uintptr_t)o % 16) == 0 &&
                   ((uintptr_t)gate % eb) == 0 && ((uintptr_t)out % eb) == 0 && ((uintptr_t)weight % 16) == 0 && weight_stride % 4 == 0;
  if (dtype == 0) {
    auto kern = vec && vdim <= 128 ? gla_out_kernel<float, true, true> : vec ? gla_out_kernel<float, true, false> : gla_out_kernel<float, false, false>;
    launch_kernel(kern, dim3((unsigned)blocks), dim3(warps * 32), 0, s, 1, o, (const float*)gate, gate_stride, weight, eps, scale,
                  (float*)out, out_stride, heads, vdim, units, sigmoid_gate, weight_stride);
  } else if (dtype == 1) {
    auto kern = vec && vdim <= 128 ? gla_out_kernel<__nv_bfloat16, true, true>
                : vec ? gla_out_kernel<__nv_bfloat16, true, false> : gla_out_kernel<__nv_bfloat16, false, false>;
    launch_kernel(kern, dim3((unsigned)blocks), dim3(warps * 32), 0, s, 1, o, (const __nv_bfloat16*)gate, gate_stride, weight, eps,
                  scale, (__nv_bfloat16*)out, out_stride, heads, vdim, units, sigmoid_gate, weight_stride);
  } else {
    return ARLE_E_BADARG;
  }
  return launch_status();
}
