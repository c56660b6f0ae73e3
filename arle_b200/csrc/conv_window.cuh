// A causal convolution of four taps per channel over the tokens of every row, several tokens a thread: the four inputs of a token
// slide through registers, so a row of x is read once (and the three before a thread's first token once more) instead of four times,
// VEC channels an access.  Sums in the order of the kernels that take a token a thread (causal_conv, conv_silu): the same bits.
// What bounds it: instructions, the exponentials and divisions of silu above all (37 an element, and a division has a branch of its own, so that
// the next one waits); memory is at a third of its rate.  Four channels a thread leave room for six blocks an SM: 2,048 tokens of 10,240
// channels, bfloat16, 84 MB 37.2 us in a graph, 1,999 tokens of 8,192 30.0, 300 of 2,304 10.0 (eight channels a thread and three blocks an SM, five
// blocks, two channels, 32 tokens a thread: all slower; eight blocks spill).  The fast exponential and division, 26.5 us, are
// not taken: they round to another bfloat16 in one of 1,000 places; in front of a look at whether they could, with the full ones behind it, 34 us, but 55
// where numbers are large.
#pragma once
#include "common.cuh"

namespace arle {

constexpr int kConvTokens = 16, kConvAhead = 4, kConvThreads = 128, kConvVec = 4;

// in_bias is added to a row's inputs (not to what the state holds); act 1: silu.
template <typename TI, typename TO, int VEC>
__global__ void __launch_bounds__(kConvThreads, sizeof(TI) + sizeof(TO) == 4 ? 6 : 5)
    conv_window_kernel(const TI* __restrict__ x, int x_stride, const float* __restrict__ in_bias, const float* __restrict__ w,
                       const float* __restrict__ out_bias, int act, const float* __restrict__ state, long slot_stride, long conv_off,
                       const int* __restrict__ q_indptr, const int* __restrict__ row_of_token, const int* __restrict__ state_slots,
                       TO* __restrict__ out, int out_stride, int T, int C) {
  pdl_launch_dependents();
  pdl_wait();
  const int c = (blockIdx.x * kConvThreads + threadIdx.x) * VEC;
  if (c >= C) return;
  const int t0 = blockIdx.y * kConvTokens, t1 = min(T, t0 + kConvTokens);
  float wt[4][VEC], ib[VEC], ob[VEC], win[3][VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    const float4 f = *reinterpret_cast<const float4*>(w + (size_t)(c + i) * 4);
    wt[0][i] = f.x, wt[1][i] = f.y, wt[2][i] = f.z, wt[3][i] = f.w;
    ib[i] = in_bias ? in_bias[c + i] : 0.f;
    ob[i] = out_bias ? out_bias[c + i] : 0.f;
  }
  // the three inputs before token t of row r
  auto fill = [&](int r, int t) {
    const int local = t - q_indptr[r];
    const float* st = state + (size_t)state_slots[r] * slot_stride + conv_off + (size_t)c * 3;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (local - 3 + j >= 0) {
        load_vec<TI, VEC>(x + (size_t)(t - 3 + j) * x_stride + c, win[j]);
#pragma unroll
        for (int i = 0; i < VEC; ++i) win[j][i] += ib[i];
      } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) win[j][i] = st[i * 3 + local + j];
      }
    }
  };
  int r = row_of_token[t0], next = q_indptr[r + 1];        // the first token of the row behind
  fill(r, t0);
  for (int tb = t0; tb < t1; tb += kConvAhead) {
    Pack<TI, VEC> ahead[kConvAhead];
#pragma unroll
    for (int g = 0; g < kConvAhead; ++g)
      if (tb + g < t1) ahead[g] = *reinterpret_cast<const Pack<TI, VEC>*>(x + (size_t)(tb + g) * x_stride + c);
#pragma unroll
    for (int g = 0; g < kConvAhead; ++g) {
      const int t = tb + g;
      if (t >= t1) break;
      if (t >= next) {
        r = row_of_token[t];
        next = q_indptr[r + 1];
        fill(r, t);
      }
      float y[VEC];
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const float in = to_f32(ahead[g].e[i]) + ib[i];
        float acc = fmaf(wt[0][i], win[0][i], ob[i]);
        acc = fmaf(wt[1][i], win[1][i], acc);
        acc = fmaf(wt[2][i], win[2][i], acc);
        acc = fmaf(wt[3][i], in, acc);
        win[0][i] = win[1][i];
        win[1][i] = win[2][i];
        win[2][i] = in;
        y[i] = act == 1 ? acc / (1.0f + expf(-acc)) : acc;
      }
      store_vec<TO, VEC>(out + (size_t)t * out_stride + c, y);
    }
  }
}

// Whether it takes these arrays: four taps, several tokens a row, channels in whole groups on their boundaries.
template <typename TI, typename TO>
inline bool conv_window_takes(const void* x, int x_stride, const float* w, const void* out, int out_stride, int T, int R, int C, int taps) {
  constexpr int VEC = kConvVec;
  return taps == 4 && T >= 4 * R && T >= 32 && C % VEC == 0 && x_stride % VEC == 0 && out_stride % VEC == 0 && vec_aligned<VEC>(x, sizeof(TI)) &&
         vec_aligned<VEC>(out, sizeof(TO)) && ((uintptr_t)w & 15) == 0 && (T + kConvTokens - 1) / kConvTokens <= 65535;
}

template <typename TI, typename TO>
inline void launch_conv_window(const void* x, int x_stride, const float* in_bias, const float* w, const float* out_bias, int act, const float* state,
                               long slot_stride, long conv_off, const int* q_indptr, const int* row_of_token, const int* state_slots, void* out,
                               int out_stride, int T, int C, cudaStream_t s) {
  constexpr int VEC = kConvVec;
  const dim3 grid((C / VEC + kConvThreads - 1) / kConvThreads, (T + kConvTokens - 1) / kConvTokens);
  launch_kernel(conv_window_kernel<TI, TO, VEC>, grid, dim3(kConvThreads), 0, s, 1, (const TI*)x, x_stride, in_bias, w, out_bias, act, state,
                slot_stride, conv_off, q_indptr, row_of_token, state_slots, (TO*)out, out_stride, T, C);
}

}  // namespace arle
