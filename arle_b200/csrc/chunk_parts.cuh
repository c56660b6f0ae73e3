// What the recurrences in chunks of 64 tokens on the tensor cores share: a row's chunks, float32 numbers as three bfloat16 ones, and products
// whose sums are rounded as float32 sums are.
#pragma once
#include "mma_utils.cuh"

namespace arle {

constexpr int kC = 64;                                     // tokens of a chunk
constexpr int kTileWords = 3 * 32 * 4;                     // a tile of 16 x 16 in three parts, as the tensor cores take it: [part][lane][4]

__device__ __forceinline__ int row_chunks(int n, int longest) { return n > longest ? (n + kC - 1) / kC : 0; }

// The row and the chunk of a slot (a warp's lanes together); false: no such slot.
__device__ __forceinline__ bool chunk_of(int slot, const int* q_indptr, int rows, int longest, int& row, int& chunk) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int r0 = 0; r0 < rows; r0 += 32) {
    const int mine = r0 + lane < rows ? row_chunks(q_indptr[r0 + lane + 1] - q_indptr[r0 + lane], longest) : 0;
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, slot < before + sum);
    if (hit) {
      const int src = __ffs(hit) - 1;
      row = r0 + src;
      chunk = slot - before - __shfl_sync(0xffffffffu, sum - mine, src);
      return true;
    }
    before += __shfl_sync(0xffffffffu, sum, 31);
  }
  return false;
}

// x = hi + mid + lo to 24 bits; an infinity stays one (hi alone).
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  float rx = x - __low2float(h), ry = y - __high2float(h);
  rx = fabsf(rx) <= fabsf(x) ? rx : 0.f;
  ry = fabsf(ry) <= fabsf(y) ? ry : 0.f;
  const __nv_bfloat162 m = __floats2bfloat162_rn(rx, ry);
  const __nv_bfloat162 l = __floats2bfloat162_rn(rx - __low2float(m), ry - __high2float(m));
  hi = *reinterpret_cast<const uint32_t*>(&h);
  mid = *reinterpret_cast<const uint32_t*>(&m);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// acc += a . b with the sum of the sixteen products rounded once on its own: the tensor core cuts off what an accumulator cannot hold, and
// over a chain of products that is a few times the error of a float32 sum.
__device__ __forceinline__ void mma_add(float (&acc)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mma_bf16(t, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] += t[i];
}

// A lane's numbers of a tile, (row g, columns 2t, 2t+1), (g+8, same), (g, 2t+8, 2t+9), (g+8, same), into memory.
__device__ __forceinline__ void split_tile(const float (&w)[8], uint32_t* to, int lane) {
  uint32_t p[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split3(w[2 * i], w[2 * i + 1], p[0][i], p[1][i], p[2][i]);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(to + (i * 32 + lane) * 4) = make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
}

// What the products of a tile of 16 weights (in three parts, as the tensor cores take them) with its values come to, row i of the tile
// with the values up to i alone.  v: the tile's first value in this lane's first column of o0; o1's columns are eight further on.
template <int VP>
__device__ __forceinline__ void add_seen(const uint32_t (&pa)[3][4], const __nv_bfloat16* v, int lane, float (&o0)[4], float (&o1)[4]) {
  const int row = lane >> 2;
#pragma unroll
  for (int reg = 0; reg < 4; ++reg) {                      // rows 0 .. 7 and 8 .. 15 of the weights in turn, keys 8 (reg / 2) ..
    float w[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 2; i >= 0; --i) {
      const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&pa[i][reg]);
      w[0] += __low2float(x), w[1] += __high2float(x);
    }
    const int half = reg & 1;
#pragma unroll 1
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float wj = __shfl_sync(0xffffffffu, w[e], (lane & ~3) | s);
        const int j = (reg >> 1) * 8 + 2 * s + e;
        if (j > row + 8 * half) continue;
        const __nv_bfloat16* x = v + j * VP;
        o0[2 * half] = fmaf(wj, __bfloat162float(x[0]), o0[2 * half]);
        o0[2 * half + 1] = fmaf(wj, __bfloat162float(x[1]), o0[2 * half + 1]);
        o1[2 * half] = fmaf(wj, __bfloat162float(x[8]), o1[2 * half]);
        o1[2 * half + 1] = fmaf(wj, __bfloat162float(x[9]), o1[2 * half + 1]);
      }
  }
}

}  // namespace arle
