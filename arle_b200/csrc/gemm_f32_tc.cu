// float32 rows times a bfloat16 W on the tensor cores, without giving up 32 bits:
//     C[M, N] = A[M, K] (float32) . W[N, K]^T (bfloat16)
//
// A number of A is cut into three bfloat16 pieces of eight bits each (cut off, not rounded: none overflows, and the three add up to it
// exactly from 2^-110 on; below that the last piece ends at bfloat16's smallest number, 2^-133, so that a number keeps fewer than 24 bits: off by
// less than 2^-133), so A . W is three products of bfloat16 numbers, each exact in float32.  What is left to chance is the sums.  The
// tensor cores add into their accumulator without rounding to nearest, so a long sum there drifts towards zero; here an accumulator in
// TMEM holds 64 numbers of k of one piece only, and float32 registers add up the three pieces' sums, the smallest first, and those of the
// blocks, k ascending, rounded to nearest.  Off from float64 by 1.2e-7 to 2.8e-7 of the result's norm at K of 1,024 to 12,288, where
// FFMAs in order are by 5.1e-7 to 2.1e-6.
//
// The order of an element's sums depends on K alone, whatever M is and whichever tile it falls into, so a token's bits do not depend on
// how its prompt was cut or on what stands beside it.
//
// Persistent CTAs walk tiles of 128 rows of W (the MMA's rows) by BN rows of A (three times BN columns of an MMA, a column for each
// piece).  Roles by warp:
//   sums    : four warps.  Warp i owns TMEM lanes 32 i .. 32 i + 31, a column of C a thread; adds up the blocks' sums of BN rows in
//             registers, stores them (lanes: neighbouring columns).
//   cutters : eight warps (four, ten).  Groups of BN / 16 warps take turns at the blocks: cut 64 numbers of k of the BN rows and lay the
//             three tiles down as the MMA reads them (128-byte swizzle).
//   loader  : one lane, W's tile and the rows of A by TMA.
//   issuer  : one lane, four MMAs a block; its warp owns the TMEM.
// NaN: a piece that is zero times an infinite W is NaN where the number itself times it is infinite.  A sum that comes out as NaN is
// formed once more from the numbers themselves, k ascending, until it is NaN there too.
// Every wait is bounded; when one runs out the error flag is raised and the CTA leaves with its copies landed, its MMAs done and its TMEM freed.
//
// What bounds it: few rows, the issuer (some 600 cycles a block of its looks at barriers, MMAs and commit; three commits a block, a barrier
// for each who waits, took 900); many rows, the chain of a block through cutters, MMAs and sums, with two accumulators (301 rows of 6,144 x 1,024:
// 1,000 cycles a block of 64 rows, issue slots 45 % used, tensor pipe and shared memory 18 % each).
// Rows of A fetched by the cutters' own loads: each proxy fence waited for them, 950 cycles a block.  All cutters at one block at a time:
// 1,400 cycles a block of 64 rows instead of 1,000.
// Measured (us, the FFMA kernels and this one): 301 rows, 6,144 x 1,024 117 and 26; 4,096 x 1,024 87 and 18; 1,024 x 2,048 62 and 17; 1,024 x
// 3,072 91 and 24; 1,024 rows of 24,576 x 4,096 4,420 and 805 (256 TFLOP/s); 16 rows of 1,024 x 3,072 84 and 19; four rows of 256 to 4,096 x 1,024 13.0 and
// 8.9, of 512 7.3 and 6.2.  One row is done sooner by FFMAs where K is short (256 to 4,096 x 512 4.7 and 6.2, x 1,024 8.0 and 8.9, x 2,048 14.6 and 14.0,
// x 4,096 27.9 and 24.3, x 12,288 80 and 66; 151,936 x 1,024 57.6 and 58.1), but a row's order of sums may not depend on how many there are; steps of one
// row are no slower as a whole (28 layers of 0.6B sizes 2,811 and 2,687, 8 layers of a hidden size of 512 583 and 584).
#include "common.cuh"
#include "tcgen05_utils.cuh"
using namespace arle;

namespace {

constexpr int kRowsW = 128, kBK = 64;
constexpr int kSumWarps = 4;

template <int BN, int CTAS>                                // CTAS: a SM
struct Layout {
  // What TMA brings (W's tile, then the rows of A as they are) and, in a ring of their own, the pieces.
  static constexpr uint32_t W = kRowsW * kBK * 2, RAW = BN * kBK * 4, STAGE = W + RAW, PIECE = BN * kBK * 2;
  static constexpr int PIECE_WARPS = CTAS == 2 ? 4 : BN == 80 ? 10 : 8, LOAD_WARP = kSumWarps + PIECE_WARPS, MMA_WARP = LOAD_WARP + 1, THREADS = (MMA_WARP + 1) * 32;
  static constexpr int GROUP = BN / 16, GROUPS = PIECE_WARPS / GROUP;      // warps that cut a block together, blocks cut side by side
  static constexpr int STAGES = BN >= 64 || CTAS == 2 ? 4 : BN == 32 ? 6 : 8, RING = BN == 80 ? 2 : BN == 64 ? 3 : BN == 32 ? 5 : STAGES;
  static_assert(RING >= GROUPS, "a group's next block has a place of its own");
  static constexpr size_t SMEM = (size_t)STAGES * STAGE + (size_t)RING * 3 * PIECE + 1024;
  static constexpr int COLS = 3 * BN, BUFFERS = BN >= 64 ? 2 : 4;      // accumulators in TMEM: a column for each piece of each row
  static constexpr uint32_t TMEM = BN == 16 ? 256 : 512;
  static_assert(COLS * BUFFERS <= (int)TMEM && CTAS * (SMEM + 2048) <= 228 * 1024, "TMEM, shared memory");
};

// Whether a phase is over, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(b));
  return a;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ unsigned long long pair(uint32_t lo, uint32_t hi) { return (unsigned long long)hi << 32 | lo; }

// The three pieces of two numbers, as pairs of bfloat16 (the first number in the low half), and what is left behind the first pieces
// added to `rest`, which infinities and NaNs turn into NaN.
__device__ __forceinline__ void cut(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2, float& rest) {
  const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
  const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
  const uint32_t va = __float_as_uint(ra), vb = __float_as_uint(rb);
  p0 = __byte_perm(ua, ub, 0x7632);
  p1 = __byte_perm(va, vb, 0x7632);
  p2 = __byte_perm(__float_as_uint(ra - __uint_as_float(va & 0xffff0000u)), __float_as_uint(rb - __uint_as_float(vb & 0xffff0000u)), 0x7632);
  rest += ra + rb;
}
// An infinity or a NaN is its own first piece, the others are zero.
__device__ __forceinline__ void cut_odd(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  if (!(fabsf(a) < INFINITY)) {
    p0 = (p0 & 0xffff0000u) | (a != a ? 0x7fffu : __float_as_uint(a) >> 16);
    p1 &= 0xffff0000u;
    p2 &= 0xffff0000u;
  }
  if (!(fabsf(b) < INFINITY)) {
    p0 = (p0 & 0xffffu) | (b != b ? 0x7fff0000u : __float_as_uint(b));
    p1 &= 0xffffu;
    p2 &= 0xffffu;
  }
}

template <int BN, int CTAS>
__global__ void __launch_bounds__(Layout<BN, CTAS>::THREADS, CTAS) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                 const __grid_constant__ CUtensorMap map_a, const float* __restrict__ A,
                                                                 int lda, const __nv_bfloat16* __restrict__ W, int ldw,
                                                                 float* __restrict__ C, int ldc, int M, int N, int K, int* __restrict__ err) {
  pdl_launch_dependents();
  pdl_wait();
  typedef Layout<BN, CTAS> L;
  constexpr int STAGES = L::STAGES, RING = L::RING;
  constexpr int kBuffers = L::BUFFERS;
  constexpr uint32_t kTmemCols = L::TMEM;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* pieces = tiles + (size_t)STAGES * L::STAGE;
  __shared__ __align__(8) uint64_t full_bar[STAGES], done_bar[STAGES], cut_full[RING], acc_empty[kBuffers];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag, loaded;                        // loaded: blocks whose copies have been issued
  __shared__ __align__(8) uint64_t last_bar;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (M + BN - 1) / BN, num_tiles = tiles_m * ((N + kRowsW - 1) / kRowsW);      // rows of A fastest: W's tile stays in L2
  const int kblocks = K / kBK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_addr(&full_bar[s]), 1);
      mbar_init(smem_addr(&done_bar[s]), 1);
    }
    for (int p = 0; p < RING; ++p) mbar_init(smem_addr(&cut_full[p]), L::GROUP);
    for (int b = 0; b < kBuffers; ++b) mbar_init(smem_addr(&acc_empty[b]), kSumWarps);
    mbar_init(smem_addr(&last_bar), 1);
    abort_flag = loaded = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == L::MMA_WARP) {
    tmem_alloc(smem_addr(&tmem_base_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const volatile int* aborted = &abort_flag;
  // Block i's products are finished: its stage, its pieces' place and its sums are free to take.  One barrier serves all who wait for it.
  // A wait tells a phase from its neighbours only, so whoever waits for block i knows that block i - STAGES is done (the loader and the
  // sums' warps waited for every block before it; a group of cutters for block i - GROUPS at the latest) and keeps block i + STAGES from
  // being issued before it has looked.
  static_assert(STAGES >= RING && STAGES >= kBuffers && STAGES >= L::GROUPS, "phases");
  auto done = [&](int i) { return mbar_wait_bounded(smem_addr(&done_bar[i % STAGES]), (i / STAGES) & 1, aborted); };

  if (warp == L::LOAD_WARP) {
    if (lane == 0) {
      int issued = 0;
      for (int t = blockIdx.x; t < num_tiles && !*aborted; t += gridDim.x) {
        const int m0 = t % tiles_m * BN, n0 = t / tiles_m * kRowsW;
        for (int kb = 0; kb < kblocks; ++kb, ++issued) {
          const int s = issued % STAGES;
          if (issued >= STAGES && !done(issued - STAGES)) {
            abort_flag = 1;
            break;
          }
          const uint32_t bar = smem_addr(&full_bar[s]), dst = smem_addr(tiles + (size_t)s * L::STAGE);
          mbar_expect_tx(bar, L::STAGE);
          tma_load_2d(dst + L::W, &map_a, kb * kBK, m0, bar);
          tma_load_2d(dst, &map_w, kb * kBK, n0, bar);
        }
      }
      loaded = issued;
    }
  } else if (warp == L::MMA_WARP) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16(kRowsW, L::COLS);
      int i = 0;
      bool ready = false;
      for (int t = blockIdx.x; t < num_tiles && !*aborted; t += gridDim.x)
        for (int kb = 0; kb < kblocks; ++kb, ++i) {
          const int s = i % STAGES, p = i % RING, buf = i % kBuffers;
          // The cutters have waited for the stage, so the pieces being there says that W's tile is there too.  A look at a barrier takes
          // some 100 cycles: the two go out together, ahead of the commit of the block before.
          if (!ready && (!mbar_wait_bounded(smem_addr(&acc_empty[buf]), ((i / kBuffers) & 1) ^ 1, aborted) ||
                         !mbar_wait_bounded(smem_addr(&cut_full[p]), (i / RING) & 1, aborted))) {
            abort_flag = 1;
            break;
          }
          tc_fence_after();
          const uint64_t wdesc = smem_desc_sw128(smem_addr(tiles + (size_t)s * L::STAGE));
          const uint64_t xdesc = smem_desc_sw128(smem_addr(pieces + (size_t)p * 3 * L::PIECE));
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            umma_bf16(tmem_base + (uint32_t)(buf * L::COLS), wdesc + 2 * k, xdesc + 2 * k, idesc, k != 0 ? 1u : 0u);
          const int next = i + 1;
          const bool sums = mbar_test(smem_addr(&acc_empty[next % kBuffers]), ((next / kBuffers) & 1) ^ 1);
          const bool cuts = mbar_test(smem_addr(&cut_full[next % RING]), (next / RING) & 1);
          umma_commit(smem_addr(&done_bar[s]));
          ready = sums && cuts;
        }
    }
  } else if (warp >= kSumWarps) {
    // Eight numbers of k a thread and unit: 16 bytes of each piece.
    constexpr int PER = 4, THREADS = L::GROUP * 32;
    static_assert(PER * THREADS == BN * 8, "units");
    const int group = (warp - kSumWarps) / L::GROUP, tid = (warp - kSumWarps) % L::GROUP * 32 + lane;
    const int my_tiles = (num_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, total = my_tiles * kblocks;
    for (int i = group; i < total; i += L::GROUPS) {
      const int s = i % STAGES, p = i % RING;
      // The place of the pieces first: block i - RING being done says that block i - STAGES is, whose phase of the stage's barrier, were it
      // still open, would look like block i's being over (the group that cut it may be another one).
      const bool ok = (i < RING || done(i - RING)) && mbar_wait_bounded(smem_addr(&full_bar[s]), (i / STAGES) & 1, aborted);
      if (!__all_sync(0xffffffffu, ok)) {
        abort_flag = 1;
        break;
      }
      const unsigned char* raw = tiles + (size_t)s * L::STAGE + L::W;
      unsigned char* dst = pieces + (size_t)p * 3 * L::PIECE;
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int idx = tid + u * THREADS, row = idx >> 3, c = idx & 7;
        // A unit's two halves: lanes 4-7 of eight read theirs the other way round, so that the eight reads fall on different banks.
        const int turn = lane & 4;
        const float4 x = *reinterpret_cast<const float4*>(raw + idx * 32 + turn * 4), y = *reinterpret_cast<const float4*>(raw + idx * 32 + 16 - turn * 4);
        const float4 a = turn ? y : x, b = turn ? x : y;
        uint4 p0, p1, p2;
        float rest = 0.f;
        cut(a.x, a.y, p0.x, p1.x, p2.x, rest);
        cut(a.z, a.w, p0.y, p1.y, p2.y, rest);
        cut(b.x, b.y, p0.z, p1.z, p2.z, rest);
        cut(b.z, b.w, p0.w, p1.w, p2.w, rest);
        if (rest != rest) {
          cut_odd(a.x, a.y, p0.x, p1.x, p2.x);
          cut_odd(a.z, a.w, p0.y, p1.y, p2.y);
          cut_odd(b.x, b.y, p0.z, p1.z, p2.z);
          cut_odd(b.z, b.w, p0.w, p1.w, p2.w);
        }
        const int at = row * (kBK * 2) + ((c ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(dst + at) = p0;
        *reinterpret_cast<uint4*>(dst + L::PIECE + at) = p1;
        *reinterpret_cast<uint4*>(dst + 2 * L::PIECE + at) = p2;
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");            // the MMA reads them through the other proxy
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(&cut_full[p])) : "memory");
    }
  } else {
    int i = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const int m0 = t % tiles_m * BN, n = t / tiles_m * kRowsW + warp * 32 + lane;
      unsigned long long acc[BN / 2];                       // two rows' sums each
#pragma unroll
      for (int j = 0; j < BN / 2; ++j) acc[j] = 0;
      for (int kb = 0; kb < kblocks; ++kb, ++i) {
        const int buf = i % kBuffers;
        ok = done(i);
        if (!ok) abort_flag = 1;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t from = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * L::COLS);
#pragma unroll
        for (int c = 0; c < BN; c += 16) {
          uint32_t p0[16], p1[16], p2[16];
          tmem_ld16(from + c, p0);
          tmem_ld16(from + BN + c, p1);
          tmem_ld16(from + 2 * BN + c, p2);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const unsigned long long sum = add2(pair(p0[j], p0[j + 1]), add2(pair(p1[j], p1[j + 1]), pair(p2[j], p2[j + 1])));
            acc[(c + j) / 2] = add2(acc[(c + j) / 2], sum);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(&acc_empty[buf])) : "memory");
      }
      if (ok && n < N) {
        bool odd = false;
        float* dst = C + (size_t)m0 * ldc + n;
#pragma unroll
        for (int j = 0; j < BN; ++j) {
          const float sum = __uint_as_float((uint32_t)(j & 1 ? acc[j / 2] >> 32 : acc[j / 2]));
          if (m0 + j < M) dst[(size_t)j * ldc] = sum;
          odd |= sum != sum;
        }
        if (odd) {
          const __nv_bfloat16* w = W + (size_t)n * ldw;
          for (int j = 0; j < BN && m0 + j < M; ++j) {
            if (dst[(size_t)j * ldc] == dst[(size_t)j * ldc]) continue;
            const float* a = A + (size_t)(m0 + j) * lda;
            float sum = 0.f;
            for (int k = 0; k < K && sum == sum; ++k) sum = fmaf(a[k], __bfloat162float(w[k]), sum);
            dst[(size_t)j * ldc] = sum;
          }
        }
      }
    }
  }
  __syncwarp();                                            // the loader's and the issuer's other lanes have been here all along
  tc_fence_before();
  __syncthreads();
  if (*aborted) {                                          // as all warps have left it: copies and MMAs under way end (bounded) before their memory is given back
    if (warp == L::LOAD_WARP && lane == 0)
      for (int i = max(0, loaded - STAGES); i < loaded; ++i) mbar_wait_plain(smem_addr(&full_bar[i % STAGES]), (i / STAGES) & 1);
    if (warp == L::MMA_WARP && lane == 0) {
      umma_commit(smem_addr(&last_bar));
      mbar_wait_plain(smem_addr(&last_bar), 0);
    }
    __syncthreads();
  }
  if (warp == L::MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0 && abort_flag && err) atomicExch(err, 2);
}

template <int BN, int CTAS>
int launch(const float* A, int lda, const __nv_bfloat16* W, int ldw, float* C, int ldc, int M, int N, int K, int* err, cudaStream_t s) {
  typedef Layout<BN, CTAS> L;
  CUtensorMap mw, ma;
  int rc = tensor_map_2d_bf16(W, N, K, ldw, kRowsW, &mw);
  if (rc == 0) rc = tensor_map_2d_f32(A, M, K, lda, BN, &ma);
  if (rc) return rc;
  auto kern = gemm_f32_tc_kernel<BN, CTAS>;
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)kern, L::SMEM);
  if (raised != cudaSuccess) return (int)raised;
  const long long num_tiles = (long long)((N + kRowsW - 1) / kRowsW) * ((M + BN - 1) / BN), room = 148 * CTAS;
  launch_kernel(kern, dim3((unsigned)(num_tiles < room ? num_tiles : room)), dim3(L::THREADS), L::SMEM, s, 1, mw, ma, A, lda, W, ldw, C, ldc, M,
                N, K, err);
  return launch_status();
}

}  // namespace

// K a multiple of 64; A's rows on 16-byte boundaries, W's too (what its TMA tensor map needs).
ARLE_API int arle_gemm_f32_tc(const float* A, int lda, const void* W, int ldw, float* C, int ldc, int M, int N, int K, int* err, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % kBK || lda % 4 || ldw % 8 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return ARLE_E_UNSUPPORTED;
  if ((long long)((N + kRowsW - 1) / kRowsW) * ((M + 15) / 16) * (K / kBK) > 0x7fffffffll) return ARLE_E_UNSUPPORTED;
  const __nv_bfloat16* w = (const __nv_bfloat16*)W;
  // Rounds of tiles times what a block of 64 numbers of k takes (us): 301 rows of 6,144 x 1,024 43.5, 33.3 and 27.1 us in tiles of 16, 32 and 64
  // rows, of 1,024 x 3,072 37.4, 25.1 and 33.3, 100 rows of 4,096 x 1,024 16.8, 12.7 and 16.9; of 4,096 x 1,024 with 301 rows 27.6 in tiles of 64 (a
  // second round for 12 of 160), 20.0 in tiles of 80 (128), which take longer where both have as many rounds (6,144 x 1,024 33.7).  Two CTAs an SM with half the stages each
  // take more tiles at a time (one row of 24,576 x 4,096 45.5 us, with one CTA 52.5) and longer for one (1,024 x 3,072 25.0, 21.0).
  auto tiles = [&](int bn) { return (long long)((N + kRowsW - 1) / kRowsW) * ((M + bn - 1) / bn); };
  auto rounds = [](long long t, int at_once) { return (float)((t + at_once - 1) / at_once); };
  const bool few = tiles(16) <= 148;
  const float c16 = few ? 0.316f : 0.47f * rounds(tiles(16), 296), c32 = 0.39f * rounds(tiles(32), 148), c64 = 0.53f * rounds(tiles(64), 148), c80 = 0.77f * rounds(tiles(80), 148);
  if (c80 < fminf(c16, fminf(c32, c64))) return launch<80, 1>(A, lda, w, ldw, C, ldc, M, N, K, err, s);
  if (c16 <= fminf(c32, c64))
    return few ? launch<16, 1>(A, lda, w, ldw, C, ldc, M, N, K, err, s) : launch<16, 2>(A, lda, w, ldw, C, ldc, M, N, K, err, s);
  if (c32 <= c64) return launch<32, 1>(A, lda, w, ldw, C, ldc, M, N, K, err, s);
  return launch<64, 1>(A, lda, w, ldw, C, ldc, M, N, K, err, s);
}
