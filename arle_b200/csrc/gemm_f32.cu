// True 32-bit matrix product for the float32 path of the engine:
//     C[M, N] = A[M, K] (float32) . W[N, K]^T      W float32 or bfloat16 (widened exactly)
// Plain FFMA, no tensor cores, no TF32, no split along K: every output element is
// the sum over k = 0..K-1 in ascending order, so its bits do not depend on M, on
// the tile it falls into, or on what else is in the batch.  Any M, N, K.
//
// The same kernel with bfloat16 A (and a bfloat16 or float32 C, rounded once from the
// float32 sum) is the plain twin of the tensor-core products: the engine's "plain"
// kernel set runs it for every projection, so that a bfloat16 discrepancy can be put
// down to the fast kernels or to the arithmetic.
//
// float32 A runs on one of four kernels (but for bfloat16 W with K from 512 on in whole blocks of 64: gemm_f32_tc.cu), all with that order of sums, so all with the same bits:
//  * gemm_f32_rows (up to 16 rows): a thread per column of C, W staged by cp.async.  Bound by W's bytes for one row, by the loads from
//    shared memory for more.
//  * gemm_f32_stages: tiles of 32 x 32 and 64 x 64, stages of 32 numbers of k as they lie in memory on their way by cp.async, three ahead.  For
//    the products of short prompts, whose few tiles an SM are bound by how long memory takes to answer (gemm_f32_tiles asks one stage ahead).
//  * gemm_f32_tiles: tiles of 64 x 128, and of 64 x 64 where a bfloat16 W's fill an SM, 8 x 4 sums a thread, the next 16 numbers of k on their
//    way while the present ones are multiplied; two neighbouring sums are one packed instruction (fma.rn.f32x2: each half the same rounded
//    fused product).  Bound by instructions, half of FFMA's rate.  No sum may be split along k, so the launcher takes the tile that leaves the busiest SM the least.
//  * gemm_f32 (rows that are not on 16-byte boundaries, and bfloat16 A): the general one, tiles of 64 x 64.
// Measured, the general kernel, gemm_f32_tiles at its best tile of 64 x 128 to 32 x 32, and these (us, W bfloat16): 301 rows, 4,096 x 1,024 168, 97
// and 86; 1,024 x 2,048 150, 88 and 62; 6,144 x 1,024 222, 117 and 117; 1,024 x 3,072 224, 130 and 90; 40 rows, 1,024 x 2,048 72 and 31; 120
// rows, 6,144 x 1,024 68 and 60; 1,024 rows of 24,576 x 4,096 8,726 and 4,420 (47 TFLOP/s); one row, 151,936 x 1,024 880 and 58 (5.3 TB/s),
// 4,096 x 1,024 76 and 12; 8 rows 883 and 117.
#include "common.cuh"
#include "mma_utils.cuh"
using namespace arle;

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256) gemm_f32_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                       TC* __restrict__ C, int M, int N, int K, int lda,
                                                       int ldw, int ldc) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256;
      const int r = idx >> 4, c = idx & 15;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.f;
      Ws[c][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn < N) C[(size_t)gm * ldc + gn] = from_f32<TC>(acc[i][j]);
    }
  }
}

template <typename TA, typename TW, typename TC>
static int launch_plain(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc,
                        cudaStream_t s) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return ARLE_E_UNSUPPORTED;
  launch_kernel(gemm_f32_kernel<TA, TW, TC>, dim3(grid), dim3(256), 0, s, 1, (const TA*)A, (const TW*)W, (TC*)C, M, N, K,
                lda, ldw, ldc);
  return launch_status();
}

// TM, TN: rows and columns of C a thread holds, in groups of four that are BM / (TM / 4) and BN / (TN / 4) apart; two neighbouring
// columns' sums stand in one 64-bit register.
template <typename TW, int BM_, int BN_, int TM, int TN>
__global__ void __launch_bounds__((BM_ / TM) * (BN_ / TN)) gemm_f32_tiles_kernel(const float* __restrict__ A, const TW* __restrict__ W,
                                                                                 float* __restrict__ C, int M, int N, int K, int lda,
                                                                                 int ldw, int ldc) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int THREADS = (BM_ / TM) * (BN_ / TN);
  constexpr int AI = BM_ * 4 / THREADS, WI = BN_ * 4 / THREADS;      // groups of four numbers of k a thread stages
  static_assert(BM_ * 4 % THREADS == 0 && BN_ * 4 % THREADS == 0, "staging");
  __shared__ __align__(16) float As[2][BK][BM_ + 4];
  __shared__ __align__(16) float Ws[2][BK][BN_ + 4];
  const int tid = threadIdx.x;
  const int tx = tid % (BN_ / TN), ty = tid / (BN_ / TN);
  const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN_;
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
  Pack<float, 4> ar[AI];
  Pack<TW, 4> wr[WI];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < AI; ++i) {
      const int idx = tid + i * THREADS, r = m0 + (idx >> 2), k = k0 + (idx & 3) * 4;
#pragma unroll
      for (int g = 0; g < 4; ++g) ar[i].e[g] = 0.f;
      if (r < M && k < K) ar[i] = *reinterpret_cast<const Pack<float, 4>*>(A + (size_t)r * lda + k);
    }
#pragma unroll
    for (int i = 0; i < WI; ++i) {
      const int idx = tid + i * THREADS, r = n0 + (idx >> 2), k = k0 + (idx & 3) * 4;
#pragma unroll
      for (int g = 0; g < 4; ++g) wr[i].e[g] = from_f32<TW>(0.f);
      if (r < N && k < K) wr[i] = *reinterpret_cast<const Pack<TW, 4>*>(W + (size_t)r * ldw + k);
    }
  };
  auto put = [&](int b) {
#pragma unroll
    for (int i = 0; i < AI; ++i) {
      const int idx = tid + i * THREADS;
#pragma unroll
      for (int g = 0; g < 4; ++g) As[b][(idx & 3) * 4 + g][idx >> 2] = ar[i].e[g];
    }
#pragma unroll
    for (int i = 0; i < WI; ++i) {
      const int idx = tid + i * THREADS;
#pragma unroll
      for (int g = 0; g < 4; ++g) Ws[b][(idx & 3) * 4 + g][idx >> 2] = to_f32(wr[i].e[g]);
    }
  };
  const int nk = (K + BK - 1) / BK;
  fetch(0);
  put(0);
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    const int b = kt & 1;
    if (kt + 1 < nk) fetch((kt + 1) * BK);
    auto frag = [&](int kk, float (&a)[TM], unsigned long long (&w)[TN / 2]) {
#pragma unroll
      for (int g = 0; g < TM / 4; ++g) load_vec<float, 4>(&As[b][kk][g * (BM_ / (TM / 4)) + ty * 4], reinterpret_cast<float(&)[4]>(a[4 * g]));
#pragma unroll
      for (int g = 0; g < TN / 4; ++g) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][g * (BN_ / (TN / 4)) + tx * 4]);
        w[2 * g] = x.x;
        w[2 * g + 1] = x.y;
      }
    };
    float a[2][TM];
    unsigned long long w[2][TN / 2];
    frag(0, a[0], w[0]);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      if (kk + 1 < BK) frag(kk + 1, a[(kk + 1) & 1], w[(kk + 1) & 1]);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        unsigned long long aa;
        asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[kk & 1][i]));
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(w[kk & 1][j]));
      }
    }
    if (kt + 1 < nk) put(b ^ 1);                       // the other buffer was last read before the barrier that ended the tile before
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + (i >> 2) * (BM_ / (TM / 4)) + ty * 4 + (i & 3);
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + (j >> 2) * (BN_ / (TN / 4)) + tx * 4 + (j & 3);
      if (gn < N) C[(size_t)gm * ldc + gn] = __uint_as_float((unsigned)(j & 1 ? acc[i][j / 2] >> 32 : acc[i][j / 2]));
    }
  }
}

// TM, TN: rows and columns of C a thread holds, BM / TM and BN / TN apart (neighbouring threads' rows of a stage are 16 bytes more than whole
// rounds of the banks apart).  A stage is 32 numbers of k of the tile's rows of A and W as they lie in memory, brought by cp.async three stages
// ahead: a thread reads four (A) or sixteen bytes of (W) numbers of k at once and runs through them in order.
constexpr int kTileK = 32, kTileStages = 4;
template <typename TW, int BM_, int BN_>
struct TileSmem {
  static constexpr int AP = kTileK + 4, WP = kTileK + 16 / (int)sizeof(TW);      // numbers from row to row
  static constexpr size_t A = (size_t)BM_ * AP * sizeof(float), W = (size_t)BN_ * WP * sizeof(TW), BYTES = kTileStages * (A + W);
};
// Number kk (0 .. 3) of k of a column from sixteen bytes of them.
__device__ __forceinline__ float nth(const uint4& v, int kk, float) { return __uint_as_float(kk == 0 ? v.x : kk == 1 ? v.y : kk == 2 ? v.z : v.w); }
__device__ __forceinline__ float nth(const uint4& v, int kk, __nv_bfloat16) {
  const uint32_t u = kk < 2 ? v.x : kk < 4 ? v.y : kk < 6 ? v.z : v.w;
  return __uint_as_float(kk & 1 ? u & 0xffff0000u : u << 16);
}

template <typename TW, int BM_, int BN_, int TM, int TN>
__global__ void __launch_bounds__((BM_ / TM) * (BN_ / TN)) gemm_f32_stages_kernel(const float* __restrict__ A, const TW* __restrict__ W,
                                                                                 float* __restrict__ C, int M, int N, int K, int lda,
                                                                                 int ldw, int ldc) {
  pdl_launch_dependents();
  pdl_wait();
  typedef TileSmem<TW, BM_, BN_> L;
  constexpr int THREADS = (BM_ / TM) * (BN_ / TN), TX = BN_ / TN, TY = BM_ / TM;
  constexpr int PER = 16 / sizeof(TW), AC = kTileK / 4, WC = kTileK / PER;       // numbers of W in 16 bytes; pieces of a row
  static_assert(BM_ * AC % THREADS == 0 && BN_ * WC % THREADS == 0, "staging");
  extern __shared__ __align__(16) unsigned char tile_sm[];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN_;
  const int nk = (K + kTileK - 1) / kTileK;
  auto load = [&](int kt) {
    float* as = reinterpret_cast<float*>(tile_sm + (kt % kTileStages) * (L::A + L::W));
    TW* ws = reinterpret_cast<TW*>(reinterpret_cast<unsigned char*>(as) + L::A);
    const int k0 = kt * kTileK;
#pragma unroll
    for (int i = 0; i < BM_ * AC / THREADS; ++i) {
      const int idx = tid + i * THREADS, r = idx / AC, k = idx % AC * 4;
      const bool ok = m0 + r < M && k0 + k < K;
      cp_async16(smem_u32(as + r * L::AP + k), ok ? A + (size_t)(m0 + r) * lda + k0 + k : A, ok ? 16 : 0);
    }
#pragma unroll
    for (int i = 0; i < BN_ * WC / THREADS; ++i) {
      const int idx = tid + i * THREADS, r = idx / WC, k = idx % WC * PER;
      const bool ok = n0 + r < N && k0 + k < K;
      cp_async16(smem_u32(ws + r * L::WP + k), ok ? W + (size_t)(n0 + r) * ldw + k0 + k : W, ok ? 16 : 0);
    }
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int kt = 0; kt < kTileStages - 1; ++kt) {
    if (kt < nk) load(kt);
    cp_commit();
  }
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<kTileStages - 2>();
    __syncthreads();                                         // the stage is here, and the one that is loaded next was used up
    if (kt + kTileStages - 1 < nk) load(kt + kTileStages - 1);
    cp_commit();
    const float* as = reinterpret_cast<const float*>(tile_sm + (kt % kTileStages) * (L::A + L::W)) + ty * L::AP;
    const TW* ws = reinterpret_cast<const TW*>(tile_sm + (kt % kTileStages) * (L::A + L::W) + L::A) + tx * L::WP;
#pragma unroll
    for (int k0 = 0; k0 < kTileK; k0 += PER) {
      uint4 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const uint4*>(ws + j * TX * L::WP + k0);
#pragma unroll
      for (int k4 = 0; k4 < PER; k4 += 4) {
        float a[TM][4];
#pragma unroll
        for (int i = 0; i < TM; ++i) load_vec<float, 4>(as + i * TY * L::AP + k0 + k4, a[i]);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const float wj = nth(w[j], k4 + kk, TW());
#pragma unroll
            for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i][kk], wj, acc[i][j]);
          }
      }
    }
  }
  cp_wait<0>();
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + i * TY;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx + j * TX;
      if (gn < N) C[(size_t)gm * ldc + gn] = acc[i][j];
    }
  }
}

// Up to 16 rows of A: a thread holds one column of C for all rows.  A block stages 128 rows of W, 64 numbers of k at a time, three
// stages; a staged row is 16 bytes longer than its numbers, so that eight lanes' 16-byte reads fall on different banks.
constexpr int kRowsN = 128, kRowsK = 64, kRowsStages = 3;

template <typename TW, int MR>
__global__ void __launch_bounds__(kRowsN) gemm_f32_rows_kernel(const float* __restrict__ A, const TW* __restrict__ W, float* __restrict__ C,
                                                               int M, int N, int K, int lda, int ldw, int ldc) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int PER = 16 / sizeof(TW);                       // numbers in 16 bytes
  constexpr int CH = kRowsK / PER, PITCH = kRowsK + PER;     // 16-byte pieces of a row, numbers to the next row
  extern __shared__ __align__(16) unsigned char rows_sm[];
  TW* ws = reinterpret_cast<TW*>(rows_sm);                                              // [stages][128][PITCH]
  float* as = reinterpret_cast<float*>(rows_sm + sizeof(TW) * kRowsStages * kRowsN * PITCH);      // [stages][MR][64]
  const int n0 = blockIdx.x * kRowsN, tid = threadIdx.x;
  const int nk = (K + kRowsK - 1) / kRowsK;
  auto load = [&](int kt) {
    const int st = kt % kRowsStages, k0 = kt * kRowsK;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int idx = tid + i * kRowsN, r = idx / CH, c = idx % CH * PER;
      const bool ok = n0 + r < N && k0 + c < K;
      cp_async16(smem_u32(ws + ((size_t)st * kRowsN + r) * PITCH + c), ok ? W + (size_t)(n0 + r) * ldw + k0 + c : W, ok ? 16 : 0);
    }
    for (int idx = tid; idx < MR * (kRowsK / 4); idx += kRowsN) {
      const int r = idx / (kRowsK / 4), c = idx % (kRowsK / 4) * 4;
      const bool ok = r < M && k0 + c < K;
      cp_async16(smem_u32(as + ((size_t)st * MR + r) * kRowsK + c), ok ? A + (size_t)r * lda + k0 + c : A, ok ? 16 : 0);
    }
  };
  float acc[MR];
#pragma unroll
  for (int r = 0; r < MR; ++r) acc[r] = 0.f;
  load(0);
  cp_commit();
  if (nk > 1) load(1);
  cp_commit();
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<1>();
    __syncthreads();
    if (kt + 2 < nk) load(kt + 2);
    cp_commit();
    const int st = kt % kRowsStages;
    const TW* w = ws + ((size_t)st * kRowsN + tid) * PITCH;
    const float* a = as + (size_t)st * MR * kRowsK;
#pragma unroll
    for (int c = 0; c < kRowsK; c += PER) {
      float wv[PER];
      load_vec<TW, PER>(w + c, wv);
#pragma unroll
      for (int g = 0; g < PER; g += 4)
#pragma unroll
        for (int r = 0; r < MR; ++r) {
          const float4 x = *reinterpret_cast<const float4*>(a + r * kRowsK + c + g);
          acc[r] = fmaf(x.x, wv[g], acc[r]);
          acc[r] = fmaf(x.y, wv[g + 1], acc[r]);
          acc[r] = fmaf(x.z, wv[g + 2], acc[r]);
          acc[r] = fmaf(x.w, wv[g + 3], acc[r]);
        }
    }
  }
  cp_wait<0>();
  if (n0 + tid < N)
#pragma unroll
    for (int r = 0; r < MR; ++r)
      if (r < M) C[(size_t)r * ldc + n0 + tid] = acc[r];
}

template <typename TW, int MR>
static int launch_rows(const float* A, const TW* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
  constexpr size_t smem = sizeof(TW) * kRowsStages * kRowsN * (kRowsK + 16 / sizeof(TW)) + sizeof(float) * kRowsStages * MR * kRowsK;
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)gemm_f32_rows_kernel<TW, MR>, smem);
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(gemm_f32_rows_kernel<TW, MR>, dim3((N + kRowsN - 1) / kRowsN), dim3(kRowsN), smem, s, 1, A, W, C, M, N, K, lda, ldw, ldc);
  return launch_status();
}

template <typename TW, int BM_, int BN_, int TM, int TN>
static int launch_tiles(const float* A, const TW* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
  dim3 grid((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_);
  if (grid.y > 65535) return ARLE_E_UNSUPPORTED;
  launch_kernel(gemm_f32_tiles_kernel<TW, BM_, BN_, TM, TN>, grid, dim3((BM_ / TM) * (BN_ / TN)), 0, s, 1, A, W, C, M, N, K, lda, ldw, ldc);
  return launch_status();
}

template <typename TW, int BM_, int BN_, int TM, int TN>
static int launch_stages(const float* A, const TW* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
  dim3 grid((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_);
  if (grid.y > 65535) return ARLE_E_UNSUPPORTED;
  constexpr size_t smem = TileSmem<TW, BM_, BN_>::BYTES;
  static SharedLimit limit;
  auto kernel = gemm_f32_stages_kernel<TW, BM_, BN_, TM, TN>;
  const cudaError_t raised = limit.raise((const void*)kernel, smem);
  if (raised != cudaSuccess) return (int)raised;
  launch_kernel(kernel, grid, dim3((BM_ / TM) * (BN_ / TN)), smem, s, 1, A, W, C, M, N, K, lda, ldw, ldc);
  return launch_status();
}

template <typename TW>
static int launch_f32(const float* A, const void* Wv, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
  const TW* W = (const TW*)Wv;
  constexpr int PER = 16 / sizeof(TW);
  if (K % PER || lda % 4 || ldw % PER || ((uintptr_t)A & 15) || ((uintptr_t)Wv & 15))
    return launch_plain<float, TW, float>(A, Wv, C, M, N, K, lda, ldw, ldc, s);
  if (M <= 16) {
    if (M == 1) return launch_rows<TW, 1>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (M <= 4) return launch_rows<TW, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (M <= 8) return launch_rows<TW, 8>(A, W, C, M, N, K, lda, ldw, ldc, s);
    return launch_rows<TW, 16>(A, W, C, M, N, K, lda, ldw, ldc, s);
  }
  // Microseconds per 1,024 of k: what a tile takes by itself on an SM, and what it adds to an SM that is full of them; in between the
  // cube root of the sum of cubes is within a tenth of what was measured at 1,024 to 6,144 columns and 40 to 1,024 rows.
  auto cost = [&](int bm, int bn, float alone, float added) {
    const float b = (float)(((long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn) + 147) / 148) * added;
    return alone * alone * alone + b * b * b;
  };
  const bool low = M <= 65535 * 32;                        // a grid has room for the rows in tiles of 32
  const float c0 = cost(64, 128, 70.f, 53.f), c1 = cost(64, 64, 36.f, 30.f), c2 = low ? cost(32, 32, 15.6f, 9.2f) : INFINITY;
  if constexpr (sizeof(TW) == 2) {
    // Full SMs don't wait for memory, and gemm_f32_tiles widens a number of W once for all threads: 1,024 rows of 5,120 x 1,024 262 us, in stages 272;
    // 700 of 4,096 x 1,024 150 and 155 (of a float32 W 148 and 146); 640 of 4,096 x 12,288 1,772 and 1,796.  But a W that L2 does not hold comes
    // from DRAM once more for the tiles beyond the five an SM that are resident: 301 rows of 12,288 x 4,096 857 to 895, in stages 830.
    const float c3 = cost(64, 64, 60.f, 29.f);
    const bool once = (long long)N * K <= 40ll << 20 || (long long)((M + 63) / 64) * ((N + 63) / 64) <= 5 * 148;
    if (once && c3 < fminf(c0, fminf(c1, c2))) return launch_tiles<TW, 64, 64, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
  }
  if (c2 <= fminf(c0, c1)) return launch_stages<TW, 32, 32, 4, 2>(A, W, C, M, N, K, lda, ldw, ldc, s);
  if (c1 <= c0) return launch_stages<TW, 64, 64, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
  return launch_tiles<TW, 64, 128, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
}

ARLE_API int arle_gemm_f32(const float* A, const void* W, int w_dtype, float* C, int M, int N, int K, int lda,
                           int ldw, int ldc, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return ARLE_E_BADARG;
  if (w_dtype == 0) return launch_f32<float>(A, W, C, M, N, K, lda, ldw, ldc, s);
  if (w_dtype == 1) return launch_f32<__nv_bfloat16>(A, W, C, M, N, K, lda, ldw, ldc, s);
  return ARLE_E_BADARG;
}

// bfloat16 A and W, float32 sums, C bfloat16 (c_dtype 1) or float32 (0).
ARLE_API int arle_gemm_plain_bf16(const void* A, const void* W, void* C, int c_dtype, int M, int N, int K, int lda,
                                  int ldw, int ldc, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return ARLE_E_BADARG;
  if (c_dtype == 1) return launch_plain<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(A, W, C, M, N, K, lda, ldw, ldc, s);
  if (c_dtype == 0) return launch_plain<__nv_bfloat16, __nv_bfloat16, float>(A, W, C, M, N, K, lda, ldw, ldc, s);
  return ARLE_E_BADARG;
}

// The same product once per head, heads side by side in a row: C[m, h, n] = sum_k A[m, h, k] . W[h, n, k], head h of a row
// starting a_head / w_head / c_head elements after head h - 1.  Small per-head matrices (a latent attention's key and
// value maps folded into its queries and outputs); k ascending as above, so a row's result does not depend on M.
template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256) gemm_heads_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C,
                                                         int M, int N, int K, int lda, int ldw, int ldc, int a_head, long w_head,
                                                         int c_head) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  A += (size_t)blockIdx.z * a_head;
  W += (size_t)blockIdx.z * w_head;
  C += (size_t)blockIdx.z * c_head;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256;
      const int r = idx >> 4, c = idx & 15;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.f;
      Ws[c][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn < N) C[(size_t)gm * ldc + gn] = from_f32<TC>(acc[i][j]);
    }
  }
}

// dtype: 0 float32 A and C (W float32 or bfloat16 by w_dtype), 1 bfloat16 A and W, C bfloat16 or (c_dtype 0) float32.
ARLE_API int arle_gemm_heads(const void* A, const void* W, void* C, int dtype, int w_dtype, int c_dtype, int M, int N, int K, int heads,
                             int lda, int ldw, int ldc, int a_head, long w_head, int c_head, cudaStream_t s) {
  if (M <= 0 || N <= 0 || heads <= 0) return 0;
  if (K <= 0) return ARLE_E_BADARG;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, heads);
  if (grid.y > 65535 || heads > 65535) return ARLE_E_UNSUPPORTED;
  if (dtype == 0 && c_dtype != 0) return ARLE_E_BADARG;
  if (dtype == 0 && w_dtype == 0)
    launch_kernel(gemm_heads_kernel<float, float, float>, dim3(grid), dim3(256), 0, s, 1, (const float*)A, (const float*)W,
                  (float*)C, M, N, K, lda, ldw, ldc, a_head, w_head, c_head);
  else if (dtype == 0 && w_dtype == 1)
    launch_kernel(gemm_heads_kernel<float, __nv_bfloat16, float>, dim3(grid), dim3(256), 0, s, 1, (const float*)A,
                  (const __nv_bfloat16*)W, (float*)C, M, N, K, lda, ldw, ldc, a_head, w_head, c_head);
  else if (dtype == 1 && w_dtype == 1 && c_dtype == 0)
    launch_kernel(gemm_heads_kernel<__nv_bfloat16, __nv_bfloat16, float>, dim3(grid), dim3(256), 0, s, 1,
                  (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, (float*)C, M, N, K, lda, ldw, ldc, a_head, w_head, c_head);
  else if (dtype == 1 && w_dtype == 1)
    launch_kernel(gemm_heads_kernel<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>, dim3(grid), dim3(256), 0, s, 1,
                  (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, (__nv_bfloat16*)C, M, N, K, lda, ldw, ldc, a_head, w_head, c_head);
  else
    return ARLE_E_BADARG;
  return launch_status();
}
