// The routed experts' products on the fifth-generation tensor cores, two SMs to a tile, with the weights in the rows of the tile:
//     out[place, n] = finish(place_scale[place] * W[expert of place][n] . x[row of place])         (float32 sums)
//
// Experts get different numbers of tokens, a few in a step of decoded tokens and some hundreds in a prompt, so a tile with a fixed
// number of token rows is mostly padding.  Here a tile is 256 rows of an expert's matrix (the M side of the MMA: two CTAs of a
// cluster with 128 rows each) by 32 .. 256 of its tokens (the N side, which the instruction descriptor gives at run time): an
// expert's c tokens are cut into ceil(c / 256) equal parts, rounded up to a multiple of 32.  Decoded tokens then cost what reading
// the weights costs, and a prompt's tiles are 84 to 95 % tokens.
//
// Operands: the weights (K-major rows) come as 128 x 64 boxes by TMA, the tokens' rows, side by side in place order, as boxes of 128, 64, 32 and
// 16 rows, one of each at most (in boxes of 16 alone, eight of them a stage, a block of K took 820 cycles instead of 660, of which the MMAs 512).
// The caller copies them there first (moe_rows: 14 us for 8,192 places of 4,096 numbers); fetched from where they stand by
// tile::gather4, four rows an instruction, the product of a prompt of 2,048 tokens with 32 matrices of 6,144 rows took 1,101 us instead of
// 491, and 32 places gained nothing either.  Each CTA of the pair loads half of a tile's tokens.  Places past an expert's last one are computed from whatever row is there and not
// stored.
//
// Per CTA, by warp (the roles and barriers of gemm_tcgen05_pair.cu): warp 8 producer; warp 9 allocates TMEM and, in the first CTA,
// issues the MMAs; warps 0-7 epilogue, two to a quarter of the
// lanes with every second 32 tokens each (four warps took longer than the products where K is 1,024).  The accumulators (256 columns) are double-buffered.  In the epilogue a lane holds one
// weight row and a register one token; neighbouring lanes exchange halves, so that a lane holds both numbers of a pair of rows
// (gate_i and up_i, or two neighbouring outputs) for every second token: the gate is applied to the float32 sums and a lane stores
// a whole pair.
// Persistent grid: the tiles of an expert with the token part running fastest, then the weight rows, so the pairs that run together
// read an expert's matrix once and share its tokens in L2.
//
// What bounds it: the weights' bytes for decoded tokens, the tensor cores (under the power cap), the part of a tile that is padding and the last
// round of tiles for prompts.  32 experts of 3 x 3,072 x 4,096, 4 of them a token, first and second product: 274 and 136 us for 64 tokens (1.61
// and 0.81 GB: 5.9 TB/s), 462 and 232 us for 2,048 tokens (0.89 PFLOP/s of tokens; 509 and 256 with four warps in the epilogue and boxes of
// 16); 16 experts of 3 x 768 x 1,024, 2,048 tokens 38.8 and 30.8 (57.0 and 43.4).  Tried and left: tiles of 512 weight rows, a block in each
// accumulator (half the reads of the tokens, no second buffer: 454 and 239); runs of tiles of equal cost for the pairs, each at experts of its own
// (598 and 306: the experts' tokens then fall out of L2).
//
// Every wait is bounded; a CTA whose wait runs out raises the error flag and runs to its end.
#include "common.cuh"
#include "tcgen05_utils.cuh"
using namespace arle;

namespace {

constexpr int BM = 128;                      // weight rows per CTA (256 per pair)
constexpr int BNMAX = 256;                   // tokens of a tile
constexpr int BK = 64;
constexpr int kEpilogueWarps = 8, kProducer = kEpilogueWarps, kIssuer = kProducer + 1;
constexpr int kThreads = (kIssuer + 1) * 32;
constexpr uint32_t kTmemCols = 512;
constexpr int kStages = 6;
constexpr int kMaxExperts = 1024;
constexpr uint32_t A_BYTES = BM * BK * 2, B_BYTES = (BNMAX / 2) * BK * 2, STAGE = A_BYTES + B_BYTES;

enum Finish { kNone = 0, kSquareRelu = 1, kSilu = 2, kGeluTanh = 3, kClamped = 4 };

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
      ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}

template <int FINISH>
__device__ __forceinline__ float finish_pair(float g, float u, float limit, float alpha) {
  if (FINISH == kSilu) return __fdividef(g, 1.0f + __expf(-g)) * u;
  if (FINISH == kGeluTanh) return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);        // as clamped_glu: the full exponential and division
}

// The tokens' rows in boxes of 16, 32, 64 and 128: half a tile's tokens are one of each at most.
constexpr int kBoxes = 4;
struct RowMaps {
  CUtensorMap of[kBoxes];
};

// The tiles of a product: expert e has cuts[e + 1] - cuts[e] equal token parts.
struct Walk {
  const int* plan;
  const int* cuts;
  int tiles_n, expert;
  __device__ __forceinline__ bool at(int t, int E, int& n_tile, int& p0, int& count, int& part) {
    if (t >= cuts[E] * tiles_n) return false;
    while (t >= cuts[expert + 1] * tiles_n) ++expert;
    const int parts = cuts[expert + 1] - cuts[expert], r = t - cuts[expert] * tiles_n;
    const int first = plan[expert], c = plan[expert + 1] - first;
    part = ((c + parts - 1) / parts + 31) & ~31;
    const int j = r % parts;
    n_tile = r / parts;
    p0 = first + j * part;
    count = min(part, c - j * part);
    return true;
  }
};

template <int FINISH>
__global__ void __launch_bounds__(kThreads, 1) moe_tcgen05_kernel(const __grid_constant__ RowMaps map_x, const __grid_constant__ CUtensorMap map_w,
                                                                  const int* __restrict__ plan, int E,
                                                                  __nv_bfloat16* __restrict__ out, int ldo, int N, int K,
                                                                  const float* __restrict__ place_scale, float limit, float alpha,
                                                                  int* __restrict__ err) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[kStages];      // first CTA's: both CTAs' copies of the stage have landed
  __shared__ __align__(8) uint64_t empty_bar[kStages];     // each CTA's: the MMAs have read the stage
  __shared__ __align__(8) uint64_t acc_full[2];            // each CTA's: accumulator buffer complete
  __shared__ __align__(8) uint64_t acc_empty[2];           // first CTA's: both CTAs' epilogues have drained the buffer
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int cuts[kMaxExperts + 1];                    // token parts of the experts before expert e

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int pair = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);
  const int kblocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_addr(&full_bar[s]), 1);
      mbar_init(smem_addr(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_addr(&acc_full[b]), 1);
      mbar_init(smem_addr(&acc_empty[b]), 2 * kEpilogueWarps);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == kIssuer) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_base_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
  if (warp == 0) {
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      int parts = 0;
      if (e < E) {
        const int c = plan[e + 1] - plan[e];
        if (c > 0) {
          const int k = (c + BNMAX - 1) / BNMAX, size = ((c + k - 1) / k + 31) & ~31;
          parts = (c + size - 1) / size;                   // rounding up can make the last part empty
        }
      }
      int sum = parts;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (e < E) cuts[e] = carry + sum - parts;
      carry += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) cuts[E] = carry;
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                      // the partner's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const volatile int* aborted = &abort_flag;
  Walk walk{plan, cuts, (N + 2 * BM - 1) / (2 * BM), 0};
  int n_tile, p0, count, part;

  if (warp == kProducer) {
    int issued = 0;
    bool dead = false;
    for (int t = pair; !dead && walk.at(t, E, n_tile, p0, count, part); t += npairs) {
      const int half = part >> 1;                          // this CTA's tokens: 16 .. 128
      const int mine = p0 + (int)rank * half;
      const bool boxed = lane < kBoxes && (half >> (4 + lane) & 1);      // lane l brings 16 << l rows, behind those of the larger boxes
      const int box_row = half & ~((32 << (lane & 3)) - 1);
      const int wrow = walk.expert * N + n_tile * 2 * BM + (int)rank * BM;
      for (int kb = 0; kb < kblocks; ++kb, ++issued) {
        const int s = issued % kStages;
        const bool ok = mbar_wait_bounded(smem_addr(&empty_bar[s]), ((issued / kStages) & 1) ^ 1, aborted);
        if (__any_sync(0xffffffffu, !ok)) {
          abort_flag = 1;
          dead = true;
          break;
        }
        const uint32_t bar_local = smem_addr(&full_bar[s]);
        const uint32_t bar = map_to_rank(bar_local, 0);
        const uint32_t a_dst = smem_addr(tiles + (size_t)s * STAGE);
        if (lane == 0) {
          if (leader) mbar_expect_tx(bar_local, 2 * (A_BYTES + (uint32_t)half * BK * 2));      // the bytes of both CTAs
          tma_load_2d_pair(a_dst, &map_w, kb * BK, wrow, bar);
        }
        __syncwarp();
        if (boxed) tma_load_2d_pair(a_dst + A_BYTES + (uint32_t)box_row * (BK * 2), &map_x.of[lane & 3], kb * BK, mine + box_row, bar);
      }
    }
  } else if (warp == kIssuer) {
    if (lane == 0 && leader) {
      int consumed = 0, iter = 0;
      for (int t = pair; !*aborted && walk.at(t, E, n_tile, p0, count, part); t += npairs, ++iter) {
        const int buf = iter & 1;
        if (!mbar_wait_bounded(smem_addr(&acc_empty[buf]), ((iter >> 1) & 1) ^ 1, aborted)) {
          abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t idesc = idesc_bf16(2 * BM, part);
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BNMAX);
        for (int kb = 0; kb < kblocks; ++kb, ++consumed) {
          const int s = consumed % kStages;
          if (!mbar_wait_bounded(smem_addr(&full_bar[s]), (consumed / kStages) & 1, aborted)) {
            abort_flag = 1;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_addr(tiles + (size_t)s * STAGE);
          const uint64_t adesc = smem_desc_sw128(a_addr), bdesc = smem_desc_sw128(a_addr + A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16_pair(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit_both(smem_addr(&empty_bar[s]));
        }
        umma_commit_both(smem_addr(&acc_full[buf]));
      }
    }
  } else {
    // epilogue of this CTA's 128 weight rows: warp i reads TMEM lanes 32 i .. 32 i + 31
    constexpr bool GATED = FINISH >= kSilu;
    int iter = 0;
    const uint32_t acc_empty_leader[2] = {map_to_rank(smem_addr(&acc_empty[0]), 0), map_to_rank(smem_addr(&acc_empty[1]), 0)};
    for (int t = pair; walk.at(t, E, n_tile, p0, count, part); t += npairs, ++iter) {
      const int buf = iter & 1;
      const bool ready = mbar_wait_bounded(smem_addr(&acc_full[buf]), (iter >> 1) & 1, aborted);
      if (!ready) abort_flag = 1;
      if (__any_sync(0xffffffffu, !ready || *aborted)) break;
      tc_fence_after();
      const int n0 = n_tile * 2 * BM + (int)rank * BM + (warp & 3) * 32 + (lane & ~1);       // this lane's pair of weight rows
      const int odd = lane & 1;
#pragma unroll 1
      for (int c = (warp >> 2) * 32; c < part; c += kEpilogueWarps * 8) {
        uint32_t r[32];
        tmem_ld32(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(buf * BNMAX + c), r);
        tmem_ld_wait();
        if (c >= count) continue;
        const float scale = place_scale && c + lane < count ? place_scale[p0 + c + lane] : 1.f;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          // even lane: its row's sum of token c + i and the next row's; odd lane: the row before's and its own of token c + i + 1
          const float own = __uint_as_float(odd ? r[i + 1] : r[i]);
          const float sent = __uint_as_float(odd ? r[i] : r[i + 1]);
          const float other = __shfl_xor_sync(0xffffffffu, sent, 1);
          float a = odd ? other : own, b = odd ? own : other;
          const int tok = c + i + odd;
          if (place_scale) {
            const float f = __shfl_sync(0xffffffffu, scale, i + odd);
            a *= f, b *= f;
          }
          if (tok >= count || n0 >= N) continue;
          if (GATED) {
            out[(size_t)(p0 + tok) * ldo + (n0 >> 1)] = __float2bfloat16_rn(finish_pair<FINISH>(a, b, limit, alpha));
          } else {
            if (FINISH == kSquareRelu) {
              a = fmaxf(a, 0.f), b = fmaxf(b, 0.f);
              a *= a, b *= b;
            }
            __nv_bfloat16* dst = out + (size_t)(p0 + tok) * ldo + n0;
            if (n0 + 1 < N && ((uintptr_t)dst & 3) == 0) {
              *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(a, b);
            } else {
              dst[0] = __float2bfloat16_rn(a);
              if (n0 + 1 < N) dst[1] = __float2bfloat16_rn(b);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty_leader[buf]);
    }
  }
  // Where a wait ran out, copies may still be under way into the pair's shared memory: wait for them (bounded) before the
  // CTA ends.  They are counted on the first CTA's barriers, so only it can look, and it does when all its warps are here: any of them may
  // be the one whose wait ran out.
  __syncthreads();
  if (warp == kProducer && lane == 0 && leader && *aborted)
    for (int s = 0; s < kStages; ++s) mbar_wait_plain(smem_addr(&full_bar[s]), 0), mbar_wait_plain(smem_addr(&full_bar[s]), 1);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                      // neither CTA frees tensor memory the other's MMAs may still write
  if (warp == kIssuer) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag && err) atomicExch(err, 4);
}

template <int FINISH>
int launch(const void* x, int ldx, int x_rows, const void* W, void* out, int ldo, const int* plan, int E, int pairs, int N, int K,
           const float* place_scale, float limit, float alpha, int* err, cudaStream_t s) {
  RowMaps mx;
  CUtensorMap mw;
  int rc = 0;
  for (int i = 0; i < kBoxes && rc == 0; ++i) rc = tensor_map_2d_bf16(x, x_rows, K, ldx, 16 << i, &mx.of[i]);
  if (rc) return rc;
  rc = tensor_map_2d_bf16(W, (long long)E * N, K, K, BM, &mw);
  if (rc) return rc;
  const size_t smem = (size_t)kStages * STAGE + 1024;
  auto kern = moe_tcgen05_kernel<FINISH>;
  static SharedLimit limit_of;
  cudaError_t e = limit_of.raise((const void*)kern, smem);
  if (e != cudaSuccess) return (int)e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // an expert with c places has at most c / 256 + 1 parts
  const long long most = ((long long)pairs / BNMAX + (pairs < E ? pairs : E)) * ((N + 2 * BM - 1) / (2 * BM));
  long long grid_pairs = sms / 2;
  if (most < grid_pairs) grid_pairs = most;
  e = launch_kernel(kern, dim3((unsigned)(2 * grid_pairs)), dim3(kThreads), smem, s, 2, mx, mw, plan, E, (__nv_bfloat16*)out, ldo, N, K,
                    place_scale, limit, alpha, err);
  if (e != cudaSuccess) return (int)e;
  return launch_status();
}

// dst[place] = x[rows[place]], 16 bytes a thread and step.
__global__ void __launch_bounds__(256) moe_rows_kernel(const __nv_bfloat16* x, int ldx, const int* rows,
                                                       __nv_bfloat16* dst, int K) {
  pdl_launch_dependents();
  pdl_wait();
  const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)rows[blockIdx.x] * ldx);
  uint4* to = reinterpret_cast<uint4*>(dst + (size_t)blockIdx.x * K);
  constexpr int AHEAD = 4;                                 // loads in front of the stores, which they could not pass
  for (int i0 = threadIdx.x; i0 < K / 8; i0 += 256 * AHEAD) {
    uint4 v[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (i0 + j * 256 < K / 8) v[j] = from[i0 + j * 256];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (i0 + j * 256 < K / 8) to[i0 + j * 256] = v[j];
  }
}

}  // namespace

// Copies the places' rows of x side by side: dst [pairs, K].
ARLE_API int arle_moe_rows(const void* x, int ldx, const int* rows, void* dst, int pairs, int K, cudaStream_t s) {
  if (pairs <= 0) return 0;
  if (K <= 0 || K % 8 || ldx % 8 || (((uintptr_t)x | (uintptr_t)dst) & 15)) return ARLE_E_UNSUPPORTED;
  launch_early(moe_rows_kernel, dim3(pairs), dim3(256), 0, s, 1, (const __nv_bfloat16*)x, ldx, rows, (__nv_bfloat16*)dst, K);
  return launch_status();
}

// x bfloat16 [x_rows, K] in place order, W bfloat16 [E][N][K] contiguous,
// out bfloat16 [pairs, N], or [pairs, N / 2] for the gated finishes (W's rows 2i and 2i + 1: gate_i and up_i).
// finish: 0 none, 1 square of relu, 2 silu gate, 3 gelu (tanh) gate, 4 clamped gate (limit, alpha).  Needs K and ldx multiples of 8
// and 16-byte aligned x and W.  err: set to 4 if a bounded wait ran out.
ARLE_API int arle_moe_gemm_tcgen05(const void* x, int ldx, int x_rows, const void* W, void* out, int ldo, const int* plan, int E,
                                   int pairs, int N, int K, const float* place_scale, int finish, float limit, float alpha, int* err,
                                   cudaStream_t s) {
  if (pairs <= 0 || N <= 0) return 0;
  if (K <= 0 || E <= 0 || finish < 0 || finish > 4 || x_rows <= 0 || (finish >= 2 && N % 2)) return ARLE_E_BADARG;
  if (E > kMaxExperts || K % 8 || ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)W & 15) || (long long)E * N > 0x7fffffffll) return ARLE_E_UNSUPPORTED;
  switch (finish) {
    case kNone: return launch<kNone>(x, ldx, x_rows, W, out, ldo, plan, E, pairs, N, K, place_scale, limit, alpha, err, s);
    case kSquareRelu: return launch<kSquareRelu>(x, ldx, x_rows, W, out, ldo, plan, E, pairs, N, K, place_scale, limit, alpha, err, s);
    case kSilu: return launch<kSilu>(x, ldx, x_rows, W, out, ldo, plan, E, pairs, N, K, place_scale, limit, alpha, err, s);
    case kGeluTanh: return launch<kGeluTanh>(x, ldx, x_rows, W, out, ldo, plan, E, pairs, N, K, place_scale, limit, alpha, err, s);
    default: return launch<kClamped>(x, ldx, x_rows, W, out, ldo, plan, E, pairs, N, K, place_scale, limit, alpha, err, s);
  }
}
