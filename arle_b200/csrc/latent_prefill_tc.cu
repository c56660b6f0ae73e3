// Causal attention of prompt portions over latent records, with the keys and values of the heads built: the counterpart of the folded
// form in latent.cu for rows of many queries.
//
// The folded form scores a query against a record of rank + dr numbers and sums records of rank numbers: 2 (2 rank + dr) operations
// a head, query and key.  With the head's keys [W_uk c | k_rot] and values W_uv c built once for all queries of the step it is
// 2 (dn + dr + dv), 3.4 times fewer at rank 512 with heads of 128 + 64 and 128, and the tiles are those of an ordinary attention, so
// they run on tcgen05 with the queries in the rows.  Building costs 2 rank (dn + dv) a head and key, what some 170 queries save.
//
//  * latent_plan: for every row of the step with at least `least` queries the first key its queries see (a multiple of 16) and where
//    its keys start in the built arrays; -1 for the others, which the folded kernel runs, and for rows whose context is long beside their
//    queries.  A row's own lengths decide.  Rows whose records do not fit beside one another are built in groups, one after the other.
//  * latent_gather: the records of those rows from the pages, side by side, each row's padded to a multiple of 16 with zeros.
//    The product that builds keys and values is the caller's (a plain matrix product over the gathered latents).
//    A latent with an infinity or a NaN is gathered as zeros with NaN in the rotated numbers beside it (a record without rotated numbers
//    gets eight, zero otherwise): its scores are NaN, so every query that sees it gets NaN as from the folded form, and no other query
//    does, since a masked score is replaced and the built values, which meet a weight of zero, are finite.
//  * latent_prefill_tc: the attention.  The scheme, the roles of the warps and the barriers are those of attention_prefill_tc.cu (two
//    query tiles of 128 a CTA that share every key tile; scores and outputs in tensor memory, P over the scores; blocks drawn from a
//    counter, heaviest first).  What differs: a key tile has NS slices of 64 numbers from the built keys and one of up to 64 from the
//    gathered records (the rotated part, the same for all heads), values have NS slices; with three slices a stage of shared memory
//    holds one slice (Q of two tiles takes 96 KB, so two whole key tiles do not fit beside it), otherwise a whole tile; an optional
//    gate multiplies the output number by number as sigmoid(gate), on the float32 sums.
//
// What bounds it: the softmax's exponentials and the tensor cores in turn, as in attention_prefill_tc.cu.  32 heads of 128 + 64 over 2,048
// tokens at rank 512: 78 us (43 GFLOP of visible keys: 0.55 PFLOP/s), with 19 us for the product that builds keys and values and 3 us for
// the gathering; the folded kernel took 2,348 us and the products of its maps 108.
#include <atomic>

#include "common.cuh"
#include "tcgen05_utils.cuh"
using namespace arle;

namespace {

constexpr int BQ = 128;                      // queries per query tile
constexpr int BQ2 = 2 * BQ;                  // queries per CTA: two query tiles
constexpr int BKV = 128;                     // keys per tile
constexpr int kThreads = 384;                // three warp groups: softmax of tile A, softmax of tile B, the rest
constexpr int kMmaWarp = 8, kKeyWarp = 9, kValueWarp = 10;
constexpr int kRegsSoftmax = 208, kRegsOther = 80;   // registers per thread after the warp groups have traded
constexpr uint32_t SUB = 128 * 128;          // bytes of a [128 rows x 64 elements] swizzled slice
constexpr int kVStages = 2;
constexpr float kRescaleStep = 8.0f;         // log2 units the maximum may grow before O is rescaled

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
// tcgen05.mma with the A operand in tensor memory: lane = row of A, each 32-bit column holds two
// consecutive bfloat16 elements of K (16 elements of K = 8 columns).
__device__ __forceinline__ void umma_bf16_a_tmem(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ float ex2_fast(float x) {          // 2^x on the special-function unit; -inf gives 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

// Descriptor of an MN-major, 128-byte swizzled operand: rows of 64 contiguous elements
// along N (128 bytes), one row per K index; groups of 8 rows 1024 bytes apart (stride
// offset), the next 64 elements of N `lbo` bytes further (leading offset).
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

template <int N>
__device__ __forceinline__ void reg_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_less() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(N)); }

// The blocks of a running launch that were drawn after every CTA's first (which is the block of its own index).  Every
// CTA draws tickets until it draws one beyond the last block; the last ticket of all sets the counter back to zero.
// Launches take the counters in turn, so launches that run at the same time (on several streams) do not share one
// unless more than kTicketSlots of them are under way.
constexpr int kTicketSlots = 64;
__device__ unsigned int g_ticket[kTicketSlots];

// Ticket number gridDim.x + (draws before this one); the draw that must be the last of the launch resets the counter.
__device__ __forceinline__ unsigned int draw_ticket(int nblocks, int slot) {
  const unsigned int raw = atomicAdd(&g_ticket[slot], 1u);
  if (raw + 1 == (unsigned int)nblocks) atomicExch(&g_ticket[slot], 0u);      // nblocks - grid blocks and grid tickets beyond them
  return raw + gridDim.x;
}

// plan: [R] (first key, place of that key in the built arrays of its group or -1).  A row is built from at most max(most * its queries,
// floor) records, a group holds at most `room`.
__global__ void __launch_bounds__(32) latent_plan_kernel(const int* q_indptr, const int* kv_lens, int R, int least,
                                                         int most, int floor, int room, int window, int2* plan) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x;
  int filled = 0;                                          // places of the group so far
  for (int r0 = 0; r0 < R; r0 += 32) {
    const int r = r0 + lane;
    int need = 0, first = 0, at = -1;
    if (r < R) {
      const int n = q_indptr[r + 1] - q_indptr[r], kv = kv_lens[r];
      first = first_visible_key(kv - n, window, 0) & ~15;
      const int records = (kv - first + 15) & ~15;
      if (n >= least && records <= max(most * n, floor)) need = records;
    }
    for (int i = 0; i < 32; ++i) {
      const int x = __shfl_sync(0xffffffffu, need, i);
      if (x == 0) continue;
      if (filled + x > room) filled = 0;                   // the next group
      if (lane == i) at = filled;
      filled += x;
    }
    if (r < R) plan[r] = make_int2(first, at);
  }
}

// Numbers of a gathered record behind its latent.
__host__ __device__ constexpr int gathered_tail(int dr) { return dr ? dr : 8; }

constexpr int kGatherThreads = 256, kGatherSteps = 16 * (512 + 64) / 8 / kGatherThreads + 1;     // 16-byte pieces a thread copies at most

// A block copies 16 neighbouring records (pages hold a multiple of 16), 16 bytes a thread and step.  kd: numbers of a stored record, ko
// of a gathered one.
__global__ void __launch_bounds__(kGatherThreads) latent_gather_kernel(const __nv_bfloat16* cache, const int* block_table,
                                                                       int bt_stride, const int* kv_lens,
                                                                       const int2* plan, int R, int page_size, int rank, int kd, int ko,
                                                                       __nv_bfloat16* out) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int bad[16];                                  // records whose latent holds an infinity or a NaN
  const int place = blockIdx.x * 16;
  int row = -1;
  for (int r = 0; r < R; ++r) {
    const int at = plan[r].y;
    if (at > place) break;
    if (at >= 0) row = r;
  }
  const int key = plan[row].x + place - plan[row].y, live = kv_lens[row] - key;       // records of the 16 that the request holds
  const int page = block_table[(size_t)row * bt_stride + key / page_size];
  const uint4* src = reinterpret_cast<const uint4*>(cache + ((size_t)page * page_size + key % page_size) * kd);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)place * ko);
  const int per = ko / 8, from = kd / 8, latent = rank / 8;
  if (threadIdx.x < 16) bad[threadIdx.x] = 0;
  __syncthreads();
  uint4 x[kGatherSteps];
#pragma unroll
  for (int it = 0; it < kGatherSteps; ++it) {
    const int i = threadIdx.x + it * kGatherThreads, rec = i / per, c = i - rec * per;
    x[it] = make_uint4(0, 0, 0, 0);
    if (rec >= min(16, live) || c >= from) continue;
    x[it] = src[rec * from + c];
    if (c < latent && (bf16x2_odd(x[it].x) || bf16x2_odd(x[it].y) || bf16x2_odd(x[it].z) || bf16x2_odd(x[it].w))) bad[rec] = 1;
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < kGatherSteps; ++it) {
    const int i = threadIdx.x + it * kGatherThreads, rec = i / per, c = i - rec * per;
    if (rec >= 16) break;
    const uint32_t instead = c < latent ? 0u : 0x7fff7fffu;
    dst[i] = bad[rec] ? make_uint4(instead, instead, instead, instead) : x[it];
  }
}

// What a CTA's roles need to know of one block: 256 queries of one request and one query head.
struct Block {
  int r, h, t0, mbeg;
  int rows_x[2], pf_x[2], pl_x[2], jlo_x[2], jhi_x[2];
  int kb, ntiles, lo, p_last;
  int at;            // place of key 0 in the built arrays (may be negative: keys before the first one needed are not there)
  // false: the block is beyond the request's queries (or the request is one that the folded kernel serves)
  __device__ bool init(int b, int nq, int nyb, const int* q_indptr, const int* kv_lens, const int2* plan, int window) {
    h = b % nq;
    const int y = (b / nq) % nyb;
    r = b / (nq * nyb);
    t0 = q_indptr[r];
    const int qlen = q_indptr[r + 1] - t0;
    // The blocks with the most keys (the last queries) come first, for all heads before any block with fewer.
    mbeg = (nyb - 1 - y) * BQ2;
    const int2 p = plan[r];
    if (mbeg >= qlen || p.y < 0) return false;
    at = p.y - p.x;
    const int pos0 = kv_lens[r] - qlen;
    int lo_x[2];
    rows_x[0] = min(BQ, qlen - mbeg);
    rows_x[1] = max(0, min(BQ, qlen - mbeg - BQ));
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      pf_x[x] = pos0 + mbeg + x * BQ;
      pl_x[x] = pf_x[x] + max(rows_x[x], 1) - 1;
      lo_x[x] = first_visible_key(pf_x[x], window, 0);
    }
    kb = lo_x[0] / BKV * BKV;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      jlo_x[x] = rows_x[x] > 0 ? (lo_x[x] / BKV * BKV - kb) / BKV : 0;
      jhi_x[x] = rows_x[x] > 0 ? (pl_x[x] - kb) / BKV + 1 : 0;
    }
    ntiles = max(jhi_x[0], jhi_x[1]);
    lo = lo_x[0];
    p_last = rows_x[1] > 0 ? pl_x[1] : pl_x[0];
    return true;
  }
  __device__ bool in_range(int x, int j) const { return j >= jlo_x[x] && j < jhi_x[x]; }
};

constexpr int kWorkReaders = 11;             // who reads a drawn ticket: the two loader warps, the MMA thread, eight softmax warps

// NS: slices of 64 unrotated key numbers, and of values; a slice of rotated numbers stands beside them.
template <int NS>
struct Shape {
  static constexpr int QS = NS + 1;                       // slices of a query or key
  static constexpr int KG = QS == 3 ? 1 : QS;             // slices of a key stage
  static constexpr int KRING = QS == 3 ? 4 : 2;           // key stages
  static constexpr int GROUPS = QS / KG;                  // key stages that a tile takes
  static constexpr int HDV = 64 * NS;
  static constexpr uint32_t QTILE = QS * SUB, KSTAGE = KG * SUB, VTILE = NS * SUB;
  static constexpr size_t SMEM = 2 * (size_t)QTILE + KRING * (size_t)KSTAGE + kVStages * (size_t)VTILE + 1024;
};

template <int NS>
__global__ void __launch_bounds__(kThreads, 1) latent_prefill_tc_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_r,
    const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out, int out_stride, const int* __restrict__ q_indptr,
    const int* __restrict__ kv_lens, const int2* __restrict__ plan, int nq, int qw, int rank, float scale_log2,
    const __nv_bfloat16* __restrict__ gate, int gate_stride, int window, int nyb, int nblocks, int ticket_slot, int places, int* __restrict__ err) {
  pdl_launch_dependents();
  pdl_wait();
  typedef Shape<NS> S_;
  constexpr int QS = S_::QS, KG = S_::KG, KRING = S_::KRING, GROUPS = S_::GROUPS, HDV = S_::HDV;
  constexpr uint32_t QTILE = S_::QTILE, KSTAGE = S_::KSTAGE, VTILE = S_::VTILE;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = base;                              // 2 x QTILE
  unsigned char* k_s = base + 2 * QTILE;                  // KRING x KSTAGE
  unsigned char* v_s = k_s + KRING * KSTAGE;              // kVStages x VTILE
  __shared__ __align__(8) uint64_t q_full, q_empty, k_full[KRING], k_empty[KRING], v_full[kVStages], v_empty[kVStages], s_full[2],
      p_full[2], o_full[2], o_empty[2], work_full[2], work_empty[2];
  __shared__ int work_id[2];                             // the drawn block, -1: none left; -2: a block without queries
  __shared__ Block work_blk[2];                          // and its shape, worked out by the thread that drew it
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool first_has_queries = false;
  if (warp == kKeyWarp && lane == 0) first_has_queries = work_blk[0].init((int)blockIdx.x, nq, nyb, q_indptr, kv_lens, plan, window);
  if (threadIdx.x == 0) {
    mbar_init(smem_addr(&q_full), 1);
    mbar_init(smem_addr(&q_empty), 1);
    for (int i = 0; i < KRING; ++i) {
      mbar_init(smem_addr(&k_full[i]), 1);
      mbar_init(smem_addr(&k_empty[i]), 1);
    }
    for (int i = 0; i < kVStages; ++i) {
      mbar_init(smem_addr(&v_full[i]), 1);
      mbar_init(smem_addr(&v_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_addr(&s_full[i]), 1);
      mbar_init(smem_addr(&p_full[i]), 4);
      mbar_init(smem_addr(&o_full[i]), 1);
      mbar_init(smem_addr(&o_empty[i]), 4);
      mbar_init(smem_addr(&work_full[i]), 1);
      mbar_init(smem_addr(&work_empty[i]), kWorkReaders);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_addr(&tmem_base_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;              // columns: S of A, S of B, O of A, O of B (128 each)
  const volatile int* aborted = &abort_flag;

  auto wait_ticket = [&](int i) -> int {
    if (!mbar_wait_bounded(smem_addr(&work_full[i & 1]), (uint32_t)((i >> 1) & 1), aborted)) return -1;
    return work_id[i & 1];
  };
  auto release_ticket = [&](int i) { mbar_arrive(smem_addr(&work_empty[i & 1])); };

  if (warp >= 8) {
    reg_less<kRegsOther>();
    if (warp == kKeyWarp || warp == kValueWarp) {
      // One warp loads the keys, one the values: boxes of 16 keys x 64 numbers, one per lane.  The key warp's first lane also
      // draws the tickets.
      const bool keys = warp == kKeyWarp;
      const int c = lane & 7, sl = lane >> 3;              // sixteen keys of the tile, slice of the stage
      const int slices = keys ? KG : NS, ring = keys ? KRING : kVStages, groups = keys ? GROUPS : 1;
      int issued = 0;                                       // stages whose loads were issued, over all blocks
      int q_loads = 0;                                      // blocks whose Q was asked for
      bool ended = false;                                   // the terminal ticket is drawn
      for (int it = 0;; ++it) {
        if (keys && lane == 0) {
          int b = -1;
          if (it == 0) {
            b = first_has_queries ? (int)blockIdx.x : -2;
          } else if (it < 2 || mbar_wait_bounded(smem_addr(&work_empty[it & 1]), (uint32_t)(((it >> 1) & 1) ^ 1), aborted)) {
            if (!*aborted) {
              const unsigned int tk = draw_ticket(nblocks, ticket_slot);
              if (tk < (unsigned int)nblocks) b = (int)tk; else ended = true;
              if (b >= 0 && !work_blk[it & 1].init(b, nq, nyb, q_indptr, kv_lens, plan, window)) b = -2;
            }
          } else {
            abort_flag = 1;
          }
          work_id[it & 1] = b;
          asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(&work_full[it & 1])) : "memory");
        }
        __syncwarp();
        const int b = __shfl_sync(0xffffffffu, lane == 0 ? wait_ticket(it) : 0, 0);
        __syncwarp();
        Block blk;
        if (b >= 0) blk = work_blk[it & 1];
        __syncwarp();
        if (lane == 0 && b != -1) release_ticket(it);
        if (b == -1) break;
        if (b == -2) continue;
        if (keys && lane == 0) {
          // Q of this block, once the S products of the block before have read theirs
          bool free_q = q_loads == 0 || mbar_wait_bounded(smem_addr(&q_empty), (uint32_t)((q_loads - 1) & 1), aborted);
          if (!free_q) abort_flag = 1;
          if (free_q) {
            const int nload = blk.rows_x[1] > 0 ? 2 : 1;
            mbar_expect_tx(smem_addr(&q_full), (uint32_t)nload * QTILE);
            for (int x = 0; x < nload; ++x)
#pragma unroll
              for (int d = 0; d < QS; ++d)
                tma_load_2d(smem_addr(q_s + x * QTILE + d * SUB), &map_q, blk.h * qw + d * 64, blk.t0 + blk.mbeg + x * BQ, smem_addr(&q_full));
            ++q_loads;
          }
        }
        bool stop = false;
        for (int j = 0; j < blk.ntiles && !stop; ++j) {
          const int key0 = blk.kb + j * BKV + c * 16;
          const bool seen = key0 <= blk.p_last && key0 + 15 >= blk.lo;
          // Value rows that no query of the block sees meet P = 0, and zero times what an earlier block left there may be NaN: they are
          // loaded from behind the last place, which fills them with zeros.
          const bool on = sl < slices && (seen || !keys);
          const int n = __popc(__ballot_sync(0xffffffffu, on));      // boxes of a stage
          for (int g = 0; g < groups; ++g) {
            const int st = issued % ring;
            const uint32_t par = (uint32_t)((issued / ring) & 1);
            const uint32_t full = smem_addr(keys ? &k_full[st] : &v_full[st]);
            int go = 1;
            if (lane == 0) {
              if (!mbar_wait_bounded(smem_addr(keys ? &k_empty[st] : &v_empty[st]), par ^ 1, aborted)) {
                abort_flag = 1;
                go = 0;
              } else {
                mbar_expect_tx(full, (uint32_t)n * 2048u);
              }
            }
            go = __shfl_sync(0xffffffffu, go, 0);
            if (!go || *aborted) {
              stop = true;
              break;
            }
            if (on) {
              const int d = g * KG + sl;                    // the key's slice
              if (!keys) tma_load_2d(smem_addr(v_s + st * VTILE + sl * SUB + c * 2048), &map_v, blk.h * HDV + sl * 64, seen ? blk.at + key0 : places, full);
              else if (d == NS) tma_load_2d(smem_addr(k_s + st * KSTAGE + sl * SUB + c * 2048), &map_r, rank, blk.at + key0, full);
              else tma_load_2d(smem_addr(k_s + st * KSTAGE + sl * SUB + c * 2048), &map_k, blk.h * HDV + d * 64, blk.at + key0, full);
            }
            ++issued;
          }
        }
        if (stop) break;
      }
      if (keys && lane == 0 && !ended) {
        // a wait ran out: the tickets are still drawn to the end, so that the counter is back at zero for the next launch
        for (int i = 0; i <= nblocks; ++i)
          if (draw_ticket(nblocks, ticket_slot) >= (unsigned int)nblocks) break;
      }
      // No copy may still be in flight when the CTA ends.
      if (lane == 0) {
        if (keys && q_loads > 0) mbar_wait_plain(smem_addr(&q_full), (uint32_t)((q_loads - 1) & 1));
        for (int s2 = 0; s2 < ring && s2 < issued; ++s2) {
          const int last = (issued - 1 - s2) / ring * ring + s2;       // last load into stage s2
          mbar_wait_plain(smem_addr(keys ? &k_full[s2] : &v_full[s2]), (uint32_t)((last / ring) & 1));
        }
      }
    } else if (warp == kMmaWarp && lane == 0) {
      constexpr uint32_t idesc_s = idesc_bf16(BQ, BKV);                  // A and B K-major
      constexpr uint32_t idesc_pv = idesc_bf16(BQ, HDV) | (1u << 16);    // B (values) MN-major
      bool ok = true;
      int g0 = 0;                                                        // key tiles of the blocks before
      int q_uses = 0;                                                    // blocks whose Q was used
      int done_p[2] = {0, 0};                                            // P tiles of each query tile consumed so far, over all blocks
      int o_blocks[2] = {0, 0};                                          // blocks in which each query tile had rows
      for (int it = 0; ok; ++it) {
        const int b = wait_ticket(it);
        Block blk;
        if (b >= 0) blk = work_blk[it & 1];
        release_ticket(it);
        if (b == -1) break;
        if (b == -2) continue;
        ok = mbar_wait_bounded(smem_addr(&q_full), (uint32_t)(q_uses & 1), aborted);
        ++q_uses;
        int k_seen = 0;                                                  // stages of the tile at hand that are known to be full
        // S of query tile x for key tile j; the query tile that is last to read a stage hands it back
        auto issue_s = [&](int x, int j) -> bool {
          const bool last = x == 1 || !blk.in_range(1, j);
#pragma unroll
          for (int g = 0; g < GROUPS; ++g) {
            const int use = (g0 + j) * GROUPS + g, kst = use % KRING;
            if (g >= k_seen) {
              if (!mbar_wait_bounded(smem_addr(&k_full[kst]), (uint32_t)((use / KRING) & 1), aborted)) return false;
              k_seen = g + 1;
              tc_fence_after();
            }
#pragma unroll
            for (int s = 0; s < KG; ++s) {
              const uint64_t ad = smem_desc_sw128(smem_addr(q_s + x * QTILE + (g * KG + s) * SUB));
              const uint64_t bd = smem_desc_sw128(smem_addr(k_s + kst * KSTAGE + s * SUB));
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_bf16(tmem_base + (uint32_t)(x * BKV), ad + 2 * k, bd + 2 * k, idesc_s, (g | s | k) != 0 ? 1u : 0u);
            }
            if (last) umma_commit(smem_addr(&k_empty[kst]));
          }
          umma_commit(smem_addr(&s_full[x]));
          return true;
        };
        // Every key tile is read by one of the query tiles at least: A's range starts the sequence and B's ends it (or A's, without
        // rows in B), and the two overlap or touch.
        if (ok) {
          if (blk.in_range(0, 0)) ok = issue_s(0, 0);
          if (ok && blk.in_range(1, 0)) ok = issue_s(1, 0);
          if (ok && blk.ntiles == 1) umma_commit(smem_addr(&q_empty));        // every S of the block is issued
        }
        int first_pv[2] = {1, 1};
        for (int j = 0; j < blk.ntiles && ok; ++j) {
          const int vst = (g0 + j) % kVStages;
          bool v_ready = false;
          k_seen = 0;
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            if (blk.in_range(x, j)) {
              if (!mbar_wait_bounded(smem_addr(&p_full[x]), (uint32_t)(done_p[x] & 1), aborted)) { ok = false; break; }
              if (!v_ready) {
                if (!mbar_wait_bounded(smem_addr(&v_full[vst]), (uint32_t)(((g0 + j) / kVStages) & 1), aborted)) { ok = false; break; }
                v_ready = true;
              }
              if (first_pv[x] && o_blocks[x] > 0) {
                // the block before has taken its O out of tensor memory
                if (!mbar_wait_bounded(smem_addr(&o_empty[x]), (uint32_t)((o_blocks[x] - 1) & 1), aborted)) { ok = false; break; }
              }
              tc_fence_after();
#pragma unroll
              for (int kk = 0; kk < 8; ++kk) {
                const uint64_t bd = smem_desc_mn_sw128(smem_addr(v_s + vst * VTILE + kk * 2048), SUB);
                umma_bf16_a_tmem(tmem_base + (uint32_t)(256 + x * 128), tmem_base + (uint32_t)(x * BKV + kk * 8), bd, idesc_pv,
                                 (first_pv[x] && kk == 0) ? 0u : 1u);
              }
              first_pv[x] = 0;
              ++done_p[x];
              if (j + 1 == blk.jhi_x[x]) {
                umma_commit(smem_addr(&o_full[x]));
                ++o_blocks[x];
              }
            }
            // S of the next key tile goes over this P: the tensor core runs them in the order issued
            if (blk.in_range(x, j + 1)) {
              if (!issue_s(x, j + 1)) { ok = false; break; }
            }
          }
          if (!ok) break;
          umma_commit(smem_addr(&v_empty[vst]));                  // tile j's values are read by what was issued so far
          if (j + 2 == blk.ntiles) umma_commit(smem_addr(&q_empty));    // every S of the block is issued
        }
        g0 += blk.ntiles;
      }
      if (!ok) abort_flag = 1;
    }
  } else {
    reg_more<kRegsSoftmax>();
    const int x = warp >> 2;                                   // query tile of this warp group
    const int row = (warp & 3) * 32 + lane;                    // query row of the tile = TMEM lane
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tmem_s = tmem_base + (uint32_t)(x * BKV), tmem_o = tmem_base + (uint32_t)(256 + x * 128);
    bool ok = true;
    int n_all = 0;                                             // S tiles of this query tile taken so far, over all blocks
    int o_all = 0;                                             // blocks in which this query tile had rows
    for (int it = 0; ok; ++it) {
      int b = lane == 0 ? wait_ticket(it) : 0;
      b = __shfl_sync(0xffffffffu, b, 0);
      __syncwarp();
      Block blk;
      if (b >= 0) blk = work_blk[it & 1];
      __syncwarp();
      if (lane == 0) release_ticket(it);
      if (b == -1) break;
      if (b == -2) continue;
      const int p_first = blk.pf_x[x], pl = blk.pl_x[x];
      const int jlo = blk.jlo_x[x], jhi = blk.jhi_x[x], rows_here = blk.rows_x[x];
      const int p_row = min(p_first + row, pl);
      const int lo_row = window > 0 ? p_row - window + 1 : 0;
      float m_used = -INFINITY, l = 0.f;
      int n = 0;
      for (int j = jlo; j < jhi; ++j) {
        const int k0 = blk.kb + j * BKV;
        const bool full_tile = k0 + BKV - 1 <= p_first && (window <= 0 || k0 >= pl - window + 1);
        bool ready = mbar_wait_bounded(smem_addr(&s_full[x]), (uint32_t)(n_all & 1), aborted);
        if (__any_sync(0xffffffffu, !ready)) { ok = false; break; }
        tc_fence_after();
        uint32_t sv[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tmem_s + lane_addr + (uint32_t)(c * 32), sv[c]);
        tmem_ld_wait();
        float mx;
        {
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
          if (full_tile) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(sv[c][i]));
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const int kj = k0 + c * 32 + i;
                if (!(kj <= p_row && kj >= lo_row)) sv[c][i] = 0xff800000u;      // -inf: masked for good
                m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(sv[c][i]));
              }
          }
          mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * scale_log2;
        }
        const float m_new = fmaxf(m_used, mx);
        const bool grow = m_new > m_used + kRescaleStep;        // also true when the row sees its first key
        const float f = (grow && m_used != -INFINITY) ? exp2f(m_used - m_new) : 1.0f;
        if (grow) m_used = m_new;
        const float m_eff = m_used == -INFINITY ? 0.f : m_used;
        l *= f;
        // O may be rescaled here without a wait: S of this key tile was issued after P.V of the tile before
        const bool rescale = n > 0 && __any_sync(0xffffffffu, f != 1.0f);
        if (rescale) {
#pragma unroll 1
          for (int c = 0; c < HDV / 32; ++c) {
            uint32_t v[32];
            tmem_ld32(tmem_o + lane_addr + (uint32_t)(c * 32), v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
            tmem_st32(tmem_o + lane_addr + (uint32_t)(c * 32), v);
          }
        }
        float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          uint32_t packed[32];                                  // 64 keys of this row as bfloat16 pairs
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float e0 = ex2_fast(fmaf(__uint_as_float(sv[2 * h2 + c][i]), scale_log2, -m_eff));
              const float e1 = ex2_fast(fmaf(__uint_as_float(sv[2 * h2 + c][i + 1]), scale_log2, -m_eff));
              l4[(i >> 1) & 3] += e0 + e1;
              packed[c * 16 + (i >> 1)] = pack_bf16x2(e0, e1);
            }
          tmem_st32(tmem_s + lane_addr + (uint32_t)(h2 * 32), packed);
        }
        tmem_st_wait();
        l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_addr(&p_full[x]));
        ++n;
        ++n_all;
      }
      if (ok && n > 0) {
        const bool ready = mbar_wait_bounded(smem_addr(&o_full[x]), (uint32_t)(o_all & 1), aborted);
        if (__any_sync(0xffffffffu, !ready)) ok = false;
      }
      if (ok && n > 0) {
        ++o_all;
        tc_fence_after();
        const float inv = 1.0f / l;
        const size_t t = (size_t)(blk.t0 + blk.mbeg + x * BQ + row);
        __nv_bfloat16* orow = out + t * out_stride + blk.h * HDV;
#pragma unroll 1
        for (int c = 0; c < HDV / 32; ++c) {
          uint32_t v[32];
          tmem_ld32(tmem_o + lane_addr + (uint32_t)(c * 32), v);
          tmem_ld_wait();
          if (c == HDV / 32 - 1) {
            // O is in registers: the next block's first product with the values may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&o_empty[x]));
          }
          if (row < rows_here) {
            uint32_t p[16];
            const __nv_bfloat16* gv = gate ? gate + t * gate_stride + blk.h * HDV + c * 32 : nullptr;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float a = __uint_as_float(v[2 * i]) * inv, b2 = __uint_as_float(v[2 * i + 1]) * inv;
              if (gate) {
                a *= __fdividef(1.0f, 1.0f + __expf(-__bfloat162float(gv[2 * i])));
                b2 *= __fdividef(1.0f, 1.0f + __expf(-__bfloat162float(gv[2 * i + 1])));
              }
              p[i] = pack_bf16x2(a, b2);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
              reinterpret_cast<uint4*>(orow + c * 32)[i] = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
          }
        }
      }
    }
    if (!ok && lane == 0) abort_flag = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && abort_flag && err) atomicExch(err, 5);
}

template <int NS>
int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mr, const CUtensorMap& mv, void* out, int out_stride, const int* q_indptr,
           const int* kv_lens, const int* plan, int nq, int qw, int rank, float scale, const void* gate, int gate_stride, int window, int rows,
           int max_q_len, int places, int* err, cudaStream_t s) {
  auto kernel = latent_prefill_tc_kernel<NS>;
  constexpr size_t smem = Shape<NS>::SMEM;
  static SharedLimit limit;
  const cudaError_t raised = limit.raise((const void*)kernel, smem);
  if (raised != cudaSuccess) return (int)raised;
  const int nyb = (max_q_len + BQ2 - 1) / BQ2;
  const long long nblocks = (long long)nq * nyb * rows;
  if (nblocks > 0x3fffffffLL) return ARLE_E_UNSUPPORTED;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int ctas = (int)(nblocks < sms ? nblocks : sms);
  static std::atomic<unsigned int> launches{0};
  const int ticket_slot = (int)(launches++ % kTicketSlots);
  cudaError_t e = launch_kernel(kernel, dim3(ctas), dim3(kThreads), smem, s, 1, mq, mk, mr, mv, (__nv_bfloat16*)out, out_stride, q_indptr, kv_lens,
                                (const int2*)plan, nq, qw, rank, scale * 1.4426950408889634f, (const __nv_bfloat16*)gate, gate_stride, window, nyb,
                                (int)nblocks, ticket_slot, places, err);
  if (e != cudaSuccess) return (int)e;
  return launch_status();
}

}  // namespace

// plan: int32 [R][2].
ARLE_API int arle_latent_plan(const int* q_indptr, const int* kv_lens, int R, int least, int most, int floor, int room, int window, int* plan,
                              cudaStream_t s) {
  if (R <= 0) return 0;
  launch_early(latent_plan_kernel, dim3(1), dim3(32), 0, s, 1, q_indptr, kv_lens, R, least, most, floor, room, window, (int2*)plan);
  return launch_status();
}

// cache bfloat16 [pages, 1, page_size, rank + dr]; out [places, rank + max(dr, 8)], places: a group's, R and the arrays by row: its
// rows.  rank up to 512, dr up to 64, multiples of 8.
ARLE_API int arle_latent_gather(const void* cache, const int* block_table, int bt_stride, const int* kv_lens, const int* plan, int R, int page_size,
                                int rank, int dr, void* out, int places, cudaStream_t s) {
  if (R <= 0 || places <= 0) return 0;
  if (page_size % 16 || rank <= 0 || rank > 512 || rank % 8 || dr < 0 || dr > 64 || dr % 8 || places % 16 || ((uintptr_t)cache & 15) ||
      ((uintptr_t)out & 15))
    return ARLE_E_UNSUPPORTED;
  launch_early(latent_gather_kernel, dim3(places / 16), dim3(kGatherThreads), 0, s, 1, (const __nv_bfloat16*)cache, block_table, bt_stride, kv_lens,
                (const int2*)plan, R, page_size, rank, rank + dr, rank + gathered_tail(dr), (__nv_bfloat16*)out);
  return launch_status();
}

// q bfloat16 [num_tokens, heads * (dn + dr)] (any row stride that is a multiple of 8): a head's unrotated numbers, then its rotated ones.
// keys [places, heads * dn] and values [places, heads * dn] (row stride kv_stride), records [places, rank + max(dr, 8)]: the built arrays
// and the gathered records of a group; rows, q_indptr, kv_lens and plan: the group's.  out [num_tokens, heads * dn] (row stride out_stride): only the plan's rows are written.
// dn 64 or 128, dr 0 or a multiple of 8 up to 64.
ARLE_API int arle_latent_prefill_tc(const void* q, int q_stride, int num_tokens, const void* keys, const void* values, int kv_stride,
                                    const void* records, int places, void* out, int out_stride, const int* q_indptr, const int* kv_lens,
                                    const int* plan, int heads, int dn, int dr, int rank, float scale, const void* gate, int gate_stride,
                                    int window, int rows, int max_q_len, int* err, cudaStream_t s) {
  if (rows <= 0 || max_q_len <= 0 || places <= 0) return 0;
  if ((dn != 64 && dn != 128) || dr < 0 || dr > 64 || dr % 8 || rank % 8 || heads <= 0 || q_stride % 8 || kv_stride % 8 || out_stride % 8 ||
      (((uintptr_t)q | (uintptr_t)keys | (uintptr_t)values | (uintptr_t)records | (uintptr_t)out) & 15))
    return ARLE_E_UNSUPPORTED;
  CUtensorMap mq, mk, mr, mv;
  int rc = tensor_map_2d_bf16(q, num_tokens, heads * (dn + dr), q_stride, BQ, &mq);
  if (!rc) rc = tensor_map_2d_bf16(keys, places, heads * dn, kv_stride, 16, &mk);
  if (!rc) rc = tensor_map_2d_bf16(values, places, heads * dn, kv_stride, 16, &mv);
  if (!rc) rc = tensor_map_2d_bf16(records, places, rank + gathered_tail(dr), rank + gathered_tail(dr), 16, &mr);
  if (rc) return rc;
  if (dn == 128)
    return launch<2>(mq, mk, mr, mv, out, out_stride, q_indptr, kv_lens, plan, heads, dn + dr, rank, scale, gate, gate_stride, window, rows, max_q_len,
                     places, err, s);
  return launch<1>(mq, mk, mr, mv, out, out_stride, q_indptr, kv_lens, plan, heads, dn + dr, rank, scale, gate, gate_stride, window, rows, max_q_len,
                   places, err, s);
}
