// Attention forward for inference: packed mixed-mask attention as in attn_fwd_sm100.cu (same tile lists, same mask bits,
// head_dim 128, bf16 in / fp32 softmax), for callers that want the output only.
//
// Per key tile: S = Q K^T and O += P V run on the tensor cores (tcgen05.mma, S and O of two query tiles in TMEM), the
// softmax warps read S with tcgen05.ld, apply the mask only on "partial" tiles, store P (bf16) to tensor memory as the A
// operand of the second product and rescale O in TMEM when a row maximum moved.  K and V tiles come through TMA rings; V
// is consumed MN-major straight from its row-major tile.
//
// The kernel of attn_fwd_sm100.cu stays for callers that want the row log-sum-exp, i.e. a backward pass: the rows of a
// warp decide together when the running maximum moves, and with 16 rows to a warp instead of 32 P is rounded at other
// scales.  Outputs are as close to fp32 softmax, but their bits differ, while every bf16 value of a training step is the
// same as before this kernel came (only sums by fp32 atomics vary: loss, gains, biases).  That holds for one step: those
// sums make the second differ from run to run (first-layer gradients by up to 1e-2), with either kernel.  Made to decide
// over 32 rows and to add row sums in the same order (bit-equal), this kernel is as slow as that one (full 8192: 1037 us).
#include "attn_common.cuh"
#include "host_common.h"

namespace snu1 {
int encode_head_tmap(CUtensorMap* out, const void* base, long long rows, int heads, long long ld, int box_rows);

namespace attn_inf {

constexpr int BQ = 128;
constexpr int BKV = 128;
constexpr int HALF_BYTES = 128 * 64 * 2;   // one 64-column box of a 128-row tile
constexpr int TILE_BYTES = 2 * HALF_BYTES;  // 32 KB
constexpr int TMEM_COLS = 512;

// One CTA owns TWO 128-row query tiles (A, B) of one head.  Each tile has its own
// softmax warps, S accumulator, O accumulator and P buffer; they share every K / V
// tile that comes through TMA, which halves the L2 -> shared-memory traffic per FLOP and
// gives the tensor cores a second, independent stream of work while the other tile is in
// its exponentials.  warp 0: TMA, warp 1: MMA issue, warps 4..11: tile A, warps 12..19: tile B.
//
// A softmax warp owns 16 rows and reads S in the 16x256b shape (four threads per row), so a thread carries 64 scores
// instead of the 128 of the row-per-thread shape: four softmax warps per scheduler instead of two.
//
// Tensor memory is full (S and O of both tiles, 512 columns), so P_A lies over S_B and P_B over S_A: when a tile's
// probabilities are ready the other tile's scores have been read (the tiles run half a step apart), and the tile's own
// next scores can be computed meanwhile.  Against P in shared memory that takes 64 KB of writes and 64 KB of operand
// reads per step off the shared-memory port (384 -> 256 KB) and makes room for a third K and a second V stage.
//
// What bounds it: the issuing warp is busy all the time (clock stamps, per step of two tiles): the two S products, whose
// operands both come from shared memory, 100 clocks per 128x128x16 instead of 64, the two P V products 64 - 70, and
// 500 clocks of waits; the softmax of a tile takes 2,400 of the 3,400 clocks.  Exponentials on the FMA pipe (every
// fourth, degree-5 polynomial) only add instructions: 7.9 -> 9.1 ms at 32 K.
//   us (TFLOP/s), 32 / 8 heads     before (P in shared memory)     now
//   full 4096 x 4096                   373  (740)                  318  (865)
//   full 8192 x 8192                  1018 (1080)                  884 (1243)
//   causal 16384                      1989 (1106)                 1815 (1212)
//   causal 32001                      7700 (1090)                 7100 (1180)
struct FwdArgs {
  __nv_bfloat16* O;
  long long ldo;
  const TokMeta* meta_q;
  const TokMeta* meta_k;
  const int* pair_list;
  const int* pair_count;
  int nk;
  int Sq, Sk, Hq, Hkv;
  float scale_log2;
  int* status;
  const int* order;      // [pairs] pair indices, longest key list first; may be null
  const int* tile_slot;  // [nq][nk] slot of a partial pair's mask bits, -1 = none; may be null
  const uint4* bits_q;   // [slots][128 query rows] 128 key bits
};

// A counter in shared memory that only grows: unlike an mbarrier's parity it can be waited for by a tile that has skipped
// any number of the other tile's steps.
__device__ __forceinline__ void count_add(int* c) {
  asm volatile("red.release.cta.shared::cta.add.s32 [%0], 1;" ::"r"(smem_u32(c)) : "memory");
}
__device__ __forceinline__ bool count_wait(const int* c, int target, volatile int* abort_flag, int* status, int where) {
  const uint32_t a = smem_u32(c);
  uint64_t t0 = 0;
  for (uint32_t spins = 0;; ++spins) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    if (v >= target) return true;
    if ((spins & 0x3ff) == 32) {
      if (*abort_flag) return false;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > kLocalWaitNs) {
        *abort_flag = 1;
        report_status(status, kWaitTimeout, where);
        return false;
      }
    }
  }
}

constexpr int K_STAGES = 3, V_STAGES = 2;
constexpr int FWD_THREADS = 640;  // five warpgroups: {TMA, MMA, 2 idle}, two for the softmax of A, two for B

__global__ void __launch_bounds__(FWD_THREADS, 1)
    attn_infer_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const FwdArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                    // 2 tiles
  uint8_t* sK = sQ + 2 * TILE_BYTES;
  uint8_t* sV = sK + K_STAGES * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + V_STAGES * TILE_BYTES);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;                  // [K_STAGES]
  uint64_t* k_empty = k_full + K_STAGES;        // [K_STAGES]
  uint64_t* v_full = k_empty + K_STAGES;        // [V_STAGES]
  uint64_t* v_empty = v_full + V_STAGES;        // [V_STAGES]
  uint64_t* s_full = v_empty + V_STAGES;        // [2] per query tile
  uint64_t* s_empty = s_full + 2;               // [2]
  uint64_t* p_full = s_empty + 2;               // [2]
  uint64_t* pv_done = p_full + 2;               // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* drained = reinterpret_cast<int*>(tmem_slot + 2);   // [2] softmax warps that have read a score tile, all tiles so far

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < K_STAGES; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < V_STAGES; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], 8);
      mbar_init(&p_full[i], 8);
      mbar_init(&pv_done[i], 1);
    }
    *abort_flag = 0;
    drained[0] = drained[1] = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // part of the programmatic chain: set up while the rotary norm in front still runs, and the output product behind may start
  // on its weights.  The plan may be of the kernel in front too: nothing is read before the wait.  256 px image, 5 steps of 12
  // layers: 9.72 -> 9.41 ms.
  pdl_wait();
  pdl_trigger();

  // heads vary fastest, tiles follow ``order`` (most key tiles first): the CTAs with the longest lists start first
  // and the last wave holds only short ones; the query heads of one key/value head run next to each other
  const int head = blockIdx.x;
  const int pair = args.order != nullptr ? args.order[blockIdx.y] : gridDim.y - 1 - blockIdx.y;
  const int kvh = head / (args.Hq / args.Hkv);
  const int q0 = pair * 2 * BQ;
  const int n = args.pair_count[pair];
  const int* list = args.pair_list + (long long)pair * args.nk;
  // columns: S_A and P_B [0,128), S_B and P_A [128,256), O_A [256,384), O_B [384,512)

  // 640 threads start with 96 registers; the softmax warps need a few more (128 x 64 + 512 x 104 = 640 x 96)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
  if (warp == 0) {
    if (lane == 0 && n > 0) {
      mbar_expect_tx(q_full, 2 * TILE_BYTES);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        tma_load_3d(sQ + t * TILE_BYTES, &tmQ, q_full, 0, head, q0 + t * BQ);
        tma_load_3d(sQ + t * TILE_BYTES + HALF_BYTES, &tmQ, q_full, 64, head, q0 + t * BQ);
      }
      auto load_k = [&](int j) -> bool {
        const int s = j % K_STAGES;
        if (!mbar_wait(&k_empty[s], ((j / K_STAGES) & 1) ^ 1, abort_flag, args.status, 1)) return false;
        const int k0 = list_tile(list[j]) * BKV;
        mbar_expect_tx(&k_full[s], TILE_BYTES);
        tma_load_3d(sK + s * TILE_BYTES, &tmK, &k_full[s], 0, kvh, k0);
        tma_load_3d(sK + s * TILE_BYTES + HALF_BYTES, &tmK, &k_full[s], 64, kvh, k0);
        return true;
      };
      bool ok = load_k(0);
      for (int j = 0; j < n && ok; ++j) {
        if (j + 1 < n) ok = load_k(j + 1);
        if (!ok) break;
        const int s = j % V_STAGES;
        if (!mbar_wait(&v_empty[s], ((j / V_STAGES) & 1) ^ 1, abort_flag, args.status, 1)) break;
        const int k0 = list_tile(list[j]) * BKV;
        mbar_expect_tx(&v_full[s], TILE_BYTES);
        tma_load_3d(sV + s * TILE_BYTES, &tmV, &v_full[s], 0, kvh, k0);
        tma_load_3d(sV + s * TILE_BYTES + HALF_BYTES, &tmV, &v_full[s], 64, kvh, k0);
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the list and one elected lane issues (see mbar_ready in attn_common.cuh).
    if (n > 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_pv = make_idesc_bf16(128, 128, false, true);
      const uint64_t q_desc = make_smem_desc(smem_u32(sQ), 0, 1024);
      const uint64_t k_desc = make_smem_desc(smem_u32(sK), 0, 1024);
      const uint64_t v_desc = make_smem_desc(smem_u32(sV), HALF_BYTES, 1024);
      bool ok = mbar_wait(q_full, 0, abort_flag, args.status, 3);   // this lane's; see mbar_wait_warp
      int s_cnt[2] = {0, 0};   // S products issued per query tile
      int pv_cnt[2] = {0, 0};  // PV products issued per query tile
      auto issue_s = [&](int entry, int j, int t) {
        if (((entry >> (24 + 2 * t)) & 3) != kTileSkip) {
          // the softmax warps must have drained the previous S of this tile
          ok &= mbar_wait(&s_empty[t], (s_cnt[t] & 1) ^ 1, abort_flag, args.status, 2);
          tc_fence_after();
          const uint64_t qd = q_desc + t * (TILE_BYTES >> 4), kd = k_desc + (j % K_STAGES) * (TILE_BYTES >> 4);
          __syncwarp();
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              constexpr uint32_t half = HALF_BYTES >> 4;
              const uint32_t off = (k >> 2) * half + (k & 3) * 2;
              umma_bf16_ss(tmem_base + t * 128, qd + off, kd + off, idesc_s, k > 0 ? 1u : 0u);
            }
            umma_commit(&s_full[t]);
          }
          __syncwarp();
          ++s_cnt[t];
        }
      };
      auto issue_pv = [&](int entry, int j, int t) {
        if (((entry >> (24 + 2 * t)) & 3) != kTileSkip) {
          ok &= mbar_wait(&p_full[t], pv_cnt[t] & 1, abort_flag, args.status, 2);
          tc_fence_after();
          const uint64_t vd = v_desc + (j % V_STAGES) * (TILE_BYTES >> 4);
          const uint32_t p_tmem = tmem_base + (t ^ 1) * 128;      // in the other tile's score columns
          const uint32_t acc0 = pv_cnt[t] > 0 ? 1u : 0u;
          __syncwarp();
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              umma_bf16_ts(tmem_base + 256 + t * 128, p_tmem + k * 8, vd + k * (2048 >> 4), idesc_pv, k > 0 ? 1u : acc0);
            umma_commit(&pv_done[t]);
          }
          __syncwarp();
          ++pv_cnt[t];
        }
      };
      auto release = [&](uint64_t* bar) {
        if (elect_one()) umma_commit(bar);
        __syncwarp();
      };
      // Order: S_A(j+1) PV_A(j) S_B(j+1) PV_B(j).  The tensor pipe runs the products in this order, so S_B(j+1) only
      // overwrites P_A(j) once PV_A(j) has read it, and S_A(j+2) P_B(j); the softmax warps see to it that a P is only
      // stored over an S that has been read.  The two tiles run half a step apart: one takes exponentials while the
      // other loads, reduces and stores.
      int e = list[0], e1 = n > 1 ? list[1] : 0;      // entries of this step and the next (read a step ahead)
      ok &= mbar_wait(&k_full[0], 0, abort_flag, args.status, 3);
      issue_s(e, 0, 0);
      issue_s(e, 0, 1);
      release(&k_empty[0]);
      if (n > 1) ok &= mbar_wait(&k_full[1], 0, abort_flag, args.status, 3);
      ok &= mbar_wait(&v_full[0], 0, abort_flag, args.status, 3);
      for (int j = 0; j < n; ++j) {      // the whole list also after a time-out
        const bool more = j + 1 < n;
        const int e2 = j + 2 < n ? list[j + 2] : 0;
        if (more) issue_s(e1, j + 1, 0);
        issue_pv(e, j, 0);
        if (more) {
          issue_s(e1, j + 1, 1);
          release(&k_empty[(j + 1) % K_STAGES]);
        }
        issue_pv(e, j, 1);
        if (more) {
          release(&v_empty[j % V_STAGES]);
          // the next step's operands, waited for while the products just issued run
          if (j + 2 < n) ok &= mbar_wait(&k_full[(j + 2) % K_STAGES], ((j + 2) / K_STAGES) & 1, abort_flag, args.status, 3);
          ok &= mbar_wait(&v_full[(j + 1) % V_STAGES], ((j + 1) / V_STAGES) & 1, abort_flag, args.status, 3);
        }
        e = e1;
        e1 = e2;
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ------------------------------ softmax --------------------------------
    // A warp owns 16 rows; its threads hold columns 2 (lane % 4) + 8 i + {0, 1} of rows lane / 4 and lane / 4 + 8.
    const int t = (warp - 4) >> 3;   // query tile of this warpgroup
    const int base = (warp & 3) * 32 + ((warp - 4) >> 2 & 1) * 16;   // first row == first TMEM lane
    const int q2 = (lane & 3) * 2;
    const int rloc[2] = {base + (lane >> 2), base + (lane >> 2) + 8};
    const int row0 = q0 + t * BQ;
    const uint32_t lane_sel = (uint32_t)base << 16;
    const uint32_t tmem_S = tmem_base + t * 128 + lane_sel;
    const uint32_t tmem_O = tmem_base + 256 + t * 128 + lane_sel;
    const uint32_t tmem_P = tmem_base + (t ^ 1) * 128 + lane_sel;   // over the other tile's scores
    uint8_t* sOt = sQ + t * TILE_BYTES;     // output rows leave through the query tile's buffer
    // stmatrix: matrices (rows 0-7, chunk i) (rows 8-15, i) (rows 0-7, i + 1) (rows 8-15, i + 1), i even
    const uint32_t st_row = smem_u32(sOt) + (base + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128;
    const uint32_t st_chunk = (uint32_t)((lane >> 4) ^ (lane & 7)) << 4;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    const float sc = args.scale_log2;
    bool ok = true;
    int cnt = 0;  // key tiles this query tile has processed
    int next = n > 0 ? list[0] : 0;          // read a step ahead
    // score tiles of the other query tile that are issued before PV_t(j): key tiles 0 .. j of B for A, 0 .. j + 1 of A for B
    int other = t == 1 && ((next >> 24) & 3) != kTileSkip;
    for (int j = 0; j < n; ++j) {        // the whole list also after a time-out, see mbar_wait_warp
      const int entry = next;
      next = j + 1 < n ? list[j + 1] : 0;
      other += t == 0 ? ((entry >> 26) & 3) != kTileSkip : ((next >> 24) & 3) != kTileSkip;
      const int cls_t = (entry >> (24 + 2 * t)) & 3;
      if (cls_t == kTileSkip) continue;
      ok &= mbar_wait(&s_full[t], cnt & 1, abort_flag, args.status, 5);
      tc_fence_after();
      float sv[2][32];   // [columns 0-63, 64-127][4 i + 2 row + e]
      {
        uint32_t r0[32], r1[32];
        tmem_ld_16x256b_x8(tmem_S, r0);
        tmem_ld_16x256b_x8(tmem_S + 64, r1);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          sv[0][c] = __uint_as_float(r0[c]);
          sv[1][c] = __uint_as_float(r1[c]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&s_empty[t]);
        count_add(&drained[t]);
      }
      if (cls_t != kTileFull) {
        const int slot =
            args.tile_slot != nullptr ? __ldg(args.tile_slot + (long long)(2 * pair + t) * args.nk + list_tile(entry)) : -1;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uint32_t w[4];
          if (slot >= 0) {
            const uint4 u = __ldg(args.bits_q + (long long)slot * 128 + rloc[r]);
            w[0] = u.x;
            w[1] = u.y;
            w[2] = u.z;
            w[3] = u.w;
          } else {
            const int k0 = list_tile(entry) * BKV, row = row0 + rloc[r];
            const TokMeta mq = row < args.Sq ? args.meta_q[row] : TokMeta{-1, 0, 0, 0};
            mask_words_by_rule<4>(mq, args.meta_k + k0, args.Sk - k0, true, w);
          }
          // Left of a causal diagonal (and inside an image block) a 32-key word is all ones for every row of the warp:
          // no per-element test there.
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (__all_sync(0xffffffffu, w[g] == 0xffffffffu)) continue;
            const uint32_t x = w[g] >> q2;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
              for (int e = 0; e < 2; ++e)
                if (!((x >> (8 * i + e)) & 1u)) sv[g >> 1][((g & 1) * 4 + i) * 4 + 2 * r + e] = -INFINITY;
            }
          }
        }
      }
      float mx[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float m0 = fmaxf(sv[0][2 * r], sv[0][2 * r + 1]), m1 = fmaxf(sv[1][2 * r], sv[1][2 * r + 1]);
#pragma unroll
        for (int i = 1; i < 8; ++i) {
          m0 = max3(m0, sv[0][4 * i + 2 * r], sv[0][4 * i + 2 * r + 1]);
          m1 = max3(m1, sv[1][4 * i + 2 * r], sv[1][4 * i + 2 * r + 1]);
        }
        mx[r] = fmaxf(m0, m1);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      }
      // Lazy rescaling: the running maximum only moves when some row of the warp outgrows it by more
      // than 2^8 (in the exponent domain); until then the exponentials are taken against the stale
      // maximum (values up to 256, exact enough in fp32 / bf16) and the accumulator O is left alone.
      // (also true for the first finite maximum, m = -inf)
      const bool rescale = __any_sync(0xffffffffu, mx[0] * sc > m[0] * sc + 8.f || mx[1] * sc > m[1] * sc + 8.f);
      float alpha[2];
      uint64_t nb2[2], acc[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m_new = rescale ? fmaxf(m[r], mx[r]) : m[r];
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        alpha[r] = rescale ? fast_exp2((m[r] - m_use) * sc) : 1.f;
        m[r] = m_new;
        nb2[r] = pack_f32x2(-m_use * sc, -m_use * sc);
        acc[r][0] = acc[r][1] = 0ull;
      }
      const uint64_t sc2 = pack_f32x2(sc, sc);
      uint32_t pk[32];      // probabilities, bf16 pairs: [2 (8-column group) + row]
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float x, y;
            unpack_f32x2(fma_f32x2(pack_f32x2(sv[h][4 * i + 2 * r], sv[h][4 * i + 2 * r + 1]), sc2, nb2[r]), x, y);
            x = fast_exp2(x);
            y = fast_exp2(y);
            acc[r][i & 1] = add_f32x2(acc[r][i & 1], pack_f32x2(x, y));
            pk[16 * h + 2 * i + r] = pack_bf16x2(x, y);
          }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float s0, s1;
        unpack_f32x2(add_f32x2(acc[r][0], acc[r][1]), s0, s1);
        l[r] = l[r] * alpha[r] + (s0 + s1);      // of this thread's columns; summed over the four threads at the end
      }
      if (cnt > 0) ok &= mbar_wait(&pv_done[t], (cnt - 1) & 1, abort_flag, args.status, 5);
      // the other tile's warps have read the scores that P goes over
      ok &= count_wait(&drained[t ^ 1], 8 * other, abort_flag, args.status, 5);
      tc_fence_after();
      tmem_st_16x128b_x16(tmem_P, pk);
      if (cnt > 0 && rescale) {
        const uint64_t al0 = pack_f32x2(alpha[0], alpha[0]), al1 = pack_f32x2(alpha[1], alpha[1]);
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t r[32];
          tmem_ld_16x256b_x8(tmem_O + c * 64, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float y0, y1;
            unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), (i & 2) ? al1 : al0),
                         y0, y1);
            r[i] = __float_as_uint(y0);
            r[i + 1] = __float_as_uint(y1);
          }
          tmem_st_16x256b_x8(tmem_O + c * 64, r);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[t]);
      ++cnt;
    }
    // Output rows leave through this warp's rows of the query tile's buffer (no product reads it any more), so that 16
    // lanes store one row's 256 bytes.
    if (cnt > 0) ok &= mbar_wait(&pv_done[t], (cnt - 1) & 1, abort_flag, args.status, 5);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
      }
      const float inv[2] = {l[0] > 0.f ? 1.f / l[0] : 0.f, l[1] > 0.f ? 1.f / l[1] : 0.f};
      if (cnt > 0) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tmem_ld_16x256b_x8(tmem_O + h * 64, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            uint32_t p[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              p[e] = pack_bf16x2(__uint_as_float(r[4 * i + 2 * e]) * inv[e & 1], __uint_as_float(r[4 * i + 2 * e + 1]) * inv[e & 1]);
            stmatrix_x4(st_row + h * HALF_BYTES + (st_chunk ^ (i << 4)), p[0], p[1], p[2], p[3]);
          }
        }
        __syncwarp();
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = base + 2 * i + (lane >> 4), c = lane & 15;
        if (row0 + r < args.Sq)
          *reinterpret_cast<uint4*>(args.O + (long long)(row0 + r) * args.ldo + head * 128 + c * 8) =
              cnt > 0 ? *reinterpret_cast<const uint4*>(sOt + (c >> 3) * HALF_BYTES + swz128_offset(r, c & 7))
                      : make_uint4(0, 0, 0, 0);       // no key tile at all for this query tile
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) {
      }
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

constexpr int FWD_SMEM = (2 + K_STAGES + V_STAGES) * TILE_BYTES + 256 + 1024;

}  // namespace attn_inf

int launch_attn_infer(const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv, void* o,
                      long long ldo, const void* meta_q, const void* meta_k, const int* pair_list, const int* pair_count,
                      int Sq, int Sk, int Hq, int Hkv, float scale, const int* tile_slot, const void* bits_q,
                      const int* pair_order, cudaStream_t st) {
  using namespace attn_inf;
  if ((reinterpret_cast<uintptr_t>(o) & 15) != 0) {
    set_last_error("attn_fwd: the output must be 16-byte aligned");
    return kHostBadArg;
  }
  CUtensorMap tmQ, tmK, tmV;
  int rc;
  if ((rc = encode_head_tmap(&tmQ, q, Sq, Hq, ldq, 128)) != kHostOk) return rc;
  if ((rc = encode_head_tmap(&tmK, k, Sk, Hkv, ldk, 128)) != kHostOk) return rc;
  if ((rc = encode_head_tmap(&tmV, v, Sk, Hkv, ldv, 128)) != kHostOk) return rc;
  FwdArgs a;
  a.O = (__nv_bfloat16*)o;
  a.ldo = ldo;
  a.meta_q = (const TokMeta*)meta_q;
  a.meta_k = (const TokMeta*)meta_k;
  a.pair_list = pair_list;
  a.pair_count = pair_count;
  a.nk = (Sk + 127) / 128;
  a.Sq = Sq;
  a.Sk = Sk;
  a.Hq = Hq;
  a.Hkv = Hkv;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.status = device_status_word();
  a.tile_slot = bits_q != nullptr ? tile_slot : nullptr;
  a.bits_q = (const uint4*)bits_q;
  a.order = pair_order;
  const int nq = (Sq + 127) / 128;
  SNU1_CUDA_CHECK(cudaFuncSetAttribute(attn_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM));
  SNU1_CUDA_CHECK(launch_pdl(attn_infer_kernel, dim3(Hq, (nq + 1) / 2), dim3(FWD_THREADS), FWD_SMEM, st, tmQ, tmK, tmV, a));
  return kHostOk;
}

}  // namespace snu1
