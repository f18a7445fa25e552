// gemm_small: y[M,N] = x[M,K] w[N,K]^T for a few rows of x (text decoding, short prompts, thumbnails), where the
// product is a stream of weights: up to 128 rows, and up to 1024 of an inference engine while the tiles are one wave (the rule and
// both of its sides stand in launch_gemm).
//
// The roles of the operands are swapped: 128 rows of w are the M side of tcgen05.mma and the rows of x the N side
// (16 .. 128), so no tensor-core row is spent on padding rows of x and the accumulator is [128 weight rows][rows
// of x] in tensor memory.  What bounds it is the stream of w from HBM: the 128 x 64 weight tiles go through a ring of
// TMA stages, and the reduction is split over the CTAs of a cluster so that (N / 128) x split CTAs, two per SM,
// keep the whole chip loading.  The partial sums meet in shared memory: every CTA owns a part of the rows of x and
// adds the cluster's partials for it in a fixed order (distributed shared memory, no atomics, deterministic).
//
// Programmatic dependent launch: the kernel is set up while the one in front of it (a norm, an attention) is still
// running, and reads nothing before griddepcontrol.wait unless the caller says that no kernel of the running chain
// writes w (``w_static``: the layers of an inference engine); then the ring is filled with weights before the wait.
//
// Measured (weights cold in L2, one launch in a chain, us; before = the 256 x 256 pair kernel, of whose 16 - 96 tiles
// these shapes fill a fraction of the chip; floor = weight bytes at 6.54 TB/s; 24576 with SwiGLU, 4096 with a residual, 151936
// with an fp32 result and without w_static):
//   N x K            rows 1: before  now  floor    rows 24: before  now    rows 128: before  now
//   6144 x 4096             27.8   11.0    7.7              27.6   12.7              29.0   16.2
//   4096 x 4096             27.4    8.4    5.1              27.5    9.6              27.6   13.0
//   24576 x 4096            63.4   34.3   30.8              54.1   35.4              56.1   42.7
//   4096 x 12288            66.5   17.3   15.4              66.3   19.7              66.5   24.2
//   151936 x 4096          335.5  185.1  190.3             263.5  197.0             280.8  253.5
// Registers: 86 and 88 for 16 and 32 rows, 148 with SwiGLU, 166 - 168 for 64 and 128 rows (two CTAs of 192 threads have 168); no spills.
#include <string.h>

#include <mutex>
#include <type_traits>

#include "host_common.h"
#include "sm100_common.cuh"

namespace snu1 {
namespace gsmall {

constexpr int BW = 128;                    // weight rows per tile (M of the instruction)
constexpr int BK = 64;
constexpr int W_STAGE = BW * BK * 2;       // 16 KB
constexpr int NUM_THREADS = 192;           // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue

// DEEP: one CTA per SM with the whole shared memory as its ring, for grids that do not fill the chip twice anyway.
template <int TN, bool DEEP>
struct Cfg {
  static constexpr int X_STAGE = TN * BK * 2;
  static constexpr int STAGE = W_STAGE + X_STAGE;
  static constexpr int STAGES = (TN <= 16 ? 6 : TN <= 32 ? 5 : TN <= 64 ? 4 : 3) * (DEEP ? 2 : 1);
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static constexpr int TMEM = TN < 32 ? 32 : TN;
  static_assert(TN * BW * 4 <= STAGES * STAGE, "partial sums reuse the ring");
};

struct Args {
  int M, N, K;
  int split;          // CTAs of a cluster = parts of the reduction
  void* C;
  long long ldc;
  int f32_out;
  const __nv_bfloat16* residual;
  long long ldr;
  float alpha;
  int w_static;       // w may be read before the preceding kernel has finished
  const int* tile_group;   // experts: weight set of row tile blockIdx.y (negative: unused tile); null: one weight set
  int w_rows;         // rows of w per weight set
  int x_shared;       // experts: every tile reads rows 0 .. of x (one row that all of them share)
  int* status;
};

// SWIGLU: w holds args.N gate rows and then as many up rows; a tile is 64 of each and gives 64 columns of
// silu(gate) * up (both rounded to bf16 first, as when the projection was stored).
template <int TN, bool SWIGLU, bool DEEP>
__global__ void __launch_bounds__(NUM_THREADS, 2)
    gemm_small_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                      const Args args) {
  using C = Cfg<TN, DEEP>;
  extern __shared__ uint8_t smem_raw[];
  // same window offset in every CTA of the cluster: the partial sums are read at this CTA's own offsets
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::STAGES;
  uint64_t* acc_full = bars + 2 * C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  constexpr int CN = SWIGLU ? BW / 2 : BW;      // columns of y per tile
  const int n0 = (blockIdx.x / args.split) * CN;
  int m0 = blockIdx.y * TN, w0 = 0;
  if (args.tile_group != nullptr) {      // rows of an expert start at multiples of 128
    pdl_wait();
    const int g = args.tile_group[blockIdx.y];
    if (g < 0) {                         // the whole cluster leaves
      pdl_trigger();
      return;
    }
    m0 = blockIdx.y * 128;
    w0 = g * args.w_rows;
  }
  const int x0 = args.x_shared ? 0 : m0;
  const int chunks = (args.K + BK - 1) / BK;
  const int c_lo = (int)((long long)chunks * rank / args.split);
  const int c_hi = (int)((long long)chunks * (rank + 1) / args.split);

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  auto load_w = [&](int s, int chunk) {
    tma_load_2d(smem + s * C::STAGE, &tmW, &full_bar[s], chunk * BK, w0 + n0);
    if (SWIGLU) tma_load_2d(smem + s * C::STAGE + W_STAGE / 2, &tmW, &full_bar[s], chunk * BK, w0 + args.N + n0);
  };
  if (warp == 0) {
    if (lane == 0) {
      const int n = c_hi - c_lo;
      const int pre = n < C::STAGES ? n : C::STAGES;
      if (!args.w_static) pdl_wait();
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(&full_bar[i], C::STAGE);
        load_w(i, c_lo + i);
      }
      pdl_wait();
      pdl_trigger();
      for (int i = 0; i < pre; ++i)
        tma_load_2d(smem + i * C::STAGE + W_STAGE, &tmX, &full_bar[i], (c_lo + i) * BK, x0);
      for (int i = pre; i < n; ++i) {
        const int s = i % C::STAGES;
        if (!mbar_wait(&empty_bar[s], ((i / C::STAGES) & 1) ^ 1, abort_flag, args.status, 1)) break;
        mbar_expect_tx(&full_bar[s], C::STAGE);
        load_w(s, c_lo + i);
        tma_load_2d(smem + s * C::STAGE + W_STAGE, &tmX, &full_bar[s], (c_lo + i) * BK, x0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the warp stays converged and one elected lane issues: see mbar_ready in attn_common.cuh
    constexpr uint32_t idesc = make_idesc_bf16(BW, TN, false, false);
    const uint64_t w_desc = make_smem_desc(smem_u32(smem), 0, 1024);
    bool ok = true;
    for (int i = 0; i < c_hi - c_lo; ++i) {
      const int s = i % C::STAGES;
      if (!mbar_wait_warp(&full_bar[s], (i / C::STAGES) & 1, abort_flag, args.status, 3)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint64_t wd = w_desc + s * (C::STAGE >> 4), xd = wd + (W_STAGE >> 4);
      const uint32_t acc0 = i > 0 ? 1u : 0u;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16_ss(tmem_base, wd + k * 2, xd + k * 2, idesc, k > 0 ? 1u : acc0);
        umma_commit(&empty_bar[s]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(acc_full);
    __syncwarp();
  }
  const int rows = min(TN, args.M - m0);
  // This CTA finishes rows [r_lo, r_hi) of the tile: 8 outputs per thread and step, two steps at a time where a thread has several.
  // What bounds it is latency (other CTAs' sums, residual), so the first residual is read while the products still run, and a
  // step's sums are asked for together: the number of parts is known to the loop.  They are asked for step by step, so that the
  // steps share them out over the cluster; part by part all CTAs wait for the same one (128 rows, 4096 x 4096: 15.8 us).  Residual
  // and sums one after the other / this, us: 24 rows 4096 x 4096 10.4 / 9.7, x 12288 21.2 / 20.2; 128 rows 13.6 / 13.2 and
  // 26.4 / 25.0; 256 rows 18.2 / 15.8 and 36.6 / 33.2.  Four steps at a time: 13.5 and 25.3 at 128 rows, 15.8 and 32.8 at 256.
  constexpr int BATCH = TN >= 64 ? 2 : 1;
  const int v_hi = rows * (rank + 1) / args.split * (CN / 8);
  const int tid = (int)threadIdx.x - 64;
  int vb = rows * rank / args.split * (CN / 8);
  uint4 res[BATCH];
  auto load_res = [&]() {
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const int vi = vb + tid + 128 * i, n = n0 + (vi % (CN / 8)) * 8;
      if (vi < v_hi && n < args.N)
        res[i] = *reinterpret_cast<const uint4*>(args.residual + (long long)(m0 + vi / (CN / 8)) * args.ldr + n);
    }
  };
  if (warp >= 2) {
    pdl_wait();
    if (args.residual != nullptr) load_res();
  }
  // partial sums: tensor memory -> [row of x][128 weight rows] in this CTA's ring (all of its products have retired)
  float* part = reinterpret_cast<float*>(smem);
  bool ok = true;
  if (warp >= 2) {
    const int quarter = warp & 3;
    const int wr = quarter * 32 + lane;
    ok = mbar_wait_warp(acc_full, 0, abort_flag, args.status, 4);
    if (ok) {
      tc_fence_after();
      const uint32_t ta = tmem_base + ((uint32_t)(quarter * 32) << 16);
      if constexpr (TN == 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(ta, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < rows) part[j * BW + wr] = __uint_as_float(r[j]);
      } else {
#pragma unroll 1
        for (int c = 0; c < TN; c += 32) {
          if (c >= rows) break;
          uint32_t r[32];
          tmem_ld_32x32b_x32(ta + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) part[(c + j) * BW + wr] = __uint_as_float(r[j]);
        }
      }
      tc_fence_before();
    }
  }
  cluster_sync_all();
  if (warp >= 2) {
    const uint32_t part_addr = smem_u32(part);
    // PARTS: how many CTAs share the reduction, 0 = args.split
    auto finish = [&](auto parts) {
      constexpr int PARTS = decltype(parts)::value;
      auto sums = [&](int c, float (&o)[BATCH][8]) {      // in the order of the parts
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
#pragma unroll
          for (int j = 0; j < 8; ++j) o[i][j] = 0.f;
          if (vb + 128 * i >= v_hi) continue;
          const int vi = min(vb + tid + 128 * i, v_hi - 1);      // a thread past the last step reads what it does not use
          const uint32_t at = part_addr + ((vi / (CN / 8)) * BW + c + (vi % (CN / 8)) * 8) * 4;
          auto add = [&](const float4& a, const float4& b) {
            o[i][0] += a.x; o[i][1] += a.y; o[i][2] += a.z; o[i][3] += a.w;
            o[i][4] += b.x; o[i][5] += b.y; o[i][6] += b.z; o[i][7] += b.w;
          };
          if constexpr (PARTS > 0) {
            float4 a[PARTS], b[PARTS];
#pragma unroll
            for (int s = 0; s < PARTS; ++s) {
              a[s] = ld_cluster_f4(at, s);
              b[s] = ld_cluster_f4(at + 16, s);
            }
#pragma unroll
            for (int s = 0; s < PARTS; ++s) add(a[s], b[s]);
          } else {
            for (int s = 0; s < args.split; ++s) add(ld_cluster_f4(at, s), ld_cluster_f4(at + 16, s));
          }
        }
      };
      for (bool first = true; vb < v_hi; vb += 128 * BATCH, first = false) {
        if (!first && args.residual != nullptr) load_res();
        float out[BATCH][8];
        sums(0, out);
        if (SWIGLU) {
          float up[BATCH][8];
          sums(CN, up);
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) out[i][j] = silu_mul(round_bf16(out[i][j]), round_bf16(up[i][j]));
        } else {
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) out[i][j] *= args.alpha;
        }
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
          const int vi = vb + tid + 128 * i, n = n0 + (vi % (CN / 8)) * 8;
          if (vi >= v_hi || n >= args.N) continue;
          float (&o)[8] = out[i];
          const long long m = m0 + vi / (CN / 8);
          if (args.f32_out) {
            float4* cp = reinterpret_cast<float4*>(reinterpret_cast<float*>(args.C) + m * args.ldc + n);
            cp[0] = make_float4(o[0], o[1], o[2], o[3]);
            cp[1] = make_float4(o[4], o[5], o[6], o[7]);
            continue;
          }
          if (args.residual != nullptr) {
            const uint32_t u[4] = {res[i].x, res[i].y, res[i].z, res[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              o[2 * j] += __uint_as_float(u[j] << 16);
              o[2 * j + 1] += __uint_as_float(u[j] & 0xffff0000u);
            }
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(args.C) + m * args.ldc + n) =
              make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
        }
      }
    };
    if (ok) {
      switch (args.split) {
        case 1: finish(std::integral_constant<int, 1>()); break;
        case 2: finish(std::integral_constant<int, 2>()); break;
        case 4: finish(std::integral_constant<int, 4>()); break;
        case 8: finish(std::integral_constant<int, 8>()); break;
        default: finish(std::integral_constant<int, 0>());
      }
    }
  }
  // nobody leaves while another CTA of the cluster may still read its partial sums
  if (*abort_flag && warp == 1) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) {
    }
  }
  tc_fence_before();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM);
  }
}

template <int TN, bool SWIGLU, bool DEEP>
static int launch(const CUtensorMap& tmW, const CUtensorMap& tmX, const Args& a, int tiles, int mt, cudaStream_t st) {
  using C = Cfg<TN, DEEP>;
  int dev = 0;
  SNU1_CUDA_CHECK(cudaGetDevice(&dev));
  static std::once_flag once[64];
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&]() {
    err = cudaFuncSetAttribute(gemm_small_kernel<TN, SWIGLU, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  });
  SNU1_CUDA_CHECK(err);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(tiles * a.split, mt, 1);
  cfg.blockDim = dim3(NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SNU1_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_small_kernel<TN, SWIGLU, DEEP>, tmW, tmX, a));
  return kHostOk;
}

}  // namespace gsmall

// tiles_m > 0: tiles_m row tiles of experts (rows 128 t .. 128 t + M - 1 of x and y belong to expert tile_group[t], whose
// weights are rows tile_group[t] * w_rows ... of w; w_total rows in all).
static int launch_gemm_small_any(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw,
                                 long long ldc, int f32_out, const void* residual, long long ldr, float alpha, int split,
                                 int w_static, int swiglu, const int* tile_group, int tiles_m, int w_rows,
                                 long long w_total, int x_shared, cudaStream_t st) {
  using namespace gsmall;
  const int tn = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  const int mt = tiles_m > 0 ? tiles_m : (M + tn - 1) / tn;
  const int cn = swiglu ? BW / 2 : BW;
  const int tiles = (N + cn - 1) / cn;
  const int chunks = (K + BK - 1) / BK;
  if (split <= 0) {
    // Split the reduction while the CTAs still fit the chip: at two per SM, or at one (with a ring of twice the depth)
    // for wide row tiles, where a part also has a larger pass over the partial sums and keeps at least 12 chunks (768 of
    // the reduction).  Powers of two: clusters of three were slower than two or four.
    // 4096 x 4096 weights, 1 row, split 1 / 2 / 4 / 8: 20.9 / 11.9 / 9.1 / 8.2 us.
    // 128 rows, us, two per SM (shallow) / one per SM (deep): 6144 x 4096 split 4 / 2: 21.0 / 16.7; 4096 x 4096 split 4:
    // 14.5 / 13.7; 4096 x 12288 split 8 / 4: 31.1 / 25.3; 64 rows: 16.6 / 14.3, 12.1 / 11.7, 25.5 / 22.2.
    const long long fit = tn >= 64 ? num_sms() : 2 * num_sms();
    split = 1;
    while (split < 8 && (long long)tiles * mt * split * 2 <= fit && chunks / (split * 2) >= (tn >= 64 ? 12 : 3)) split *= 2;
  }
  // every part needs a chunk (a CTA without one has no product that would set its accumulator), a cluster has 8 CTAs at most
  split = split < chunks ? split : chunks;
  split = split < 8 ? split : 8;
  CUtensorMap tmW, tmX;
  int rc;
  {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)w_total};
    uint64_t strides[1] = {(uint64_t)ldw * 2};
    uint32_t box[2] = {BK, (uint32_t)cn};
    if ((rc = encode_tmap_bf16(&tmW, w, 2, dims, strides, box)) != kHostOk) return rc;
  }
  {
    uint64_t dims[2] = {(uint64_t)K, tiles_m > 0 && !x_shared ? (uint64_t)tiles_m * 128 : (uint64_t)M};
    uint64_t strides[1] = {(uint64_t)ldx * 2};
    uint32_t box[2] = {BK, (uint32_t)tn};
    if ((rc = encode_tmap_bf16(&tmX, x, 2, dims, strides, box)) != kHostOk) return rc;
  }
  Args a;
  memset(&a, 0, sizeof(a));
  a.M = tiles_m > 0 ? tiles_m * 128 : M;
  a.tile_group = tile_group;
  a.w_rows = w_rows;
  a.x_shared = x_shared;
  a.N = N;
  a.K = K;
  a.split = split;
  a.C = c;
  a.ldc = ldc;
  a.f32_out = f32_out;
  a.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  a.ldr = ldr;
  a.alpha = alpha;
  a.w_static = w_static;
  a.status = device_status_word();
#define SNU1_SMALL(TN, DEEP)                                                   \
  return swiglu ? launch<TN, true, DEEP>(tmW, tmX, a, tiles, mt, st) : launch<TN, false, DEEP>(tmW, tmX, a, tiles, mt, st)
  const bool deep = tn >= 64 && (long long)tiles * mt * split <= num_sms();
  switch (tn) {
    case 16: SNU1_SMALL(16, false);
    case 32: SNU1_SMALL(32, false);
    case 64: if (deep) SNU1_SMALL(64, true); SNU1_SMALL(64, false);
    default: if (deep) SNU1_SMALL(128, true); SNU1_SMALL(128, false);
  }
#undef SNU1_SMALL
}

int launch_gemm_small(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw,
                      long long ldc, int f32_out, const void* residual, long long ldr, float alpha, int split,
                      int w_static, int swiglu, cudaStream_t st) {
  return launch_gemm_small_any(x, w, c, M, N, K, ldx, ldw, ldc, f32_out, residual, ldr, alpha, split, w_static, swiglu,
                               nullptr, 0, 0, (long long)N * (swiglu ? 2 : 1), 0, st);
}

}  // namespace snu1

// The same product with the reduction split given (0: chosen by size; more parts than the reduction has 64s, or than 8, are
// not made); snu1_gemm_bf16 comes to launch_gemm_small by itself, with the checks of its own.
SNU1_API int snu1_gemm_small(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw,
                             long long ldc, int f32_out, const void* residual, long long ldr, float alpha, int split,
                             void* stream) {
  using namespace snu1;
  if (M <= 0 || N <= 0 || N % 8 || K <= 0 || K % 8 || ldx % 8 || ldw % 8 || ldc % (f32_out ? 4 : 8) ||
      (M + 127) / 128 > 65535 || (reinterpret_cast<uintptr_t>(c) & 15) != 0) {
    set_last_error("gemm_small: M=%d N=%d K=%d ldx=%lld ldw=%lld ldc=%lld (N, K, ldx, ldw multiples of 8, ldc of %d, y 16-byte "
                   "aligned)", M, N, K, ldx, ldw, ldc, f32_out ? 4 : 8);
    return kHostBadArg;
  }
  if (residual != nullptr && (f32_out || ldr % 8 || (reinterpret_cast<uintptr_t>(residual) & 15) != 0)) {
    set_last_error("gemm_small: a residual needs a bf16 result, 16-byte alignment and a stride of a multiple of 8");
    return kHostBadArg;
  }
  return launch_gemm_small(x, w, c, M, N, K, ldx, ldw, ldc, f32_out, residual, ldr, alpha, split, 0, 0,
                           reinterpret_cast<cudaStream_t>(stream));
}

// Expert products of a few rows: row tile t (rows 128 t .. 128 t + rows - 1 of x and y, rows <= 128) times the weights of
// expert tile_group[t], w[experts][w_rows][K] contiguous; tiles with a negative entry are skipped.  swiglu: w_rows = 2 N,
// y = silu(gate) * up, else w_rows = N.  x_shared: x has the one set of rows that every tile reads.  Rows of a tile past those in
// use are computed from whatever x holds there.
// One token, 8 of 128 experts, 768 x 2048: gate / up with activation 37.4 (pair kernel over padded tiles) -> 12 us, down
// 23.6 -> 8 us (floors 7.6 and 3.8).
SNU1_API int snu1_gemm_experts(const void* x, const void* w, void* y, int tiles, int rows, int N, int K, long long ldx,
                               long long ldy, const int* tile_group, int experts, int swiglu, int x_shared, void* stream) {
  using namespace snu1;
  if (tiles <= 0 || tiles > 65535 || rows <= 0 || rows > 128 || N <= 0 || N % 8 || K <= 0 || K % 8 || ldx % 8 || ldy % 8 ||
      experts <= 0 || tile_group == nullptr || (reinterpret_cast<uintptr_t>(y) & 15) != 0) {
    set_last_error("gemm_experts: tiles=%d rows=%d N=%d K=%d (N, K and strides multiples of 8, y 16-byte aligned)", tiles,
                   rows, N, K);
    return kHostBadArg;
  }
  const int w_rows = swiglu ? 2 * N : N;
  return launch_gemm_small_any(x, w, y, rows, N, K, ldx, K, ldy, 0, nullptr, 0, 1.0f, 0, 0, swiglu, tile_group, tiles,
                               w_rows, (long long)experts * w_rows, x_shared, reinterpret_cast<cudaStream_t>(stream));
}
