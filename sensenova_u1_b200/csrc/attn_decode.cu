// Decode attention: one query row per document against the document's rows of the K/V cache.
//
// What bounds it is the stream of K and V from HBM, so the work is split over keys and not over query tiles: the
// tile kernel (attn_fwd_sm100.cu) gives one CTA per head all key tiles of all documents, 32 CTAs on 148 SMs that walk
// up to 150 tiles one after another.  Here a cluster of ``split`` CTAs owns (document, K/V head), every CTA takes a
// contiguous part of the document's rows, and the partial results (row maximum, sum, weighted V) meet in distributed
// shared memory in a fixed order (no atomics, no scratch, deterministic).  With one row per document the products are
// 1 - 2 multiply-adds per byte, far below the tensor cores' balance: packed fp32 FMAs, probabilities and sums in fp32.
//
// Eight lanes share a key (16 of its 128 elements each), a warp works on four keys at a time.  Every lane copies the
// 16-byte pieces that it will read itself into its own slots of a three-stage ring (cp.async), so two steps of 64 keys
// per CTA are on their way during the arithmetic of a third, without registers and without block barriers; two CTAs
// fit an SM: 128 KB of loads in flight.
//
// Measured (32 / 8 heads, bf16, us per launch inside a graph, caches cold in L2; floor = K and V at 6.65 TB/s):
//   documents x keys           tile kernel    this kernel    floor
//   1 x 70                           7.0            5.3       0.04
//   1 x 840                         15.8            7.6       0.5
//   1 x 32000                        388             56        20
//   24 x 62 .. 1500 (18600)          312             32        11
#include <string.h>

#include <mutex>

#include "attn_common.cuh"
#include "host_common.h"

namespace snu1 {
namespace attn_dec {

constexpr int THREADS = 128;
constexpr int GROUPS = THREADS / 8;   // keys in flight per step of the CTA
constexpr int U = 4;                  // keys per group and step
constexpr int STAGES = 3;
constexpr int MAX_SPLIT = 16;         // CTAs of a cluster (more than 8 need the non-portable size)
constexpr int SMEM = STAGES * U * (4 * THREADS + GROUPS) * 16;

struct Args {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  __nv_bfloat16* o;
  long long ldq, ldk, ldv, ldo;
  const TokMeta* meta_q;
  const TokMeta* meta_k;
  const int* first;          // [rows] first cache row of the document
  const long long* last;     // [rows] cache row of the query itself
  int Sk, Hq, Hkv, split;
  float scale_log2;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Sums over the eight lanes of a key: lane ``sub`` returns head (sub >> 1) of four, (sub >> 2) of two.  Every exchange
// halves the heads that a lane still carries.
template <int HG>
__device__ __forceinline__ float head_sum(const float (&s)[HG], int sub) {
  float r;
  if constexpr (HG == 4) {
    const bool b = (sub & 4) != 0, c = (sub & 2) != 0;
    float k0 = b ? s[2] : s[0], k1 = b ? s[3] : s[1];
    k0 += __shfl_xor_sync(0xffffffffu, b ? s[0] : s[2], 4);
    k1 += __shfl_xor_sync(0xffffffffu, b ? s[1] : s[3], 4);
    r = c ? k1 : k0;
    r += __shfl_xor_sync(0xffffffffu, c ? k0 : k1, 2);
  } else if constexpr (HG == 2) {
    const bool b = (sub & 4) != 0;
    r = b ? s[1] : s[0];
    r += __shfl_xor_sync(0xffffffffu, b ? s[0] : s[1], 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
  } else {
    r = s[0];
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
  }
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}
// the value that the lanes of head ``h`` hold, in all lanes of the key
template <int HG>
__device__ __forceinline__ float head_value(float x, int h, int lane) {
  return __shfl_sync(0xffffffffu, x, (lane & 24) | (HG == 4 ? h * 2 : HG == 2 ? h * 4 : 0));
}

// HG query heads of one K/V head.  Grid: (split, K/V heads x groups of HG query heads, rows).
template <int HG>
__global__ void __launch_bounds__(THREADS, 2) attn_decode_kernel(const Args a) {
  extern __shared__ uint4 ring[];                       // [STAGES][U][K lo, K hi, V lo, V hi][THREADS], then the metadata
  int4* ring_meta = reinterpret_cast<int4*>(ring + STAGES * U * 4 * THREADS);          // [STAGES][U][GROUPS]
  __shared__ float s_acc[THREADS / 32][HG][128];
  __shared__ float s_m[THREADS / 32][HG], s_l[THREADS / 32][HG];
  __shared__ float c_acc[HG][128], c_m[HG], c_l[HG];    // this CTA's partial result, read by the cluster
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & 7, grp = warp * 4 + (lane >> 3);
  const int row = blockIdx.z;
  const int rank = a.split > 1 ? (int)cluster_ctarank() : 0;
  const int rep = a.Hq / a.Hkv, per_kv = rep / HG;
  const int kvh = blockIdx.y / per_kv;
  const int h0 = kvh * rep + (blockIdx.y % per_kv) * HG;
  pdl_wait();
  pdl_trigger();

  const int lo = max(0, a.first[row]);
  const int hi = (int)min((long long)a.Sk, a.last[row] + 1);
  const int len = max(0, hi - lo);
  const int k_lo = lo + (int)((long long)len * rank / a.split);
  const int k_hi = lo + (int)((long long)len * (rank + 1) / a.split);
  const int steps = (k_hi - k_lo + GROUPS * U - 1) / (GROUPS * U);
  const __nv_bfloat16* kb = a.k + (long long)kvh * 128 + sub * 8;
  const __nv_bfloat16* vb = a.v + (long long)kvh * 128 + sub * 8;
  auto load = [&](int it) {
    if (it < steps) {
      const int st = it % STAGES;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int key = k_lo + (it * U + u) * GROUPS + grp;
        const long long r = key < k_hi ? key : k_lo;    // past the end: any row of the range, masked below
        const uint32_t dst = smem_u32(ring + (st * U + u) * 4 * THREADS + threadIdx.x);
        cp_async16(dst, kb + r * a.ldk);
        cp_async16(dst + THREADS * 16, kb + r * a.ldk + 64);
        cp_async16(dst + 2 * THREADS * 16, vb + r * a.ldv);
        cp_async16(dst + 3 * THREADS * 16, vb + r * a.ldv + 64);
        if (sub == u) cp_async16(smem_u32(ring_meta + (st * U + u) * GROUPS + grp), a.meta_k + r);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) load(i);

  // lane ``sub`` holds elements [8 sub, 8 sub + 8) and [64 + 8 sub, 64 + 8 sub + 8)
  uint64_t q2[HG][8];
  const uint64_t sc2 = pack_f32x2(a.scale_log2, a.scale_log2);
#pragma unroll
  for (int h = 0; h < HG; ++h) {
    const __nv_bfloat16* qp = a.q + row * a.ldq + (long long)(h0 + h) * 128 + sub * 8;
    const uint4 u0 = *reinterpret_cast<const uint4*>(qp), u1 = *reinterpret_cast<const uint4*>(qp + 64);
    const uint32_t w[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) q2[h][i] = mul_f32x2(bf16x2_to_f32x2(w[i]), sc2);
  }
  const TokMeta mq = a.meta_q[row];

  uint64_t acc[HG][8];
#pragma unroll
  for (int h = 0; h < HG; ++h)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[h][i] = 0ull;
  float m = -INFINITY, l = 0.f;                         // of this lane's head, over the keys of its group
  for (int it = 0; it < steps; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncwarp();                                       // the metadata was copied by other lanes
    load(it + STAGES - 1);                              // into the stage that the warp left in the previous step
    const int st = it % STAGES;
    const uint4* slot = ring + st * U * 4 * THREADS + threadIdx.x;
    float s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 r0 = slot[u * 4 * THREADS], r1 = slot[(u * 4 + 1) * THREADS];
      const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
      uint64_t k2[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) k2[i] = bf16x2_to_f32x2(w[i]);
      float d[HG];
#pragma unroll
      for (int h = 0; h < HG; ++h) {
        uint64_t d0 = mul_f32x2(q2[h][0], k2[0]), d1 = mul_f32x2(q2[h][1], k2[1]);
#pragma unroll
        for (int i = 2; i < 8; i += 2) {
          d0 = fma_f32x2(q2[h][i], k2[i], d0);
          d1 = fma_f32x2(q2[h][i + 1], k2[i + 1], d1);
        }
        float x, y;
        unpack_f32x2(add_f32x2(d0, d1), x, y);
        d[h] = x + y;
      }
      const int4 t = ring_meta[(st * U + u) * GROUPS + grp];
      const bool ok = k_lo + (it * U + u) * GROUPS + grp < k_hi && mask_allowed(mq, TokMeta{t.x, t.y, t.z, t.w});
      const float v = head_sum<HG>(d, sub);
      s[u] = ok ? v : -INFINITY;
    }
    float mx = s[0];
#pragma unroll
    for (int u = 1; u < U; ++u) mx = fmaxf(mx, s[u]);
    if (__any_sync(0xffffffffu, mx > m)) {
      const float mn = fmaxf(m, mx);
      const float f = m == -INFINITY ? 0.f : fast_exp2(m - mn);
      l *= f;
      m = mn;
#pragma unroll
      for (int h = 0; h < HG; ++h) {
        const float fh = head_value<HG>(f, h, lane);
        const uint64_t f2 = pack_f32x2(fh, fh);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[h][i] = mul_f32x2(acc[h][i], f2);
      }
    }
    const float mu = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s[u] = fast_exp2(s[u] - mu);
      l += s[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 r0 = slot[(u * 4 + 2) * THREADS], r1 = slot[(u * 4 + 3) * THREADS];
      const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
      uint64_t v2[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v2[i] = bf16x2_to_f32x2(w[i]);
#pragma unroll
      for (int h = 0; h < HG; ++h) {
        const float p = head_value<HG>(s[u], h, lane);
        const uint64_t p2 = pack_f32x2(p, p);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[h][i] = fma_f32x2(p2, v2[i], acc[h][i]);
      }
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // the four key groups of a warp, then the four warps
#pragma unroll
  for (int h = 0; h < HG; ++h) {
    const float mh = head_value<HG>(m, h, lane), lh = head_value<HG>(l, h, lane);
    float mw = fmaxf(mh, __shfl_xor_sync(0xffffffffu, mh, 8));
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 16));
    const float f = mh == -INFINITY ? 0.f : fast_exp2(mh - mw);
    float lw = lh * f;
    lw += __shfl_xor_sync(0xffffffffu, lw, 8);
    lw += __shfl_xor_sync(0xffffffffu, lw, 16);
    float o[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) unpack_f32x2(acc[h][i], o[2 * i], o[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      o[i] *= f;
      o[i] += __shfl_xor_sync(0xffffffffu, o[i], 8);
      o[i] += __shfl_xor_sync(0xffffffffu, o[i], 16);
    }
    if (lane < 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s_acc[warp][h][sub * 8 + i] = o[i];
        s_acc[warp][h][64 + sub * 8 + i] = o[8 + i];
      }
      if (lane == 0) {
        s_m[warp][h] = mw;
        s_l[warp][h] = lw;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < HG; ++h) {
    float mc = s_m[0][h];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) mc = fmaxf(mc, s_m[w][h]);
    float x = 0.f, lc = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
      const float f = s_m[w][h] == -INFINITY ? 0.f : fast_exp2(s_m[w][h] - mc);
      x += f * s_acc[w][h][threadIdx.x];
      lc += f * s_l[w][h];
    }
    c_acc[h][threadIdx.x] = x;
    if (threadIdx.x == 0) {
      c_m[h] = mc;
      c_l[h] = lc;
    }
  }
  if (a.split > 1) cluster_sync_all();
  else __syncthreads();
  // every CTA of the cluster finishes its share of the HG x 128 outputs, two at a time
  constexpr int PAIRS = HG * 64;
  for (int i = PAIRS * rank / a.split + threadIdx.x; i < PAIRS * (rank + 1) / a.split; i += THREADS) {
    const int h = i >> 6, c = (i & 63) * 2;
    float x, y, lt;
    if (a.split == 1) {
      x = c_acc[h][c];
      y = c_acc[h][c + 1];
      lt = c_l[h];
    } else {
      float mt = -INFINITY;
      for (int r = 0; r < a.split; ++r) mt = fmaxf(mt, ld_cluster(c_m[h], r));
      x = y = lt = 0.f;
      for (int r = 0; r < a.split; ++r) {
        const float mr = ld_cluster(c_m[h], r);
        const float f = mr == -INFINITY ? 0.f : fast_exp2(mr - mt);
        x += f * ld_cluster(c_acc[h][c], r);
        y += f * ld_cluster(c_acc[h][c + 1], r);
        lt += f * ld_cluster(c_l[h], r);
      }
    }
    const float inv = lt > 0.f ? 1.f / lt : 0.f;       // a row without keys gives zeros
    *reinterpret_cast<uint32_t*>(a.o + row * a.ldo + (long long)(h0 + h) * 128 + c) = pack_bf16x2(x * inv, y * inv);
  }
  if (a.split > 1) cluster_sync_all();   // nobody leaves while its partial result is read
}

template <int HG>
static int launch(const Args& a, int rows, cudaStream_t st) {
  int dev = 0;
  SNU1_CUDA_CHECK(cudaGetDevice(&dev));
  static std::once_flag once[64];
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&]() {
    err = cudaFuncSetAttribute(attn_decode_kernel<HG>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(attn_decode_kernel<HG>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  SNU1_CUDA_CHECK(err);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = a.split;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(a.split, a.Hq / HG, rows);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SNU1_CUDA_CHECK(cudaLaunchKernelEx(&cfg, attn_decode_kernel<HG>, a));
  return kHostOk;
}

}  // namespace attn_dec
}  // namespace snu1

using namespace snu1;

// rows queries [rows][Hq][128], query r against cache rows [first[r], last[r]] that the mask rule lets it read.
// max_keys: the longest range the caller expects (a hint for the split).  split <= 0: chosen by size.
SNU1_API int snu1_attn_decode(const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv,
                              void* o, long long ldo, const void* meta_q, const void* meta_k, const int* first,
                              const long long* last, int rows, int Sk, int Hq, int Hkv, float scale, int max_keys,
                              int split, void* stream) {
  if (Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0 || rows <= 0 || rows > 65535 || Sk <= 0 || split > attn_dec::MAX_SPLIT) {
    set_last_error("attn_decode: bad head counts / lengths");
    return kHostBadArg;
  }
  if (ldq % 8 || ldk % 8 || ldv % 8 || ldo % 8 ||
      ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
        reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(meta_q) | reinterpret_cast<uintptr_t>(meta_k)) &
       15) != 0) {
    set_last_error("attn_decode: rows must be 16-byte aligned");
    return kHostBadArg;
  }
  attn_dec::Args a;
  a.q = (const __nv_bfloat16*)q;
  a.k = (const __nv_bfloat16*)k;
  a.v = (const __nv_bfloat16*)v;
  a.o = (__nv_bfloat16*)o;
  a.ldq = ldq;
  a.ldk = ldk;
  a.ldv = ldv;
  a.ldo = ldo;
  a.meta_q = (const TokMeta*)meta_q;
  a.meta_k = (const TokMeta*)meta_k;
  a.first = first;
  a.last = last;
  a.Sk = Sk;
  a.Hq = Hq;
  a.Hkv = Hkv;
  a.scale_log2 = scale * 1.4426950408889634f;
  const int rep = Hq / Hkv;
  const int hg = rep % 4 == 0 ? 4 : rep % 2 == 0 ? 2 : 1;
  if (split <= 0) {
    // Until the chip is full (two CTAs per SM), at least one step of 64 keys per CTA; a part costs about 3 us besides
    // its keys.  24 x 62 .. 1500 keys, split 1 / 2 / 4 / 8: 34.4 / 32.1 / 34.8 / 53.1 us; 1 x 840, 1 / 4 / 8 / 16:
    // 19.0 / 9.1 / 7.6 / 7.6; 1 x 32000, 4 / 8 / 16: 134 / 79 / 56.
    split = 1;
    while (split < attn_dec::MAX_SPLIT && (long long)rows * (Hq / hg) * split < 2 * 148 && max_keys / (split * 2) >= attn_dec::GROUPS * attn_dec::U)
      split *= 2;
  }
  a.split = split;
  cudaStream_t st = (cudaStream_t)stream;
  if (hg == 4) return attn_dec::launch<4>(a, rows, st);
  if (hg == 2) return attn_dec::launch<2>(a, rows, st);
  return attn_dec::launch<1>(a, rows, st);
}
