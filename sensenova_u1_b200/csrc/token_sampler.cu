// Top-k / top-p token sampling of fp32 logits in one launch per step.
//
// As separate operations (top-k, mask, full sort of the vocabulary, softmax three times, scan, scatter, division, argmax)
// a step took 27 launches and 330 us per row of 151,936 logits, most of it in single-CTA softmaxes and the sort of values
// that the top-k mask had just removed.  Here a cluster of eight CTAs holds a row in shared memory, finds the k-th largest
// value by a radix select (8 bits a pass, histograms summed over distributed shared memory), the at most k - 1 larger ones
// are sorted in one CTA, and only they (and ties of the k-th) meet the noise.  What bounds it: the row is read once
// (0.6 MB), then cluster barriers and the sort.  One row of 151,936, k = 50, p = 0.9: 330 -> 44 us, and 4 us for the noise.
//
// The rule: x = logits / temperature; values below the k-th largest go (ties of it stay); of the rest, sorted by value, a
// token stays while the probability before it is at most top_p; the token is the argmax of p / noise with noise ~ Exp(1).
// Ties are ordered by their index.
#include <string.h>

#include <mutex>

#include "host_common.h"
#include "sm100_common.cuh"

namespace snu1 {
namespace tok {

constexpr int THREADS = 512;
constexpr int CTAS = 8;
constexpr int MAX_K = 1024;

struct Args {
  const float* logits;
  const float* noise;
  long long* out;
  long long ld;
  int V, k;
  float inv_t, top_p;
};

struct Shared {
  unsigned hist[4][256];
  unsigned total[256];
  unsigned key[MAX_K];       // this CTA's larger values, in the first CTA all of them
  int idx[MAX_K];
  unsigned key_all[MAX_K];
  int idx_all[MAX_K];
  int count, ties;
  int digit;
  unsigned rest;
  float best_val[THREADS / 32];
  int best_idx[THREADS / 32];
  float cta_val;             // best of this CTA's ties
  int cta_idx;
  float draw_val;            // best of the larger values (first CTA)
  int draw_idx;
  float scan[THREADS / 32];
  // of the first CTA, read by the others
  float max, sum, tie_prob;
  int tie_keep;
};

// order-preserving integer of a float; NaN above everything (as sorting does), -0 equal to 0
__device__ __forceinline__ unsigned to_key(float x) {
  if (x != x) return 0xffffffffu;
  const unsigned b = __float_as_uint(x + 0.f);
  return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float from_key(unsigned k) {
  return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k);
}
// larger value wins, on equality the smaller index; NaN never wins against a number
__device__ __forceinline__ void take(float& v, int& i, float ov, int oi) {
  if (oi >= 0 && (i < 0 || ov > v || (ov == v && oi < i))) {
    v = ov;
    i = oi;
  }
}
__device__ __forceinline__ void block_best(Shared& s, float& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) take(v, i, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, i, o));
  if ((threadIdx.x & 31) == 0) {
    s.best_val[threadIdx.x >> 5] = v;
    s.best_idx[threadIdx.x >> 5] = i;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < THREADS / 32; ++w) take(v, i, s.best_val[w], s.best_idx[w]);
}

__global__ void __launch_bounds__(THREADS) top_k_top_p_kernel(const Args a) {
  extern __shared__ unsigned keys[];
  __shared__ Shared s;
  const uint32_t rank = cluster_ctarank();
  const int row = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lo = (int)((long long)a.V * rank / CTAS), n = (int)((long long)a.V * (rank + 1) / CTAS) - lo;
  for (int i = tid; i < 4 * 256; i += THREADS) s.hist[0][i] = 0;
  if (tid == 0) s.count = s.ties = 0;
  pdl_wait();
  pdl_trigger();
  const float* lg = a.logits + row * a.ld + lo;
  for (int i = tid; i < n; i += THREADS) keys[i] = to_key(lg[i] * a.inv_t);
  __syncthreads();

  // k-th largest key: digits from the top
  unsigned prefix = 0, rest = a.k;
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    const int shift = 24 - 8 * p;
    for (int i0 = 0; i0 < n; i0 += THREADS) {
      const int i = i0 + tid;
      const unsigned key = i < n ? keys[i] : 0;
      const bool in = i < n && (p == 0 || (key >> (shift + 8)) == prefix);
      const unsigned d = in ? (key >> shift) & 255u : 256u;
      const unsigned same = __match_any_sync(0xffffffffu, d);      // most logits share a few digits
      if (in && (same & ((1u << lane) - 1)) == 0) atomicAdd(&s.hist[p][d], __popc(same));
    }
    cluster_sync_all();
    if (tid < 256) {
      unsigned t = 0;
      for (int r = 0; r < CTAS; ++r) t += ld_cluster(s.hist[p][tid], r);
      s.total[tid] = t;
    }
    __syncthreads();
    if (warp == 0) {             // lane l: digits 255 - 8 l .. 248 - 8 l
      unsigned c = 0;
      for (int j = 0; j < 8; ++j) c += s.total[255 - 8 * lane - j];
      unsigned incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      unsigned before = incl - c;
      if (before < rest && incl >= rest) {
        for (int j = 0; j < 8; ++j) {
          const unsigned t = s.total[255 - 8 * lane - j];
          if (before + t >= rest) {
            s.digit = 255 - 8 * lane - j;
            s.rest = rest - before;
            break;
          }
          before += t;
        }
      }
    }
    __syncthreads();
    prefix = (prefix << 8) | (unsigned)s.digit;
    rest = s.rest;
  }
  const unsigned kth = prefix;
  const int larger = a.k - (int)rest;                 // values above the k-th
  const int ties = (int)s.total[s.digit];             // values equal to it
  // this CTA's larger values and its number of ties (a thread's elements are contiguous: ties are ranked by index)
  const int per = (n + THREADS - 1) / THREADS;
  int my_ties = 0;
  for (int j = 0; j < per; ++j) {
    const int i = tid * per + j;
    if (i >= n) break;
    const unsigned key = keys[i];
    my_ties += key == kth;
    if (key > kth) {
      const int c = atomicAdd(&s.count, 1);
      s.key[c] = key;
      s.idx[c] = lo + i;
    }
  }
  int tie_rank;                                       // ties before this thread's, in this CTA
  {
    int incl = my_ties;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s.best_idx[warp] = incl;
    __syncthreads();
    tie_rank = incl - my_ties;
    int all = 0;
    for (int w = 0; w < THREADS / 32; ++w) {
      if (w < warp) tie_rank += s.best_idx[w];
      all += s.best_idx[w];
    }
    if (tid == 0) s.ties = all;
  }
  cluster_sync_all();
  if (rank == 0) {
    // gather, sort by (value, -index), softmax and cut
    int at = 0;
    for (int r = 0; r < CTAS; ++r) {
      const int c = ld_cluster(s.count, r);
      for (int i = tid; i < c; i += THREADS) {
        s.key_all[at + i] = ld_cluster(s.key[i], r);
        s.idx_all[at + i] = ld_cluster(s.idx[i], r);
      }
      at += c;
    }
    int size = 2;
    while (size < larger) size <<= 1;
    __syncthreads();
    for (int i = larger + tid; i < size; i += THREADS) {
      s.key_all[i] = 0;
      s.idx_all[i] = 0x7fffffff;
    }
    __syncthreads();
    for (int kk = 2; kk <= size; kk <<= 1)
      for (int j = kk >> 1; j > 0; j >>= 1) {
        for (int i = tid; i < size; i += THREADS) {
          const int o = i ^ j;
          if (o > i) {
            const unsigned ka = s.key_all[i], kb = s.key_all[o];
            const int ia = s.idx_all[i], ib = s.idx_all[o];
            const bool a_first = ka > kb || (ka == kb && ia < ib);
            if (a_first != ((i & kk) == 0)) {
              s.key_all[i] = kb;
              s.key_all[o] = ka;
              s.idx_all[i] = ib;
              s.idx_all[o] = ia;
            }
          }
        }
        __syncthreads();
      }
    const float mx = from_key(larger > 0 ? s.key_all[0] : kth);
    const float e_tie = expf(from_key(kth) - mx);
    // two neighbours per thread: sum, then the probability before each (exclusive scan)
    float e[2];
    for (int j = 0; j < 2; ++j) {
      const int i = 2 * tid + j;
      e[j] = i < larger ? expf(from_key(s.key_all[i]) - mx) : 0.f;
    }
    // sum over the block before the thread's own, and with it.  The former is never the latter less x: that leaves a
    // rounding instead of 0 before the first, and the likeliest token would go at a top_p below it
    auto scan = [&](float x, float& before) {
      float incl = x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      before = __shfl_up_sync(0xffffffffu, incl, 1);
      if (lane == 0) before = 0.f;
      __syncthreads();
      if (lane == 31) s.scan[warp] = incl;
      __syncthreads();
      float base = 0.f;
      for (int w = 0; w < warp; ++w) base += s.scan[w];
      before += base;
      return incl + base;
    };
    float b0, unused;
    const float incl = scan(e[0] + e[1], b0);
    if (tid == THREADS - 1) s.sum = incl;
    __syncthreads();
    const float above = s.sum, sum = above + ties * e_tie;
    __syncthreads();
    const float b1 = b0 + e[0];
    const bool k0 = !(b0 / sum > a.top_p) || a.top_p >= 1.f, k1 = !(b1 / sum > a.top_p) || a.top_p >= 1.f;
    const float kept = scan((k0 ? e[0] : 0.f) + (k1 ? e[1] : 0.f), unused);
    if (tid == THREADS - 1) {
      int keep = ties;
      if (a.top_p < 1.f) {
        const float left = a.top_p - above / sum, pt = e_tie / sum;
        keep = left < 0.f ? 0 : pt > 0.f && left / pt < (float)ties ? min(ties, (int)(left / pt) + 1) : ties;
      }
      s.tie_keep = keep;
      s.max = mx;
      s.sum = kept + keep * e_tie;
      s.tie_prob = e_tie / s.sum;
    }
    __syncthreads();
    const float total = s.sum;
    float bv = 0.f;
    int bi = -1;
    for (int j = 0; j < 2; ++j) {
      const int i = 2 * tid + j;
      if (i < larger && (j == 0 ? k0 : k1)) take(bv, bi, e[j] / total / a.noise[(long long)row * a.V + s.idx_all[i]], s.idx_all[i]);
    }
    block_best(s, bv, bi);
    if (tid == 0) {
      s.draw_val = bv;
      s.draw_idx = bi;
    }
  }
  cluster_sync_all();
  // ties of the k-th value that stay, ranked by index over the cluster
  {
    const int keep = ld_cluster(s.tie_keep, 0);
    const float pt = ld_cluster(s.tie_prob, 0);
    int before = tie_rank;
    for (uint32_t r = 0; r < rank; ++r) before += ld_cluster(s.ties, r);
    float bv = 0.f;
    int bi = -1;
    if (my_ties > 0 && before < keep)
      for (int j = 0; j < per && before < keep; ++j) {
        const int i = tid * per + j;
        if (i >= n) break;
        if (keys[i] == kth) {
          take(bv, bi, pt / a.noise[(long long)row * a.V + lo + i], lo + i);
          ++before;
        }
      }
    __syncthreads();
    block_best(s, bv, bi);
    if (tid == 0) {
      s.cta_val = bv;
      s.cta_idx = bi;
    }
  }
  cluster_sync_all();
  if (rank == 0 && tid == 0) {
    float bv = s.draw_val;
    int bi = s.draw_idx;
    for (int r = 0; r < CTAS; ++r) take(bv, bi, ld_cluster(s.cta_val, r), ld_cluster(s.cta_idx, r));
    a.out[row] = bi < 0 ? 0 : bi;
  }
  cluster_sync_all();      // nobody leaves while its shared memory is read
}

}  // namespace tok
}  // namespace snu1

// logits, noise: fp32 [rows][V] (logits with row stride ld, noise contiguous); out: int64 [rows].  0 < k < V, k <= 1024.
SNU1_API int snu1_sample_top_k_top_p(const float* logits, long long ld, const float* noise, long long* out, int rows, int V,
                                     int k, float inv_t, float top_p, void* stream) {
  using namespace snu1;
  const int smem = (V / tok::CTAS + 1) * 4;
  if (rows <= 0 || rows > 65535 || k <= 0 || k >= V || k > tok::MAX_K || smem > 180 * 1024) {
    set_last_error("sample_top_k_top_p: rows=%d V=%d k=%d", rows, V, k);
    return kHostBadArg;
  }
  int dev = 0;
  SNU1_CUDA_CHECK(cudaGetDevice(&dev));
  static std::once_flag once[64];
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&]() {
    err = cudaFuncSetAttribute(tok::top_k_top_p_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 180 * 1024);
  });
  SNU1_CUDA_CHECK(err);
  tok::Args a = {logits, noise, out, ld, V, k, inv_t, top_p};
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = tok::CTAS;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(tok::CTAS, rows, 1);
  cfg.blockDim = dim3(tok::THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SNU1_CUDA_CHECK(cudaLaunchKernelEx(&cfg, tok::top_k_top_p_kernel, a));
  return kHostOk;
}
