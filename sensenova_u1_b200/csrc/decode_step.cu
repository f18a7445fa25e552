// What stands between the LM head and the decoder layers of a decode step: the likeliest token of a row, and everything that
// follows from a token (output slot, embedding row, position, cache row, token metadata).
//
// Bound by launches: as a dozen tensor operations (reduction, index copies, gathers, stacks, increments) this took 30 us of
// a step of 1.1 ms; two launches of 3 and 2 us do the same.  One row of 151,936 logits: argmax 9.9 -> 3.4 us.
#include <string.h>

#include "attn_common.cuh"
#include "host_common.h"

namespace snu1 {
namespace dstep {

constexpr int THREADS = 512;
constexpr int CTAS = 8;        // of a row: one CTA alone reads 0.6 MB in 10 us

// whether (v, i) comes before (ov, oi): NaN above everything, then the larger value, then the smaller index
__device__ __forceinline__ bool before(float v, int i, float ov, int oi) {
  const bool n = v != v, on = ov != ov;
  if (n != on) return n;
  if (!n && v != ov) return v > ov;
  return i < oi;
}

__global__ void __launch_bounds__(THREADS) argmax_kernel(const float* __restrict__ x, long long ld, int V, long long* __restrict__ out) {
  __shared__ float s_v[THREADS / 32];
  __shared__ int s_i[THREADS / 32];
  __shared__ float c_v;
  __shared__ int c_i;
  const int rank = (int)cluster_ctarank(), row = blockIdx.y, tid = threadIdx.x;
  const int lo = (int)((long long)V * rank / CTAS), hi = (int)((long long)V * (rank + 1) / CTAS);
  pdl_wait();
  pdl_trigger();
  const float* p = x + row * ld;
  float v = -INFINITY;
  int i = V;                   // behind every element, also an infinite one
#pragma unroll 8
  for (int k = lo + tid; k < hi; k += THREADS) {
    const float t = p[k];
    if (before(t, k, v, i)) {
      v = t;
      i = k;
    }
  }
  auto best = [&](float ov, int oi) {
    if (before(ov, oi, v, i)) {
      v = ov;
      i = oi;
    }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    best(ov, oi);
  }
  if ((tid & 31) == 0) {
    s_v[tid >> 5] = v;
    s_i[tid >> 5] = i;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < THREADS / 32; ++w) best(s_v[w], s_i[w]);
    c_v = v;
    c_i = i;
  }
  cluster_sync_all();
  if (rank == 0 && tid == 0) {
    for (int r = 1; r < CTAS; ++r) {
      const float ov = ld_cluster(c_v, r);
      const int oi = ld_cluster(c_i, r);
      best(ov, oi);
    }
    out[row] = i;
  }
  cluster_sync_all();          // nobody leaves while its result is read
}

struct Advance {
  const long long* token;      // [rows]
  const __nv_bfloat16* embed;  // [V][H]
  int V, H, rows, Sk;
  int* done;                   // [rows] tokens so far
  const int* pos0;             // [rows] position and cache row of the first token
  const long long* row0;
  long long* out;              // [rows][ld_out]
  int ld_out;
  __nv_bfloat16* x;            // [rows][H]
  int* pos3;                   // [3][rows]
  TokMeta* meta_q;             // [rows]
  TokMeta* meta_k;             // [Sk]
  long long* kv_row;           // [rows]
  int* status;
};

__global__ void __launch_bounds__(256) advance_kernel(const Advance a) {
  const int r = blockIdx.x;
  pdl_wait();
  pdl_trigger();
  const long long t = a.token[r];
  const bool ok = t >= 0 && t < a.V;
  const uint4* src = reinterpret_cast<const uint4*>(a.embed + (ok ? t : 0) * a.H);
  uint4* dst = reinterpret_cast<uint4*>(a.x + (long long)r * a.H);
  for (int i = threadIdx.x; i < a.H / 8; i += 256) dst[i] = ok ? src[i] : make_uint4(0, 0, 0, 0);
  if (threadIdx.x == 0) {
    const int n = a.done[r], pos = a.pos0[r] + n;
    const long long row = a.row0[r] + n;
    const bool in = n >= 0 && n < a.ld_out && row >= 0 && row < a.Sk;
    if (n >= 0 && n < a.ld_out) a.out[(long long)r * a.ld_out + n] = t;
    a.pos3[r] = pos;
    a.pos3[a.rows + r] = a.pos3[2 * a.rows + r] = 0;
    const TokMeta m{r, pos, 0, 0};
    a.meta_q[r] = m;
    if (row >= 0 && row < a.Sk) a.meta_k[row] = m;
    a.kv_row[r] = row;
    a.done[r] = n + 1;
    if (!ok || !in) report_status(a.status, kBadShape, 5);
  }
}

}  // namespace dstep
}  // namespace snu1

using namespace snu1;

// out[r] = index of the largest element of row r of x [rows][V] fp32 (NaN counts as largest; of equal ones the first).
SNU1_API int snu1_argmax_rows(const float* x, long long ld, int rows, int V, long long* out, void* stream) {
  if (rows < 1 || rows > 65535 || V < 1 || ld < V) {
    set_last_error("argmax_rows: rows=%d V=%d ld=%lld", rows, V, ld);
    return kHostBadArg;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = dstep::CTAS;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(dstep::CTAS, rows, 1);
  cfg.blockDim = dim3(dstep::THREADS, 1, 1);
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SNU1_CUDA_CHECK(cudaLaunchKernelEx(&cfg, dstep::argmax_kernel, x, ld, V, out));
  return kHostOk;
}

// What follows from the tokens of a decode step (csrc above: Advance), one document per row.
SNU1_API int snu1_decode_advance(const long long* token, const void* embed, int V, int H, int rows, int Sk, int* done, const int* pos0,
                                 const long long* row0, long long* out, int ld_out, void* x, int* pos3, void* meta_q, void* meta_k,
                                 long long* kv_row, void* stream) {
  if (rows < 1 || V < 1 || H < 8 || H % 8 || Sk < 1 || ld_out < 1 ||
      ((reinterpret_cast<uintptr_t>(embed) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(meta_q) |
        reinterpret_cast<uintptr_t>(meta_k)) & 15)) {
    set_last_error("decode_advance: rows=%d V=%d H=%d (a multiple of 8, 16-byte aligned) Sk=%d", rows, V, H, Sk);
    return kHostBadArg;
  }
  dstep::Advance a{token, (const __nv_bfloat16*)embed, V, H, rows, Sk, done, pos0, row0, out, ld_out, (__nv_bfloat16*)x, pos3,
                   (TokMeta*)meta_q, (TokMeta*)meta_k, kv_row, device_status_word()};
  SNU1_CUDA_CHECK(launch_pdl(dstep::advance_kernel, dim3(rows), dim3(256), 0, (cudaStream_t)stream, a));
  return kHostOk;
}
