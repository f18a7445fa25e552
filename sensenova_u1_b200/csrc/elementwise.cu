// Memory-bound kernels of the MoT decoder layer: RMSNorm with per-branch gains,
// the q/k half-head RMSNorm fused with the three-axis rotary embedding, and
// SwiGLU; forward and backward.  All of them work on the packed row layout
// "generation rows | understanding rows", where every 128-row tile belongs to
// one branch (tile_group), so a branch switch never needs a gather or a concat
// (reference: training/sensenovalm/model/modeling_qwen3_moe_mot.py:323-369).
//
// Math references: RMSNorm src/sensenova_u1/models/neo_unify/modeling_qwen3.py:183-200,
// q/k half norms and t/h/w RoPE :444-468, rotate-half :219-250, SwiGLU :203-217.
#include "host_common.h"
#include "sm100_common.cuh"

namespace snu1 {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) t += scratch[i];
  return t;
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]);
  u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]);
  u.w = pack_bf16x2(f[6], f[7]);
  return u;
}

// ---------------------------------------------------------------------------
// RMSNorm over the hidden dimension, gain chosen per 128-row tile.
// ---------------------------------------------------------------------------
constexpr int RN_THREADS = 256;

__global__ void __launch_bounds__(RN_THREADS)
    rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gain,
                       const int* __restrict__ tile_group, __nv_bfloat16* __restrict__ y,
                       float* __restrict__ rstd_out, int rows, int H, float eps) {
  __shared__ float scratch[RN_THREADS / 32];
  const int nvec = H / 8;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    int g = tile_group ? tile_group[row >> 7] : 0;
    if (g < 0) g = 0;
    const uint4* xr = reinterpret_cast<const uint4*>(x + (long long)row * H);
    const uint4* gr = reinterpret_cast<const uint4*>(gain + (long long)g * H);
    uint4* yr = reinterpret_cast<uint4*>(y + (long long)row * H);
    float ss = 0.f;
    for (int v = threadIdx.x; v < nvec; v += RN_THREADS) {
      float f[8];
      unpack8(xr[v], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    }
    ss = block_sum<RN_THREADS>(ss, scratch);
    const float rstd = rsqrtf(ss / H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
    for (int v = threadIdx.x; v < nvec; v += RN_THREADS) {
      float f[8], w[8];
      unpack8(xr[v], f);
      unpack8(gr[v], w);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * w[i];
      yr[v] = pack8(f);
    }
  }
}

// One warp per row, the row held in registers (VPL 16-byte vectors per lane): no block barrier, one read of x,
// VPL independent loads in flight per lane.  Used when H = 256 * VPL; other widths take the kernel above.
template <int VPL>
__global__ void __launch_bounds__(RN_THREADS, 2)
    rmsnorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gain,
                            const int* __restrict__ tile_group, __nv_bfloat16* __restrict__ y,
                            float* __restrict__ rstd_out, int rows, float eps) {
  constexpr int H = 256 * VPL;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (RN_THREADS / 32);
  for (int row = blockIdx.x * (RN_THREADS / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    int g = tile_group ? tile_group[row >> 7] : 0;
    if (g < 0) g = 0;
    const uint4* xr = reinterpret_cast<const uint4*>(x + (long long)row * H);
    const uint4* gr = reinterpret_cast<const uint4*>(gain + (long long)g * H);
    uint4* yr = reinterpret_cast<uint4*>(y + (long long)row * H);
    uint4 v[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) v[j] = xr[lane + 32 * j];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      float f[8];
      unpack8(v[j], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / H + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      float f[8], w[8];
      unpack8(v[j], f);
      unpack8(__ldg(gr + lane + 32 * j), w);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * w[i];
      yr[lane + 32 * j] = pack8(f);
    }
  }
}

// One CTA per row, VPT vectors per thread: for products of few rows, where the warp kernel would leave most SMs without
// work and one warp with 16 loads of its own.  Part of the programmatic-launch chain of a decoder layer.
template <int VPT>
__global__ void __launch_bounds__(RN_THREADS)
    rmsnorm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gain,
                           const int* __restrict__ tile_group, __nv_bfloat16* __restrict__ y,
                           float* __restrict__ rstd_out, int H, float eps) {
  __shared__ float scratch[RN_THREADS / 32];
  const int row = blockIdx.x, nvec = H / 8;
  pdl_wait();
  pdl_trigger();
  int g = tile_group ? tile_group[row >> 7] : 0;
  if (g < 0) g = 0;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (long long)row * H);
  const uint4* gr = reinterpret_cast<const uint4*>(gain + (long long)g * H);
  uint4* yr = reinterpret_cast<uint4*>(y + (long long)row * H);
  uint4 v[VPT], w[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int c = threadIdx.x + j * RN_THREADS;
    v[j] = w[j] = make_uint4(0, 0, 0, 0);
    if (c < nvec) {
      v[j] = xr[c];
      w[j] = __ldg(gr + c);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    float f[8];
    unpack8(v[j], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  ss = block_sum<RN_THREADS>(ss, scratch);
  const float rstd = rsqrtf(ss / H + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int c = threadIdx.x + j * RN_THREADS;
    if (c < nvec) {
      float f[8], gg[8];
      unpack8(v[j], f);
      unpack8(w[j], gg);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * gg[i];
      yr[c] = pack8(f);
    }
  }
}

// dx = rstd * (g*dy - xhat * mean(g*dy*xhat)) (+ dres);  dgain[g] += sum_rows dy * xhat.
// Each CTA owns ROWS_PER_CTA consecutive rows of one tile and keeps its gain
// gradient in registers until the end, then adds it to the fp32 accumulator.
constexpr int RN_ROWS_PER_CTA = 32;
constexpr int RN_MAX_VEC_PER_THREAD = 4;  // H <= 8 * 256 * 4 = 8192

__global__ void __launch_bounds__(RN_THREADS)
    rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                       const __nv_bfloat16* __restrict__ gain, const float* __restrict__ rstd_in,
                       const int* __restrict__ tile_group, const __nv_bfloat16* __restrict__ dres,
                       __nv_bfloat16* __restrict__ dx, float* __restrict__ dgain, int rows, int H) {
  __shared__ float scratch[RN_THREADS / 32];
  const int nvec = H / 8;
  const int row0 = blockIdx.x * RN_ROWS_PER_CTA;
  if (row0 >= rows) return;
  int g = tile_group ? tile_group[row0 >> 7] : 0;
  const bool tile_ok = g >= 0;
  if (g < 0) g = 0;
  const uint4* gr = reinterpret_cast<const uint4*>(gain + (long long)g * H);
  float dg[RN_MAX_VEC_PER_THREAD][8];
#pragma unroll
  for (int j = 0; j < RN_MAX_VEC_PER_THREAD; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) dg[j][i] = 0.f;

  for (int r = 0; r < RN_ROWS_PER_CTA; ++r) {
    const int row = row0 + r;
    if (row >= rows) break;
    const uint4* xr = reinterpret_cast<const uint4*>(x + (long long)row * H);
    const uint4* dyr = reinterpret_cast<const uint4*>(dy + (long long)row * H);
    const float rstd = rstd_in[row];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < RN_MAX_VEC_PER_THREAD; ++j) {
      const int v = threadIdx.x + j * RN_THREADS;
      if (v < nvec) {
        float xf[8], dyf[8], w[8];
        unpack8(xr[v], xf);
        unpack8(dyr[v], dyf);
        unpack8(gr[v], w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xh = xf[i] * rstd;
          dot += dyf[i] * w[i] * xh;
          dg[j][i] += dyf[i] * xh;
        }
      }
    }
    dot = block_sum<RN_THREADS>(dot, scratch) / H;
    uint4* dxr = reinterpret_cast<uint4*>(dx + (long long)row * H);
    const uint4* drr = dres ? reinterpret_cast<const uint4*>(dres + (long long)row * H) : nullptr;
#pragma unroll
    for (int j = 0; j < RN_MAX_VEC_PER_THREAD; ++j) {
      const int v = threadIdx.x + j * RN_THREADS;
      if (v < nvec) {
        float xf[8], dyf[8], w[8], o[8];
        unpack8(xr[v], xf);
        unpack8(dyr[v], dyf);
        unpack8(gr[v], w);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rstd * (dyf[i] * w[i] - xf[i] * rstd * dot);
        if (drr) {
          float rf[8];
          unpack8(drr[v], rf);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += rf[i];
        }
        dxr[v] = pack8(o);
      }
    }
  }
  if (dgain && tile_ok) {
#pragma unroll
    for (int j = 0; j < RN_MAX_VEC_PER_THREAD; ++j) {
      const int v = threadIdx.x + j * RN_THREADS;
      if (v < nvec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) atomicAdd(dgain + (long long)g * H + v * 8 + i, dg[j][i]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// q/k half-head RMSNorm + three-axis RoPE.  head_dim is 128: dims [0,64) carry
// the temporal axis, [64,96) the row axis, [96,128) the column axis.  One warp
// handles one head of one token; lane l owns elements [4l, 4l+4).
//   gains: [groups][4][64] = (q_t, q_hw, k_t, k_hw)
//   pos:   [3][rows] int32 (t, h, w)
// ---------------------------------------------------------------------------
constexpr int QK_THREADS = 128;

struct RopeTable {
  float c[64];  // cos for t pairs [0,32), h pairs [32,48), w pairs [48,64)
  float s[64];
};

__device__ __forceinline__ void fill_rope_table(RopeTable* tab, const int* pos, int rows, int row,
                                                const float* inv_t, const float* inv_hw) {
  for (int i = threadIdx.x; i < 64; i += blockDim.x) {
    float ang;
    if (i < 32) ang = (float)pos[row] * inv_t[i];
    else if (i < 48) ang = (float)pos[rows + row] * inv_hw[i - 32];
    else ang = (float)pos[2 * rows + row] * inv_hw[i - 48];
    float sn, cs;
    sincosf(ang, &sn, &cs);
    tab->c[i] = cs;
    tab->s[i] = sn;
  }
}

// lane -> (table base index, partner xor, sign) for its 4 elements
__device__ __forceinline__ void rope_lane_info(int lane, int& tab0, int& pxor, bool& first_half) {
  if (lane < 16) {  // t block, pairs (i, i+32), 8 lanes per half
    pxor = 8;
    first_half = lane < 8;
    tab0 = (lane & 7) * 4;
  } else if (lane < 24) {  // h block, pairs (i, i+16), 4 lanes per half
    pxor = 4;
    first_half = lane < 20;
    tab0 = 32 + (lane & 3) * 4;
  } else {  // w block
    pxor = 4;
    first_half = lane < 28;
    tab0 = 48 + (lane & 3) * 4;
  }
}

__global__ void __launch_bounds__(QK_THREADS)
    qknorm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld_in,
                           __nv_bfloat16* __restrict__ out, long long ld_out,
                           const __nv_bfloat16* __restrict__ gains,
                           const int* __restrict__ tile_group, const int* __restrict__ pos,
                           const float* __restrict__ inv_t, const float* __restrict__ inv_hw,
                           int rows, int n_q_heads, int n_kv_heads, float eps) {
  __shared__ RopeTable tab;
  const int row = blockIdx.x;
  int g = tile_group ? tile_group[row >> 7] : 0;
  if (g < 0) g = 0;
  fill_rope_table(&tab, pos, rows, row, inv_t, inv_hw);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tab0, pxor;
  bool first;
  rope_lane_info(lane, tab0, pxor, first);
  const int nheads = n_q_heads + n_kv_heads;
  for (int h = warp; h < nheads; h += QK_THREADS / 32) {
    const bool is_k = h >= n_q_heads;
    const __nv_bfloat16* src = qkv + (long long)row * ld_in + h * 128 + lane * 4;
    const uint2 raw = *reinterpret_cast<const uint2*>(src);
    float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    float v[4] = {a.x, a.y, b.x, b.y};
    float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);  // 16-lane halves
    const float rstd = rsqrtf(ss / 64.f + eps);
    const int which = (is_k ? 2 : 0) + (lane >= 16 ? 1 : 0);
    const __nv_bfloat16* gp = gains + ((long long)g * 4 + which) * 64 + (lane & 15) * 4;
    float n[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) n[i] = v[i] * rstd * __bfloat162float(gp[i]);
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, n[i], pxor);
      const float cs = tab.c[tab0 + i], sn = tab.s[tab0 + i];
      o[i] = first ? (n[i] * cs - other * sn) : (n[i] * cs + other * sn);
    }
    uint2 packed;
    packed.x = pack_bf16x2(o[0], o[1]);
    packed.y = pack_bf16x2(o[2], o[3]);
    *reinterpret_cast<uint2*>(out + (long long)row * ld_out + h * 128 + lane * 4) = packed;
  }
}

// The same for a decoder layer of the inference engine, fused with the write into the K/V cache: q goes to ``q_out``,
// k (normalised and rotated) and v to cache row kv_rows[row].  Sixteen lanes of 8 elements own a head.  A CTA
// has one row, or 16 heads of it when rows are few; the heads are loaded before the sine table is ready.  Few rows are
// bound by the launch, many by the chain position -> sine -> norm -> store of a CTA rather than by memory
// ((n_q + 2 n_kv) heads read and written once: 30 us at 8192 rows; four rows per CTA with shared tables: 45 - 48 us).
// 32 / 8 heads, us, against the kernel above and two index copies:
//   rows       1     24    128    300   1024   8192
//   before   9.1   11.0   11.4   11.8   16.5   93.9
//   now      1.8    1.9    2.4    3.8    6.4   46.2
constexpr int QC_THREADS = 256;
constexpr int QC_GROUPS = QC_THREADS / 16;

template <int PER>   // heads per group of lanes
__global__ void __launch_bounds__(QC_THREADS)
    qknorm_rope_cache_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld_in, __nv_bfloat16* __restrict__ q_out,
                             long long ld_q, __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc,
                             long long cache_rows, const long long* __restrict__ kv_rows,
                             const __nv_bfloat16* __restrict__ gains, const int* __restrict__ pos,
                             const float* __restrict__ inv_t, const float* __restrict__ inv_hw, int rows, int n_q,
                             int n_kv, int hpc, float eps, int* status) {
  __shared__ float2 tab[64];      // cos, sin
  const int row = blockIdx.x;
  const int sub = threadIdx.x & 15;
  const int grp = threadIdx.x >> 4;
  const int n_heads = n_q + 2 * n_kv;
  const int h_lo = blockIdx.y * hpc, h_hi = min(n_heads, h_lo + hpc);
  pdl_wait();
  pdl_trigger();
  uint4 raw[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int h = h_lo + grp + j * QC_GROUPS;
    raw[j] = make_uint4(0, 0, 0, 0);
    if (h < h_hi) raw[j] = *reinterpret_cast<const uint4*>(qkv + (long long)row * ld_in + h * 128 + sub * 8);
  }
  const long long dst = kv_rows[row];
  const bool dst_ok = dst >= 0 && dst < cache_rows;
  if (!dst_ok && threadIdx.x == 0) report_status(status, kBadShape, 5);
  if (threadIdx.x < 64) {
    const int i = threadIdx.x;
    float ang;
    if (i < 32) ang = (float)pos[row] * inv_t[i];
    else if (i < 48) ang = (float)pos[rows + row] * inv_hw[i - 32];
    else ang = (float)pos[2 * rows + row] * inv_hw[i - 48];
    float sn, cs;
    sincosf(ang, &sn, &cs);
    tab[i] = make_float2(cs, sn);
  }
  // lane -> first entry of the table, partner, half of the rotation pair
  int tab0, pxor;
  bool first;
  if (sub < 8) {           // t block, pairs (i, i + 32)
    pxor = 4;
    first = (sub & 4) == 0;
    tab0 = (sub & 3) * 8;
  } else {                 // h and w blocks, pairs (i, i + 16)
    pxor = 2;
    first = (sub & 2) == 0;
    tab0 = (sub < 12 ? 32 : 48) + (sub & 1) * 8;
  }
  const uint4 gq = *reinterpret_cast<const uint4*>(gains + (sub >= 8 ? 64 : 0) + (sub & 7) * 8);
  const uint4 gk = *reinterpret_cast<const uint4*>(gains + 128 + (sub >= 8 ? 64 : 0) + (sub & 7) * 8);
  __syncthreads();
  float2 t[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    t[i] = tab[tab0 + i];
    if (first) t[i].y = -t[i].y;
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int h = h_lo + grp + j * QC_GROUPS;
    if (h_lo + (threadIdx.x >> 5) * 2 + j * QC_GROUPS >= h_hi) break;          // both groups of the warp are done
    const bool rot = h < n_q + n_kv;                                           // the heads of v are only copied
    float v[8], g[8], o[8];
    unpack8(raw[j], v);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
#pragma unroll
    for (int x = 4; x > 0; x >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, x);   // halves of 64 elements
    const float rstd = rsqrtf(ss / 64.f + eps);
    unpack8(h >= n_q ? gk : gq, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = v[i] * rstd * g[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = v[i] * t[i].x + __shfl_xor_sync(0xffffffffu, v[i], pxor) * t[i].y;
    if (h >= h_hi) continue;
    const uint4 u = rot ? pack8(o) : raw[j];
    if (h < n_q) *reinterpret_cast<uint4*>(q_out + (long long)row * ld_q + h * 128 + sub * 8) = u;
    else if (dst_ok) {
      __nv_bfloat16* c = rot ? kc + (h - n_q) * 128 : vc + (h - n_q - n_kv) * 128;
      *reinterpret_cast<uint4*>(c + dst * n_kv * 128 + sub * 8) = u;
    }
  }
}

// Backward: d_in = d(norm)(R^T d_out); dgains[g][which][64] += sum d_n * xhat.
// `d` is updated in place (ld_d), qkv holds the saved pre-norm projections.
__global__ void __launch_bounds__(QK_THREADS)
    qknorm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld_in,
                           __nv_bfloat16* __restrict__ d, long long ld_d,
                           const __nv_bfloat16* __restrict__ gains, float* __restrict__ dgains,
                           const int* __restrict__ tile_group, const int* __restrict__ pos,
                           const float* __restrict__ inv_t, const float* __restrict__ inv_hw,
                           int rows, int rows_per_cta, int n_q_heads, int n_kv_heads, float eps) {
  __shared__ RopeTable tab;
  __shared__ float sdg[4 * 64];
  for (int i = threadIdx.x; i < 256; i += QK_THREADS) sdg[i] = 0.f;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tab0, pxor;
  bool first;
  rope_lane_info(lane, tab0, pxor, first);
  const int nheads = n_q_heads + n_kv_heads;
  const int row_begin = blockIdx.x * rows_per_cta;
  int g = tile_group ? tile_group[row_begin >> 7] : 0;  // rows_per_cta divides 128
  const bool tile_ok = g >= 0;
  if (g < 0) g = 0;
  float acc_q[4] = {0.f, 0.f, 0.f, 0.f};
  float acc_k[4] = {0.f, 0.f, 0.f, 0.f};
  for (int r = 0; r < rows_per_cta; ++r) {
    const int row = row_begin + r;
    if (row >= rows) break;
    __syncthreads();
    fill_rope_table(&tab, pos, rows, row, inv_t, inv_hw);
    __syncthreads();
    for (int h = warp; h < nheads; h += QK_THREADS / 32) {
      const bool is_k = h >= n_q_heads;
      const uint2 raw =
          *reinterpret_cast<const uint2*>(qkv + (long long)row * ld_in + h * 128 + lane * 4);
      float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
      float v[4] = {a.x, a.y, b.x, b.y};
      float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float rstd = rsqrtf(ss / 64.f + eps);
      __nv_bfloat16* dp = d + (long long)row * ld_d + h * 128 + lane * 4;
      const uint2 draw = *reinterpret_cast<const uint2*>(dp);
      float2 da = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&draw.x));
      float2 db = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&draw.y));
      float dy[4] = {da.x, da.y, db.x, db.y};
      const int which = (is_k ? 2 : 0) + (lane >= 16 ? 1 : 0);
      const __nv_bfloat16* gp = gains + ((long long)g * 4 + which) * 64 + (lane & 15) * 4;
      float dn[4], xh[4], dxh[4];
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, dy[i], pxor);
        const float cs = tab.c[tab0 + i], sn = tab.s[tab0 + i];
        dn[i] = first ? (dy[i] * cs + other * sn) : (dy[i] * cs - other * sn);
        xh[i] = v[i] * rstd;
        dxh[i] = dn[i] * __bfloat162float(gp[i]);
        dot += dxh[i] * xh[i];
        if (is_k) acc_k[i] += dn[i] * xh[i];
        else acc_q[i] += dn[i] * xh[i];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      dot *= (1.f / 64.f);
      float dx[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) dx[i] = rstd * (dxh[i] - xh[i] * dot);
      uint2 packed;
      packed.x = pack_bf16x2(dx[0], dx[1]);
      packed.y = pack_bf16x2(dx[2], dx[3]);
      *reinterpret_cast<uint2*>(dp) = packed;
    }
  }
  // lane l holds gain-gradient partials for gain (lane>=16 ? hw : t), elements (l&15)*4..+4
  const int half = lane >= 16 ? 1 : 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    atomicAdd(&sdg[(0 + half) * 64 + (lane & 15) * 4 + i], acc_q[i]);
    atomicAdd(&sdg[(2 + half) * 64 + (lane & 15) * 4 + i], acc_k[i]);
  }
  __syncthreads();
  if (dgains && tile_ok)
    for (int i = threadIdx.x; i < 256; i += QK_THREADS) atomicAdd(dgains + (long long)g * 256 + i, sdg[i]);
}

// The same with 16 lanes of 8 elements per head (16-byte aligned rows): the sine tables of the CTA's 16 rows are filled
// once, then the rows are walked without barriers and the next heads are on their way while these are worked on.  The
// kernel above takes two barriers and the table's latency per row.
// 32 / 8 heads, 16384 rows (floor 76 us): 234 -> 184 us, 8192 rows 213 -> 99, 4096 rows 148 -> 51.
constexpr int QB_ROWS = 16;
constexpr int QB_PER = 3;       // heads per group of lanes and step

__global__ void __launch_bounds__(QC_THREADS, 2)
    qknorm_rope_bwd_wide_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld_in, __nv_bfloat16* __restrict__ d,
                                long long ld_d, const __nv_bfloat16* __restrict__ gains, float* __restrict__ dgains,
                                const int* __restrict__ tile_group, const int* __restrict__ pos,
                                const float* __restrict__ inv_t, const float* __restrict__ inv_hw, int rows, int n_q,
                                int n_kv, float eps) {
  __shared__ float2 tab[QB_ROWS][64];
  __shared__ float sdg[4 * 64];
  const int row0 = blockIdx.x * QB_ROWS, nrows = min(QB_ROWS, rows - row0);
  const int lane = threadIdx.x & 31, sub = threadIdx.x & 15, grp = threadIdx.x >> 4;
  const int nheads = n_q + n_kv;
  const int steps = (nheads + QB_PER * QC_GROUPS - 1) / (QB_PER * QC_GROUPS);   // per row
  int g = tile_group ? tile_group[row0 >> 7] : 0;
  const bool tile_ok = g >= 0;
  if (g < 0) g = 0;
  uint4 vn[QB_PER], dn[QB_PER];
  auto load = [&](int it) {
    const long long row = row0 + it / steps;
    const int h0 = (it % steps) * QB_PER * QC_GROUPS + grp;
#pragma unroll
    for (int j = 0; j < QB_PER; ++j) {
      const int h = h0 + j * QC_GROUPS;
      const bool in = h < nheads;
      vn[j] = in ? *reinterpret_cast<const uint4*>(qkv + row * ld_in + h * 128 + sub * 8) : make_uint4(0, 0, 0, 0);
      dn[j] = in ? *reinterpret_cast<const uint4*>(d + row * ld_d + h * 128 + sub * 8) : make_uint4(0, 0, 0, 0);
    }
  };
  load(0);
  sdg[threadIdx.x] = 0.f;
  for (int i = threadIdx.x; i < nrows * 64; i += QC_THREADS) {
    const int row = row0 + (i >> 6), c = i & 63;
    float ang;
    if (c < 32) ang = (float)pos[row] * inv_t[c];
    else if (c < 48) ang = (float)pos[rows + row] * inv_hw[c - 32];
    else ang = (float)pos[2 * rows + row] * inv_hw[c - 48];
    float sn, cs;
    sincosf(ang, &sn, &cs);
    tab[i >> 6][c] = make_float2(cs, sn);
  }
  int tab0, pxor;
  bool first;
  if (sub < 8) {
    pxor = 4;
    first = (sub & 4) == 0;
    tab0 = (sub & 3) * 8;
  } else {
    pxor = 2;
    first = (sub & 2) == 0;
    tab0 = (sub < 12 ? 32 : 48) + (sub & 1) * 8;
  }
  const __nv_bfloat16* gp = gains + (long long)g * 256 + (sub >= 8 ? 64 : 0) + (sub & 7) * 8;
  float gq[8], gk[8], acc_q[8], acc_k[8];
  unpack8(*reinterpret_cast<const uint4*>(gp), gq);
  unpack8(*reinterpret_cast<const uint4*>(gp + 128), gk);
#pragma unroll
  for (int i = 0; i < 8; ++i) acc_q[i] = acc_k[i] = 0.f;
  __syncthreads();
  for (int it = 0; it < nrows * steps; ++it) {
    const int r = it / steps, h0 = (it % steps) * QB_PER * QC_GROUPS;
    uint4 vc[QB_PER], dc[QB_PER];
#pragma unroll
    for (int j = 0; j < QB_PER; ++j) {
      vc[j] = vn[j];
      dc[j] = dn[j];
    }
    if (it + 1 < nrows * steps) load(it + 1);
#pragma unroll
    for (int j = 0; j < QB_PER; ++j) {
      const int h = h0 + grp + j * QC_GROUPS;
      if (h0 + (threadIdx.x >> 5) * 2 + j * QC_GROUPS >= nheads) break;      // both groups of the warp are done
      const bool is_k = h >= n_q;
      float v[8], dy[8];
      unpack8(vc[j], v);
      unpack8(dc[j], dy);
      // two quads per lane, summed over the half head in the order of the narrow kernel's 16 lanes
      float s0 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
      float s1 = v[4] * v[4] + v[5] * v[5] + v[6] * v[6] + v[7] * v[7];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      }
      const float ss = s0 + s1;
      const float rstd = rsqrtf(ss / 64.f + eps);
      float dxh[8], dot2[2] = {0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, dy[i], pxor);
        const float2 t = tab[r][tab0 + i];
        const float dnorm = first ? (dy[i] * t.x + other * t.y) : (dy[i] * t.x - other * t.y);
        v[i] *= rstd;
        dxh[i] = dnorm * (is_k ? gk[i] : gq[i]);
        dot2[i >> 2] += dxh[i] * v[i];
        const float a = dnorm * v[i];
        if (!is_k) acc_q[i] += a;
        else if (h < nheads) acc_k[i] += a;    // past the last head v is 0 * rstd, not a number where eps is 0
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        dot2[0] += __shfl_xor_sync(0xffffffffu, dot2[0], o);
        dot2[1] += __shfl_xor_sync(0xffffffffu, dot2[1], o);
      }
      const float dot = (dot2[0] + dot2[1]) * (1.f / 64.f);
      if (h >= nheads) continue;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = rstd * (dxh[i] - v[i] * dot);
      *reinterpret_cast<uint4*>(d + (long long)(row0 + r) * ld_d + h * 128 + sub * 8) = pack8(v);
    }
  }
  // the two groups of a warp hold the same elements
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc_q[i] += __shfl_xor_sync(0xffffffffu, acc_q[i], 16);
    acc_k[i] += __shfl_xor_sync(0xffffffffu, acc_k[i], 16);
    if (lane < 16) {
      const int e = (sub >= 8 ? 64 : 0) + (sub & 7) * 8 + i;
      atomicAdd(&sdg[e], acc_q[i]);
      atomicAdd(&sdg[128 + e], acc_k[i]);
    }
  }
  __syncthreads();
  if (dgains && tile_ok) atomicAdd(dgains + (long long)g * 256 + threadIdx.x, sdg[threadIdx.x]);
}

// ---------------------------------------------------------------------------
// SwiGLU on the fused projection [rows][gate(F) | up(F)].
// ---------------------------------------------------------------------------
// rows_dev (optional): the number of rows in use, read on the device, for buffers sized for a worst case
// One row per CTA step, columns strided over the threads: no 64-bit division per element vector.
__global__ void __launch_bounds__(256)
    swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, long long rows, int F,
                      const int* __restrict__ rows_dev) {
  if (rows_dev != nullptr && *rows_dev < rows) rows = *rows_dev;
  const int fv = F / 8;
  const int rpc = fv >= 256 ? 1 : 256 / fv;   // narrow rows (expert FFNs): several rows per CTA step
  const int tr = rpc == 1 ? 0 : threadIdx.x / fv;
  const int tc = threadIdx.x - tr * fv;
  for (long long r0 = (long long)blockIdx.x * rpc; r0 < rows; r0 += (long long)gridDim.x * rpc) {
    const long long r = r0 + tr;
    if (tr >= rpc || r >= rows) continue;
    const uint4* base = reinterpret_cast<const uint4*>(gu + r * 2 * F);
    uint4* out = reinterpret_cast<uint4*>(act + r * F);
#pragma unroll 2
    for (int c = tc; c < fv; c += 256) {
      float gt[8], up[8], o[8];
      unpack8(base[c], gt);
      unpack8(base[fv + c], up);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = silu_mul(gt[j], up[j]);
      }
      out[c] = pack8(o);
    }
  }
}

__global__ void __launch_bounds__(256)
    swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dact,
                      __nv_bfloat16* __restrict__ dgu, long long rows, int F, const int* __restrict__ rows_dev) {
  if (rows_dev != nullptr && *rows_dev < rows) rows = *rows_dev;
  const int fv = F / 8;
  const int rpc = fv >= 256 ? 1 : 256 / fv;
  const int tr = rpc == 1 ? 0 : threadIdx.x / fv;
  const int tc = threadIdx.x - tr * fv;
  for (long long r0 = (long long)blockIdx.x * rpc; r0 < rows; r0 += (long long)gridDim.x * rpc) {
    const long long r = r0 + tr;
    if (tr >= rpc || r >= rows) continue;
    const uint4* base = reinterpret_cast<const uint4*>(gu + r * 2 * F);
    const uint4* dab = reinterpret_cast<const uint4*>(dact + r * F);
    uint4* ob = reinterpret_cast<uint4*>(dgu + r * 2 * F);
#pragma unroll 2
    for (int c = tc; c < fv; c += 256) {
      float gt[8], up[8], da[8], dgt[8], dup[8];
      unpack8(base[c], gt);
      unpack8(base[fv + c], up);
      unpack8(dab[c], da);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float sg = fmaf(0.5f, fast_tanh(0.5f * gt[j]), 0.5f);
        const float silu = gt[j] * sg;
        dup[j] = da[j] * silu;
        dgt[j] = da[j] * up[j] * (sg + silu * (1.f - sg));
      }
      ob[c] = pack8(dgt);
      ob[fv + c] = pack8(dup);
    }
  }
}

}  // namespace snu1

using namespace snu1;

// Rows up to which the forward norm gives a CTA to every row.  H = 4096, us per launch, warp kernel / row kernel:
//   rows       1     24    128    512   1184   2048
//            2.8    4.1    4.2    4.6    5.2    6.4     (H = 2048: 1.9 .. 2.9)
//            1.4    1.7    1.7    2.6    3.9      -     (H = 2048: 1.3 .. 2.7)
// Beyond, both are bound by memory and the warp kernel needs no barrier.
static constexpr int kRowKernelRows = 148 * 8;

SNU1_API int snu1_rmsnorm_fwd(const void* x, const void* gain, const int* tile_group, void* y,
                              float* rstd, int rows, int H, float eps, void* stream) {
  if (H % 8 != 0 || rows <= 0) {
    set_last_error("rmsnorm_fwd: H must be a multiple of 8 (H=%d rows=%d)", H, rows);
    return kHostBadArg;
  }
  if (rows <= kRowKernelRows && H <= 8 * RN_THREADS * 4) {
    const __nv_bfloat16 *xp = (const __nv_bfloat16*)x, *gp = (const __nv_bfloat16*)gain;
    const int vpt = (H / 8 + RN_THREADS - 1) / RN_THREADS;
    auto k = vpt <= 1 ? rmsnorm_fwd_row_kernel<1> : vpt == 2 ? rmsnorm_fwd_row_kernel<2> : rmsnorm_fwd_row_kernel<4>;
    SNU1_CUDA_CHECK(launch_pdl(k, dim3(rows), dim3(RN_THREADS), 0, (cudaStream_t)stream, xp, gp, tile_group,
                               (__nv_bfloat16*)y, rstd, H, eps));
    return kHostOk;
  }
  {
    const int wgrid = (rows + 7) / 8 < 148 * 8 ? (rows + 7) / 8 : 148 * 8;
    const __nv_bfloat16 *xp = (const __nv_bfloat16*)x, *gp = (const __nv_bfloat16*)gain;
    __nv_bfloat16* yp = (__nv_bfloat16*)y;
    cudaStream_t st = (cudaStream_t)stream;
    bool done = true;
    switch (H) {
      case 256: rmsnorm_fwd_warp_kernel<1><<<wgrid, RN_THREADS, 0, st>>>(xp, gp, tile_group, yp, rstd, rows, eps); break;
      case 512: rmsnorm_fwd_warp_kernel<2><<<wgrid, RN_THREADS, 0, st>>>(xp, gp, tile_group, yp, rstd, rows, eps); break;
      case 1024: rmsnorm_fwd_warp_kernel<4><<<wgrid, RN_THREADS, 0, st>>>(xp, gp, tile_group, yp, rstd, rows, eps); break;
      case 2048: rmsnorm_fwd_warp_kernel<8><<<wgrid, RN_THREADS, 0, st>>>(xp, gp, tile_group, yp, rstd, rows, eps); break;
      case 4096: rmsnorm_fwd_warp_kernel<16><<<wgrid, RN_THREADS, 0, st>>>(xp, gp, tile_group, yp, rstd, rows, eps); break;
      default: done = false;
    }
    if (done) {
      SNU1_CUDA_CHECK(cudaGetLastError());
      return kHostOk;
    }
  }
  int grid = rows < 148 * 8 ? rows : 148 * 8;
  rmsnorm_fwd_kernel<<<grid, RN_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)gain, tile_group, (__nv_bfloat16*)y, rstd,
      rows, H, eps);
  SNU1_CUDA_CHECK(cudaGetLastError());
  return kHostOk;
}

SNU1_API int snu1_rmsnorm_bwd(const void* dy, const void* x, const void* gain, const float* rstd,
                              const int* tile_group, const void* dres, void* dx, float* dgain,
                              int rows, int H, void* stream) {
  if (H % 8 != 0 || H > 8 * RN_THREADS * RN_MAX_VEC_PER_THREAD || rows <= 0) {
    set_last_error("rmsnorm_bwd: unsupported H=%d (multiple of 8, at most %d)", H,
                   8 * RN_THREADS * RN_MAX_VEC_PER_THREAD);
    return kHostBadArg;
  }
  int grid = (rows + RN_ROWS_PER_CTA - 1) / RN_ROWS_PER_CTA;
  rmsnorm_bwd_kernel<<<grid, RN_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)gain, rstd,
      tile_group, (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, dgain, rows, H);
  SNU1_CUDA_CHECK(cudaGetLastError());
  return kHostOk;
}

SNU1_API int snu1_qknorm_rope_fwd(const void* qkv, long long ld_in, void* out, long long ld_out,
                                  const void* gains, const int* tile_group, const int* pos,
                                  const float* inv_t, const float* inv_hw, int rows, int n_q_heads,
                                  int n_kv_heads, float eps, void* stream) {
  if (rows <= 0 || ld_in % 4 != 0 || ld_out % 4 != 0) {
    set_last_error("qknorm_rope_fwd: bad rows / strides");
    return kHostBadArg;
  }
  qknorm_rope_fwd_kernel<<<rows, QK_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)qkv, ld_in, (__nv_bfloat16*)out, ld_out, (const __nv_bfloat16*)gains,
      tile_group, pos, inv_t, inv_hw, rows, n_q_heads, n_kv_heads, eps);
  SNU1_CUDA_CHECK(cudaGetLastError());
  return kHostOk;
}

// q heads of ``qkv`` -> q_out, k and v heads -> rows kv_rows[] of the caches ([cache_rows][n_kv][128], contiguous).  A row
// index outside the cache is skipped and reported through the status word.
SNU1_API int snu1_qknorm_rope_cache(const void* qkv, long long ld_in, void* q_out, long long ld_q, void* kc, void* vc,
                                    long long cache_rows, const long long* kv_rows, const void* gains, const int* pos,
                                    const float* inv_t, const float* inv_hw, int rows, int n_q, int n_kv, float eps,
                                    void* stream) {
  const int heads = n_q + 2 * n_kv;
  if (rows <= 0 || n_q <= 0 || n_kv <= 0 || ld_in % 8 || ld_q % 8 ||
      ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(kc) |
        reinterpret_cast<uintptr_t>(vc) | reinterpret_cast<uintptr_t>(gains)) & 15) != 0) {
    set_last_error("qknorm_rope_cache: rows=%d, %d + %d heads; rows must be 16-byte aligned", rows, n_q, n_kv);
    return kHostBadArg;
  }
  // few rows: a CTA per 16 heads, so that every group of lanes has one; otherwise a CTA per row (of up to 128 heads)
  const int hpc = rows <= 148 ? QC_GROUPS : heads < 8 * QC_GROUPS ? heads : 8 * QC_GROUPS;
  const int per = (hpc + QC_GROUPS - 1) / QC_GROUPS;
  auto k = per <= 1 ? qknorm_rope_cache_kernel<1> : per <= 3 ? qknorm_rope_cache_kernel<3> : qknorm_rope_cache_kernel<8>;
  SNU1_CUDA_CHECK(launch_pdl(k, dim3(rows, (heads + hpc - 1) / hpc), dim3(QC_THREADS), 0, (cudaStream_t)stream,
                             (const __nv_bfloat16*)qkv, ld_in, (__nv_bfloat16*)q_out, ld_q, (__nv_bfloat16*)kc,
                             (__nv_bfloat16*)vc, cache_rows, kv_rows, (const __nv_bfloat16*)gains, pos, inv_t, inv_hw,
                             rows, n_q, n_kv, hpc, eps, device_status_word()));
  return kHostOk;
}

SNU1_API int snu1_qknorm_rope_bwd(const void* qkv, long long ld_in, void* d, long long ld_d,
                                  const void* gains, float* dgains, const int* tile_group,
                                  const int* pos, const float* inv_t, const float* inv_hw, int rows,
                                  int n_q_heads, int n_kv_heads, float eps, void* stream) {
  if (rows <= 0 || ld_in % 4 != 0 || ld_d % 4 != 0) {
    set_last_error("qknorm_rope_bwd: bad rows / strides");
    return kHostBadArg;
  }
  if (ld_in % 8 == 0 && ld_d % 8 == 0 &&
      ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(gains)) & 15) == 0) {
    qknorm_rope_bwd_wide_kernel<<<(rows + QB_ROWS - 1) / QB_ROWS, QC_THREADS, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)qkv, ld_in, (__nv_bfloat16*)d, ld_d, (const __nv_bfloat16*)gains, dgains, tile_group, pos,
        inv_t, inv_hw, rows, n_q_heads, n_kv_heads, eps);
    SNU1_CUDA_CHECK(cudaGetLastError());
    return kHostOk;
  }
  const int rows_per_cta = 16;
  const int grid = (rows + rows_per_cta - 1) / rows_per_cta;
  qknorm_rope_bwd_kernel<<<grid, QK_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)qkv, ld_in, (__nv_bfloat16*)d, ld_d, (const __nv_bfloat16*)gains,
      dgains, tile_group, pos, inv_t, inv_hw, rows, rows_per_cta, n_q_heads, n_kv_heads, eps);
  SNU1_CUDA_CHECK(cudaGetLastError());
  return kHostOk;
}

// rows_dev may be null; otherwise only min(rows, *rows_dev) rows are processed (count known on the device only)
SNU1_API int snu1_swiglu_fwd_dyn(const void* gu, void* act, long long rows, int F, const int* rows_dev, void* stream) {
  if (F % 8 != 0 || rows <= 0) {
    set_last_error("swiglu_fwd: F must be a multiple of 8");
    return kHostBadArg;
  }
  const int rpc = F / 8 >= 256 ? 1 : 256 / (F / 8);
  const long long steps = (rows + rpc - 1) / rpc;
  int grid = (int)(steps < 148 * 8 ? steps : 148 * 8);
  swiglu_fwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)gu,
                                                            (__nv_bfloat16*)act, rows, F, rows_dev);
  SNU1_CUDA_CHECK(cudaGetLastError());
  return kHostOk;
}

SNU1_API int snu1_swiglu_fwd(const void* gu, void* act, long long rows, int F, void* stream) {
  return snu1_swiglu_fwd_dyn(gu, act, rows, F, nullptr, stream);
}

SNU1_API int snu1_swiglu_bwd_dyn(const void* gu, const void* dact, void* dgu, long long rows, int F,
                                 const int* rows_dev, void* stream) {
  if (F % 8 != 0 || rows <= 0) {
    set_last_error("swiglu_bwd: F must be a multiple of 8");
    return kHostBadArg;
  }
  const int rpc = F / 8 >= 256 ? 1 : 256 / (F / 8);
  const long long steps = (rows + rpc - 1) / rpc;
  int grid = (int)(steps < 148 * 8 ? steps : 148 * 8);
  swiglu_bwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)gu, (const __nv_bfloat16*)dact, (__nv_bfloat16*)dgu, rows, F, rows_dev);
  SNU1_CUDA_CHECK(cudaGetLastError());
  return kHostOk;
}

SNU1_API int snu1_swiglu_bwd(const void* gu, const void* dact, void* dgu, long long rows, int F,
                             void* stream) {
  return snu1_swiglu_bwd_dyn(gu, dact, dgu, rows, F, nullptr, stream);
}
