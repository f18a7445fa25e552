// decode_stack: all decoder layers of one decode step (one token of one or two documents) in ONE launch.
//
// What bounds a decode step is the stream of weights from HBM.  As a chain of launches (norm, product, rotary norm, attention,
// product, norm, product, product) every product ends with a tail and the next one starts with a ramp in which memory idles:
// 80 us per 8B layer for 386 MB.  Here one CTA per SM stays for the whole step and two independent roles share it:
//
//  * a producer warp walks all weights of all layers in the order of use and copies this CTA's rows into a ring of shared
//    memory stages (16 rows x 1024 of the reduction, cp.async.bulk).  It waits for ring space only, never for activations,
//    so the next product's weights arrive while activations travel, a norm or the attention of the layer runs;
//  * eight consumer warps run the phases QKV | attention | output | gate and up with SwiGLU | down.
//
// Activations go from CTA to CTA through L2 without a barrier: a word is two bf16 and the number of the phase in one 64-bit access;
// readers poll the words that they need.  (With a grid barrier per phase - fence, arrival, poll, then the loads - a boundary
// took 6 us, more than the ring covers, and a layer longer than as a chain of launches.)  A word is not overwritten before all
// its readers are through: the writer of the next layer's word has consumed, through the phases in between, results of every
// reader.
//
// Products: every CTA owns an even number of consecutive weight rows (gate and up rows of the same outputs), so that no CTA
// has more than a per cent or two above the others; the rows of the residual stream stay in its shared memory.  Every warp
// takes an eighth of each stage's reduction: the weights are the A operand of mma.sync m16n8k16 (16-byte fragment loads: the
// reduction index is permuted within 32 the same way on both sides), the rows of x the B operand.  mma.sync is enough: one
// multiply-add per row of x and weight, the tensor pipe is idle nearly all the time.  Partial sums of the warps meet in shared
// memory in a fixed order.
//
// Attention: a unit is (row of x, four query heads, part of the keys); the parts meet in the same way as activations do, each
// CTA finishing a share of the outputs in a fixed order.  The unit normalises and rotates its own q heads; the new key and
// value are taken from shared memory and stored to the cache by one unit.
//
// Measured, us per 8B layer (386 MB; 59.8 at the measured copy bandwidth), chain of launches / this kernel:
//   keys                50     839    1500    2000    3000    5000        2 x 50   2 x 1500      3 x 50    4 x 50
//                 78.8/70.9 82.6/73.6 85.4/78.0 86.0/79.9 87.9/85.0 93.5/100  79.6/75.2 93.7/88.5  80.3/86.4 81.3/108
//   two documents, keys of each  500, 50  1500, 50  1750, 50  2000, 50  2 x 1750  2 x 2000  2 x 2500   2 x 3000  3000, 50
//                               83.1/76.8 91.3/87.5 90.8/90.9 91.0/92.4 93.7/91.8 94.0/93.7 96.8/98.4 97.1/101.4 91.6/99.7
// With three rows or more x takes the ring's place (4 and 3 stages) and the small phases grow; long documents are better off
// with the attention kernel's deeper pipeline.  Hence the lines at two rows, and at 3072 keys of one document or 1792 of the
// longer of two.
// What bounds it now: 8 us from the last stage of QKV to the first of the output product (two hops of 2 us and the unit's own
// chain), of which the ring covers 4.4.  Tried: asking L2 for stages beyond the ring (2 us per layer slower at any distance), one
// accumulator per tile (a product waits 70 clocks for the one before it).  Nine warps leave 168
// registers a thread (three of them share a quarter of the SM); one row spills 444 bytes, two rows 548 (stores).
// The split follows the keys that the request may reach (max_keys), so a short document with a large budget has small parts.  50 keys,
// chain / this kernel, budget of 32 tokens 80.0/70.7, 500 82.9/71.7, 1000 86.3/73.2, 3000 85.1/73.3.
//
// The launch is cooperative (all CTAs are resident).  Every wait is bounded; a CTA that gives up raises a flag that the
// others poll, and the kernel then refuses later launches on the same scratch.
#include <string.h>

#include <mutex>

#include "attn_common.cuh"
#include "host_common.h"

namespace snu1 {
namespace dstack {

constexpr int CW = 8;                       // consumer warps
constexpr int CT = CW * 32;
constexpr int THREADS = CT + 32;
constexpr int MAXM = 2;                     // rows of x
constexpr int UR = 16;                      // weight rows per tile
constexpr int KC = 1024;                    // reduction per stage
constexpr int PITCH = KC * 2 + 64;          // rows 64 bytes apart in the banks: fragment loads without conflicts
constexpr int STAGE = UR * PITCH;
constexpr int MAX_STAGES = 6, MIN_STAGES = 5;
constexpr int MAXU = 12;                    // tiles whose sums a pass keeps in registers
constexpr int PK = KC / CW;                 // a warp's part of a stage's reduction
constexpr int RED = 4096;                   // floats of the reduction buffer
constexpr int XROW = PK * 2;           // bytes of a warp's part of one row of x in a stage's reduction
constexpr int HG = 4;                       // query heads per attention unit
constexpr int MAX_LAYERS = 48;              // per launch: the table of pointers is a kernel argument
constexpr int MAX_SPLIT = 32;
constexpr int OWN = 64;                     // rows of the residual stream per CTA at most
constexpr int PART = HG * 128 + 2 * HG;     // words of one part's result: weighted V, maximum, sum
constexpr int U = 4, GROUPS = CW * 2;       // attention: keys per group of 16 lanes and step, groups

struct Smem {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES];
  float q[HG][128];
  uint4 kv[2][16];                          // new key and value of the unit's K/V head
  float am[CW][HG], al[CW][HG];
  float ss[CW][MAXM];
  int abort, stop;
};
constexpr int SMEM = 227 * 1024;
// After the ring: x of a phase (it serves the reductions when all warps are through with x), the residual rows, the sines.
__host__ __device__ constexpr int x_bytes(int M, int K) {
  const int b = K / KC * CW * M * XROW;
  return b > RED * 4 ? b : RED * 4;
}
__host__ __device__ constexpr int rest_bytes(int M) { return 2 * OWN * M * 4 + M * 64 * 8 + (int)sizeof(Smem) + 128; }
__host__ __device__ constexpr int stages_for(int M, int K) {
  const int n = (SMEM - rest_bytes(M) - x_bytes(M, K)) / STAGE;
  return n < MAX_STAGES ? n : MAX_STAGES;
}
static_assert(stages_for(1, 12288) == 6 && stages_for(2, 12288) == 5, "a ring of 170 - 200 KB for the 8B model");

struct Layer {
  const __nv_bfloat16 *wqkv, *wo, *w13, *w2, *attn_norm, *qk_norm, *ffn_norm;
  __nv_bfloat16 *kc, *vc;
};

struct Args {
  Layer layer[MAX_LAYERS];
  int layers;
  int M, H, F, Hq, Hkv, split, Sk;
  int stages, x_size;
  long long cache_rows;
  const __nv_bfloat16* x_in;                // [M][H]
  __nv_bfloat16* x_out;                     // [M][H]
  // words (two values, phase number) between CTAs
  uint2 *x, *x1, *qkv, *o, *act;            // [M][H / 2], [M][H / 2], [M][(Hq + 2 Hkv) 64], [M][Hq 64], [M][F / 2]
  uint2* part;                              // [M][Hq / HG][split][PART]: one fp32 value per word
  unsigned int* count;                      // [CTAs] launches so far, by this CTA; [CTAs]: non-zero after a launch that gave up
  const TokMeta *meta_q, *meta_k;
  const int* first;
  const long long* last;                    // cache row of the new token
  const int* pos;                           // [3][M]
  const float *inv_t, *inv_hw;
  float eps, inv_h, scale_log2;
  int* status;
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1, bool first) {
  if (first) c[0] = c[1] = c[2] = c[3] = 0.f;
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

enum Phase { QKV, OUT, UP, DOWN };

// One product of one layer as both roles see it.  Every CTA owns ``per`` consecutive rows of w (gate and up: and the same rows
// of the second half), an even number; tiles of ``tile`` rows.
struct Product {
  const __nv_bfloat16* w;
  int K, lo, hi, tile;
  __device__ __forceinline__ int count() const { return lo < hi ? (hi - lo + tile - 1) / tile : 0; }
};
__device__ __forceinline__ Product product(const Args& a, int l, int ph) {
  const Layer& L = a.layer[l];
  const int rows = ph == QKV ? (a.Hq + 2 * a.Hkv) * 128 : ph == UP ? a.F : a.H;
  const int per = ((rows + gridDim.x - 1) / gridDim.x + 1) & ~1;
  const int lo = min(rows, (int)blockIdx.x * per);
  return {ph == QKV ? L.wqkv : ph == OUT ? L.wo : ph == UP ? L.w13 : L.w2, ph == OUT ? a.Hq * 128 : ph == DOWN ? a.F : a.H, lo,
          min(rows, lo + per), ph == UP ? UR / 2 : UR};
}

// Documents, heads and keys of attention unit ``ua``.
struct Unit {
  int sp, hgp, m, kvh, lo, hi;
  long long last;
};
__device__ __forceinline__ Unit attention_unit(const Args& a, int ua) {
  const int NG = a.Hq / HG, per_kv = a.Hq / a.Hkv / HG;
  Unit u;
  u.sp = ua % a.split;
  u.hgp = ua / a.split % NG;
  u.m = ua / (a.split * NG);
  u.kvh = u.hgp / per_kv;
  u.last = a.last[u.m];
  const int lo = max(0, a.first[u.m]);
  const int len = max(0, (int)max(0ll, min((long long)a.Sk, u.last + 1)) - lo);
  u.lo = lo + (int)((long long)len * u.sp / a.split);
  u.hi = lo + (int)((long long)len * (u.sp + 1) / a.split);
  return u;
}

// What layer l's small phases read from memory, asked for a phase ahead by the producer warp: a load that misses L2 queues
// behind all the weights that the rings have asked for (4 us).  ``u``: the attention unit of this CTA.
__device__ __forceinline__ void fetch_small(const Args& a, const Unit& u, int l, int lane) {
  constexpr int MAX_KEYS = 256;              // of a unit: 19 MB over the chip
  if (l >= a.layers) return;
  const Layer& L = a.layer[l];
  if (blockIdx.x == 0 && lane == 0) {
    l2_prefetch(L.attn_norm, a.H * 2);
    l2_prefetch(L.ffn_norm, a.H * 2);
    l2_prefetch(L.qk_norm, 512);
  }
  for (int k = u.lo + lane; k < min(u.hi, u.lo + MAX_KEYS); k += 32) {
    l2_prefetch(L.kc + ((long long)k * a.Hkv + u.kvh) * 128, 256);
    l2_prefetch(L.vc + ((long long)k * a.Hkv + u.kvh) * 128, 256);
  }
}

// weights are read once: they leave L2 first and let the activations and the cache rows stay
__device__ __forceinline__ uint64_t evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ void produce(const Args& a, uint8_t* ring, Smem& s, int lane) {
  volatile int* abort_flag = &s.abort;
  const uint32_t stages = a.stages;
  const uint64_t policy = evict_first();
  uint32_t it = 0, st = 0, par = 1;                          // a fresh stage counts as empty
  bool ok = true;
  Unit unit{};
  if ((int)blockIdx.x < a.M * (a.Hq / HG) * a.split) unit = attention_unit(a, blockIdx.x);
  fetch_small(a, unit, 0, lane);
  for (int l = 0; l < a.layers && ok; ++l) {
    for (int ph = QKV; ph <= DOWN && ok; ++ph) {
      const Product p = product(a, l, ph);
      const int n = p.count(), r = ph == UP ? lane & 7 : lane, rows = lane < UR ? p.hi - p.lo - r : 0;
      const __nv_bfloat16* w = p.w + (long long)(p.lo + r + (ph == UP && lane >= 8 ? a.F : 0)) * p.K;
      const long long next = (long long)p.tile * p.K;
      if (ph == UP) fetch_small(a, unit, l + 1, lane);
      for (int c = 0; c < p.K && ok; c += KC) {
        const __nv_bfloat16* src = w + c;
        for (int u = 0; u < n; ++u, src += next) {
          if (!mbar_wait_warp(&s.empty[st], par, abort_flag, a.status, 1)) {
            ok = false;
            break;
          }
          if (lane == 0) mbar_expect_tx(&s.full[st], (ph == UP ? 2 : 1) * min(p.tile, p.hi - p.lo - u * p.tile) * (KC * 2));
          __syncwarp();
          if (u * p.tile < rows) bulk_load(ring + st * STAGE + lane * PITCH, src, KC * 2, &s.full[st], policy);
          ++it;
          if (++st == stages) {
            st = 0;
            par ^= 1;
          }
        }
      }
    }
  }
  // nobody leaves while a copy into this CTA's shared memory is on its way (after a time-out nobody else waits for it)
  if (lane == 0) {
    int never = 0;
    for (uint32_t i = it > stages ? it - stages : 0; i < it; ++i)
      mbar_wait(&s.full[i % stages], (i / stages) & 1, &never, a.status, 1);
  }
}

// ---- words between CTAs: a payload (low half) and its phase number (high half) in ONE element of 64 bits.  That they become
// visible together is promised of an element only: of v2.u32 / v4.u32 every 32 bits are an access of their own.  The same time: a
// layer of 50 keys took 71.3 us with those, 70.9 with these and a barrier more. ----
__device__ __forceinline__ uint2 halves(uint64_t w) { return make_uint2((uint32_t)w, (uint32_t)(w >> 32)); }
__device__ __forceinline__ uint4 ld_words(const uint2* p) {
  uint64_t a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  const uint2 x = halves(a), y = halves(b);
  return make_uint4(x.x, x.y, y.x, y.y);
}
__device__ __forceinline__ uint2 ld_word(const uint2* p) {
  uint64_t a;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return halves(a);
}
__device__ __forceinline__ void st_word(uint2* p, uint32_t v, uint32_t phase) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((uint64_t)phase << 32 | v) : "memory");
}
// Polls until ``ready()`` holds in all lanes of the warp (``ready`` loads what is missing); false when it took too long or
// another CTA gave up.
template <typename F>
__device__ __forceinline__ bool poll(const Args& a, Smem& s, F ready) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (!__all_sync(0xffffffffu, ready())) {
    if ((++spins & 0x3f) != 16) continue;
    const uint64_t now = globaltimer_ns();
    if (t0 == 0) t0 = now;
    const bool late = now - t0 > kLocalWaitNs;
    unsigned int* dead = a.count + gridDim.x;
    if (late) {
      atomicExch(dead, 1u);
      report_status(a.status, kWaitTimeout, 7);
    }
    if (__any_sync(0xffffffffu, late || *(volatile int*)&s.abort || *(volatile unsigned int*)dead)) {
      *(volatile int*)&s.abort = 1;
      return false;
    }
  }
  return true;
}

// One phase of the consumers: y = f(norm(x) w^T).  x is in words of phase ``in`` (``x_in``: plain rows, the input of the
// launch).  ``gain``: x is normalised on the way (rounded to bf16 as the norm kernel stores it).  ``own``: this CTA's rows of the
// residual stream, added to the product; the sum goes to ``own_out`` as well.  y: words of phase ``out``, or plain rows in
// ``y_out``.  A time-out only sets s.abort: everything after it works on whatever is there, and the layers end.
template <int M, bool UP_PHASE>
__device__ __forceinline__ void multiply(const Args& a, uint8_t* ring, uint8_t* xbuf, Smem& s, const Product& p, uint32_t& st,
                                         uint32_t& par, const uint2* x, const __nv_bfloat16* x_in, uint32_t in,
                                         const __nv_bfloat16* gain, const float* own, float* own_out, uint2* y,
                                         __nv_bfloat16* y_out, int ldy, uint32_t out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  constexpr int OR = UP_PHASE ? UR / 2 : UR;                 // rows of y per tile
  volatile int* abort_flag = &s.abort;
  const int n = p.count();
  if (n == 0) return;
  const uint32_t stages = a.stages;
  const int chunks = p.K / KC, todo = chunks * M;
  // this warp's part of x: [stage][row][128 elements], the 64-byte quarters of odd rows exchanged against bank conflicts
  uint8_t* xs = xbuf + warp * todo * XROW;
  auto xat = [&](int i, int r) { return reinterpret_cast<uint2*>(xs + i * XROW + (((lane >> 1) ^ ((r & 1) << 2)) << 4) + (lane & 1) * 8); };
  constexpr int B = M == 1 ? 6 : 4 * M;                      // rows of stages on their way; all of them for a normalised x
  const int at0 = warp * PK + lane * 4, half_k = p.K / 2;    // this lane's four elements of row i % M, stage i / M
  for (int i0 = 0; i0 < todo; i0 += B) {
    uint4 v[B];
    const uint2* xw = x + at0 / 2 + i0 / M * (KC / 2);       // B is a multiple of M
    uint2 gw[B / M + 1];
    if (gain != nullptr) {
#pragma unroll
      for (int j = 0; j < B / M; ++j)
        if (j < chunks) gw[j] = __ldg(reinterpret_cast<const uint2*>(gain + j * KC + at0));
    }
    if (x_in != nullptr) {
#pragma unroll
      for (int b = 0; b < B; ++b)
        if (i0 + b < todo) {
          const uint2 w = *reinterpret_cast<const uint2*>(x_in + b % M * p.K + (i0 + b) / M * KC + at0);
          v[b] = make_uint4(w.x, in, w.y, in);
        }
    } else {
      poll(a, s, [&]() {
#pragma unroll
        for (int b = 0; b < B; ++b)
          if (i0 + b < todo) v[b] = ld_words(xw + b % M * half_k + b / M * (KC / 2));
        bool ok = true;
#pragma unroll
        for (int b = 0; b < B; ++b)
          if (i0 + b < todo) ok &= v[b].y == in && v[b].w == in;
        return ok;
      });
    }
    if (gain != nullptr) {
      float ss[M];
#pragma unroll
      for (int m = 0; m < M; ++m) ss[m] = 0.f;
#pragma unroll
      for (int b = 0; b < B; ++b)
        if (b < todo) {
          const float f0 = __uint_as_float(v[b].x << 16), f1 = __uint_as_float(v[b].x & 0xffff0000u);
          const float f2 = __uint_as_float(v[b].z << 16), f3 = __uint_as_float(v[b].z & 0xffff0000u);
          ss[b % M] += f0 * f0 + f1 * f1 + f2 * f2 + f3 * f3;
        }
#pragma unroll
      for (int m = 0; m < M; ++m) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss[m] += __shfl_xor_sync(0xffffffffu, ss[m], o);
        if (lane == 0) s.ss[warp][m] = ss[m];
      }
      named_bar_sync(1, CT);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < CW; ++w) t += s.ss[w][m];
        ss[m] = rsqrtf(t * a.inv_h + a.eps);
      }
#pragma unroll
      for (int b = 0; b < B; ++b)
        if (b < todo) {
          auto scale2 = [&](uint32_t f, uint32_t w) {
            return pack_bf16x2(__uint_as_float(f << 16) * ss[b % M] * __uint_as_float(w << 16),
                               __uint_as_float(f & 0xffff0000u) * ss[b % M] * __uint_as_float(w & 0xffff0000u));
          };
          v[b].x = scale2(v[b].x, gw[b / M].x);
          v[b].z = scale2(v[b].z, gw[b / M].y);
        }
    }
#pragma unroll
    for (int b = 0; b < B; ++b)
      if (i0 + b < todo) *xat(i0 + b, b % M) = make_uint2(v[b].x, v[b].z);
  }
  __syncwarp();
  float acc[MAXU][4];
#pragma unroll
  for (int u = 0; u < MAXU; ++u) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.f;
  const uint8_t* w0 = ring + g * PITCH + warp * PK * 2 + q * 16;
  const uint8_t* xp = xs + g * XROW;
  const int swz = (g & 1) << 2;
  for (int j = 0; j < chunks; ++j, xp += M * XROW) {
    uint4 xb[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      xb[b] = make_uint4(0, 0, 0, 0);
      if (g < M) xb[b] = *reinterpret_cast<const uint4*>(xp + (((b * 4 + q) ^ swz) << 4));
    }
#pragma unroll
    for (int u = 0; u < MAXU; ++u) {
      if (u >= n) break;              // one jump: the bodies are far apart for the instruction cache
      mbar_wait_warp(&s.full[st], par, abort_flag, a.status, 3);
      const uint8_t* wp = w0 + st * STAGE;
      float t[4][4];                  // four chains of two products: one waits for the one before it in its accumulator
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const uint4 lo = *reinterpret_cast<const uint4*>(wp + b * 64);
        const uint4 hi = *reinterpret_cast<const uint4*>(wp + 8 * PITCH + b * 64);
        mma16816(t[b], lo.x, hi.x, lo.y, hi.y, xb[b].x, xb[b].y, true);
        mma16816(t[b], lo.z, hi.z, lo.w, hi.w, xb[b].z, xb[b].w, false);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.empty[st]);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][i] += (t[0][i] + t[1][i]) + (t[2][i] + t[3][i]);
      if (++st == stages) {
        st = 0;
        par ^= 1;
      }
    }
  }
  // sums over the warps: [tile][warp][row of x][weight row]
  float* red = reinterpret_cast<float*>(xbuf);
  constexpr int RU = MAXU < RED / (CW * UR * M) ? MAXU : RED / (CW * UR * M);       // tiles per reduction
#pragma unroll
  for (int r0 = 0; r0 < MAXU; r0 += RU) {
    if (r0 >= n) break;
    named_bar_sync(1, CT);
#pragma unroll
    for (int u = r0; u < r0 + RU && u < MAXU; ++u) {
      if (u >= n) break;
      float* d = red + ((u - r0) * CW + warp) * M * UR + g;
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (2 * q + j < M) {
          d[(2 * q + j) * UR] = acc[u][j];
          d[(2 * q + j) * UR + 8] = acc[u][2 + j];
        }
    }
    named_bar_sync(1, CT);
    // two rows of y per thread
    for (int i = threadIdx.x; i < min(RU, n - r0) * M * (OR / 2); i += CT) {
      const int r = i % (OR / 2) * 2, rest = i / (OR / 2), u = rest / M, m = rest % M;
      const int row = p.lo + (r0 + u) * OR + r;
      if (row >= p.hi) continue;
      float2 v = make_float2(0.f, 0.f), up = v;
#pragma unroll
      for (int w = 0; w < CW; ++w) {
        const float* d = red + ((u * CW + w) * M + m) * UR + r;
        const float2 f = *reinterpret_cast<const float2*>(d);
        v.x += f.x;
        v.y += f.y;
        if (UP_PHASE) {
          const float2 f2 = *reinterpret_cast<const float2*>(d + UR / 2);
          up.x += f2.x;
          up.y += f2.y;
        }
      }
      if (UP_PHASE) {
        v.x = silu_mul(round_bf16(v.x), round_bf16(up.x));
        v.y = silu_mul(round_bf16(v.y), round_bf16(up.y));
      }
      const int at = m * OWN + row - p.lo;
      if (own != nullptr) {
        v.x += own[at];
        v.y += own[at + 1];
      }
      const uint32_t h = pack_bf16x2(v.x, v.y);
      if (y_out != nullptr) *reinterpret_cast<uint32_t*>(y_out + (long long)m * ldy + row) = h;
      else st_word(y + (m * ldy + row) / 2, h, out);
      if (own_out != nullptr) {
        own_out[at] = __uint_as_float(h << 16);
        own_out[at + 1] = __uint_as_float(h & 0xffff0000u);
      }
    }
  }
  named_bar_sync(1, CT);                                       // the next phase's x may overwrite the sums
}

// Keys and values of one step of a unit: 16 lanes per key, 8 of its elements each, U keys per group of lanes.
struct Keys {
  uint4 k[U], v[U];
  int4 meta[U];
};
__device__ __forceinline__ void load_keys(const Args& a, const Layer& L, const Unit& t, int k0, Keys& x) {
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 4;
  const __nv_bfloat16 *kb = L.kc + t.kvh * 128 + (lane & 15) * 8, *vb = L.vc + t.kvh * 128 + (lane & 15) * 8;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int key = k0 + u * GROUPS + grp;
    const int r = key < t.hi ? key : t.lo;                   // past the end: a row of the range, masked later
    if (r >= t.hi) continue;
    x.meta[u] = *reinterpret_cast<const int4*>(a.meta_k + r);
    if (r == t.last) continue;                               // the new key: taken from shared memory later
    const long long at = (long long)r * a.Hkv * 128;
    x.k[u] = *reinterpret_cast<const uint4*>(kb + at);
    x.v[u] = *reinterpret_cast<const uint4*>(vb + at);
  }
}
// Sums over the 16 lanes of a key: lane ``sub`` returns head sub / 4 (every exchange halves the heads that a lane carries).
__device__ __forceinline__ float heads_sum(const float (&d)[HG], int sub) {
  static_assert(HG == 4, "two exchanges");
  const bool b = (sub & 8) != 0, c = (sub & 4) != 0;
  float k0 = b ? d[2] : d[0], k1 = b ? d[3] : d[1];
  k0 += __shfl_xor_sync(0xffffffffu, b ? d[0] : d[2], 8);
  k1 += __shfl_xor_sync(0xffffffffu, b ? d[1] : d[3], 8);
  float r = c ? k1 : k0;
  r += __shfl_xor_sync(0xffffffffu, c ? k0 : k1, 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}
// the value that the lanes of head ``h`` hold, in all lanes of the key
__device__ __forceinline__ float of_head(float x, int h, int lane) { return __shfl_sync(0xffffffffu, x, (lane & 16) | h * 4); }

// Attention of the new rows against their documents' cache rows.  ``in``, ``out``, ``mid``: phase numbers of qkv, of the result and
// of the parts of it.
__device__ __forceinline__ void attend(const Args& a, Smem& s, float* red, const float2* rope, const Layer& L, Unit t, uint32_t in,
                                       uint32_t out, uint32_t mid) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 15, grp = threadIdx.x >> 4;
  const int NG = a.Hq / HG, per_kv = a.Hq / a.Hkv / HG;
  const int units = a.M * NG * a.split;
  const long long ldk = (long long)a.Hkv * 128;
  // One turn: there are never more units than CTAs (snu1_decode_stack_takes leaves at most 60 of (row, four heads), the split fills the
  // rest).  Without the loop the compiler spills twice as much, us per layer with / without: 3000 keys 85.7/90.9, 2 x 1000 84.0/90.8.
  for (int ua = blockIdx.x; ua < units; ua += gridDim.x) {
    if (ua != (int)blockIdx.x) t = attention_unit(a, ua);
    Keys x{};
    load_keys(a, L, t, t.lo, x);                             // on their way while the projections are awaited
    named_bar_sync(1, CT);                                   // the unit before has left the buffers
    const int sp = t.sp, hgp = t.hgp, m = t.m, kvh = t.kvh, h0 = hgp * HG, k_lo = t.lo, k_hi = t.hi;
    const long long last = t.last;
    const int4 mqr = *reinterpret_cast<const int4*>(a.meta_q + m);
    const TokMeta mq{mqr.x, mqr.y, mqr.z, mqr.w};
    if (warp < (HG + 2) / 2) {
      // q heads, the key and the value of this row: 16 lanes of 8 elements each
      const int head = grp;
      const int src = head < HG ? h0 + head : head == HG ? a.Hq + kvh : a.Hq + a.Hkv + kvh;
      const uint2* qp = a.qkv + ((long long)m * (a.Hq + 2 * a.Hkv) + src) * 64 + sub * 4;
      const __nv_bfloat16* gp = L.qk_norm + (head >= HG ? 128 : 0) + (sub >= 8 ? 64 : 0) + (sub & 7) * 8;
      const uint4 gr = __ldg(reinterpret_cast<const uint4*>(gp));
      uint4 w0, w1;
      poll(a, s, [&]() {
        w0 = ld_words(qp);
        w1 = ld_words(qp + 2);
        return w0.y == in && w0.w == in && w1.y == in && w1.w == in;
      });
      const uint4 raw = make_uint4(w0.x, w0.z, w1.x, w1.z);
      float v[8], g[8], o[8];
      unpack8(raw, v);
      unpack8(gr, g);
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
#pragma unroll
      for (int x = 4; x > 0; x >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, x);      // halves of 64 elements
      const float rstd = rsqrtf(ss / 64.f + a.eps);
      // pairs (i, i + 32) of the t block, (i, i + 16) of the h and w blocks
      const int pxor = sub < 8 ? 4 : 2;
      const bool lower = (sub & pxor) == 0;
      const int tab = sub < 8 ? (sub & 3) * 8 : (sub < 12 ? 32 : 48) + (sub & 1) * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = v[i] * rstd * g[i];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 t = rope[m * 64 + tab + i];
        const float other = __shfl_xor_sync(0xffffffffu, v[i], pxor);
        o[i] = v[i] * t.x + other * (lower ? -t.y : t.y);
      }
      if (head < HG) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s.q[head][sub * 8 + i] = round_bf16(o[i]) * a.scale_log2;
      } else {
        const uint4 u = head == HG ? pack8(o) : raw;
        s.kv[head - HG][sub] = u;
        if (sp == a.split - 1 && hgp % per_kv == 0) {
          if (last >= 0 && last < a.cache_rows)
            *reinterpret_cast<uint4*>((head == HG ? L.kc : L.vc) + last * ldk + kvh * 128 + sub * 8) = u;
          else if (sub == 0)
            report_status(a.status, kBadShape, 5);
        }
      }
    }
    named_bar_sync(1, CT);

    uint64_t q2[HG][4], acc[HG][4];
#pragma unroll
    for (int h = 0; h < HG; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = *reinterpret_cast<const float2*>(&s.q[h][sub * 8 + i * 2]);
        q2[h][i] = pack_f32x2(f.x, f.y);
        acc[h][i] = 0ull;
      }
    float mx = -INFINITY, l = 0.f;                           // of this lane's head, over the keys of its group
    for (int k0 = k_lo; k0 < k_hi; k0 += GROUPS * U) {
      if (k0 != k_lo) load_keys(a, L, t, k0, x);
      float sc[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int key = k0 + u * GROUPS + grp;
        if ((key < k_hi ? key : k_lo) == last) {
          x.k[u] = s.kv[0][sub];
          x.v[u] = s.kv[1][sub];
        }
        const uint32_t w[4] = {x.k[u].x, x.k[u].y, x.k[u].z, x.k[u].w};
        float d[HG];
#pragma unroll
        for (int h = 0; h < HG; ++h) {
          uint64_t d0 = mul_f32x2(q2[h][0], bf16x2_to_f32x2(w[0])), d1 = mul_f32x2(q2[h][1], bf16x2_to_f32x2(w[1]));
          d0 = fma_f32x2(q2[h][2], bf16x2_to_f32x2(w[2]), d0);
          d1 = fma_f32x2(q2[h][3], bf16x2_to_f32x2(w[3]), d1);
          float e, o;
          unpack_f32x2(add_f32x2(d0, d1), e, o);
          d[h] = e + o;
        }
        const float v = heads_sum(d, sub);
        const bool in = key < k_hi && mask_allowed(mq, TokMeta{x.meta[u].x, x.meta[u].y, x.meta[u].z, x.meta[u].w});
        sc[u] = in ? v : -INFINITY;
      }
      float top = sc[0];
#pragma unroll
      for (int u = 1; u < U; ++u) top = fmaxf(top, sc[u]);
      if (__any_sync(0xffffffffu, top > mx)) {
        const float mn = fmaxf(mx, top);
        const float f = mx == -INFINITY ? 0.f : fast_exp2(mx - mn);
        l *= f;
        mx = mn;
#pragma unroll
        for (int h = 0; h < HG; ++h) {
          const float fh = of_head(f, h, lane);
          const uint64_t f2 = pack_f32x2(fh, fh);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[h][i] = mul_f32x2(acc[h][i], f2);
        }
      }
      const float mu = mx == -INFINITY ? 0.f : mx;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        sc[u] = fast_exp2(sc[u] - mu);
        l += sc[u];
        const uint32_t w[4] = {x.v[u].x, x.v[u].y, x.v[u].z, x.v[u].w};
#pragma unroll
        for (int h = 0; h < HG; ++h) {
          const float p = of_head(sc[u], h, lane);
          const uint64_t p2 = pack_f32x2(p, p);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[h][i] = fma_f32x2(p2, bf16x2_to_f32x2(w[i]), acc[h][i]);
        }
      }
    }
    // the two key groups of a warp, then the warps
    {
      const float mo = __shfl_xor_sync(0xffffffffu, mx, 16), mw = fmaxf(mx, mo);
      const float f = mx == -INFINITY ? 0.f : fast_exp2(mx - mw);
      float lw = l * f;
      lw += __shfl_xor_sync(0xffffffffu, lw, 16);
      if (lane < 16 && (lane & 3) == 0) {
        s.am[warp][lane >> 2] = mw;
        s.al[warp][lane >> 2] = lw;
      }
      float* wacc = red + warp * HG * 128 + sub * 8;
#pragma unroll
      for (int h = 0; h < HG; ++h) {
        const float fh = of_head(f, h, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float x0, x1;
          unpack_f32x2(acc[h][i], x0, x1);
          x0 *= fh;
          x1 *= fh;
          x0 += __shfl_xor_sync(0xffffffffu, x0, 16);
          x1 += __shfl_xor_sync(0xffffffffu, x1, 16);
          if (lane < 16) *reinterpret_cast<float2*>(wacc + h * 128 + i * 2) = make_float2(x0, x1);
        }
      }
    }
    named_bar_sync(1, CT);
    uint2* part = a.part + ((long long)(m * NG + hgp) * a.split + sp) * PART;
    uint2* op = a.o + ((long long)m * a.Hq + h0) * 64;
    {
      const int i = threadIdx.x * 2, h = i >> 7;             // HG * 128 results, two per thread
      static_assert(HG * 128 == CT * 2, "two results per thread");
      float mc = s.am[0][h];
#pragma unroll
      for (int w = 1; w < CW; ++w) mc = fmaxf(mc, s.am[w][h]);
      float2 o = make_float2(0.f, 0.f);
      float lc = 0.f;
#pragma unroll
      for (int w = 0; w < CW; ++w) {
        const float f = s.am[w][h] == -INFINITY ? 0.f : fast_exp2(s.am[w][h] - mc);
        const float2 r = *reinterpret_cast<const float2*>(red + w * HG * 128 + i);
        o.x += f * r.x;
        o.y += f * r.y;
        lc += f * s.al[w][h];
      }
      if (a.split == 1) {
        const float inv = lc > 0.f ? 1.f / lc : 0.f;         // a row without keys gives zeros
        st_word(op + i / 2, pack_bf16x2(o.x * inv, o.y * inv), out);
      } else {
        st_word(part + i, __float_as_uint(o.x), mid);
        st_word(part + i + 1, __float_as_uint(o.y), mid);
        if ((i & 127) == 0) {
          st_word(part + HG * 128 + h, __float_as_uint(mc), mid);
          st_word(part + HG * 128 + HG + h, __float_as_uint(lc), mid);
        }
      }
    }
    // ``red`` is the memory of x: a warp goes on to the output product's x, which may be there already, once every warp has its sums.
    // The wait lies beside that for the other parts.
    named_bar_sync(1, CT);
    if (a.split > 1) {
      // this CTA's share of the results, from all parts
      const uint2* p0 = a.part + (long long)(m * NG + hgp) * a.split * PART;
      const int p_lo = HG * 64 * sp / a.split, p_hi = HG * 64 * (sp + 1) / a.split;
      const int lanes = (p_hi - p_lo + 31) / 32 * 32;        // whole warps
      if ((int)threadIdx.x < lanes) {
        const int i = min(p_lo + (int)threadIdx.x, p_hi - 1) * 2, h = i >> 7;
        float mc = -INFINITY, lc = 0.f;
        float2 o = make_float2(0.f, 0.f);
        constexpr int PB = 4;                                // parts on their way
        for (int r0 = 0; r0 < a.split; r0 += PB) {           // running maximum: one pass over the parts, in order
          uint4 v[PB];
          uint2 wm[PB], wl[PB];
          poll(a, s, [&]() {
            bool ok = true;
#pragma unroll
            for (int b = 0; b < PB; ++b) {
              const uint2* pr = p0 + min(r0 + b, a.split - 1) * PART;
              v[b] = ld_words(pr + i);
              wm[b] = ld_word(pr + HG * 128 + h);
              wl[b] = ld_word(pr + HG * 128 + HG + h);
            }
#pragma unroll
            for (int b = 0; b < PB; ++b) ok &= v[b].y == mid && v[b].w == mid && wm[b].y == mid && wl[b].y == mid;
            return ok;
          });
#pragma unroll
          for (int b = 0; b < PB; ++b) {
            if (r0 + b >= a.split) break;
            const float mr = __uint_as_float(wm[b].x), mn = fmaxf(mc, mr);
            const float f0 = mc == -INFINITY ? 0.f : fast_exp2(mc - mn), f1 = mr == -INFINITY ? 0.f : fast_exp2(mr - mn);
            o.x = o.x * f0 + f1 * __uint_as_float(v[b].x);
            o.y = o.y * f0 + f1 * __uint_as_float(v[b].z);
            lc = lc * f0 + f1 * __uint_as_float(wl[b].x);
            mc = mn;
          }
        }
        const float inv = lc > 0.f ? 1.f / lc : 0.f;
        if (p_lo + (int)threadIdx.x < p_hi) st_word(op + i / 2, pack_bf16x2(o.x * inv, o.y * inv), out);
      }
    }
  }
}

template <int M>
__global__ void __launch_bounds__(THREADS, 1) decode_stack_kernel(const __grid_constant__ Args a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint8_t* xbuf = ring + a.stages * STAGE;
  float* own = reinterpret_cast<float*>(xbuf + a.x_size);                    // [2][M][OWN] x and x1
  float2* rope = reinterpret_cast<float2*>(own + 2 * OWN * a.M);
  Smem& s = *reinterpret_cast<Smem*>(rope + a.M * 64);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x;
  if (*(volatile unsigned int*)(a.count + G) != 0) {         // a launch before gave up: phase numbers may differ
    if (threadIdx.x == 0) report_status(a.status, kWaitTimeout, 7);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < a.stages; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], CW);
    }
    s.abort = 0;
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < a.M * 64; i += THREADS) {
    const int m = i >> 6, j = i & 63;
    const float ang = j < 32 ? (float)a.pos[m] * a.inv_t[j] : (float)a.pos[(j < 48 ? 1 : 2) * a.M + m] * a.inv_hw[(j - 32) & 15];
    float sn, cs;
    sincosf(ang, &sn, &cs);
    rope[i] = make_float2(cs, sn);
  }
  const Product rows = product(a, 0, DOWN);
  for (int i = threadIdx.x; i < a.M * (rows.hi - rows.lo); i += THREADS) {
    const int m = i / (rows.hi - rows.lo), r = i % (rows.hi - rows.lo);
    own[m * OWN + r] = __bfloat162float(a.x_in[(long long)m * a.H + rows.lo + r]);
  }
  const uint32_t launch = a.count[blockIdx.x] + 1;           // the same in all CTAs
  __syncthreads();
  if (warp == CW) {
    produce(a, ring, s, lane);
    return;
  }
  if (threadIdx.x == 0) a.count[blockIdx.x] = launch;
  uint32_t st = 0, par = 0;                                  // ring position of the consumers
  uint32_t now = launch * (MAX_LAYERS * 8);                  // number of the current phase
  const bool attends = (int)blockIdx.x < a.M * (a.Hq / HG) * a.split;
  Unit unit{};
  if (attends) unit = attention_unit(a, blockIdx.x);
  float* own1 = own + OWN * a.M;
  for (int l = 0; l < a.layers; ++l, now += 8) {
    // phases of a layer: 0 qkv, 1 parts of attention, 2 attention, 3 x1, 4 act, 5 x
    const Layer& L = a.layer[l];
    for (int ph = QKV; ph <= DOWN; ++ph) {
      const Product p = product(a, l, ph);
      if (ph == UP) {
        multiply<M, true>(a, ring, xbuf, s, p, st, par, a.x1, nullptr, now + 3, L.ffn_norm, nullptr, nullptr, a.act, nullptr, a.F, now + 4);
      } else {
        const bool qkv = ph == QKV, o = ph == OUT;
        multiply<M, false>(a, ring, xbuf, s, p, st, par, qkv ? a.x : o ? a.o : a.act, qkv && l == 0 ? a.x_in : nullptr,
                        qkv ? now - 8 + 5 : o ? now + 2 : now + 4, qkv ? L.attn_norm : nullptr, qkv ? nullptr : o ? own : own1,
                        qkv ? nullptr : o ? own1 : own, qkv ? a.qkv : o ? a.x1 : a.x, ph == DOWN && l + 1 == a.layers ? a.x_out : nullptr,
                        qkv ? (a.Hq + 2 * a.Hkv) * 128 : a.H, qkv ? now : o ? now + 3 : now + 5);
        if (qkv && attends) attend(a, s, reinterpret_cast<float*>(xbuf), rope, L, unit, now, now + 2, now + 1);
      }
    }
    // a time-out anywhere: all warps leave together (until then every wait fails soon)
    named_bar_sync(1, CT);
    if (threadIdx.x == 0) {
      s.stop = s.abort;
      if (s.stop) atomicExch(a.count + G, 1u);
    }
    named_bar_sync(1, CT);
    if (s.stop) break;
  }
}

}  // namespace dstack
}  // namespace snu1

using namespace snu1;

// Scratch of one engine, in words of 8 bytes.
static long long decode_stack_words(int rows, int H, int F, int Hq, int Hkv) {
  using namespace dstack;
  return (long long)rows * (H + (Hq + 2 * Hkv) * 64 + Hq * 64 + F / 2) + (long long)(rows * (Hq / HG) + num_sms()) * PART;
}

// Whether the kernel is built for these sizes: the words of scratch it needs, or 0.
SNU1_API long long snu1_decode_stack_takes(int rows, int H, int F, int Hq, int Hkv) {
  using namespace dstack;
  if (rows < 1 || rows > MAXM || H < KC || H % KC || F < KC || F % KC || Hq < 1 || Hkv < 1 || Hq % Hkv || (Hq / Hkv) % HG || Hq * 128 % KC)
    return 0;
  const int K = H > F ? (H > Hq * 128 ? H : Hq * 128) : (F > Hq * 128 ? F : Hq * 128);
  // one pass over x with all sums in registers, a normalised x in one batch of words
  const int per = ((F + num_sms() - 1) / num_sms() + 1) & ~1, qper = (((Hq + 2 * Hkv) * 128 + num_sms() - 1) / num_sms() + 1) & ~1;
  if (stages_for(rows, K) < MIN_STAGES || (H + num_sms() - 1) / num_sms() + 1 > OWN || per > MAXU * (UR / 2) || qper > MAXU * UR ||
      H / KC > (rows == 1 ? 6 : 4))
    return 0;
  return decode_stack_words(rows, H, F, Hq, Hkv);
}

// Table entry of one layer: wqkv, wo, w13, w2, attn_norm, qk_norm, ffn_norm, k cache, v cache (device addresses).  words: scratch
// of at least snu1_decode_stack_takes() words, count [SMs + 1]; both zero before the first launch and then left alone.
SNU1_API int snu1_decode_stack(const long long* table, int layers, int rows, int H, int F, int Hq, int Hkv, int Sk,
                               long long cache_rows, const void* x_in, void* x_out, void* words, long long n_words, void* count,
                               const void* meta_q, const void* meta_k, const int* first, const long long* last, const int* pos,
                               const float* inv_t, const float* inv_hw, int max_keys, float eps, float scale, void* stream) {
  using namespace dstack;
  const long long need = snu1_decode_stack_takes(rows, H, F, Hq, Hkv);
  if (layers < 1 || Sk < 1 || need == 0 || n_words < need) {
    set_last_error("decode_stack: rows=%d H=%d F=%d heads %d / %d, %lld words of scratch (%lld needed)", rows, H, F, Hq, Hkv, n_words,
                   need);
    return kHostBadArg;
  }
  uintptr_t bits = 0;
  for (const void* p : {x_in, (const void*)x_out, (const void*)words, meta_q, meta_k}) bits |= reinterpret_cast<uintptr_t>(p);
  for (int i = 0; i < layers * 9; ++i) bits |= (uintptr_t)table[i];
  if (bits & 15) {
    set_last_error("decode_stack: operands must be 16-byte aligned");
    return kHostBadArg;
  }
  void (*const kernels[MAXM])(const Args) = {decode_stack_kernel<1>, decode_stack_kernel<2>};
  void (*const kernel)(const Args) = kernels[rows - 1];
  int dev = 0;
  SNU1_CUDA_CHECK(cudaGetDevice(&dev));
  static std::once_flag once[64];
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&]() {
    for (auto k : kernels)
      if (err == cudaSuccess) err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  });
  SNU1_CUDA_CHECK(err);
  const int G = num_sms(), NG = Hq / HG;
  Args a;
  memset(&a, 0, sizeof(a));
  a.M = rows;
  a.H = H;
  a.F = F;
  a.Hq = Hq;
  a.Hkv = Hkv;
  a.Sk = Sk;
  a.cache_rows = cache_rows;
  const int K = H > F ? (H > Hq * 128 ? H : Hq * 128) : (F > Hq * 128 ? F : Hq * 128);
  a.stages = stages_for(rows, K);
  a.x_size = x_bytes(rows, K);
  // one unit per CTA, at least 64 keys each
  int split = G / (rows * NG);
  split = split < (max_keys + 63) / 64 ? split : (max_keys + 63) / 64;
  a.split = split < 1 ? 1 : split > MAX_SPLIT ? MAX_SPLIT : split;
  a.x_out = (__nv_bfloat16*)x_out;
  a.x = (uint2*)words;
  a.x1 = a.x + (long long)rows * H / 2;
  a.qkv = a.x1 + (long long)rows * H / 2;
  a.o = a.qkv + (long long)rows * (Hq + 2 * Hkv) * 64;
  a.act = a.o + (long long)rows * Hq * 64;
  a.part = a.act + (long long)rows * F / 2;
  a.count = (unsigned int*)count;
  a.meta_q = (const TokMeta*)meta_q;
  a.meta_k = (const TokMeta*)meta_k;
  a.first = first;
  a.last = last;
  a.pos = pos;
  a.inv_t = inv_t;
  a.inv_hw = inv_hw;
  a.eps = eps;
  a.inv_h = 1.f / H;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.status = device_status_word();
  for (int l0 = 0; l0 < layers; l0 += MAX_LAYERS) {
    a.layers = layers - l0 < MAX_LAYERS ? layers - l0 : MAX_LAYERS;
    static_assert(sizeof(Layer) == 9 * sizeof(long long), "one table entry per layer");
    memcpy(a.layer, table + (long long)l0 * 9, a.layers * sizeof(Layer));
    a.x_in = (const __nv_bfloat16*)(l0 == 0 ? x_in : x_out);
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(G, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = (cudaStream_t)stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SNU1_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, a));
  }
  return kHostOk;
}
