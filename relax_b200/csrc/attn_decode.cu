// Single-query attention of a decode step over the fp16 KV cache, as ONE launch: softmax(q . K^T / sqrt(128)) . V per
// (batch, head), optionally with the rotary embedding of q and k and the append of k and v in front (ROPE).
//
// The reference has no attention op; the semantics are the composition of its elementwise ops, statistics in fp32,
// one fp16 rounding of the rotated q and k and one of the result, which is what the oracle's restatement does too.
//
// Work: a cluster of 1, 2, 4 or 8 CTAs of four, five or eight warps per (head, batch).  The cache entries older than the new token are cut into units of 16
// tokens that are dealt out over all warps of the cluster.  Lane l of a warp holds dims 8 (l % 16).. + 7 of token
// 2 j + l / 16 of a unit, so that a load is 16 bytes a lane, a score takes four shuffles for two tokens, and the two halves of
// a warp keep their own online softmax until the end.  The keys of the next unit are requested as soon as this one's scores are
// formed, its values as soon as this one's are added up.  The new token is one more term, taken by the warp with the fewest
// units: with ROPE from the qkv row (it is never read back from the cache), else from the cache.
//
// The partial (max, sum, acc[128]) of a CTA goes to the CTAs of the cluster through their shared memory, owner o getting dims
// [o * 128 / c, (o + 1) * 128 / c); one cluster barrier, then every owner merges its dims in rank order.  No scratch in global
// memory, no counters, no second launch.  (Clusters of 16 CTAs were slower: one starts only where 16 places in a GPC are free at
// once.)
//
// What bounds it: HBM from about 400 pairs on (64 x 32 heads at 1002: 150 us, reading 7.0 TB/s; 16 x 32 at 2012 76 us, 6.9; a copy, half
// of it writes, moves 6.45), below that latency.  Against three launches (rotary + append, 128-token chunks, merge) a layer of a decode step
// took, us, before / after: hidden 4096, 1 row at 2012 53.4 / 51.6, 2 at 1501 61.7 / 54.4, 8 at 151 71.5 / 65.7, 16 at 2012
// 144.7 / 133.4, 64 at 1002 232.6 / 222; hidden 2048, 5 rows at 334 40.5 / 37.6; hidden 1024, 64 at 61 39.9 / 33.2.
#include "internal.h"
#include "sm100_ptx.cuh"

namespace b200 {

namespace {

constexpr int kUnit = 16;                // tokens a warp takes at a time
constexpr int kTok = kUnit / 2;          // per half of a warp
constexpr int kMaxCluster = 8;
constexpr int kCarveoutPercent = 30;     // of the SM's memory as shared memory

struct AttnParams {
  const __half* q;                       // [B, nh, 128] rotated queries, or (ROPE) qkv rows [q heads | k heads | v heads]
  const float* cos_t;                    // ROPE: fp32 [max_pos, 64]
  const float* sin_t;
  const int* pos;
  __half* k_cache;                       // [B, max_ctx, nh, 128]
  __half* v_cache;
  __half* out;                           // [B, nh * 128]
  int nh, max_ctx;
  float scale_log2e;
  int early_loads;                       // B200_ATTN_EARLY_KV_LOADS
  int early_release;                     // the next launch may begin in the first instruction
};

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// Eight consecutive fp16.  A16: the pointers are 16-byte aligned; else 8 bytes are what the loads may assume.
template <bool A16>
__device__ __forceinline__ uint4 load8(const __half* p) {
  if (A16) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
  }
  const uint2 a = reinterpret_cast<const uint2*>(p)[0], b = reinterpret_cast<const uint2*>(p)[1];
  return make_uint4(a.x, a.y, b.x, b.y);
}
template <bool A16>
__device__ __forceinline__ void store8(__half* p, const uint4& v) {
  if (A16) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    reinterpret_cast<uint2*>(p)[0] = make_uint2(v.x, v.y);
    reinterpret_cast<uint2*>(p)[1] = make_uint2(v.z, v.w);
  }
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __half22float2(h[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
__device__ __forceinline__ float dot8(const float (&q)[8], const uint4& k) {
  float f[8];
  unpack8(k, f);
  float s = q[0] * f[0];
#pragma unroll
  for (int j = 1; j < 8; ++j) s = fmaf(q[j], f[j], s);
  return s;
}

// W warps.  At least 128 registers a thread, 16 (W = 5: 15) warps an SM: each has 8 KB of keys and values in flight.
template <int W, bool ROPE, bool A16>
__global__ void __launch_bounds__(W * 32, 16 / W)
attn_decode_kernel(const AttnParams p) {
  if (p.early_release) ptx::pdl_launch_dependents();
  const int c = gridDim.x, rank = blockIdx.x;            // (the cluster spans the grid's x)
  const int h = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = lane >> 4, d0 = (lane & 15) * 8;
  if (c > 1) ptx::cluster_arrive_relaxed();                   // (every CTA of the cluster runs before anything is stored in it)

  // early_loads: the caller promises that the position and the cache entries older than the new token were complete before the
  // launch in front of this one began.  Without the promise nothing is read before the wait.
  if (!p.early_loads) {
    ptx::pdl_wait();
    if (!p.early_release) ptx::pdl_launch_dependents();
  }
  const int pos = min(*p.pos, p.max_ctx - 1);            // tokens older than the new one
  const int units = (pos + kUnit - 1) / kUnit;
  const int nw = c * W, gw = warp * c + rank;
  const int64_t stride = (int64_t)p.nh * 128;
  const __half* kb = p.k_cache + ((int64_t)b * p.max_ctx * p.nh + h) * 128 + d0;
  const __half* vb = p.v_cache + ((int64_t)b * p.max_ctx * p.nh + h) * 128 + d0;
  uint4 kv[kTok], vv[kTok];
  auto load_unit = [&](uint4 (&dst)[kTok], const __half* base, int u) {
#pragma unroll
    for (int j = 0; j < kTok; ++j) {
      const int t = min(u * kUnit + 2 * j + half, pos - 1);     // clamped: a token past the end is loaded but not used
      dst[j] = load8<A16>(base + t * stride);
    }
  };
  if (gw < units) {
    load_unit(kv, kb, gw);
    load_unit(vv, vb, gw);
  }
  float cs[8], sn[8];
  if (ROPE && pos >= 0) {
    const float4* cp = reinterpret_cast<const float4*>(p.cos_t + (int64_t)pos * 64 + (d0 & 63));
    const float4* sp = reinterpret_cast<const float4*>(p.sin_t + (int64_t)pos * 64 + (d0 & 63));
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    cs[0] = c0.x; cs[1] = c0.y; cs[2] = c0.z; cs[3] = c0.w; cs[4] = c1.x; cs[5] = c1.y; cs[6] = c1.z; cs[7] = c1.w;
    sn[0] = s0.x; sn[1] = s0.y; sn[2] = s0.z; sn[3] = s0.w; sn[4] = s1.x; sn[5] = s1.y; sn[6] = s1.z; sn[7] = s1.w;
  }
  if (p.early_loads) {
    ptx::pdl_wait();
    if (!p.early_release) ptx::pdl_launch_dependents();
  }

  // dims i and i + 64 are a pair: this lane's partner is lane ^ 8.  First half a * cos - b * sin, second b * cos + a * sin, rounded
  // to fp16 as a q or k tensor would be.
  const float sign = d0 < 64 ? -1.f : 1.f;
  auto rotate = [&](const uint4& raw) {
    float f[8];
    unpack8(raw, f);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float other = __shfl_xor_sync(0xffffffffu, f[j], 8);
      r[j] = f[j] * cs[j] + sign * other * sn[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) oh[j] = __floats2half2_rn(r[2 * j], r[2 * j + 1]);
    return o;
  };
  const __half* row = p.q + (int64_t)b * 3 * p.nh * 128;         // (ROPE)
  uint4 qraw = load8<A16>(ROPE ? row + h * 128 + d0 : p.q + ((int64_t)b * p.nh + h) * 128 + d0);
  const bool newest = gw == nw - 1 && pos >= 0;
  uint4 nk, nv;
  if (newest) {
    if (ROPE) {
      nk = load8<A16>(row + (p.nh + h) * 128 + d0);
      nv = load8<A16>(row + (2 * p.nh + h) * 128 + d0);
    } else {
      nk = load8<A16>(kb + pos * stride);
      nv = load8<A16>(vb + pos * stride);
    }
  }
  if (ROPE) qraw = rotate(qraw);
  float qf[8];
  unpack8(qraw, qf);
#pragma unroll
  for (int j = 0; j < 8; ++j) qf[j] *= p.scale_log2e;

  float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (newest) {
    if (ROPE) {
      nk = rotate(nk);
      if (half == 0) {
        store8<A16>(p.k_cache + (((int64_t)b * p.max_ctx + pos) * p.nh + h) * 128 + d0, nk);
        store8<A16>(p.v_cache + (((int64_t)b * p.max_ctx + pos) * p.nh + h) * 128 + d0, nv);
      }
    }
    float s = dot8(qf, nk);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (half == 0) {
      m = s;
      l = 1.f;
      unpack8(nv, acc);
    }
  }

  for (int u = gw; u < units; u += nw) {
    float s[kTok];
#pragma unroll
    for (int j = 0; j < kTok; ++j) s[j] = dot8(qf, kv[j]);
    if (u + nw < units) load_unit(kv, kb, u + nw);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < kTok; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
    float mn = m;
#pragma unroll
    for (int j = 0; j < kTok; ++j) {
      if (u * kUnit + 2 * j + half >= pos) s[j] = -INFINITY;      // log2-domain scores; masked tokens get weight 0
      mn = fmaxf(mn, s[j]);
    }
    const float mr = mn == -INFINITY ? 0.f : mn;                  // (half of a warp may have seen masked tokens only)
    const float corr = exp2f(m - mr);
    l *= corr;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= corr;
#pragma unroll
    for (int j = 0; j < kTok; ++j) {
      const float pj = exp2f(s[j] - mr);
      float f[8];
      unpack8(vv[j], f);
      l += pj;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(pj, f[i], acc[i]);
    }
    if (u + nw < units) load_unit(vv, vb, u + nw);
    m = mn;
  }

  // ---- the two halves of the warp, the warps of the CTA, the CTAs of the cluster ------------------------------------
  __shared__ float sm_m[W], sm_l[W];
  __shared__ __align__(16) float sm_acc[W][128];
  __shared__ float in_m[kMaxCluster], in_l[kMaxCluster], in_acc[kMaxCluster][128];     // from every rank: this owner's dims
  {
    const float mo = __shfl_xor_sync(0xffffffffu, m, 16);
    const float M = fmaxf(m, mo);
    const float mr = M == -INFINITY ? 0.f : M;
    const float f = exp2f(m - mr);                                 // (-inf: 0)
    l *= f;
    l += __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      acc[i] *= f;
      acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
    }
    if (lane == 0) { sm_m[warp] = M; sm_l[warp] = l; }
    // each half stores four of a lane's eight dims
    *reinterpret_cast<float4*>(&sm_acc[warp][d0 + 4 * half]) =
        half ? make_float4(acc[4], acc[5], acc[6], acc[7]) : make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
  __syncthreads();
  const int d = threadIdx.x;
  float M = -INFINITY, L = 0.f, A = 0.f;
  if (d < 128) {
#pragma unroll
    for (int w = 0; w < W; ++w) M = fmaxf(M, sm_m[w]);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float f = sm_m[w] == -INFINITY ? 0.f : exp2f(sm_m[w] - M);
      L += sm_l[w] * f;
      A += sm_acc[w][d] * f;
    }
  }
  __half* out = p.out + ((int64_t)b * p.nh + h) * 128;
  if (c == 1) {
    if (d < 128) out[d] = __float2half_rn(A / L);
    return;
  }
  const int per = 128 / c;                                         // dims of an owner
  ptx::cluster_wait();                                             // (the one at the start)
  if (d < 128) {
    const int owner = d / per;
    st_cluster_f32(ptx::map_to_rank(ptx::smem_u32(&in_acc[rank][d - owner * per]), owner), A);
    if (d < c) {
      st_cluster_f32(ptx::map_to_rank(ptx::smem_u32(&in_m[rank]), d), M);
      st_cluster_f32(ptx::map_to_rank(ptx::smem_u32(&in_l[rank]), d), L);
    }
  }
  ptx::cluster_arrive();
  ptx::cluster_wait();
  if (d < per) {
    M = -INFINITY;
    for (int r = 0; r < c; ++r) M = fmaxf(M, in_m[r]);
    L = A = 0.f;
    for (int r = 0; r < c; ++r) {
      const float f = in_m[r] == -INFINITY ? 0.f : exp2f(in_m[r] - M);
      L += in_l[r] * f;
      A += in_acc[r][d] * f;
    }
    out[rank * per + d] = __float2half_rn(A / L);
  }
}

bool aligned(const void* p, unsigned n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

int launch_attn(const char* what, bool rope, AttnParams p, int64_t B, cudaStream_t stream) {
  p.scale_log2e = 1.4426950408889634f / sqrtf(128.f);
  const bool a16 = aligned(p.q, 16) && aligned(p.k_cache, 16) && aligned(p.v_cache, 16);
  // Warps per (head, batch): as many as the GPU holds at once, and no more than there are units.  64 only where half of the places
  // are enough (32 pairs at context 2012: 32 warps 51.6, 64 warps 52.4 us a layer of a step).  Above 592 pairs four warps each are
  // more than one wave; up to two waves of them leave too much of the second one empty (800 pairs at 1201: 4 warps 125, 8 warps
  // 115 us), and so does a little more than two over a long context (1280 pairs at 1501 156.3 / 145.2; but at 301, inside a step, a layer took 114
  // us with four and 117 with eight).
  // Five warps are three CTAs an SM: from 297 to 444 pairs, where eight warps each are more than one wave and four leave places empty, one
  // CTA of five, and from 593 to 666, over a cache of more than 640 tokens, two, which fill their last wave.  A layer of a step (hidden 4096,
  // inter 2816), us, before / now: 320 pairs at 301 68.7 / 67.7, at 1001 89.3 / 84.8, at 2011 117.8 / 109.2; 416 70.7 / 70.0, 93.1 / 90.8, 124.1 / 120.5;
  // 640 at 301 72.2 / 72.8, at 1001 108.3 / 105.3, at 2011 160.1 / 149.3; behind the lines, at 2011, 448 126.9 / 150.3, 672 163.4 / 166.0.
  const int64_t pairs = B * p.nh;
  const int64_t slots = (int64_t)sm_count() * 16;
  const int64_t last = pairs * 4 % slots;                  // of the last wave of four warps a pair
  const bool second = pairs * 4 > slots && pairs * 2 < slots && p.max_ctx > 4 * kUnit;
  const bool later = pairs * 2 >= slots && last > 0 && 2 * last < slots && p.max_ctx > 80 * kUnit;
  int t = second || later ? 8 : 4;
  while (pairs * 2 * t <= (t == 32 ? slots / 2 : slots) && t < 64 && t * kUnit < p.max_ctx) t *= 2;
  const int64_t fives = (int64_t)sm_count() * 3;           // CTAs of five warps in a wave
  if (pairs * 8 > slots && pairs <= fives && p.max_ctx > 4 * kUnit) t = 5;
  if (pairs * 4 > slots && pairs * 2 <= 3 * fives && p.max_ctx > 40 * kUnit) t = 10;
  const int w = t % 5 == 0 ? 5 : t < 8 ? 4 : 8, c = t / w;
  auto pick = [&](auto k4, auto k5, auto k8) { return w == 8 ? k8 : w == 5 ? k5 : k4; };
  auto kern = rope ? (a16 ? pick(attn_decode_kernel<4, true, true>, attn_decode_kernel<5, true, true>, attn_decode_kernel<8, true, true>)
                          : pick(attn_decode_kernel<4, true, false>, attn_decode_kernel<5, true, false>, attn_decode_kernel<8, true, false>))
                   : (a16 ? pick(attn_decode_kernel<4, false, true>, attn_decode_kernel<5, false, true>, attn_decode_kernel<8, false, true>)
                          : pick(attn_decode_kernel<4, false, false>, attn_decode_kernel<5, false, false>, attn_decode_kernel<8, false, false>));
  // The keys and values in flight are lines of the L1 cache, so most of the SM's memory has to be cache: behind a matmul that
  // had it as shared memory, and without this, 16 warps were held to 25 KB in flight.  A layer of a step, us, before / after: 16 rows
  // at 2012 148 / 133, 5 rows at 2001 (hidden 5120) 141 / 117, 64 at 1002 (hidden 4096) 239 / 222.
  static SmemLimit carveout[12];
  const int variant = (w == 8 ? 8 : w == 5 ? 4 : 0) + rope * 2 + a16;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    carveout[variant].raise(dev, 1, [&](size_t) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveoutPercent);
      return e == cudaSuccess ? 0 : 1;
    });
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "%s: shared-memory carve-out: %s", what, cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c, (unsigned)p.nh, (unsigned)B);
  cfg.blockDim = dim3((unsigned)w * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = options().gemv_pdl ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, kern, p);
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "%s launch: %s", what, cudaGetErrorString(e));
  count_launch();
  return B200_OK;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

// The scratch arguments below are of an earlier form of the kernel (partial results in global memory, arrival counters behind
// them).  Nothing is stored there any more; what was refused without one still is.
static int64_t chunks_of(int64_t max_ctx) { return (max_ctx + 127) / 128; }

int64_t b200_attn_decode_scratch_bytes(int64_t B, int64_t nh, int64_t max_ctx) {
  return B * nh * chunks_of(max_ctx) * 130 * (int64_t)sizeof(float);
}

int64_t b200_attn_decode_fused_scratch_bytes(int64_t B, int64_t nh, int64_t max_ctx) {
  return b200_attn_decode_scratch_bytes(B, nh, max_ctx) + B * nh * (int64_t)sizeof(int);
}

static int check_sizes(const char* who, int64_t B, int64_t nh, int64_t max_ctx) {
  if (B <= 0 || nh <= 0 || max_ctx <= 0) return fail(B200_EINVAL, "%s: bad sizes", who);
  if (B > 65535 || nh > 65535 || max_ctx > 0x3fffffffLL)
    return fail(B200_EINVAL, "%s: batch and heads are limited to 65535 (grid dimensions), max_ctx to 2^30", who);
  return B200_OK;
}

static int attn_plain(const char* who, const void* q, const void* k_cache, const void* v_cache, const void* pos, void* out, int64_t B,
                      int64_t nh, int64_t max_ctx, uint32_t flags, bool early_release, void* stream) {
  int rc = check_sizes(who, B, nh, max_ctx);
  if (rc) return rc;
  if (flags & ~(uint32_t)B200_ATTN_EARLY_KV_LOADS) return fail(B200_EINVAL, "%s: unknown flag bits %#x", who, flags);
  if (!q || !k_cache || !v_cache || !pos || !out) return fail(B200_EINVAL, "%s: null pointer", who);
  if ((rc = ensure_device())) return rc;
  AttnParams p = {};
  p.q = (const __half*)q; p.k_cache = (__half*)k_cache; p.v_cache = (__half*)v_cache; p.pos = (const int*)pos; p.out = (__half*)out;
  p.nh = (int)nh; p.max_ctx = (int)max_ctx;
  p.early_loads = (flags & B200_ATTN_EARLY_KV_LOADS) != 0;
  p.early_release = early_release;
  return launch_attn(who, false, p, B, static_cast<cudaStream_t>(stream));
}

static int attn_rope(const char* who, const void* qkv, const void* cos_t, const void* sin_t, const void* pos, void* k_cache,
                     void* v_cache, void* out, int64_t B, int64_t nh, int64_t max_ctx, bool early_loads, bool early_release, void* stream) {
  int rc = check_sizes(who, B, nh, max_ctx);
  if (rc) return rc;
  if (!qkv || !cos_t || !sin_t || !pos || !k_cache || !v_cache || !out) return fail(B200_EINVAL, "%s: null pointer", who);
  if ((rc = ensure_device())) return rc;
  AttnParams p = {};
  p.q = (const __half*)qkv; p.cos_t = (const float*)cos_t; p.sin_t = (const float*)sin_t; p.pos = (const int*)pos;
  p.k_cache = (__half*)k_cache; p.v_cache = (__half*)v_cache; p.out = (__half*)out;
  p.nh = (int)nh; p.max_ctx = (int)max_ctx;
  p.early_loads = early_loads;
  p.early_release = early_release;
  return launch_attn(who, true, p, B, static_cast<cudaStream_t>(stream));
}

int b200_attn_decode(const void* q, const void* k_cache, const void* v_cache, const void* pos, void* out, void* scratch,
                     int64_t B, int64_t nh, int64_t max_ctx, uint32_t flags, void* stream) {
  if (!scratch) return fail(B200_EINVAL, "attn_decode: null pointer");
  return attn_plain("attn_decode", q, k_cache, v_cache, pos, out, B, nh, max_ctx, flags, false, stream);
}

int b200_attn_decode_early_release(const void* q, const void* k_cache, const void* v_cache, const void* pos, void* out,
                                   void* scratch, int64_t B, int64_t nh, int64_t max_ctx, uint32_t flags, void* stream) {
  if (!scratch) return fail(B200_EINVAL, "attn_decode_early_release: null pointer");
  return attn_plain("attn_decode_early_release", q, k_cache, v_cache, pos, out, B, nh, max_ctx, flags, true, stream);
}

int b200_attn_decode_fused(const void* qkv, const void* cos_t, const void* sin_t, const void* pos, void* k_cache, void* v_cache,
                           void* out, void* scratch, int64_t B, int64_t nh, int64_t max_ctx, void* stream) {
  if (!scratch) return fail(B200_EINVAL, "attn_decode_fused: null pointer");
  return attn_rope("attn_decode_fused", qkv, cos_t, sin_t, pos, k_cache, v_cache, out, B, nh, max_ctx, false, false, stream);
}

int b200_attn_decode_rope(const void* qkv, const void* cos_t, const void* sin_t, const void* pos, void* k_cache, void* v_cache,
                          void* out, void* scratch, int64_t B, int64_t nh, int64_t max_ctx, void* stream) {
  if (!scratch) return fail(B200_EINVAL, "attn_decode_rope: null pointer");
  return attn_rope("attn_decode_rope", qkv, cos_t, sin_t, pos, k_cache, v_cache, out, B, nh, max_ctx, false, false, stream);
}

int b200_attn_decode_step(const void* qkv, const void* cos_t, const void* sin_t, const void* pos, void* k_cache, void* v_cache,
                          void* out, int64_t B, int64_t nh, int64_t max_ctx, uint32_t flags, void* stream) {
  const char* who = "attn_decode_step";
  if (flags & ~(uint32_t)(B200_ATTN_EARLY_KV_LOADS | B200_ATTN_EARLY_RELEASE)) return fail(B200_EINVAL, "%s: unknown flag bits %#x", who, flags);
  if (!aligned(qkv, 8) || !aligned(k_cache, 8) || !aligned(v_cache, 8) || !aligned(cos_t, 16) || !aligned(sin_t, 16) || !aligned(out, 2))
    return fail(B200_EINVAL, "%s: qkv and the caches must be 8-byte aligned, the tables 16-byte", who);
  return attn_rope(who, qkv, cos_t, sin_t, pos, k_cache, v_cache, out, B, nh, max_ctx, (flags & B200_ATTN_EARLY_KV_LOADS) != 0,
                   (flags & B200_ATTN_EARLY_RELEASE) != 0, stream);
}

// Attention without caller-provided scratch.  The limit is that of the fixed array that once held its partial results.
constexpr int64_t kStaticAttnSlots = 8192;                       // e.g. 16 sequences x 32 heads x 2048 tokens

int b200_attn_decode_static(const void* q, const void* k_cache, const void* v_cache, const void* pos, void* out, int64_t B,
                            int64_t nh, int64_t max_ctx, uint32_t flags, void* stream) {
  int rc = check_sizes("attn_decode_static", B, nh, max_ctx);
  if (rc) return rc;
  if (!q || !k_cache || !v_cache || !pos || !out) return fail(B200_EINVAL, "attn_decode_static: null pointer");
  const int64_t nsplit = chunks_of(max_ctx);
  // (B, nh <= 65535 and nsplit <= 2^23: the product below cannot overflow 64 bits)
  if (B * nh * nsplit > kStaticAttnSlots)
    return fail(B200_EINVAL,
                "attn_decode_static: batch %lld x heads %lld x %lld chunks of 128 tokens = %lld partial results, the built-in "
                "scratch holds %lld; use b200_attn_decode with a caller-owned buffer",
                (long long)B, (long long)nh, (long long)nsplit, (long long)(B * nh * nsplit), (long long)kStaticAttnSlots);
  return attn_plain("attn_decode_static", q, k_cache, v_cache, pos, out, B, nh, max_ctx, flags, false, stream);
}

}  // extern "C"
