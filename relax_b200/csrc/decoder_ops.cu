// Glue kernels of one Llama-style decode step around the quantised matmuls: RMSNorm (with the
// residual add fused), rotary embedding + KV-cache append and SwiGLU (the attention: attn_decode.cu).
//
// The reference has no op for RMSNorm, RoPE or attention (its op list stops at mean / sqrt /
// divide / multiply / strided_slice / concat / softmax / silu, python/tvm/relax/transform/
// legalize_ops.py:378-381,506-514); the semantics here are the composition of those ops with
// statistics in fp32 and one fp16 rounding at each kernel's output, which is what the oracle's
// decoder restatement does too.
//
// All of them are latency bound and tiny next to the weight streams.
#include "internal.h"
#include "sm100_ptx.cuh"

namespace b200 {

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Where a kernel lets its successor start (griddepcontrol.launch_dependents).  The entry points' ordinary forms do so
// right after their own wait: everything up to the launch before them is then complete, which is what an attention
// with early loads of old cache entries and of the position relies on when one of them is directly in front.  The
// early-release forms (kEarly) do so in their first instruction, for a caller that knows that nothing is read
// early behind them but weights: a matmul's set-up and first weight loads then run beside them.
template <bool kEarly>
__device__ __forceinline__ void wait_and_release() {
  if (kEarly) ptx::pdl_launch_dependents();
  ptx::pdl_wait();
  if (!kEarly) ptx::pdl_launch_dependents();
}

// y[b,:] = fp16( f32(x) * rsqrt(mean(f32(x)^2) + eps) * f32(w) ); optionally x += delta first (the
// updated x is written back: it is the residual stream).  One CTA per row, H % 8 == 0.  A thread's share of the row,
// of delta and of w (up to kRmsWords words of 8 values: H <= 8192) is loaded in one go and stays in registers; a longer
// row makes the trip for w after the statistics, through a copy of x in shared memory.
constexpr int kRmsWords = 4;
template <bool kAdd, bool kEarly>
__global__ void __launch_bounds__(256)
rmsnorm_kernel(__half* __restrict__ x, const __half* __restrict__ delta, const __half* __restrict__ w,
               __half* __restrict__ y, int H, float eps) {
  wait_and_release<kEarly>();
  extern __shared__ float xs[];                 // H floats (H > 8192)
  __shared__ float red[8];
  const int b = blockIdx.x;
  __half* xr = x + (int64_t)b * H;
  const bool one_go = H <= kRmsWords * 256 * 8;
  float ss = 0.f;
  uint4 v[kRmsWords], wv[kRmsWords];
  // the residual stream is stored in fp16: round the sum once, then normalise what was stored
  auto add = [&](uint4& val, const uint4& dv) {
    __half2* h = reinterpret_cast<__half2*>(&val);
    const __half2* dh = reinterpret_cast<const __half2*>(&dv);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(h[j]), t = __half22float2(dh[j]);
      h[j] = __floats2half2_rn(f.x + t.x, f.y + t.y);
    }
  };
  auto squares = [&](const uint4& val) {
    const __half2* h = reinterpret_cast<const __half2*>(&val);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(h[j]);
      ss += f.x * f.x;
      ss += f.y * f.y;
    }
  };
  if (one_go) {
    uint4 dv[kRmsWords];
#pragma unroll
    for (int r = 0; r < kRmsWords; ++r) {
      const int i = (threadIdx.x + r * 256) * 8;
      v[r] = wv[r] = dv[r] = make_uint4(0, 0, 0, 0);
      if (i < H) {
        v[r] = *reinterpret_cast<const uint4*>(xr + i);
        if (kAdd) dv[r] = *reinterpret_cast<const uint4*>(delta + (int64_t)b * H + i);
        wv[r] = *reinterpret_cast<const uint4*>(w + i);
      }
    }
#pragma unroll
    for (int r = 0; r < kRmsWords; ++r) {
      const int i = (threadIdx.x + r * 256) * 8;
      if (i >= H) continue;
      if (kAdd) {
        add(v[r], dv[r]);
        *reinterpret_cast<uint4*>(xr + i) = v[r];
      }
      squares(v[r]);
    }
  } else {
    for (int i = threadIdx.x * 8; i < H; i += 256 * 8) {
      uint4 val = *reinterpret_cast<const uint4*>(xr + i);
      if (kAdd) {
        add(val, *reinterpret_cast<const uint4*>(delta + (int64_t)b * H + i));
        *reinterpret_cast<uint4*>(xr + i) = val;
      }
      squares(val);
      const __half2* h = reinterpret_cast<const __half2*>(&val);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h[j]);
        xs[i + 2 * j] = f.x;
        xs[i + 2 * j + 1] = f.y;
      }
    }
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = rsqrtf(tot / (float)H + eps);
  auto scaled = [&](const float (&f)[8], const uint4& wr) {
    const __half2* wh = reinterpret_cast<const __half2*>(&wr);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 wf = __half22float2(wh[j]);
      oh[j] = __floats2half2_rn(f[2 * j] * inv * wf.x, f[2 * j + 1] * inv * wf.y);
    }
    return o;
  };
  if (one_go) {
#pragma unroll
    for (int r = 0; r < kRmsWords; ++r) {
      const int i = (threadIdx.x + r * 256) * 8;
      if (i >= H) continue;
      const __half2* h = reinterpret_cast<const __half2*>(&v[r]);
      float f[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = __half22float2(h[j]);
        f[2 * j] = t.x;
        f[2 * j + 1] = t.y;
      }
      *reinterpret_cast<uint4*>(y + (int64_t)b * H + i) = scaled(f, wv[r]);
    }
  } else {
    for (int i = threadIdx.x * 8; i < H; i += 256 * 8) {
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = xs[i + j];
      *reinterpret_cast<uint4*>(y + (int64_t)b * H + i) = scaled(f, *reinterpret_cast<const uint4*>(w + i));
    }
  }
}

// Rotary embedding (rotate-half pairing i <-> i+64 inside a 128-wide head) of q and k, then k and v
// go to the cache at position pos[0].  qkv row layout: [q heads | k heads | v heads], nh heads each.
// cos/sin tables fp32 [max_pos, 64].  grid (nh, B), 64 threads.
__global__ void __launch_bounds__(64)
rope_kv_append_kernel(const __half* __restrict__ qkv, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                      const int* __restrict__ pos_ptr, __half* __restrict__ q_out, __half* __restrict__ k_cache,
                      __half* __restrict__ v_cache, int nh, int max_ctx) {
  ptx::pdl_wait();
  ptx::pdl_launch_dependents();
  const int h = blockIdx.x, b = blockIdx.y, i = threadIdx.x;
  const int pos = pos_ptr[0];
  const float c = cos_t[(int64_t)pos * 64 + i], s = sin_t[(int64_t)pos * 64 + i];
  const __half* row = qkv + (int64_t)b * 3 * nh * 128;
  const __half* q = row + h * 128;
  const __half* k = row + (nh + h) * 128;
  const __half* v = row + (2 * nh + h) * 128;
  const float q0 = __half2float(q[i]), q1 = __half2float(q[i + 64]);
  const float k0 = __half2float(k[i]), k1 = __half2float(k[i + 64]);
  __half* qo = q_out + ((int64_t)b * nh + h) * 128;
  qo[i] = __float2half_rn(q0 * c - q1 * s);
  qo[i + 64] = __float2half_rn(q1 * c + q0 * s);
  const int64_t slot = (((int64_t)b * max_ctx + pos) * nh + h) * 128;
  k_cache[slot + i] = __float2half_rn(k0 * c - k1 * s);
  k_cache[slot + i + 64] = __float2half_rn(k1 * c + k0 * s);
  v_cache[slot + i] = v[i];
  v_cache[slot + i + 64] = v[i + 64];
}

// out[b,i] = fp16( silu(f32(g)) * f32(u) ), gu row = [gate (I) | up (I)].  I % 8 == 0.
template <bool kEarly>
__global__ void __launch_bounds__(256)
silu_mul_kernel(const __half* __restrict__ gu, __half* __restrict__ out, int I, int64_t total8) {
  wait_and_release<kEarly>();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total8) return;
  const int per_row = I / 8;
  const int64_t b = idx / per_row;
  const int i = (int)(idx - b * per_row) * 8;
  uint4 gv = *reinterpret_cast<const uint4*>(gu + b * 2 * I + i);
  uint4 uv = *reinterpret_cast<const uint4*>(gu + b * 2 * I + I + i);
  const __half2* gh = reinterpret_cast<const __half2*>(&gv);
  const __half2* uh = reinterpret_cast<const __half2*>(&uv);
  uint4 o;
  __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 g = __half22float2(gh[j]), u = __half22float2(uh[j]);
    float a = g.x / (1.f + __expf(-g.x)) * u.x;
    float c = g.y / (1.f + __expf(-g.y)) * u.y;
    oh[j] = __floats2half2_rn(a, c);
  }
  *reinterpret_cast<uint4*>(out + b * I + i) = o;
}

// out[b,:] = table[ids[b],:] (fp16 rows of H, H % 8 == 0).  grid (B), 128 threads.  kStats: the row's sum of squares goes to
// stats[b][0] and zeros to the other H / 16 - 1 places of its partial sums.
template <bool kStats>
__global__ void __launch_bounds__(128)
embed_rows_kernel(const __half* __restrict__ table, const int* __restrict__ ids, __half* __restrict__ out, float* __restrict__ stats,
                  int H, int vocab) {
  ptx::pdl_wait();
  const int b = blockIdx.x;
  int id = ids[b];
  id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);          // clamp: never read outside the table
  const uint4* src = reinterpret_cast<const uint4*>(table + (int64_t)id * H);
  uint4* dst = reinterpret_cast<uint4*>(out + (int64_t)b * H);
  ptx::pdl_launch_dependents();
  float ss = 0.f;
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    const uint4 v = src[i];
    dst[i] = v;
    if (kStats) {
      const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h[j]);
        ss += f.x * f.x + f.y * f.y;
      }
    }
  }
  if (kStats) {
    __shared__ float red[4];
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    for (int i = threadIdx.x; i < H / 16; i += blockDim.x)
      stats[(int64_t)b * (H / 16) + i] = i == 0 ? (red[0] + red[1]) + (red[2] + red[3]) : 0.f;
  }
}

// *pos += delta (one thread): advances the decode position on the device so that a captured
// graph can be replayed token after token.
__global__ void advance_pos_kernel(int* pos, int delta) {
  ptx::pdl_wait();
  ptx::pdl_launch_dependents();
  if (threadIdx.x == 0 && blockIdx.x == 0) *pos += delta;
}

template <typename K, typename... A>
int launch(const char* what, K kern, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = options().gemv_pdl ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "%s launch: %s", what, cudaGetErrorString(e));
  count_launch();
  return B200_OK;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

static int rmsnorm_impl(const char* who, void* x, const void* delta, const void* w, void* y, int64_t B, int64_t H, float eps,
                        bool early, void* stream) {
  if (B < 0 || H <= 0 || H % 8 != 0 || H > 16384) return fail(B200_EINVAL, "%s: need 0 < H <= 16384, H %% 8 == 0", who);
  if (B == 0) return B200_OK;
  if (!x || !w || !y) return fail(B200_EINVAL, "%s: null pointer", who);
  int rc = ensure_device();
  if (rc) return rc;
  auto kern = delta ? (early ? rmsnorm_kernel<true, true> : rmsnorm_kernel<true, false>)
                    : (early ? rmsnorm_kernel<false, true> : rmsnorm_kernel<false, false>);
  return launch(delta ? "add_rmsnorm" : "rmsnorm", kern, dim3((unsigned)B), dim3(256),
                H > kRmsWords * 256 * 8 ? (size_t)H * 4 : 0, static_cast<cudaStream_t>(stream), (__half*)x, (const __half*)delta,
                (const __half*)w, (__half*)y, (int)H, eps);
}

int b200_rmsnorm(void* x, const void* delta, const void* w, void* y, int64_t B, int64_t H, float eps, void* stream) {
  return rmsnorm_impl("rmsnorm", x, delta, w, y, B, H, eps, false, stream);
}

int b200_rmsnorm_early_release(void* x, const void* delta, const void* w, void* y, int64_t B, int64_t H, float eps, void* stream) {
  return rmsnorm_impl("rmsnorm_early_release", x, delta, w, y, B, H, eps, true, stream);
}

int b200_rope_kv_append(const void* qkv, const void* cos_t, const void* sin_t, const void* pos, void* q_out,
                        void* k_cache, void* v_cache, int64_t B, int64_t nh, int64_t max_ctx, void* stream) {
  if (B <= 0 || nh <= 0 || max_ctx <= 0) return fail(B200_EINVAL, "rope_kv_append: bad sizes");
  if (!qkv || !cos_t || !sin_t || !pos || !q_out || !k_cache || !v_cache) return fail(B200_EINVAL, "rope_kv_append: null pointer");
  int rc = ensure_device();
  if (rc) return rc;
  return launch("rope_kv_append", rope_kv_append_kernel, dim3((unsigned)nh, (unsigned)B), dim3(64), 0,
                static_cast<cudaStream_t>(stream), (const __half*)qkv, (const float*)cos_t, (const float*)sin_t,
                (const int*)pos, (__half*)q_out, (__half*)k_cache, (__half*)v_cache, (int)nh, (int)max_ctx);
}

static int embed_rows_impl(const char* who, const void* table, const void* ids, void* out, void* stats, int64_t B, int64_t H,
                           int64_t vocab, void* stream) {
  if (B < 0 || H <= 0 || H % 8 != 0 || vocab <= 0) return fail(B200_EINVAL, "%s: need H %% 8 == 0, vocab > 0", who);
  if (B == 0) return B200_OK;
  if (!table || !ids || !out) return fail(B200_EINVAL, "%s: null pointer", who);
  int rc = ensure_device();
  if (rc) return rc;
  return launch("embed_rows", stats ? embed_rows_kernel<true> : embed_rows_kernel<false>, dim3((unsigned)B), dim3(128), 0,
                static_cast<cudaStream_t>(stream), (const __half*)table, (const int*)ids, (__half*)out, (float*)stats, (int)H, (int)vocab);
}

int b200_embed_rows(const void* table, const void* ids, void* out, int64_t B, int64_t H, int64_t vocab, void* stream) {
  return embed_rows_impl("embed_rows", table, ids, out, nullptr, B, H, vocab, stream);
}

int b200_embed_rows_stats(const void* table, const void* ids, void* out, void* stats, int64_t B, int64_t H, int64_t vocab, void* stream) {
  if (!stats) return fail(B200_EINVAL, "embed_rows_stats: null pointer");
  if (H % 16 != 0) return fail(B200_EINVAL, "embed_rows_stats: need H %% 16 == 0");
  return embed_rows_impl("embed_rows_stats", table, ids, out, stats, B, H, vocab, stream);
}

int b200_advance_pos(void* pos, int64_t delta, void* stream) {
  if (!pos) return fail(B200_EINVAL, "advance_pos: null pointer");
  int rc = ensure_device();
  if (rc) return rc;
  return launch("advance_pos", advance_pos_kernel, dim3(1), dim3(32), 0, static_cast<cudaStream_t>(stream), (int*)pos,
                (int)delta);
}

static int silu_mul_impl(const char* who, const void* gu, void* out, int64_t B, int64_t I, bool early, void* stream) {
  if (B < 0 || I <= 0 || I % 8 != 0) return fail(B200_EINVAL, "%s: need I %% 8 == 0", who);
  if (B == 0) return B200_OK;
  if (!gu || !out) return fail(B200_EINVAL, "%s: null pointer", who);
  int rc = ensure_device();
  if (rc) return rc;
  const int64_t total8 = B * (I / 8);
  return launch("silu_mul", early ? silu_mul_kernel<true> : silu_mul_kernel<false>, dim3((unsigned)((total8 + 255) / 256)), dim3(256), 0,
                static_cast<cudaStream_t>(stream), (const __half*)gu, (__half*)out, (int)I, total8);
}

int b200_silu_mul(const void* gu, void* out, int64_t B, int64_t I, void* stream) {
  return silu_mul_impl("silu_mul", gu, out, B, I, false, stream);
}

int b200_silu_mul_early_release(const void* gu, void* out, int64_t B, int64_t I, void* stream) {
  return silu_mul_impl("silu_mul_early_release", gu, out, B, I, true, stream);
}

}  // extern "C"
