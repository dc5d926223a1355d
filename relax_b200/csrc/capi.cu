// C ABI of the kernel library: argument validation, kernel-family dispatch, error state.
// Everything a caller outside this library may bind is declared in include/b200_q4f16.h.
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "internal.h"

namespace b200 {

namespace {
thread_local char g_err[512] = {0};
thread_local int64_t g_launches = 0;
thread_local cudaStream_t g_stream = nullptr;
}  // namespace

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

void count_launch(int n) { g_launches += n; }

Options& options() {
  static Options o;
  return o;
}

thread_local int g_call_layout = -1;
int current_layout() { return g_call_layout >= 0 ? g_call_layout : (int)options().weights_layout; }
LayoutScope::LayoutScope(int layout) : saved(g_call_layout) {
  if (layout >= 0) g_call_layout = layout;
}
LayoutScope::~LayoutScope() { g_call_layout = saved; }

// Per-process cache of "device d is usable" (index = device ordinal).
int ensure_device() {
  static int ok[64] = {0};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(B200_ENODEVICE, "no CUDA device: %s", cudaGetErrorString(e));
  if (dev >= 0 && dev < 64 && ok[dev]) return B200_OK;
  cudaDeviceProp p;
  e = cudaGetDeviceProperties(&p, dev);
  if (e != cudaSuccess) return fail(B200_ENODEVICE, "cudaGetDeviceProperties: %s", cudaGetErrorString(e));
  if (p.major != 10)
    return fail(B200_ENODEVICE, "device %d is sm_%d%d; this library is built for sm_100a only and has no fallback",
                dev, p.major, p.minor);
  if (dev >= 0 && dev < 64) ok[dev] = 1;
  return B200_OK;
}

int raise_smem_limit(SmemLimit& limit, const void* kern, size_t bytes, const char* who) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    limit.raise(dev, bytes, [&](size_t n) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
      return e == cudaSuccess ? 0 : 1;
    });
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "%s: cudaFuncSetAttribute(%zu): %s", who, bytes, cudaGetErrorString(e));
  return B200_OK;
}

int sm_count() {
  static int n[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!n[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    n[dev] = v;
  }
  return n[dev];
}

namespace {

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_common(const char* who, const void* wq, const void* scales, int64_t N, int64_t K) {
  if (N < 0 || K < 0) return fail(B200_EINVAL, "%s: negative size N=%lld K=%lld", who, (long long)N, (long long)K);
  if (K % 32 != 0) return fail(B200_EINVAL, "%s: K=%lld is not a multiple of the group size 32", who, (long long)K);
  if (N > 0x7fffffffLL / 32 || K > 0x3fffffffLL)
    return fail(B200_EINVAL, "%s: N=%lld K=%lld exceeds the supported range", who, (long long)N, (long long)K);
  if (N > 0 && K > 0) {
    if (!wq || !scales) return fail(B200_EINVAL, "%s: null weight or scale pointer", who);
    if (!aligned16(wq)) return fail(B200_EINVAL, "%s: packed weights must be 16-byte aligned", who);
    if (reinterpret_cast<uintptr_t>(scales) & 1u) return fail(B200_EINVAL, "%s: scales must be 2-byte aligned", who);
  }
  return B200_OK;
}

int check_matmul(const char* who, const void* x, const void* wq, const void* scales, const void* y, int64_t M,
                 int64_t N, int64_t K) {
  if (M < 0) return fail(B200_EINVAL, "%s: negative M=%lld", who, (long long)M);
  int rc = check_common(who, wq, scales, N, K);
  if (rc) return rc;
  if (M > 0x7fffffffLL / 64) return fail(B200_EINVAL, "%s: M=%lld exceeds the supported range", who, (long long)M);
  if (M > 0 && K > 0 && (!x || !aligned16(x))) return fail(B200_EINVAL, "%s: x must be non-null and 16-byte aligned", who);
  if (M > 0 && N > 0 && (!y || (reinterpret_cast<uintptr_t>(y) & 1u)))
    return fail(B200_EINVAL, "%s: y must be non-null and 2-byte aligned", who);
  return B200_OK;
}

// y = 0 when the reduction is empty (K == 0): the sum over no terms.
int zero_output(void* y, int64_t M, int64_t N, cudaStream_t s) {
  if (M * N == 0) return B200_OK;
  cudaError_t e = cudaMemsetAsync(y, 0, (size_t)(M * N) * 2, s);
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "cudaMemsetAsync: %s", cudaGetErrorString(e));
  return B200_OK;
}

enum Family { kAuto, kGemv, kGemm, kGemmWs };

// Whether the automatic choice asks the weight-stationary kernel first.
// 9 rows and more, and 5..8 where K is long: the weight-stationary kernel, whose weights stream once up to 128 rows.
// Measured on B200, skinny / weight-stationary kernel in us at 4, 8 and 16 rows: N = K = 4096 6.0 / 6.1, 7.7 / 6.4,
// 11.1 / 6.5; N = 22016 16.5 / 17.9, 17.9 / 18.1, 24.4 / 18.4; N = 4096, K = 11008 11.8 / 12.2, 18.9 / 12.3, 29.3 / 12.5;
// N = 1280, K = 8192 6.6 / 5.9, 9.7 / 6.0, 17.0 / 6.1 (the skinny kernel stages all of x in every CTA, and its
// arithmetic grows from 8 columns on).  At 5..8 rows and a shorter K the skinny kernel is the better one inside a
// decode step, where two of its CTAs fit an SM and it starts beside the kernel before it (8 layers of hidden
// 2048 at 5 rows: 413 us with it, 440 without).  Above 128 rows it cuts the tokens into tiles to suit the shape; the
// prefill kernel with its 256-token tiles keeps the long prompts that one wave of them holds (prefill_kernel_is_ahead in
// ws_plan.h: the launcher says B200_ENOTREADY) and loses the rest (44 against 11.8 us at M = 129, N = K = 4096, 164 against
// 134-140 at M = 2048, N = 11008).
// Where K is not a multiple of 256 (or the scales are not 16-byte aligned) the other choice up to 16 rows is the
// register-streaming kernel, whose time grows with the rows: it keeps one row and small products, M * N * K < 50 M, at two
// rows < 100 M where K < 5000 (streaming / weight-stationary in us: 4 x 4096 x 2080 5.1 / 5.3, 16 x 1024 x 1056 4.5 / 4.5;
// 2 x 8192 x 3200 9.4 / 10.7, 2 x 11008 x 4128 13.3 / 16.2, with weights from HBM 15.3 / 15.6, 2 x 22016 x 2080 13.7 / 15.1, but
// 2 x 8192 x 5152 21.6 / 19.0 and 2 x 16384 x 3200 16.1 / 13.7; 3 x 8640 x 3200 13.8 / 11.0, 8 x 4096 x 2080 7.0 / 5.5,
// 16 x 22016 x 4128 86 / 24; above 16 rows, against the prefill kernel, 32 x 8640 x 3200 43 / 11.5, 2048 x 11008 x 4128 188 / 159).
// (Above a gemm.ws_max_m that was lowered the skinny and prefill kernels take over, and a variant of the skinny kernel
// asked for by option keeps its rows.)
bool weight_stationary_first(int64_t M, int64_t N, int64_t K, bool ragged) {
  const int64_t streamed = M == 2 && K < 5000 ? 100000000 : 50000000;
  const bool ahead = M > 16 || (ragged ? M >= 2 && M * N * K >= streamed : M >= 9 || (M >= 5 && K >= 8192));
  return ahead && M <= options().gemm_ws_max_m && (M > 16 || options().gemv_variant == 0);
}

// Of that, the skinny kernel's form for a ragged K takes two to four rows of the weight-stationary kernel's share and up to eight of the
// streaming kernel's where K is long enough for its start-up.  Weight-stationary / skinny in us: 2 x 8640 x 3200 11.0 / 7.4,
// 3 x 8640 x 3200 9.7 / 7.6, 4 x 12288 x 1056 6.3 / 6.0, 4 x 5120 x 5152 11.1 / 9.6, 2 x 4096 x 9248 12.3 / 9.8, 4 x 4096 x 7200 10.9 / 9.9,
// but 5 x 4096 x 4128 8.4 / 8.6, 8 x 22016 x 2080 13.8 / 15.3, 8 x 4096 x 7200 11.1 / 12.8, 6 x 2560 x 6944 8.3 / 11.2; streaming / skinny:
// 3 x 2048 x 5152 9.5 / 5.1, 8 x 512 x 2080 4.9 / 3.8, 4 x 4096 x 2080 5.2 / 4.7, but 2 x 4096 x 1056 3.1 / 3.4, 8 x 4096 x 1056 4.4 / 4.5.
// Not from three rows on: few chunks of very many tiles (4 x 28672 x 1056 10.1 / 10.8, 4 x 24576 x 544 6.9 / 8.9), and a long K of one to two tiles an
// SM (4 x 3072 x 9248 11.1 / 13.8, 3 x 4096 x 9248 12.5 / 13.6).  Not against the streaming kernel: where a wave of tiles leaves more than half of
// the next one empty, with two rows (2 x 6144 x 2592 5.9 / 6.6) and for a short K (2 x 3072 x 2080 3.8 / 4.7, 3 x 6144 x 2080 5.7 / 6.5).
bool skinny_ragged(int64_t M, int64_t N, int64_t K) {
  if (M < 2 || M > 8 || options().gemv_variant != 0) return false;
  const int64_t tiles = (N + 15) / 16, sms = sm_count();
  if (weight_stationary_first(M, N, K, true)) {
    if (M > 4) return false;
    return M == 2 || !((K <= 1280 && N >= 14000) || (K > 8192 && tiles > sms && tiles <= 2 * sms));
  }
  const bool one_wave = 2 * tiles > 2 * sms && 2 * tiles < 3 * sms, two_waves = tiles > 2 * sms && tiles < 3 * sms;
  if (M <= 4 && K < 2304 && (one_wave || two_waves)) return false;
  return K >= 2048 && !(M == 2 && two_waves);
}

int matmul_impl(Family fam, const char* who, const void* x, const void* wq, const void* scales, void* y, int64_t M,
                int64_t N, int64_t K, void* stream) {
  int rc = check_matmul(who, x, wq, scales, y, M, N, K);
  if (rc) return rc;
  if (fam == kGemv && (M < 1 || M > 16))
    return fail(B200_EINVAL, "%s: the skinny kernel takes 1 <= M <= 16, got %lld", who, (long long)M);
  rc = ensure_device();
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (M == 0 || N == 0) return B200_OK;
  if (K == 0) return zero_output(y, M, N, s);
  const bool use_gemv = fam == kGemv || (fam == kAuto && M <= 16);
  auto xh = static_cast<const __half*>(x);
  auto wh = static_cast<const uint32_t*>(wq);
  auto sh = static_cast<const __half*>(scales);
  auto yh = static_cast<__half*>(y);
  const bool ragged = K % 256 != 0 || !aligned16(scales);
  if (fam == kAuto && ragged && skinny_ragged(M, N, K)) {
    rc = launch_gemv_pipe_ragged(xh, wh, sh, yh, M, N, K, s);
    if (rc != B200_ENOTREADY) return rc;
  }
  if (fam == kGemmWs || (fam == kAuto && weight_stationary_first(M, N, K, ragged))) {
    rc = fam == kGemmWs && (M > 128 || ragged) ? B200_ENOTREADY : launch_gemm_ws(xh, wh, sh, yh, M, N, K, s);
    if (rc != B200_ENOTREADY) return rc;
    if (fam == kGemmWs) return fail(B200_EINVAL, "%s: the weight-stationary kernel takes 1 <= M <= 128, K %% 256 == 0, 16-byte aligned scales", who);
  }
  if (use_gemv) return launch_gemv(xh, wh, sh, yh, M, N, K, s);
  return launch_gemm(xh, wh, sh, yh, M, N, K, s);
}

// ---- DLPack validation -------------------------------------------------------------------
bool is_dtype(const B200DLTensor* t, int code, int bits) {
  return t->dtype.code == code && t->dtype.bits == bits && t->dtype.lanes == 1;
}

int check_tensor(const char* who, const char* name, const B200DLTensor* t, int code, int bits, int* dev) {
  if (!t) return fail(B200_EINVAL, "%s: %s is null", who, name);
  if (t->ndim != 2) return fail(B200_EINVAL, "%s: %s must have 2 dimensions, has %d", who, name, t->ndim);
  if (!t->shape) return fail(B200_EINVAL, "%s: %s has no shape", who, name);
  if (!is_dtype(t, code, bits))
    return fail(B200_EINVAL, "%s: %s must be %s%d, got code=%d bits=%d lanes=%d", who, name,
                code == 2 ? "float" : "uint", bits, t->dtype.code, t->dtype.bits, t->dtype.lanes);
  if (t->device.device_type != 2 /* kDLCUDA */)
    return fail(B200_EINVAL, "%s: %s is not on a CUDA device (device_type=%d)", who, name, t->device.device_type);
  if (*dev < 0) *dev = t->device.device_id;
  else if (*dev != t->device.device_id)
    return fail(B200_EINVAL, "%s: %s is on device %d, other arguments on device %d", who, name, t->device.device_id, *dev);
  if (t->strides && t->shape[0] != 0 && t->shape[1] != 0) {  // compact row-major only (strides of size-1 dimensions are free)
    int64_t expect = 1;
    for (int i = 1; i >= 0; --i) {
      if (t->shape[i] != 1 && t->strides[i] != expect)
        return fail(B200_EINVAL, "%s: %s is not contiguous", who, name);
      expect *= t->shape[i];
    }
  }
  if (t->shape[0] < 0 || t->shape[1] < 0) return fail(B200_EINVAL, "%s: %s has a negative extent", who, name);
  return B200_OK;
}

void* data_ptr(const B200DLTensor* t) { return static_cast<char*>(t->data) + t->byte_offset; }

int check_current_device(const char* who, int dev) {
  int cur = -1;
  cudaError_t e = cudaGetDevice(&cur);
  if (e != cudaSuccess) return fail(B200_ENODEVICE, "%s: no CUDA device: %s", who, cudaGetErrorString(e));
  if (cur != dev)
    return fail(B200_EINVAL, "%s: tensors live on device %d but the current device is %d", who, dev, cur);
  return B200_OK;
}

}  // namespace
}  // namespace b200

using namespace b200;

// Small host transfers as kernels.  A copy-engine transfer on either side of a 5 us matmul costs
// more than the matmul (each switch between the copy engine and the SMs is a few microseconds), so
// activations and results up to kHostKernelBytes travel by a kernel that reads or writes the pinned host
// buffer through its device mapping: 16 bytes per thread and one CTA per 4 KB, up to kHostCopyCtas of them, so that a
// read of up to 32 KB makes one round trip over the bus; more requests at a time than that slow the larger copies down.
// Measured, a call among others in us with one CTA per 16 KB / one per 4 KB / the same up to eight: 1 x 4096 x 4096
// 14.0 / 12.4 / 12.3, 3 x 8640 x 3200 22.6 / 20.3 / 20.4, 4 x 12288 x 4096 21.0 / 23.8 / 21.8, 6 x 4096 x 8192 20.6 / 22.4 / 20.5,
// 16 x 4096 x 4096 24.7 / 22.1 / 20.6, 16 x 8192 x 8192 34.9 / 32.0 / 30.8; waited for, 8 x 4096 x 11008 33.6 / 34.9 / 30.6.
// The copies are launched as programmatic dependents.  A copy lets the next launch begin once it has waited itself: the matmul
// then starts beside it (it reads only weights before its own wait), but not beside the call in front, whose matmul it
// would take the SMs from.  Without the attribute on the copy of x / with it, us a call among others: 1 x 4096 x 4096 12.4 / 11.1,
// 1 x 8192 x 8192 18.2 / 16.4, 4 x 22016 x 4096 28.0 / 25.9, 6 x 4096 x 4096 17.2 / 14.4, 16 x 4096 x 4096 19.2 / 18.3.
// The skinny matmul can store the result to the host buffer itself, next to y_dev, in pieces of 32 bytes (one row) or 16: a launch less, but
// most of those stores come at the end of the matmul and take the bus longer than a copy does.  Launched by the host, one or two rows of a
// short call are bound by the launches, and a CTA with several long tiles sends the stores of the first beside the last; elsewhere the copy is
// faster.  Copy / direct, us a call among others, 1 x 512 x 1024 12.1 / 10.0, 1 x 4096 x 4096 12.3 / 10.2, 2 x 2048 x 4096 12.1 / 10.6, 2 x 8192 x 1024
// 12.1 / 11.1, 1 x 16384 x 4096 18.1 / 17.5, 2 x 22016 x 4096 22.5 / 21.4, but 1 x 12288 x 2048 12.1 / 12.6, 1 x 4096 x 8192 12.2 / 12.8, 1 x 4096 x 11008
// 14.3 / 15.3, 2 x 8192 x 2048 12.1 / 12.3, 2 x 22016 x 1024 14.2 / 16.1, 3 x 12288 x 2048 13.5 / 15.8, 4 x 4096 x 4096 12.5 / 13.3, 4 x 22016 x 1024 16.4 / 23.3.
// Replayed from a graph, where launches follow each other without the host, it is faster for up to four rows unless they have many outputs of
// a short K: 1 x 512 x 1024 6.3 / 4.8, 1 x 4096 x 11008 11.8 / 10.9, 3 x 12288 x 4096 14.2 / 12.8, 4 x 22016 x 11008 45.8 / 42.4, but 3 x 12288 x 1024 9.0 / 9.9,
// 4 x 22016 x 1024 12.4 / 17.7.
// Pageable host memory and larger transfers use cudaMemcpyAsync.
namespace b200 {
namespace {
constexpr size_t kHostKernelBytes = 256 * 1024;
constexpr size_t kHostCopyCtas = 8;

// Whether the matmul stores its result to the host buffer itself.
bool host_direct(int64_t M, int64_t N, int64_t K, cudaStream_t s) {
  if (M > 4) return false;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &status) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (status == cudaStreamCaptureStatusActive) return M <= 2 || K >= 4096 || M * N <= 12288 + 8 * K;
  return M <= 2 && (M * N * K <= 1 << 24 || (N >= 12288 && K >= 4096));
}

__global__ void __launch_bounds__(256) host_copy_kernel(const unsigned char* __restrict__ src, unsigned char* __restrict__ dst,
                                                        size_t bytes) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const size_t n16 = bytes >> 4;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x)
    reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  if (blockIdx.x == 0)
    for (size_t i = (n16 << 4) + threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
}

// Device-side address of a pinned (page-locked, mapped) host buffer, or null for anything else.
void* mapped_host_pointer(const void* host) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (a.type != cudaMemoryTypeHost) return nullptr;
  return a.devicePointer;
}

// dst <- src (one of them a mapped host buffer) on `s`, a programmatic dependent of the kernel before it in the stream (the copy
// waits for that kernel's completion itself).
int host_copy(const void* src, void* dst, size_t bytes, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  const size_t ctas = (bytes + 4095) / 4096;
  cfg.gridDim = dim3((unsigned)(ctas < kHostCopyCtas ? ctas : kHostCopyCtas));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, host_copy_kernel, static_cast<const unsigned char*>(src),
                                     static_cast<unsigned char*>(dst), bytes);
  if (e != cudaSuccess) return fail(B200_ELAUNCH, "q4f16_matmul_host: copy kernel: %s", cudaGetErrorString(e));
  count_launch();
  return B200_OK;
}
}  // namespace
}  // namespace b200

extern "C" {

const char* b200_last_error(void) { return g_err; }
int b200_abi_version(void) { return 102; }

int b200_set_stream(void* s) {
  g_stream = static_cast<cudaStream_t>(s);
  return B200_OK;
}
void* b200_get_stream(void) { return g_stream; }

int64_t b200_launch_count(void) { return g_launches; }
void b200_reset_launch_count(void) { g_launches = 0; }

int b200_device_error_flags(void) {
  int rc = ensure_device();
  if (rc) return rc;
  if (cudaDeviceSynchronize() != cudaSuccess) return fail(B200_EDEVICE, "device_error_flags: %s", cudaGetErrorString(cudaGetLastError()));
  return device_error_flags_read_and_clear();
}

int b200_set_option(const char* name, int64_t v) {
  if (!name) return fail(B200_EINVAL, "set_option: null name");
  Options& o = options();
  if (!strcmp(name, "gemv.variant")) { if (v < 0 || v > 2) return fail(B200_EINVAL, "gemv.variant in 0..2"); o.gemv_variant = v; }
  else if (!strcmp(name, "gemv.warps")) { if (v < 0 || v > 16) return fail(B200_EINVAL, "gemv.warps in 0..16"); o.gemv_warps = v; }
  else if (!strcmp(name, "gemv.stages")) { if (v < 0 || v > 16) return fail(B200_EINVAL, "gemv.stages in 0..16"); o.gemv_stages = v; }
  else if (!strcmp(name, "gemv.pdl")) { o.gemv_pdl = v != 0; }
  else if (!strcmp(name, "gemv.ctas_per_sm")) { if (v < 0 || v > 8) return fail(B200_EINVAL, "gemv.ctas_per_sm in 0..8"); o.gemv_ctas_per_sm = v; }
  else if (!strcmp(name, "gemv.exact")) { if (v < 0 || v > 2) return fail(B200_EINVAL, "gemv.exact is 0 (by shape), 1 (exact form) or 2 (fast form)"); o.gemv_exact = v; }
  else if (!strcmp(name, "gemv.peer_wait_ms")) { if (v < 1 || v > 60000) return fail(B200_EINVAL, "gemv.peer_wait_ms in 1..60000"); o.gemv_peer_wait_ms = v; }
  else if (!strcmp(name, "layer.wait_ms")) { if (v < 1 || v > 60000) return fail(B200_EINVAL, "layer.wait_ms in 1..60000"); o.layer_wait_ms = v; }
  else if (!strcmp(name, "layer.stages")) { if (v < 0 || v > 5) return fail(B200_EINVAL, "layer.stages in 0..5"); o.layer_stages = v; }
  else if (!strcmp(name, "layer.max_ctas")) { if (v < 0 || v > 1024) return fail(B200_EINVAL, "layer.max_ctas in 0..1024"); o.layer_max_ctas = v; }
  else if (!strcmp(name, "gemm.ws_ksplit")) { if (v < 0 || v > 8 || (v & (v - 1))) return fail(B200_EINVAL, "gemm.ws_ksplit is 0, 1, 2, 4 or 8"); o.gemm_ws_ksplit = v; }
  else if (!strcmp(name, "gemm.ws_x_stages")) { if (v < 0 || v > 8) return fail(B200_EINVAL, "gemm.ws_x_stages in 0..8"); o.gemm_ws_x_stages = v; }
  else if (!strcmp(name, "gemm.ws_w_stages")) { if (v != 0) return fail(B200_EINVAL, "gemm.ws_w_stages is 0: the dequantised weights sit in a fixed ring in tensor memory"); }
  else if (!strcmp(name, "gemm.ws_r_stages")) { if (v < 0 || v == 1 || v > 8) return fail(B200_EINVAL, "gemm.ws_r_stages is 0 or in 2..8"); o.gemm_ws_r_stages = v; }
  else if (!strcmp(name, "gemm.ws_xk")) { if (v != 0) return fail(B200_EINVAL, "gemm.ws_xk is 0: the K blocks per stage follow from the token tile"); }
  else if (!strcmp(name, "gemm.ws_max_m")) { if (v < 0 || v > kWsNoLimit) return fail(B200_EINVAL, "gemm.ws_max_m in 0..%lld (no limit)", (long long)kWsNoLimit); o.gemm_ws_max_m = v; }
  else if (!strcmp(name, "weights.layout")) { if (v != B200_LAYOUT_REFERENCE && v != B200_LAYOUT_PAIRED) return fail(B200_EINVAL, "weights.layout is 0 (reference) or 1 (paired)"); o.weights_layout = v; }
  else if (!strcmp(name, "gemm.max_ctas")) { if (v < 0 || v > 1024) return fail(B200_EINVAL, "gemm.max_ctas in 0..1024"); o.gemm_max_ctas = v; }
  else return fail(B200_EINVAL, "set_option: unknown option '%s'", name);
  return B200_OK;
}

int64_t b200_get_option(const char* name) {
  if (!name) return -1;
  Options& o = options();
  if (!strcmp(name, "gemv.variant")) return o.gemv_variant;
  if (!strcmp(name, "gemv.warps")) return o.gemv_warps;
  if (!strcmp(name, "gemv.stages")) return o.gemv_stages;
  if (!strcmp(name, "gemv.pdl")) return o.gemv_pdl;
  if (!strcmp(name, "gemv.ctas_per_sm")) return o.gemv_ctas_per_sm;
  if (!strcmp(name, "gemv.exact")) return o.gemv_exact;
  if (!strcmp(name, "gemv.peer_wait_ms")) return o.gemv_peer_wait_ms;
  if (!strcmp(name, "gemm.max_ctas")) return o.gemm_max_ctas;
  if (!strcmp(name, "layer.wait_ms")) return o.layer_wait_ms;
  if (!strcmp(name, "layer.stages")) return o.layer_stages;
  if (!strcmp(name, "layer.max_ctas")) return o.layer_max_ctas;
  if (!strcmp(name, "gemm.ws_ksplit")) return o.gemm_ws_ksplit;
  if (!strcmp(name, "gemm.ws_max_m")) return o.gemm_ws_max_m;
  if (!strcmp(name, "gemm.ws_x_stages")) return o.gemm_ws_x_stages;
  if (!strcmp(name, "gemm.ws_w_stages") || !strcmp(name, "gemm.ws_xk")) return 0;
  if (!strcmp(name, "gemm.ws_r_stages")) return o.gemm_ws_r_stages;
  if (!strcmp(name, "weights.layout")) return o.weights_layout;
  return -1;
}

int b200_q4f16_dequantize(const void* wq, const void* scales, void* w_out, int64_t N, int64_t K, void* stream) {
  int rc = check_common("q4f16_dequantize", wq, scales, N, K);
  if (rc) return rc;
  if (N > 0 && K > 0 && (!w_out || !aligned16(w_out)))
    return fail(B200_EINVAL, "q4f16_dequantize: output must be non-null and 16-byte aligned");
  rc = ensure_device();
  if (rc) return rc;
  return launch_dequantize(static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                           static_cast<__half*>(w_out), N, K, static_cast<cudaStream_t>(stream));
}

static int check_layout(const char* who, int32_t layout) {
  if (layout != B200_LAYOUT_REFERENCE && layout != B200_LAYOUT_PAIRED)
    return fail(B200_EINVAL, "%s: unknown weight layout %d (0 reference, 1 paired)", who, (int)layout);
  return B200_OK;
}

static int repack_impl(const char* who, const void* in, void* out, int64_t N, int64_t K, int32_t layout, bool to_layout,
                       void* stream) {
  int rc = check_layout(who, layout);
  if (rc) return rc;
  if (N < 0 || K < 0) return fail(B200_EINVAL, "%s: negative shape N=%lld K=%lld", who, (long long)N, (long long)K);
  if (K % 32 != 0) return fail(B200_EINVAL, "%s: K=%lld is not a multiple of the group size 32", who, (long long)K);
  if (N > 0 && K > 0 && (!in || !out)) return fail(B200_EINVAL, "%s: null pointer", who);
  if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 3u) != 0)
    return fail(B200_EINVAL, "%s: buffers must be 4-byte aligned", who);
  if (N > 0 && K > 0 && in != out) {
    const char* a = static_cast<const char*>(in);
    const char* b = static_cast<const char*>(out);
    const int64_t bytes = N * (K / 2);
    if (a < b + bytes && b < a + bytes) return fail(B200_EINVAL, "%s: input and output overlap without being the same buffer", who);
  }
  if ((rc = ensure_device())) return rc;
  return launch_repack(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out), N * (K / 8), layout, to_layout,
                       static_cast<cudaStream_t>(stream));
}

int64_t b200_lm_head_scratch_bytes(void) {
  if (ensure_device()) return -1;
  return lm_head_scratch_bytes();
}

static int lm_head_impl(const void* h, const void* stats, const void* norm_w, float eps, void* h_out, const void* w, void* logits,
                        int32_t* tokens, void* scratch, int64_t B, int64_t V, int64_t H, int64_t token_offset, void* stream) {
  if (B < 1 || B > 16) return fail(B200_EINVAL, "lm_head: takes 1 <= B <= 16 rows, got %lld", (long long)B);
  if (V < 1 || V > 0x7fffff00LL || H < 32 || H % 32 != 0)
    return fail(B200_EINVAL, "lm_head: need 1 <= V < 2^31, H >= 32 and H %% 32 == 0 (V=%lld H=%lld)", (long long)V, (long long)H);
  if (!h || !w || (!logits && !tokens)) return fail(B200_EINVAL, "lm_head: null pointer (h, w, and one of logits / tokens are required)");
  if (tokens && !scratch) return fail(B200_EINVAL, "lm_head: tokens need the scratch buffer (b200_lm_head_scratch_bytes)");
  if (!aligned16(h) || !aligned16(w) || (scratch && !aligned16(scratch)) || (reinterpret_cast<uintptr_t>(logits) & 1u) ||
      (reinterpret_cast<uintptr_t>(tokens) & 3u))
    return fail(B200_EINVAL, "lm_head: h, w and scratch must be 16-byte aligned");
  if (token_offset < 0 || token_offset + V > 0x7fffffffLL) return fail(B200_EINVAL, "lm_head: token_offset + V overflows int32");
  int rc = ensure_device();
  if (rc) return rc;
  rc = launch_lm_head(static_cast<const __half*>(h), static_cast<const float*>(stats), static_cast<const __half*>(norm_w), eps,
                      static_cast<__half*>(h_out), static_cast<const __half*>(w), static_cast<__half*>(logits), tokens,
                      static_cast<float*>(scratch), B, V, H, token_offset, static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(B200_EINVAL, "lm_head: %lld rows of H=%lld do not fit in shared memory", (long long)B, (long long)H);
  return rc;
}

int b200_lm_head(const void* h, const void* w, void* logits, int32_t* tokens, void* scratch, int64_t B, int64_t V,
                 int64_t H, int64_t token_offset, void* stream) {
  return lm_head_impl(h, nullptr, nullptr, 0.f, nullptr, w, logits, tokens, scratch, B, V, H, token_offset, stream);
}

int b200_lm_head_norm(const void* x, const void* stats, const void* norm_w, float eps, void* h_out, const void* w, void* logits,
                      int32_t* tokens, void* scratch, int64_t B, int64_t V, int64_t H, int64_t token_offset, void* stream) {
  if (B > 8) return fail(B200_EINVAL, "lm_head_norm: takes 1 <= B <= 8 rows, got %lld", (long long)B);
  if (H % 64 != 0) return fail(B200_EINVAL, "lm_head_norm: needs H %% 64 == 0");
  if (!stats || !norm_w || !aligned16(stats) || !aligned16(norm_w))
    return fail(B200_EINVAL, "lm_head_norm: statistics and norm weight must be non-null and 16-byte aligned");
  if (h_out == x || !aligned16(h_out)) return fail(B200_EINVAL, "lm_head_norm: h_out must be 16-byte aligned and not x");
  return lm_head_impl(x, stats, norm_w, eps, h_out, w, logits, tokens, scratch, B, V, H, token_offset, stream);
}

int b200_argmax_rows(const void* logits, int32_t* tokens, int64_t B, int64_t V, void* stream) {
  if (B < 0 || B > 0x7fffffffLL || V < 1 || V > 0x7ffffff0LL) return fail(B200_EINVAL, "argmax_rows: need B >= 0 and 1 <= V < 2^31");
  if (B == 0) return B200_OK;
  if (!logits || !tokens || (reinterpret_cast<uintptr_t>(logits) & 1u) || (reinterpret_cast<uintptr_t>(tokens) & 3u))
    return fail(B200_EINVAL, "argmax_rows: null or misaligned pointer");
  if (int rc = ensure_device()) return rc;
  return launch_argmax_rows(static_cast<const __half*>(logits), tokens, B, V, static_cast<cudaStream_t>(stream));
}

int b200_q4f16_repack(const void* wq, void* packed_out, int64_t N, int64_t K, int32_t layout, void* stream) {
  return repack_impl("q4f16_repack", wq, packed_out, N, K, layout, true, stream);
}

int b200_q4f16_unpack(const void* packed, void* wq_out, int64_t N, int64_t K, int32_t layout, void* stream) {
  return repack_impl("q4f16_unpack", packed, wq_out, N, K, layout, false, stream);
}

int b200_q4f16_matmul_layout(const void* x, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                             int32_t layout, void* stream) {
  int rc = check_layout("q4f16_matmul_layout", layout);
  if (rc) return rc;
  LayoutScope scope(layout);
  return matmul_impl(kAuto, "q4f16_matmul_layout", x, wq, scales, y, M, N, K, stream);
}

int b200_q4f16_dequantize_layout(const void* wq, const void* scales, void* w_out, int64_t N, int64_t K, int32_t layout,
                                 void* stream) {
  int rc = check_layout("q4f16_dequantize_layout", layout);
  if (rc) return rc;
  LayoutScope scope(layout);
  return b200_q4f16_dequantize(wq, scales, w_out, N, K, stream);
}

int b200_q4f16_matmul(const void* x, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                      void* stream) {
  return matmul_impl(kAuto, "q4f16_matmul", x, wq, scales, y, M, N, K, stream);
}
int b200_q4f16_gemv(const void* x, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                    void* stream) {
  return matmul_impl(kGemv, "q4f16_gemv", x, wq, scales, y, M, N, K, stream);
}
int b200_q4f16_gemm(const void* x, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                    void* stream) {
  return matmul_impl(kGemm, "q4f16_gemm", x, wq, scales, y, M, N, K, stream);
}

int b200_q4f16_gemv_rmsnorm(const void* x, const void* delta, const void* norm_w, void* x_out, float eps, const void* wq,
                            const void* scales, void* y, int64_t M, int64_t N, int64_t K, void* stream) {
  const char* who = "q4f16_gemv_rmsnorm";
  int rc = check_matmul(who, x, wq, scales, y, M, N, K);
  if (rc) return rc;
  if (M < 1 || M > 16) return fail(B200_EINVAL, "%s: takes 1 <= M <= 16, got %lld", who, (long long)M);
  if (N < 1 || K < 256 || K % 256 != 0) return fail(B200_EINVAL, "%s: needs N >= 1 and K a positive multiple of 256", who);
  if (!aligned16(scales)) return fail(B200_EINVAL, "%s: scales must be 16-byte aligned", who);
  if (!norm_w || !aligned16(norm_w)) return fail(B200_EINVAL, "%s: norm weight must be non-null and 16-byte aligned", who);
  if ((delta && !aligned16(delta)) || (x_out && !aligned16(x_out))) return fail(B200_EINVAL, "%s: delta / x_out must be 16-byte aligned", who);
  if (x_out == x) return fail(B200_EINVAL, "%s: x_out must not alias x (other CTAs still read x)", who);
  rc = ensure_device();
  if (rc) return rc;
  rc = launch_gemv_pipe_rmsnorm(static_cast<const __half*>(x), static_cast<const __half*>(delta), static_cast<const __half*>(norm_w),
                                static_cast<__half*>(x_out), eps, static_cast<const uint32_t*>(wq),
                                static_cast<const __half*>(scales), static_cast<__half*>(y), M, N, K,
                                static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(B200_EINVAL, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

int b200_q4f16_gemv_rmsnorm_rope(const void* x, const void* delta, const void* norm_w, void* x_out, float eps, const void* wq,
                                 const void* scales, const void* cos_t, const void* sin_t, const void* pos, void* q_out,
                                 void* k_cache, void* v_cache, int64_t heads, int64_t K, void* stream) {
  const char* who = "q4f16_gemv_rmsnorm_rope";
  if (heads < 1 || heads > 4096) return fail(B200_EINVAL, "%s: heads %lld out of range", who, (long long)heads);
  const int64_t N = 3 * heads * 128;
  int rc = check_matmul(who, x, wq, scales, q_out, 1, N, K);
  if (rc) return rc;
  if (K < 256 || K % 256 != 0) return fail(B200_EINVAL, "%s: needs K a positive multiple of 256", who);
  if (!aligned16(scales)) return fail(B200_EINVAL, "%s: scales must be 16-byte aligned", who);
  if (!norm_w || !aligned16(norm_w)) return fail(B200_EINVAL, "%s: norm weight must be non-null and 16-byte aligned", who);
  if ((delta && !aligned16(delta)) || (x_out && !aligned16(x_out))) return fail(B200_EINVAL, "%s: delta / x_out must be 16-byte aligned", who);
  if (x_out == x) return fail(B200_EINVAL, "%s: x_out must not alias x (other CTAs still read x)", who);
  if (!cos_t || !sin_t || !pos || !k_cache || !v_cache) return fail(B200_EINVAL, "%s: null table, position or cache pointer", who);
  rc = ensure_device();
  if (rc) return rc;
  // B200_ENOTREADY (no message): the launch would not use the fast form; the caller runs b200_q4f16_gemv_rmsnorm and
  // b200_rope_kv_append instead
  return launch_gemv_pipe_rmsnorm_rope(static_cast<const __half*>(x), static_cast<const __half*>(delta),
                                       static_cast<const __half*>(norm_w), static_cast<__half*>(x_out), eps, nullptr,
                                       static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                                       static_cast<const float*>(cos_t), static_cast<const float*>(sin_t),
                                       static_cast<const int*>(pos), static_cast<__half*>(q_out), static_cast<__half*>(k_cache),
                                       static_cast<__half*>(v_cache), heads, K, static_cast<cudaStream_t>(stream));
}

int b200_q4f16_gemv_gate_up_applies(const void* scales, int64_t M, int64_t I, int64_t K) {
  if (M < 1 || M > 16 || I < 8 || I % 8 != 0 || I > 0x3fffffffLL / 32 || K < 256 || K % 256 != 0 || !scales || !aligned16(scales)) return 0;
  return options().gemv_variant != 1 && !weight_stationary_first(M, 2 * I, K, false);
}

int b200_q4f16_gemv_gate_up(const void* x, const void* delta, const void* norm_w, void* x_out, float eps, const void* wq,
                            const void* scales, void* act, int64_t M, int64_t I, int64_t K, void* stream) {
  const char* who = "q4f16_gemv_gate_up";
  if (I < 8 || I % 8 != 0 || I > 0x3fffffffLL / 32) return fail(B200_EINVAL, "%s: needs I a positive multiple of 8, got %lld", who, (long long)I);
  int rc = check_matmul(who, x, wq, scales, act, M, 2 * I, K);
  if (rc) return rc;
  if (M < 1 || M > 16) return fail(B200_EINVAL, "%s: takes 1 <= M <= 16, got %lld", who, (long long)M);
  if (K < 256 || K % 256 != 0) return fail(B200_EINVAL, "%s: needs K a positive multiple of 256", who);
  if (!aligned16(scales)) return fail(B200_EINVAL, "%s: scales must be 16-byte aligned", who);
  if (!norm_w && (delta || x_out)) return fail(B200_EINVAL, "%s: delta and x_out go with a norm weight", who);
  if (!aligned16(norm_w)) return fail(B200_EINVAL, "%s: norm weight must be 16-byte aligned", who);
  if ((delta && !aligned16(delta)) || (x_out && !aligned16(x_out))) return fail(B200_EINVAL, "%s: delta / x_out must be 16-byte aligned", who);
  if (x_out == x) return fail(B200_EINVAL, "%s: x_out must not alias x (other CTAs still read x)", who);
  rc = ensure_device();
  if (rc) return rc;
  rc = launch_gemv_pipe_gate_up(static_cast<const __half*>(x), static_cast<const __half*>(delta), static_cast<const __half*>(norm_w),
                                static_cast<__half*>(x_out), eps, nullptr, static_cast<const uint32_t*>(wq),
                                static_cast<const __half*>(scales), static_cast<__half*>(act), M, I, K,
                                static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(rc, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

// SwiGLU in the epilogue of the weight-stationary kernel, where the automatic dispatch gives the matmul to it and that is the faster way.
int b200_q4f16_gate_up_applies(const void* scales, int64_t M, int64_t I, int64_t K) {
  if (M < 1 || M > 128 || I < 1 || I > 0x3fffffffLL / 32 || K < 32 || K % 32 != 0 || !scales) return 0;
  const bool ragged = K % 256 != 0 || !aligned16(scales);
  return weight_stationary_first(M, 2 * I, K, ragged) && gemm_ws_gate_up_is_ahead(M, I, K, ragged);
}

int b200_q4f16_gate_up(const void* x, const void* wq, const void* scales, void* act, int64_t M, int64_t I, int64_t K, void* stream) {
  const char* who = "q4f16_gate_up";
  if (I < 1 || I > 0x3fffffffLL / 32) return fail(B200_EINVAL, "%s: needs I >= 1, got %lld", who, (long long)I);
  int rc = check_matmul(who, x, wq, scales, act, M, 2 * I, K);
  if (rc) return rc;
  if (M < 1 || M > 128 || K < 32) return fail(B200_EINVAL, "%s: takes 1 <= M <= 128 and K >= 32", who);
  if ((rc = ensure_device())) return rc;
  rc = launch_gemm_ws(static_cast<const __half*>(x), static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                      static_cast<__half*>(act), M, 2 * I, K, static_cast<cudaStream_t>(stream), true);
  if (rc == B200_ENOTREADY) return fail(rc, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

// ---- the residual stream with its statistics -------------------------------------------------------------------
// Common to the forms that normalise x by statistics left behind: up to eight rows.
static int check_norm_stats(const char* who, const void* stats, const void* norm_w, const void* scales, int64_t M, int64_t K) {
  if (M < 1 || M > 8) return fail(B200_EINVAL, "%s: takes 1 <= M <= 8, got %lld", who, (long long)M);
  if (K < 256 || K % 256 != 0) return fail(B200_EINVAL, "%s: needs K a positive multiple of 256", who);
  if (!aligned16(scales)) return fail(B200_EINVAL, "%s: scales must be 16-byte aligned", who);
  if (!norm_w || !aligned16(norm_w)) return fail(B200_EINVAL, "%s: norm weight must be non-null and 16-byte aligned", who);
  if (!stats || !aligned16(stats)) return fail(B200_EINVAL, "%s: statistics must be non-null and 16-byte aligned", who);
  return ensure_device();
}

int b200_q4f16_gemv_add_applies(const void* scales, int64_t M, int64_t N, int64_t K) {
  if (M < 1 || M > 8 || N < 16 || N % 16 != 0 || N > 0x7fffffffLL / 32 || K < 256 || K % 256 != 0 || !scales || !aligned16(scales)) return 0;
  return options().gemv_variant != 1 && !weight_stationary_first(M, N, K, false);
}

int b200_q4f16_gemv_add(const void* x, const void* wq, const void* scales, void* y, void* stats, int64_t M, int64_t N, int64_t K,
                        int32_t swiglu, void* stream) {
  const char* who = "q4f16_gemv_add";
  int rc = check_matmul(who, x, wq, scales, y, M, N, K);
  if (rc) return rc;
  if (M < 1 || M > 8) return fail(B200_EINVAL, "%s: takes 1 <= M <= 8, got %lld", who, (long long)M);
  if (N < 16 || N % 16 != 0 || K < 256 || K % 256 != 0)
    return fail(B200_EINVAL, "%s: needs N a positive multiple of 16 and K a positive multiple of 256", who);
  if (!aligned16(scales)) return fail(B200_EINVAL, "%s: scales must be 16-byte aligned", who);
  if (!stats || (reinterpret_cast<uintptr_t>(stats) & 3u)) return fail(B200_EINVAL, "%s: statistics must be non-null and 4-byte aligned", who);
  if (x == y) return fail(B200_EINVAL, "%s: y must not alias x (other CTAs still read x)", who);
  if ((rc = ensure_device())) return rc;
  rc = launch_gemv_pipe_add(static_cast<const __half*>(x), static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                            static_cast<__half*>(y), static_cast<float*>(stats), M, N, K, swiglu, static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(rc, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

int b200_q4f16_gemv_norm_applies(const void* scales, int64_t M, int64_t N, int64_t K) {
  if (M < 1 || M > 8 || N < 1 || N > 0x7fffffffLL / 32 || K < 256 || K % 256 != 0 || K > 0x3fffffffLL || !scales || !aligned16(scales)) return 0;
  return options().gemv_variant != 1 && !weight_stationary_first(M, N, K, false) && gemv_pipe_norm_fits(M, N, K);
}

int b200_q4f16_gemv_norm(const void* x, const void* stats, const void* norm_w, float eps, const void* wq, const void* scales, void* y,
                         int64_t M, int64_t N, int64_t K, void* stream) {
  const char* who = "q4f16_gemv_norm";
  int rc = check_matmul(who, x, wq, scales, y, M, N, K);
  if (rc) return rc;
  if (N < 1) return fail(B200_EINVAL, "%s: needs N >= 1", who);
  if ((rc = check_norm_stats(who, stats, norm_w, scales, M, K))) return rc;
  rc = launch_gemv_pipe_norm(static_cast<const __half*>(x), static_cast<const float*>(stats), static_cast<const __half*>(norm_w), eps,
                             static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales), static_cast<__half*>(y), M, N, K,
                             static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(rc, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

int b200_q4f16_gemv_norm_gate_up(const void* x, const void* stats, const void* norm_w, float eps, const void* wq, const void* scales,
                                 void* act, int64_t M, int64_t I, int64_t K, void* stream) {
  const char* who = "q4f16_gemv_norm_gate_up";
  if (I < 8 || I % 8 != 0 || I > 0x3fffffffLL / 32) return fail(B200_EINVAL, "%s: needs I a positive multiple of 8, got %lld", who, (long long)I);
  int rc = check_matmul(who, x, wq, scales, act, M, 2 * I, K);
  if (rc) return rc;
  if ((rc = check_norm_stats(who, stats, norm_w, scales, M, K))) return rc;
  rc = launch_gemv_pipe_gate_up(static_cast<const __half*>(x), nullptr, static_cast<const __half*>(norm_w), nullptr, eps,
                                static_cast<const float*>(stats), static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                                static_cast<__half*>(act), M, I, K, static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(rc, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

int b200_q4f16_gemv_norm_rope(const void* x, const void* stats, const void* norm_w, float eps, const void* wq, const void* scales,
                              const void* cos_t, const void* sin_t, const void* pos, void* q_out, void* k_cache, void* v_cache,
                              int64_t heads, int64_t K, void* stream) {
  const char* who = "q4f16_gemv_norm_rope";
  if (heads < 1 || heads > 4096) return fail(B200_EINVAL, "%s: heads %lld out of range", who, (long long)heads);
  int rc = check_matmul(who, x, wq, scales, q_out, 1, 3 * heads * 128, K);
  if (rc) return rc;
  if (!cos_t || !sin_t || !pos || !k_cache || !v_cache) return fail(B200_EINVAL, "%s: null table, position or cache pointer", who);
  if ((rc = check_norm_stats(who, stats, norm_w, scales, 1, K))) return rc;
  // B200_ENOTREADY (no message): the launch would not use the fast form; the caller runs b200_q4f16_gemv_norm and
  // b200_attn_decode_step instead
  return launch_gemv_pipe_rmsnorm_rope(static_cast<const __half*>(x), nullptr, static_cast<const __half*>(norm_w), nullptr, eps,
                                       static_cast<const float*>(stats), static_cast<const uint32_t*>(wq),
                                       static_cast<const __half*>(scales), static_cast<const float*>(cos_t),
                                       static_cast<const float*>(sin_t), static_cast<const int*>(pos), static_cast<__half*>(q_out),
                                       static_cast<__half*>(k_cache), static_cast<__half*>(v_cache), heads, K,
                                       static_cast<cudaStream_t>(stream));
}

int b200_q4f16_gemv_swiglu(const void* gu, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                           void* stream) {
  const char* who = "q4f16_gemv_swiglu";
  int rc = check_matmul(who, gu, wq, scales, y, M, N, K);
  if (rc) return rc;
  if (M < 1 || M > 16) return fail(B200_EINVAL, "%s: takes 1 <= M <= 16, got %lld", who, (long long)M);
  if (N < 1 || K < 256 || K % 256 != 0) return fail(B200_EINVAL, "%s: needs N >= 1 and K a positive multiple of 256", who);
  if (!aligned16(scales)) return fail(B200_EINVAL, "%s: scales must be 16-byte aligned", who);
  rc = ensure_device();
  if (rc) return rc;
  rc = launch_gemv_pipe_swiglu(static_cast<const __half*>(gu), static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                               static_cast<__half*>(y), M, N, K, static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(B200_EINVAL, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

int b200_q4f16_gemv_allreduce(const void* x, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                              int32_t swiglu, const B200PeerReduce* red, void* stream) {
  const char* who = "q4f16_gemv_allreduce";
  int rc = check_matmul(who, x, wq, scales, y, M, N, K);
  if (rc) return rc;
  if (M < 1 || M > 16) return fail(B200_EINVAL, "%s: takes 1 <= M <= 16, got %lld", who, (long long)M);
  if (N < 8 || N % 8 != 0 || K < 256 || K % 256 != 0)
    return fail(B200_EINVAL, "%s: needs N a positive multiple of 8 and K a positive multiple of 256", who);
  if (!aligned16(scales) || !aligned16(y)) return fail(B200_EINVAL, "%s: scales and y must be 16-byte aligned", who);
  if (!red) return fail(B200_EINVAL, "%s: null reduction descriptor", who);
  if (red->world < 1 || red->world > 8 || red->rank < 0 || red->rank >= red->world)
    return fail(B200_EINVAL, "%s: world %d / rank %d out of range (1..8)", who, red->world, red->rank);
  if (red->world > 1) {
    if (!red->epoch || !red->done_counter || !red->out || !aligned16(red->out) || red->flag_base < 0)
      return fail(B200_EINVAL, "%s: epoch, done_counter and a 16-byte aligned out are required", who);
    for (int r = 0; r < red->world; ++r)
      if (!red->peer_y[r] || !aligned16(red->peer_y[r]) || !red->peer_flags[r])
        return fail(B200_EINVAL, "%s: peer %d has a null or misaligned buffer", who, r);
    if (red->peer_y[red->rank] != y) return fail(B200_EINVAL, "%s: y must be this rank's entry of peer_y", who);
  }
  rc = ensure_device();
  if (rc) return rc;
  rc = launch_gemv_pipe_allreduce(static_cast<const __half*>(x), static_cast<const uint32_t*>(wq),
                                  static_cast<const __half*>(scales), static_cast<__half*>(y), M, N, K, swiglu, red,
                                  static_cast<cudaStream_t>(stream));
  if (rc == B200_ENOTREADY) return fail(B200_EINVAL, "%s: shape outside the fused kernel's domain", who);
  return rc;
}

int b200_allreduce_peer(int64_t count, const B200PeerReduce* red, void* stream) {
  const char* who = "allreduce_peer";
  if (count < 0 || count % 8 != 0) return fail(B200_EINVAL, "%s: count must be a non-negative multiple of 8, got %lld", who, (long long)count);
  if (!red) return fail(B200_EINVAL, "%s: null reduction descriptor", who);
  if (red->world < 2 || red->world > 8 || red->rank < 0 || red->rank >= red->world)
    return fail(B200_EINVAL, "%s: world %d / rank %d out of range (2..8)", who, red->world, red->rank);
  if (!red->epoch || !red->out || !aligned16(red->out) || red->flag_base < 0)
    return fail(B200_EINVAL, "%s: epoch and a 16-byte aligned out are required", who);
  for (int r = 0; r < red->world; ++r)
    if (!red->peer_y[r] || !aligned16(red->peer_y[r]) || !red->peer_flags[r])
      return fail(B200_EINVAL, "%s: peer %d has a null or misaligned buffer", who, r);
  int rc = ensure_device();
  if (rc) return rc;
  return launch_peer_allreduce(count, red, static_cast<cudaStream_t>(stream));
}

int b200_q4f16_gemm_ws(const void* x, const void* wq, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                       void* stream) {
  return matmul_impl(kGemmWs, "q4f16_gemm_ws", x, wq, scales, y, M, N, K, stream);
}

int b200_q4f16_matmul_host(const void* x_host, void* x_dev, const void* wq, const void* scales, void* y_dev,
                           void* y_host, int64_t M, int64_t N, int64_t K, void* stream) {
  if (M < 0 || N < 0 || K < 0) return fail(B200_EINVAL, "q4f16_matmul_host: negative size");
  if ((M * K > 0 && (!x_host || !x_dev)) || (M * N > 0 && (!y_host || !y_dev)))
    return fail(B200_EINVAL, "q4f16_matmul_host: null host or staging buffer");
  int rc = check_matmul("q4f16_matmul_host", x_dev, wq, scales, y_dev, M, N, K);
  if (rc) return rc;
  rc = ensure_device();
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  const size_t xb = (size_t)(M * K) * 2, yb = (size_t)(M * N) * 2;
  if (xb > 0) {
    void* xm = xb <= kHostKernelBytes && !(reinterpret_cast<uintptr_t>(x_host) & 15) ? mapped_host_pointer(x_host) : nullptr;
    if (xm) {
      if ((rc = host_copy(xm, x_dev, xb, s))) return rc;
    } else {
      e = cudaMemcpyAsync(x_dev, x_host, xb, cudaMemcpyHostToDevice, s);
      if (e != cudaSuccess) return fail(B200_ELAUNCH, "q4f16_matmul_host: H2D copy: %s", cudaGetErrorString(e));
    }
  }
  void* ym = yb > 0 && yb <= kHostKernelBytes && !(reinterpret_cast<uintptr_t>(y_host) & 15) ? mapped_host_pointer(y_host) : nullptr;
  if (ym && xb > 0 && options().gemv_variant != 1 && K % 256 == 0 && aligned16(scales) && !weight_stationary_first(M, N, K, false) &&
      host_direct(M, N, K, s)) {
    rc = launch_gemv_pipe_twice(static_cast<const __half*>(x_dev), static_cast<const uint32_t*>(wq), static_cast<const __half*>(scales),
                                static_cast<__half*>(y_dev), static_cast<__half*>(ym), M, N, K, s);
    if (rc != B200_ENOTREADY) return rc;
  }
  rc = matmul_impl(kAuto, "q4f16_matmul_host", x_dev, wq, scales, y_dev, M, N, K, stream);
  if (rc) return rc;
  if (yb > 0) {
    if (ym) {
      if ((rc = host_copy(y_dev, ym, yb, s))) return rc;
    } else {
      e = cudaMemcpyAsync(y_host, y_dev, yb, cudaMemcpyDeviceToHost, s);
      if (e != cudaSuccess) return fail(B200_ELAUNCH, "q4f16_matmul_host: D2H copy: %s", cudaGetErrorString(e));
    }
  }
  return B200_OK;
}

int b200_q4f16_matmul_dl(const B200DLTensor* x, const B200DLTensor* wq, const B200DLTensor* scales, B200DLTensor* y) {
  return b200_q4f16_matmul_dl_family(x, wq, scales, y, B200_FAMILY_AUTO);
}

int b200_q4f16_matmul_dl_family(const B200DLTensor* x, const B200DLTensor* wq, const B200DLTensor* scales, B200DLTensor* y,
                                int32_t family) {
  const char* who = "b200.q4f16_matmul";
  int dev = -1, rc;
  // bits 0-7: kernel family; bits 8-15: weight layout + 1 (0 = the process-wide option)
  const int32_t layout_code = (family >> 8) & 0xff;
  if ((family & ~0xffff) != 0 || layout_code > 2)
    return fail(B200_EINVAL, "%s: malformed family/layout code 0x%x", who, (unsigned)family);
  family &= 0xff;
  if (family != B200_FAMILY_AUTO && family != B200_FAMILY_GEMV && family != B200_FAMILY_GEMM)
    return fail(B200_EINVAL, "%s: unknown kernel family %d (0 auto, 1 skinny, 2 tensor-core)", who, (int)family);
  LayoutScope scope(layout_code - 1);
  if ((rc = check_tensor(who, "x", x, 2, 16, &dev))) return rc;
  if ((rc = check_tensor(who, "wq", wq, 1, 32, &dev))) return rc;
  if ((rc = check_tensor(who, "scales", scales, 2, 16, &dev))) return rc;
  if ((rc = check_tensor(who, "y", y, 2, 16, &dev))) return rc;
  int64_t M = x->shape[0], K = x->shape[1], N = wq->shape[0];
  if (K % 32 != 0) return fail(B200_EINVAL, "%s: K=%lld is not a multiple of the group size 32", who, (long long)K);
  if (wq->shape[1] != K / 8)
    return fail(B200_EINVAL, "%s: wq is [%lld,%lld], expected [N,%lld] for K=%lld", who, (long long)wq->shape[0],
                (long long)wq->shape[1], (long long)(K / 8), (long long)K);
  if (scales->shape[0] != N || scales->shape[1] != K / 32)
    return fail(B200_EINVAL, "%s: scales is [%lld,%lld], expected [%lld,%lld]", who, (long long)scales->shape[0],
                (long long)scales->shape[1], (long long)N, (long long)(K / 32));
  if (y->shape[0] != M || y->shape[1] != N)
    return fail(B200_EINVAL, "%s: y is [%lld,%lld], expected [%lld,%lld]", who, (long long)y->shape[0],
                (long long)y->shape[1], (long long)M, (long long)N);
  if ((rc = check_current_device(who, dev))) return rc;
  const Family fam = family == B200_FAMILY_GEMV ? kGemv : family == B200_FAMILY_GEMM ? kGemm : kAuto;
  return matmul_impl(fam, who, data_ptr(x), data_ptr(wq), data_ptr(scales), data_ptr(y), M, N, K, g_stream);
}

int b200_q4f16_dequantize_dl(const B200DLTensor* wq, const B200DLTensor* scales, B200DLTensor* w_out) {
  const char* who = "b200.q4f16_dequantize";
  int dev = -1, rc;
  if ((rc = check_tensor(who, "wq", wq, 1, 32, &dev))) return rc;
  if ((rc = check_tensor(who, "scales", scales, 2, 16, &dev))) return rc;
  if ((rc = check_tensor(who, "w", w_out, 2, 16, &dev))) return rc;
  int64_t N = wq->shape[0], K = wq->shape[1] * 8;
  if (K % 32 != 0) return fail(B200_EINVAL, "%s: K=%lld is not a multiple of the group size 32", who, (long long)K);
  if (scales->shape[0] != N || scales->shape[1] != K / 32)
    return fail(B200_EINVAL, "%s: scales is [%lld,%lld], expected [%lld,%lld]", who, (long long)scales->shape[0],
                (long long)scales->shape[1], (long long)N, (long long)(K / 32));
  if (w_out->shape[0] != N || w_out->shape[1] != K)
    return fail(B200_EINVAL, "%s: output is [%lld,%lld], expected [%lld,%lld]", who, (long long)w_out->shape[0],
                (long long)w_out->shape[1], (long long)N, (long long)K);
  if ((rc = check_current_device(who, dev))) return rc;
  return b200_q4f16_dequantize(data_ptr(wq), data_ptr(scales), data_ptr(w_out), N, K, g_stream);
}

// ---- packed-function symbols (legacy TVM C backend ABI) ------------------------------------
// TVMValue is an 8-byte union; tensors come as v_handle with type code 7 or 13.
static int packed_tensors(const char* who, void* args, int* type_codes, int num_args, int want,
                          const B200DLTensor** out) {
  if (num_args != want) return fail(B200_EINVAL, "%s: expected %d arguments, got %d", who, want, num_args);
  if (!args || !type_codes) return fail(B200_EINVAL, "%s: null argument array", who);
  void** vals = static_cast<void**>(args);
  for (int i = 0; i < want; ++i) {
    if (type_codes[i] != 7 && type_codes[i] != 13)
      return fail(B200_EINVAL, "%s: argument %d has type code %d, expected a tensor (7 or 13)", who, i, type_codes[i]);
    out[i] = static_cast<const B200DLTensor*>(vals[i]);
  }
  return B200_OK;
}

int32_t b200_q4f16_matmul_packed(void* args, int* type_codes, int num_args, void* out_value, int* out_type_code,
                                 void* resource_handle) {
  (void)out_value; (void)resource_handle;
  const B200DLTensor* t[4];
  if (packed_tensors("b200.q4f16_matmul", args, type_codes, num_args, 4, t)) return -1;
  if (b200_q4f16_matmul_dl(t[0], t[1], t[2], const_cast<B200DLTensor*>(t[3]))) return -1;
  if (out_type_code) *out_type_code = 4;  // kTVMNullptr: DPS functions return nothing
  return 0;
}

int32_t b200_q4f16_dequantize_packed(void* args, int* type_codes, int num_args, void* out_value, int* out_type_code,
                                     void* resource_handle) {
  (void)out_value; (void)resource_handle;
  const B200DLTensor* t[3];
  if (packed_tensors("b200.q4f16_dequantize", args, type_codes, num_args, 3, t)) return -1;
  if (b200_q4f16_dequantize_dl(t[0], t[1], const_cast<B200DLTensor*>(t[2]))) return -1;
  if (out_type_code) *out_type_code = 4;
  return 0;
}

}  // extern "C"
