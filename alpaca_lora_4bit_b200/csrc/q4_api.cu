// Error plumbing and version query of the q4b200 C ABI.
#include <stdarg.h>
#include <string.h>

#include "q4_common.cuh"

namespace q4 {

char* err_buf() {
  static thread_local char buf[512] = "";
  return buf;
}

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(err_buf(), 512, fmt, ap);
  va_end(ap);
  return code;
}

int check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return Q4_OK;
  return fail(Q4_E_CUDA, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

int check_device() {
  static int ok[64] = {0};      // 0 unknown, 1 ok, -1 bad
  int dev = 0;
  if (int e = check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return e;
  if (dev >= 0 && dev < 64 && ok[dev] == 1) return Q4_OK;
  int major = 0, minor = 0;
  if (int e = check_cuda(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev), "device attribute")) return e;
  if (int e = check_cuda(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev), "device attribute")) return e;
  if (major != 10) return fail(Q4_E_DEVICE, "device %d is sm_%d%d; this library is built for sm_100a only", dev, major, minor);
  if (dev >= 0 && dev < 64) ok[dev] = 1;
  return Q4_OK;
}

}  // namespace q4

extern "C" int q4_version(void) { return Q4_VERSION; }
extern "C" const char* q4_last_error_string(void) { return q4::err_buf(); }

// ---- tensor-map encoding through the driver entry point (no link-time dependency on libcuda) ----
#include "q4_async.cuh"

namespace q4 {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = (EncodeTiledFn)p;
  return fn;
}

int make_tmap_2d(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t cols,
                 uint64_t rows, uint64_t row_pitch_bytes, uint32_t box_cols, uint32_t box_rows,
                 CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(Q4_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  if (!aligned16(base) || row_pitch_bytes % 16 || (uint64_t)box_cols * elem_bytes % 16)
    return fail(Q4_E_ALIGN, "tensor map: base, row pitch and box width must be multiples of 16 bytes");
  int dev = 0;
  if (int e = check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return e;
  // A descriptor depends only on the address and the geometry, not on the bytes behind it, and a
  // decode step asks for the same few hundred descriptors token after token: keep the last ones
  // of this thread (direct-mapped, keyed by everything that goes into the descriptor).
  struct Entry { const void* base; uint64_t cols, rows, pitch; uint32_t box_cols, box_rows; int dt, swizzle, dev, valid; CUtensorMap map; };
  constexpr int SLOTS = 512;
  static thread_local Entry cache[SLOTS];
  const size_t h = ((reinterpret_cast<uintptr_t>(base) >> 8) * 0x9E3779B97F4A7C15ull + cols * 31 + rows * 17 + box_rows) % SLOTS;
  Entry& e = cache[h];
  if (e.valid && e.base == base && e.cols == cols && e.rows == rows && e.pitch == row_pitch_bytes && e.box_cols == box_cols &&
      e.box_rows == box_rows && e.dt == (int)dt && e.swizzle == (int)swizzle && e.dev == dev) {
    *out = e.map;
    return Q4_OK;
  }
  // The driver call needs this thread to have a current context; a thread that has only inherited
  // the device setting (an autograd worker, say) binds the primary context with cudaSetDevice.
  if (int err = check_cuda(cudaSetDevice(dev), "cudaSetDevice")) return err;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {row_pitch_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(Q4_E_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  e.base = base; e.cols = cols; e.rows = rows; e.pitch = row_pitch_bytes; e.box_cols = box_cols; e.box_rows = box_rows;
  e.dt = (int)dt; e.swizzle = (int)swizzle; e.dev = dev; e.map = *out; e.valid = 1;
  return Q4_OK;
}

int sm_count() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev] > 0 ? n[dev] : 148;
}

}  // namespace q4

namespace q4 {
// The head of a workspace as a node of a captured graph.  Programmatic on both sides, so that the product behind it is launched
// meanwhile: every kernel that takes a workspace waits for the earlier kernel before it touches it.
__global__ void __launch_bounds__(256) clear_kernel(uint4* p, int n) {
  pdl_launch_dependents();
  pdl_wait();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) p[i] = make_uint4(0, 0, 0, 0);
}
}  // namespace q4

extern "C" int q4_clear(void* p, size_t bytes, q4_stream_t stream) {
  using namespace q4;
  if (!p) return fail(Q4_E_BADARG, "clear: null pointer");
  if (!aligned16(p) || bytes % 16 || bytes > (1u << 30)) return fail(Q4_E_ALIGN, "clear: %zu bytes, a multiple of 16 on a 16-byte boundary", bytes);
  if (bytes == 0) return Q4_OK;
  if (int e = check_device()) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(bytes < (32u << 12) ? (unsigned)((bytes + 4095) >> 12) : 32); cfg.blockDim = dim3(256); cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&cfg, clear_kernel, (uint4*)p, (int)(bytes / 16)), "clear launch");
}

extern "C" int q4_capture_id(q4_stream_t stream, unsigned long long* out) {
  using namespace q4;
  if (!out) return fail(Q4_E_BADARG, "capture_id: null pointer");
  cudaStreamCaptureStatus status;
  unsigned long long id = 0;
  if (int e = check_cuda(cudaStreamGetCaptureInfo((cudaStream_t)stream, &status, &id), "capture_id")) return e;
  *out = status == cudaStreamCaptureStatusActive ? id : 0;
  return Q4_OK;
}

