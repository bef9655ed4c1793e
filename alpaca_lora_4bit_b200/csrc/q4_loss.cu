// The loss of a causal language model over 16-bit logits: cross entropy in fp32, forward and backward, without the fp32
// copy of the logits that the framework makes (`logits.float()`, log-softmax, negative log-likelihood).
//
// Bound by HBM and the exponentials: the forward reads the logits once and, where a gradient may be asked for, writes the copy
// that the backward reads (the caller may write to its own before then); the backward reads that and writes the gradient.
// The framework's kernels move 24 bytes an element instead of 8: at 1024 x 32000 fp16 the casts took 93 us, log-softmax 71
// and its backward 110, the two kernels of the likelihood 31; here 24 and 20 us and 2 for the mean (20 and 20 at the rate of a
// copy; 22 and 22 when the forward wrote nothing and the backward read the caller's logits).  A CTA of 256 threads per row, so that four rows on an SM cover each other's loads and reductions (512 threads:
// 30 us); a thread keeps a running maximum and the sum of exponentials relative to it, so a row of any length is read once,
// and all sums are added in a fixed order.
#include <cuda_bf16.h>
#include "q4_common.cuh"

namespace q4 {

constexpr int CE_THREADS = 256, CE_BATCH = 4;
constexpr float LOG2E = 1.4426950408889634f;
template <bool BF16>
constexpr uint32_t CE_NONE = BF16 ? 0xFF80FF80u : 0xFC00FC00u;           // two -inf

template <bool BF16>
__device__ __forceinline__ float2 ce_pair(uint32_t v) {
  if (BF16) return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
  return __half22float2(as_h2(v));
}
template <bool BF16>
__device__ __forceinline__ uint32_t ce_pack(float a, float b) {
  if (BF16) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  return as_u32(__floats2half2_rn(a, b));
}
template <bool BF16>
__device__ __forceinline__ float ce_one(const uint16_t* p) {
  return BF16 ? __uint_as_float((uint32_t)*p << 16) : __half2float(*reinterpret_cast<const __half*>(p));
}

// The class of a row: its own label or, for rows of `seq` tokens each, the next token's (the last has none).
__device__ __forceinline__ long long ce_label(const long long* labels, int row, int seq, long long ignore) {
  if (seq == 0) return labels[row];
  return row % seq + 1 < seq ? labels[row + 1] : ignore;
}

// Sums relative to two maxima as one; -inf (nothing seen, or only -inf) adds nothing.
__device__ __forceinline__ void ce_merge(float& m, float& s, float m2, float s2) {
  const float mm = fmaxf(m, m2);
  s = (m == -INFINITY ? 0.f : s * expf(m - mm)) + (m2 == -INFINITY ? 0.f : s2 * expf(m2 - mm));
  m = mm;
}

template <bool BF16>
__global__ void __launch_bounds__(CE_THREADS, 4)
ce_fwd_kernel(const uint16_t* __restrict__ logits, const long long* __restrict__ labels, float2* __restrict__ stats, float* __restrict__ row_loss,
              uint16_t* __restrict__ kept, long long* __restrict__ classes, int V, int seq, long long ignore) {
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint4* src = reinterpret_cast<const uint4*>(logits + (size_t)row * V);
  uint4* copy = reinterpret_cast<uint4*>(kept + (size_t)row * V);          // (a null `kept`: never written)
  // four vectors at a time, the next four on their way meanwhile: one rescaling for 32 elements
  uint4 v[CE_BATCH];
  auto fetch = [&](int i0) __attribute__((always_inline)) {
#pragma unroll
    for (int j = 0; j < CE_BATCH; ++j) {
      const int i = i0 + j * CE_THREADS;
      v[j] = i < V / 8 ? ldg_stream(src + i) : make_uint4(CE_NONE<BF16>, CE_NONE<BF16>, CE_NONE<BF16>, CE_NONE<BF16>);
    }
  };
  fetch(threadIdx.x);
  const long long label = ce_label(labels, row, seq, ignore);
  if (classes && threadIdx.x == 0) classes[row] = label;
  if (label == ignore) {
    if (threadIdx.x == 0) row_loss[row] = 0.f;
    if (kept)
      for (int i = threadIdx.x; i < V / 8; i += CE_THREADS) copy[i] = src[i];
    return;
  }
  const bool known = label >= 0 && label < V;
  const float at_label = known ? ce_one<BF16>(logits + (size_t)row * V + label) : NAN;
  float m = -INFINITY, s = 0.f;
  bool bad = false;
#pragma unroll 1
  for (int i0 = threadIdx.x; i0 < V / 8; i0 += CE_BATCH * CE_THREADS) {
    uint32_t w[4 * CE_BATCH];
#pragma unroll
    for (int j = 0; j < CE_BATCH; ++j) { w[4 * j] = v[j].x; w[4 * j + 1] = v[j].y; w[4 * j + 2] = v[j].z; w[4 * j + 3] = v[j].w; }
    if (kept) {
#pragma unroll
      for (int j = 0; j < CE_BATCH; ++j)
        if (i0 + j * CE_THREADS < V / 8) copy[i0 + j * CE_THREADS] = v[j];
    }
    fetch(i0 + CE_BATCH * CE_THREADS);
    float top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int e = 0; e < 4 * CE_BATCH; ++e) {
      const float2 x = ce_pair<BF16>(w[e]);
      top = fmaxf(top, fmaxf(x.x, x.y));
      bad |= x.x != x.x || x.y != x.y;                     // (the maximum passes a NaN over)
    }
    if (top > m) {
      s = m == -INFINITY ? 0.f : s * expf(m - top);
      m = top;
    }
    if (m == -INFINITY) continue;
#pragma unroll
    for (int e = 0; e < 4 * CE_BATCH; ++e) {
      // (the difference first: a product m log2(e) is rounded at the size of the logits)
      const float2 x = ce_pair<BF16>(w[e]);
      sum += exp2f((x.x - m) * LOG2E) + exp2f((x.y - m) * LOG2E);
    }
    s += sum;
  }
  if (bad) s = NAN;
  __shared__ float2 red[CE_THREADS / 32];
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) ce_merge(m, s, __shfl_xor_sync(0xffffffffu, m, d), __shfl_xor_sync(0xffffffffu, s, d));
  if (lane == 0) red[warp] = make_float2(bad ? NAN : m, s);
  const int any_bad = __syncthreads_or(bad);
  if (warp != 0) return;
  m = lane < CE_THREADS / 32 ? red[lane].x : -INFINITY;
  s = lane < CE_THREADS / 32 ? red[lane].y : 0.f;
#pragma unroll
  for (int d = CE_THREADS / 64; d >= 1; d >>= 1) ce_merge(m, s, __shfl_xor_sync(0xffffffffu, m, d), __shfl_xor_sync(0xffffffffu, s, d));
  if (lane == 0) {
    if (any_bad || !known) m = s = NAN;
    const float ls = logf(s);
    stats[row] = make_float2(m, ls);
    row_loss[row] = ls - (at_label - m);
  }
}

// The mean loss of the rows that have a class, and their number
__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ row_loss, const long long* __restrict__ labels, float* __restrict__ loss, float* __restrict__ count, int rows,
               int seq, long long ignore) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float s = 0.f;
  int n = 0;
  for (int r = threadIdx.x; r < rows; r += 1024) { s += row_loss[r]; n += ce_label(labels, r, seq, ignore) != ignore; }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) { s += __shfl_xor_sync(0xffffffffu, s, d); n += __shfl_xor_sync(0xffffffffu, n, d); }
  __shared__ float rs[32];
  __shared__ int rn[32];
  if (lane == 0) { rs[warp] = s; rn[warp] = n; }
  __syncthreads();
  if (threadIdx.x == 0) {
    s = 0.f; n = 0;
    for (int w = 0; w < 32; ++w) { s += rs[w]; n += rn[w]; }
    *loss = s / (float)n;
    *count = (float)n;
  }
}

// grad = (softmax - one at the class) * grad_loss / number of rows that have one, zero for the others
template <bool BF16>
__global__ void __launch_bounds__(CE_THREADS)
ce_bwd_kernel(const uint16_t* __restrict__ logits, const long long* __restrict__ labels, const float2* __restrict__ stats,
              const float* __restrict__ grad_loss, const float* __restrict__ count, uint16_t* __restrict__ grad, int V, int seq, long long ignore) {
  const int row = blockIdx.x;
  const long long label = ce_label(labels, row, seq, ignore);
  const uint4* src = reinterpret_cast<const uint4*>(logits + (size_t)row * V);
  uint4* dst = reinterpret_cast<uint4*>(grad + (size_t)row * V);
  if (label == ignore) {
    for (int i = threadIdx.x; i < V / 8; i += CE_THREADS) dst[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  const float g = *grad_loss / *count;
  const float2 st = stats[row];
  const int at = (int)(label >> 3), which = (int)(label & 7);
#pragma unroll 4
  for (int i = threadIdx.x; i < V / 8; i += CE_THREADS) {
    const uint4 v = ldg_stream(src + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = ce_pair<BF16>(w[e]);
      const float la = (x.x - st.x) - st.y, lb = (x.y - st.x) - st.y;
      float a = exp2f(la * LOG2E), b = exp2f(lb * LOG2E);
      if (i == at) {                                       // softmax - 1, also where it is next to nothing
        if (which == 2 * e) a = expm1f(la);
        if (which == 2 * e + 1) b = expm1f(lb);
      }
      o[e] = ce_pack<BF16>(a * g, b * g);
    }
    dst[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

static int ce_check(const void* logits, int rows, int V, int seq, const char* what) {
  if (rows <= 0 || V <= 0 || seq < 0) return fail(Q4_E_BADARG, "%s: rows=%d V=%d seq=%d", what, rows, V, seq);
  if (V % 8 || (seq > 0 && rows % seq)) return fail(Q4_E_SHAPE, "%s: V=%d must be a multiple of 8 and %d rows whole sequences of %d", what, V, rows, seq);
  if (!aligned16(logits)) return fail(Q4_E_ALIGN, "%s: logits must be 16-byte aligned", what);
  return check_device();
}

}  // namespace q4

using namespace q4;

extern "C" int q4_causal_loss_fwd(const void* logits, const long long* labels, float* stats, float* row_loss, float* loss, float* count, int rows,
                                  int V, int seq, long long ignore, int bf16, q4_stream_t stream) {
  return q4_causal_loss_fwd_keep(logits, labels, stats, row_loss, loss, count, nullptr, nullptr, rows, V, seq, ignore, bf16, stream);
}

extern "C" int q4_causal_loss_fwd_keep(const void* logits, const long long* labels, float* stats, float* row_loss, float* loss, float* count,
                                       void* kept, long long* classes, int rows, int V, int seq, long long ignore, int bf16, q4_stream_t stream) {
  if (!logits || !labels || !stats || !row_loss || !loss || !count) return fail(Q4_E_BADARG, "causal_loss: null pointer");
  if (int e = ce_check(logits, rows, V, seq, "causal_loss")) return e;
  if (!aligned16(kept)) return fail(Q4_E_ALIGN, "causal_loss: the copy of the logits must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  if (bf16) ce_fwd_kernel<true><<<rows, CE_THREADS, 0, st>>>((const uint16_t*)logits, labels, (float2*)stats, row_loss, (uint16_t*)kept, classes, V, seq, ignore);
  else ce_fwd_kernel<false><<<rows, CE_THREADS, 0, st>>>((const uint16_t*)logits, labels, (float2*)stats, row_loss, (uint16_t*)kept, classes, V, seq, ignore);
  ce_mean_kernel<<<1, 1024, 0, st>>>(row_loss, labels, loss, count, rows, seq, ignore);
  return check_cuda(cudaGetLastError(), "causal_loss launch");
}

extern "C" int q4_causal_loss_bwd(const void* logits, const long long* labels, const float* stats, const float* grad_loss, const float* count,
                                  void* grad, int rows, int V, int seq, long long ignore, int bf16, q4_stream_t stream) {
  if (!logits || !labels || !stats || !grad_loss || !count || !grad) return fail(Q4_E_BADARG, "causal_loss_bwd: null pointer");
  if (int e = ce_check(logits, rows, V, seq, "causal_loss_bwd")) return e;
  if (!aligned16(grad)) return fail(Q4_E_ALIGN, "causal_loss_bwd: the gradient must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  if (bf16) ce_bwd_kernel<true><<<rows, CE_THREADS, 0, st>>>((const uint16_t*)logits, labels, (const float2*)stats, grad_loss, count, (uint16_t*)grad, V, seq, ignore);
  else ce_bwd_kernel<false><<<rows, CE_THREADS, 0, st>>>((const uint16_t*)logits, labels, (const float2*)stats, grad_loss, count, (uint16_t*)grad, V, seq, ignore);
  return check_cuda(cudaGetLastError(), "causal_loss_bwd launch");
}
