// predictor_kernels.cu -- kernels of the early-termination network.
//
// The network (a strided temporal convolution stack and an MLP, see
// openems_b200/predictor_net.py) runs forward and backward on these kernels:
// every matrix product goes through the tcgen05 BF16 GEMM (gemm_tc.cuh) with
// f32 accumulation; activations are kept as f32 (B, T, C) row-major with bf16
// copies for the GEMM operands; weights are f32 masters with bf16 copies.
// All entry points take device pointers and a CUDA stream (NULL = default)
// and return an oems_status; what they allocate is the error word (once per
// device) and, for split reductions, stream-ordered workspace from the
// device's pool.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "../../include/oems.h"
#include "../../include/oems_predictor.h"
#include "gemm_tc.cuh"

namespace oems {
extern thread_local std::string g_last_error;
// stream-ordered memory of the current device's pool, kept for reuse until
// oems_release_cached_memory (engine.cu)
cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t s);
}

namespace {

oems_status pfail(oems_status st, const std::string& m) {
  oems::g_last_error = m;
  return st;
}

#define PK_CUDA(x)                                                              \
  do {                                                                          \
    cudaError_t e_ = (x);                                                       \
    if (e_ != cudaSuccess) return pfail(OEMS_ERR_CUDA, cudaGetErrorString(e_)); \
  } while (0)

int* g_err[64] = {nullptr};

oems_status err_word(int** out) {
  int dev = 0;
  PK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return pfail(OEMS_ERR_CUDA, "device index out of range");
  if (!g_err[dev]) {
    PK_CUDA(cudaMalloc(&g_err[dev], sizeof(int)));
    PK_CUDA(cudaMemset(g_err[dev], 0, sizeof(int)));
  }
  *out = g_err[dev];
  return OEMS_OK;
}

// Stream-ordered workspace of one call.  get: false where it is not to be
// had, and the call takes the form that needs none.
struct Workspace {
  void* p = nullptr;
  cudaStream_t s;
  explicit Workspace(void* stream) : s(reinterpret_cast<cudaStream_t>(stream)) {}
  bool get(size_t bytes) {
    if (oems::pool_alloc(&p, bytes, s) == cudaSuccess) return true;
    cudaGetLastError();
    p = nullptr;
    return false;
  }
  ~Workspace() {
    if (p) cudaFreeAsync(p, s);
  }
};

inline bool aligned16(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library)
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

oems_status encode_fn(EncodeTiled* out) {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(f);
  });
  if (!fn) return pfail(OEMS_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  *out = fn;
  return OEMS_OK;
}

// Tensor map of a row-major bf16 matrix [rows, k] with row pitch ld
// elements: boxes of 64 K-elements (128 bytes, the swizzle span) x box_rows
// rows, 128-byte swizzle, zero fill outside the matrix.
oems_status bf16_map(EncodeTiled enc, CUtensorMap* m, const void* ptr, int ld, int k, int rows, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return pfail(OEMS_ERR_CUDA, "GEMM: cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return OEMS_OK;
}

template <int BN>
cudaError_t launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const oems::GemmArgs& p, int grid, void* stream) {
  const size_t smem = oems::GemmCfg<BN>::smem;
  cudaError_t e = cudaFuncSetAttribute(oems::k_gemm_tc<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  oems::k_gemm_tc<BN><<<grid, 192, smem, S(stream)>>>(ta, tb, p);
  return cudaGetLastError();
}
inline int blocks(long long n, int t) { return (int)((n + t - 1) / t); }
inline int grid_for(long long n, int cap) { return std::max(1, std::min(blocks(n, 256), cap)); }

__global__ void k_f32_to_bf16(const float* x, __nv_bfloat16* y, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16_rn(x[i]);
}

// y[c * ldy + r] = x[r * ldx + c] for r < R, c < C (bf16), through a 32 x 32 tile
__global__ void k_transpose_bf16(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy, int R, int C) {
  __shared__ __nv_bfloat16 t[32][33];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    if (r < R && c < C) t[i][threadIdx.x] = x[(size_t)r * ldx + c];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (r < R && c < C) y[(size_t)c * ldy + r] = t[threadIdx.x][i];
  }
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// The transpose for pitches and sizes that are multiples of 8: 64 x 64 tiles,
// 16-byte loads and stores (the 2-byte form moves 64-byte rows at 1.4 TB/s;
// 65536 x 640: 21 -> 9 us an average launch of the network's shapes).
__global__ void __launch_bounds__(256) k_transpose_bf16_8(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy,
                                                          int R, int C) {
  __shared__ __nv_bfloat16 t[64][66];
  const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = (threadIdx.x >> 3) + 32 * h, c = (threadIdx.x & 7) * 8;
    if (r0 + i < R && c0 + c < C) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(x + (size_t)(r0 + i) * ldx + c0 + c));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) *reinterpret_cast<uint32_t*>(&t[i][c + 2 * u]) = w[u];
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = (threadIdx.x >> 3) + 32 * h, r = (threadIdx.x & 7) * 8;
    if (c0 + c < C && r0 + r < R) {
      uint32_t w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        w[u] = (uint32_t)__bfloat16_as_ushort(t[r + 2 * u][c]) | (uint32_t)__bfloat16_as_ushort(t[r + 2 * u + 1][c]) << 16;
      *reinterpret_cast<uint4*>(y + (size_t)(c0 + c) * ldy + r0 + r) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// cols[(b, t), k * C + c] = x[b, t * s + k, c]  (bf16, row pitch ldc)
__global__ void k_im2col(const float* x, __nv_bfloat16* cols, int B, int T, int C, int ks, int s, int Tout,
                         int ldc) {
  const long long n = (long long)B * Tout * ks * C;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    long long r = i / C;
    const int k = (int)(r % ks);
    r /= ks;
    const int t = (int)(r % Tout);
    const int b = (int)(r / Tout);
    cols[((long long)b * Tout + t) * ldc + (long long)k * C + c] =
        __float2bfloat16_rn(x[((long long)b * T + (long long)t * s + k) * C + c]);
  }
}

// dx[b, tau, c] = sum over (t, k) with t * s + k = tau of dcols[(b, t), k * C + c]
__global__ void k_col2im(const float* dcols, int ldc, float* dx, int B, int T, int C, int ks, int s, int Tout) {
  const long long n = (long long)B * T * C;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const long long r = i / C;
    const int tau = (int)(r % T);
    const int b = (int)(r / T);
    float acc = 0.f;
    for (int k = 0; k < ks; ++k) {
      const int u = tau - k;
      if (u < 0 || u % s) continue;
      const int t = u / s;
      if (t >= Tout) continue;
      acc += dcols[((long long)b * Tout + t) * ldc + (long long)k * C + c];
    }
    dx[i] = acc;
  }
}

// Causal dilated im2col: output length T; row (b, t) holds, at k C + c,
// x[b, t - (ks - 1 - k) dil, c] (0 before the start), so tap ks - 1 is the
// current step and the others reach back by multiples of the dilation.
__global__ void k_im2col_causal(const float* x, __nv_bfloat16* cols, int B, int T, int C, int ks, int dil, int ldc) {
  const long long n = (long long)B * T * ks * C;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    long long r = i / C;
    const int k = (int)(r % ks);
    r /= ks;
    const int t = (int)(r % T);
    const int b = (int)(r / T);
    const int u = t - (ks - 1 - k) * dil;
    const float v = u >= 0 ? x[((long long)b * T + u) * C + c] : 0.0f;
    cols[((long long)b * T + t) * ldc + (long long)k * C + c] = __float2bfloat16_rn(v);
  }
}

// The same for C and ldc multiples of 8 and 16-byte bases: 8 channels a
// thread (two 16-byte loads, one 16-byte store, one division chain where the
// general form has eight): 256 x 256 x 128 channels, 5 taps: 200 -> 25 us.
__global__ void __launch_bounds__(256) k_im2col_causal8(const float* x, __nv_bfloat16* cols, long long rows, int T,
                                                        int C, int ks, int dil, int ldc) {
  const int per = ks * (C >> 3);  // 8-channel groups of a row
  const long long n = rows * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / per;
    const int g = (int)(i - row * per), k = g / (C >> 3), c = (g - k * (C >> 3)) * 8;
    const int back = (ks - 1 - k) * dil, t = (int)(row % T);
    uint4 o = make_uint4(0, 0, 0, 0);
    if (t >= back) {
      const float4* s = reinterpret_cast<const float4*>(x + (row - back) * C + c);
      const float4 a = __ldg(s), b = __ldg(s + 1);
      o = make_uint4(bf16x2(a.x, a.y), bf16x2(a.z, a.w), bf16x2(b.x, b.y), bf16x2(b.z, b.w));
    }
    *reinterpret_cast<uint4*>(cols + row * ldc + (long long)k * C + c) = o;
  }
}

// Adjoint: dx[b, tau, c] = sum over k of dcols[(b, tau + (ks - 1 - k) dil), k C + c]
// (terms past the end dropped), summed in k order.
__global__ void k_col2im_causal(const float* dcols, int ldc, float* dx, int B, int T, int C, int ks, int dil) {
  const long long n = (long long)B * T * C;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const long long r = i / C;
    const int tau = (int)(r % T);
    const int b = (int)(r / T);
    float acc = 0.f;
    for (int k = 0; k < ks; ++k) {
      const int t = tau + (ks - 1 - k) * dil;
      if (t >= T) continue;
      acc += dcols[((long long)b * T + t) * ldc + (long long)k * C + c];
    }
    dx[i] = acc;
  }
}

// The same for C and ldc multiples of 4 and 16-byte bases, 4 channels a thread.
__global__ void __launch_bounds__(256) k_col2im_causal4(const float* dcols, int ldc, float* dx, long long rows, int T,
                                                        int C, int ks, int dil) {
  const int per = C >> 2;
  const long long n = rows * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / per;
    const int c = (int)(i - row * per) * 4, tau = (int)(row % T);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < ks; ++k) {
      const int on = (ks - 1 - k) * dil;
      if (tau + on >= T) continue;
      const float4 v = __ldcs(reinterpret_cast<const float4*>(dcols + (row + on) * ldc + (long long)k * C + c));
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
    *reinterpret_cast<float4*>(dx + row * C + c) = acc;
  }
}

// y = max(x, 0) in place, with a bf16 copy of y (pitch ldb, rows of width w)
__global__ void k_relu(float* x, __nv_bfloat16* xb, long long rows, int w, int ldb) {
  const long long n = rows * w;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = fmaxf(x[i], 0.f);
    x[i] = v;
    if (xb) xb[(i / w) * ldb + i % w] = __float2bfloat16_rn(v);
  }
}

// The same for widths and pitches that are multiples of 4, with a bf16 copy.
__global__ void __launch_bounds__(256) k_relu4(float* x, __nv_bfloat16* xb, long long rows, int w, int ldb) {
  const int per = w >> 2;
  const long long n = rows * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float4 v = reinterpret_cast<float4*>(x)[i];
    v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
    reinterpret_cast<float4*>(x)[i] = v;
    const long long row = i / per;
    *reinterpret_cast<uint2*>(xb + row * ldb + (i - row * per) * 4) = make_uint2(bf16x2(v.x, v.y), bf16x2(v.z, v.w));
  }
}

// dy *= (y > 0)
__global__ void k_relu_bwd(float* dy, const float* y, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (!(y[i] > 0.f)) dy[i] = 0.f;
}

// db[c] = sum_r dy[r, c]: one block per column, fixed order
__global__ void k_colsum(const float* dy, long long rows, int w, float* db) {
  const int c = blockIdx.x;
  __shared__ float part[256];
  float acc = 0.f;
  for (long long r = threadIdx.x; r < rows; r += blockDim.x) acc += dy[r * w + c];
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) part[threadIdx.x] += part[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) db[c] = part[0];
}

// Long columns: block b sums rows [b per, b per + per) of every column into
// part[b] (kV columns a thread, 32 row lanes, so rows are read whole and four
// of a lane's are in flight); the second launch adds the parts, 8 lanes each
// its own, in a fixed order.  65536 x 128: 37 us with a block per column.
template <int kV>
__global__ void __launch_bounds__(1024) k_colsum_part(const float* dy, long long rows, int w, long long per, float* part) {
  __shared__ float red[32][32 * kV];
  const int lane = threadIdx.x >> 5, q = threadIdx.x & 31;
  const long long r0 = blockIdx.x * per, r1 = min(rows, r0 + per);
  for (int c0 = 0; c0 < w; c0 += 32 * kV) {
    const int c = c0 + q * kV;
    float acc[kV];
#pragma unroll
    for (int v = 0; v < kV; ++v) acc[v] = 0.f;
    if (c < w) {
#pragma unroll 4
      for (long long r = r0 + lane; r < r1; r += 32) {
        if constexpr (kV == 4) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(dy + r * w + c));
          acc[0] += x.x;
          acc[1] += x.y;
          acc[2] += x.z;
          acc[3] += x.w;
        } else {
          acc[0] += __ldg(dy + r * w + c);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < kV; ++v) red[lane][q * kV + v] = acc[v];
    __syncthreads();
    for (int x = threadIdx.x; x < 32 * kV && c0 + x < w; x += blockDim.x) {
      float sum = 0.f;
#pragma unroll 8
      for (int l = 0; l < 32; ++l) sum += red[l][x];
      part[(long long)blockIdx.x * w + c0 + x] = sum;
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256) k_colsum_add(const float* part, int parts, int w, float* db) {
  __shared__ float red[8][32];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), lane = threadIdx.x >> 5;
  float acc = 0.f;
  if (c < w)
#pragma unroll 4
    for (int p = lane; p < parts; p += 8) acc += __ldg(part + (long long)p * w + c);
  red[lane][threadIdx.x & 31] = acc;
  __syncthreads();
  if (lane == 0 && c < w) {
    for (int l = 1; l < 8; ++l) acc += red[l][threadIdx.x];
    db[c] = acc;
  }
}

// g = 2 (p - t) w_row / n ; loss partials per block (sum of w_row (p - t)^2)
__global__ void k_mse(const float* p, const float* t, const float* wrow, float* g, long long rows, int w,
                      double* partial) {
  __shared__ double part[256];
  const long long n = rows * w;
  double acc = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float d = p[i] - t[i];
    const float wr = wrow ? wrow[i / w] : 1.f;
    g[i] = 2.f * d * wr / (float)n;
    acc += (double)wr * d * d;
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) part[threadIdx.x] += part[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = part[0];
}

// Adam (Kingma & Ba) with decoupled weight decay, f32 masters, bf16 copy
__global__ void k_adam(float* w, __nv_bfloat16* wb, const float* g, float* m, float* v, long long n, float lr,
                       float b1, float b2, float eps, float wd, float c1, float c2) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] * (1.f - lr * wd) - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16_rn(wi);
  }
}

}  // namespace

extern "C" {

oems_status oems_tc_gemm_bf16(const void* a, int lda, const void* b, int ldb, float* c, int ldc, int M, int N, int K,
                              float beta, const float* bias, void* stream) {
  if (!a || !b || !c) return pfail(OEMS_ERR_INVALID_ARGUMENT, "NULL operand");
  if (M <= 0 || N <= 0 || K <= 0) return pfail(OEMS_ERR_CONFIG, "GEMM sizes must be positive");
  if (K % 8 || lda % 8 || ldb % 8 || lda < K || ldb < K || ldc < N)
    return pfail(OEMS_ERR_CONFIG, "GEMM: K and the A / B row pitches must be multiples of 8 elements");
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15)
    return pfail(OEMS_ERR_CONFIG, "GEMM: A and B must be 16-byte aligned");
  int* err = nullptr;
  oems_status st = err_word(&err);
  if (st != OEMS_OK) return st;
  oems::GemmArgs p{};
  p.c = c;
  p.bias = bias;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.K = K;
  p.beta = beta;
  p.err = err;
  EncodeTiled enc = nullptr;
  st = encode_fn(&enc);
  if (st != OEMS_OK) return st;
  int dev = 0, sms = 0;
  PK_CUDA(cudaGetDevice(&dev));
  PK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // tile width: one CTA per SM (the stage ring takes ~192 KB of shared
  // memory), so the estimate is waves x a tile's cost, taken as its MMA
  // columns plus a fixed 64 for loading A and draining the accumulator
  const long long tm = (M + 127) / 128;
  int BN = 64;
  long long best = -1;
  for (int cand : {256, 128, 64}) {
    const long long waves = (tm * ((N + cand - 1) / cand) + sms - 1) / sms;
    const long long cost = waves * (cand + 64);
    if (best < 0 || cost < best) best = cost, BN = cand;
  }
  // few tiles and a long K (the weight gradients: 128 x 640 outputs over K =
  // 65,536 ran on 10 of 148 SMs, 215 us): the K range in parts of at least 8
  // blocks, as many as the SMs take in one wave.  Fewer than half the SMs
  // busy, or the sum of the parts costs more than it gives; so it does for
  // outputs past 2^18 below K = 4,096 (640 x 640 and 1000 x 512 at 2,048: 17.4
  // and 20.0 us in parts, 16.5 whole; level at 3,072; 20.6 against 24.7 and level
  // at 4,096; 128 x 1024 at 2,048 14.4 against 16.5).
  const int nkb = (K + 63) / 64;
  p.splits = 1;
  p.kb_per = nkb;
  Workspace ws(stream);
  if (tm * ((N + BN - 1) / BN) * 2 <= sms && nkb >= ((long long)M * N > (1 << 18) ? 64 : 32)) {
    long long fewest = -1;
    int split_bn = BN;
    for (int cand : {256, 128, 64}) {
      const long long t = tm * ((N + cand - 1) / cand);
      const long long parts = std::max<long long>(1, std::min<long long>(sms / t, nkb / 8));
      const long long cost = ((nkb + parts - 1) / parts) * (cand + 64);
      if (t <= sms && (fewest < 0 || cost < fewest)) fewest = cost, split_bn = cand;
    }
    const long long t = tm * ((N + split_bn - 1) / split_bn);
    const int parts = (int)std::max<long long>(1, std::min<long long>(sms / t, nkb / 8));
    const int per = (nkb + parts - 1) / parts, splits = (nkb + per - 1) / per;
    if (splits == 1 || ws.get((size_t)splits * M * N * sizeof(float))) {
      BN = split_bn;
      p.kb_per = per;
      p.splits = splits;
      p.part = static_cast<float*>(ws.p);
    }
  }
  CUtensorMap ta, tb;
  st = bf16_map(enc, &ta, a, lda, K, M, 128);
  if (st == OEMS_OK) st = bf16_map(enc, &tb, b, ldb, K, N, BN);
  if (st != OEMS_OK) return st;
  const long long tiles = tm * ((N + BN - 1) / BN) * p.splits;
  const int grid = (int)std::min<long long>(tiles, sms);
  if (BN == 256) {
    PK_CUDA(launch_gemm<256>(ta, tb, p, grid, stream));
  } else if (BN == 128) {
    PK_CUDA(launch_gemm<128>(ta, tb, p, grid, stream));
  } else {
    PK_CUDA(launch_gemm<64>(ta, tb, p, grid, stream));
  }
  if (p.splits > 1) oems::k_gemm_sum<<<grid_for((long long)M * N, 2048), 256, 0, S(stream)>>>(p);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_tc_wait_probe(void* stream) {
  int* err = nullptr;
  oems_status st = err_word(&err);
  if (st != OEMS_OK) return st;
  oems::k_tc_wait_probe<<<1, 32, 0, S(stream)>>>(err);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_tc_check(void* stream) {
  int* err = nullptr;
  oems_status st = err_word(&err);
  if (st != OEMS_OK) return st;
  int h = 0;
  PK_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, S(stream)));
  PK_CUDA(cudaStreamSynchronize(S(stream)));
  if (h) {
    PK_CUDA(cudaMemset(err, 0, sizeof(int)));
    return pfail(OEMS_ERR_TIMEOUT, "a tensor-core GEMM gave up waiting for its MMAs");
  }
  return OEMS_OK;
}

oems_status oems_pk_f32_to_bf16(const float* x, void* y, int64_t n, void* stream) {
  k_f32_to_bf16<<<grid_for(n, 4096), 256, 0, S(stream)>>>(x, static_cast<__nv_bfloat16*>(y), n);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_transpose_bf16(const void* x, int ldx, void* y, int ldy, int R, int C, void* stream) {
  if (R % 8 == 0 && C % 8 == 0 && ldx % 8 == 0 && ldy % 8 == 0 && aligned16(x, y)) {
    const dim3 g8((C + 63) / 64, (R + 63) / 64);
    if (g8.y <= 65535) {
      k_transpose_bf16_8<<<g8, 256, 0, S(stream)>>>(static_cast<const __nv_bfloat16*>(x), ldx,
                                                    static_cast<__nv_bfloat16*>(y), ldy, R, C);
      PK_CUDA(cudaGetLastError());
      return OEMS_OK;
    }
  }
  const dim3 grid((C + 31) / 32, (R + 31) / 32);
  k_transpose_bf16<<<grid, dim3(32, 8), 0, S(stream)>>>(static_cast<const __nv_bfloat16*>(x), ldx,
                                                       static_cast<__nv_bfloat16*>(y), ldy, R, C);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_im2col(const float* x, void* cols, int B, int T, int C, int ks, int s, int ldc, void* stream) {
  if (T < ks) return pfail(OEMS_ERR_CONFIG, "im2col: sequence shorter than the kernel");
  const int Tout = (T - ks) / s + 1;
  const long long n = (long long)B * Tout * ks * C;
  k_im2col<<<grid_for(n, 8192), 256, 0, S(stream)>>>(x, static_cast<__nv_bfloat16*>(cols), B, T, C, ks, s, Tout,
                                                     ldc);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_col2im(const float* dcols, int ldc, float* dx, int B, int T, int C, int ks, int s, void* stream) {
  const int Tout = (T - ks) / s + 1;
  const long long n = (long long)B * T * C;
  k_col2im<<<grid_for(n, 8192), 256, 0, S(stream)>>>(dcols, ldc, dx, B, T, C, ks, s, Tout);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_im2col_causal(const float* x, void* cols, int B, int T, int C, int ks, int dil, int ldc,
                                  void* stream) {
  if (ks < 1 || dil < 1 || ldc < ks * C) return pfail(OEMS_ERR_CONFIG, "im2col_causal: bad kernel, dilation or pitch");
  if (C % 8 == 0 && ldc % 8 == 0 && aligned16(x, cols)) {
    const long long rows = (long long)B * T;
    k_im2col_causal8<<<grid_for(rows * ks * (C / 8), 148 * 16), 256, 0, S(stream)>>>(
        x, static_cast<__nv_bfloat16*>(cols), rows, T, C, ks, dil, ldc);
    PK_CUDA(cudaGetLastError());
    return OEMS_OK;
  }
  const long long n = (long long)B * T * ks * C;
  k_im2col_causal<<<grid_for(n, 8192), 256, 0, S(stream)>>>(x, static_cast<__nv_bfloat16*>(cols), B, T, C, ks, dil,
                                                            ldc);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_col2im_causal(const float* dcols, int ldc, float* dx, int B, int T, int C, int ks, int dil,
                                  void* stream) {
  if (ks < 1 || dil < 1 || ldc < ks * C) return pfail(OEMS_ERR_CONFIG, "col2im_causal: bad kernel, dilation or pitch");
  // (below 2^17 values the launch is all, and the plain kernel's the shorter: 8 x
  // 64 x 128 4.0 us, 4.2 four channels a thread; 8 x 256 x 128 6.2 against 4.2)
  if (C % 4 == 0 && ldc % 4 == 0 && aligned16(dcols, dx) && (long long)B * T * C >= (1 << 17)) {
    const long long rows = (long long)B * T;
    k_col2im_causal4<<<grid_for(rows * (C / 4), 148 * 16), 256, 0, S(stream)>>>(dcols, ldc, dx, rows, T, C, ks, dil);
    PK_CUDA(cudaGetLastError());
    return OEMS_OK;
  }
  const long long n = (long long)B * T * C;
  k_col2im_causal<<<grid_for(n, 8192), 256, 0, S(stream)>>>(dcols, ldc, dx, B, T, C, ks, dil);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_relu(float* x, void* xb, int64_t rows, int w, int ldb, void* stream) {
  if (xb && w % 4 == 0 && ldb % 4 == 0 && aligned16(x, xb)) {
    k_relu4<<<grid_for(rows * (w / 4), 148 * 16), 256, 0, S(stream)>>>(x, static_cast<__nv_bfloat16*>(xb), rows, w, ldb);
    PK_CUDA(cudaGetLastError());
    return OEMS_OK;
  }
  const long long n = rows * w;
  k_relu<<<grid_for(n, 8192), 256, 0, S(stream)>>>(x, static_cast<__nv_bfloat16*>(xb), rows, w, ldb);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_relu_bwd(float* dy, const float* y, int64_t n, void* stream) {
  k_relu_bwd<<<grid_for(n, 8192), 256, 0, S(stream)>>>(dy, y, n);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_colsum(const float* dy, int64_t rows, int w, float* db, void* stream) {
  // The parts (two launches, 10 us and more) against a block per column: they
  // pay from 12,288 rows of 33 to 128 columns on (10.3 us both; 4,096 x 128 9.6
  // against 6.2, 65,536 x 128 12.3 against 36.9), 6,144 of 192 and 256 (10.3),
  // 4,096 of 512 and 640 (11.4 against 12.3, 13.3 against 14.7) and 24,576 of 16
  // (10.3); at 2,048 x 640 13.3 against 10.3.
  const bool long_columns = rows >= (w < 32 ? 24576 : 4096) && rows * std::max(w, 128) >= 1570000;
  const int parts = 148;
  Workspace ws(stream);
  if (long_columns && ws.get((size_t)parts * w * sizeof(float))) {
    const long long per = (rows + parts - 1) / parts;
    float* part = static_cast<float*>(ws.p);
    if (w % 4 == 0 && aligned16(dy, dy))
      k_colsum_part<4><<<parts, 1024, 0, S(stream)>>>(dy, rows, w, per, part);
    else
      k_colsum_part<1><<<parts, 1024, 0, S(stream)>>>(dy, rows, w, per, part);
    k_colsum_add<<<blocks(w, 32), 256, 0, S(stream)>>>(part, parts, w, db);
    PK_CUDA(cudaGetLastError());
    return OEMS_OK;
  }
  k_colsum<<<w, 256, 0, S(stream)>>>(dy, rows, w, db);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_mse(const float* p, const float* t, const float* wrow, float* g, int64_t rows, int w,
                        double* partial, int nblocks, void* stream) {
  if (nblocks < 1 || nblocks > 4096) return pfail(OEMS_ERR_CONFIG, "mse: 1..4096 blocks");
  k_mse<<<nblocks, 256, 0, S(stream)>>>(p, t, wrow, g, rows, w, partial);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

oems_status oems_pk_adam(float* w, void* wb, const float* g, float* m, float* v, int64_t n, float lr, float b1,
                         float b2, float eps, float wd, int step, void* stream) {
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<grid_for(n, 4096), 256, 0, S(stream)>>>(w, static_cast<__nv_bfloat16*>(wb), g, m, v, n, lr, b1, b2, eps,
                                                   wd, c1, c2);
  PK_CUDA(cudaGetLastError());
  return OEMS_OK;
}

}  // extern "C"
