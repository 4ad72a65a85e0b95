// The encoder's block analysis on the GPU: forwardDCT and satd
// (ebiv/transform.go:44-119) over a batch of n x n residual blocks, the inner
// loops of the encoder's rate-distortion search (every intra-mode trial and
// every inter candidate transforms or Hadamard-scores its residual).
//
// n threads per block, thread l with column l of the block in registers.
// forwardDCT: tmp[k][l] = round(sum_i C[k][i] * src[i][l]) down the column,
// then, through shared memory, row l: dst[l][m] = round(sum_j C[m][j] *
// tmp[l][j]) (int64 accumulation, rounding shift by 13, the int32 narrowing of
// the reference).  satd: the Walsh-Hadamard butterflies of the columns, then
// the rows (int32 arithmetic, wrapping as Go's does, in which the order of the
// two makes no difference), and the sum of absolute values (int64) as a
// reduction over the block's threads.
//
// Bound by the block's 2 n^3 products, so nothing else is done per product:
// the samples stay in registers and four words of the basis come with one load
// that all threads share.  32,400 blocks of 8x8: 32 us with a warp per block,
// a lane per output and two loads a product, 9 us now.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <new>

#include "../../include/ebivgpu.h"
#include "ebiv_format.h"

namespace ebiv {
namespace dev {

constexpr int kAnaThreads = 128;
constexpr int kDCTScaleBits = 13;  // the DCT basis is scaled by 2^13 (ebiv/transform.go:15-40)

// One output of a 1-D transform: row k of the basis with v.
template <int N>
__device__ __forceinline__ int32_t dctDot(const int4* c, int k, const int32_t (&v)[N]) {
  int64_t acc = 1LL << (kDCTScaleBits - 1);
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const int4 w = c[(k * N + i) / 4];
    acc += (int64_t)w.x * v[i];
    acc += (int64_t)w.y * v[i + 1];
    acc += (int64_t)w.z * v[i + 2];
    acc += (int64_t)w.w * v[i + 3];
  }
  return (int32_t)(acc >> kDCTScaleBits);
}

template <int N>
__device__ __forceinline__ void hadamard(int32_t (&v)[N]) {
#pragma unroll
  for (int span = 1; span < N; span <<= 1)
#pragma unroll
    for (int a = 0; a < N; a++)
      if (!(a & span)) {
        const uint32_t x = (uint32_t)v[a], y = (uint32_t)v[a + span];
        v[a] = (int32_t)(x + y);
        v[a + span] = (int32_t)(x - y);
      }
}

template <int N>
__global__ void __launch_bounds__(kAnaThreads) kAnalyze(const int32_t* __restrict__ src, int count,
                                                        const int32_t* __restrict__ basis, int32_t* __restrict__ dst,
                                                        int64_t* __restrict__ satdOut) {
  constexpr int kBlocks = kAnaThreads / N, kPitch = N + 1;
  __shared__ int4 sC[N * N / 4];
  __shared__ int32_t sTmp[kBlocks][N * kPitch];
  if (threadIdx.x < N * N / 4) sC[threadIdx.x] = reinterpret_cast<const int4*>(basis)[threadIdx.x];
  __syncthreads();
  const int l = threadIdx.x % N;
  const size_t b = (size_t)blockIdx.x * kBlocks + threadIdx.x / N;
  const bool mine = b < (size_t)count;  // every thread of a warp stays for its barriers
  const int32_t* s = src + b * (N * N);
  int32_t* tmp = sTmp[threadIdx.x / N];
  int32_t v[N], t[N];
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = mine ? s[i * N + l] : 0;
  if (dst) {
#pragma unroll 8
    for (int k = 0; k < N; k++) tmp[k * kPitch + l] = dctDot<N>(sC, k, v);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < N; j++) t[j] = tmp[l * kPitch + j];
    int4* const d = reinterpret_cast<int4*>(dst + b * (N * N) + l * N);
#pragma unroll 2
    for (int m = 0; m < N; m += 4) {
      const int4 o = make_int4(dctDot<N>(sC, m, t), dctDot<N>(sC, m + 1, t), dctDot<N>(sC, m + 2, t), dctDot<N>(sC, m + 3, t));
      if (mine) d[m / 4] = o;
    }
    __syncwarp();
  }
  if (satdOut) {
    hadamard<N>(v);
#pragma unroll
    for (int i = 0; i < N; i++) tmp[i * kPitch + l] = v[i];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < N; j++) t[j] = tmp[l * kPitch + j];
    hadamard<N>(t);
    int64_t sum = 0;
#pragma unroll
    for (int j = 0; j < N; j++) sum += t[j] < 0 ? -(int64_t)t[j] : (int64_t)t[j];
    for (int o = N / 2; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (l == 0 && mine) satdOut[b] = sum;
  }
}

template <int N>
static void launchAnalyze(const int32_t* src, int count, const int32_t* basis, int32_t* dst, int64_t* satd, cudaStream_t s) {
  constexpr int kBlocks = kAnaThreads / N;
  kAnalyze<N><<<(int)(((size_t)count + kBlocks - 1) / kBlocks), kAnaThreads, 0, s>>>(src, count, basis, dst, satd);
}

}  // namespace dev
}  // namespace ebiv

using namespace ebiv;

struct ebivgpu_analysis {
  int32_t* dSrc = nullptr;
  int32_t* dDst = nullptr;
  int64_t* dSatd = nullptr;
  int32_t* dBasis = nullptr;  // the three DCT matrices, 256 words each
  size_t cap = 0;             // blocks of 256 words the buffers hold
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  ~ebivgpu_analysis() {
    if (stream) cudaStreamSynchronize(stream);
    cudaFree(dSrc);
    cudaFree(dDst);
    cudaFree(dSatd);
    cudaFree(dBasis);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (stream) cudaStreamDestroy(stream);
  }
};

extern "C" {

int ebivgpu_analysis_create(ebivgpu_analysis** out) {
  if (!out) return kErrArg;
  ebivgpu_analysis* a = new (std::nothrow) ebivgpu_analysis();
  if (!a) return kErrArg;
  const CodingTables& t = codingTables();
  int32_t basis[3 * 256];
  std::memset(basis, 0, sizeof(basis));
  for (int k = 0; k < 3; k++) std::memcpy(basis + 256 * k, t.dct[k], sizeof(int32_t) * kLumaTx[k] * kLumaTx[k]);
  if (cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&a->ev0) != cudaSuccess || cudaEventCreate(&a->ev1) != cudaSuccess ||
      cudaMalloc(&a->dBasis, sizeof(basis)) != cudaSuccess ||
      cudaMemcpy(a->dBasis, basis, sizeof(basis), cudaMemcpyHostToDevice) != cudaSuccess) {
    delete a;
    return kErrDevice;
  }
  *out = a;
  return kOK;
}

void ebivgpu_analysis_destroy(ebivgpu_analysis* a) { delete a; }

int ebivgpu_fdct_satd(ebivgpu_analysis* a, const int32_t* residuals, int n, int count, int32_t* coeffs,
                      int64_t* satd, double* kernel_ms) {
  if (!a || (!residuals && count) || count < 0 || (n != 4 && n != 8 && n != 16)) return kErrArg;
  if (count == 0) return kOK;
  const size_t nn = (size_t)n * n;
  if ((size_t)count > a->cap) {
    cudaFree(a->dSrc);
    cudaFree(a->dDst);
    cudaFree(a->dSatd);
    a->dSrc = a->dDst = nullptr;
    a->dSatd = nullptr;
    a->cap = 0;
    if (cudaMalloc(&a->dSrc, (size_t)count * 256 * 4) != cudaSuccess ||
        cudaMalloc(&a->dDst, (size_t)count * 256 * 4) != cudaSuccess ||
        cudaMalloc(&a->dSatd, (size_t)count * 8) != cudaSuccess)
      return kErrDevice;
    a->cap = (size_t)count;
  }
  const int k = n == 4 ? 0 : (n == 8 ? 1 : 2);
  if (cudaMemcpyAsync(a->dSrc, residuals, (size_t)count * nn * 4, cudaMemcpyHostToDevice, a->stream) != cudaSuccess)
    return kErrDevice;
  cudaEventRecord(a->ev0, a->stream);
  (n == 4 ? dev::launchAnalyze<4> : (n == 8 ? dev::launchAnalyze<8> : dev::launchAnalyze<16>))(
      a->dSrc, count, a->dBasis + 256 * k, coeffs ? a->dDst : nullptr, satd ? a->dSatd : nullptr, a->stream);
  if (cudaGetLastError() != cudaSuccess) return kErrDevice;
  cudaEventRecord(a->ev1, a->stream);
  if ((coeffs && cudaMemcpyAsync(coeffs, a->dDst, (size_t)count * nn * 4, cudaMemcpyDeviceToHost, a->stream)) ||
      (satd && cudaMemcpyAsync(satd, a->dSatd, (size_t)count * 8, cudaMemcpyDeviceToHost, a->stream)) ||
      cudaStreamSynchronize(a->stream) != cudaSuccess)
    return kErrDevice;
  if (kernel_ms) {
    float ms = 0;
    cudaEventElapsedTime(&ms, a->ev0, a->ev1);
    *kernel_ms = ms;
  }
  return kOK;
}

}  // extern "C"
