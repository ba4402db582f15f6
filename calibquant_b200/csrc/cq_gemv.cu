// The output projection of a decode step of a few requests: y = x W^T for up to four rows of x, W [N][K] row-major, fp32 sums
// rounded once to the data type.  It is bound by reading W once; a library GEMM took 8.8 us for 4096 x 4096 and one request
// (3.8 TB/s) and 12 us of host time to issue, more than its share of the GPU; this takes 7.1 us.
//   * A warp owns one row of W, its lanes 16-byte pieces in turn, four loads in flight; x comes from L1.  All warps of the sizes
//     in use are resident at once: nothing is split along K, nothing is exchanged.
// More than four rows: the multiplications begin to cost as much as the reading, and a matrix product takes over; at the tensor level also
// for rows of more than 4096 elements (14336 -> 4096, one row: 31.8 us against 26.5), where a warp's chain of loads is the longer.
// (The projection to queries, keys and values stays with the matrix product: a rounding of a query or key that falls the other
// way moves the extreme logits, and with them the calibration of a whole row, by more than the data type's precision.)
#include "cq_common.cuh"

namespace cq {
namespace gemv {

constexpr int WARPS = 8, U = 4, MAX_ROWS = 4;

// sums of a row of W with the B rows of x, complete in every lane
template <typename T, int B>
__device__ __forceinline__ void dot(const T* __restrict__ x, const T* __restrict__ w, int K, int lane, float (&acc)[B]) {
  using T2 = typename Elem<T>::T2;
#pragma unroll
  for (int b = 0; b < B; ++b) acc[b] = 0.f;
  const int pieces = K / 8;
  for (int c0 = lane; c0 < pieces; c0 += 32 * U) {
    uint4 wv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      wv[u] = make_uint4(0u, 0u, 0u, 0u);
      if (c0 + 32 * u < pieces) wv[u] = __ldg(reinterpret_cast<const uint4*>(w) + c0 + 32 * u);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c0 + 32 * u >= pieces) break;
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + (int64_t)b * K) + c0 + 32 * u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 xf = Elem<T>::to_f2(reinterpret_cast<const T2*>(&xv)[i]), wf = Elem<T>::to_f2(reinterpret_cast<const T2*>(&wv[u])[i]);
          acc[b] = fmaf(wf.x, xf.x, acc[b]);
          acc[b] = fmaf(wf.y, xf.y, acc[b]);
        }
      }
    }
  }
#pragma unroll
  for (int b = 0; b < B; ++b) acc[b] = warp_sum(acc[b]);
}

template <typename T, int B>
__global__ void __launch_bounds__(WARPS * 32)
linear_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ out, int N, int K) {
  const int lane = threadIdx.x & 31, row = blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (row >= N) return;
  float acc[B];
  dot<T, B>(x, w + (int64_t)row * K, K, lane, acc);
#pragma unroll
  for (int b = 0; b < B; ++b)
    if (lane == b) out[(int64_t)b * N + row] = Elem<T>::from_f(acc[b]);
}

}  // namespace gemv
}  // namespace cq

using namespace cq;

extern "C" int cq_linear_small(const void* x, const void* weight, void* out, int rows, int n, int k, int dtype, void* stream) {
  if (rows == 0 || n == 0) return CQ_OK;
  if (!x || !weight || !out || rows < 0 || n < 0 || k <= 0) return CQ_ERR_BAD_ARG;
  if (dtype != CQ_DTYPE_F16 && dtype != CQ_DTYPE_BF16) return CQ_ERR_BAD_ARG;
  if (rows > gemv::MAX_ROWS || k % 8) return CQ_ERR_UNSUPPORTED;
  if (!aligned16(x) || !aligned16(weight)) return CQ_ERR_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)((n + gemv::WARPS - 1) / gemv::WARPS);
#define CQ_LIN(T, B) gemv::linear_kernel<T, B><<<grid, gemv::WARPS * 32, 0, st>>>(static_cast<const T*>(x), static_cast<const T*>(weight), static_cast<T*>(out), n, k)
#define CQ_LIN_T(T) do { if (rows == 1) CQ_LIN(T, 1); else if (rows == 2) CQ_LIN(T, 2); else if (rows == 3) CQ_LIN(T, 3); else CQ_LIN(T, 4); } while (0)
  if (dtype == CQ_DTYPE_F16) CQ_LIN_T(__half); else CQ_LIN_T(__nv_bfloat16);
#undef CQ_LIN_T
#undef CQ_LIN
  return check_launch();
}
