// Projections of a decode step of a few requests: y = x W^T for up to four rows of x, W [N][K] row-major, fp32 sums rounded once
// to the data type.  The step is bound by reading W once; a library GEMM reached 4.1 TB/s on the 6144 x 4096 projection of one
// request (12.1 us) and cost 12 us of host time to issue, more than its share of the GPU.
//   * A warp owns one row of W (or the two rows of a rotary pair), its lanes 16-byte pieces in turn, four loads per row in flight;
//     x comes from L1.  All warps of the sizes in use are resident at once: nothing is split along K, nothing is exchanged.
//   * The projection to queries, keys and values ends with what follows it anyway: the pair (d, d + 64) of a head is rotated
//     and goes to the query tensor or to its place in the full-precision cache.
// More than four rows: the multiplications (32 a 16-byte piece and row pair) begin to cost as much as the reading, and a
// matrix product takes over.
// One request, hidden 4096, bfloat16: projection, split, rotation and append 10.0 us (12.1 + 2.4 us and two launches before),
// output projection 7.1 us (8.8 us).
#include "cq_common.cuh"

namespace cq {
namespace gemv {

constexpr int WARPS = 8, U = 4, MAX_ROWS = 4;

// sums of R rows of W (w + r * pitch) with the B rows of x, complete in every lane
template <typename T, int B, int R>
__device__ __forceinline__ void dot(const T* __restrict__ x, const T* __restrict__ w, int64_t pitch, int K, int lane, float (&acc)[R][B]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int b = 0; b < B; ++b) acc[r][b] = 0.f;
  const int pieces = K / 8;
  for (int c0 = lane; c0 < pieces; c0 += 32 * U) {
    uint4 wv[U][R];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        wv[u][r] = make_uint4(0u, 0u, 0u, 0u);
        if (c0 + 32 * u < pieces) wv[u][r] = __ldg(reinterpret_cast<const uint4*>(w + r * pitch) + c0 + 32 * u);
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c0 + 32 * u >= pieces) break;
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + (int64_t)b * K) + c0 + 32 * u);
        const typename Elem<T>::T2* xp = reinterpret_cast<const typename Elem<T>::T2*>(&xv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 xf = Elem<T>::to_f2(xp[i]);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float2 wf = Elem<T>::to_f2(reinterpret_cast<const typename Elem<T>::T2*>(&wv[u][r])[i]);
            acc[r][b] = fmaf(wf.x, xf.x, acc[r][b]);
            acc[r][b] = fmaf(wf.y, xf.y, acc[r][b]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int b = 0; b < B; ++b) acc[r][b] = warp_sum(acc[r][b]);
}

template <typename T, int B>
__global__ void __launch_bounds__(WARPS * 32)
linear_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ out, int N, int K) {
  const int lane = threadIdx.x & 31, row = blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (row >= N) return;
  float acc[1][B];
  dot<T, B, 1>(x, w + (int64_t)row * K, 0, K, lane, acc);
#pragma unroll
  for (int b = 0; b < B; ++b)
    if (lane == b) out[(int64_t)b * N + row] = Elem<T>::from_f(acc[0][b]);
}

// W: per KV head n_rep query heads, key, value of 128 rows each; a warp: rows d and d + 64 of one of them
template <typename T, int B>
__global__ void __launch_bounds__(WARPS * 32)
qkv_rope_append_kernel(const T* __restrict__ x, const T* __restrict__ w, int K, const T* __restrict__ cos_t, const T* __restrict__ sin_t,
                       int rope_len, const int64_t* __restrict__ position_ids, int n_kv_heads, int n_rep, T* __restrict__ q_out,
                       T* __restrict__ k_cache, T* __restrict__ v_cache, int64_t cache_stride_b, int64_t cache_stride_h, int index) {
  const int lane = threadIdx.x & 31, unit = blockIdx.x * WARPS + (threadIdx.x >> 5);
  const int head = unit >> 6, d = unit & 63, per_kv = n_rep + 2;
  if (head >= n_kv_heads * per_kv) return;
  float acc[2][B];
  dot<T, B, 2>(x, w + ((int64_t)head * kHeadDim + d) * K, (int64_t)64 * K, K, lane, acc);
  const int hk = head / per_kv, slot = head % per_kv;      // slot < n_rep: query head; n_rep: key; n_rep+1: value
#pragma unroll
  for (int b = 0; b < B; ++b) {
    if (lane != b) continue;
    const float x0 = rnd<T>(acc[0][b]), x1 = rnd<T>(acc[1][b]);
    T* dst = slot < n_rep ? q_out + ((int64_t)(b * n_kv_heads + hk) * n_rep + slot) * kHeadDim
                          : (slot == n_rep ? k_cache : v_cache) + b * cache_stride_b + hk * cache_stride_h + (int64_t)index * kHeadDim;
    if (slot == n_rep + 1) {                               // values are not rotated
      dst[d] = Elem<T>::from_f(x0);
      dst[d + 64] = Elem<T>::from_f(x1);
      continue;
    }
    int64_t pos = position_ids[b];
    pos = pos < 0 ? 0 : (pos >= rope_len ? rope_len - 1 : pos);
    const T* cr = cos_t + pos * kHeadDim;
    const T* sr = sin_t + pos * kHeadDim;
    // x*cos rounded, then + rotate_half(x)*sin with one more rounding, as where the rotation stands alone
    const float a0 = rnd<T>(x0 * Elem<T>::to_f(cr[d])), a1 = rnd<T>(x1 * Elem<T>::to_f(cr[d + 64]));
    dst[d] = Elem<T>::from_f(__fadd_rn(a0, __fmul_rn(-x1, Elem<T>::to_f(sr[d]))));
    dst[d + 64] = Elem<T>::from_f(__fadd_rn(a1, __fmul_rn(x0, Elem<T>::to_f(sr[d + 64]))));
  }
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

extern "C" int cq_qkv_rope_append(const void* x, const void* weight, int k, const void* cos_table, const void* sin_table, int rope_len,
                                  const int64_t* position_ids, int batch, int n_kv_heads, int n_rep, int head_dim, void* q_out, void* k_cache,
                                  void* v_cache, int64_t cache_stride_b, int64_t cache_stride_h, int capacity, int append_index, int dtype,
                                  void* stream) {
  if (batch == 0) return CQ_OK;
  if (!x || !weight || !cos_table || !sin_table || !position_ids || !q_out || !k_cache || !v_cache) return CQ_ERR_BAD_ARG;
  if (batch < 0 || k <= 0 || n_kv_heads <= 0 || n_rep <= 0 || rope_len <= 0 || append_index < 0 || append_index >= capacity) return CQ_ERR_BAD_ARG;
  if (dtype != CQ_DTYPE_F16 && dtype != CQ_DTYPE_BF16) return CQ_ERR_BAD_ARG;
  if (head_dim != kHeadDim || batch > gemv::MAX_ROWS || k % 8) return CQ_ERR_UNSUPPORTED;
  const int64_t units = (int64_t)n_kv_heads * (n_rep + 2) * 64;
  if (units > 0x3fffffff) return CQ_ERR_UNSUPPORTED;
  if (!aligned16(x) || !aligned16(weight)) return CQ_ERR_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)(units / gemv::WARPS);
#define CQ_QKV(T, B) gemv::qkv_rope_append_kernel<T, B><<<grid, gemv::WARPS * 32, 0, st>>>(static_cast<const T*>(x), static_cast<const T*>(weight), k, \
      static_cast<const T*>(cos_table), static_cast<const T*>(sin_table), rope_len, position_ids, n_kv_heads, n_rep, static_cast<T*>(q_out),           \
      static_cast<T*>(k_cache), static_cast<T*>(v_cache), cache_stride_b, cache_stride_h, append_index)
#define CQ_QKV_T(T) do { if (batch == 1) CQ_QKV(T, 1); else if (batch == 2) CQ_QKV(T, 2); else if (batch == 3) CQ_QKV(T, 3); else CQ_QKV(T, 4); } while (0)
  if (dtype == CQ_DTYPE_F16) CQ_QKV_T(__half); else CQ_QKV_T(__nv_bfloat16);
#undef CQ_QKV_T
#undef CQ_QKV
  return check_launch();
}
