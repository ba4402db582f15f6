// Pieces shared by the decode kernels that contract packed codes on the warp MMA (cq_decode_mma.cu: separate score,
// attn.V and merge launches; cq_decode_cluster.cu: the whole step in one launch): code expansion, 16-bit arithmetic
// with the reference's rounding points, calibration, tensor maps, launches.
#pragma once

#include <cuda.h>
#include <string.h>

#include "cq_common.cuh"
#include "cq_ptx.cuh"

namespace cq {
namespace mma {

using namespace ptx;

constexpr float LOG2E = 1.4426950408889634f;

// ---- per-lane constants for expanding packed codes into MMA A operands -------------------------
// A lane (g = lane/4) owns rows g and g+8 of a 16-row m-tile; they are mapped to two adjacent
// packed elements e, e+1 of the 32-element group the m-tile belongs to (m-tile i = 0, 1 of the group).
// Which element a row stands for is free, as long as the epilogue agrees:
//   2 bits: e = 16 i + 2g, so m-tile i is one word of the group;
//   4 bits: e = 16 (g/4) + 8 i + 2 (g%4): the lane's two m-tiles are the adjacent words 2(g/4), 2(g/4)+1 of the
//           group's four, fetched by one 8-byte load;
//   1 bit:  e = 4g + 2i, so both m-tiles take their bits from the same byte of the same word
//           and share one byte permute.
template <int BITS>
struct Expand {
  static __device__ __forceinline__ int elem(int i, int g) {
    return BITS == 1 ? 4 * g + 2 * i : BITS == 4 ? 16 * (g >> 2) + 8 * i + 2 * (g & 3) : 16 * i + 2 * g;
  }
  static __device__ __forceinline__ int bit_off(int i, int g) { return elem(i, g) * BITS; }
};

__device__ __forceinline__ uint32_t prmt_sel(int byte) {
  return (uint32_t)(byte | (byte << 4) | ((4 + byte) << 8) | ((4 + byte) << 12));
}

// barrier among a subset of the CTA's warps (the producer warp takes no part)
__device__ __forceinline__ void named_barrier_sync(int id, int n_threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n_threads) : "memory");
}

// ---- data-dtype helpers.  The MMA operands are always fp16: bf16 scales, minima and queries fit
// ---- fp16 exactly (8 significant bits) within its range, so they are converted on the way in,
// ---- while every value the reference rounds to the data dtype is rounded to T here too.
template <typename T> struct D16;
template <> struct D16<__half> {
  using T2 = __half2;
  static __device__ __forceinline__ uint32_t to_h2(uint32_t v) { return v; }
  static __device__ __forceinline__ T2 round2(float a, float b) { return __floats2half2_rn(a, b); }
  static __device__ __forceinline__ T2 bcast(float a) { return __float2half2_rn(a); }
  static __device__ __forceinline__ T2 pair2(__half a, __half b) { return __halves2half2(a, b); }
  static __device__ __forceinline__ float2 to_f2(T2 v) { return __half22float2(v); }
  static __device__ __forceinline__ float big() { return 65504.f; }
  // two probabilities rounded to the data dtype, as an fp16 pair
  static __device__ __forceinline__ uint32_t prob_pair(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  // rnd(x / sqrt(128)) as the reference's division gives it: 1/sqrt(128) as two fp16 terms (the
  // second one carries the 1e-4 relative error of the first), product formed by one FMA, one rounding.
  // A plain multiply by fp16(1/sqrt(128)) lands on the neighbouring fp16 value for one logit in ten.
  static __device__ __forceinline__ T2 inv_sqrt_d(T2 x) {
    const __half2 c_hi = __float2half2_rn(0.08837890625f);                       // fp16(1/sqrt(128))
    const __half2 c_lo = __float2half2_rn(0.08838834764831845f - 0.08837890625f);
    return __hfma2(x, c_hi, __hmul2(x, c_lo));
  }
};
template <> struct D16<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static __device__ __forceinline__ uint32_t to_h2(uint32_t v) {
    const __half2 h = __floats2half2_rn(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ T2 round2(float a, float b) { return __floats2bfloat162_rn(a, b); }
  static __device__ __forceinline__ T2 bcast(float a) { return __float2bfloat162_rn(a); }
  static __device__ __forceinline__ T2 pair2(__nv_bfloat16 a, __nv_bfloat16 b) { return __halves2bfloat162(a, b); }
  static __device__ __forceinline__ float2 to_f2(T2 v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ float big() { return 3.0e38f; }
  static __device__ __forceinline__ uint32_t prob_pair(float a, float b) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
    return to_h2(*reinterpret_cast<const uint32_t*>(&r));
  }
  // bf16(1/sqrt(128)) would be off by up to 2^-9 (a systematic error on every logit): multiply in fp32
  static __device__ __forceinline__ T2 inv_sqrt_d(T2 x) {
    const float2 f = __bfloat1622float2(x);
    return __floats2bfloat162_rn(f.x * 0.08838834764831845f, f.y * 0.08838834764831845f);
  }
};

template <typename T>
struct CalibH {   // per head: 16-bit pairs for packed arithmetic in the data dtype
  typename D16<T>::T2 mn, range, rdenom, rdenom_lo;
};

// rnd(rnd(rnd(s - mn) / denom) * range) + mn with the reference's rounding after every operation.  The
// quotient is a product with the reciprocal carried as two 16-bit terms, formed by one FMA: it differs from
// the rounded quotient in one case in 2^11 (fp16).
template <typename T>
__device__ __forceinline__ typename D16<T>::T2 calibrate2(typename D16<T>::T2 v, const CalibH<T>& cal) {
  v = __hsub2(v, cal.mn);
  v = __hfma2(v, cal.rdenom, __hmul2(v, cal.rdenom_lo));
  return __hadd2(__hmul2(v, cal.range), cal.mn);
}

template <typename T>
__device__ __forceinline__ void set_calib(CalibH<T>& cal, float lo, float hi) {
  const float denom = rnd<T>(rnd<T>(hi - lo) + 1e-8f);
  const float range = rnd<T>(rnd<T>(hi + (-3.f)) - lo);
  cal.mn = D16<T>::bcast(lo);
  cal.rdenom = D16<T>::bcast(1.f / denom);
  cal.rdenom_lo = D16<T>::bcast(1.f / denom - rnd<T>(1.f / denom));
  cal.range = D16<T>::bcast(range);
}

// 2^x by the hardware approximation (relative error 2^-22, far below the 16-bit rounding that follows)
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---- host side -----------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// rows x cols matrix (cols contiguous), box = box_cols columns x 128 rows.
// A decode loop asks for the same few descriptors at every step (one cache per layer), so the encoded
// maps are remembered per host thread: a descriptor is a pure function of the key below.
inline bool make_map(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int elem_bytes,
                     uint64_t cols, uint64_t rows, CUtensorMapSwizzle sw, uint32_t box_cols, uint32_t box_rows = 128) {
  struct Entry { const void* base; uint64_t cols, rows; int dt, sw; uint32_t box_cols, box_rows; CUtensorMap map; };
  constexpr int N = 256;
  thread_local Entry cache[N];
  thread_local int used = 0, next = 0;
  for (int i = 0; i < used; ++i) {
    const Entry& e = cache[i];
    if (e.base == base && e.cols == cols && e.rows == rows && e.dt == (int)dt && e.sw == (int)sw && e.box_cols == box_cols &&
        e.box_rows == box_rows) {
      *m = e.map;
      return true;
    }
  }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * (uint64_t)elem_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  if (fn(m, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  Entry& e = cache[next];
  e.base = base; e.cols = cols; e.rows = rows; e.dt = (int)dt; e.sw = (int)sw; e.box_cols = box_cols; e.box_rows = box_rows; e.map = *m;
  next = (next + 1) % N;
  if (used < N) ++used;
  return true;
}

// The value codes of the attn.V kernel at 2 and 4 bits: [tokens of all KV heads][4*BITS words], boxes of 256 token
// rows swizzled over the row width (32 or 64 bytes).  At 1 bit the kernel copies the rows untiled and ignores the map.
template <int BITS>
inline bool make_v_map(CUtensorMap* tm_v, const void* code, uint64_t tokens) {
  if (BITS == 1) { memset(tm_v, 0, sizeof(*tm_v)); return true; }
  return make_map(tm_v, code, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, 4 * BITS, tokens,
                  BITS == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B, 4 * BITS, 256);
}

}  // namespace mma
}  // namespace cq
