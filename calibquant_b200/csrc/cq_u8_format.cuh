// What the kernels on the uint8 format share: where an MMA operand register finds its codes, and the score type.
#pragma once

#include "cq_common.cuh"

namespace cq {
namespace calib {

// Operand layout of the score products (A = codes with rows = tokens, k = channels; see lut_scores_mma_kernel).
template <int BITS>
struct LutMap {
  // channel that k-block kb, lane column c, slot (0: a0.lo, 1: a0.hi, 2: a2.lo, 3: a2.hi) reads, and the
  // bit position of its field inside the 16-bit half
  static __device__ __forceinline__ void get(int kb, int c, int slot, int& chan, int& pos) {
    if (BITS == 1) {             // word j = kb/2 (32 channels), bytes s, s+2 with s = kb%2
      const int j = kb >> 1, s = kb & 1;
      const int byte = s + 2 * (slot & 1);
      pos = 2 * c + (slot >> 1);
      chan = 32 * j + 8 * byte + (7 - pos);
    } else if (BITS == 2) {      // word kb (16 channels): a0 from bytes 0,2, a2 from bytes 1,3; field c
      const int byte = (slot >> 1) + 2 * (slot & 1);
      pos = 2 * c;
      chan = 16 * kb + 4 * byte + (3 - c);
    } else {                     // words 2kb (a0) and 2kb+1 (a2), 8 channels each; nibble (c&1) of byte c>>1 (+2)
      const int word = 2 * kb + (slot >> 1);
      const int byte = (c >> 1) + 2 * (slot & 1);
      pos = 0;                   // shifted down to bit 0 before masking
      chan = 8 * word + 2 * byte + (1 - (c & 1));
    }
  }
};

// Score type of the fused decode step: `fused_kernel(...) / sd - bias_k` is an fp16 tensor minus a tensor of
// the data dtype, so torch keeps fp16 for fp16 data and promotes to fp32 for bf16 data.
template <typename T> struct StepScore;
template <> struct StepScore<__half> {
  using type = __half;
  static __device__ __forceinline__ float r(float v) { return rnd<__half>(v); }
  static __device__ __forceinline__ __half make(float v) { return __float2half_rn(v); }
  static __device__ __forceinline__ float load(__half v) { return __half2float(v); }
};
template <> struct StepScore<__nv_bfloat16> {
  using type = float;
  static __device__ __forceinline__ float r(float v) { return v; }
  static __device__ __forceinline__ float make(float v) { return v; }
  static __device__ __forceinline__ float load(float v) { return v; }
};


}  // namespace calib
}  // namespace cq
