// uint8 format, quantize + encode of a span in one launch: extremes per channel, scale and zero point, codes.
//
// What bounded it before: four launches per tensor, the last one a CTA per 2048 tokens of a (batch, head): 16 CTAs for
// 2 x 8 heads x 1280 tokens, each working through the division-by-bisection thresholds alone (26 us; extremes 15 us).
// Here a (batch, head) is a cluster of S CTAs, each with a slice of its tokens: extremes of the slice -> every CTA of the
// cluster by remote stores -> scale, zero point and thresholds, in every CTA -> codes of the slice, whose second reading comes from L2
// (the slices at work at one time are a few tens of MB).  HBM bound where the span is large.
// Thread = 8 consecutive channels (16 bytes) of every 32nd token.
// 2 x 1280 tokens, 8 heads, fp16, 2 bits: 44 us for the four launches, 9.5 us for this one.
#include "cq_cluster.cuh"
#include "cq_common.cuh"
#include "cq_u8_quant.cuh"

namespace cq {
namespace calib {

using namespace cluster;

constexpr int QE_THREADS = 512, QE_LANES = QE_THREADS / 16, MAX_S = 8, KEEP = 8;

// KEPT: the slice has at most KEEP rows per thread; they are loaded at once and stay in registers for the second use
template <typename T, int BITS, bool KEPT>
__global__ void __launch_bounds__(QE_THREADS, 2)
quant_encode_kernel(const T* __restrict__ x, int heads, int t_len, int64_t sb, int64_t st, int64_t sh, float clip,
                    T* __restrict__ scale, T* __restrict__ zp, uint8_t* __restrict__ enc) {
  using T2 = typename Elem<T>::T2;
  constexpr int LEVELS = (1 << BITS) - 1, U = 4;
  __shared__ uint32_t red_s[QE_THREADS / 32][16][8];
  __shared__ float2 ext_s[MAX_S][kHeadDim];              // [CTA of the cluster][channel] (minimum, maximum)
  __shared__ __align__(16) T sz_s[2][kHeadDim];
  __shared__ __align__(16) T thr_s[BITS <= 2 ? LEVELS : 1][kHeadDim];
  const int S = (int)cluster_size(), rank = (int)cluster_rank();
  const int bh = blockIdx.x / S, b = bh / heads, h = bh % heads;
  const int tid = threadIdx.x, col = tid & 15, tl = tid >> 4;
  const int t_begin = (int)((int64_t)t_len * rank / S), t_end = (int)((int64_t)t_len * (rank + 1) / S);      // not empty: S <= t_len
  // Short spans are bound by what lies between the launches of a prompt: the next launch (the values' span, the attention)
  // comes up while this one runs, and this one waits here for the end of the one before it, which wrote x and may read what is
  // written here.  Split, both spans, attention, back to back: 2 x 1280 tokens 73.7 -> 71.4 us, 1 x 256 31.1 -> 29.3, 1 x 1280
  // 51.5 -> 49.8, 4 x 3328 431 -> 430.  (With the split launching it early too, clusters found their places among the split's
  // CTAs, two on an SM: 4 x 3328 took 436.)
  ptx::pdl_launch_dependents();
  x = ptx::pdl_wait_for(x);
  const T* base = x + b * sb + h * sh + col * 8;

  uint4 kept[KEPT ? KEEP : 1];
  if (KEPT) {
#pragma unroll
    for (int u = 0; u < KEEP; ++u) kept[KEPT ? u : 0] = ptx::ld_global16(base + (int64_t)min(t_begin + tl + u * QE_LANES, t_end - 1) * st);
  }
  // extremes of the slice; every thread starts from a row of it, so no neutral element is needed
  {
    const uint4 first = KEPT ? kept[0] : ptx::ld_global16(base + (int64_t)min(t_begin + tl, t_end - 1) * st);
    T2 mn[4], mx[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) mn[i] = mx[i] = reinterpret_cast<const T2*>(&first)[i];
    auto take = [&](const uint4& v) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        mn[i] = __hmin2(mn[i], reinterpret_cast<const T2*>(&v)[i]);
        mx[i] = __hmax2(mx[i], reinterpret_cast<const T2*>(&v)[i]);
      }
    };
    if (KEPT) {
#pragma unroll
      for (int u = 0; u < KEEP; ++u) take(kept[KEPT ? u : 0]);
    } else
    for (int t = t_begin + tl; t < t_end; t += U * QE_LANES) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = ptx::ld_global16(base + (int64_t)min(t + u * QE_LANES, t_end - 1) * st);
#pragma unroll
      for (int u = 0; u < U; ++u) take(v[u]);
    }
    // the two token lanes of a warp, then the warps
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t a = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<uint32_t*>(&mn[i]), 16);
      const uint32_t c = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<uint32_t*>(&mx[i]), 16);
      mn[i] = __hmin2(mn[i], *reinterpret_cast<const T2*>(&a));
      mx[i] = __hmax2(mx[i], *reinterpret_cast<const T2*>(&c));
    }
    if ((tid & 31) < 16) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        red_s[tid >> 5][col][i] = *reinterpret_cast<uint32_t*>(&mn[i]);
        red_s[tid >> 5][col][4 + i] = *reinterpret_cast<uint32_t*>(&mx[i]);
      }
    }
  }
  __syncthreads();
  cluster_arrive();                                      // no CTA stores into one that has not started
  cluster_wait();
  if (tid < kHeadDim) {
    const int c8 = tid >> 3, e = tid & 7;
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll
    for (int w = 0; w < QE_THREADS / 32; ++w) {
      const float2 a = Elem<T>::to_f2(*reinterpret_cast<const T2*>(&red_s[w][c8][e >> 1]));
      const float2 c = Elem<T>::to_f2(*reinterpret_cast<const T2*>(&red_s[w][c8][4 + (e >> 1)]));
      lo = fminf(lo, (e & 1) ? a.y : a.x);
      hi = fmaxf(hi, (e & 1) ? c.y : c.x);
    }
    const uint32_t mine = smem_u32(&ext_s[rank][tid]);
    for (int r = 0; r < S; ++r) st_peer2(map_peer(mine, (uint32_t)r), lo, hi);
  }
  cluster_arrive();
  cluster_wait();
  int bad = 0;
  if (tid < kHeadDim) {
    float lo = INFINITY, hi = -INFINITY;
    for (int r = 0; r < S; ++r) { lo = fminf(lo, ext_s[r][tid].x); hi = fmaxf(hi, ext_s[r][tid].y); }
    float s, z;
    scale_zero<T>(lo, hi, clip, LEVELS, s, z);
    sz_s[0][tid] = Elem<T>::from_f(s);
    sz_s[1][tid] = Elem<T>::from_f(z);
    if (rank == 0) {
      scale[(int64_t)bh * kHeadDim + tid] = sz_s[0][tid];
      zp[(int64_t)bh * kHeadDim + tid] = sz_s[1][tid];
    }
    bad = !(s > 0.f) || isinf(s) || isnan(z) || isinf(z);
  }
  const bool plain = BITS > 2 || __syncthreads_or(bad);      // per-element arithmetic: 4 bits, or a channel with a degenerate scale
  if (BITS > 2) __syncthreads();
  if (!plain) {
    for (int i = tid; i < LEVELS * kHeadDim; i += QE_THREADS) {
      const int k = i / kHeadDim, c = i % kHeadDim;
      thr_s[BITS <= 2 ? k : 0][c] = threshold<T>(Elem<T>::to_f(sz_s[0][c]), Elem<T>::to_f(sz_s[1][c]), k, LEVELS);
    }
    __syncthreads();
  }
  uint8_t* dst = enc + ((int64_t)bh * t_len) * (kHeadDim * BITS / 8);
  // a thread's BITS bytes of a token; neighbours join theirs to 4-byte stores (all lanes take part)
  auto store = [&](int t, uint32_t v) {
    if (BITS == 1) v |= __shfl_down_sync(0xffffffffu, v, 1) << 8;
    if (BITS <= 2) v |= __shfl_down_sync(0xffffffffu, v, BITS == 1 ? 2 : 1) << 16;
    if (t < t_end && col % (4 / BITS) == 0) *reinterpret_cast<uint32_t*>(dst + (int64_t)t * (kHeadDim * BITS / 8) + col * BITS) = v;
  };
  const int t_last = t_begin + (t_end - t_begin + QE_LANES - 1) / QE_LANES * QE_LANES;      // whole rounds, for the shuffles
  if (plain) {
    float s[8], z[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { s[i] = Elem<T>::to_f(sz_s[0][col * 8 + i]); z[i] = Elem<T>::to_f(sz_s[1][col * 8 + i]); }
    auto encode = [&](int t, const uint4& raw) {
      const T* xv = reinterpret_cast<const T*>(&raw);
      uint32_t v = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {                      // byte = 8 / BITS channels, most significant field first
        const uint32_t code = (uint32_t)ref_code<T>(Elem<T>::to_f(xv[i]), s[i], z[i], LEVELS);
        v |= code << (8 * (i * BITS / 8) + 8 - BITS - (i * BITS) % 8);
      }
      store(t, v);
    };
    if (KEPT) {
#pragma unroll
      for (int u = 0; u < KEEP; ++u)
        if (t_begin + u * QE_LANES < t_end) encode(t_begin + tl + u * QE_LANES, kept[KEPT ? u : 0]);
    } else {
      // two rows requested together (one after the other 1 x 8 x 4096 tokens at 4 bits took 16.0 us, so 14.5; 16 x 3328 82.1, 78.8; four:
      // 14.0, 82.0)
      for (int t0 = t_begin + tl; t0 < t_last; t0 += 2 * QE_LANES) {
        uint4 v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) v[u] = ptx::ld_global16(base + (int64_t)min(t0 + u * QE_LANES, t_end - 1) * st);
#pragma unroll
        for (int u = 0; u < 2; ++u) encode(t0 + u * QE_LANES, v[u]);
      }
    }
    return;
  }
  if constexpr (BITS <= 2) {
    T2 thr[LEVELS][4];
#pragma unroll
    for (int k = 0; k < LEVELS; ++k) {
      const uint4 w = *reinterpret_cast<const uint4*>(&thr_s[k][col * 8]);
#pragma unroll
      for (int i = 0; i < 4; ++i) thr[k][i] = reinterpret_cast<const T2*>(&w)[i];
    }
    auto encode = [&](int t, const uint4& raw) {
      const T2* xv = reinterpret_cast<const T2*>(&raw);
      uint32_t r = 0;
      if (BITS == 1) {
        // channel i at bit 7 - i; pair p = channels (2p, 2p+1) -> bits 7-2p (low half), 22-2p (high half)
#pragma unroll
        for (int i = 0; i < 4; ++i) r |= __hgt2_mask(xv[i], thr[0][i]) & ((0x80u >> (2 * i)) | (0x400000u >> (2 * i)));
        r = (r | (r >> 16)) & 0xffu;
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          T2 cnt = __hgt2(xv[i], thr[0][i]);             // the code as a number of the data type
#pragma unroll
          for (int k = 1; k < LEVELS; ++k) cnt = __hadd2(cnt, __hgt2(xv[i], thr[k][i]));
          const T2 m = __hadd2(cnt, Pk2<T>::magic());    // 0..3 in the low mantissa bits
          const uint32_t w = *reinterpret_cast<const uint32_t*>(&m) & 0x00030003u;
          r |= (((w & 0xffffu) << 2) | (w >> 16)) << (8 * (i >> 1) + 4 - 4 * (i & 1));      // (code 2i, code 2i+1) as four bits
        }
      }
      store(t, r);
    };
    if (KEPT) {
#pragma unroll
      for (int u = 0; u < KEEP; ++u)
        if (t_begin + u * QE_LANES < t_end) encode(t_begin + tl + u * QE_LANES, kept[KEPT ? u : 0]);
    } else {
      for (int t0 = t_begin + tl; t0 < t_last; t0 += U * QE_LANES) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = ptx::ld_global16(base + (int64_t)min(t0 + u * QE_LANES, t_end - 1) * st);
#pragma unroll
        for (int u = 0; u < U; ++u) encode(t0 + u * QE_LANES, v[u]);
      }
    }
  }
}

// The smallest cluster that puts two CTAs on every SM, as long as a CTA has 64 tokens (two rounds of its threads)
static int cluster_of(int64_t bh, int t_len) {
  const int sms = sm_count();
  int S = 1;
  while (S < MAX_S && bh * S < 2 * sms && t_len >= 128 * S) S *= 2;
  return S;
}

template <typename T, int BITS>
static int launch_quant_encode(const void* x, int batch, int t_len, int heads, const int64_t* strides, float clip, void* scale, void* zp,
                               uint8_t* enc, cudaStream_t st) {
  const int64_t bh = (int64_t)batch * heads;
  const int S = cluster_of(bh, t_len);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(bh * S));
  cfg.blockDim = dim3(QE_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const bool fits = (t_len + S - 1) / S <= KEEP * QE_LANES;
  if (cudaLaunchKernelEx(&cfg, fits ? quant_encode_kernel<T, BITS, true> : quant_encode_kernel<T, BITS, false>, static_cast<const T*>(x), heads, t_len, strides[0], strides[1], strides[2], clip,
                         static_cast<T*>(scale), static_cast<T*>(zp), enc) != cudaSuccess) {
    (void)cudaGetLastError();
    return CQ_ERR_LAUNCH;
  }
  return check_launch();
}

}  // namespace calib
}  // namespace cq

using namespace cq;

extern "C" int cq_calib_quant_encode(const void* x, int batch, int t_len, int heads, int head_dim, const int64_t* strides, int bits, float clip,
                                     int dtype, void* scale, void* zero_point, uint8_t* enc_out, void* stream) {
  if (!x || !strides || !scale || !zero_point || !enc_out || batch <= 0 || t_len <= 0 || heads <= 0) return CQ_ERR_BAD_ARG;
  if (dtype != CQ_DTYPE_F16 && dtype != CQ_DTYPE_BF16) return CQ_ERR_BAD_ARG;
  if ((bits != 1 && bits != 2 && bits != 4) || head_dim != kHeadDim) return CQ_ERR_UNSUPPORTED;
  if (!aligned16(x) || strides[0] % 8 || strides[1] % 8 || strides[2] % 8 || reinterpret_cast<uintptr_t>(enc_out) % 4) return CQ_ERR_BAD_ARG;
  if ((int64_t)batch * heads > 0x0fffffff) return CQ_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Few (batch, head) pairs with long spans at 4 bits: a quotient per element, on clusters that fill less than the GPU.  The separate
  // launches deal tokens over all SMs (1 x 16384, one head 43 us against 63; 2 x 16384 x 8 84 against 109; 2 x 3328 x 8, 416
  // tokens a CTA, 37 against 29; 8 x 16384 x 8, two CTAs on every SM, 298 against 260)
  const int64_t ctas = (int64_t)batch * heads * calib::cluster_of((int64_t)batch * heads, t_len);
  if (bits == 4 && ctas < 2 * cq::sm_count() && t_len > 1024 * calib::cluster_of((int64_t)batch * heads, t_len)) {
    const int rc = cq_calib_minmax(x, batch, t_len, heads, head_dim, strides, bits, clip, dtype, scale, zero_point, stream);
    return rc ? rc : cq_calib_quantize(x, batch, t_len, heads, head_dim, strides, bits, dtype, scale, zero_point, 0, nullptr, enc_out, stream);
  }
#define CQ_QE(T, B) calib::launch_quant_encode<T, B>(x, batch, t_len, heads, strides, clip, scale, zero_point, enc_out, st)
  if (dtype == CQ_DTYPE_F16) return bits == 1 ? CQ_QE(__half, 1) : bits == 2 ? CQ_QE(__half, 2) : CQ_QE(__half, 4);
  return bits == 1 ? CQ_QE(__nv_bfloat16, 1) : bits == 2 ? CQ_QE(__nv_bfloat16, 2) : CQ_QE(__nv_bfloat16, 4);
#undef CQ_QE
}
