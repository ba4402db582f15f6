// Decode step on the uint8 format as ONE launch: a thread-block cluster per (batch row, KV head).
//
// What bounded the step as four launches (scores, softmax of a whole row per CTA, attn.V, finish): 107 us at 16 x 3328
// tokens, 1 bit, of which 28 us were softmax CTAs that walked the full-precision keys one warp per key and 22 us were
// finish CTAs that walked the full-precision values one row after the other; the scores went through memory as fp32.
// Here a CTA owns a share of the visual tokens (items of 64, dealt out over its warps in 16-token tiles) and of the full-precision
// tokens (tiles of 16), keeps its scores in shared memory and does both products of both spans on the warp MMA:
//   1. visual scores, extremes -> every peer (remote stores), full-precision scores while they travel;
//   2. calibration and mask, local maximum and sum of exponentials -> every peer: the global sum has to be known before
//      a probability is rounded, because the reference rounds the normalised ones and multiplies their sum with the zero
//      point of V (the two terms cancel);
//   3. probabilities in place, attn.V of the codes, the two full-precision segments;
//   4. partial sums scattered over the cluster by output slice, every CTA finishes its slice in the reference's order of
//      roundings.
// Codes are read straight from global memory (the lanes of a row share their 16-byte loads; the span is on its way into L2
// since the first instruction).  Two CTAs of eight warps per SM.  What bounds it now is the instructions of a warp waiting for each
// other: 14 000 and 9000 of 46 600 cycles in the loops of the two products, 9400 in the two passes over the scores.  16 x 8 heads x
// 3328 bfloat16 keys, 1 bit, with the maximum from the extremes, shares of 16-token tiles, the next words ahead and two chains of
// products together: 32.8 -> 30.7 us; 3 x 8 x 418 at 4 bits 16.7 -> 13.1; 12 x 8 x 1479 fp16 24.6 -> 21.1.  Nothing waits for another
// cluster; waits are bounded.
// The sums of the full-precision scores run over the channels in the order of the loads, so a score may round to the other of two
// neighbouring numbers than in another order; against 64 bits the step is as near either way.
#include <mutex>
#include <type_traits>

#include "cq_cluster.cuh"
#include "cq_common.cuh"
#include "cq_ptx.cuh"
#include "cq_u8_format.cuh"
#include "cq_u8_cluster.cuh"

namespace cq {
namespace calib {
namespace cl {

using namespace ptx;
using namespace cluster;

constexpr int NW = 8, THREADS = NW * 32;
constexpr int ITEM = 64;                        // visual tokens by which the span is dealt out over the cluster
constexpr int MAX_CLUSTER = 8;
constexpr uint32_t WAIT_TRIES = 1u << 22;
constexpr float LOG2E = 1.4426950408889634f;
constexpr int RED_STRIDE = kHeadDim + 4;

struct Args {
  int hq, hkv, n_rep, t_vis, t_fp, t_sys, calibrate, scale_heads;
  int n_items;                 // ceil(t_vis / 64)
  int pitch, fp_pitch;         // score rows in tokens: visual (multiple of 64, + 8), full-precision (multiple of 16, + 8)
  int64_t fp_stride_b, fp_stride_h, mask_stride_b;
  const int32_t* t_fp_dev;
};

__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <typename T>
__device__ __forceinline__ void mma_t(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {   // rows 8..15 unused
  if constexpr (std::is_same<T, __nv_bfloat16>::value) mma_bf16(d, a0, 0u, a2, 0u, b0, b1);
  else mma_f16(d, a0, 0u, a2, 0u, b0, b1);
}

// Rows of a cluster-wide reduction: (max, min or sum) per head and CTA.
struct Pair { float a, b; };

template <typename T, int BITS>
__global__ void __launch_bounds__(THREADS, 2)
u8_step_kernel(const Args a, const T* q, const uint8_t* enc_k, const uint8_t* enc_v, const T* scale_k, const T* zp_k,
               const T* scale_v, const T* zp_v, const T* k_fp, const T* v_fp, const T* mask,
               __nv_bfloat16* __restrict__ out, int* __restrict__ status) {
  using SS = StepScore<T>;
  using SO = typename SS::type;
  constexpr int SB = sizeof(SO);
  constexpr int ROWB = kHeadDim * BITS / 8, WORDS = ROWB / 4;
  constexpr uint32_t FIELD = (1u << BITS) - 1u;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar[3];
  __shared__ float w_s[kMaxRep][kHeadDim];                           // rnd(q * scale_key); later the sums of two segments
  __shared__ float bias_s[kMaxRep];
  __shared__ float red_s[NW][kMaxRep][2];
  __shared__ Pair peer_s[2][MAX_CLUSTER][kMaxRep];
  __shared__ float m_s[kMaxRep], f_s[kMaxRep], e_s[kMaxRep], psum_s[NW][kMaxRep];
  __shared__ float recv_s[3][kMaxRep * kHeadDim + MAX_CLUSTER];      // codes, system, text: [source CTA][slice element]
  __shared__ float recv_p[MAX_CLUSTER][kMaxRep];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int rank = (int)cluster_rank(), S = (int)cluster_size();
  const int pair = blockIdx.x / S, b = pair / a.hkv, hk = pair % a.hkv;
  const int64_t row0 = (int64_t)b * a.hq + (int64_t)hk * a.n_rep;
  const int i0 = rank * a.n_items / S, n_it = (rank + 1) * a.n_items / S - i0;
  const int tok0 = i0 * ITEM, n_tok = min(n_it * ITEM, a.t_vis - tok0);      // may be <= 0 without items

  // on its way during the set-up; a launch before this one may still be advancing the live count, which is good enough for a
  // prefetch and read again behind the wait
  int live = a.t_fp_dev ? *reinterpret_cast<const volatile int32_t*>(a.t_fp_dev) : a.t_fp;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bar[i], S);
    mbar_fence_init();
  }
  __syncthreads();
  cluster_arrive();
  const uint8_t* ek = enc_k + ((int64_t)pair * a.t_vis + tok0) * ROWB;
  const uint8_t* ev = enc_v + ((int64_t)pair * a.t_vis + tok0) * ROWB;
  for (int i = tid; i < n_tok * ROWB / 128; i += THREADS) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(ek + (int64_t)i * 128));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(ev + (int64_t)i * 128));
  }
  // this CTA's share of the full-precision tokens (16-token tiles dealt out over the cluster)
  int t_fp, n_f, f0;
  int64_t fp_off;
  auto fp_range = [&]() {
    t_fp = min(live, a.t_fp);
    const int n_t16 = (t_fp + 15) / 16;
    f0 = rank * n_t16 / S * 16;
    n_f = min(t_fp, (rank + 1) * n_t16 / S * 16) - f0;
    fp_off = (int64_t)b * a.fp_stride_b + (int64_t)hk * a.fp_stride_h + (int64_t)f0 * kHeadDim;
  };
  fp_range();
  for (int i = tid; i < n_f * 4; i += THREADS)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(((i & 1) ? v_fp : k_fp) + fp_off + (int64_t)(i >> 1) * 64));

  unsigned char* sc_b = smem;                                               // scores [n_rep][pitch] of SO
  float* fs = reinterpret_cast<float*>(smem + (size_t)a.n_rep * a.pitch * SB);   // full-precision scores [n_rep][fp_pitch]
  T* fpr = reinterpret_cast<T*>(fs);                                        // ... later their probabilities, [n_rep][2*fp_pitch]
  pdl_wait();
  if (a.t_fp_dev) live = *reinterpret_cast<const volatile int32_t*>(a.t_fp_dev);

  // ---- query side: weights rnd(q * scale_key), bias_k = rnd(rnd(sum rnd(rnd(scale*zp) * q)) / sqrt(D))
  if (warp < a.n_rep) {
    const int r = warp;
    const int64_t srow = a.scale_heads == a.hq ? row0 + r : (int64_t)b * a.scale_heads + hk;
    float bs = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = lane + 32 * i;
      const float qv = Elem<T>::to_f(q[(row0 + r) * kHeadDim + d]);
      const float sk = Elem<T>::to_f(scale_k[srow * kHeadDim + d]), zk = Elem<T>::to_f(zp_k[srow * kHeadDim + d]);
      bs += rnd<T>(rnd<T>(sk * zk) * qv);
      w_s[r][d] = rnd<T>(qv * sk);
    }
    bs = warp_sum(bs);
    if (lane == 0) bias_s[r] = rnd<T>(__fdiv_rn(rnd<T>(bs), 11.313708498984761f));
  }
  __syncthreads();
  fp_range();

  // this warp's share of the CTA's 16-token tiles, in both products
  const int n_m16 = n_tok > 0 ? (n_tok + 15) / 16 : 0, m_first = warp * n_m16 / NW, m_last = (warp + 1) * n_m16 / NW;

  // ================= 1. visual scores =================
  // A register (two k values of one token) = one AND of the token's code word; B carries the weights in the channel order
  // that follows, times the power of two of the field's position (every product weighs 2^-20)
  {
    uint32_t b0[8], b1[8];
#pragma unroll
    for (int kb = 0; kb < 8; ++kb) {
      float v[4];
#pragma unroll
      for (int slot = 0; slot < 4; ++slot) {
        int chan, pos;
        LutMap<BITS>::get(kb, c, slot, chan, pos);
        v[slot] = g < a.n_rep ? w_s[g][chan] * __uint_as_float((uint32_t)(127 + 4 - pos) << 23) : 0.f;
      }
      const __half2 lo = __floats2half2_rn(v[0], v[1]), hi = __floats2half2_rn(v[2], v[3]);
      b0[kb] = *reinterpret_cast<const uint32_t*>(&lo);
      b1[kb] = *reinterpret_cast<const uint32_t*>(&hi);
    }
    const uint32_t m_a0 = BITS == 4 ? 0x000f000fu : (FIELD << (2 * c)) * 0x00010001u;
    const uint32_t m_a2 = BITS == 1 ? (1u << (2 * c + 1)) * 0x00010001u : m_a0;
    const int sh4 = 4 * (c & 1) + 8 * (c >> 1);
    const float bias[2] = {2 * c < a.n_rep ? bias_s[2 * c] : 0.f, 2 * c + 1 < a.n_rep ? bias_s[2 * c + 1] : 0.f};
    float lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY};
    // The warps take contiguous shares of the 16-token tiles (dealt out as items of 64 tokens, four rounds of eight warps were 3.25
    // items' work), MT at a time, and request the words of the next ones before they work on those at hand.
    constexpr int MT = BITS == 1 ? 2 : 1;
    struct Words { uint32_t w[MT][2][WORDS]; };
    auto load = [&](Words& W, int m0) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int t = min(16 * (m0 + m) + g + 8 * hf, n_tok - 1);
          const uint4* rp = reinterpret_cast<const uint4*>(ek + (int64_t)t * ROWB);
#pragma unroll
          for (int q4 = 0; q4 < WORDS / 4; ++q4) {
            const uint4 v = rp[q4];
            W.w[m][hf][4 * q4] = v.x; W.w[m][hf][4 * q4 + 1] = v.y; W.w[m][hf][4 * q4 + 2] = v.z; W.w[m][hf][4 * q4 + 3] = v.w;
          }
        }
    };
    auto compute = [&](const Words& W, int m0) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};       // a tile past the share computes along, so that the chains of two interleave
#pragma unroll
        for (int kb = 0; kb < 8; ++kb) {
          uint32_t a0, a1, a2, a3;
          if (BITS == 1) {
            const uint32_t x0 = W.w[m][0][kb >> 1] >> (8 * (kb & 1)), x1 = W.w[m][1][kb >> 1] >> (8 * (kb & 1));
            a0 = x0 & m_a0; a1 = x1 & m_a0; a2 = x0 & m_a2; a3 = x1 & m_a2;
          } else if (BITS == 2) {
            const uint32_t x0 = W.w[m][0][kb], x1 = W.w[m][1][kb];
            a0 = x0 & m_a0; a1 = x1 & m_a0; a2 = (x0 >> 8) & m_a0; a3 = (x1 >> 8) & m_a0;
          } else {
            a0 = (W.w[m][0][2 * kb] >> sh4) & m_a0; a1 = (W.w[m][1][2 * kb] >> sh4) & m_a0;
            a2 = (W.w[m][0][2 * kb + 1] >> sh4) & m_a0; a3 = (W.w[m][1][2 * kb + 1] >> sh4) & m_a0;
          }
          mma_f16(acc, a0, a1, a2, a3, b0[kb], b1[kb]);
        }
        // acc[0..1] = (token g, heads 2c, 2c+1), acc[2..3] = (token g+8, same heads): fp16 product, / sqrt(D) (a product
        // with the fp32 reciprocal: one score in 4000 lands on the neighbouring fp16 value), - bias_k in the score type
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = 2 * c + (e & 1), t = 16 * (m0 + m) + g + 8 * (e >> 1);
          if (r < a.n_rep && t < n_tok && m0 + m < m_last) {
            const float v = SS::r(rnd<__half>(rnd<__half>(acc[e] * 1048576.f) * 0.08838834764831845f) - bias[e & 1]);
            reinterpret_cast<SO*>(sc_b)[r * a.pitch + t] = SS::make(v);
            lo[e & 1] = fminf(lo[e & 1], v);
            hi[e & 1] = fmaxf(hi[e & 1], v);
          }
        }
      }
    };
    if (BITS == 1) {
      Words W0, W1;
      if (m_first < m_last) load(W0, m_first);
#pragma unroll 1
      for (int m = m_first; m < m_last; m += 2 * MT) {
        if (m + MT < m_last) load(W1, m + MT);
        compute(W0, m);
        if (m + 2 * MT < m_last) load(W0, m + 2 * MT);
        if (m + MT < m_last) compute(W1, m + MT);
      }
    } else if (BITS == 2) {      // one body and moves: 8 x 8 x 2000 tokens 17.3 -> 16.8 us, 16 x 8 x 3328 33.6 -> 32.4
      Words W;
      if (m_first < m_last) load(W, m_first);
#pragma unroll 1
      for (int m = m_first; m < m_last; m += MT) {
        Words next;
        load(next, min(m + MT, m_last - 1));
        compute(W, m);
        W = next;
      }
    } else {                     // no registers for words ahead
#pragma unroll 1
      for (int m = m_first; m < m_last; m += MT) { Words W; load(W, m); compute(W, m); }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        lo[i] = fminf(lo[i], __shfl_xor_sync(0xffffffffu, lo[i], o));
        hi[i] = fmaxf(hi[i], __shfl_xor_sync(0xffffffffu, hi[i], o));
      }
      if (g == 0) { red_s[warp][2 * c + i][0] = lo[i]; red_s[warp][2 * c + i][1] = hi[i]; }
    }
  }
  __syncthreads();
  cluster_wait();
  // a per-head pair of this CTA to every peer, then one arrival per peer
  auto push = [&](int slot, auto value) {
    if (tid < S * a.n_rep) {
      const int peer = tid / a.n_rep, h = tid % a.n_rep;
      const Pair v = value(h);
      st_peer2(map_peer(smem_u32(&peer_s[slot][rank][h]), peer), v.a, v.b);
    }
    __syncthreads();
    if (tid < S) arrive_peer(map_peer(smem_u32(&bar[slot]), tid));
  };
  bool failed = false;
  auto wait = [&](int slot) {
    if (!wait_peers(&bar[slot], WAIT_TRIES)) {
      failed = true;
      if (tid == 0) atomicExch(status, CQ_ERR_TIMEOUT);
    }
  };
  push(0, [&](int h) {
    Pair p{INFINITY, -INFINITY};
#pragma unroll
    for (int w = 0; w < NW; ++w) { p.a = fminf(p.a, red_s[w][h][0]); p.b = fmaxf(p.b, red_s[w][h][1]); }
    return p;
  });

  // ---- full-precision scores of this CTA's tokens: rnd(rnd(q . k) / sqrt(D)) + mask.  Keys (and values below) in pieces of 16 (8)
  // bytes; a lane's piece holds neighbouring channels, which the products take in the order they come
  const bool q_wide = reinterpret_cast<uintptr_t>(q) % 16 == 0;
  const int n_ft = (n_f + 15) / 16;
  const T* mrow = mask ? mask + (int64_t)b * a.mask_stride_b : nullptr;
  for (int ft = warp; ft < n_ft; ft += NW) {
    const T* qrow = q + (row0 + (g < a.n_rep ? g : 0)) * kHeadDim + 8 * c;
    const T* k_lo = k_fp + fp_off + (int64_t)min(16 * ft + g, n_f - 1) * kHeadDim + 8 * c;
    const T* k_hi = k_fp + fp_off + (int64_t)min(16 * ft + g + 8, n_f - 1) * kHeadDim + 8 * c;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    uint4 lo[4], hi[4], qv[4];      // channels 32m + 8c .. + 7: four pairs, two k-steps
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      lo[m] = *reinterpret_cast<const uint4*>(k_lo + 32 * m);
      hi[m] = *reinterpret_cast<const uint4*>(k_hi + 32 * m);
      if (q_wide) {                 // columns past the last head repeat the first; they are not kept
        qv[m] = *reinterpret_cast<const uint4*>(qrow + 32 * m);
      } else {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(qrow + 32 * m);
        qv[m] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        mma_bf16(acc, lo[m].x, hi[m].x, lo[m].y, hi[m].y, qv[m].x, qv[m].y);
        mma_bf16(acc, lo[m].z, hi[m].z, lo[m].w, hi[m].w, qv[m].z, qv[m].w);
      } else {
        mma_f16(acc, lo[m].x, hi[m].x, lo[m].y, hi[m].y, qv[m].x, qv[m].y);
        mma_f16(acc, lo[m].z, hi[m].z, lo[m].w, hi[m].w, qv[m].z, qv[m].w);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int h = 2 * c + (e & 1), t = 16 * ft + g + 8 * (e >> 1);
      if (h < a.n_rep) {
        float v = -INFINITY;
        if (t < n_f) {
          v = rnd<T>(__fdiv_rn(rnd<T>(acc[e]), 11.313708498984761f));
          const int f = f0 + t;
          if (mrow) v = SS::r(v + Elem<T>::to_f(mrow[f < a.t_sys ? f : a.t_vis + f]));
        }
        fs[h * a.fp_pitch + t] = v;
      }
    }
  }

  // ================= 2. calibration, mask, local maximum and sum of exponentials =================
  wait(0);
  const int n_vec = n_it * (ITEM / 8);
  auto load8 = [&](int h, int v, float (&x)[8]) {
    const unsigned char* p = sc_b + (size_t)(h * a.pitch + 8 * v) * SB;
    if constexpr (SB == 2) {
      const uint4 w = *reinterpret_cast<const uint4*>(p);
      const __half2* h2 = reinterpret_cast<const __half2*>(&w);
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = __half22float2(h2[j]); x[2 * j] = f.x; x[2 * j + 1] = f.y; }
    } else {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float4 f = reinterpret_cast<const float4*>(p)[j];
        x[4 * j] = f.x; x[4 * j + 1] = f.y; x[4 * j + 2] = f.z; x[4 * j + 3] = f.w;
      }
    }
  };
  __syncthreads();      // every warp's full-precision scores
  // fp16 rows without a mask round the calibration's product and sum once (against 64-bit arithmetic 8 x 1024 keys at 1 bit are
  // off by 4.36e-3, with two roundings by 4.59e-3) and take a product with the reciprocal, which for numbers of 11 significant
  // bits rounds to the same fp16 number as the quotient.  Other rows round every operation; their quotient is that product
  // corrected by its residual (Markstein 1990), 1.2 us less than divisions at 16 x 8 heads x 3328 bfloat16 keys.
  // Without a mask the calibration is monotonous, so the largest calibrated score is that of one of the extremes, and known before
  // the pass that calibrates, which then sums the exponentials as well; in fp32 rows it leaves them in place of the scores, and the
  // later pass multiplies them.  (Calibration, sum and probabilities as three passes, two of them with exponentials, took 11 300
  // cycles of 50 200 at 16 x 8 heads x 3328 keys; now 9400.)
  const bool early = !mrow;
  struct Calib { float lo, hi, span, denom, rden; };
  auto calib_of = [&](int h) {
    Calib k{INFINITY, -INFINITY, 0.f, 0.f, 0.f};
    for (int p = 0; p < S; ++p) { k.lo = fminf(k.lo, peer_s[0][p][h].a); k.hi = fmaxf(k.hi, peer_s[0][p][h].b); }
    k.span = SS::r(SS::r(k.hi + -3.f) - k.lo);
    k.denom = SS::r(SS::r(k.hi - k.lo) + 1e-8f);
    k.rden = 1.f / k.denom;
    return k;
  };
  auto calibrated = [&](float x, const Calib& k) {
    const float d = SS::r(x - k.lo), n = d * k.rden;
    return SS::r(SS::r(SS::r(fmaf(fmaf(-n, k.denom, d), k.rden, n)) * k.span) + k.lo);
  };
  auto calibrated2 = [&](float x, float y, const Calib& k) {      // two of an fp16 row without a mask
    const __half2 lo2 = __float2half2_rn(k.lo);
    const float2 d = __half22float2(__hsub2(__floats2half2_rn(x, y), lo2));
    return __half22float2(__hfma2(__floats2half2_rn(d.x * k.rden, d.y * k.rden), __float2half2_rn(k.span), lo2));
  };
  auto store8 = [&](int h, int v, const float (&x)[8]) {
    unsigned char* p = sc_b + (size_t)(h * a.pitch + 8 * v) * SB;
    if constexpr (SB == 2) {
      uint4 w;
      __half2* h2 = reinterpret_cast<__half2*>(&w);
#pragma unroll
      for (int j = 0; j < 4; ++j) h2[j] = __floats2half2_rn(x[2 * j], x[2 * j + 1]);
      *reinterpret_cast<uint4*>(p) = w;
    } else {
#pragma unroll
      for (int j = 0; j < 2; ++j) reinterpret_cast<float4*>(p)[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
    }
  };
  if (early) {
    if (warp < a.n_rep) {
      const Calib k = calib_of(warp);
      float m = k.hi;
      if (a.calibrate) {
        const float2 y = SB == 2 ? calibrated2(k.lo, k.hi, k) : make_float2(calibrated(k.lo, k), calibrated(k.hi, k));
        m = fmaxf(y.x, y.y);
      }
      for (int t = lane; t < n_f; t += 32) m = fmaxf(m, fs[warp * a.fp_pitch + t]);
      m = warp_max(m);
      if (lane == 0) m_s[warp] = m;
    }
    __syncthreads();
    for (int h = 0; h < a.n_rep; ++h) {
      const Calib k = calib_of(h);
      const float m = m_s[h], ml = m == -INFINITY ? 0.f : m * LOG2E;
      float l = 0.f;
      for (int v = (tid + 256 - (h * n_vec & 255)) & 255; v < n_vec; v += THREADS) {
        float x[8];
        load8(h, v, x);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          if (a.calibrate) {
            const float2 y = SB == 2 ? calibrated2(x[j], x[j + 1], k) : make_float2(calibrated(x[j], k), calibrated(x[j + 1], k));
            x[j] = y.x; x[j + 1] = y.y;
          }
#pragma unroll
          for (int i = j; i < j + 2; ++i) {
            if (8 * v + i >= n_tok) x[i] = -INFINITY;
            const float e = ex2(fmaf(x[i], LOG2E, -ml));
            l += e;
            if (SB == 4) x[i] = e;
          }
        }
        store8(h, v, x);
      }
      for (int t = tid; t < n_f; t += THREADS) l += ex2(fmaf(fs[h * a.fp_pitch + t], LOG2E, -ml));
      l = warp_sum(l);
      if (lane == 0) red_s[warp][h][1] = l;
    }
  } else {
    for (int h = 0; h < a.n_rep; ++h) {
      const Calib k = calib_of(h);
      float m = -INFINITY;
      for (int v = (tid + 256 - (h * n_vec & 255)) & 255; v < n_vec; v += THREADS) {
        float x[8];
        load8(h, v, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int t = 8 * v + j;
          if (a.calibrate) x[j] = calibrated(x[j], k);
          if (t < n_tok) x[j] = SS::r(x[j] + Elem<T>::to_f(mrow[a.t_sys + tok0 + t]));
          else x[j] = -INFINITY;
          m = fmaxf(m, x[j]);
        }
        store8(h, v, x);
      }
      for (int t = tid; t < n_f; t += THREADS) m = fmaxf(m, fs[h * a.fp_pitch + t]);
      m = warp_max(m);
      if (lane == 0) red_s[warp][h][0] = m;
    }
    __syncthreads();
    if (tid < a.n_rep) {
      float m = -INFINITY;
#pragma unroll
      for (int w = 0; w < NW; ++w) m = fmaxf(m, red_s[w][tid][0]);
      m_s[tid] = m;
    }
    __syncthreads();
    for (int h = 0; h < a.n_rep; ++h) {
      const float m = m_s[h], ml = m == -INFINITY ? 0.f : m * LOG2E;
      float l = 0.f;
      for (int v = (tid + 256 - (h * n_vec & 255)) & 255; v < n_vec; v += THREADS) {
        float x[8];
        load8(h, v, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) l += ex2(fmaf(x[j], LOG2E, -ml));
      }
      for (int t = tid; t < n_f; t += THREADS) l += ex2(fmaf(fs[h * a.fp_pitch + t], LOG2E, -ml));
      l = warp_sum(l);
      if (lane == 0) red_s[warp][h][1] = l;
    }
  }
  __syncthreads();
  push(1, [&](int h) {
    float l = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) l += red_s[w][h][1];
    return Pair{m_s[h], l};
  });
  wait(1);
  if (tid < a.n_rep) {
    float m = -INFINITY, l = 0.f;
    for (int p = 0; p < S; ++p) m = fmaxf(m, peer_s[1][p][tid].a);
    for (int p = 0; p < S; ++p) {
      const Pair v = peer_s[1][p][tid];
      if (v.a != -INFINITY) l += v.b * exp2f((v.a - m) * LOG2E);
    }
    e_s[tid] = exp2f((m_s[tid] - m) * LOG2E) / l;      // what turns this CTA's exponentials into probabilities
    m_s[tid] = m;
    f_s[tid] = 1.f / l;
  }
  __syncthreads();

  // ================= 3. probabilities, attn.V =================
  // in place: the 8 tokens of a vector become 16 bytes of fp16 at the vector's first byte
  for (int h = 0; h < a.n_rep; ++h) {
    const float ml = m_s[h] * LOG2E, inv = f_s[h], scale = e_s[h];
    float ps = 0.f;
    for (int v = (tid + 256 - (h * n_vec & 255)) & 255; v < n_vec; v += THREADS) {
      float x[8];
      load8(h, v, x);
      uint4 w;
      __half2* h2 = reinterpret_cast<__half2*>(&w);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p0 = rnd<T>(SB == 4 && early ? x[2 * j] * scale : ex2(fmaf(x[2 * j], LOG2E, -ml)) * inv);
        const float p1 = rnd<T>(SB == 4 && early ? x[2 * j + 1] * scale : ex2(fmaf(x[2 * j + 1], LOG2E, -ml)) * inv);
        ps += p0 + p1;
        h2[j] = __floats2half2_rn(p0, p1);
      }
      *reinterpret_cast<uint4*>(sc_b + (size_t)(h * a.pitch + 8 * v) * SB) = w;
    }
    ps = warp_sum(ps);
    if (lane == 0) psum_s[warp][h] = ps;
    // the full-precision probabilities in the data type: element t of a row replaces half of the float t / 2, which only
    // this warp-strided pass reads, so a warp takes whole rows
    if (warp == (h & (NW - 1)))
      for (int t0 = 0; t0 < 16 * n_ft; t0 += 32) {
        const int t = t0 + lane;
        const float x = t < 16 * n_ft ? fs[h * a.fp_pitch + t] : -INFINITY;
        __syncwarp();
        if (t < 16 * n_ft) fpr[h * 2 * a.fp_pitch + t] = Elem<T>::from_f(ex2(fmaf(x, LOG2E, -ml)) * inv);
        __syncwarp();
      }
  }
  __syncthreads();

  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 32; ++i) (&acc[0][0])[i] = 0.f;
  {
    // A = codes (rows = channels, k = tokens): one byte permute pairs two token rows, rows g / g+8 are adjacent fields of
    // byte g/2 (4 bits: the nibbles of byte g%4 of the words 2(g/4), 2(g/4)+1 of every 32-channel quarter)
    const uint32_t byte = BITS == 4 ? (uint32_t)(g & 3) : (uint32_t)(g >> 1);
    const uint32_t sel = byte | (byte << 4) | ((4 + byte) << 8) | ((4 + byte) << 12);
    constexpr int NM = BITS == 1 ? 2 : 1;
    uint32_t m0[NM], m1[NM];
#pragma unroll
    for (int i = 0; i < NM; ++i) {
      const int p0 = BITS == 4 ? 0 : 4 * (g & 1) + 2 * i;
      m0[i] = (FIELD << p0) * 0x00010001u;
      m1[i] = (FIELD << (p0 + BITS)) * 0x00010001u;
    }
    const unsigned char* prow = sc_b + (size_t)((g < a.n_rep ? g : 0) * a.pitch) * SB;
    struct Words { uint32_t w[4][WORDS]; };       // rows of tokens 2c, 2c+1, 2c+8, 2c+9 (4 bits: the lane's word pairs)
    auto load = [&](Words& W, int m) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {               // tokens past the end have p = 0
        const uint8_t* r = ev + (int64_t)min(16 * m + 2 * c + (i & 1) + 8 * (i >> 1), n_tok - 1) * ROWB;
        if (BITS == 4) {
#pragma unroll
          for (int qd = 0; qd < 4; ++qd) {
            const uint2 v = *reinterpret_cast<const uint2*>(r + 16 * qd + 8 * (g >> 2));
            W.w[i][2 * qd] = v.x; W.w[i][2 * qd + 1] = v.y;
          }
        } else {
#pragma unroll
          for (int q4 = 0; q4 < WORDS / 4; ++q4) {
            const uint4 v = reinterpret_cast<const uint4*>(r)[q4];
            W.w[i][4 * q4] = v.x; W.w[i][4 * q4 + 1] = v.y; W.w[i][4 * q4 + 2] = v.z; W.w[i][4 * q4 + 3] = v.w;
          }
        }
      }
    };
    auto compute = [&](const Words& W, int m) {   // columns past the last head take the first one's; they are not kept
      const uint32_t p0 = *reinterpret_cast<const uint32_t*>(prow + (size_t)(16 * m) * SB + 4 * c);
      const uint32_t p1 = *reinterpret_cast<const uint32_t*>(prow + (size_t)(16 * m + 8) * SB + 4 * c);
      constexpr int NWD = 8 / NM;                 // words a row: m-tiles NM wd .. NM wd + NM - 1
#pragma unroll
      for (int wd = 0; wd < NWD; ++wd) {
        const uint32_t x = prmt(W.w[0][wd], W.w[1][wd], sel), y = prmt(W.w[2][wd], W.w[3][wd], sel);
#pragma unroll
        for (int i = 0; i < NM; ++i)
          mma_f16(acc[wd * NM + i], x & m0[i], x & m1[i], y & m0[i], y & m1[i], p0, p1);
      }
    };
    if (BITS == 1) {                              // the next tile's words are requested ahead; more bits leave no registers for it
      Words W0, W1;
      if (m_first < m_last) load(W0, m_first);
#pragma unroll 1
      for (int m = m_first; m < m_last; m += 2) {
        if (m + 1 < m_last) load(W1, m + 1);
        compute(W0, m);
        if (m + 2 < m_last) load(W0, m + 2);
        if (m + 1 < m_last) compute(W1, m + 1);
      }
    } else {
#pragma unroll 1                                  // two bodies at 2 bits: 8 x 8 x 2000 tokens 18.2 us, one 17.3
      for (int m = m_first; m < m_last; ++m) { Words W; load(W, m); compute(W, m); }
    }
  }
  // full-precision segments: warp w owns channels 32 (w / 2) .. + 31 of every other 16 tokens; system and text keys are summed
  // apart, as the reference adds their rounded products one after the other
  float fo[2][4][4] = {};
  {
    const T* vf = v_fp + fp_off + 32 * (warp >> 1) + 4 * g;
    const T* prow = fpr + (size_t)(g < a.n_rep ? g : 0) * 2 * a.fp_pitch + 2 * c;
    const int n_sys = min(max(min(a.t_sys, t_fp) - f0, 0), n_f);
#pragma unroll 2
    for (int ft = warp & 1; ft < n_ft; ft += 2) {
      uint2 v[4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
        v[r] = *reinterpret_cast<const uint2*>(vf + (int64_t)min(16 * ft + 2 * c + (r & 1) + 8 * (r >> 1), n_f - 1) * kHeadDim);
      const uint32_t p[2] = {*reinterpret_cast<const uint32_t*>(prow + 16 * ft), *reinterpret_cast<const uint32_t*>(prow + 16 * ft + 8)};
#pragma unroll
      for (int seg = 0; seg < 2; ++seg) {
        if (seg == 0 ? 16 * ft >= n_sys : 16 * ft + 16 <= n_sys) continue;
        uint32_t ps[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = 16 * ft + 8 * i + 2 * c;
          const uint32_t keep = ((t < n_sys) == (seg == 0) ? 0xffffu : 0u) | ((t + 1 < n_sys) == (seg == 0) ? 0xffff0000u : 0u);
          ps[i] = p[i] & keep;
        }
        // n-tile j: column n stands for channel 32 (w / 2) + 4n + j
        mma_t<T>(fo[seg][0], ps[0], ps[1], prmt(v[0].x, v[1].x, 0x5410), prmt(v[2].x, v[3].x, 0x5410));
        mma_t<T>(fo[seg][1], ps[0], ps[1], prmt(v[0].x, v[1].x, 0x7632), prmt(v[2].x, v[3].x, 0x7632));
        mma_t<T>(fo[seg][2], ps[0], ps[1], prmt(v[0].y, v[1].y, 0x5410), prmt(v[2].y, v[3].y, 0x5410));
        mma_t<T>(fo[seg][3], ps[0], ps[1], prmt(v[0].y, v[1].y, 0x7632), prmt(v[2].y, v[3].y, 0x7632));
      }
    }
  }
  __syncthreads();      // scores and probabilities have been used: their memory holds the warps' sums from here on
  float* red = reinterpret_cast<float*>(smem);                          // [warp][head][RED_STRIDE]
  float* seg_s = red + NW * a.n_rep * RED_STRIDE;                       // [token parity][system | text][head][channel]
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    constexpr int NM = BITS == 1 ? 2 : 1;
    int d0, d1;
    float s0, s1;
    if (BITS == 4) {
      const int W = 4 * (j >> 1) + 2 * (g >> 2) + (j & 1);
      d0 = 8 * W + 2 * (g & 3) + 1; d1 = 8 * W + 2 * (g & 3);
      s0 = 16777216.f; s1 = 1048576.f;
    } else {            // MSB first: the field at bit p of byte y is channel (8/BITS)*y + 8/BITS - 1 - p/BITS
      const int p0 = 4 * (g & 1) + 2 * (j % NM), base = (j / NM) * (32 / BITS) + (8 / BITS) * (g >> 1) + 8 / BITS - 1;
      d0 = base - p0 / BITS; d1 = base - (p0 + BITS) / BITS;
      s0 = __uint_as_float((uint32_t)(127 + 24 - p0) << 23); s1 = __uint_as_float((uint32_t)(127 + 24 - p0 - BITS) << 23);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (2 * c + e < a.n_rep) {
        float* row = red + (warp * a.n_rep + 2 * c + e) * RED_STRIDE;
        row[d0] = acc[j][e] * s0;
        row[d1] = acc[j][2 + e] * s1;
      }
  }
  if (g < a.n_rep) {
#pragma unroll
    for (int seg = 0; seg < 2; ++seg)
#pragma unroll
      for (int i = 0; i < 2; ++i)      // fragment columns 2c, 2c+1 of n-tile j = channels 32 (w / 2) + 8c + j, + 4
        *reinterpret_cast<float4*>(seg_s + (((warp & 1) * 2 + seg) * a.n_rep + g) * kHeadDim + 32 * (warp >> 1) + 8 * c + 4 * i) =
            make_float4(fo[seg][0][i], fo[seg][1][i], fo[seg][2][i], fo[seg][3][i]);
  }
  __syncthreads();

  // ================= 4. sums over the cluster, output =================
  const int n_out = a.n_rep * kHeadDim, slice = (n_out + S - 1) / S;
  for (int e = tid; e < n_out; e += THREADS) {
    const int h = e >> 7, d = e & 127, peer = e / slice, at = rank * slice + e % slice;
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) o += red[(w * a.n_rep + h) * RED_STRIDE + d];
    st_peer(map_peer(smem_u32(&recv_s[0][at]), peer), o);
    st_peer(map_peer(smem_u32(&recv_s[1][at]), peer), seg_s[h * kHeadDim + d] + seg_s[(2 * a.n_rep + h) * kHeadDim + d]);
    st_peer(map_peer(smem_u32(&recv_s[2][at]), peer), seg_s[(a.n_rep + h) * kHeadDim + d] + seg_s[(3 * a.n_rep + h) * kHeadDim + d]);
    if (d < S) {
      float ps = 0.f;
#pragma unroll
      for (int w = 0; w < NW; ++w) ps += psum_s[w][h];
      st_peer(map_peer(smem_u32(&recv_p[rank][h]), d), ps);
    }
  }
  __syncthreads();
  if (tid < S) arrive_peer(map_peer(smem_u32(&bar[2]), tid));
  wait(2);
  if (failed) {
    cluster_arrive();      // a late peer may still store into this CTA's shared memory
    cluster_wait();
    return;
  }
  for (int i = tid; i < slice && rank * slice + i < n_out; i += THREADS) {
    const int e = rank * slice + i, h = e >> 7, d = e & 127;
    float acc_v = 0.f, sys = 0.f, txt = 0.f, ps = 0.f;
    for (int p = 0; p < S; ++p) {
      acc_v += recv_s[0][p * slice + i];
      sys += recv_s[1][p * slice + i];
      txt += recv_s[2][p * slice + i];
      ps += recv_p[p][h];
    }
    const int64_t srow = a.scale_heads == a.hq ? row0 + h : (int64_t)b * a.scale_heads + hk;
    const float sv = Elem<T>::to_f(scale_v[srow * kHeadDim + d]), zv = Elem<T>::to_f(zp_v[srow * kHeadDim + d]);
    float o = SS::r(rnd<__half>(acc_v) * sv);
    o = SS::r(o - rnd<T>(rnd<T>(sv * zv) * rnd<T>(ps)));
    o = SS::r(o + rnd<T>(sys));
    o = SS::r(o + rnd<T>(txt));
    out[row0 * kHeadDim + e] = __float2bfloat16_rn(o);
  }
}

// ---- host side ---------------------------------------------------------------------------------------------
struct Plan { int S, pitch, fp_pitch, smem; };

// Clusters as for the group format: the largest with which the grid is resident at once; where the batch alone fills
// the GPU, one CTA per KV head, or as many as its scores need.
inline bool make_plan(const cq_u8_decode_args* a, Plan* p) {
  const int n_rep = a->n_q_heads / a->n_kv_heads, n_items = (a->t_vis + ITEM - 1) / ITEM, sb = a->dtype == CQ_DTYPE_F16 ? 2 : 4;
  const int64_t pairs = (int64_t)a->batch * a->n_kv_heads;
  int S = MAX_CLUSTER;
  while (S > 1 && (pairs > max_clusters(S) || S > n_items)) S /= 2;
  for (; S <= MAX_CLUSTER; S *= 2) {
    p->S = S;
    p->pitch = (n_items + S - 1) / S * ITEM + 8;
    p->fp_pitch = ((a->t_fp + 15) / 16 + S - 1) / S * 16 + 8;
    const size_t rows = (size_t)n_rep * ((size_t)p->pitch * sb + (size_t)p->fp_pitch * 4);
    const size_t red = (size_t)(NW * n_rep * RED_STRIDE + 4 * n_rep * kHeadDim) * 4;
    const size_t smem = rows > red ? rows : red;
    if (smem <= 88 * 1024) { p->smem = (int)smem; return true; }
  }
  return false;
}

template <typename T, int BITS>
static int launch(const cq_u8_decode_args* a, const Plan& p, int* status, cudaStream_t st) {
  auto kern = u8_step_kernel<T, BITS>;
  static bool configured[64] = {};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return CQ_ERR_LAUNCH;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!configured[dev]) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 88 * 1024) != cudaSuccess) return CQ_ERR_LAUNCH;
      configured[dev] = true;
    }
  }
  Args d;
  d.hq = a->n_q_heads; d.hkv = a->n_kv_heads; d.n_rep = d.hq / d.hkv;
  d.t_vis = a->t_vis; d.t_fp = a->t_fp; d.t_sys = a->t_sys; d.calibrate = a->calibrate ? 1 : 0; d.scale_heads = a->n_scale_heads;
  d.n_items = (a->t_vis + ITEM - 1) / ITEM;
  d.pitch = p.pitch; d.fp_pitch = p.fp_pitch;
  d.fp_stride_b = a->fp_stride_b; d.fp_stride_h = a->fp_stride_h; d.mask_stride_b = a->mask_stride_b;
  d.t_fp_dev = a->t_fp_dev;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((int64_t)a->batch * a->n_kv_heads * p.S));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.S; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  auto t = [](const void* x) { return static_cast<const T*>(x); };
  if (cudaLaunchKernelEx(&cfg, kern, d, t(a->q), a->enc_k, a->enc_v, t(a->scale_key), t(a->zero_point_key), t(a->scale_value),
                         t(a->zero_point_value), t(a->k_fp), t(a->v_fp), t(a->mask), static_cast<__nv_bfloat16*>(a->out),
                         status) != cudaSuccess)
    return CQ_ERR_LAUNCH;
  return check_launch();
}

}  // namespace cl
}  // namespace calib

bool u8_cluster_eligible(const cq_u8_decode_args* a) {
  calib::cl::Plan p;
  if (a->t_vis <= 0 || reinterpret_cast<uintptr_t>(a->q) % 4) return false;
  if (a->t_fp > 0 && (!aligned16(a->k_fp) || !aligned16(a->v_fp) || a->fp_stride_b % 8 || a->fp_stride_h % 8)) return false;
  return calib::cl::make_plan(a, &p);
}

int u8_cluster_run(const cq_u8_decode_args* a, void* status_word, cudaStream_t st) {
  using namespace calib::cl;
  Plan p;
  if (!make_plan(a, &p)) return CQ_ERR_UNSUPPORTED;
  int* status = static_cast<int*>(status_word);
  if (a->dtype == CQ_DTYPE_F16)
    return a->bits == 1 ? launch<__half, 1>(a, p, status, st) : a->bits == 2 ? launch<__half, 2>(a, p, status, st) : launch<__half, 4>(a, p, status, st);
  return a->bits == 1 ? launch<__nv_bfloat16, 1>(a, p, status, st)
         : a->bits == 2 ? launch<__nv_bfloat16, 2>(a, p, status, st) : launch<__nv_bfloat16, 4>(a, p, status, st);
}

}  // namespace cq
