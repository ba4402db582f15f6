// QJL sign-sketch key quantizer and its GQA score estimator (the reference's `qjl` baseline method).
//
// quantize: keys come in groups of G tokens; per group a set of outlier channels is given.  For every
// token the sign bits of  S k_inlier  and  S k_outlier  (S = sketch_dim x 128 projection, k split by
// the outlier mask) are packed LSB-first, 8 per byte, plus the norm of the outlier part.
// score:    for a query q and a key sketched that way
//     score = sqrt(pi/2)/s * |k_in| * sum_p sgn_p * (qS - q_out S)_p  +  sqrt(pi/2)/s_o * |k_out| * sum_{p<s_o} sgn'_p * (q_out S)_p
// with q_out = q restricted to the group's outlier channels and |k_in| = sqrt(|k|^2 - |k_out|^2).
//
// quant_kernel and score_kernel are CUDA-core kernels: one CTA per (group, chunk of 32 tokens); thread =
// (token, block of 32 projections); the sign sums run over "bit set" terms only:
// sum_p sgn_p x_p = 2 sum_{bit_p} x_p - sum_p x_p.  They serve unaligned buffers, sketch dims that are not multiples of
// 128 and, for the quantizer, other groups than 32 keys; otherwise the tcgen05 kernels of cq_qjl_build.cu (quantizer) and
// cq_qjl_score.cu (groups of 32 keys, 256 projections, up to four query heads per KV head), or score_rows_kernel (outlier
// projection and sign sums on the warp MMA, a group per warp) run.
#include <type_traits>

#include "cq_common.cuh"
#include "cq_ptx.cuh"

namespace cq {
namespace qjl_build {      // cq_qjl_build.cu: groups of 32 keys, 256 projections
bool eligible(const void* keys, int group_size, int head_dim, int sketch, int o_sketch, int oc, const int64_t* strides, const void* kq,
              const void* koq);
int run(const void* keys, int batch, int heads, int n_groups, const int64_t* strides, const uint8_t* given, const void* proj, int proj_dtype,
        int o_sketch, int oc, int dtype, uint8_t* idx, uint8_t* kq, uint8_t* koq, void* knorm, void* onorm, cudaStream_t st);
}  // namespace qjl_build
namespace qjl_score {      // cq_qjl_score.cu: groups of 32 keys, 256 projections, up to four query heads per KV head
bool eligible(const uint8_t* kq, const uint8_t* koq, int group_size, int sketch, int o_sketch, int n_rep);
int run(const uint8_t* kq, const uint8_t* koq, const void* kn, const void* kon, const uint8_t* idx, const float* qs, const void* q,
        const void* proj, int proj_dtype, int n_kbh, int n_rep, int n_groups, int o_sketch, int oc, int dtype, float* scores, cudaStream_t st);
}  // namespace qjl_score
namespace qjl {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int MAX_SKETCH = 256;       // projections per token handled by one CTA (32 per warp)
constexpr int D_CHUNK = 16;           // channels of the projection staged per step

template <typename TP> __device__ __forceinline__ float proj_f(TP v);
template <> __device__ __forceinline__ float proj_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float proj_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float proj_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// keys [groups][G][128], outlier_idx [groups][oc], proj [sketch][128] -> key_quant [groups][G][sketch/8],
// key_outlier_quant [groups][G][o_sketch/8], outlier_norm [groups][G]
template <typename T, typename TP>
__global__ void __launch_bounds__(THREADS)
quant_kernel(const T* __restrict__ keys, const uint8_t* __restrict__ outlier_idx, const TP* __restrict__ proj,
             uint8_t* __restrict__ key_quant, uint8_t* __restrict__ key_outlier_quant, T* __restrict__ outlier_norm,
             int G, int sketch, int o_sketch, int oc) {
  __shared__ float key_s[kHeadDim][33];            // [channel][token], padded
  __shared__ float proj_s[D_CHUNK][MAX_SKETCH];    // [channel in chunk][projection]
  __shared__ uint8_t mask_s[kHeadDim];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
  const int64_t grp = blockIdx.x;
  const int tok0 = blockIdx.y * 32;
  const int n_tok = min(32, G - tok0);
  if (tid < kHeadDim) mask_s[tid] = 0;
  __syncthreads();
  if (tid < oc) mask_s[outlier_idx[grp * oc + tid] & (kHeadDim - 1)] = 1;
  const T* kbase = keys + (grp * G + tok0) * kHeadDim;
  for (int i = tid; i < 32 * kHeadDim; i += THREADS) {
    const int t = i >> 7, d = i & (kHeadDim - 1);
    key_s[d][t] = t < n_tok ? Elem<T>::to_f(kbase[t * kHeadDim + d]) : 0.f;
  }
  float acc_in[32], acc_out[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) { acc_in[j] = 0.f; acc_out[j] = 0.f; }
  const int p0 = warp * 32;                         // this warp's projections
  for (int d0 = 0; d0 < kHeadDim; d0 += D_CHUNK) {
    __syncthreads();                                // previous chunk consumed (first pass: key_s, mask_s written)
    for (int i = tid; i < sketch * D_CHUNK; i += THREADS) {
      const int p = i / D_CHUNK, dd = i % D_CHUNK;
      proj_s[dd][p] = proj_f<TP>(proj[(int64_t)p * kHeadDim + d0 + dd]);
    }
    __syncthreads();
    if (p0 < sketch) {
#pragma unroll 4
      for (int dd = 0; dd < D_CHUNK; ++dd) {
        const float kv = key_s[d0 + dd][lane];
        const float4* pr = reinterpret_cast<const float4*>(&proj_s[dd][p0]);
        if (mask_s[d0 + dd]) {                      // uniform over the CTA
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = pr[j];
            acc_out[4 * j] = fmaf(v.x, kv, acc_out[4 * j]); acc_out[4 * j + 1] = fmaf(v.y, kv, acc_out[4 * j + 1]);
            acc_out[4 * j + 2] = fmaf(v.z, kv, acc_out[4 * j + 2]); acc_out[4 * j + 3] = fmaf(v.w, kv, acc_out[4 * j + 3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = pr[j];
            acc_in[4 * j] = fmaf(v.x, kv, acc_in[4 * j]); acc_in[4 * j + 1] = fmaf(v.y, kv, acc_in[4 * j + 1]);
            acc_in[4 * j + 2] = fmaf(v.z, kv, acc_in[4 * j + 2]); acc_in[4 * j + 3] = fmaf(v.w, kv, acc_in[4 * j + 3]);
          }
        }
      }
    }
  }
  if (lane < n_tok && p0 < sketch) {
    uint32_t w_in = 0, w_out = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      w_in |= (acc_in[j] > 0.f ? 1u : 0u) << j;
      w_out |= (acc_out[j] > 0.f ? 1u : 0u) << j;
    }
    const int64_t tok = grp * G + tok0 + lane;
    *reinterpret_cast<uint32_t*>(key_quant + tok * (sketch / 8) + p0 / 8) = w_in;
    if (p0 < o_sketch) *reinterpret_cast<uint32_t*>(key_outlier_quant + tok * (o_sketch / 8) + p0 / 8) = w_out;
  }
  if (warp == 0 && lane < n_tok) {
    float ss = 0.f;
    for (int d = 0; d < kHeadDim; ++d)
      if (mask_s[d]) ss = fmaf(key_s[d][lane], key_s[d][lane], ss);
    outlier_norm[grp * G + tok0 + lane] = Elem<T>::from_f(sqrtf(ss));
  }
}

// One CTA per (batch x KV head, group, chunk of 32 tokens).  R = query heads per KV head held per thread.
template <typename T, typename TP, int R>
__global__ void __launch_bounds__(THREADS)
score_kernel(const uint8_t* __restrict__ key_quant, const uint8_t* __restrict__ key_outlier_quant,
             const T* __restrict__ key_norm, const T* __restrict__ key_outlier_norm,
             const uint8_t* __restrict__ outlier_idx, const float* __restrict__ query_sketch,
             const T* __restrict__ query, const TP* __restrict__ proj_score, float* __restrict__ scores,
             int n_groups, int G, int n_rep, int sketch, int o_sketch, int oc) {
  __shared__ __align__(16) float qin_s[MAX_SKETCH][R];     // (q S - q_out S)_p per head
  __shared__ __align__(16) float qout_s[MAX_SKETCH][R];    // (q_out S)_p per head
  __shared__ float q_s[R][kHeadDim];
  __shared__ float part_s[WARPS][32][2 * R];
  __shared__ float tot_s[2][R];
  __shared__ uint8_t otl_s[kHeadDim];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
  const int64_t kbh = blockIdx.x;                           // batch * n_kv_heads + kv head
  const int n = blockIdx.y, tok0 = blockIdx.z * 32;
  const int n_tok = min(32, G - tok0);
  const int64_t qrow0 = kbh * n_rep;                        // first query head of this KV head
  const int64_t grp = kbh * n_groups + n;
  for (int i = tid; i < R * kHeadDim; i += THREADS) {
    const int r = i >> 7, d = i & (kHeadDim - 1);
    q_s[r][d] = r < n_rep ? Elem<T>::to_f(query[(qrow0 + r) * kHeadDim + d]) : 0.f;
  }
  if (tid < oc) otl_s[tid] = outlier_idx[grp * oc + tid] & (kHeadDim - 1);
  if (tid < 2 * R) tot_s[tid / R][tid % R] = 0.f;
  __syncthreads();
  // sketches of the query's outlier part and of the rest, per projection; their totals per head
  for (int p = tid; p < sketch; p += THREADS) {
    float o[R];
#pragma unroll
    for (int r = 0; r < R; ++r) o[r] = 0.f;
    for (int i = 0; i < oc; ++i) {
      const int d = otl_s[i];
      const float pv = proj_f<TP>(proj_score[(int64_t)d * sketch + p]);
#pragma unroll
      for (int r = 0; r < R; ++r) o[r] = fmaf(q_s[r][d], pv, o[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float qs = r < n_rep ? query_sketch[(qrow0 + r) * sketch + p] : 0.f;
      qin_s[p][r] = qs - o[r];
      qout_s[p][r] = o[r];
    }
  }
  __syncthreads();
  // totals per head over the projections: (which, head) pairs dealt over the warps, lanes stride p
  for (int pr = warp; pr < 2 * R; pr += WARPS) {
    const int which = pr / R, r = pr % R;
    const int lim = which == 0 ? sketch : o_sketch;
    float t = 0.f;
    for (int p = lane; p < lim; p += 32) t += which == 0 ? qin_s[p][r] : qout_s[p][r];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) tot_s[which][r] = t;
  }
  // set-bit sums of this warp's 32 projections for token `lane`
  float s_in[R], s_out[R];
#pragma unroll
  for (int r = 0; r < R; ++r) { s_in[r] = 0.f; s_out[r] = 0.f; }
  const int p0 = warp * 32;
  if (lane < n_tok && p0 < sketch) {
    const int64_t tok = grp * G + tok0 + lane;
    const uint32_t w_in = *reinterpret_cast<const uint32_t*>(key_quant + tok * (sketch / 8) + p0 / 8);
    const uint32_t w_out = p0 < o_sketch ? *reinterpret_cast<const uint32_t*>(key_outlier_quant + tok * (o_sketch / 8) + p0 / 8) : 0u;
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const bool b_in = (w_in >> k) & 1u, b_out = (w_out >> k) & 1u;
#pragma unroll
      for (int r4 = 0; r4 < R; r4 += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&qin_s[p0 + k][r4]);
        const float4 b = *reinterpret_cast<const float4*>(&qout_s[p0 + k][r4]);
        if (b_in) { s_in[r4] += a.x; s_in[r4 + 1] += a.y; s_in[r4 + 2] += a.z; s_in[r4 + 3] += a.w; }
        if (b_out) { s_out[r4] += b.x; s_out[r4 + 1] += b.y; s_out[r4 + 2] += b.z; s_out[r4 + 3] += b.w; }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) { part_s[warp][lane][r] = s_in[r]; part_s[warp][lane][R + r] = s_out[r]; }
  __syncthreads();
  for (int i = tid; i < 32 * R; i += THREADS) {
    const int t = i / R, r = i % R;
    if (t >= n_tok || r >= n_rep) continue;
    float si = 0.f, so = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) { si += part_s[w][t][r]; so += part_s[w][t][R + r]; }
    const float inner = 2.f * si - tot_s[0][r], outer = 2.f * so - tot_s[1][r];
    const int64_t tok = grp * G + tok0 + t;
    const float norm_o = Elem<T>::to_f(key_outlier_norm[tok]);
    const float norm_k = Elem<T>::to_f(key_norm[tok]);
    // |k_in|: the two norms are rounded separately, so the difference can dip below zero
    const float norm_in = sqrtf(fmaxf(norm_k * norm_k - norm_o * norm_o, 0.f));
    const float scl = 1.2533141373155001f / (float)sketch, scl_o = 1.2533141373155001f / (float)o_sketch;
    scores[(qrow0 + r) * ((int64_t)n_groups * G) + (int64_t)n * G + tok0 + t] =
        scl * norm_in * inner + scl_o * norm_o * outer;
  }
}

// The same estimate on the warp MMA (sketch dims that are multiples of 128; other groups, sketches and head counts than those of
// cq_qjl_score.cu), persistent: one CTA of 16 warps per SM keeps
// the projection in shared memory as fp16 hi/lo rows (hi = fp16(x), lo = fp16(x - hi): fp32-exact sums), every warp works
// off (group, 32 tokens) items by itself, without a CTA barrier.
//
// What bounded the earlier form: the query's outlier projection q_out S, which every group needs for its own 32 outlier
// channels, as 32 x 256 x n_rep FMAs with an indexed load each (2650 cycles per group and SM, issue-bound), and two CTA
// barriers per group.  Here it is a product with gathered rows: A = rows of S (transposed by ldmatrix; the row addresses ARE the
// gather), B = the query's outlier channels, D = 16 projections x 8 columns, the heads.  q_out S and q S - q_out S are the
// operands of the outlier and of the inlier sketch; a movmatrix turns each into the layout that the sign product wants its B
// operand in, so nothing passes through shared memory.  Columns 0-3 keep the fp16 value, columns 4-7 the remainder of the same
// head; with five to eight heads both are kept and the sign product runs twice.
//   * k-step b takes bits b and b + 16 of every sign word of a token: lane c needs only its words c and c + 4, and an operand
//     register costs one shift and one LOP3.  The table's columns are in that order.
//   * 8 products a k-step (n_rep <= 4).  With the gathered rows as B operand (no transposition, half of the 16 rows idle) and q S
//     and q_out S against the inlier signs separately it was 14, and 153 us for 8 x 8 x 16384 keys; now 129.
//   * The rows of an 8 x 8 matrix hit the bank group (channel mod 8): the 32 channels are dealt over the four matrices of a
//     load by rank within their residue class (the order of the contraction is free).
constexpr int SW = 16, STHREADS = SW * 32;
constexpr int S_PITCH = MAX_SKETCH + 8;               // halves per projection row: channel d starts in bank group d % 8
constexpr int S_TAB_BYTES = 2 * kHeadDim * S_PITCH * 2;
constexpr int S_SIGN_BYTES = 2 * 32 * (MAX_SKETCH / 8);          // signs of 32 tokens, both sketches
constexpr int S_QF_BYTES = (MAX_SKETCH / 16) * 32 * 16;          // q S as accumulators: [k-step][lane] x 4
constexpr int S_SMEM = S_TAB_BYTES + SW * 2 * S_SIGN_BYTES + S_QF_BYTES + kMaxRep * kHeadDim * 2 + SW * 64;

// projection at position 16 b + 8 half + 2 c + e of a table row: bit b + 16 e of word c + 4 half (256 projections), or
// bit b + 8 half + 16 e of word c (128 projections)
__device__ __forceinline__ int sign_proj(int pos, int sketch) {
  const int b = pos >> 4, half = (pos >> 3) & 1, c = (pos >> 1) & 3, e = pos & 1;
  return sketch == 256 ? 32 * (c + 4 * half) + b + 16 * e : 32 * c + b + 8 * half + 16 * e;
}

// ONE: at most 32 outlier channels and groups of at most 32 tokens: one block of channels, one item per group
template <typename T, typename TP, int R, bool ONE>
__global__ void __launch_bounds__(STHREADS, 1)
score_rows_kernel(const uint8_t* __restrict__ key_quant, const uint8_t* __restrict__ key_outlier_quant,
                  const T* __restrict__ key_norm, const T* __restrict__ key_outlier_norm,
                  const uint8_t* __restrict__ outlier_idx, const float* __restrict__ query_sketch,
                  const T* __restrict__ query, const TP* __restrict__ proj_score, float* __restrict__ scores,
                  int n_kbh, int n_groups, int G, int n_rep, int sketch, int o_sketch, int oc) {
  extern __shared__ __align__(16) unsigned char smem[];
  __half* tab = reinterpret_cast<__half*>(smem);                                              // [hi|lo][channel][S_PITCH]
  unsigned char* sign_s = smem + S_TAB_BYTES;                                                 // [warp][buffer][in|out][token][bytes]
  float4* qf_s = reinterpret_cast<float4*>(sign_s + SW * 2 * S_SIGN_BYTES);                   // [k-step][lane]
  __half* q_s = reinterpret_cast<__half*>(qf_s + (MAX_SKETCH / 16) * 32);                 // [head][channel]
  uint8_t* order_s = reinterpret_cast<uint8_t*>(q_s + kMaxRep * kHeadDim);                    // [warp][64]: channel per slot, free slots
  constexpr bool SCALED = std::is_same<T, __nv_bfloat16>::value;
  __shared__ float2 scale_s[kMaxRep];                                                         // query rows: power of two, its inverse
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
  // the projection, rows of channels, positions in sign order: lane = eight adjacent positions, so that neighbouring lanes
  // read neighbouring projections and write neighbouring 16-byte pieces
  const int per_row = sketch / 8, nb = sketch / 16;
#pragma unroll 2
  for (int i = tid; i < kHeadDim * per_row; i += STHREADS) {
    const int d = i / per_row, b = i % nb, half = i % per_row / nb, pos = 16 * b + 8 * half;
    float x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = proj_f<TP>(proj_score[(int64_t)d * sketch + sign_proj(pos + k, sketch)]);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __half2 h = __floats2half2_rn(x[2 * k], x[2 * k + 1]);
      const float2 f = __half22float2(h);
      const __half2 l = __floats2half2_rn(x[2 * k] - f.x, x[2 * k + 1] - f.y);
      hi[k] = *reinterpret_cast<const uint32_t*>(&h);
      lo[k] = *reinterpret_cast<const uint32_t*>(&l);
    }
    *reinterpret_cast<uint4*>(tab + d * S_PITCH + pos) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(tab + (kHeadDim + d) * S_PITCH + pos) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  const int n_chunks = ONE ? 1 : (G + 31) / 32, per_kbh = n_groups * n_chunks;
  const int64_t n_items = (int64_t)n_kbh * per_kbh;
  const int64_t it_first = blockIdx.x * n_items / gridDim.x, it_end = (blockIdx.x + 1) * n_items / gridDim.x;
  const int rb = sketch / 8, orb = o_sketch / 8;
  unsigned char* my_sign = sign_s + warp * 2 * S_SIGN_BYTES;
  uint8_t* order = order_s + warp * 64;
  const uint32_t tab_b = ptx::smem_u32(tab);
  const float keep = R == 8 || c >= 2 ? 1.f : 0.f;      // R == 4: the lanes (columns 4-7) of the remainders

  for (int64_t seg = it_first; seg < it_end;) {       // runs of items of one (batch, KV head)
    const int64_t kbh = seg / per_kbh;
    const int64_t seg_end = min(it_end, (kbh + 1) * per_kbh);
    const int64_t qrow0 = kbh * n_rep;
    __syncthreads();
    // the queries as fp16 operands.  bfloat16 rows are scaled by a power of two that puts the largest element into [4, 8): their
    // range is fp32's, and the sums with 128 channels stay within fp16's
    if (warp < kMaxRep) {
      float x[kHeadDim / 32], m = 0.f, up = 1.f, down = 1.f;
#pragma unroll
      for (int i = 0; i < kHeadDim / 32; ++i) {
        x[i] = warp < n_rep ? Elem<T>::to_f(query[(qrow0 + warp) * kHeadDim + 32 * i + lane]) : 0.f;
        m = fmaxf(m, fabsf(x[i]));
      }
      m = warp_max(m);
      if (SCALED && m > 0.f && m < INFINITY) {
        const uint32_t e = max(__float_as_uint(m) >> 23, 7u);      // biased exponent; numbers below 2^-120 are not worth more
        up = __uint_as_float((127u + 127u + 2u - e) << 23);
        down = __uint_as_float((e - 2u) << 23);
      }
#pragma unroll
      for (int i = 0; i < kHeadDim / 32; ++i) q_s[warp * kHeadDim + 32 * i + lane] = __float2half_rn(x[i] * up);
      if (SCALED && lane == 0) scale_s[warp] = make_float2(up, down);
    }
    __syncthreads();
    // q S as accumulators: rows = positions g, g + 8 of a k-step, columns 2c, 2c+1 = heads (R == 4: heads 0-3 twice).  Not given:
    // a product with the table, one k-step of positions per warp
    if (query_sketch) {
      for (int i = tid; i < sketch * 2; i += STHREADS) {
        const int b = i >> 5, l = i & 31;
        float x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int head = (2 * (l & 3) + (k & 1)) & (R == 4 ? 3 : 7), pos = 16 * b + (l >> 2) + 8 * (k >> 1);
          x[k] = head < n_rep ? query_sketch[(qrow0 + head) * sketch + sign_proj(pos, sketch)] * (SCALED ? scale_s[head].x : 1.f) : 0.f;
        }
        qf_s[i] = make_float4(x[0], x[1], x[2], x[3]);
      }
    } else if (warp < sketch / 16) {
      float u[2][4] = {};      // by the hi and the lo rows
      const __half* qh = q_s + (R == 4 ? (g & 3) : g) * kHeadDim + 2 * c;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const uint32_t q0 = *reinterpret_cast<const uint32_t*>(qh + 16 * ks), q1 = *reinterpret_cast<const uint32_t*>(qh + 16 * ks + 8);
#pragma unroll
        for (int hl = 0; hl < 2; ++hl) {
          uint32_t b0, b1, b2, b3;
          ptx::ldmatrix_x4_trans(tab_b + (uint32_t)(((hl * kHeadDim + 16 * ks + (lane & 15)) * S_PITCH + 16 * warp) * 2 + (lane >> 4) * 16), b0, b1, b2, b3);
          ptx::mma_f16(u[hl], b0, b2, b1, b3, q0, q1);
        }
      }
      qf_s[warp * 32 + lane] = make_float4(u[0][0] + u[1][0], u[0][1] + u[1][1], u[0][2] + u[1][2], u[0][3] + u[1][3]);
    }
    __syncthreads();
    // an item's sign words (contiguous: 32 tokens x sketch / 8 bytes each) through a double buffer of this warp
    auto fetch = [&](int64_t item, int buf) {
      if (item < seg_end) {
        const int loc = (int)(item - kbh * per_kbh), nn = ONE ? loc : loc / n_chunks, tok0 = ONE ? 0 : (loc - nn * n_chunks) * 32;
        const int n_tok = min(32, G - tok0);
        const int64_t grp = kbh * n_groups + nn;
        const uint8_t* a = key_quant + (grp * G + tok0) * rb;
        const uint8_t* o = key_outlier_quant + (grp * G + tok0) * orb;
        const uint32_t dst = ptx::smem_u32(my_sign + buf * S_SIGN_BYTES);
        // rows of 32 bytes: the two 16-byte halves of every other four rows are exchanged, so that eight rows hit all banks
        auto put = [&](uint32_t to, const uint8_t* from, int row_bytes) {
          for (int i = lane; i < n_tok * row_bytes / 16; i += 32)
            ptx::cp_async_zfill<16>(to + (uint32_t)((row_bytes == 32 ? i ^ ((i >> 3) & 1) : i) * 16), from + i * 16, 16);
        };
        put(dst, a, rb);
        put(dst + S_SIGN_BYTES / 2, o, orb);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int64_t item = seg + warp;
    fetch(item, 0);
    for (int buf = 0; item < seg_end; item += SW, buf ^= 1) {
      const int loc = (int)(item - kbh * per_kbh), n = ONE ? loc : loc / n_chunks, tok0 = ONE ? 0 : (loc - n * n_chunks) * 32;
      const int n_tok = min(32, G - tok0);
      const int64_t grp = kbh * n_groups + n;
      fetch(item + SW, buf ^ 1);
      float nk[4], no[4];                             // norms of the lane's tokens g + 8 i
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t t = grp * G + tok0 + min(g + 8 * i, n_tok - 1);
        nk[i] = Elem<T>::to_f(key_norm[t]);
        no[i] = Elem<T>::to_f(key_outlier_norm[t]);
      }
      // [values | remainders][in | out][m-tile][fragment].  The tensor core truncates as it adds, so eight k-steps are summed at a
      // time, and values and remainders of more than four heads apart: in one accumulator every remainder truncated the sum
      // of the values, and scores of six heads were off by 8.7e-6 of their size instead of 2.3e-6 (141.6 us for 8 x 8 x 16384
      // keys, apart 155.7)
      constexpr int NV = R / 4;
      float acc[NV][2][2][4], sum[2][2][4];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        (&sum[0][0][0])[i] = 0.f;
#pragma unroll
        for (int v = 0; v < NV; ++v) (&acc[v][0][0][0])[i] = 0.f;
      }
      // u accumulates over blocks of 32 outlier channels; there is one block unless oc > 32 (an empty one where oc is 0)
      const int blocks = ONE ? 1 : max(1, (oc + 31) / 32);
      uint32_t qa[2][2], row[2];                      // A fragments and ldmatrix row of the block at hand
      auto load_block = [&](int blk) {
        const int i = blk * 32 + lane;
        const bool have = i < oc;
        const int d = have ? outlier_idx[grp * oc + i] & (kHeadDim - 1) : 0x80 | lane;      // bit 7: no channel
        const uint32_t same = __match_any_sync(0xffffffffu, d & 7), lt = (1u << lane) - 1u;
        const int rank = __popc(same & lt);
        const bool over = rank >= 4;
        const uint32_t taken = __reduce_or_sync(0xffffffffu, over ? 0u : 1u << (rank * 8 + (d & 7)));
        const uint32_t ov = __ballot_sync(0xffffffffu, over);
        if (!((taken >> lane) & 1u)) order[32 + __popc(~taken & lt)] = (uint8_t)lane;       // free slots in order
        __syncwarp();
        order[over ? order[32 + __popc(ov & lt)] : rank * 8 + (d & 7)] = (uint8_t)d;
        __syncwarp();
        const int head = R == 4 ? (g & 3) : g;
        auto qv = [&](int slot) -> uint32_t {
          const int ch = order[slot];
          return ch & 0x80 ? 0u : (uint32_t)__half_as_ushort(q_s[head * kHeadDim + ch]);
        };
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          qa[ks][0] = qv(16 * ks + 2 * c) | (qv(16 * ks + 2 * c + 1) << 16);
          qa[ks][1] = qv(16 * ks + 2 * c + 8) | (qv(16 * ks + 2 * c + 9) << 16);
          // matrices 0, 1 of a load: rows k 0-7 and 8-15 at positions 0-7; 2, 3: the same rows at positions 8-15
          row[ks] = tab_b + (uint32_t)((order[16 * ks + (lane & 15)] & 0x7f) * S_PITCH * 2) + (uint32_t)(lane >> 4) * 16u;
        }
        __syncwarp();
      };
      if (ONE || blocks == 1) load_block(0);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      // sign words of the lane: rows g + 8 i, inverted, words c and c + 4 (128 projections: word c twice, eight bits apart).
      // k-steps run from the top: the bits at hand are always 15 and 31
      uint32_t x[2][4][2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int bytes = s == 0 ? rb : orb;
        const unsigned char* base = my_sign + buf * S_SIGN_BYTES + s * (S_SIGN_BYTES / 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = g + 8 * i, sw = bytes == 32 ? (r >> 2) & 1 : 0;
          const uint32_t w = ~*reinterpret_cast<const uint32_t*>(base + r * bytes + (sw << 4) + 4 * c);
          if (bytes == 32) {
            x[s][i][0] = w;
            x[s][i][1] = ~*reinterpret_cast<const uint32_t*>(base + r * bytes + ((1 ^ sw) << 4) + 4 * c);
          } else {
            x[s][i][0] = sketch == 256 ? w : w << 8;
            x[s][i][1] = w;
          }
        }
      }
      __syncwarp();      // the sign buffer may be refilled
      const uint32_t two = 1u + (sketch > 0);         // not a constant: the shift becomes a multiplication, off the busy ALU pipe
      const bool short_out = o_sketch < sketch;      // 128 of 256: only the first half of every k-step is in the outlier sketch
#pragma unroll 2
      for (int b = sketch / 16 - 1; b >= 0; --b) {
        float u[2][4];                                // q_out S by the hi and the lo rows: rows = positions, columns = heads
        for (int blk = 0; blk < blocks; ++blk) {
          if (!ONE && blocks > 1) load_block(blk);
#pragma unroll
          for (int ks = 0; ks < 2; ++ks)
#pragma unroll
            for (int hl = 0; hl < 2; ++hl) {
              uint32_t b0, b1, b2, b3;
              ptx::ldmatrix_x4_trans(row[ks] + (uint32_t)(hl * kHeadDim * S_PITCH * 2 + 32 * b), b0, b1, b2, b3);
              if (ks == 0 && blk == 0) ptx::mma_f16_zero(u[hl], b0, b2, b1, b3, qa[0][0], qa[0][1]);
              else ptx::mma_f16(u[hl], b0, b2, b1, b3, qa[ks][0], qa[ks][1]);
            }
        }
        // the two operands: fp16 value, or what it leaves over (R == 8: both), as [position][head] -> B fragments
        const float4 qs = qf_s[b * 32 + lane];
        const float qv[4] = {qs.x, qs.y, qs.z, qs.w};
        uint32_t bv[2][2], bl[2][2];                  // [in | out][positions 0-7 | 8-15]
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const float o0 = u[0][2 * half] + u[1][2 * half], o1 = u[0][2 * half + 1] + u[1][2 * half + 1];
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const float x0 = s ? o0 : qv[2 * half] - o0, x1 = s ? o1 : qv[2 * half + 1] - o1;
            const __half2 h = __floats2half2_rn(x0, x1);
            const float2 f = __half22float2(h);
            const __half2 l = __floats2half2_rn(fmaf(-keep, f.x, x0), fmaf(-keep, f.y, x1));
            bl[s][half] = ptx::movmatrix_trans(*reinterpret_cast<const uint32_t*>(&l));
            bv[s][half] = R == 4 ? bl[s][half] : ptx::movmatrix_trans(*reinterpret_cast<const uint32_t*>(&h));
          }
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          uint32_t a[4][2];                           // +-2^-24, negative where the bit is 0
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              a[i][e] = (x[s][i][e] & 0x80008000u) | 0x00010001u;
              asm("mad.lo.u32 %0, %0, %1, 0;" : "+r"(x[s][i][e]) : "r"(two));
            }
          const uint32_t b1v = s == 1 && short_out ? 0u : bv[s][1], b1l = s == 1 && short_out ? 0u : bl[s][1];
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            ptx::mma_f16(acc[0][s][mt], a[2 * mt][0], a[2 * mt + 1][0], a[2 * mt][1], a[2 * mt + 1][1], bv[s][0], b1v);
            if (R == 8) ptx::mma_f16(acc[NV - 1][s][mt], a[2 * mt][0], a[2 * mt + 1][0], a[2 * mt][1], a[2 * mt + 1][1], bl[s][0], b1l);
          }
        }
        if (b % 8 == 0) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            (&sum[0][0][0])[i] += R == 4 ? (&acc[0][0][0][0])[i] : (&acc[0][0][0][0])[i] + (&acc[NV - 1][0][0][0])[i];
#pragma unroll
            for (int v = 0; v < NV; ++v) (&acc[v][0][0][0])[i] = 0.f;
          }
        }
      }
      // columns 2c, 2c+1 = heads (R == 4: values in columns 0-3, remainders in 4-7)
      const float scl = 1.2533141373155001f / (float)sketch * 16777216.f, scl_o = 1.2533141373155001f / (float)o_sketch * 16777216.f;
      float norm_in[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)      // the two norms are rounded separately, so the difference can dip below zero
        norm_in[i] = scl * sqrtf(fmaxf(nk[i] * nk[i] - no[i] * no[i], 0.f));
      float* dst = scores + (qrow0 + 2 * c) * ((int64_t)n_groups * G) + (int64_t)n * G + tok0 + g;
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = 2 * mt + (e >> 1);
          float v = norm_in[i] * sum[0][mt][e] + scl_o * no[i] * sum[1][mt][e];
          if (R == 4) v += __shfl_xor_sync(0xffffffffu, v, 2);
          if (SCALED) v *= scale_s[(2 * c + (e & 1)) & (R - 1)].y;
          if (2 * c + (e & 1) < n_rep && g + 8 * i < n_tok && (R == 8 || c < 2)) dst[(e & 1) * ((int64_t)n_groups * G) + 8 * i] = v;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    seg = seg_end;
  }
}

// ---- the quantizer on the warp MMA ---------------------------------------------------------------
// For group sizes and sketches that the tcgen05 kernel of cq_qjl_build.cu does not take (groups of 32, 256 projections).
// The sums of a chunk are a [32 tokens x 128] x [128 x sketch] product.  A persistent CTA (one per SM)
// keeps the whole projection in shared memory as fp16 hi/lo pairs in B-fragment order (hi = fp16(x),
// lo = fp16(x - hi): the fp32 accumulator then holds the fp32-rounded sum) and walks (group, chunk)
// items: keys staged as fp16 rows, A fragments by ldmatrix, once as they are (all channels) and once
// ANDed with the group's outlier mask; inlier sum = all - outlier.  Warp = 16 projections.
constexpr int QW = 16, QTHREADS = QW * 32;
constexpr int KPITCH = 136;                           // halves per staged key row: ldmatrix rows hit distinct banks
constexpr int Q_PF_BYTES = 2 * 32 * 8 * 32 * 8;       // [hi|lo][n-tile][k-step][lane] x (b0, b1)
constexpr int Q_KEY_BYTES = 2 * 32 * KPITCH * 2;      // two staged chunks
constexpr int Q_SMEM = Q_PF_BYTES + Q_KEY_BYTES + 32 + 128;

template <typename T> struct Half8;
template <> struct Half8<__half> {
  static __device__ __forceinline__ uint4 conv(uint4 v) { return v; }
};
template <> struct Half8<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t two(uint32_t w) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
    const __half2 h = __floats2half2_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ uint4 conv(uint4 v) { return make_uint4(two(v.x), two(v.y), two(v.z), two(v.w)); }
};

template <typename T, typename TP>
__global__ void __launch_bounds__(QTHREADS, 1)
quant_mma_kernel(const T* __restrict__ keys, const uint8_t* __restrict__ outlier_idx, const TP* __restrict__ proj,
                 uint8_t* __restrict__ key_quant, uint8_t* __restrict__ key_outlier_quant,
                 T* __restrict__ outlier_norm, int64_t n_groups, int G, int sketch, int o_sketch, int oc) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint2* pf = reinterpret_cast<uint2*>(smem);
  __half* key_s = reinterpret_cast<__half*>(smem + Q_PF_BYTES);
  uint32_t* mask_s = reinterpret_cast<uint32_t*>(smem + Q_PF_BYTES + Q_KEY_BYTES);     // [2][4]
  uint8_t* byte_s = smem + Q_PF_BYTES + Q_KEY_BYTES + 32;                               // [128], warp 0 only
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, c = lane & 3;
  // projection fragments: b0 = (P[p][d], P[p][d+1]), b1 = (P[p][d+8], P[p][d+9]) with p = 8 nt + g, d = 16 ks + 2c
  for (int i = tid; i < 32 * 8 * 32; i += QTHREADS) {
    const int nt = i >> 8, ks = (i >> 5) & 7, l = i & 31;
    const int p = 8 * nt + (l >> 2), d = 16 * ks + 2 * (l & 3);
    uint32_t hi[2] = {0u, 0u}, lo[2] = {0u, 0u};
    if (p < sketch) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float x0 = proj_f<TP>(proj[(int64_t)p * kHeadDim + d + 8 * j]);
        const float x1 = proj_f<TP>(proj[(int64_t)p * kHeadDim + d + 8 * j + 1]);
        const __half h0 = __float2half_rn(x0), h1 = __float2half_rn(x1);
        const __half l0 = __float2half_rn(x0 - __half2float(h0)), l1 = __float2half_rn(x1 - __half2float(h1));
        hi[j] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
        lo[j] = (uint32_t)__half_as_ushort(l0) | ((uint32_t)__half_as_ushort(l1) << 16);
      }
    }
    pf[((0 * 32 + nt) * 8 + ks) * 32 + l] = make_uint2(hi[0], hi[1]);
    pf[((1 * 32 + nt) * 8 + ks) * 32 + l] = make_uint2(lo[0], lo[1]);
  }
  const int n_chunks = (G + 31) / 32;
  const int64_t n_items = n_groups * n_chunks;
  // loader role: token row lt, eight channels from 8 * seg
  const int lt = tid >> 4, seg = tid & 15;
  auto fetch = [&](int64_t item) -> uint4 {
    const int64_t grp = item / n_chunks;
    const int tok0 = (int)(item % n_chunks) * 32;
    if (tok0 + lt >= G) return make_uint4(0u, 0u, 0u, 0u);
    return *reinterpret_cast<const uint4*>(keys + ((grp * G + tok0 + lt) * kHeadDim + 8 * seg));
  };
  int64_t item = blockIdx.x;
  uint4 cur = make_uint4(0u, 0u, 0u, 0u);
  if (item < n_items) cur = fetch(item);
  const int p0 = 16 * warp;
  for (int it = 0; item < n_items; item += gridDim.x, ++it) {
    const int buf = it & 1;
    const int64_t grp = item / n_chunks;
    const int tok0 = (int)(item % n_chunks) * 32;
    const int n_tok = min(32, G - tok0);
    *reinterpret_cast<uint4*>(key_s + (buf * 32 + lt) * KPITCH + 8 * seg) = Half8<T>::conv(cur);
    if (warp == 0) {                                  // the group's outlier channels as a 128-bit mask
      reinterpret_cast<uint32_t*>(byte_s)[lane] = 0u;
      __syncwarp();
      for (int i = lane; i < oc; i += 32) byte_s[outlier_idx[grp * oc + i] & (kHeadDim - 1)] = 1;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t w = __ballot_sync(0xffffffffu, byte_s[32 * j + lane] != 0);
        if (lane == 0) mask_s[buf * 4 + j] = w;
      }
      __syncwarp();
    }
    __syncthreads();
    uint4 nxt = make_uint4(0u, 0u, 0u, 0u);
    if (item + gridDim.x < n_items) nxt = fetch(item + gridDim.x);
    const uint32_t mw[4] = {mask_s[buf * 4], mask_s[buf * 4 + 1], mask_s[buf * 4 + 2], mask_s[buf * 4 + 3]};
    {  // norm of the outlier part, from the values as loaded
      const uint32_t mbyte = (mw[seg >> 2] >> (8 * (seg & 3))) & 0xffu;
      const T* e = reinterpret_cast<const T*>(&cur);
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x = Elem<T>::to_f(e[j]);
        if ((mbyte >> j) & 1u) ss = fmaf(x, x, ss);
      }
#pragma unroll
      for (int o = 8; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (seg == 0 && lt < n_tok) outlier_norm[grp * G + tok0 + lt] = Elem<T>::from_f(sqrtf(ss));
    }
    if (p0 < sketch) {
      float acc_t[2][2][4], acc_o[2][2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) { acc_t[mt][nt][e] = 0.f; acc_o[mt][nt][e] = 0.f; }
      const uint32_t a_base = ptx::smem_u32(key_s + (buf * 32 + (lane & 7) + 8 * ((lane >> 3) & 1)) * KPITCH + 8 * (lane >> 4));
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        // channels 16ks + (2c, 2c+1) and + (2c+8, 2c+9): all-ones halves where the channel is an outlier
        const uint32_t m = mw[ks >> 1] >> (16 * (ks & 1) + 2 * c);
        const uint32_t m_lo = ((m & 1u) ? 0x0000ffffu : 0u) | ((m & 2u) ? 0xffff0000u : 0u);
        const uint32_t m_hi = ((m & 0x100u) ? 0x0000ffffu : 0u) | ((m & 0x200u) ? 0xffff0000u : 0u);
        uint2 b[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int v = 0; v < 2; ++v) b[nt][v] = pf[((v * 32 + 2 * warp + nt) * 8 + ks) * 32 + lane];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          uint32_t a0, a1, a2, a3;
          ptx::ldmatrix_x4(a_base + (uint32_t)((mt * 16 * KPITCH + ks * 16) * 2), a0, a1, a2, a3);
          const uint32_t o0 = a0 & m_lo, o1 = a1 & m_lo, o2 = a2 & m_hi, o3 = a3 & m_hi;
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              ptx::mma_f16(acc_t[mt][nt], a0, a1, a2, a3, b[nt][v].x, b[nt][v].y);
              ptx::mma_f16(acc_o[mt][nt], o0, o1, o2, o3, b[nt][v].x, b[nt][v].y);
            }
        }
      }
      // acc[..][0..1] = (token g, projections 2c, 2c+1 of the n-tile), acc[..][2..3] = (token g + 8, same)
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t bits_in = 0u, bits_out = 0u;
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float out = acc_o[mt][nt][2 * hh + e], in = acc_t[mt][nt][2 * hh + e] - out;
              bits_in |= (in > 0.f ? 1u : 0u) << (8 * nt + 2 * c + e);
              bits_out |= (out > 0.f ? 1u : 0u) << (8 * nt + 2 * c + e);
            }
          bits_in |= __shfl_xor_sync(0xffffffffu, bits_in, 1); bits_in |= __shfl_xor_sync(0xffffffffu, bits_in, 2);
          bits_out |= __shfl_xor_sync(0xffffffffu, bits_out, 1); bits_out |= __shfl_xor_sync(0xffffffffu, bits_out, 2);
          const int t = 16 * mt + g + 8 * hh;
          if (c == 0 && t < n_tok) {
            const int64_t tok = grp * G + tok0 + t;
            *reinterpret_cast<uint16_t*>(key_quant + tok * (sketch / 8) + 2 * warp) = (uint16_t)bits_in;
            if (p0 < o_sketch)
              *reinterpret_cast<uint16_t*>(key_outlier_quant + tok * (o_sketch / 8) + 2 * warp) = (uint16_t)bits_out;
          }
        }
    }
    cur = nxt;
  }
}

static bool sizes_ok(int G, int sketch, int o_sketch, int oc) {
  return G > 0 && sketch > 0 && sketch <= MAX_SKETCH && sketch % 32 == 0 && o_sketch > 0 && o_sketch <= sketch &&
         o_sketch % 32 == 0 && oc >= 0 && oc <= kHeadDim;
}

static bool mma_ptrs_ok(const void* a, const void* b) { return aligned16(a) && aligned16(b); }

}  // namespace qjl
}  // namespace cq

using namespace cq;

extern "C" int cq_qjl_quant(const void* keys, const uint8_t* outlier_indices, const void* proj, int proj_dtype,
                            int64_t n_groups_total, int group_size, int head_dim, int sketch_dim,
                            int outlier_sketch_dim, int outlier_count, int dtype, uint8_t* key_quant,
                            uint8_t* key_outlier_quant, void* outlier_norms, void* stream) {
  if (n_groups_total == 0) return CQ_OK;
  if (!keys || !outlier_indices || !proj || !key_quant || !key_outlier_quant || !outlier_norms || n_groups_total < 0)
    return CQ_ERR_BAD_ARG;
  if (dtype != CQ_DTYPE_F16 && dtype != CQ_DTYPE_BF16) return CQ_ERR_BAD_ARG;
  if (proj_dtype != CQ_DTYPE_F32 && proj_dtype != dtype) return CQ_ERR_BAD_ARG;
  if (head_dim != kHeadDim || !qjl::sizes_ok(group_size, sketch_dim, outlier_sketch_dim, outlier_count))
    return CQ_ERR_UNSUPPORTED;
  if (n_groups_total > 0x7fffffff) return CQ_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t strides[3] = {0, 0, kHeadDim};      // one dense run of groups
  if (qjl_build::eligible(keys, group_size, head_dim, sketch_dim, outlier_sketch_dim, outlier_count, strides, key_quant, key_outlier_quant))
    return qjl_build::run(keys, 1, 1, (int)n_groups_total, strides, outlier_indices, proj, proj_dtype, outlier_sketch_dim, outlier_count,
                          dtype, nullptr, key_quant, key_outlier_quant, nullptr, outlier_norms, st);
  // other sizes, aligned rows: the warp MMA, one persistent CTA per SM (8 x 8 x 32768 keys: 3.0 ms, on the CUDA cores 12.6)
  if (aligned16(keys) && (reinterpret_cast<uintptr_t>(key_quant) & 1u) == 0 &&
      (reinterpret_cast<uintptr_t>(key_outlier_quant) & 1u) == 0) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      return CQ_ERR_LAUNCH;
    const int64_t items = n_groups_total * ((group_size + 31) / 32);
    const unsigned grid_mma = (unsigned)(items < sms ? items : sms);
#define CQ_QJL_QUANT_MMA(T, TP)                                                                                 \
    do {                                                                                                        \
      auto kern = qjl::quant_mma_kernel<T, TP>;                                                                 \
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, qjl::Q_SMEM) != cudaSuccess)  \
        return CQ_ERR_LAUNCH;                                                                                   \
      kern<<<grid_mma, qjl::QTHREADS, qjl::Q_SMEM, st>>>(static_cast<const T*>(keys), outlier_indices,          \
          static_cast<const TP*>(proj), key_quant, key_outlier_quant, static_cast<T*>(outlier_norms),           \
          n_groups_total, group_size, sketch_dim, outlier_sketch_dim, outlier_count);                           \
    } while (0)
    if (dtype == CQ_DTYPE_F16) {
      if (proj_dtype == CQ_DTYPE_F32) CQ_QJL_QUANT_MMA(__half, float); else CQ_QJL_QUANT_MMA(__half, __half);
    } else {
      if (proj_dtype == CQ_DTYPE_F32) CQ_QJL_QUANT_MMA(__nv_bfloat16, float); else CQ_QJL_QUANT_MMA(__nv_bfloat16, __nv_bfloat16);
    }
#undef CQ_QJL_QUANT_MMA
    return cudaGetLastError() == cudaSuccess ? CQ_OK : CQ_ERR_LAUNCH;
  }
  dim3 grid((unsigned)n_groups_total, (unsigned)((group_size + 31) / 32));
#define CQ_QJL_QUANT(T, TP)                                                                                   \
  qjl::quant_kernel<T, TP><<<grid, qjl::THREADS, 0, st>>>(static_cast<const T*>(keys), outlier_indices,       \
      static_cast<const TP*>(proj), key_quant, key_outlier_quant, static_cast<T*>(outlier_norms), group_size,  \
      sketch_dim, outlier_sketch_dim, outlier_count)
  if (dtype == CQ_DTYPE_F16) {
    if (proj_dtype == CQ_DTYPE_F32) CQ_QJL_QUANT(__half, float); else CQ_QJL_QUANT(__half, __half);
  } else {
    if (proj_dtype == CQ_DTYPE_F32) CQ_QJL_QUANT(__nv_bfloat16, float); else CQ_QJL_QUANT(__nv_bfloat16, __nv_bfloat16);
  }
#undef CQ_QJL_QUANT
  return cudaGetLastError() == cudaSuccess ? CQ_OK : CQ_ERR_LAUNCH;
}

extern "C" int cq_qjl_gqa_score(const uint8_t* key_quant, const uint8_t* key_outlier_quant, const void* key_norm,
                                const void* key_outlier_norm, const uint8_t* outlier_indices,
                                const float* query_sketch, const void* query, const void* proj_score,
                                int proj_dtype, int batch, int n_kv_heads, int n_rep, int n_groups, int group_size,
                                int head_dim, int sketch_dim, int outlier_sketch_dim, int outlier_count, int dtype,
                                float* scores, void* stream) {
  if (batch == 0 || n_groups == 0) return CQ_OK;
  if (!key_quant || !key_outlier_quant || !key_norm || !key_outlier_norm || !outlier_indices || !query || !proj_score || !scores)
    return CQ_ERR_BAD_ARG;
  if (batch < 0 || n_kv_heads <= 0 || n_rep <= 0 || n_groups < 0) return CQ_ERR_BAD_ARG;
  if (dtype != CQ_DTYPE_F16 && dtype != CQ_DTYPE_BF16) return CQ_ERR_BAD_ARG;
  if (proj_dtype != CQ_DTYPE_F32 && proj_dtype != dtype) return CQ_ERR_BAD_ARG;
  if (head_dim != kHeadDim || n_rep > kMaxRep || !qjl::sizes_ok(group_size, sketch_dim, outlier_sketch_dim, outlier_count))
    return CQ_ERR_UNSUPPORTED;
  if (n_groups > 65535) return CQ_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // sketch rows that are whole 16-byte words: the persistent tensor-core kernel, one CTA per SM
  const bool use_mma = sketch_dim % 128 == 0 && outlier_sketch_dim % 128 == 0 && qjl::mma_ptrs_ok(key_quant, key_outlier_quant) && aligned16(proj_score);
  if (!query_sketch && !use_mma) return CQ_ERR_UNSUPPORTED;
  // 8 x 8 x 16384 keys, four heads: 133 us on the warp MMA, 87 here; 1 x 8 x 512 15.2 and 10.0, 1 x 8 x 8192 15.9 and 14.9, a single
  // group 10.5 and 10.0; eight outlier channels 1 x 8 x 8192 15.5 and 15.0
  if (use_mma && qjl_score::eligible(key_quant, key_outlier_quant, group_size, sketch_dim, outlier_sketch_dim, n_rep))
    return qjl_score::run(key_quant, key_outlier_quant, key_norm, key_outlier_norm, outlier_indices, query_sketch, query, proj_score, proj_dtype,
                          batch * n_kv_heads, n_rep, n_groups, outlier_sketch_dim, outlier_count, dtype, scores, st);
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return CQ_ERR_LAUNCH;
  const int64_t items = (int64_t)batch * n_kv_heads * n_groups * ((group_size + 31) / 32);
  // a CTA per 16 items, or per KV head where a head has fewer: a CTA goes from head to head behind barriers
  const int64_t per_head = (int64_t)n_groups * ((group_size + 31) / 32), per_cta = per_head < qjl::SW ? per_head : qjl::SW;
  const unsigned grid_mma = (unsigned)((items + per_cta - 1) / per_cta < sms ? (items + per_cta - 1) / per_cta : sms);
  const dim3 grid((unsigned)(batch * n_kv_heads), (unsigned)n_groups, (unsigned)((group_size + 31) / 32));
#define CQ_QJL_ARGS(T, TP) key_quant, key_outlier_quant, static_cast<const T*>(key_norm), static_cast<const T*>(key_outlier_norm), \
      outlier_indices, query_sketch, static_cast<const T*>(query), static_cast<const TP*>(proj_score), scores
#define CQ_QJL_SCORE(T, TP, R)                                                                                 \
  do {                                                                                                         \
    if (use_mma) {                                                                                             \
      auto kern = group_size <= 32 && outlier_count <= 32 ? qjl::score_rows_kernel<T, TP, R, true> : qjl::score_rows_kernel<T, TP, R, false>;                                                            \
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, qjl::S_SMEM) != cudaSuccess) \
        return CQ_ERR_LAUNCH;                                                                                  \
      kern<<<grid_mma, qjl::STHREADS, qjl::S_SMEM, st>>>(CQ_QJL_ARGS(T, TP), batch * n_kv_heads, n_groups, group_size, n_rep, \
                                                         sketch_dim, outlier_sketch_dim, outlier_count);       \
    } else {                                                                                                   \
      qjl::score_kernel<T, TP, R><<<grid, qjl::THREADS, 0, st>>>(CQ_QJL_ARGS(T, TP), n_groups, group_size, n_rep, sketch_dim, \
                                                                 outlier_sketch_dim, outlier_count);           \
    }                                                                                                          \
  } while (0)
#define CQ_QJL_SCORE_R(T, TP) do { if (n_rep <= 4) CQ_QJL_SCORE(T, TP, 4); else CQ_QJL_SCORE(T, TP, 8); } while (0)
  if (dtype == CQ_DTYPE_F16) {
    if (proj_dtype == CQ_DTYPE_F32) CQ_QJL_SCORE_R(__half, float); else CQ_QJL_SCORE_R(__half, __half);
  } else {
    if (proj_dtype == CQ_DTYPE_F32) CQ_QJL_SCORE_R(__nv_bfloat16, float); else CQ_QJL_SCORE_R(__nv_bfloat16, __nv_bfloat16);
  }
#undef CQ_QJL_SCORE_R
#undef CQ_QJL_SCORE
#undef CQ_QJL_ARGS
  return cudaGetLastError() == cudaSuccess ? CQ_OK : CQ_ERR_LAUNCH;
}
