// QJL score estimate on the 5th-generation tensor cores (groups of 32 keys, 256 projections, up to four query heads per KV head):
//     score = sqrt(pi/2)/s * |k_in| * sum_p sgn_p * (q S - q_out S)_p  +  sqrt(pi/2)/s_o * |k_out| * sum_{p<s_o} sgn'_p * (q_out S)_p
// with q_out = q restricted to the group's outlier channels.
//
// What bounded the form before this one (score_rows_kernel, which stays for other sizes): 2781 warp instructions per group of 32
// keys at 55 % of the issue slots, two thirds of them around the warp MMA: gathered rows of S, the conversion of every
// accumulator into the next product's operand, one shift and one LOP per pair of sign bits; 129 us for 8 x 8 x 16384 keys.
// Here both products are tcgen05.mma over persistent CTAs, S resident in shared memory as fp16 hi + lo rows:
//   1. q_out S of up to 16 groups x 4 heads at once: A = S^T (256 projections = two M tiles), B = the heads' queries with all but
//      the group's outlier channels zeroed.  No gather: the dense product costs the tensor pipe less than addressing rows cost
//      the warps.  A KV head's first tile carries the unmasked queries as well: q S.
//   2. sums over set sign bits of a unit of 128 keys (4 groups): A = the bits, written by the warps into tensor memory as fp16
//      powers of two; B = [projection][q_out S hi | lo of 4 groups x 4 heads, q S hi | lo of 4 heads] as read back from (1).
//      Only a key's own group's columns count (3/4 of the work is idle).
//      sum_p sgn_p x_p = 2 sum_{bit p} x_p - sum_p x_p, the latter from channel sums of S: sum_p (q_out S)_p = q_out (S 1).
// A bit stays where it is in its word: one AND makes two operand elements, of weight 2^(i-24) for bit i.  The rows of B carry the
// inverse.  Bits 4-11 of each half word are used in place, the others after one rotation by eight, so the weights span 2^7.
// Six roles of warps (below) hand these steps on through mbarriers.  What bounds it now is that chain and no unit by itself: a unit
// of 8 x 8 x 16384 keys takes about 2700 cycles, and without 16 of its 40 products the call takes 84.0 us instead of 87.2, with half
// of the first product 81.5, without the sums of the masked queries 84.1 (an outlier sketch of 128 bits, whose second half is
// multiplied although it is zero, would gain 1 % without it).
// 8 x 8 x 16384 keys, 32 query heads: 129 -> 87 us on the way from the warp MMA; 1 x 8 x 512 keys 15.3 -> 10.0 us; error against 64-bit sums
// 4.6e-6 -> 3.5e-7 (the product truncates less often than the warp MMA).  The inlier part by itself, of a query that lies 300 to 1 in
// the outlier channels, is off by 6.4e-5, on the warp MMA by 4.2e-5: q S and q_out S are summed apart and subtracted after the signs,
// and an fp32 difference ahead of them cost 5 us for 5.9e-5; the whole score of such a query 2.2e-6 and 5.0e-6.
// Every wait is bounded; on a timeout the CTA writes the status word and NaN for its scores, frees its tensor memory and returns.
#include <type_traits>

#include "cq_common.cuh"
#include "cq_ptx.cuh"
#include "cq_tc.cuh"

namespace cq {
namespace qjl_score {

using namespace ptx;
using namespace tc;

constexpr int G = 32, SKETCH = 256, R = 4;                 // keys of a group, projections, query heads per KV head (at most)
constexpr int UNIT_G = 4, MAX_TG = 16;                     // groups of a unit, of a tile (at most)
constexpr int SLOTS = 8;                                   // tiles whose totals are kept
// warps by role: sign bits, sketches of the query, scores, masked queries, and one issuer for either product.  (Where one warp did
// several of these, each waited for the slowest of its own steps: 118 us with two roles and one issuer, 8 x 8 x 16384 keys.)
constexpr int N_SIGN = 8, N_SKETCH = 8, N_SCORE = 4, N_QUERY = 4;
constexpr int W_SKETCH = N_SIGN, W_SCORE = W_SKETCH + N_SKETCH, W_QUERY = W_SCORE + N_SCORE, W_ISSUE = W_QUERY + N_QUERY;
constexpr int N_WARPS = W_ISSUE + 2, THREADS = N_WARPS * 32;
constexpr int TAB_BYTES = SKETCH * kHeadDim * 2, TAB_PANEL = TAB_BYTES / 2;      // S^T hi (lo behind it): two panels of [256 rows][128 bytes]
constexpr int Q_ROWS = MAX_TG * R + 16, Q_BYTES = Q_ROWS * kHeadDim * 2, Q_PANEL = Q_BYTES / 2;
constexpr int X_BYTES = SKETCH * 128;                      // sketches of a unit: [projection][64 columns]
constexpr int SMEM = 2 * TAB_BYTES + Q_BYTES + 2 * X_BYTES + 1024;
// tensor memory: (1) by M tile; sign bits of half the projections: inlier sketch, outlier sketch; (2)
constexpr uint32_t T_OUT = 0, T_OUT_TILE = 96, T_SIGN = 176, T_SIGN_HALF = 128, T_SUM_IN = 432, T_SUM_OUT = 480;
constexpr int N_IN = 48, N_OUT = 32;                       // columns: q_out S hi 16 | lo 16 | q S hi 4 | lo 4 | zeros 8

struct Args {
  int n_kbh, n_groups, n_rep, o_sketch, oc;
  int tg, tiles_per_kbh;       // groups of a tile
  int n_tiles;
  uint32_t idesc_q, idesc_q_first, idesc_in, idesc_out;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}

template <typename TP> __device__ __forceinline__ float proj_f(TP v);
template <> __device__ __forceinline__ float proj_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float proj_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float proj_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ float2 h2_floats(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
// (a, b) as fp16, and what that leaves over
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  hi = h2_bits(h);
  lo = h2_bits(__floats2half2_rn(a - f.x, b - f.y));
}

// A channel named more than once counts as often.  The products have it once; what the further mentions add to a key's scores is
// summed here in fp32 (none of the quantizers names a channel twice; as a factor of the fp16 query, three mentions of an element
// lost its last bits).  With oc < 0 they become NaN.  A call, so that it takes no registers from the kernel.
template <typename T, typename TP>
__device__ __noinline__ void further_mentions(const uint8_t* idx, int oc, const uint8_t* sign_in, const uint8_t* sign_out, int o_sketch, float nk,
                                              float no, const T* query, int n_rep, const TP* proj, float* scores, int64_t row_len) {
  const float norm_in = 1.2533141373155001f / (float)SKETCH * sqrtf(fmaxf(nk * nk - no * no, 0.f)), norm_out = 1.2533141373155001f / (float)o_sketch * no;
  if (oc < 0)
    for (int h = 0; h < n_rep; ++h) scores[h * row_len] = __int_as_float(0x7fc00000);
  uint64_t seen_lo = 0, seen_hi = 0;
  for (int i = 0; i < oc; ++i) {
    const int d = idx[i] & (kHeadDim - 1);
    const uint64_t bit = 1ull << (d & 63);
    const bool again = ((d < 64 ? seen_lo : seen_hi) & bit) != 0;
    if (d < 64) seen_lo |= bit; else seen_hi |= bit;
    if (!again) continue;
    float in = 0.f, out = 0.f;                       // signs times the channel's projections
    for (int p = 0; p < SKETCH; ++p) {
      const float x = proj_f<TP>(proj[(int64_t)d * SKETCH + p]);
      in += (sign_in[p >> 3] >> (p & 7)) & 1 ? x : -x;
      if (p < o_sketch) out += (sign_out[p >> 3] >> (p & 7)) & 1 ? x : -x;
    }
    for (int h = 0; h < n_rep; ++h)
      scores[h * row_len] += Elem<T>::to_f(query[(int64_t)h * kHeadDim + d]) * (norm_out * out - norm_in * in);
  }
}

template <typename T, typename TP>
__global__ void __launch_bounds__(THREADS, 1)
score_kernel(const Args a, const uint8_t* __restrict__ key_quant, const uint8_t* __restrict__ key_outlier_quant,
             const T* __restrict__ key_norm, const T* __restrict__ key_outlier_norm, const uint8_t* __restrict__ outlier_idx,
             const float* __restrict__ query_sketch, const T* __restrict__ query, const TP* __restrict__ proj,
             float* __restrict__ scores, int* __restrict__ status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* tab_s = smem;
  unsigned char* q_s = smem + 2 * TAB_BYTES;
  unsigned char* x_s = q_s + Q_BYTES;
  __shared__ __align__(8) uint64_t bar_q, bar_out, bar_out_free, bar_x[2], bar_x_free[2], bar_sign[2], bar_done[2], bar_sum_free;
  __shared__ uint32_t tmem_s;
  __shared__ __align__(16) float sum_in_s[kHeadDim], sum_out_s[kHeadDim];      // per channel: sums of S over all / the outlier sketch's projections
  // A slot per tile.  With tiles of one unit the queries of tile t are built while the scores of t - 5 may still be read: they follow
  // the first product of t - 1, that one the sketches of t - 2, these (two operand buffers) the sums of t - 4, and these the
  // arrival of the scores of t - 5, which comes before their reading of the slot.
  static_assert(SLOTS > 5 && (SLOTS & (SLOTS - 1)) == 0, "a ring of more tiles than the queries are ahead of the scores");
  __shared__ float tot_in_s[SLOTS][MAX_TG][R], tot_out_s[SLOTS][MAX_TG][R];    // sums of q_out S
  __shared__ float tot_q_s[SLOTS][R], down_s[SLOTS][R], up_s[SLOTS][R];        // sums of q S; powers of two of the queries' scaling
  __shared__ float smax_s[N_WARPS];
  __shared__ int again_s;                                                      // does a group of the CTA name a channel more than once?
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile0 = (int)((int64_t)blockIdx.x * a.n_tiles / gridDim.x), tile1 = (int)((int64_t)(blockIdx.x + 1) * a.n_tiles / gridDim.x);
  // A tile: number within the CTA, KV head, first group within the head.  (Divided out anew at every use, the positions were half
  // of the kernel's instructions.)
  struct Tile { int i, kbh, first, units; bool fresh; };         // fresh: the CTA's first tile of the KV head
  auto settle = [&](Tile& t) { t.units = (min(a.tg, a.n_groups - t.first) + UNIT_G - 1) / UNIT_G; };
  auto first_tile = [&]() {
    Tile t{0, tile0 / a.tiles_per_kbh, tile0 % a.tiles_per_kbh * a.tg, 0, true};
    settle(t);
    return t;
  };
  auto after = [&](Tile t) {
    ++t.i;
    t.first += a.tg;
    t.fresh = t.first >= a.n_groups;
    if (t.fresh) { t.first = 0; ++t.kbh; }
    settle(t);
    return t;
  };
  const int n_tiles = tile1 - tile0;

  if (tid == 0) {
    again_s = 0;
    mbar_init(&bar_q, N_QUERY);
    mbar_init(&bar_out, 1);
    mbar_init(&bar_out_free, N_SKETCH);
    for (int i = 0; i < 2; ++i) { mbar_init(&bar_x[i], N_SKETCH); mbar_init(&bar_x_free[i], 1); mbar_init(&bar_sign[i], N_SIGN); mbar_init(&bar_done[i], 1); }
    mbar_init(&bar_sum_free, N_SCORE);
    mbar_fence_init();
  }
  if (warp == W_ISSUE) tmem_alloc(&tmem_s, 512);
  // S^T, rows of projections, as hi and lo in the swizzled K-major layout; lanes take neighbouring projections
  float smax = 0.f;
  float* const part_s = reinterpret_cast<float*>(x_s);      // sums over 32 projections: [projection / 32][channel]; until the first sketches
#pragma unroll 2
  for (int i = tid; i < SKETCH * 16; i += THREADS) {
    const int p = i & 255, pc = i >> 8;
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { x[j] = proj_f<TP>(proj[(int64_t)(pc * 8 + j) * SKETCH + p]); smax = fmaxf(smax, fabsf(x[j])); }
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      split2(x[2 * j], x[2 * j + 1], hi[j], lo[j]);
      // The sums are of the numbers that the products take: against sums of S itself, the rounding of small elements counted
      // twice where the bit is set (elements of 1e-3: scores off by 2.5e-5, so by 1.7e-5)
      const float2 h = h2_floats(hi[j]), l = h2_floats(lo[j]);
      x[2 * j] = h.x + l.x;
      x[2 * j + 1] = h.y + l.y;
    }
    // over the warp's 32 projections, channels dealt out over the lanes as the sums get fewer
#pragma unroll
    for (int n = 4, o = 16; n >= 1; n /= 2, o /= 2)
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const bool up = lane & o;
        const float other = __shfl_xor_sync(0xffffffffu, up ? x[j] : x[j + n], o);
        x[j] = (up ? x[j + n] : x[j]) + other;
      }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
    if ((lane & 3) == 0) part_s[(p >> 5) * kHeadDim + pc * 8 + (lane >> 2)] = x[0];
    unsigned char* dst = tab_s + (pc >> 3) * TAB_PANEL + p * 128 + (((pc & 7) ^ (p & 7)) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + TAB_BYTES) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  smax = warp_max(smax);
  if (lane == 0) smax_s[warp] = smax;
  // rows of no query
  for (int i = tid; i < Q_BYTES / 16; i += THREADS) reinterpret_cast<uint4*>(q_s)[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;
  bool ok = true;

  if (warp >= W_ISSUE) {
    // ================= products =================
    // the whole warp runs the loop and one elected lane issues, so that the operands are uniform
    const uint32_t lead = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    auto wait = [&](uint64_t* bar, uint32_t phase) { ok = ok && __all_sync(0xffffffffu, mbar_wait_suspended(bar, phase & 1u)) != 0; };
    uint32_t v = 0;
    if (warp == W_ISSUE) {
      const uint64_t td = smem_desc(smem_u32(tab_s), 16, 1024), qd = smem_desc(smem_u32(q_s), 16, 1024);
      for (Tile t = first_tile(); t.i < n_tiles && ok; t = after(t)) {
        wait(&bar_q, (uint32_t)t.i);
        if (t.i > 0) wait(&bar_out_free, (uint32_t)t.i - 1);
        if (!ok) break;
        tc_fence_after();
        if (lead) {
          const uint32_t idesc = t.fresh ? a.idesc_q_first : a.idesc_q;
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int hl = 1; hl >= 0; --hl)      // the tensor core truncates as it adds: first what is small
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                umma(tm + T_OUT + (uint32_t)mt * T_OUT_TILE,
                     td + (uint64_t)((hl * TAB_BYTES + (ks >> 2) * TAB_PANEL + mt * 128 * 128 + (ks & 3) * 32) >> 4),
                     qd + (uint64_t)(((ks >> 2) * Q_PANEL + (ks & 3) * 32) >> 4), idesc, (hl == 0 || ks > 0) ? 1u : 0u);
          umma_commit(&bar_out);
        }
        __syncwarp();
      }
    } else {
      const uint64_t xd = smem_desc(smem_u32(x_s), X_BYTES, 1024);
      for (Tile t = first_tile(); t.i < n_tiles && ok; t = after(t))
        for (int u = 0; u < t.units && ok; ++u, ++v) {
          wait(&bar_x[v & 1], v >> 1);
          if (v > 0) wait(&bar_sum_free, v - 1);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            wait(&bar_sign[half], v);
            if (!ok) break;
            tc_fence_after();
            if (lead) {
              const uint64_t b = xd + (uint64_t)(((v & 1) * X_BYTES) >> 4);
#pragma unroll
              for (int ks = 0; ks < 8; ++ks) {
                const uint32_t sign = tm + T_SIGN + (uint32_t)(half * T_SIGN_HALF + ks * 8), acc = (half > 0 || ks > 0) ? 1u : 0u;
                const uint64_t bk = b + (uint64_t)(((half * 8 + ks) * 2048) >> 4);
                umma_ts(tm + T_SUM_IN, sign, bk, a.idesc_in, acc);
                umma_ts(tm + T_SUM_OUT, sign + T_SIGN_HALF / 2, bk, a.idesc_out, acc);
              }
              umma_commit(&bar_done[half]);
              if (half == 1) umma_commit(&bar_x_free[v & 1]);
            }
            __syncwarp();
          }
        }
    }
    if (!ok && lead) atomicExch(status, CQ_ERR_TIMEOUT);
    __syncwarp();
  } else {
    const int quad = warp & 3;
    const uint32_t lanes = (uint32_t)(32 * quad) << 16;
    auto wait = [&](uint64_t* bar, uint32_t phase) { if (ok) ok = mbar_wait_suspended(bar, phase & 1u); };
    auto arrive = [&](uint64_t* bar) { __syncwarp(); if (lane == 0) mbar_arrive(bar); };
    if (warp >= W_QUERY) {
      // ================= masked queries =================
      const int wq = warp - W_QUERY;
      for (int w = 0; w < N_WARPS; ++w) smax = fmaxf(smax, smax_s[w]);
      {
        const int d = tid - W_QUERY * 32;
        float sum = 0.f, sum_o = 0.f;
#pragma unroll
        for (int i = 0; i < SKETCH / 32; ++i) {
          const float x = part_s[i * kHeadDim + d];
          sum += x;
          if (32 * i < a.o_sketch) sum_o += x;
        }
        sum_in_s[d] = sum;
        sum_out_s[d] = sum_o;
        asm volatile("bar.sync 1, %0;" ::"n"(N_QUERY * 32) : "memory");
      }
      // ---- queries with their group's outlier channels: a warp takes every fourth group, a lane head lane / 8, channels
      // 8 (lane % 8) .. + 7 and + 64
      uint32_t qw[8];                       // the lane's sixteen channels, scaled by a power of two
      const int qh = lane >> 3, qc = lane & 7;
      auto put_row = [&](int row, const uint32_t (&w)[8]) {
        unsigned char* dst = q_s + row * 128 + ((qc ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(dst + Q_PANEL) = make_uint4(w[4], w[5], w[6], w[7]);
      };
      auto dot = [&](const uint32_t (&w)[8], const float* ch) {       // with per-channel factors, summed over the head's eight lanes
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 f = h2_floats(w[i]);
          const float2 c = *reinterpret_cast<const float2*>(ch + (i >> 2) * 64 + qc * 8 + (i & 3) * 2);
          s = fmaf(f.x, c.x, s);
          s = fmaf(f.y, c.y, s);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
      };
      // up to 32 outlier channels of the warp's groups, requested a tile ahead of their use
      constexpr int PER = MAX_TG / N_QUERY;
      uint8_t ch_ahead[PER] = {};
      auto fetch_channels = [&](const Tile& t) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          const int gi = wq + N_QUERY * j, n = t.first + gi;
          if (t.i < n_tiles && gi < a.tg && n < a.n_groups && lane < a.oc) ch_ahead[j] = outlier_idx[((int64_t)t.kbh * a.n_groups + n) * a.oc + lane];
        }
      };
      auto build_queries = [&](const Tile& t) {
        const int slot = t.i & (SLOTS - 1);
        if (t.fresh) {
          // scaled so that the elements, their sums with 128 channels and a given q S stay below 2^15: fp16 operands keep what they
          // can of the remainders
          const T* src = query + ((int64_t)t.kbh * a.n_rep + qh) * kHeadDim + qc * 8;
          float x[16], m = 0.f, up = 1.f, down = 1.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            x[i] = qh < a.n_rep ? Elem<T>::to_f(src[(i >> 3) * 64 + (i & 7)]) : 0.f;
            m = fmaxf(m, fabsf(x[i]));
          }
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
          float tq = 0.f, sketch_max = 0.f;      // of a given q S
          if (query_sketch) {
            if (qh < a.n_rep)
              for (int p = qc; p < SKETCH; p += 8) {
                const float v = query_sketch[((int64_t)t.kbh * a.n_rep + qh) * SKETCH + p];
                tq += v;
                sketch_max = fmaxf(sketch_max, fabsf(v));
              }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
              tq += __shfl_xor_sync(0xffffffffu, tq, o);
              sketch_max = fmaxf(sketch_max, __shfl_xor_sync(0xffffffffu, sketch_max, o));
            }
          }
          // (in units of a power of two near the largest element: 128 channels of bfloat16 numbers can leave fp32's range)
          const int em = m > 0.f ? max(-126, min(126, (int)(__float_as_uint(m) >> 23) - 127)) : 0;
          const float unit = __uint_as_float((uint32_t)(127 - em) << 23);
          const float bound = fmaxf(fmaxf(128.f * smax, 1.f) * (m * unit), sketch_max * unit);
          if (bound > 0.f && bound < INFINITY) {
            const int e = (int)(__float_as_uint(bound) >> 23) - 127;       // bound < 2^(e+1)
            const int s = max(-126, min(126, 14 - e - em));
            up = __uint_as_float((uint32_t)(127 + s) << 23);
            down = __uint_as_float((uint32_t)(127 - s) << 23);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) qw[i] = h2_bits(__floats2half2_rn(x[2 * i] * up, x[2 * i + 1] * up));
          if (wq == 0) {
            put_row(a.tg * R + qh, qw);
            tq = query_sketch ? tq * up : dot(qw, sum_in_s);
            if (qc == 0) { tot_q_s[slot][qh] = tq; down_s[slot][qh] = down; up_s[slot][qh] = up; }
          }
        } else if (wq == 0 && qc == 0) {
          tot_q_s[slot][qh] = tot_q_s[(slot + SLOTS - 1) & (SLOTS - 1)][qh]; down_s[slot][qh] = down_s[(slot + SLOTS - 1) & (SLOTS - 1)][qh];
        }
        int missing = 0;                       // mentions less channels
#pragma unroll 1
        for (int j = 0; j < PER; ++j) {
          const int gi = wq + N_QUERY * j, n = t.first + gi;
          if (gi >= a.tg) break;
          uint32_t ch = ch_ahead[0];
#pragma unroll
          for (int i = 1; i < PER; ++i) ch = i == j ? ch_ahead[i] : ch;
          const uint8_t* idx = outlier_idx + ((int64_t)t.kbh * a.n_groups + n) * a.oc;
          uint32_t mask[4] = {0u, 0u, 0u, 0u};
          if (n < a.n_groups) {
            for (int i0 = 0; i0 < a.oc; i0 += 32) {
              const bool have = i0 + lane < a.oc;
              const int d = i0 == 0 ? ch & (kHeadDim - 1) : have ? idx[i0 + lane] & (kHeadDim - 1) : 0;
#pragma unroll
              for (int m = 0; m < 4; ++m) mask[m] |= __reduce_or_sync(0xffffffffu, have && (d >> 5) == m ? 1u << (d & 31) : 0u);
            }
          }
          const uint32_t lo8 = (qc < 4 ? mask[0] : mask[1]) >> (8 * (qc & 3)), hi8 = (qc < 4 ? mask[2] : mask[3]) >> (8 * (qc & 3));
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t m = (i < 4 ? lo8 : hi8) >> (2 * (i & 3));
            w[i] = qw[i] & (((m & 1u) ? 0x0000ffffu : 0u) | ((m & 2u) ? 0xffff0000u : 0u));
          }
          if (n < a.n_groups) missing += a.oc - (__popc(mask[0]) + __popc(mask[1]) + __popc(mask[2]) + __popc(mask[3]));
          put_row(gi * R + qh, w);
          const float ti = dot(w, sum_in_s), to = a.o_sketch == SKETCH ? ti : dot(w, sum_out_s);
          if (qc == 0) { tot_in_s[slot][gi][qh] = ti; tot_out_s[slot][gi][qh] = to; }
        }
        fence_proxy_async_smem();
        if (missing != 0) again_s = 1;         // (tested group by group it cost 8 x 8 x 16384 keys 2.4 us)
        arrive(&bar_q);
        fetch_channels(after(t));
      };

      Tile t = first_tile();
      fetch_channels(t);
      for (; t.i < n_tiles; t = after(t)) {
        if (t.i > 0) wait(&bar_out, (uint32_t)t.i - 1);      // the queries of the tile before have been read
        build_queries(t);
      }
    } else if (warp >= W_SKETCH && warp < W_SCORE) {
      // ================= q_out S of a unit, from tensor memory to the second product's operand =================
      // Lane = projection 128 mt + 32 quad + lane; its row follows the order of the sign bits (see expand), its factor undoes their
      // weight
      const int mt = (warp - W_SKETCH) >> 2;
      const int z = (lane - 4) & 31, row = 128 * mt + 32 * quad + 2 * (z & 15) + (z >> 4);
      const float weight = __uint_as_float((uint32_t)(127 - (z & 7)) << 23);
      unsigned char* const x_row = x_s + (row >> 3) * 1024 + (row & 7) * 128;
      const uint32_t sw = row & 7, from = tmem + lanes + T_OUT + (uint32_t)mt * T_OUT_TILE;
      auto put = [&](unsigned char* to, uint32_t chunk, uint4 v) { *reinterpret_cast<uint4*>(to + ((chunk ^ sw) << 4)) = v; };
      uint4 sq = make_uint4(0u, 0u, 0u, 0u);           // q S of the lane's projection: hi of four heads, lo of four heads
      uint32_t v = 0;
      for (Tile t = first_tile(); t.i < n_tiles; t = after(t)) {
        wait(&bar_out, (uint32_t)t.i);
        tc_fence_after();
        if (t.fresh) {
          uint32_t r[4];
          tmem_ld4_nowait(from + (uint32_t)(a.tg * R), r);
          tmem_ld_wait();
          if (query_sketch) {
            const float* qs = query_sketch + (int64_t)t.kbh * a.n_rep * SKETCH + 128 * mt + 32 * quad + lane;
#pragma unroll
            for (int h = 0; h < R; ++h) r[h] = h < a.n_rep ? __float_as_uint(qs[h * SKETCH] * up_s[t.i & (SLOTS - 1)][h]) : 0u;
          }
          split2(__uint_as_float(r[0]) * weight, __uint_as_float(r[1]) * weight, sq.x, sq.z);
          split2(__uint_as_float(r[2]) * weight, __uint_as_float(r[3]) * weight, sq.y, sq.w);
        }
        for (int u = 0; u < t.units; ++u, ++v) {
          uint32_t r[16];
          tmem_ld16_nowait(from + (uint32_t)(u * 16), r);
          if (v >= 2) wait(&bar_x_free[v & 1], (v >> 1) - 1);
          tmem_ld_wait();
          if (u == t.units - 1) { tc_fence_before(); arrive(&bar_out_free); }
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) split2(__uint_as_float(r[2 * i]) * weight, __uint_as_float(r[2 * i + 1]) * weight, hi[i], lo[i]);
          unsigned char* to = x_row + (v & 1) * X_BYTES;
          put(to, 0, make_uint4(hi[0], hi[1], hi[2], hi[3]));
          put(to, 1, make_uint4(hi[4], hi[5], hi[6], hi[7]));
          put(to, 2, make_uint4(lo[0], lo[1], lo[2], lo[3]));
          put(to, 3, make_uint4(lo[4], lo[5], lo[6], lo[7]));
          put(to, 4, sq);
          fence_proxy_async_smem();
          arrive(&bar_x[v & 1]);
        }
      }
    } else if (warp < W_SKETCH) {
      // ================= sign bits =================
      // of the lane's key 32 quad + lane, sk 0: inlier, 1: outlier sketch; words 4 half .. + 3.  Operand element 2 r + e of a word: bit
      // 4 + r + 16 e of the word (r < 8), of the word rotated by eight (r >= 8: bit r - 4)
      const int sk = warp >> 2;
      const int rb = sk == 0 ? SKETCH / 8 : a.o_sketch / 8;
      const uint8_t* const sign_src = (sk == 0 ? key_quant : key_outlier_quant) + lane * rb;
      uint4 word[2];
      auto fetch = [&](const Tile& t, int u) {
        const int n = t.first + u * UNIT_G + quad;
        word[0] = word[1] = make_uint4(0u, 0u, 0u, 0u);
        if (n < a.n_groups) {
          const uint8_t* src = sign_src + ((int64_t)t.kbh * a.n_groups + n) * (G * rb);
          word[0] = *reinterpret_cast<const uint4*>(src);
          if (rb == SKETCH / 8) word[1] = *reinterpret_cast<const uint4*>(src + 16);
        }
      };
      const uint32_t sign_at = tmem + lanes + T_SIGN + (uint32_t)(sk * (T_SIGN_HALF / 2));
      auto expand = [&](int half) {
        const uint32_t w[4] = {word[half].x, word[half].y, word[half].z, word[half].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t y0 = w[j], y1 = __funnelshift_r(y0, y0, 8);
          uint32_t e[16];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            e[r] = y0 & (0x00100010u << r);
            e[8 + r] = y1 & (0x00100010u << r);
          }
          tmem_st16(sign_at + (uint32_t)(half * T_SIGN_HALF + j * 16), e);
        }
        tmem_st_wait();
        tc_fence_before();
        arrive(&bar_sign[half]);
      };
      uint32_t v = 0;
      Tile t = first_tile();
      if (n_tiles > 0) fetch(t, 0);
      while (t.i < n_tiles) {
        const Tile next = after(t);
        for (int u = 0; u < t.units; ++u, ++v) {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (v > 0) wait(&bar_done[half], v - 1);
            tc_fence_after();
            expand(half);
          }
          const bool more = u + 1 < t.units;
          if (more || next.i < n_tiles) fetch(more ? t : next, more ? u + 1 : 0);
        }
        t = next;
      }
    } else {
      // ================= sums of a unit -> scores of its keys =================
      const float scl = 1.2533141373155001f / (float)SKETCH, scl_o = 1.2533141373155001f / (float)a.o_sketch;
      T norm_k = {}, norm_o = {};          // as loaded, a unit ahead: a conversion would wait for the load
      auto fetch = [&](const Tile& t, int u) {
        const int n = t.first + u * UNIT_G + quad;
        if (t.i < n_tiles && n < a.n_groups) {
          const int64_t key = ((int64_t)t.kbh * a.n_groups + n) * G + lane;
          norm_k = key_norm[key];
          norm_o = key_outlier_norm[key];
        }
      };
      const uint32_t in = tmem + lanes + T_SUM_IN, out = tmem + lanes + T_SUM_OUT + (uint32_t)(quad * R);
      const int64_t row_len = (int64_t)a.n_groups * G;
      uint32_t v = 0;
      Tile t = first_tile();
      fetch(t, 0);
      while (t.i < n_tiles) {
        const Tile next = after(t);
        const int slot = t.i & (SLOTS - 1);
        for (int u = 0; u < t.units; ++u, ++v) {
          const float nk = Elem<T>::to_f(norm_k), no = Elem<T>::to_f(norm_o);
          const bool more = u + 1 < t.units;
          fetch(more ? t : next, more ? u + 1 : 0);
          // the two norms are rounded separately, so the difference can dip below zero
          const float norm_in = scl * sqrtf(fmaxf(nk * nk - no * no, 0.f)), norm_out = scl_o * no;
          wait(&bar_done[1], v);
          tc_fence_after();
          uint32_t s_in[4][4], s_out[2][4];      // q_out S hi, lo, q S hi, lo by the inlier signs; q_out S hi, lo by the outlier signs
          tmem_ld4_nowait(in + (uint32_t)(quad * R), s_in[0]);
          tmem_ld4_nowait(in + (uint32_t)(16 + quad * R), s_in[1]);
          tmem_ld4_nowait(in + 32u, s_in[2]);
          tmem_ld4_nowait(in + 36u, s_in[3]);
          tmem_ld4_nowait(out, s_out[0]);
          tmem_ld4_nowait(out + 16u, s_out[1]);
          tmem_ld_wait();
          tc_fence_before();
          arrive(&bar_sum_free);
          const int gi = u * UNIT_G + quad, n = t.first + gi;
          if (n < a.n_groups && ok) {
            constexpr float TWICE = 2097152.f;             // 2 * 2^20: what the operand bits' common weight leaves
            auto f = [](uint32_t w) { return __uint_as_float(w); };
            float* dst = scores + (int64_t)t.kbh * a.n_rep * row_len + n * G + lane;
#pragma unroll
            for (int h = 0; h < R; ++h) {
              const float o_in = f(s_in[0][h]) + f(s_in[1][h]), q_in = f(s_in[2][h]) + f(s_in[3][h]), o_out = f(s_out[0][h]) + f(s_out[1][h]);
              const float inner = fmaf(TWICE, q_in - o_in, tot_in_s[slot][gi][h] - tot_q_s[slot][h]);
              const float outer = fmaf(TWICE, o_out, -tot_out_s[slot][gi][h]);
              if (h < a.n_rep) dst[h * row_len] = (norm_in * inner + norm_out * outer) * down_s[slot][h];
            }
          }
        }
        t = next;
      }
      // every further mention of a channel, once the products' scores are written (within the loop it cost every call 6 %); NaN where a
      // wait ran out, so that no score of the CTA stays what it was in memory
      if (!ok) again_s = 1;
      __syncwarp();
      if (again_s)
        for (Tile t = first_tile(); t.i < n_tiles; t = after(t))
          for (int n = t.first + quad; n < min(t.first + a.tg, a.n_groups); n += UNIT_G) {
            const int64_t group = (int64_t)t.kbh * a.n_groups + n, key = group * G + lane;
            further_mentions<T, TP>(outlier_idx + group * a.oc, ok ? a.oc : -1, key_quant + key * (SKETCH / 8), key_outlier_quant + key * (a.o_sketch / 8), a.o_sketch,
                                    Elem<T>::to_f(key_norm[key]), Elem<T>::to_f(key_outlier_norm[key]), query + (int64_t)t.kbh * a.n_rep * kHeadDim,
                                    a.n_rep, proj, scores + (int64_t)t.kbh * a.n_rep * row_len + n * G + lane, row_len);
          }
    }
    if (!ok && lane == 0) atomicExch(status, CQ_ERR_TIMEOUT);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == W_ISSUE) tmem_dealloc(tmem, 512);
}

static __device__ int g_status;

template <typename T, typename TP>
static int launch(const Args& a, int grid, const uint8_t* kq, const uint8_t* koq, const void* kn, const void* kon, const uint8_t* idx,
                  const float* qs, const void* q, const void* proj, float* scores, cudaStream_t st) {
  void* status = nullptr;
  if (cudaGetSymbolAddress(&status, g_status) != cudaSuccess ||
      cudaFuncSetAttribute(score_kernel<T, TP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)
    return CQ_ERR_LAUNCH;
  score_kernel<T, TP><<<(unsigned)grid, THREADS, SMEM, st>>>(a, kq, koq, static_cast<const T*>(kn), static_cast<const T*>(kon), idx, qs,
                                                            static_cast<const T*>(q), static_cast<const TP*>(proj), scores,
                                                            static_cast<int*>(status));
  return check_launch();
}

bool eligible(const uint8_t* kq, const uint8_t* koq, int group_size, int sketch, int o_sketch, int n_rep) {
  return group_size == G && sketch == SKETCH && (o_sketch == 128 || o_sketch == 256) && n_rep <= R && aligned16(kq) && aligned16(koq);
}

int run(const uint8_t* kq, const uint8_t* koq, const void* kn, const void* kon, const uint8_t* idx, const float* qs, const void* q,
        const void* proj, int proj_dtype, int n_kbh, int n_rep, int n_groups, int o_sketch, int oc, int dtype, float* scores, cudaStream_t st) {
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return CQ_ERR_LAUNCH;
  Args a;
  a.n_kbh = n_kbh; a.n_groups = n_groups; a.n_rep = n_rep; a.o_sketch = o_sketch; a.oc = oc;
  // groups per tile: the first product costs a tile about as much as two thirds of a unit, whatever its width; smaller tiles where
  // they fill the SMs better, or where they hold the same groups (four heads of 4 groups: 11.2 us with tiles of 16, 10.0 with tiles of
  // 4; on the warp MMA 10.8)
  a.n_tiles = 0;
  double best = 1e30;
  for (int tg = MAX_TG; tg >= UNIT_G; tg /= 2) {
    const int per = (n_groups + tg - 1) / tg;
    const int64_t tiles = (int64_t)n_kbh * per;
    if (tiles > 0x7fffffff) continue;
    const int units = tg < n_groups ? tg / UNIT_G : (n_groups + UNIT_G - 1) / UNIT_G;
    const double cost = (double)((tiles + sms - 1) / sms) * (units + 0.7);
    if (cost <= best) { best = cost; a.tg = tg; a.tiles_per_kbh = per; a.n_tiles = (int)tiles; }
  }
  if (a.n_tiles == 0) return CQ_ERR_UNSUPPORTED;
  a.idesc_q = make_idesc(0, 0, 128, a.tg * R);
  a.idesc_q_first = make_idesc(0, 0, 128, a.tg * R + 16);
  a.idesc_in = make_idesc(0, 1, 128, N_IN);
  a.idesc_out = make_idesc(0, 1, 128, N_OUT);
  const int grid = a.n_tiles < sms ? a.n_tiles : sms;
#define CQ_SCORE(T, TP) launch<T, TP>(a, grid, kq, koq, kn, kon, idx, qs, q, proj, scores, st)
  if (dtype == CQ_DTYPE_F16) return proj_dtype == CQ_DTYPE_F32 ? CQ_SCORE(__half, float) : CQ_SCORE(__half, __half);
  return proj_dtype == CQ_DTYPE_F32 ? CQ_SCORE(__nv_bfloat16, float) : CQ_SCORE(__nv_bfloat16, __nv_bfloat16);
#undef CQ_SCORE
}

int status() {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_status, sizeof(int)) == cudaSuccess ? v : CQ_ERR_LAUNCH;
}

}  // namespace qjl_score
}  // namespace cq
