// QJL key sketching on the 5th-generation tensor cores: norms, outlier channels and both sign sketches of grouped keys in
// one persistent launch (groups of 32 keys, 256 projections).
//
// What bounded the step before: five torch launches in front of the quantizer (a copy of the strided keys, two norm
// reductions, top-k and its sort: 175 us for 4 x 8 x 6656 keys) and the quantizer itself on the warp MMA (223 us: 2048
// m16n8k16 products per group at 8 cycles of a scheduler's pipe each, 97 us if nothing else took time).
// Here a tile is 128 keys = 4 groups, the M of a tcgen05.mma:
//   D_all = K S^T, D_out = K_out S^T    K_out = the keys with all but their group's outlier channels zeroed; S as fp16
//                                       hi + lo rows (fp32-exact sums), resident in shared memory as the B operand
//   sketch bits: D_all - D_out > 0 and D_out > 0
// 16 worker warps load a tile (strided, 16-byte pieces), take the norms, rank the 128 channels of a group by
// (norm, lower index first), write both A tiles in the 128-byte-swizzled K-major layout and read the accumulators back;
// the 17th warp issues the products.  The two 128-projection halves of the accumulators are handed over separately, so that one
// half is read while the other is being computed, and the statistics of the next tile lie under the products of this one.
// 4 x 8 x 6688 bfloat16 keys, 32 outlier channels: 406 us for the six launches before, 80 us for this one.
// Every wait is bounded; on a timeout the CTA writes the status word, frees its tensor memory and returns.
#include <type_traits>

#include "cq_common.cuh"
#include "cq_ptx.cuh"
#include "cq_tc.cuh"

namespace cq {
namespace qjl_score {      // cq_qjl_score.cu
int status();
}
namespace qjl_build {

using namespace ptx;
using namespace tc;

constexpr int G = 32, TILE = 128, SKETCH = 256;
constexpr int WORKERS = 512, THREADS = WORKERS + 32, NW = WORKERS / 32;
constexpr int A_BYTES = TILE * kHeadDim * 2;              // one A tile: two 64-channel panels of [128 rows][128 bytes]
constexpr int B_BYTES = SKETCH * kHeadDim * 2;            // one B table: two panels of [256 rows][128 bytes]
constexpr int A_PANEL = A_BYTES / 2, B_PANEL = B_BYTES / 2;
constexpr int PART_BYTES = NW * kHeadDim * 4;             // per group: channel sums of the worker warps
constexpr int SMEM = 2 * B_BYTES + 2 * A_BYTES + 4 * PART_BYTES + 4 * kHeadDim * 2 + 1024;
constexpr uint32_t WAIT_TRIES = 1u << 22;
constexpr int64_t NOWHERE = INT64_MIN;                      // a group past the end

struct Args {
  int64_t n_groups_total;      // batch * heads * n_groups
  int heads, n_groups, oc, o_sketch;
  int64_t stride_b, stride_h, stride_t;
  uint32_t idesc;
};

__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory"); }
__device__ __forceinline__ void group_sync(int gg) { asm volatile("bar.sync %0, %1;" ::"r"(2 + gg), "n"(WORKERS / 4) : "memory"); }

template <typename T>
__device__ __forceinline__ uint32_t half_pair(uint32_t v) {
  if (std::is_same<T, __nv_bfloat16>::value) {             // bfloat16 -> fp16 (8 significant bits fit)
    const __half2 h = __floats2half2_rn(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  return v;
}

template <typename TP> __device__ __forceinline__ float proj_f(TP v);
template <> __device__ __forceinline__ float proj_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float proj_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float proj_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// given_idx: the outlier channels of every group (then idx_out and key_norm are not written), or nullptr.
template <typename T, typename TP>
__global__ void __launch_bounds__(THREADS, 1)
build_kernel(const Args a, const T* __restrict__ keys, const uint8_t* __restrict__ given_idx, const TP* __restrict__ proj,
             uint8_t* __restrict__ idx_out, uint8_t* __restrict__ key_quant, uint8_t* __restrict__ key_outlier_quant,
             T* __restrict__ key_norm, T* __restrict__ outlier_norm, int* __restrict__ status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* b_s = smem;                              // hi, lo
  unsigned char* a_s = smem + 2 * B_BYTES;                // all, outliers
  float* part_s = reinterpret_cast<float*>(a_s + 2 * A_BYTES);                        // [group][warp][channel]
  T* norm_s = reinterpret_cast<T*>(part_s + 4 * PART_BYTES / 4);                      // [group][channel] norms to rank
  __shared__ __align__(8) uint64_t bar_a, bar_d[2], bar_free[2];
  __shared__ uint32_t tmem_s;
  __shared__ uint32_t mask_s[4][4];
  __shared__ int64_t base_s[2][4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t n_tiles = (a.n_groups_total + 3) / 4;

  if (tid == 0) {
    mbar_init(&bar_a, WORKERS);
    for (int i = 0; i < 2; ++i) { mbar_init(&bar_d[i], 1); mbar_init(&bar_free[i], WORKERS); }
    mbar_fence_init();
  }
  if (warp == NW) tmem_alloc(&tmem_s, 512);
      // where the four groups of a tile start (64-bit divisions: one thread per group, a tile ahead)
  auto place = [&](int64_t tile, int slot) {
    if (tid >= 4) return;
    const int64_t grp = tile * 4 + tid;
    int64_t at = NOWHERE;
    if (grp < a.n_groups_total) {
      const int64_t bh = grp / a.n_groups, n = grp - bh * a.n_groups, b = bh / a.heads;
      at = b * a.stride_b + (bh - b * a.heads) * a.stride_h + n * G * a.stride_t;
    }
    base_s[slot][tid] = at;
  };
  // loader role: 16-byte piece ch of row r0 of each of the four groups
  const int ch = tid & 15, r0 = tid >> 4;
  uint4 v[4];
  auto load = [&](int slot) {
#pragma unroll
    for (int gg = 0; gg < 4; ++gg) {
      const int64_t at = base_s[slot][gg];
      v[gg] = make_uint4(0u, 0u, 0u, 0u);
      if (at != NOWHERE) v[gg] = *reinterpret_cast<const uint4*>(keys + at + r0 * a.stride_t + ch * 8);
    }
  };
  place(blockIdx.x, 0);
  place((int64_t)blockIdx.x + gridDim.x, 1);
  __syncthreads();
  if (warp < NW) load(0);      // in flight while the table is built
  // S, rows of projections, as hi and lo in the swizzled K-major layout
  const bool wide = reinterpret_cast<uintptr_t>(proj) % 16 == 0;
#pragma unroll 2
  for (int i = tid; i < SKETCH * 16; i += THREADS) {
    const int p = i >> 4, pc = i & 15;
    const TP* src = proj + (int64_t)p * kHeadDim + pc * 8;
    __align__(16) TP piece[8];
    if (wide) {
#pragma unroll
      for (int j = 0; j < (int)(sizeof(TP) * 8 / 16); ++j) reinterpret_cast<uint4*>(piece)[j] = reinterpret_cast<const uint4*>(src)[j];
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) piece[j] = src[j];
    }
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float x0 = proj_f<TP>(piece[2 * j]), x1 = proj_f<TP>(piece[2 * j + 1]);
      const __half2 h = __floats2half2_rn(x0, x1);
      const float2 f = __half22float2(h);
      const __half2 l = __floats2half2_rn(x0 - f.x, x1 - f.y);
      hi[j] = *reinterpret_cast<const uint32_t*>(&h);
      lo[j] = *reinterpret_cast<const uint32_t*>(&l);
    }
    unsigned char* dst = b_s + (pc >> 3) * B_PANEL + p * 128 + (((pc & 7) ^ (p & 7)) << 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + B_BYTES) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;      // columns: all [0, 256), outliers [256, 512)
  bool ok = true;

  if (warp == NW) {
    // ================= products =================
    // the whole warp runs the loop and one elected lane issues, so that the operands are uniform
    const uint32_t lead = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    auto all = [](bool r) { return __all_sync(0xffffffffu, r) != 0; };
    const uint64_t ad = smem_desc(smem_u32(a_s), 16, 1024), bd = smem_desc(smem_u32(b_s), 16, 1024);
    uint32_t i = 0;
    for (int64_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++i) {
      ok = all(mbar_wait_bounded(&bar_a, i & 1, WAIT_TRIES));
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (i > 0) ok = ok && all(mbar_wait_bounded(&bar_free[half], (i - 1) & 1, WAIT_TRIES));
        if (!ok) break;
        tc_fence_after();
        if (lead) {
#pragma unroll
          for (int src = 0; src < 2; ++src)
#pragma unroll
            for (int hl = 0; hl < 2; ++hl)
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)      // 16 channels per step; 128 projections further down a panel for half 1
                umma(tm + (uint32_t)(src * 256 + half * 128), ad + (uint64_t)((src * A_BYTES + (ks >> 2) * A_PANEL + (ks & 3) * 32) >> 4),
                     bd + (uint64_t)((hl * B_BYTES + (ks >> 2) * B_PANEL + half * 128 * 128 + (ks & 3) * 32) >> 4), a.idesc, (hl > 0 || ks > 0) ? 1u : 0u);
          umma_commit(&bar_d[half]);
        }
      }
    }
    if (!ok && lead) atomicExch(status, CQ_ERR_TIMEOUT);
    __syncwarp();
  } else {
    // ================= workers =================
    auto value = [&](int j, int e) -> float {      // element e of the thread's piece of group j
      const uint32_t w = reinterpret_cast<const uint32_t*>(&v[j])[e >> 1];
      const typename Elem<T>::T2 p = *reinterpret_cast<const typename Elem<T>::T2*>(&w);
      const float2 f = Elem<T>::to_f2(p);
      return (e & 1) ? f.y : f.x;
    };
    // sums of four rows (one per group) over the sixteen lanes of a row -> norms; every lane ends with one of the four
    auto row_norms = [&](int64_t tile, const float (&s)[4], T* dst) {
      const bool b3 = lane & 8, b2 = lane & 4;
      const float p = (b3 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, b3 ? s[0] : s[2], 8);
      const float q = (b3 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, b3 ? s[1] : s[3], 8);
      float x = (b2 ? q : p) + __shfl_xor_sync(0xffffffffu, b2 ? p : q, 4);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      const int64_t grp = tile * 4 + (b3 ? 2 : 0) + (b2 ? 1 : 0);
      if ((lane & 3) == 0 && grp < a.n_groups_total) dst[grp * G + r0] = Elem<T>::from_f(sqrtf(x));
    };
    // key norms, channel norms -> outlier channels of the four groups (mask words in mask_s), outlier norms
    auto statistics = [&](int64_t tile) {
      if (!given_idx) {
        const int gg = warp >> 2, c0 = 32 * (warp & 3) + lane;      // ranking role: one channel of one group per lane
        float rs[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float cs[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) { const float x = value(j, e); cs[e] = x * x; }
          rs[j] = ((cs[0] + cs[1]) + (cs[2] + cs[3])) + ((cs[4] + cs[5]) + (cs[6] + cs[7]));
          // two rows per warp: each half keeps four of the eight channel sums
          float out[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) out[e] = (lane < 16 ? cs[e] : cs[4 + e]) + __shfl_xor_sync(0xffffffffu, lane < 16 ? cs[4 + e] : cs[e], 16);
          *reinterpret_cast<float4*>(part_s + (j * NW + warp) * kHeadDim + ch * 8 + (lane < 16 ? 0 : 4)) = make_float4(out[0], out[1], out[2], out[3]);
        }
        workers_sync();
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) s += part_s[(gg * NW + w) * kHeadDim + c0];
        // a channel's norm as the data type holds it; not a number ranks with infinity
        T mine = Elem<T>::from_f(sqrtf(s));
        if (!(Elem<T>::to_f(mine) <= 3.4e38f)) mine = Elem<T>::from_f(INFINITY);
        norm_s[gg * kHeadDim + c0] = mine;
        row_norms(tile, rs, key_norm);
        group_sync(gg);
        // rank = channels with a greater norm + channels with the same one and a lower index: >= for the 32-channel blocks
        // before this warp's, > after it, > and the matching lower lanes within it; two compares and two counts an instruction
        const unsigned short mbits = *reinterpret_cast<const unsigned short*>(&mine);
        const typename Elem<T>::T2 mine2 = {mine, mine};
        typename Elem<T>::T2 count = {Elem<T>::from_f(0.f), Elem<T>::from_f(0.f)};
        const uint4* all = reinterpret_cast<const uint4*>(norm_s + gg * kHeadDim);
#pragma unroll
        for (int blk = 0; blk < 4; ++blk) {
          const bool before = blk < (warp & 3);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 o = all[4 * blk + i];
            const typename Elem<T>::T2* p = reinterpret_cast<const typename Elem<T>::T2*>(&o);
            if (before) {
#pragma unroll
              for (int k = 0; k < 4; ++k) count = __hadd2(count, __hge2(p[k], mine2));
            } else {
#pragma unroll
              for (int k = 0; k < 4; ++k) count = __hadd2(count, __hgt2(p[k], mine2));
            }
          }
        }
        const float2 cf = Elem<T>::to_f2(count);
        const int rank = (int)(cf.x + cf.y) + __popc(__match_any_sync(0xffffffffu, mbits) & ((1u << lane) - 1u));
        const int64_t grp = tile * 4 + gg;
        const uint32_t m = __ballot_sync(0xffffffffu, rank < a.oc);
        if (lane == 0) mask_s[gg][warp & 3] = m;
        if (rank < a.oc && grp < a.n_groups_total) idx_out[grp * a.oc + rank] = (uint8_t)c0;
      } else {
        workers_sync();      // the masks of the tile before have been taken
        if (tid < 16) mask_s[tid >> 2][tid & 3] = 0u;
        workers_sync();
        for (int i = tid; i < 4 * a.oc; i += WORKERS) {
          const int64_t grp = tile * 4 + i / a.oc;
          if (grp < a.n_groups_total) {
            const int c = given_idx[grp * a.oc + i % a.oc] & (kHeadDim - 1);
            atomicOr(&mask_s[i / a.oc][c >> 5], 1u << (c & 31));
          }
        }
      }
      workers_sync();
    };
    uint32_t mbyte[4];      // this thread's eight channels in the outlier masks of the four groups
    auto take_masks = [&](int64_t tile) {
#pragma unroll
      for (int gg = 0; gg < 4; ++gg) mbyte[gg] = (mask_s[gg][ch >> 2] >> (8 * (ch & 3))) & 0xffu;
      float rs[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        rs[j] = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float x = value(j, e);
          if ((mbyte[j] >> e) & 1u) rs[j] = fmaf(x, x, rs[j]);
        }
      }
      row_norms(tile, rs, outlier_norm);
    };
    auto stage = [&]() {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = G * j + r0;
        const uint32_t m = mbyte[j];
        uint32_t w[4], o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          w[k] = half_pair<T>(reinterpret_cast<const uint32_t*>(&v[j])[k]);
          const uint32_t keep = ((m >> (2 * k)) & 1u ? 0x0000ffffu : 0u) | ((m >> (2 * k + 1)) & 1u ? 0xffff0000u : 0u);
          o[k] = w[k] & keep;
        }
        unsigned char* dst = a_s + (ch >> 3) * A_PANEL + r * 128 + (((ch & 7) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(dst + A_BYTES) = make_uint4(o[0], o[1], o[2], o[3]);
      }
      fence_proxy_async_smem();
      mbar_arrive(&bar_a);
    };
    // accumulators of one half: warp w reads its 32 rows (TMEM lanes 32 (w % 4) ..), columns 32 (w / 4) .. + 31
    auto read_half = [&](int64_t tile, int half, uint32_t phase) {
      if (ok) ok = mbar_wait_bounded(&bar_d[half], phase, WAIT_TRIES);
      tc_fence_after();
      const uint32_t base = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(half * 128 + 32 * (warp >> 2));
      // signs: in = all - out > 0, out > 0, each the sign bit of the opposite difference (which is +0 for equal numbers, and so 0
      // for a zero of either sign), shifted into the word: one addition and one funnel shift a bit.  Eight columns to a chain;
      // sixteen columns at a time, which is what the registers beside the next tile's keys hold
      uint32_t in_w = 0u, out_w = 0u;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t all[16], o[16];
        tmem_ld16_nowait(base + 16 * part, all);
        tmem_ld16_nowait(base + 256 + 16 * part, o);
        tmem_ld_wait();
        if (part == 1) { tc_fence_before(); mbar_arrive(&bar_free[half]); }
#pragma unroll
        for (int c8 = 0; c8 < 2; ++c8) {
          uint32_t iw = 0u, ow = 0u;
#pragma unroll
          for (int i = 7; i >= 0; --i) {
            const float x = __uint_as_float(o[8 * c8 + i]);
            iw = __funnelshift_l(__float_as_uint(x - __uint_as_float(all[8 * c8 + i])), iw, 1);
            ow = __funnelshift_l(__float_as_uint(0.f - x), ow, 1);
          }
          in_w |= iw << (16 * part + 8 * c8);
          out_w |= ow << (16 * part + 8 * c8);
        }
      }
      const int row = 32 * (warp & 3) + lane;
      const int64_t grp = tile * 4 + (row >> 5);
      if (ok && grp < a.n_groups_total) {
        const int64_t tok = tile * TILE + row;
        const int word = 4 * half + (warp >> 2);
        *reinterpret_cast<uint32_t*>(key_quant + tok * (SKETCH / 8) + 4 * word) = in_w;
        if (32 * word < a.o_sketch)
          *reinterpret_cast<uint32_t*>(key_outlier_quant + tok * (a.o_sketch / 8) + 4 * word) = out_w;
      }
    };

    uint32_t i = 0;
    int64_t tile = blockIdx.x, prev = -1;
    if (tile < n_tiles) { statistics(tile); take_masks(tile); }
    for (; tile < n_tiles; tile += gridDim.x, ++i) {
      if (prev >= 0 && ok) ok = mbar_wait_bounded(&bar_d[1], (i - 1) & 1, WAIT_TRIES);      // the A tiles have been read
      stage();
      const int64_t next = tile + gridDim.x;
      if (next < n_tiles) load((i + 1) & 1);
      place(next + gridDim.x, i & 1);      // read after the barriers of the statistics; this slot was last read before them
      if (prev >= 0) read_half(prev, 1, (i - 1) & 1);
      if (next < n_tiles) { statistics(next); take_masks(next); }
      read_half(tile, 0, i & 1);
      prev = tile;
    }
    if (prev >= 0) read_half(prev, 1, (i - 1) & 1);
    if (!ok && lane == 0) atomicExch(status, CQ_ERR_TIMEOUT);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == NW) tmem_dealloc(tmem, 512);
}

static __device__ int g_status;

template <typename T, typename TP>
static int launch(const Args& a, const void* keys, const uint8_t* given, const void* proj, uint8_t* idx, uint8_t* kq, uint8_t* koq,
                  void* knorm, void* onorm, cudaStream_t st) {
  int dev = 0, sms = 0;
  void* status = nullptr;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0 ||
      cudaGetSymbolAddress(&status, g_status) != cudaSuccess ||
      cudaFuncSetAttribute(build_kernel<T, TP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)
    return CQ_ERR_LAUNCH;
  const int64_t tiles = (a.n_groups_total + 3) / 4;
  build_kernel<T, TP><<<(unsigned)(tiles < sms ? tiles : sms), THREADS, SMEM, st>>>(
      a, static_cast<const T*>(keys), given, static_cast<const TP*>(proj), idx, kq, koq, static_cast<T*>(knorm), static_cast<T*>(onorm),
      static_cast<int*>(status));
  return check_launch();
}

bool eligible(const void* keys, int group_size, int head_dim, int sketch, int o_sketch, int oc, const int64_t* strides, const void* kq,
              const void* koq) {
  for (int i = 0; i < 3; ++i)
    if (strides[i] % 8) return false;
  return group_size == G && head_dim == kHeadDim && sketch == SKETCH && o_sketch > 0 && o_sketch <= SKETCH && o_sketch % 32 == 0 &&
         oc >= 0 && oc <= kHeadDim && aligned16(keys) && reinterpret_cast<uintptr_t>(kq) % 4 == 0 && reinterpret_cast<uintptr_t>(koq) % 4 == 0;
}

// keys: element (b, h, t, d) at keys[b*strides[0] + h*strides[1] + t*strides[2] + d]
int run(const void* keys, int batch, int heads, int n_groups, const int64_t* strides, const uint8_t* given, const void* proj, int proj_dtype,
        int o_sketch, int oc, int dtype, uint8_t* idx, uint8_t* kq, uint8_t* koq, void* knorm, void* onorm, cudaStream_t st) {
  Args a;
  a.n_groups_total = (int64_t)batch * heads * n_groups;
  a.heads = heads; a.n_groups = n_groups; a.oc = oc; a.o_sketch = o_sketch;
  a.stride_b = strides[0]; a.stride_h = strides[1]; a.stride_t = strides[2];
  a.idesc = make_idesc(0, 0, TILE, 128);
#define CQ_BUILD(T, TP) launch<T, TP>(a, keys, given, proj, idx, kq, koq, knorm, onorm, st)
  if (dtype == CQ_DTYPE_F16) return proj_dtype == CQ_DTYPE_F32 ? CQ_BUILD(__half, float) : CQ_BUILD(__half, __half);
  return proj_dtype == CQ_DTYPE_F32 ? CQ_BUILD(__nv_bfloat16, float) : CQ_BUILD(__nv_bfloat16, __nv_bfloat16);
#undef CQ_BUILD
}

}  // namespace qjl_build
}  // namespace cq

extern "C" int cq_qjl_status(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, cq::qjl_build::g_status, sizeof(int)) != cudaSuccess) return CQ_ERR_LAUNCH;
  return v != 0 ? v : cq::qjl_score::status();
}

extern "C" int cq_qjl_build(const void* keys, int batch, int heads, int n_groups, int group_size, int head_dim, const int64_t* strides,
                            const void* proj, int proj_dtype, int sketch_dim, int outlier_sketch_dim, int outlier_count, int dtype,
                            uint8_t* outlier_indices, uint8_t* key_quant, uint8_t* key_outlier_quant, void* key_norms,
                            void* outlier_norms, void* stream) {
  if (batch == 0 || heads == 0 || n_groups == 0) return CQ_OK;
  if (!keys || !strides || !proj || !outlier_indices || !key_quant || !key_outlier_quant || !key_norms || !outlier_norms)
    return CQ_ERR_BAD_ARG;
  if (batch < 0 || heads < 0 || n_groups < 0) return CQ_ERR_BAD_ARG;
  if (dtype != CQ_DTYPE_F16 && dtype != CQ_DTYPE_BF16) return CQ_ERR_BAD_ARG;
  if (proj_dtype != CQ_DTYPE_F32 && proj_dtype != dtype) return CQ_ERR_BAD_ARG;
  if (!cq::qjl_build::eligible(keys, group_size, head_dim, sketch_dim, outlier_sketch_dim, outlier_count, strides, key_quant, key_outlier_quant))
    return CQ_ERR_UNSUPPORTED;
  return cq::qjl_build::run(keys, batch, heads, n_groups, strides, nullptr, proj, proj_dtype, outlier_sketch_dim, outlier_count, dtype,
                            outlier_indices, key_quant, key_outlier_quant, key_norms, outlier_norms, static_cast<cudaStream_t>(stream));
}
