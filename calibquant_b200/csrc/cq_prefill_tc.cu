// Dense causal prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// One work item = 256 query rows as two 128-row tiles A and B that share the K/V stream: the same rows of two heads of a KV
// head, or (odd number of heads per KV head) adjacent rows of one head.  One CTA per SM; it starts with the item of its own
// block index and then takes over blocks of the grid that have not been launched yet (cluster launch control), so tensor
// memory, barriers and the pipeline are set up once per SM and the hardware's launch order and load balance are kept.  Roles:
//   warp 9 (one lane)  TMA producer: the item's Q tiles, then its 128-key K/V tiles through a two-stage ring
//                        that runs on across items; asks for the next block when an item's loads are issued
//   warp 8             MMA issuer (one elected lane):
//        S_X = Q_X K^T   tcgen05.mma kind::f16, A = Q_X and B = K from shared memory (K-major), D in the
//                        tile's 128 TMEM columns
//        O_X += P_X V    A = P_X read from TENSOR MEMORY (16-bit pairs the softmax warps stored over the
//                        first 64 columns of S_X), B = V from shared memory (MN-major), D accumulates in
//                        the tile's O columns over all key tiles
//   warps 0-3 / 4-7    softmax of tile A / B: thread = one query row (= TMEM lane).  It reads its 128
//                        logits once (tcgen05.ld), applies scale, causal mask and the online softmax
//                        with a lazy maximum, and stores P back to TMEM (tcgen05.st).  No cross-thread
//                        exchange: the two tiles run out of phase, so one tile's
//                        exponentials overlap the other tile's products on the tensor pipe.
// Lazy maximum: a row keeps its reference maximum until the true one exceeds it by more than 2^8, and
// only then are that row's O columns and running sum rescaled (tcgen05.ld / st between two PV
// products); probabilities stay below 256 and O is read back once, at the end.
// Epilogue: the normalised rows of a tile are staged in shared memory (swizzled box layout) and written
// with two tiled TMA stores, which also clip the rows past the end of the sequence.
// TMEM columns: S_A [0,128) S_B [128,256) O_A [256,384) O_B [384,512).  Operand tiles in shared
// memory use the 128-byte swizzle: a [128 rows x 64 elements] TMA box lands directly in the
// canonical UMMA layout (8-row atoms of 1024 bytes).
// Bound: the tensor pipe takes 64 cycles per M128 N128 K16 product (measured, from shared and from tensor memory alike), 2050
// for the 32 products of a key tile; the 2 x 128 x 128 exponentials take 2048 cycles of the special-function unit.  What
// is above that is the chain of one tile (S -> softmax -> P V -> next S) that the other tile does not cover.
// 16 x 3392 tokens, 32 query / 8 KV heads, bfloat16: 1642 us (918 TFLOP/s, causal) with one lane running the issuer's loop and
// spilling softmax warps; 1481 with the register split; 1384 (1090 TFLOP/s) with uniform issue.
//
// Every mbarrier wait is bounded; on a timeout the CTA records CQ_ERR_TIMEOUT in the status word,
// skips its remaining waits, frees its TMEM and returns.
#include <cuda.h>
#include <stdlib.h>

#include <type_traits>

#include "cq_common.cuh"
#include "cq_ptx.cuh"
#include "cq_tc.cuh"

namespace cq {
namespace prefill_tc {

using namespace ptx;
using namespace tc;

constexpr int BM = 128, BN = 128;
constexpr int PANEL_BYTES = 128 * 128;          // [128 rows][64 x 16-bit]
constexpr int TILE_BYTES = 2 * PANEL_BYTES;     // [128 rows][128 x 16-bit]
constexpr int SMEM_BYTES = TILE_BYTES * 7 + 1024;   // Q x2, K x2, V x2, output staging (+ alignment slack)
constexpr int SOFTMAX_THREADS = 256, MMA_WARP = 8, TMA_WARP = 9, THREADS = SOFTMAX_THREADS + 128;
// A row's 128 logits and 32 words of probabilities do not fit the 168 registers that 384 threads start with: the softmax
// warpgroups take what the third one (producer, issuer, two idle warps) gives up.  256 x 200 + 128 x 96 = 63 488 of the
// launch's 384 x 168 = 64 512.
constexpr int SOFTMAX_REGS = 200, CONTROL_REGS = 96;
constexpr uint32_t WAIT_TRIES = 1u << 22;
constexpr long long WAIT_CYCLES = 1ll << 30;     // ~0.5 s: bound of the waits on the S / P hand-offs
constexpr uint32_t TMEM_COLS = 512;
constexpr float RESCALE_LOG2 = 8.f;          // a row is rescaled when its maximum grew by more than 2^8

struct Params {
  int t_len, hq, hkv;
  int pair;              // 1: the two tiles of an item are the same queries of two heads; 0: adjacent tiles of one head
  int by_length;         // 1: block order (head, batch row, query rows), all longest rows first; 0: (query rows, head, batch row)
  float scale_log2;
  uint32_t idesc_s, idesc_pv;
  int is_bf16;
  int* status;
};

__device__ __forceinline__ void tma_load_4d(void* dst, const void* tmap, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(smem_u32(dst)), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

// 4-D tiled store shared -> global (rows past the tensor's extent are clipped), tracked by the thread's bulk group
__device__ __forceinline__ void tma_store_4d(const void* tmap, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
      ::"l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(src))
      : "memory");
}
// closes the thread's bulk group and waits until its stores have read their shared-memory source
__device__ __forceinline__ void tma_store_commit_wait_read() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// Cluster launch control: a running CTA asks for the grid's next CTA that has not been launched yet.  On success
// that CTA is never launched and the 16-byte response names its block index, so the caller does its work: the
// hardware's own launch order and load balance, without the launch gap and the set-up of a new CTA.
// After a request has failed (nothing left to cancel) no further request may be issued.
__device__ __forceinline__ void clc_try_cancel(void* resp, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(resp)), "r"(smem_u32(bar)) : "memory");
}
// decodes a response; false: the request failed, there is no further work
__device__ __forceinline__ bool clc_read(const void* resp, int& bx, int& by, int& bz) {
  uint32_t valid = 0, x = 0, y = 0, z = 0;
  asm volatile(
      "{\n\t.reg .pred p1;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p1, r;\n\t"
      "selp.u32 %3, 1, 0, p1;\n\t"
      "@p1 clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n\t}"
      : "+r"(x), "+r"(y), "+r"(z), "+r"(valid)
      : "r"(smem_u32(resp))
      : "memory");
  fence_proxy_async_smem();       // the slot is written again through the async proxy
  bx = (int)x; by = (int)y; bz = (int)z;
  return valid != 0;
}
// A use counter in shared memory (monotonic, so a waiter may be any number of uses behind or ahead, which the
// parity of an mbarrier phase cannot express): bounded wait until it has reached `target`.
__device__ __forceinline__ bool wait_count(const uint32_t* ctr, uint32_t target, uint32_t max_tries) {
#pragma unroll 1
  for (uint32_t i = 0; i < max_tries; ++i) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(ctr)) : "memory");
    if (v >= target) return true;
    __nanosleep(32);
  }
  return false;
}
__device__ __forceinline__ void publish_count(uint32_t* ctr, uint32_t v) {
  asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(ctr)), "r"(v) : "memory");
}
// barrier among the four softmax warps of one query tile that also tells whether ALL of them passed `flag`
__device__ __forceinline__ bool tile_all(int id, bool flag) {
  uint32_t out;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(out) : "r"((uint32_t)flag), "r"(id) : "memory");
  return out != 0;
}
// barrier among the four softmax warps of one query tile
__device__ __forceinline__ void tile_barrier(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

// register split between warpgroups; every warp of a group runs it
template <int N> __device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// sm_100 arithmetic that halves the instruction count of the softmax: 3-input maximum, and fp32
// operations on register pairs
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// (x0, x1) = (a0, a1) * (b, b) + (c, c)
__device__ __forceinline__ void fma_pair(float& x0, float& x1, float a0, float a1, float b, float c) {
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%5, %5};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(x0), "=f"(x1) : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
// (s0, s1) += (a0, a1)
__device__ __forceinline__ void add_pair(float& s0, float& s1, float a0, float a1) {
  asm("{\n\t.reg .b64 ra, rs;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rs, {%0, %1};\n\t"
      "add.rn.f32x2 rs, rs, ra;\n\tmov.b64 {%0, %1}, rs;\n\t}"
      : "+f"(s0), "+f"(s1) : "f"(a0), "f"(a1));
}

template <bool IS_BF16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
  if (IS_BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// One work item = one block index of the grid.  A CTA starts with its own index and then takes over blocks that have not been
// launched yet (cluster launch control), in block order.  Where the keys and values do not fit L2 the query rows run fastest
// (longest first): the CTAs running at the same time then work on the query blocks and heads of a few KV heads, whose K/V
// tiles stay in L2, as with one CTA per block; items sorted by length lost that and ran 6 % slower at 16 x 3392 tokens.
// Where they do fit, all longest items come first, so that the CTAs end together: 2 x 1401 tokens 51 -> 42 us, 1 x 3433 114 -> 94, 3 x 2500 173 -> 150, 2 x 6697 654 -> 624.
struct Item {
  int h, b, hk, q0, n_a, n_b, n_max;        // tile X = 0 (A), 1 (B): head h + X pair, queries q0 + X (1 - pair) BM ..
};
__device__ __forceinline__ Item decode_item(const Params& p, int bx, int by, int bz) {
  Item w;
  const int qt = p.by_length ? (int)gridDim.z - 1 - bz : (int)gridDim.x - 1 - bx;         // longest rows first
  w.h = (p.by_length ? bx : by) << p.pair;
  w.b = p.by_length ? by : bz;
  w.hk = w.h / (p.hq / p.hkv);
  w.q0 = qt * (2 - p.pair) * BM;
  const int t_tiles = (p.t_len + BN - 1) / BN, q1 = p.pair ? w.q0 : w.q0 + BM;
  // key tiles of query tile A, B; B may lie wholly past the end
  w.n_a = min((w.q0 + BM + BN - 1) / BN, t_tiles);
  w.n_b = q1 < p.t_len ? min((q1 + BM + BN - 1) / BN, t_tiles) : 0;
  w.n_max = max(w.n_a, w.n_b);
  return w;
}

template <bool IS_BF16>
__global__ void __launch_bounds__(THREADS, 1)
prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, Params p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* q_s = smem;                    // tiles A, B
  unsigned char* k_s = q_s + 2 * TILE_BYTES;    // 2 stages
  unsigned char* v_s = k_s + 2 * TILE_BYTES;    // 2 stages
  unsigned char* o_s = v_s + 2 * TILE_BYTES;    // output staging, used by the two tiles in turn
  // Barriers.  Their phases run on across the CTA's items: every role keeps the count of completions it has seen.
  //   bar_q[X]       Q_X of an item has landed                         (once per item)
  //   bar_q_free[X]  the last S_X of an item has completed: Q_X may be overwritten   (once per item)
  //   bar_kv_full/free[stage]   K/V ring                               (once per key tile of the CTA)
  //   bar_s[X]       S_X ready;  bar_p[X][half]  P_X of keys 0-63 / 64-127 stored (128 arrivals);
  //   bar_pv[X]      O_X += P_X V done                                 (once per key tile of X)
  //   stage_done     (a counter, not a barrier) uses of the staging buffer whose stores have read it
  //   bar_clc_full/free[slot]   the response naming the CTA's next item has arrived / has been read by the MMA
  //                  thread and the eight softmax warps (item i's successor travels through slot i % 2)
  __shared__ __align__(8) uint64_t bar_q[2], bar_q_free[2], bar_kv_full[2], bar_kv_free[2], bar_s[2], bar_p[2][2],
      bar_pv[2], bar_clc_full[2], bar_clc_free[2];
  __shared__ __align__(16) uint4 clc_resp[2];
  __shared__ uint32_t stage_done;
  __shared__ uint32_t tmem_base_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar_q[s], 1);
      mbar_init(&bar_q_free[s], 1);
      mbar_init(&bar_kv_full[s], 1);
      mbar_init(&bar_kv_free[s], 1);
      mbar_init(&bar_s[s], 1);
      mbar_init(&bar_p[s][0], SOFTMAX_THREADS / 2);
      mbar_init(&bar_p[s][1], SOFTMAX_THREADS / 2);
      mbar_init(&bar_pv[s], 1);
      mbar_init(&bar_clc_full[s], 1);
      mbar_init(&bar_clc_free[s], 1 + SOFTMAX_THREADS / 32);
    }
    stage_done = 0;
    mbar_fence_init();
  }
  // The launch before this one may still run up to here.  The wait comes before the tensor memory is taken: a kernel that
  // this one waits for must not have to wait for it.
  pdl_wait();
  if (warp == MMA_WARP) tmem_alloc(&tmem_base_s, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;

  if (warp >= SOFTMAX_THREADS / 32) {
    setmaxnreg_dec<CONTROL_REGS>();
    if (warp == TMA_WARP) {
      // ================= TMA producer (one lane) =================
      if (lane == 0) {
        bool ok = true;
        uint32_t kv = 0;                          // K/V tiles this CTA has loaded so far
        int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
        for (uint32_t it = 0; ok; ++it) {         // items of this CTA
          const Item w = decode_item(p, bx, by, bz);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            // Q_x of the previous item is read until its last S_x has completed
            if (it > 0) ok = ok && mbar_wait_bounded(&bar_q_free[x], (it - 1) & 1, WAIT_TRIES);
            if (!ok) break;
            mbar_expect_tx(&bar_q[x], TILE_BYTES);
            const int hx = w.h + x * p.pair, qx0 = w.q0 + x * (1 - p.pair) * BM;
            tma_load_4d(q_s + x * TILE_BYTES, &tm_q, 0, hx, qx0, w.b, &bar_q[x]);
            tma_load_4d(q_s + x * TILE_BYTES + PANEL_BYTES, &tm_q, 64, hx, qx0, w.b, &bar_q[x]);
          }
          for (int j = 0; j < w.n_max && ok; ++j, ++kv) {
            const uint32_t s = kv & 1;
            if (kv >= 2) ok = mbar_wait_bounded(&bar_kv_free[s], ((kv - 2) >> 1) & 1, WAIT_TRIES);
            if (!ok) break;
            mbar_expect_tx(&bar_kv_full[s], 2 * TILE_BYTES);
            tma_load_4d(k_s + s * TILE_BYTES, &tm_k, 0, w.hk, j * BN, w.b, &bar_kv_full[s]);
            tma_load_4d(k_s + s * TILE_BYTES + PANEL_BYTES, &tm_k, 64, w.hk, j * BN, w.b, &bar_kv_full[s]);
            tma_load_4d(v_s + s * TILE_BYTES, &tm_v, 0, w.hk, j * BN, w.b, &bar_kv_full[s]);
            tma_load_4d(v_s + s * TILE_BYTES + PANEL_BYTES, &tm_v, 64, w.hk, j * BN, w.b, &bar_kv_full[s]);
          }
          if (!ok) break;
          // All loads of this item are on their way (the other roles are about two key tiles behind): ask for the
          // item's successor now, not earlier, so that a CTA does not sit on a block another CTA could start.
          const uint32_t slot = it & 1;
          if (it >= 2) ok = mbar_wait_bounded(&bar_clc_free[slot], ((it >> 1) - 1) & 1, WAIT_TRIES);
          if (!ok) break;
          mbar_expect_tx(&bar_clc_full[slot], 16);
          clc_try_cancel(&clc_resp[slot], &bar_clc_full[slot]);
          ok = mbar_wait_bounded(&bar_clc_full[slot], (it >> 1) & 1, WAIT_TRIES);
          if (!ok || !clc_read(&clc_resp[slot], bx, by, bz)) break;
        }
        if (!ok) atomicExch(p.status, CQ_ERR_TIMEOUT);
      }
      __syncwarp();
    } else if (warp == MMA_WARP) {
      // ================= MMA issuer =================
      // The whole warp runs the loop and one elected lane issues: control flow and operands are uniform, so that a product costs
      // the issuing lane a few instructions (one lane alone in the loop, with the stage as an index, could not keep the pipe fed)
      const uint32_t lead = elect_one();
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint32_t q_b = smem_u32(q_s), k_b = smem_u32(k_s), v_b = smem_u32(v_s);
      // descriptors of the operand tiles; a k-step only moves the start address (14-bit field of
      // 16-byte units in the low word, which cannot carry: shared memory ends below 256 KB)
      const uint64_t qd = smem_desc(q_b, 16, 1024), kd = smem_desc(k_b, 16, 1024), vd = smem_desc(v_b, PANEL_BYTES, 1024);
      auto issue_s = [&](auto xc, auto sc) {        // S_x = Q_x K^T on the K tile of that stage, known to be there
        constexpr int x = decltype(xc)::value, st = decltype(sc)::value;
        if (lead) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {          // 16 channels per step; panel = ks/4, 32 B per step
            constexpr uint64_t tile = TILE_BYTES >> 4;
            const uint64_t off = (uint64_t)(((ks >> 2) * PANEL_BYTES + (ks & 3) * 32) >> 4);
            umma(tm + (uint32_t)x * 128u, qd + (x * tile + off), kd + (st * tile + off), p.idesc_s, ks > 0);
          }
          umma_commit(&bar_s[x]);
        }
      };
      // O_x += P_x(j) V(j) of half the keys, 16 keys = 8 TMEM columns per step
      auto issue_pv = [&](auto xc, auto sc, auto hc, bool acc) {
        constexpr int x = decltype(xc)::value, st = decltype(sc)::value, hf = decltype(hc)::value;
        if (lead) {
#pragma unroll
          for (int ks = 4 * hf; ks < 4 * hf + 4; ++ks)
            umma_ts(tm + 256u + (uint32_t)x * 128u, tm + (uint32_t)x * 128u + (uint32_t)ks * 8u,
                    vd + (uint64_t)((st * TILE_BYTES + ks * 2048) >> 4), p.idesc_pv, (ks > 0 || acc) ? 1u : 0u);
        }
      };
      auto commit = [&](uint64_t* bar) { if (lead) umma_commit(bar); };
      using C0 = std::integral_constant<int, 0>;
      using C1 = std::integral_constant<int, 1>;
      // every decision is the whole warp's, a timeout of one lane included
      auto all = [](bool r) { return __all_sync(0xffffffffu, r) != 0; };
      bool ok = true;
      uint32_t kv = 0, cnt[2] = {0, 0};             // K/V tiles, key tiles of A / B done so far
      int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
      Item w = decode_item(p, bx, by, bz);
      bool begun = false;                           // the item's S_A(0) has been issued behind the item before
      for (uint32_t it = 0; ok; ++it) {
        auto first_s = [&](auto xc) {
          constexpr int x = decltype(xc)::value;
          const int n = x == 0 ? w.n_a : w.n_b;
          if (x == 0 && begun) return;
          ok = ok && all(mbar_wait_bounded(&bar_q[x], it & 1, WAIT_TRIES));
          if (!ok) return;
          tc_fence_after();
          if (n > 0) { if (kv & 1) issue_s(xc, C1{}); else issue_s(xc, C0{}); }
          if (n <= 1) commit(&bar_q_free[x]);       // that was the item's last S_x (or it has none)
        };
        ok = all(mbar_wait_bounded(&bar_kv_full[kv & 1], (kv >> 1) & 1, WAIT_TRIES));
        first_s(C0{});
        first_s(C1{});
        // the item's successor: 0 not asked yet, 1 known, 2 there is none
        int next = 0;
        Item w2 = w;
        auto take_next = [&]() {
          next = clc_read(&clc_resp[it & 1], bx, by, bz) ? 1 : 2;
          __syncwarp();
          if (lead) mbar_arrive(&bar_clc_free[it & 1]);
          if (next == 1) w2 = decode_item(p, bx, by, bz);
        };
        begun = false;
        bool next_k_ready = false;
        // key tile j of query tile x, whose K/V tile is in stage st
        auto step = [&](auto xc, auto sc, int j) {
          constexpr int x = decltype(xc)::value, st = decltype(sc)::value;
          using Other = std::integral_constant<int, st ^ 1>;
          const int n = x == 0 ? w.n_a : w.n_b;
          if (j >= n) return;
          // the first four steps start as soon as the probabilities of keys 0-63 are stored, while the softmax warps work
          // on keys 64-127
          ok = all(mbar_wait_cycles(&bar_p[x][0], (cnt[x] + j) & 1, WAIT_CYCLES));
          if (!ok) return;
          tc_fence_after();
          issue_pv(xc, sc, C0{}, j > 0);
          ok = all(mbar_wait_cycles(&bar_p[x][1], (cnt[x] + j) & 1, WAIT_CYCLES));
          if (!ok) return;
          tc_fence_after();
          issue_pv(xc, sc, C1{}, true);
          commit(&bar_pv[x]);
          // S_x(j+1) overwrites the columns P_x(j) lives in; the tensor pipe runs in issue order
          if (j + 1 < n) {
            if (!next_k_ready) {
              ok = all(mbar_wait_bounded(&bar_kv_full[st ^ 1], ((kv + j + 1) >> 1) & 1, WAIT_TRIES));
              if (!ok) return;
              tc_fence_after();
              next_k_ready = true;
            }
            issue_s(xc, Other{});
            if (j + 2 == n) commit(&bar_q_free[x]);     // the item's last S_x
          } else if (x == 0 && w.n_a == w.n_b) {
            // A is through with the item, B still has P V of its last tile to come: the successor's S_A goes in between,
            // as within an item, if its operands are there already (otherwise after B, where waiting holds up nothing).
            // Tiles of unequal length would come into phase here and lose the overlap of softmax and products
            if (all(mbar_try_wait(&bar_clc_full[it & 1], (it >> 1) & 1))) take_next();
            if (next == 1 && all(mbar_try_wait(&bar_q[0], (it + 1) & 1)) && all(mbar_try_wait(&bar_kv_full[st ^ 1], ((kv + j + 1) >> 1) & 1))) {
              tc_fence_after();
              issue_s(C0{}, Other{});                   // n_a > 0 in every item
              if (w2.n_a == 1) commit(&bar_q_free[0]);
              begun = true;
            }
          }
        };
        for (int j = 0; j < w.n_max && ok; ++j) {
          const uint32_t s = (kv + j) & 1;
          next_k_ready = false;
          if (s == 0) {
            step(C0{}, C0{}, j);
            if (ok) step(C1{}, C0{}, j);
          } else {
            step(C0{}, C1{}, j);
            if (ok) step(C1{}, C1{}, j);
          }
          if (!ok) break;
          commit(&bar_kv_free[s]);                  // K(j), V(j) are free once everything issued so far has drained
        }
        kv += (uint32_t)w.n_max;
        cnt[0] += (uint32_t)w.n_a;
        cnt[1] += (uint32_t)w.n_b;
        if (!ok) break;
        if (next == 0) {
          ok = all(mbar_wait_bounded(&bar_clc_full[it & 1], (it >> 1) & 1, WAIT_TRIES));
          if (!ok) break;
          take_next();
        }
        if (next == 2) break;
        w = w2;
      }
      if (!ok && lead) atomicExch(p.status, CQ_ERR_TIMEOUT);
      __syncwarp();
    }
  } else {
    setmaxnreg_inc<SOFTMAX_REGS>();
    // ===== softmax: warps 0-3 tile A, 4-7 tile B; thread = one query row =====
    const int x = warp >> 2, quarter = warp & 3;
    const int r_in = quarter * 32 + lane;               // row inside the tile = TMEM lane
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem + (uint32_t)x * 128u + lane_off;
    const uint32_t tO = tmem + 256u + (uint32_t)x * 128u + lane_off;
    bool ok = true;                                     // stays false after a timeout; later waits are skipped
    uint32_t cnt = 0, uses = 0;                         // key tiles of this tile / uses of the staging buffer so far
    int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
    for (uint32_t it = 0;; ++it) {
      const Item w = decode_item(p, bx, by, bz);
      const int n_x = x == 0 ? w.n_a : w.n_b;
      const int hx = w.h + x * p.pair, qx0 = w.q0 + x * (1 - p.pair) * BM;
      const int row = qx0 + r_in;
      float m_ref = -INFINITY, l_run = 0.f;             // reference maximum (log2 units), row sum
      for (int j = 0; j < n_x; ++j) {
        const int key0 = j * BN;
        const bool need_mask = (key0 + BN - 1 > qx0) || (key0 + BN > p.t_len);
        if (ok) ok = mbar_wait_cycles(&bar_s[x], (cnt + j) & 1, WAIT_CYCLES);
        tc_fence_after();
        uint32_t sv[4][32];                             // this row's 128 logits, read once
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) tmem_ld32_nowait(tS + cc * 32, sv[cc]);
        tmem_ld_wait();
        if (need_mask) {                                // diagonal and last key tiles only
          const int lim = min(row, p.t_len - 1) - key0; // columns above lim are masked
#pragma unroll
          for (int cc = 0; cc < 4; ++cc)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (cc * 32 + i > lim) sv[cc][i] = 0xff800000u;   // -inf
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(sv[cc][i]), __uint_as_float(sv[cc][i + 1]));
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        const float m_true = fmaxf(m_ref, mx * p.scale_log2);
        const bool grow = m_true - m_ref > RESCALE_LOG2;  // also true for the first tile (m_ref = -inf)
        if (j > 0 && __any_sync(0xffffffffu, grow)) {
          // O_x holds the products of tiles 0..j-1; the last of them must have completed
          if (ok) ok = mbar_wait_bounded(&bar_pv[x], (cnt + j - 1) & 1, WAIT_TRIES);
          tc_fence_after();
          const float alpha = grow ? exp2f(m_ref - m_true) : 1.f;
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            uint32_t r[32];
            tmem_ld32(tO + cc * 32, r);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st32(tO + cc * 32, r);
          }
          l_run *= alpha;
        }
        if (grow) m_ref = m_true;
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
        float rs4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int cc = 0; cc < 4; cc += 2) {
          uint32_t wv[32];                              // 64 probabilities as 16-bit pairs = 32 TMEM columns
#pragma unroll
          for (int i = 0; i < 64; i += 2) {
            // masked logits are -inf: ex2 gives 0
            float x0, x1;
            fma_pair(x0, x1, __uint_as_float(sv[cc + (i >> 5)][i & 31]), __uint_as_float(sv[cc + (i >> 5)][(i & 31) + 1]),
                     p.scale_log2, -m_use);
            const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
            add_pair(rs4[i & 2], rs4[(i & 2) + 1], p0, p1);
            wv[i >> 1] = pack16<IS_BF16>(p0, p1);
          }
          tmem_st32(tS + (cc >> 1) * 32, wv);           // over the first 64 columns of S_x
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(&bar_p[x][cc >> 1]);
        }
        l_run += (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]);
      }
      if (n_x > 0) {
        if (ok) ok = mbar_wait_bounded(&bar_pv[x], (cnt + n_x - 1) & 1, WAIT_TRIES);
        // the staging buffer is used by A, then B, of every item: wait until the use before this one has been read
        const uint32_t use = uses + (x == 1 && w.n_a > 0 ? 1u : 0u);
        if (ok) ok = wait_count(&stage_done, use, WAIT_TRIES);
        if (ok) {
          tc_fence_after();
          const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
          // The normalised rows go through shared memory in the layout of a 128-byte-swizzled TMA box and leave
          // as two tiled stores: a thread's row is 256 contiguous bytes in global memory, but the 32 rows of a
          // warp are a row pitch apart, and direct 16-byte stores from the registers cost the CTA ~5000 cycles.
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            uint32_t r[32];
            tmem_ld32(tO + cc * 32, r);
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 wq;
              wq.x = pack16<IS_BF16>(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv);
              wq.y = pack16<IS_BF16>(__uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
              wq.z = pack16<IS_BF16>(__uint_as_float(r[i + 4]) * inv, __uint_as_float(r[i + 5]) * inv);
              wq.w = pack16<IS_BF16>(__uint_as_float(r[i + 6]) * inv, __uint_as_float(r[i + 7]) * inv);
              const int chunk = (cc & 1) * 4 + (i >> 3);        // 16-byte chunk of the 128-byte panel row
              *reinterpret_cast<uint4*>(o_s + (cc >> 1) * PANEL_BYTES + r_in * 128 + ((chunk ^ (r_in & 7)) << 4)) = wq;
            }
          }
        }
        tc_fence_before();                              // O_x has been read: the next item's first P.V may overwrite it
        fence_proxy_async_smem();
        tile_barrier(1 + x);
        if (quarter == 0 && lane == 0) {
          if (ok) {
            tma_store_4d(&tm_o, o_s, 0, hx, qx0, w.b);
            tma_store_4d(&tm_o, o_s + PANEL_BYTES, 64, hx, qx0, w.b);
            tma_store_commit_wait_read();
          } else {
            atomicExch(p.status, CQ_ERR_TIMEOUT);
          }
          publish_count(&stage_done, use + 1);          // also after a timeout, so that nobody waits for this use
        }
      }
      cnt += (uint32_t)n_x;
      uses += (w.n_a > 0 ? 1u : 0u) + (w.n_b > 0 ? 1u : 0u);
      // the next item, if there is one
      if (ok) ok = mbar_wait_bounded(&bar_clc_full[it & 1], (it >> 1) & 1, WAIT_TRIES);
      bool more = ok && clc_read(&clc_resp[it & 1], bx, by, bz);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_clc_free[it & 1]);
      more = tile_all(1 + x, more);                     // the tile's four warps go on, or leave, together
      if (!more) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem, TMEM_COLS);
}

// ---- host ---------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
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

// [B, T, H, D] with element strides (sb, st, sh), D contiguous -> 4-D map (d, h, t, b), box 64 x 1 x 128 x 1
static bool make_map(CUtensorMap* m, const void* base, int is_bf16, int batch, int t_len, int heads,
                     const int64_t* strides) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {128, (cuuint64_t)heads, (cuuint64_t)t_len, (cuuint64_t)batch};
  cuuint64_t gstr[3] = {(cuuint64_t)strides[2] * 2, (cuuint64_t)strides[1] * 2, (cuuint64_t)strides[0] * 2};
  cuuint32_t box[4] = {64, 1, 128, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(m, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
            const_cast<void*>(base), dims, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace prefill_tc

bool prefill_tc_eligible(const int64_t* qs, const int64_t* ks, const int64_t* vs, const int64_t* os) {
  if (!prefill_tc::encode_fn()) return false;
  const int64_t* all[] = {qs, ks, vs, os};
  for (const int64_t* s : all)
    for (int i = 0; i < 3; ++i)
      if (s[i] % 8 || s[i] <= 0) return false;
  return true;
}

int prefill_tc_run(const void* q, const void* k, const void* v, void* out, int batch, int t_len, int hq, int hkv,
                   const int64_t* qs, const int64_t* ks, const int64_t* vs, const int64_t* os, int is_bf16,
                   int* status, cudaStream_t st) {
  using namespace prefill_tc;
  CUtensorMap tq, tk, tv, to;
  if (!make_map(&tq, q, is_bf16, batch, t_len, hq, qs) || !make_map(&tk, k, is_bf16, batch, t_len, hkv, ks) ||
      !make_map(&tv, v, is_bf16, batch, t_len, hkv, vs) || !make_map(&to, out, is_bf16, batch, t_len, hq, os))
    return CQ_ERR_LAUNCH;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return CQ_ERR_LAUNCH;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(prefill_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(prefill_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
      return CQ_ERR_LAUNCH;
    configured[dev] = true;
  }
  Params p;
  p.t_len = t_len; p.hq = hq; p.hkv = hkv;
  // Two heads of one KV head, same queries, share every K/V tile and have the same number of them, so that neither tile of an
  // item waits for the other at its end.  Needs an even number of heads per KV head; a prompt of one tile gives twice the
  // items (half of the chip would idle) with the heads apart
  p.pair = (hq / hkv) % 2 == 0 && t_len > BM ? 1 : 0;
  p.scale_log2 = 1.4426950408889634f / sqrtf(128.f);
  p.idesc_s = make_idesc(is_bf16, 0, BM, BN);
  p.idesc_pv = make_idesc(is_bf16, 1, BM, BN);
  p.is_bf16 = is_bf16;
  p.status = status;
  const int rows = p.pair ? BM : 2 * BM;
  const unsigned tiles = (unsigned)((t_len + rows - 1) / rows), heads = (unsigned)(p.pair ? hq / 2 : hq);
  p.by_length = (int64_t)batch * t_len * hkv * 2 * 128 * 2 <= (int64_t)64 << 20 && tiles <= 65535u ? 1 : 0;      // half of L2
  const dim3 grid = p.by_length ? dim3(heads, (unsigned)batch, tiles) : dim3(tiles, heads, (unsigned)batch);
  return launched(launch_pdl(is_bf16 ? prefill_tc_kernel<true> : prefill_tc_kernel<false>, grid, dim3(THREADS), SMEM_BYTES, st, tq, tk, tv, to, p));
}

}  // namespace cq
