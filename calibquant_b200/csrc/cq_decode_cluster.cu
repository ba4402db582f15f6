// Decode-step attention on the group format as ONE launch: a thread-block cluster per (batch row, KV head).
//
// What bounded the step before this kernel: separate score, attn.V, full-precision and merge launches meant three
// dependent grids per step (3-4 us each at short contexts, where the arithmetic takes 1-6 us), a side stream with two
// events for the full-precision tokens (4 us of host time), the logits through L2 and back, and two computing warps per
// scheduler, so that the per-tile work around the MMA loops (scale fragments, epilogue, probabilities) was exposed
// latency: 456 cycles per 32-token group and scheduler against ~200 that the MMA, ALU and shared-memory pipes need.
//
// Here every CTA of a cluster owns a contiguous range of the visual span (units of 256 tokens = 8 groups) and a share of
// the full-precision tokens, and keeps its logits in shared memory:
//   1. scores of its units (warp = 16-byte chunks of the 128 channel rows), running minimum / maximum;
//   2. the extremes go to every peer's shared memory (remote stores + a remote mbarrier arrival per peer); while they
//      travel, the CTA works off its full-precision tokens;
//   3. calibration, exponentials, probabilities in place over the logits;
//   4. attn.V of its units, the warps' accumulators summed, one partial (max, sum, acc[128]) per head;
//   5. the partials are scattered over the cluster by output slice (remote stores + arrivals), every CTA merges its slice.
// Key units and then value units pass through one ring of TMA slots that the warps refill themselves as they finish units,
// so the first value units are on their way before the phase changes.
// Two CTAs per SM (16 warps): one CTA's barriers, exchanges and exponentials lie under the other's MMA loops.
// Every wait is bounded; nothing depends on another cluster, so no grid-wide residency is needed.
#include <mutex>
#include <type_traits>

#include "cq_cluster.cuh"
#include "cq_decode_shared.cuh"
#include "cq_decode_tile.cuh"

namespace cq {
namespace mma {

namespace cl {

using namespace cluster;

constexpr int NW = 8, THREADS = NW * 32;        // 16 warps per SM in two CTAs: 128 registers per thread
constexpr int UNIT_TOK = 256, UNIT_G = 8;       // tokens / groups of a unit
constexpr int FPC = 128;                        // full-precision tokens worked off at a time (16 per warp)
constexpr int PF_PITCH = FPC + 8;
constexpr int RED_STRIDE = 136;                 // 128 channels + 4 group biases + the row sum + pad
constexpr int MAX_CLUSTER = 8;
constexpr uint32_t WAIT_TRIES = 1u << 22;

__host__ __device__ constexpr int unit_bytes(int bits) { return 4096 * bits + 4096; }
// slots of the ring: 60-64 KB, so that two CTAs with ~32 KB of logits each fit an SM
__host__ __device__ constexpr int n_slots(int bits) { return bits == 1 ? 8 : bits == 2 ? 5 : 3; }
__host__ __device__ constexpr int ring_bytes(int bits) { return n_slots(bits) * unit_bytes(bits); }
__host__ __device__ constexpr int v_item(int bits) { return bits == 1 ? 128 : 64; }      // tokens a warp takes at a time in the attn.V phase
constexpr int SLOT_WEIGHT = 8;                  // what the items of a unit add up to (see release())

struct Args {
  int batch, hq, hkv, n_rep, t_vis, t_fp, t_sys, calibrate;
  int n_units;                 // ceil(t_vis / 256)
  int pitch;                   // logit row pitch in elements
  int64_t fp_stride_b, fp_stride_h, mask_stride_b;
  const int32_t* t_fp_dev;
  const void* mask;
};

__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
template <typename T>
__device__ __forceinline__ void mma_t(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) mma_bf16(d, a0, a1, a2, a3, b0, b1);
  else mma_f16(d, a0, a1, a2, a3, b0, b1);
}

// Byte transposition of packed codes, in place.  An A fragment takes, per lane (g, c) and k-step of 16 rows, the codes of
// rows 2c, 2c+1, 2c+8, 2c+9 - but of each row's words only the byte (or nibble) of its own matrix row g.  Read straight
// from the rows, every lane fetched four 16-byte pieces per k-step and used an eighth: shared-memory bandwidth, not the MMA
// or the integer pipe, bounded both phases (252 of 355 cycles per 32 tokens and scheduler).  Here lane (kt, c) of the warp
// takes the four rows of one k-step, transposes byte against row (8 permutes per word) and writes 16-byte cells
// [byte j][word p] = (row 2c, row 2c+8, row 2c+1, row 2c+9): afterwards one load per k-step brings all a lane needs, its
// low and third byte are the first operand pair and a shift by 8 gives the second.  Half the shared-memory wavefronts for
// the same number of integer instructions (the permutes replace those that paired the rows).
// Odd k-steps take the rows of a pair in swapped order, which spreads the eight lanes of a load phase over all banks; the
// other operand follows (queries, scales and probabilities of odd k-steps are swapped pairwise as well).
// Rows and cells lie at pitch PITCH with the TMA swizzle of that width; `ch` is the 16-byte column.
template <int PITCH>
__device__ __forceinline__ uint32_t cell(uint32_t base, int d, int ch) {
  const int sw = PITCH == 16 ? 0 : PITCH == 32 ? (d >> 2) & 1 : PITCH == 64 ? (d >> 1) & 3 : d & 7;
  return base + (uint32_t)(d * PITCH + (PITCH == 16 ? 0 : (ch ^ sw) << 4));
}
__device__ __forceinline__ int cell_row(int kt, int j, int c) { return ((kt >> 1) * 4 + j) * 8 + (kt & 1) * 4 + c; }
template <int PITCH>
__device__ __forceinline__ void transpose_bytes(uint32_t base, int ch, int kt, int c) {
  uint32_t w[4][4], x[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint4 v = lds128(cell<PITCH>(base, 16 * kt + ((2 * c + (r & 1)) ^ (kt & 1)) + 8 * (r >> 1), ch));
    w[r][0] = v.x; w[r][1] = v.y; w[r][2] = v.z; w[r][3] = v.w;
  }
  __syncwarp();
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uint32_t t0 = prmt(w[0][p], w[2][p], 0x5140), t1 = prmt(w[0][p], w[2][p], 0x7362);
    const uint32_t u0 = prmt(w[1][p], w[3][p], 0x5140), u1 = prmt(w[1][p], w[3][p], 0x7362);
    x[0][p] = prmt(t0, u0, 0x5410); x[1][p] = prmt(t0, u0, 0x7632);
    x[2][p] = prmt(t1, u1, 0x5410); x[3][p] = prmt(t1, u1, 0x7632);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    sts128(cell<PITCH>(base, cell_row(kt, j, c), ch), make_uint4(x[j][0], x[j][1], x[j][2], x[j][3]));
}

// Lane constants for expanding packed codes (see Expand): the byte permute selector, the two masks per m-tile and the
// powers of two that turn the accumulators of subnormal operands back.  At 1 bit the two m-tiles of a group take their
// bits from the same byte at different offsets; at 2 and 4 bits they take the same field of different words.
template <int BITS>
struct Lane {
  static constexpr int NM = BITS == 1 ? 2 : 1;
  int j;                       // the byte of a word (cell) this lane takes
  uint32_t m0[NM], m1[NM];
  float sc0[NM], sc1[NM];
  __device__ __forceinline__ explicit Lane(int g) {
    constexpr uint32_t FIELD = (1u << BITS) - 1u;
#pragma unroll
    for (int i = 0; i < NM; ++i) {
      const int off = Expand<BITS>::bit_off(i, g) & 31;
      const int sh = off & 7;
      if (i == 0) j = off >> 3;
      m0[i] = (FIELD << sh) * 0x00010001u;
      m1[i] = (FIELD << (sh + BITS)) * 0x00010001u;
      sc0[i] = __uint_as_float((uint32_t)(127 + 24 - sh) << 23);
      sc1[i] = __uint_as_float((uint32_t)(127 + 24 - sh - BITS) << 23);
    }
  }
};

// RAGGED: spans that are a multiple of 32 tokens but not of 256.  The row pitches of the packed keys (t_vis*bits/8 bytes) and
// of their scales and minima (t_vis/16 bytes) are then none a tensor map can describe: a whole warp copies the code words
// of a unit with cp.async (4, 8 or 16 bytes, what the pitch allows; past the last group zeros), the scale and minimum
// fragments come straight from global memory, groups past the end are neither kept nor counted in the extremes.
template <typename T, int BITS, bool SPLIT, bool RAGGED>
__global__ void __launch_bounds__(THREADS, 2)
step_kernel(const __grid_constant__ CUtensorMap tm_code, const __grid_constant__ CUtensorMap tm_ks,
            const __grid_constant__ CUtensorMap tm_kmn, const __grid_constant__ CUtensorMap tm_v, const Args a,
            const T* q, const int32_t* v_code, const T* v_scale, const T* v_mn,   // inputs: written by an overlapping launch, no read-only loads
            const T* k_fp, const T* v_fp, T* __restrict__ out, int* __restrict__ status,
            const int32_t* k_code, const T* k_scale, const T* k_mn) {
  using T2 = typename D16<T>::T2;
  constexpr int NS = n_slots(BITS), UB = unit_bytes(BITS), CODE = 4096 * BITS;
  constexpr int GU = 4 / BITS, CHUNKS = UNIT_G / GU;       // groups per 16-byte chunk of a channel row, chunks of a key unit
  constexpr int ROW = 32 * BITS;                 // bytes of a channel row in a key unit
  constexpr int TOKB = 16 * BITS;                // code bytes of a token in a value unit
  constexpr int VI = v_item(BITS), V_SHARE = UNIT_TOK / VI;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[NS], stat_bar, part_bar;
  __shared__ uint32_t done_s[NS];                // weights of the items done with the load in a slot
  __shared__ int issued_s[NS];                   // loads issued to a slot so far
  __shared__ float mm_s[NW][kMaxRep][2];                            // per warp: minimum / maximum of its logits
  __shared__ float2 peer_mm[MAX_CLUSTER][kMaxRep];                  // the same per CTA of the cluster
  __shared__ __align__(16) uint32_t cal_s[kMaxRep][8];              // calibration constants, -max * log2(e), max
  __shared__ __align__(16) T pf_s[kMaxRep * PF_PITCH];              // full-precision scores, then probabilities
  __shared__ float fp_m[kMaxRep], fp_l[kMaxRep], fp_alpha[kMaxRep];
  __shared__ float recv_o[kMaxRep * kHeadDim + MAX_CLUSTER];        // partials from the peers: [source CTA][slice element]
  __shared__ float2 recv_ml[MAX_CLUSTER][kMaxRep];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int rank = (int)cluster_rank(), S = (int)cluster_size();
  const int pair = blockIdx.x / S, b = pair / a.hkv, hk = pair % a.hkv;
  const int64_t row0 = (int64_t)b * a.hq + (int64_t)hk * a.n_rep;
  const int u0 = rank * a.n_units / S, n_u = (rank + 1) * a.n_units / S - u0;      // this CTA's units

  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(&full_bar[s], RAGGED ? 32 : 1); done_s[s] = 0u; issued_s[s] = 0; }
    mbar_init(&stat_bar, S);
    mbar_init(&part_bar, S);
    mbar_fence_init();
    fence_proxy_async_smem();
  }
  __syncthreads();
  cluster_arrive();          // waited for before the first remote store: every peer's barriers exist then

  // The ring holds the CTA's key units and then its value units, in order: load k goes to slot k % NS.
  // Called by one thread, by a whole warp where RAGGED.
  const int n_groups = a.t_vis / kGroup;
  auto issue = [&](int k) {
    const int s = k % NS;
    unsigned char* base = smem + s * UB;
    // told before the copies: what a waiting warp has to know is that the slot's barrier has entered this load's phase, which
    // the release of the load before (seen by this thread) made sure of.  (A fence behind the copies cost ~800 cycles a load.)
    __threadfence_block();
    *reinterpret_cast<volatile int*>(&issued_s[s]) = k / NS + 1;
    if (RAGGED && k < n_u) {
      const int gr0 = (u0 + k) * UNIT_G;
      const int32_t* src = k_code + ((int64_t)pair * kHeadDim * n_groups + gr0) * BITS;
#pragma unroll 8
      for (int i = lane; i < kHeadDim * UNIT_G; i += 32) {       // (channel row, group): BITS words each
        const int d = i / UNIT_G, gi = i % UNIT_G;
        const bool live = gr0 + gi < n_groups;
        const uint32_t dst = cell<ROW>(smem_u32(base), d, gi * BITS / 4) + (uint32_t)(gi * BITS * 4) % 16u;
        cp_async_zfill<4 * BITS>(dst, src + ((int64_t)d * n_groups + (live ? gi : 0)) * BITS, live ? 4 * BITS : 0);
      }
      cp_async_mbar_arrive_noinc(&full_bar[s]);
    } else if (RAGGED && lane > 0) {
      mbar_arrive(&full_bar[s]);
    } else if (k < n_u) {
      const int u = u0 + k;
      mbar_expect_tx(&full_bar[s], UB);
      tma_load_2d(base, &tm_code, u * UNIT_G * BITS, pair * kHeadDim, &full_bar[s]);
      tma_load_2d(base + CODE, &tm_ks, u * UNIT_G, pair * kHeadDim, &full_bar[s]);
      tma_load_2d(base + CODE + 2048, &tm_kmn, u * UNIT_G, pair * kHeadDim, &full_bar[s]);
    } else {
      const int u = u0 + k - n_u, nt = min(UNIT_TOK, a.t_vis - u * UNIT_TOK);
      const int64_t tok = (int64_t)pair * a.t_vis + (int64_t)u * UNIT_TOK;
      // a tiled load always delivers the whole box of 256 rows (rows past the last token are never read)
      mbar_expect_tx(&full_bar[s], (uint32_t)((BITS == 1 ? nt : UNIT_TOK) * TOKB + nt * 16));
      if (BITS == 1) bulk_load_1d(base, v_code + tok * 4, (uint32_t)(nt * TOKB), &full_bar[s]);
      else tma_load_2d(base, &tm_v, 0, (int)tok, &full_bar[s]);
      bulk_load_1d(base + CODE, v_scale + tok * 4, (uint32_t)(nt * 8), &full_bar[s]);
      bulk_load_1d(base + CODE + 2048, v_mn + tok * 4, (uint32_t)(nt * 8), &full_bar[s]);
    }
  };
  // A warp is done with its share of load k; whoever completes the unit refills the slot.  There is no producer warp: a
  // ninth warp per CTA would cost every warp a quarter of its registers.
  auto release = [&](int k, uint32_t weight) {
    __syncwarp();
    bool last = false;
    if (lane == 0) {
      const int s = k % NS;
      __threadfence_block();
      last = atomicAdd(&done_s[s], weight) + weight == SLOT_WEIGHT;
      if (last) done_s[s] = 0u;
    }
    if (RAGGED) last = __shfl_sync(0xffffffffu, (int)last, 0) != 0;
    if (last && k + NS < 2 * n_u) {
      __threadfence_block();
      fence_proxy_async_smem();          // the warps wrote into the slot (in-place transposition)
      issue(k + NS);
    }
  };
  // Warps skip units that hold none of their items, so a warp can come to a slot before the load ahead of its own has
  // landed there, when the parity of its own phase still reads as completed: it waits first until its load has been issued
  // (which follows the release of the load before), then for the data.
  bool failed = false;
  auto wait_full = [&](int k) {
    const int s = k % NS, turn = k / NS + 1;
    uint32_t tries = 0;
#pragma unroll 1
    while (*reinterpret_cast<volatile int*>(&issued_s[s]) != turn && ++tries < WAIT_TRIES) __nanosleep(32);
    __threadfence_block();
    const bool ok = tries < WAIT_TRIES && mbar_wait_bounded(&full_bar[s], (uint32_t)((k / NS) & 1), WAIT_TRIES);
    failed = !__all_sync(0xffffffffu, ok);
    if (failed && lane == 0) atomicExch(status, CQ_ERR_TIMEOUT);
    return !failed;
  };
  // The query, the newest full-precision token and freshly packed operands come from the launches before this one: nothing is
  // read before they have completed.  Steps that follow each other directly lose the overlap of the first loads with the tail
  // of the step before (timed before the wider pieces below: 1 x 8 x 256 tokens 11.1 us with the packed operands read ahead of the
  // wait, 11.4 so; 4 x 8 x 5152 23.2, 24.0; 64 x 8 x 6656 164.5, 169.0; with them 10.9, 24.4 and 160.6).  (Requested into L2 ahead of
  // the wait 16 x 8 x 3328 took 33.0: a bulk prefetch costs its thread as much as the load.)
  pdl_wait();
  const int t_live = a.t_fp_dev ? *reinterpret_cast<const volatile int32_t*>(a.t_fp_dev) : a.t_fp;      // on its way beside the loads below
  // the first loads of the slots, one by each warp (one after the other they took one thread 7000
  // cycles; 4 x 8 x 5152 masked tokens 24.0 -> 23.2 us, no difference where the ring's first units suffice for a while)
  static_assert(NS <= NW, "a warp per slot");
  if (warp < min(NS, n_u) && (RAGGED || lane == 0)) issue(warp);
  __syncwarp();
  // this CTA's share of the full-precision tokens (16-token tiles dealt out over the cluster), on its way into L2
  auto fp_range = [&](int& f0, int& f1) {
    const int t_fp = min(t_live, a.t_fp), n_t16 = (t_fp + 15) / 16;
    f0 = rank * n_t16 / S * 16;
    f1 = min(t_fp, (rank + 1) * n_t16 / S * 16);
  };
  {
    int f0, f1;
    fp_range(f0, f1);
    const int64_t off = (int64_t)b * a.fp_stride_b + (int64_t)hk * a.fp_stride_h;
    for (int i = tid; i < (f1 - f0) * 4; i += THREADS) {
      const T* p = ((i & 1) ? v_fp : k_fp) + off + (int64_t)(f0 + (i >> 2)) * kHeadDim + ((i >> 1) & 1) * 64;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
  }

  const uint32_t ring = smem_u32(smem), lg = ring + ring_bytes(BITS);      // logits [n_rep][pitch] behind the ring
  const Lane<BITS> L(g);
  // value units of the first ring behind the key units, whose data is needed first: 16 x 8 x 3328 tokens 30.7 -> 28.7 us
  if (warp >= n_u && warp < min(NS, 2 * n_u) && (RAGGED || lane == 0)) issue(warp);
  __syncwarp();

  // ================= 1. scores =================
  {
    // B operand: q * ks.  SPLIT (at most four query heads): column 2h carries the product rounded to fp16, column
    // 2h+1 the exact remainder; otherwise the eight columns are heads.
    const int q_head = SPLIT ? (g >> 1) : g;
    const bool lo_lane = SPLIT && (g & 1);
    const int out_head = SPLIT ? c : 2 * c;      // first head of this lane's accumulator columns
    uint32_t qA[8], qB[8];
    {
      const T* qrow = q + (row0 + q_head) * kHeadDim + 2 * c;
#pragma unroll
      for (int kt = 0; kt < 8; ++kt) {
        qA[kt] = q_head < a.n_rep ? D16<T>::to_h2(*reinterpret_cast<const uint32_t*>(qrow + kt * 16)) : 0u;
        qB[kt] = q_head < a.n_rep ? D16<T>::to_h2(*reinterpret_cast<const uint32_t*>(qrow + kt * 16 + 8)) : 0u;
        if (kt & 1) { qA[kt] = prmt(qA[kt], qA[kt], 0x1032); qB[kt] = prmt(qB[kt], qB[kt], 0x1032); }
      }
    }
    // warps per unit: whole units per warp save scale fragments (fetched for eight groups at once), shares of a unit
    // fill the warps when there are few units; cost in tenths of a group
    int share = 1, best = 0x7fffffff;
#pragma unroll
    for (int s = 1; s <= (CHUNKS < 4 ? CHUNKS : 4); s *= 2) {
      const int cost = (n_u * s + NW - 1) / NW * (80 / s + 20);
      if (cost < best && s * NS >= NW) { best = cost; share = s; }      // the ring has to hold an item for every warp
    }
    T2 mnA = D16<T>::bcast(D16<T>::big()), mxA = D16<T>::bcast(-D16<T>::big()), mnB = mnA, mxB = mxA;
    for (int it = warp; it < n_u * share; it += NW) {
      const int u = it / share, sub = it % share;
      if (!wait_full(u)) break;
      const uint32_t base = ring + (uint32_t)(u % NS * UB);
      uint32_t ksA[8], ksB[8];                   // scales of group g of the unit, channels of k-tile kt in fragment order
      float cb[4] = {0.f, 0.f, 0.f, 0.f};        // bias[group g][columns 2c, 2c+1]
      {
        const int mat = lane >> 3, r = (lane & 7) ^ (mat >> 1), G = (u0 + u) * UNIT_G + g;
        const bool live = !RAGGED || G < n_groups;
        const T* ksr = k_scale + (int64_t)pair * kHeadDim * n_groups + (live ? G : 0);
        const T* mnr = k_mn + (int64_t)pair * kHeadDim * n_groups + (live ? G : 0);
        const uint32_t srow = base + CODE + (uint32_t)((16 * (mat >> 1) + 8 * (mat & 1) + r) * 16);
#pragma unroll
        for (int kp = 0; kp < 4; ++kp) {         // 32 channels: k-tiles 2kp and 2kp+1
          uint32_t s0, s1, s2, s3, z0, z1, z2, z3;
          if (RAGGED) {
            auto pairs = [&](const T* rows, uint32_t& f0, uint32_t& f1, uint32_t& f2, uint32_t& f3) {
              uint32_t* f[4] = {&f0, &f1, &f2, &f3};
#pragma unroll
              for (int m = 0; m < 4; ++m) {      // channels 32kp + 8m + 2c, + 1; swapped in odd k-tiles
                const int64_t d = 32 * kp + 8 * m + 2 * c, e = m >> 1;
                const T2 v = D16<T>::pair2(rows[(d + e) * n_groups], rows[(d + 1 - e) * n_groups]);
                *f[m] = live ? *reinterpret_cast<const uint32_t*>(&v) : 0u;
              }
            };
            pairs(ksr, s0, s1, s2, s3);
            pairs(mnr, z0, z1, z2, z3);
          } else {
            ldmatrix_x4_trans(srow + kp * 512, s0, s1, s2, s3);
            ldmatrix_x4_trans(srow + 2048 + kp * 512, z0, z1, z2, z3);
          }
          ksA[2 * kp] = D16<T>::to_h2(s0); ksB[2 * kp] = D16<T>::to_h2(s1);
          ksA[2 * kp + 1] = D16<T>::to_h2(s2); ksB[2 * kp + 1] = D16<T>::to_h2(s3);
          mma_f16(cb, D16<T>::to_h2(z0), 0u, D16<T>::to_h2(z1), 0u, qA[2 * kp], qB[2 * kp]);
          mma_f16(cb, D16<T>::to_h2(z2), 0u, D16<T>::to_h2(z3), 0u, qA[2 * kp + 1], qB[2 * kp + 1]);
        }
      }
#pragma unroll 1
      for (int ch = sub * CHUNKS / share; ch < (sub + 1) * CHUNKS / share; ++ch) {
        transpose_bytes<ROW>(base, ch, lane >> 2, c);
        __syncwarp();
        // Below 4 bits the first products have a zero addend in place of cleared accumulators: 64 x 8 x 6656 at 2 bits 158.1 ->
        // 156.2 us, 16 x 8 x 3328 at 1 bit 24.4 -> 23.9 (at 4 bits 9.8 -> 10.0 for 5 x 8 x 256, nothing elsewhere).
        float acc[GU][2][4];
        if (BITS == 4)
#pragma unroll
          for (int i = 0; i < GU * 8; ++i) (&acc[0][0][0])[i] = 0.f;
        auto mma = [](float (&d)[4], bool first, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
          if (BITS < 4 && first) mma_f16_zero(d, a0, a1, a2, a3, b0, b1);
          else mma_f16(d, a0, a1, a2, a3, b0, b1);
        };
#pragma unroll
        for (int kt = 0; kt < 8; ++kt) {
          const uint32_t ca = cell<ROW>(base, cell_row(kt, L.j, c), ch);
          uint32_t W[4];
          if (BITS == 4) {                       // the lane's word pair of the group's four
            const uint2 v = lds64(ca + (uint32_t)(g >> 2) * 8u);
            W[0] = v.x; W[1] = v.y; W[2] = W[3] = 0u;
          } else {
            const uint4 v = lds128(ca);
            W[0] = v.x; W[1] = v.y; W[2] = v.z; W[3] = v.w;
          }
#pragma unroll
          for (int x = 0; x < GU; ++x) {
            const int src = 4 * (ch * GU + x) + c;
            const uint32_t ksa = __shfl_sync(0xffffffffu, ksA[kt], src), ksb = __shfl_sync(0xffffffffu, ksB[kt], src);
            uint32_t b0 = hmul2_u32(qA[kt], ksa), b1 = hmul2_u32(qB[kt], ksb);
            if (lo_lane) {                       // q*ks - rnd(q*ks), formed exactly by the FMA
              b0 = hfma2_neg_u32(qA[kt], ksa, b0);
              b1 = hfma2_neg_u32(qB[kt], ksb, b1);
            }
            if (BITS == 1) {
              const uint32_t lo = W[x], hi = W[x] >> 8;
              mma(acc[x][0], kt == 0, lo & L.m0[0], lo & L.m1[0], hi & L.m0[0], hi & L.m1[0], b0, b1);
              mma(acc[x][1], kt == 0, lo & L.m0[L.NM - 1], lo & L.m1[L.NM - 1], hi & L.m0[L.NM - 1], hi & L.m1[L.NM - 1], b0, b1);
            } else {
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const uint32_t lo = W[(BITS == 4 ? 0 : 2 * x) + i], hi = lo >> 8;
                mma(acc[x][i], kt == 0, lo & L.m0[0], lo & L.m1[0], hi & L.m0[0], hi & L.m1[0], b0, b1);
              }
            }
          }
        }
        // ---- epilogue: bias, the reference's roundings, 1/sqrt(D), logits to shared memory
#pragma unroll
        for (int x = 0; x < GU; ++x) {
          const int gi = ch * GU + x;            // group of the unit
          if (RAGGED && (u0 + u) * UNIT_G + gi >= n_groups) continue;
          const float bias0 = __shfl_sync(0xffffffffu, cb[0], 4 * gi + c);
          const float bias1 = SPLIT ? 0.f : __shfl_sync(0xffffffffu, cb[1], 4 * gi + c);
          const uint32_t la = lg + (uint32_t)((out_head * a.pitch + u * UNIT_TOK + gi * 32) * 2), lb = la + (uint32_t)(a.pitch * 2);
          T2 sa[2], sb[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int m = BITS == 1 ? i : 0;
            if (SPLIT) {
              sa[i] = D16<T>::inv_sqrt_d(D16<T>::round2(fmaf(acc[x][i][0] + acc[x][i][1], L.sc0[m], bias0),
                                                        fmaf(acc[x][i][2] + acc[x][i][3], L.sc1[m], bias0)));
            } else {
              sa[i] = D16<T>::inv_sqrt_d(D16<T>::round2(fmaf(acc[x][i][0], L.sc0[m], bias0), fmaf(acc[x][i][2], L.sc1[m], bias0)));
              sb[i] = D16<T>::inv_sqrt_d(D16<T>::round2(fmaf(acc[x][i][1], L.sc0[m], bias1), fmaf(acc[x][i][3], L.sc1[m], bias1)));
            }
          }
          auto put = [&](uint32_t row, const T2 (&v)[2]) {      // a lane's four tokens; at 1 bit they are adjacent
            if (BITS == 1) {
              sts64(row + 8 * g, *reinterpret_cast<const uint32_t*>(&v[0]), *reinterpret_cast<const uint32_t*>(&v[1]));
            } else {
#pragma unroll
              for (int i = 0; i < 2; ++i)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(row + 2 * Expand<BITS>::elem(i, g)),
                             "r"(*reinterpret_cast<const uint32_t*>(&v[i])) : "memory");
            }
          };
          if (out_head < a.n_rep) {
            put(la, sa);
            mnA = __hmin2(mnA, __hmin2(sa[0], sa[1])); mxA = __hmax2(mxA, __hmax2(sa[0], sa[1]));
          }
          if (!SPLIT && out_head + 1 < a.n_rep) {
            put(lb, sb);
            mnB = __hmin2(mnB, __hmin2(sb[0], sb[1])); mxB = __hmax2(mxB, __hmax2(sb[0], sb[1]));
          }
        }
      }
      release(u, SLOT_WEIGHT / share);
    }
    // extremes of this warp per head
    const float2 n0 = D16<T>::to_f2(mnA), x0 = D16<T>::to_f2(mxA), n1 = D16<T>::to_f2(mnB), x1 = D16<T>::to_f2(mxB);
    float lo_a = fminf(n0.x, n0.y), hi_a = fmaxf(x0.x, x0.y), lo_b = fminf(n1.x, n1.y), hi_b = fmaxf(x1.x, x1.y);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      lo_a = fminf(lo_a, __shfl_xor_sync(0xffffffffu, lo_a, o));
      hi_a = fmaxf(hi_a, __shfl_xor_sync(0xffffffffu, hi_a, o));
      if (!SPLIT) {
        lo_b = fminf(lo_b, __shfl_xor_sync(0xffffffffu, lo_b, o));
        hi_b = fmaxf(hi_b, __shfl_xor_sync(0xffffffffu, hi_b, o));
      }
    }
    if (g == 0) {
      mm_s[warp][out_head][0] = lo_a; mm_s[warp][out_head][1] = hi_a;
      if (!SPLIT) { mm_s[warp][out_head + 1][0] = lo_b; mm_s[warp][out_head + 1][1] = hi_b; }
    }
  }
  __syncthreads();

  // ================= 2. extremes to the peers =================
  cluster_wait();
  if (tid < S * a.n_rep) {
    const int peer = tid / a.n_rep, h = tid % a.n_rep;
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; ++w) { lo = fminf(lo, mm_s[w][h][0]); hi = fmaxf(hi, mm_s[w][h][1]); }
    st_peer2(map_peer(smem_u32(&peer_mm[rank][h]), peer), lo, hi);
  }
  __syncthreads();
  if (tid < S) arrive_peer(map_peer(smem_u32(&stat_bar), tid));

  // ---- full-precision tokens of this CTA, 128 at a time: scores as 16-token MMA tiles, running maximum per head, probabilities
  // rounded to the data type, P.V with warp w owning channels 32 (w / 2) .. + 31 of every other 64 tokens.  Keys and values come
  // straight from global memory in pieces of 16 and 8 bytes: a lane's piece holds neighbouring channels, which the products take in
  // the order they come.  (In the fragments' own 4-byte pieces the 80 loads of a thread, eight rows each, took 6900 cycles a chunk.)
  // At 4 bits values come in 4-byte pieces, channels 16 w .. + 15 of all tokens: half the sums to keep through attn.V, where that
  // width has no registers left (with other kernels between the steps 2 x 8 x 5120 tokens 19.35 us with 8-byte pieces, 18.9 so;
  // 4 x 8 x 5120 masked 20.2, 19.7).  Ragged spans keep the wide ones (4 x 8 x 5152 masked, one step after the other, 24.3 against 24.7).
  constexpr int VW = BITS == 4 && !RAGGED ? 1 : 2;
  float fo[2 * VW][4] = {};
  if (tid < kMaxRep) { fp_m[tid] = -INFINITY; fp_l[tid] = 0.f; }
  {
    int f0, f1;
    fp_range(f0, f1);
    const T* kf = k_fp + (int64_t)b * a.fp_stride_b + (int64_t)hk * a.fp_stride_h;
    const T* vf = v_fp + (int64_t)b * a.fp_stride_b + (int64_t)hk * a.fp_stride_h + (VW == 2 ? 32 * (warp >> 1) + 4 * g : 16 * warp + 2 * g);
    const T* mrow = a.mask ? static_cast<const T*>(a.mask) + (int64_t)b * a.mask_stride_b : nullptr;
    for (int t0 = f0; t0 < f1; t0 += FPC) {
      const int nt = min(FPC, f1 - t0);
      if (16 * warp < nt) {
        const int tt = 16 * warp;
        const T* qrow = q + (row0 + (g < a.n_rep ? g : 0)) * kHeadDim + 8 * c;
        const T* k_lo = kf + (int64_t)(t0 + min(tt + g, nt - 1)) * kHeadDim + 8 * c;       // rows past the end repeat
        const T* k_hi = kf + (int64_t)(t0 + min(tt + g + 8, nt - 1)) * kHeadDim + 8 * c;   // the last token
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        uint4 lo[4], hi[4], qv[4];      // channels 32m + 8c .. + 7: four pairs, two k-steps
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          lo[m] = *reinterpret_cast<const uint4*>(k_lo + 32 * m);
          hi[m] = *reinterpret_cast<const uint4*>(k_hi + 32 * m);
          qv[m] = *reinterpret_cast<const uint4*>(qrow + 32 * m);      // columns past the last head repeat the first; they are not kept
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          mma_t<T>(acc, lo[m].x, hi[m].x, lo[m].y, hi[m].y, qv[m].x, qv[m].y);
          mma_t<T>(acc, lo[m].z, hi[m].z, lo[m].w, hi[m].w, qv[m].z, qv[m].w);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {       // acc[0..1] = (token tt+g, heads 2c, 2c+1), acc[2..3] = (token tt+g+8, same)
          const int h = 2 * c + (e & 1), t = tt + g + 8 * (e >> 1);
          if (h < a.n_rep && t < nt) pf_s[h * PF_PITCH + t] = Elem<T>::from_f(__fdiv_rn(rnd<T>(acc[e]), 11.313708498984761f));
        }
      }
      using Piece = typename std::conditional<VW == 2, uint2, uint32_t>::type;
      constexpr int NK = FPC / (16 * VW);
      const int th = VW == 2 ? 64 * (warp & 1) : 0;
      Piece v[NK][4];                       // tokens th + 16k + 2c + {0, 1, 8, 9}, 2 VW channels; on their way during the softmax
#pragma unroll
      for (int k = 0; k < NK; ++k)
#pragma unroll
        for (int r = 0; r < 4; ++r)         // past the end p is 0 and the value repeats the last token
          v[k][r] = th + 16 * k < nt ? *reinterpret_cast<const Piece*>(vf + (int64_t)(t0 + min(th + 16 * k + 2 * c + (r & 1) + 8 * (r >> 1), nt - 1)) * kHeadDim)
                                     : Piece{};
      __syncthreads();
      if (warp < a.n_rep) {                 // warp = head
        const int h = warp;
        float xv[4], m = fp_m[h];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = j * 32 + lane;
          xv[j] = t < nt ? Elem<T>::to_f(pf_s[h * PF_PITCH + t]) : -INFINITY;
          if (mrow && t < nt) {             // token f sits before (system) or after (text) the visual span
            const int f = t0 + t;
            xv[j] = rnd<T>(xv[j] + Elem<T>::to_f(mrow[f < a.t_sys ? f : a.t_vis + f]));
          }
          m = fmaxf(m, xv[j]);
        }
        m = warp_max(m);
        const float ref = m == -INFINITY ? 0.f : m;
        const float alpha = exp2f((fp_m[h] - ref) * LOG2E);              // 0 for the first chunk
        float l = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = j * 32 + lane;
          const float p = t < nt ? rnd<T>(exp2f((xv[j] - ref) * LOG2E)) : 0.f;
          pf_s[h * PF_PITCH + t] = Elem<T>::from_f(p);
          l += p;
        }
        l = warp_sum(l);
        __syncwarp();
        if (lane == 0) { fp_l[h] = fp_l[h] * alpha + l; fp_m[h] = m; fp_alpha[h] = alpha; }
      }
      __syncthreads();
      {
        const float alpha = g < a.n_rep ? fp_alpha[g] : 0.f;
#pragma unroll
        for (int j = 0; j < 2 * VW; ++j) { fo[j][0] *= alpha; fo[j][1] *= alpha; }
        const T* prow = pf_s + (g < a.n_rep ? g : 0) * PF_PITCH + th + 2 * c;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          if (th + 16 * k >= nt) break;
          const uint32_t p0 = *reinterpret_cast<const uint32_t*>(prow + 16 * k), p1 = *reinterpret_cast<const uint32_t*>(prow + 16 * k + 8);
          // n-tile j: column n stands for channel 32 (w / 2) + 4n + j (4 bits: 16w + 2n + j)
#pragma unroll
          for (int i = 0; i < VW; ++i) {
            auto word = [&](int r) { return reinterpret_cast<const uint32_t*>(&v[k][r])[i]; };
            mma_t<T>(fo[2 * i], p0, 0u, p1, 0u, prmt(word(0), word(1), 0x5410), prmt(word(2), word(3), 0x5410));
            mma_t<T>(fo[2 * i + 1], p0, 0u, p1, 0u, prmt(word(0), word(1), 0x7632), prmt(word(2), word(3), 0x7632));
          }
        }
      }
      __syncthreads();       // the probabilities have been used
    }
  }

  // ================= 3. probabilities =================
  if (!wait_peers(&stat_bar, WAIT_TRIES)) {
    if (tid == 0) atomicExch(status, CQ_ERR_TIMEOUT);
    failed = true;
  }
  if (tid < a.n_rep) {
    float lo = INFINITY, hi = -INFINITY;
    for (int p = 0; p < S; ++p) { lo = fminf(lo, peer_mm[p][tid].x); hi = fmaxf(hi, peer_mm[p][tid].y); }
    CalibH<T> cal;
    cal.mn = cal.range = cal.rdenom = cal.rdenom_lo = D16<T>::bcast(0.f);
    float m = hi;
    if (a.calibrate) {
      set_calib<T>(cal, lo, hi);
      m = D16<T>::to_f2(calibrate2<T>(D16<T>::bcast(hi), cal)).x;        // the maximum, calibrated like any logit
    }
    uint32_t* e = cal_s[tid];
    e[0] = *reinterpret_cast<const uint32_t*>(&cal.mn); e[1] = *reinterpret_cast<const uint32_t*>(&cal.range);
    e[2] = *reinterpret_cast<const uint32_t*>(&cal.rdenom); e[3] = *reinterpret_cast<const uint32_t*>(&cal.rdenom_lo);
    e[4] = __float_as_uint(-m * LOG2E);
    e[5] = __float_as_uint(m);
  }
  __syncthreads();
  {
    // 8 tokens of one head per thread and step (a unit is 32 such vectors: the head is uniform over a warp); the
    // reference rounds probabilities to the data type, they are then exact in fp16, the type the MMA takes
    const int n_vec = n_u * (UNIT_TOK / 8);
    const T* mvis = a.mask ? static_cast<const T*>(a.mask) + (int64_t)b * a.mask_stride_b + a.t_sys : nullptr;
    for (int h = 0; h < a.n_rep; ++h) {
      const uint4 cw = *reinterpret_cast<const uint4*>(cal_s[h]);
      const float mneg = __uint_as_float(cal_s[h][4]);
      CalibH<T> ch;
      ch.mn = *reinterpret_cast<const T2*>(&cw.x); ch.range = *reinterpret_cast<const T2*>(&cw.y);
      ch.rdenom = *reinterpret_cast<const T2*>(&cw.z); ch.rdenom_lo = *reinterpret_cast<const T2*>(&cw.w);
      // start at another warp for every head, so that short spans use all of them
      for (int v = (tid + 256 - (h * n_vec & 255)) & 255; v < n_vec; v += NW * 32) {
        const uint32_t addr = lg + (uint32_t)((h * a.pitch + 8 * v) * 2);
        const uint4 x = lds128(addr);
        const uint32_t xi[4] = {x.x, x.y, x.z, x.w};
        uint32_t po[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          T2 y = *reinterpret_cast<const T2*>(&xi[j]);
          if (a.calibrate) y = calibrate2<T>(y, ch);
          if (mvis) {
            const int t = u0 * UNIT_TOK + 8 * v + 2 * j;
            if (t < a.t_vis) y = __hadd2(y, D16<T>::pair2(mvis[t], mvis[t + 1]));
          }
          const float2 f = D16<T>::to_f2(y);
          po[j] = D16<T>::prob_pair(ex2_approx(fmaf(f.x, LOG2E, mneg)), ex2_approx(fmaf(f.y, LOG2E, mneg)));
        }
        sts128(addr, make_uint4(po[0], po[1], po[2], po[3]));
      }
    }
  }
  __syncthreads();

  // ================= 4. attn.V =================
  // A rows = channels (codes, transposed in place as in the score phase), B = p * vs with columns = heads; the minima and
  // the row sum of p ride on one more MMA per 16 tokens (rows = heads; columns 0-3: the four channel groups, 4: ones).
  float acc[8][4], vb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 32; ++i) (&acc[0][0])[i] = 0.f;
  {
    const uint32_t zoff = (uint32_t)(g < 4 ? g : 0) * 4u;
    const uint32_t z_and = g < 4 ? 0xffffffffu : 0u, z_or = g == 4 ? 0x3c003c00u : 0u;
    const uint32_t lgh = lg + (uint32_t)((g < a.n_rep ? g : 0) * a.pitch * 2);      // columns past the last head are not kept
    const uint32_t odd = (lane >> 3) & 1;      // pairs of odd k-steps are swapped (see transpose_bytes)
    const uint32_t sel_lo = odd ? 0x1054u : 0x5410u, sel_hi = odd ? 0x3276u : 0x7632u;
    for (int it = warp; it < n_u * V_SHARE && !failed; it += NW) {
      const int u = it / V_SHARE, tq = it % V_SHARE * VI, k = n_u + u;
      if (!wait_full(k)) break;
      const int nt = min(VI, a.t_vis - (u0 + u) * UNIT_TOK - tq);      // live tokens of the item: a multiple of 32, may be <= 0
      if (nt > 0) {
        const uint32_t base = ring + (uint32_t)(k % NS * UB), code_b = base + (uint32_t)tq * TOKB;
        const uint32_t vs_b = base + CODE + (uint32_t)tq * 8u, vm_b = vs_b + 2048u;
        if (BITS == 1) transpose_bytes<16>(code_b, 0, lane >> 2, c);
        if (BITS == 2) transpose_bytes<32>(code_b, lane >> 4, (lane >> 2) & 3, c);
        if (BITS == 4) { transpose_bytes<64>(code_b, lane >> 4, (lane >> 2) & 3, c); transpose_bytes<64>(code_b, 2 + (lane >> 4), (lane >> 2) & 3, c); }
        // scales and minima re-laid out in place: a 16-byte unit holds two tokens x four channel groups and becomes four
        // token pairs, the B-fragment order; bf16 becomes fp16
#pragma unroll
        for (int arr = 0; arr < 2; ++arr)
#pragma unroll
          for (int i = 0; i < VI / 64; ++i) {
            const uint32_t addr = (arr == 0 ? vs_b : vm_b) + (uint32_t)(i * 32 + lane) * 16u;
            uint4 v = lds128(addr);
            v.x = D16<T>::to_h2(v.x); v.y = D16<T>::to_h2(v.y); v.z = D16<T>::to_h2(v.z); v.w = D16<T>::to_h2(v.w);
            sts128(addr, make_uint4(prmt(v.x, v.z, sel_lo), prmt(v.x, v.z, sel_hi), prmt(v.y, v.w, sel_lo), prmt(v.y, v.w, sel_hi)));
          }
        __syncwarp();
#pragma unroll
        for (int kq = 0; kq < VI / 16; ++kq) {
          if ((BITS == 4 || kq % 2 == 0) && kq * 16 >= nt) break;      // live tokens come in groups of 32 (at 4 bits 24.2 -> 24.4 us, 4 x 8 x 5152)
          const int t0 = kq * 16 + 2 * c;                              // first token of the lane's first pair, in the item
          uint32_t pp0 = lds32(lgh + (uint32_t)(u * UNIT_TOK + tq + t0) * 2u), pp1 = lds32(lgh + (uint32_t)(u * UNIT_TOK + tq + t0 + 8) * 2u);
          if (kq & 1) { pp0 = prmt(pp0, pp0, 0x1032); pp1 = prmt(pp1, pp1, 0x1032); }
          const uint4 s0 = lds128(vs_b + (uint32_t)t0 * 8u), s1 = lds128(vs_b + (uint32_t)(t0 + 8) * 8u);
          const uint32_t z0 = lds32(vm_b + (uint32_t)t0 * 8u + zoff), z1 = lds32(vm_b + (uint32_t)(t0 + 8) * 8u + zoff);
          const uint32_t bA[4] = {hmul2_u32(pp0, s0.x), hmul2_u32(pp0, s0.y), hmul2_u32(pp0, s0.z), hmul2_u32(pp0, s0.w)};
          const uint32_t bB[4] = {hmul2_u32(pp1, s1.x), hmul2_u32(pp1, s1.y), hmul2_u32(pp1, s1.z), hmul2_u32(pp1, s1.w)};
          mma_f16(vb, pp0, 0u, pp1, 0u, (z0 & z_and) | z_or, (z1 & z_and) | z_or);
          const int row = cell_row(kq, L.j, c);
          if (BITS == 1) {          // word m = channels 32m .. 32m+31 = m-tiles 2m, 2m+1
            const uint4 w = lds128(cell<16>(code_b, row, 0));
            const uint32_t W[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const uint32_t lo = W[m], hi = W[m] >> 8;
              mma_f16(acc[2 * m], lo & L.m0[0], lo & L.m1[0], hi & L.m0[0], hi & L.m1[0], bA[m], bB[m]);
              mma_f16(acc[2 * m + 1], lo & L.m0[L.NM - 1], lo & L.m1[L.NM - 1], hi & L.m0[L.NM - 1], hi & L.m1[L.NM - 1], bA[m], bB[m]);
            }
          } else {                  // m-tile j: 2 bits: word j of the row; 4 bits: word j % 2 of the lane's pair in channel group j / 2
#pragma unroll
            for (int q4 = 0; q4 < BITS; ++q4) {
              uint32_t W[4];
              if (BITS == 2) {
                const uint4 w = lds128(cell<32>(code_b, row, q4));
                W[0] = w.x; W[1] = w.y; W[2] = w.z; W[3] = w.w;
              } else {
                const uint2 w = lds64(cell<64>(code_b, row, q4) + (uint32_t)(g >> 2) * 8u);
                W[0] = w.x; W[1] = w.y; W[2] = W[3] = 0u;
              }
              constexpr int NJ = 8 / BITS;
#pragma unroll
              for (int j = 0; j < NJ; ++j) {
                const int jj = q4 * NJ + j;
                const uint32_t lo = W[j], hi = W[j] >> 8;
                mma_f16(acc[jj], lo & L.m0[0], lo & L.m1[0], hi & L.m0[0], hi & L.m1[0], bA[jj >> 1], bB[jj >> 1]);
              }
            }
          }
        }
      }
      release(k, SLOT_WEIGHT / V_SHARE);
    }
  }
  __syncthreads();            // the ring is idle: it holds the warps' sums from here on
  float* fp_o = reinterpret_cast<float*>(smem) + NW * kMaxRep * RED_STRIDE;      // [token half (one at 4 bits)][head][channel]
  {
    float* mine = reinterpret_cast<float*>(smem) + warp * kMaxRep * RED_STRIDE;
    if (g < a.n_rep) {                       // fragment columns 2c, 2c+1 of n-tile j = channels 32 (w / 2) + 8c + j, + 4 (4 bits: 16w + 4c + j, + 2)
      if constexpr (VW == 2) {
        float4* dst = reinterpret_cast<float4*>(fp_o + ((warp & 1) * kMaxRep + g) * kHeadDim + 32 * (warp >> 1) + 8 * c);
        dst[0] = make_float4(fo[0][0], fo[1][0], fo[2][0], fo[3][0]);
        dst[1] = make_float4(fo[0][1], fo[1][1], fo[2][1], fo[3][1]);
      } else {
        *reinterpret_cast<float4*>(fp_o + g * kHeadDim + 16 * warp + 4 * c) = make_float4(fo[0][0], fo[1][0], fo[0][1], fo[1][1]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = BITS == 1 ? (j & 1) : 0;
      const int chn = 32 * (j >> 1) + Expand<BITS>::elem(j & 1, g);
      if (2 * c < a.n_rep) {
        mine[(2 * c) * RED_STRIDE + chn] = acc[j][0] * L.sc0[i];
        mine[(2 * c) * RED_STRIDE + chn + 1] = acc[j][2] * L.sc1[i];
      }
      if (2 * c + 1 < a.n_rep) {
        mine[(2 * c + 1) * RED_STRIDE + chn] = acc[j][1] * L.sc0[i];
        mine[(2 * c + 1) * RED_STRIDE + chn + 1] = acc[j][3] * L.sc1[i];
      }
    }
    if (g < a.n_rep && c < 3) {              // bias columns 0..3 (c = 0, 1) and the row sum (column 4)
      mine[g * RED_STRIDE + 128 + 2 * c] = vb[0];
      if (c < 2) mine[g * RED_STRIDE + 128 + 2 * c + 1] = vb[1];
    }
  }
  __syncthreads();

  // ================= 5. merge over the cluster =================
  const int n_out = a.n_rep * kHeadDim, slice = (n_out + S - 1) / S;

  for (int e = tid; e < n_out; e += NW * 32) {
    const int h = e >> 7, d = e & 127;
    float o = 0.f, l = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float* r = reinterpret_cast<const float*>(smem) + (w * kMaxRep + h) * RED_STRIDE;
      o += r[d] + r[128 + (d >> 5)];
      l += r[132];
    }
    // this CTA's visual and full-precision parts under one reference
    const float m_v = n_u > 0 ? __uint_as_float(cal_s[h][5]) : -INFINITY, m_f = fp_m[h], m = fmaxf(m_v, m_f);
    const float wv = m_v == -INFINITY ? 0.f : exp2f((m_v - m) * LOG2E), wf = m_f == -INFINITY ? 0.f : exp2f((m_f - m) * LOG2E);
    o = o * wv + (VW == 2 ? fp_o[e] + fp_o[kMaxRep * kHeadDim + e] : fp_o[e]) * wf;
    const int peer = e / slice;
    st_peer(map_peer(smem_u32(&recv_o[rank * slice + e % slice]), peer), o);
    if (d < S) st_peer2(map_peer(smem_u32(&recv_ml[rank][h]), d), m, l * wv + fp_l[h] * wf);
  }
  __syncthreads();
  if (tid < S) arrive_peer(map_peer(smem_u32(&part_bar), tid));
  if (!wait_peers(&part_bar, WAIT_TRIES)) {
    if (tid == 0) atomicExch(status, CQ_ERR_TIMEOUT);
    cluster_arrive();      // a late peer may still store into this CTA's shared memory
    cluster_wait();
    return;
  }
  for (int i = tid; i < slice && rank * slice + i < n_out; i += NW * 32) {
    const int e = rank * slice + i, h = e >> 7;
    float m = -INFINITY, l = 0.f, o = 0.f;
    for (int p = 0; p < S; ++p) m = fmaxf(m, recv_ml[p][h].x);
    for (int p = 0; p < S; ++p) {
      const float2 v = recv_ml[p][h];
      const float w = v.x == -INFINITY ? 0.f : exp2f((v.x - m) * LOG2E);
      l = fmaf(v.y, w, l);
      o = fmaf(recv_o[p * slice + i], w, o);
    }
    out[row0 * kHeadDim + e] = Elem<T>::from_f(o / l);
  }
}

// ---- host side ---------------------------------------------------------------------------------------------
struct Plan { int S, pitch, smem; };

constexpr int STATIC_SMEM = 9 * 1024;           // upper bound of the kernel's static shared memory
constexpr int SMEM_TWO = 113 * 1024 - STATIC_SMEM;

// Estimates in microseconds, fitted to steps timed both ways and with every cluster size (7376 shapes: batch 1-64, 32 to 32768
// visual and up to 1000 full-precision tokens, 1 to 8 query heads, all bit widths; they held to about a tenth).  The single launch has
// become 2 to 6 % faster since and the constants were not fitted anew: of 400 drawn shapes timed in both forms, one step after the other,
// 79 took more than 3 % longer than the other form would, 27 % at most (2 x 8 x 8192 at 4 bits 19.4 us against 15.2).
struct Cost {
  double unit, unit_ragged;      // a CTA's time per 256 visual tokens
  double split, split_ragged;    // the separate launches', per 256 tokens of a KV head and SM
};
inline Cost cost_of(int bits) {
  return bits == 1 ? Cost{1.15, 1.8, 1.1, 1.6} : bits == 2 ? Cost{1.5, 2.1, 1.27, 2.05} : Cost{1.95, 3.2, 1.53, 2.6};
}

// One launch, with which cluster, or the separate launches of cq_decode_mma.cu.
//   * All clusters resident at once: whatever the estimates say, over the cluster sizes whose logits fit and whose CTAs all have
//     a visual unit or 64 full-precision tokens.  (256 visual and 1000 text tokens in one CTA per KV head take 37 us, in
//     clusters of eight 12.6, in separate launches 13.8; 20 x 8 x 5152 at 4 bits fit clusters of one only: 127 against 73.)
//     A grid of at most a CTA per SM has half the warps: it stops paying at eight units a CTA, at 4 bits four (2 x 8 x 18432 tokens
//     at 1 bit 30.9 us against 28.7; 2 x 8 x 9216 at 4 bits 20.5 against 15.2).  The estimate has to win by 4 %, so that ties stay
//     where the step does not depend on its neighbours' tails.
//   * More pairs than that, 1 and 2 bits, clusters of one or two with up to 16 units and three chunks a CTA: several rounds,
//     where the last one is at least 0.85 full and there are at most four, or where the second of two is a quarter to a half
//     full, when its CTAs have an SM each (294 shapes timed: 0.95 of the separate launches' time, 26 of them slower by more than
//     3 %; 64 x 8 x 6656 at 2 bits and six heads 169 against 179, 161 now; 80 x 8 x 3328, 2.16 rounds, would take 111 against 107).
inline bool make_plan(const cq_decode_args* a, Plan* p) {
  const int n_rep = a->n_q_heads / a->n_kv_heads, n_units = (a->t_vis + UNIT_TOK - 1) / UNIT_TOK;
  const int fp_chunks = (a->t_fp + FPC - 1) / FPC, most = n_units > (a->t_fp + 63) / 64 ? n_units : (a->t_fp + 63) / 64;
  const int64_t pairs = (int64_t)a->batch * a->n_kv_heads;
  const int sms = sm_count();
  const bool ragged = a->t_vis % UNIT_TOK != 0;
  const Cost c = cost_of(a->bits);
  const double heads = n_rep > 4 ? 1.2 : 1.0, load = (double)pairs * n_units / sms;
  const auto units_of = [&](int S) { return (n_units + S - 1) / S; };
  const auto chunks_of = [&](int S) { return (((a->t_fp + 15) / 16 + S - 1) / S + 7) / 8; };      // 16-token tiles are dealt out
  const auto fits = [&](int S, Plan* q) {
    const int pitch = units_of(S) * UNIT_TOK + 8;
    const int64_t smem = 1024 + ring_bytes(a->bits) + (int64_t)n_rep * pitch * 2;
    if (smem > SMEM_TWO) return false;
    q->S = S; q->pitch = pitch; q->smem = (int)smem;
    return true;
  };
  double best = 14.5 + (ragged ? 2.5 + c.split_ragged * heads * load : c.split * heads * load) + (a->t_fp ? 3.4 : 0.0) + 2.18 * pairs * fp_chunks / sms +
                0.13 * pairs * n_rep / sms - (load < 4.0 ? 4.4 - 1.1 * load : 0.0);
  bool resident = false, found = false;
  Plan q;
  for (int S = 1; S <= MAX_CLUSTER; S *= 2) {
    if (S > most || !fits(S, &q) || pairs > max_clusters(S)) continue;
    resident = true;
    const bool two = pairs * S > sms;
    if (!two && units_of(S) > (a->bits == 4 ? 4 : 8)) continue;
    const double t = 7.0 + (two ? 1.55 : 1.0) * ((ragged ? c.unit_ragged : c.unit) * heads * units_of(S) + chunks_of(S) * (2.2 + 0.22 * n_rep));
    if (t * 1.04 < best) { best = t * 1.04; *p = q; found = true; }
  }
  if (resident || a->bits > 2 || ragged) return found;
  for (int S = 1; S <= 2; S *= 2) {
    if (S > n_units || !fits(S, p)) continue;
    const int64_t fit = max_clusters(S), rounds = (pairs + fit - 1) / fit;
    return units_of(S) <= 16 && chunks_of(S) <= 3 &&
           ((rounds <= 4 && pairs * 20 >= rounds * fit * 17) || (pairs * 4 >= fit * 5 && pairs * 2 <= fit * 3));
  }
  return false;
}

template <typename T, int BITS, bool SPLIT, bool RAGGED>
static int launch(const cq_decode_args* a, const Plan& p, int* status, cudaStream_t st) {
  auto kern = step_kernel<T, BITS, SPLIT, RAGGED>;
  static bool configured[64] = {};
  static std::mutex mu;                          // host threads may share a device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return CQ_ERR_LAUNCH;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!configured[dev]) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TWO) != cudaSuccess) return CQ_ERR_LAUNCH;
      configured[dev] = true;
    }
  }
  Args d;
  d.batch = a->batch; d.hq = a->n_q_heads; d.hkv = a->n_kv_heads; d.n_rep = d.hq / d.hkv;
  d.t_vis = a->t_vis; d.t_fp = a->t_fp; d.t_sys = a->t_sys; d.calibrate = a->calibrate ? 1 : 0;
  d.n_units = (a->t_vis + UNIT_TOK - 1) / UNIT_TOK;
  d.pitch = p.pitch;
  d.fp_stride_b = a->fp_stride_b; d.fp_stride_h = a->fp_stride_h; d.mask_stride_b = a->mask_stride_b;
  d.t_fp_dev = a->t_fp_dev; d.mask = a->mask;
  const uint64_t pairs = (uint64_t)a->batch * a->n_kv_heads, rows = pairs * kHeadDim, n_groups = (uint64_t)a->t_vis / 32;
  CUtensorMap tm_code, tm_ks, tm_kmn, tm_v;
  constexpr CUtensorMapSwizzle sw = BITS == 1 ? CU_TENSOR_MAP_SWIZZLE_32B : BITS == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
  if (RAGGED) {
    memset(&tm_code, 0, sizeof(tm_code)); memset(&tm_ks, 0, sizeof(tm_ks)); memset(&tm_kmn, 0, sizeof(tm_kmn));
  } else if (!make_map(&tm_code, a->k_code, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, n_groups * BITS, rows, sw, UNIT_G * BITS) ||
      !make_map(&tm_ks, a->k_scale, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, n_groups, rows, CU_TENSOR_MAP_SWIZZLE_NONE, UNIT_G) ||
      !make_map(&tm_kmn, a->k_mn, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, n_groups, rows, CU_TENSOR_MAP_SWIZZLE_NONE, UNIT_G)) {
    return CQ_ERR_LAUNCH;
  }
  if (!make_v_map<BITS>(&tm_v, a->v_code, pairs * a->t_vis)) return CQ_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pairs * p.S));
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
  if (cudaLaunchKernelEx(&cfg, kern, tm_code, tm_ks, tm_kmn, tm_v, d, static_cast<const T*>(a->q), a->v_code,
                         static_cast<const T*>(a->v_scale), static_cast<const T*>(a->v_mn), static_cast<const T*>(a->k_fp),
                         static_cast<const T*>(a->v_fp), static_cast<T*>(a->out), status, a->k_code,
                         static_cast<const T*>(a->k_scale), static_cast<const T*>(a->k_mn)) != cudaSuccess)
    return CQ_ERR_LAUNCH;
  return check_launch();
}

}  // namespace cl
}  // namespace mma

bool cluster_path_eligible(const cq_decode_args* a) {
  mma::cl::Plan p;
  return mma_path_eligible(a) && mma::cl::make_plan(a, &p);
}

int cluster_path_run(const cq_decode_args* a, void* workspace, cudaStream_t st, int* status_word) {
  using namespace mma::cl;
  Plan p;
  if (!make_plan(a, &p)) return CQ_ERR_UNSUPPORTED;
  int* status = status_word ? status_word : static_cast<int*>(workspace);
  const bool split = a->n_q_heads / a->n_kv_heads <= 4, ragged = a->t_vis % UNIT_TOK != 0;
#define CQ_STEP(T, B)                                                                                          \
  (split ? (ragged ? launch<T, B, true, true>(a, p, status, st) : launch<T, B, true, false>(a, p, status, st)) \
         : (ragged ? launch<T, B, false, true>(a, p, status, st) : launch<T, B, false, false>(a, p, status, st)))
  if (a->dtype == CQ_DTYPE_F16) return a->bits == 1 ? CQ_STEP(__half, 1) : a->bits == 2 ? CQ_STEP(__half, 2) : CQ_STEP(__half, 4);
  return a->bits == 1 ? CQ_STEP(__nv_bfloat16, 1) : a->bits == 2 ? CQ_STEP(__nv_bfloat16, 2) : CQ_STEP(__nv_bfloat16, 4);
#undef CQ_STEP
}

}  // namespace cq
