// Flash attention backward as two tcgen05 kernels (head_dim 128 or 64), the default backward of attention.cu's forward.
//
//   dkv kernel   one CTA per 128-key tile walks the query tiles that see it, in transposed form so that keys are the
//                TMEM lanes:  S^T = Kh Qh^T,  dP^T = V dO^T,  P^T = exp2(S^T c1 - lse2) masked,  dV += P^T dO,
//                dS^T = P^T (dP^T - delta) scale,  dK += dS^T Qh.
//                dS^T also goes to memory where there is scratch for it.
//   dq kernel    one CTA per 128-query tile walks its key tiles (queries are the lanes):  dQ += dS Kh with the stored dS^T, or, without
//                the scratch, S and dP again, dS, dQ += dS Kh.
//
// P^T, dS^T and dS reach their MMAs without shared memory: the compute warps write them back to TMEM as packed bf16 pairs over the
// columns of the fp32 tile they were computed from, and the next MMA takes its A operand from TMEM.  Every accumulator
// (dK, dV, dQ) lives in TMEM for the whole CTA: no atomics, no per-tile drain, deterministic results.  In the single-kernel
// form (attention_bwd.cu) TMEM is full and the five GEMMs serialise with the exponentiation and a dQ drain through fp32 atomics.
// Outputs are bf16: dq-hat | dk-hat as [B*T, 2A] for the RoPE / QK-norm backward, dV straight into its third of dqkv.
// Operand views, masking and scaling are those of attention_bwd.cu; the saved log-sum-exp is consumed through a
// pre-pass that also computes delta = rowsum(dO * O).
#include "common.cuh"

namespace bones {

constexpr int ST = 128;
constexpr uint32_t SATOM = ST * 64 * 2;    // 16 KB: one 128-byte-swizzled atom of [128 rows][64 cols]; a tile has D / 64
constexpr float kLog2e = 1.4426950408889634f;

// Cycle accounting of the dK / dV kernel's roles, compiled in only with -DBONES_ATTN_PROF (a measuring build; the regular
// library carries none of it).  Each role sums the clocks it spends in each of its waits and in its work and stores the
// sums in its CTA's 32 slots of the buffer given to `bones_attn_set_prof`:
//   MMA warp: 0 wait item + K/V  1 wait Q  2 wait dO  3 wait P ready  4 wait accumulators free  5 wait dS ready  6 issue  7 total
//             8 tiles;  compute warp 2: 10 wait statistics  11 wait S  12 P  13 wait dP  14 dS  15 wait done  16 drain  17 total;
//   producer: 20 waits  21 issue.
#ifdef BONES_ATTN_PROF
__device__ long long* g_attn_prof = nullptr;
#define APROF_DECL(n) long long ap_[n] = {}; long long ap_t_ = clock64(); const long long ap_t0_ = ap_t_
#define APROF_ADD(i) do { const long long n_ = clock64(); ap_[i] += n_ - ap_t_; ap_t_ = n_; } while (0)
#define APROF_COUNT(i) (++ap_[i])
#define APROF_STORE(slot, i) do { if (g_attn_prof) g_attn_prof[(long long)blockIdx.x * 32 + (slot)] = ap_[i]; } while (0)
#define APROF_TOTAL(slot) do { if (g_attn_prof) g_attn_prof[(long long)blockIdx.x * 32 + (slot)] = clock64() - ap_t0_; } while (0)
#else
#define APROF_DECL(n)
#define APROF_ADD(i)
#define APROF_COUNT(i)
#define APROF_STORE(slot, i)
#define APROF_TOTAL(slot)
#endif

struct SplitParams {
  int B, T, H;
  int Tp;                // T rounded up to whole tiles: row length of the statistics
  float c1, scale;
  int window_tiles;
  const int* doc_start;
  const float2* stats;   // [B, H, Tp]: (-lse * log2(e), delta); (-inf, 0) past T, so that the queries there have P = 0
  __nv_bfloat16* dqk;    // [B*T, 2A]: dq-hat | dk-hat
  __nv_bfloat16* ds;     // dS^T of every tile pair, [slot][16 strips of 8 queries][128 keys][8], for the dQ kernel that reads it; or null
  int slots;             // tile pairs of a (sequence, head) in that buffer
  __nv_bfloat16* dv;     // rows of dv_ld elements
  long long dv_ld;
  int* err;
  int* items;            // device counter the persistent CTAs of a launch draw their work items from (zero at launch)
};

__device__ __forceinline__ int split_first_tile(const SplitParams& p, int b, int qt) {
  int lo = 0;
  if (p.doc_start) lo = min(max(p.doc_start[(long long)b * p.T + qt * ST] / ST, 0), qt);
  if (p.window_tiles > 0) lo = max(lo, qt - p.window_tiles + 1);
  return lo;
}
// Where the tile pair (query tile qt, key tile kt) of a (sequence, head) stands in the buffer of dS^T: the query tiles one after
// another, each with the key tiles that causality and the band allow (those of earlier documents are neither written nor read).
__host__ __device__ __forceinline__ int ds_before(int qt, int w) {        // slots of the query tiles before qt; w: window_tiles
  return w <= 0 || qt <= w ? qt * (qt + 1) / 2 : w * (w + 1) / 2 + (qt - w) * w;
}
__device__ __forceinline__ long long ds_slot(const SplitParams& p, int b, int h, int qt, int kt) {
  const int first = p.window_tiles > 0 ? max(0, qt - p.window_tiles + 1) : 0;
  return ((long long)b * p.H + h) * p.slots + ds_before(qt, p.window_tiles) + kt - first;
}
// Descriptors are the tile's base descriptor plus a compile-time step in the address field (16-byte units; shared-memory
// addresses stay below 2^18, so the field never carries): one 64-bit add per operand and MMA in the issuing loop instead
// of the mask-shift-or chain of a fresh descriptor.
__device__ __forceinline__ uint64_t sdesc_k(uint32_t tile, int k) {   // K-major view, UMMA_K step k
  return umma_smem_desc(tile, 0, 1024, kLayoutSw128) + (uint64_t)(((k >> 2) * SATOM + (k & 3) * 32) >> 4);
}
__device__ __forceinline__ uint64_t sdesc_mn(uint32_t tile, int k) {  // MN-major view of the same bytes
  return umma_smem_desc(tile, SATOM, 1024, kLayoutSw128) + (uint64_t)((k * 2048) >> 4);
}
// Compute warps: four per 32-lane TMEM quadrant, each thread one row and 32 of the tile's 128 columns.  With two per
// quadrant (64 columns a thread) the exponentials and the dS arithmetic of a tile took 3 300 clocks one after the other
// against 2 048 clocks of MMAs; the same work over twice the warps hides a little more of its latency (0.836 -> 0.812 ms
// for the whole backward at B = 16, T = 2048, H = 10).  A P phase still takes about 2 000 clocks: TMEM load, 1 024
// clocks of exponentials on the special-function units, TMEM store, one after the other in every warp at once.
// Computing every other exponential with a cubic on the FMA pipe was measured and made both kernels slower (the
// arithmetic of the dS phase competes for the same issue slots), so all exponentials stay on `ex2.approx`.
constexpr int SCW = 16;                      // compute warps per CTA
constexpr int STHREADS = 64 + 32 * SCW;      // producer warp + MMA warp + compute warps
// TMEM column of UMMA_K step k of a packed bf16 A operand: each compute warp packs its 32 fp32 columns (c0 = 0, 32,
// 64, 96) into the first 16 columns of its own range, two K steps of 8 packed columns each
__device__ __forceinline__ uint32_t packed_col(int k) { return (uint32_t)((k >> 1) * 32 + (k & 1) * 8); }

__device__ __forceinline__ float ex2_fast(float x) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x));
  return e;
}
// 32 fp32 values -> 16 packed bf16 pairs -> 16 TMEM columns starting at taddr
__device__ __forceinline__ void store_packed32(uint32_t taddr, const float* v) {
  uint32_t pk[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) pk[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
  BONES_TMEM_ST16(taddr, pk);
  tmem_st_wait();
}
// C accumulator columns of this thread's row -> C bf16 in global memory (32-byte sectors); dst null: nothing is stored
template <int C>
__device__ __forceinline__ void drain_row(uint32_t taddr, __nv_bfloat16* dst) {
  uint32_t v[C];
  __syncwarp();
  if constexpr (C == 32) BONES_TMEM_LD32(taddr, v);
  else BONES_TMEM_LD16(taddr, v);
  tmem_ld_wait();
  if (!dst) return;
  uint4 u[C / 8];
#pragma unroll
  for (int g = 0; g < C / 8; ++g) {
    u[g].x = pack_bf16(__uint_as_float(v[g * 8 + 0]), __uint_as_float(v[g * 8 + 1]));
    u[g].y = pack_bf16(__uint_as_float(v[g * 8 + 2]), __uint_as_float(v[g * 8 + 3]));
    u[g].z = pack_bf16(__uint_as_float(v[g * 8 + 4]), __uint_as_float(v[g * 8 + 5]));
    u[g].w = pack_bf16(__uint_as_float(v[g * 8 + 6]), __uint_as_float(v[g * 8 + 7]));
  }
#pragma unroll
  for (int g = 0; g < C / 8; g += 2) st_global_v8(dst + g * 8, u[g], u[g + 1]);
}

// stats[b,h,t] = (-lse * log2(e), sum_d dO * O); D / 8 lanes per (head, two positions), 16 bytes of each operand and
// position per lane (64 bytes of loads in flight: 36.6 -> 30.8 us at 32768 rows of 10 heads, where the copy rate gives 26).
// Items run in the order of the output, [b, h, t] with t fastest: a group still reads 2 D contiguous bytes of each
// operand, and the statistics and the log-sum-exp values of neighbouring groups are neighbours in memory (with the
// head fastest they were T elements apart: one 32-byte sector per 8-byte result).  Positions T .. Tp - 1 get (-inf, 0).
// The first thread zeroes the work-item counters of the two kernels that follow on the stream.
template <int D>
__global__ void attn_bwd_stats_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ y,
                                      const float* __restrict__ lse, float2* __restrict__ stats, int* counters, int B, int T, int Tp, int H) {
  constexpr int LANES = D / 8;
  if (blockIdx.x == 0 && threadIdx.x < 2) counters[threadIdx.x] = 0;
  const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
  const int lane = threadIdx.x & (LANES - 1);
  const long long total = (long long)B * H * Tp / 2;
  const long long it = (item < total ? item : total - 1) * 2;      // every lane takes part in the shuffles; Tp is even
  const long long bh = it / Tp;
  const int tp = (int)(it - bh * Tp);
  const long long b = bh / H;
  const int h = (int)(bh - b * H);
  uint4 u[2], v[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const long long off = ((b * T + min(tp + j, T - 1)) * H + h) * D + lane * 8;
    u[j] = *reinterpret_cast<const uint4*>(dy + off);
    v[j] = *reinterpret_cast<const uint4*>(y + off);
  }
  float s[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t aw[4] = {u[j].x, u[j].y, u[j].z, u[j].w}, cw[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
    s[j] = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 fa = unpack_bf16(aw[i]), fc = unpack_bf16(cw[i]);
      s[j] += fa.x * fc.x + fa.y * fc.y;
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
  }
  if (lane < 2 && item < total) {
    const int t = tp + lane;
    stats[it + lane] = t < T ? make_float2(-lse[bh * T + t] * kLog2e, lane ? s[1] : s[0]) : make_float2(__int_as_float(0xff800000), 0.f);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// dK / dV  (transposed: TMEM lanes are keys, columns are queries).  A Q tile lives from S^T(i) (issued during tile
//          i-1) to dK(i), so Q has a ring of three; dO (with the tile's statistics) is first needed a tile later and
//          has a ring of two.
//          Persistent: one CTA per SM draws (key tile, head, batch) items from a device counter, the key tiles of one
//          (head, batch) side by side.  Barrier phases and the Q / dO rings run on across items; K and V are
//          single-buffered and reloaded as soon as the item's last S^T and dP^T MMAs have been issued, so the next
//          item's first tiles are computed while the compute warps drain dK and dV.
// ---------------------------------------------------------------------------------------------------------------
// shared-memory offsets, by the tile's D / 64 atoms: seven tiles, two stages of 128 x (float2 stats) travelling with dO, barriers
__host__ __device__ constexpr uint32_t dkv_bars(int D) { return (uint32_t)(D / 64) * SATOM * 7 + 2 * 1024; }
constexpr uint32_t DKV_SLACK = 512;                 // room for aligning the tiles to 1024 bytes

struct DkvItem {
  int kt, h, b, n;
};
__device__ __forceinline__ DkvItem dkv_item(const SplitParams& p, int w, int n_tiles) {
  DkvItem it;
  const int grp = w / n_tiles;
  it.kt = w % n_tiles;                                // longest walks (small kt) of a (head, batch) first
  it.h = grp % p.H;
  it.b = grp / p.H;
  // Up to the last query tile that sees this key tile: every pair that a dQ item reads (it takes all key tiles from its first one
  // on) is walked here, whatever the document starts are.  The lanes of the (whole) warp look at 32 tiles at a time.
  const int cap = p.window_tiles > 0 ? min(n_tiles - it.kt, p.window_tiles) : n_tiles - it.kt;
  it.n = cap;
  if (p.doc_start) {
    it.n = 1;                                         // a key tile is always seen by its own query tile
    for (int c = 1; c < cap; c += 32) {
      const int i = c + (int)(threadIdx.x & 31);
      const uint32_t sees = __ballot_sync(0xffffffffu, i < cap && split_first_tile(p, it.b, it.kt + i) <= it.kt);
      if (sees) it.n = c + 32 - __clz(sees);
    }
  }
  return it;
}

template <int D>
__global__ void __launch_bounds__(STHREADS, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_qk, const __grid_constant__ CUtensorMap tm_v,
                    const __grid_constant__ CUtensorMap tm_dy, const SplitParams p) {
  constexpr uint32_t STILE = (D / 64) * SATOM;
  constexpr int DT = D / 4;                            // accumulator columns a compute thread drains
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  if (base - raw > DKV_SLACK) {                       // the seven tiles would not fit behind the alignment gap
    if (threadIdx.x == 0) atomicCAS(p.err, 0, ERR_WAIT_AUX);
    return;
  }
  uint8_t* gen = smem_raw + (base - raw);
  const uint32_t sK = base, sV = base + STILE;
  auto sQ = [&](int s) { return base + STILE * (2 + s); };       // three stages
  auto sdO = [&](int s) { return base + STILE * (5 + s); };      // two stages
  const uint32_t bars = base + dkv_bars(D);
  enum { B_KV = 0, B_KVFREE, B_Q0, B_Q1, B_Q2, B_QFREE0, B_QFREE1, B_QFREE2, B_DO0, B_DO1, B_DOFREE0, B_DOFREE1, B_SFULL, B_DPFULL,
         B_PREADY, B_DSREADY, B_DONE, B_ACCFREE, B_COUNT };
  auto bar = [&](int i) { return bars + 8u * i; };
  const uint32_t tmem_slot = bars + 8u * B_COUNT;
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(gen + dkv_bars(D) + 8 * B_COUNT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + dkv_bars(D) + 8 * B_COUNT + 8);
  const uint32_t ring_bars = bars + 176u;
  volatile int* ring_slots = reinterpret_cast<volatile int*>(gen + dkv_bars(D) + 208);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int A = p.H * D;
  const int n_tiles = p.Tp / ST;
  const int total = n_tiles * p.H * p.B;

  if (threadIdx.x == 0) {
    mbar_init(bar(B_KV), 1);
    mbar_init(bar(B_KVFREE), 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(bar(B_Q0 + s), 1);
      mbar_init(bar(B_QFREE0 + s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(B_DO0 + s), 1);
      mbar_init(bar(B_DOFREE0 + s), 1);
    }
    mbar_init(bar(B_SFULL), 1);
    mbar_init(bar(B_DPFULL), 1);
    mbar_init(bar(B_PREADY), SCW);
    mbar_init(bar(B_DSREADY), SCW);
    mbar_init(bar(B_DONE), 1);
    mbar_init(bar(B_ACCFREE), SCW);
    for (int s = 0; s < 4; ++s) mbar_init(ring_bars + 8u * s, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_qk);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_dy);
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_g;
  const uint32_t tS = tmem, tdP = tmem + 128, tdV = tmem + 256, tdK = tmem + 384;

  // The producer and MMA roles run on all 32 lanes of their warp with warp-uniform state and issue from the elected lane
  // (`elect_one` in common.cuh).  Work items are drawn by lane 0 and handed round with a shuffle.  A lane whose bounded
  // wait ran out turns `dead`: it walks on without waiting or issuing; when lane 0 is dead no further item is drawn.
  if (warp == 0) {
    int g = 0, it = 0;
    bool dead = false;
    APROF_DECL(2);
    for (;; ++it) {
      int w = -1;
      if (lane == 0 && !dead) w = item_publish(ring_bars, ring_slots, it, p.items, total);
      w = warp_uniform(w);
      if (w < 0) break;
      DkvItem im = dkv_item(p, w, n_tiles);
      im.n = warp_uniform(im.n);
      APROF_ADD(1);
      if (it >= 1 && !dead) dead = !mbar_wait(bar(B_KVFREE), (uint32_t)((it - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
      APROF_ADD(0);
      if (elect_one() && !dead) {
        mbar_arrive_expect_tx(bar(B_KV), 2 * STILE);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_3d(sK + c * SATOM, &tm_qk, bar(B_KV), A + im.h * D + c * 64, im.kt * ST, im.b);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_3d(sV + c * SATOM, &tm_v, bar(B_KV), 2 * A + im.h * D + c * 64, im.kt * ST, im.b);
      }
      const float2* stat_row = p.stats + ((long long)im.b * p.H + im.h) * p.Tp;
      for (int i = 0; i < im.n; ++i, ++g) {
        const int qs = g % 3, ds = g & 1;
        const int r = (im.kt + i) * ST;
        APROF_ADD(1);
        if (g >= 3 && !dead) dead = !mbar_wait(bar(B_QFREE0 + qs), (uint32_t)(((g - 3) / 3) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        APROF_ADD(0);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(bar(B_Q0 + qs), STILE);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sQ(qs) + c * SATOM, &tm_qk, bar(B_Q0 + qs), im.h * D + c * 64, r, im.b);
        }
        APROF_ADD(1);
        if (g >= 2 && !dead) dead = !mbar_wait(bar(B_DOFREE0 + ds), (uint32_t)(((g - 2) >> 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        APROF_ADD(0);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(bar(B_DO0 + ds), STILE + 1024);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sdO(ds) + c * SATOM, &tm_dy, bar(B_DO0 + ds), im.h * D + c * 64, r, im.b);
          bulk_load(base + STILE * 7 + ds * 1024, stat_row + (im.kt + i) * ST, 1024, bar(B_DO0 + ds));
        }
      }
    }
    APROF_ADD(1);
    if (lane == 0) { APROF_STORE(20, 0); APROF_STORE(21, 1); }
  } else if (warp == 1) {
    const uint32_t id_kk = umma_idesc_f16(128, 128, 1, 0, 0);
    const uint32_t id_km = umma_idesc_f16(128, D, 1, 0, 1);
    bool dead = false;
    APROF_DECL(8);
    auto issue_s = [&](int t) {                           // S^T(t) = Kh Qh(t)^T
      APROF_ADD(6);
      if (!dead) dead = !mbar_wait(bar(B_Q0 + t % 3), (uint32_t)((t / 3) & 1), abort_flag, p.err, ERR_WAIT_FULL);
      APROF_ADD(1);
      tc_fence_after();
      if (elect_one() && !dead) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tS, sdesc_k(sK, k), sdesc_k(sQ(t % 3), k), id_kk, k ? 1u : 0u);
        tc_commit(bar(B_SFULL));
      }
    };
    auto issue_dp = [&](int t, bool last) {               // dP^T(t) = V dO(t)^T; after the item's last one K and V are free
      APROF_ADD(6);
      if (!dead) dead = !mbar_wait(bar(B_DO0 + (t & 1)), (uint32_t)((t >> 1) & 1), abort_flag, p.err, ERR_WAIT_FULL);
      APROF_ADD(2);
      tc_fence_after();
      if (elect_one() && !dead) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tdP, sdesc_k(sV, k), sdesc_k(sdO(t & 1), k), id_kk, k ? 1u : 0u);
        tc_commit(bar(B_DPFULL));
        if (last) tc_commit(bar(B_KVFREE));
      }
    };
    int g = 0, it = 0;
    for (;; ++it) {
      int w = -1;
      APROF_ADD(6);
      if (!dead) w = item_take(ring_bars, ring_slots, it, abort_flag, p.err);
      w = warp_uniform(w);
      if (w < 0) break;
      DkvItem im = dkv_item(p, w, n_tiles);
      im.n = warp_uniform(im.n);
      if (!dead) dead = !mbar_wait(bar(B_KV), (uint32_t)(it & 1), abort_flag, p.err, ERR_WAIT_FULL);
      APROF_ADD(0);
      // the first tile's S^T and dP^T go behind the previous item's last dV / dK MMAs on the same (in-order) pipe
      issue_s(g);
      issue_dp(g, im.n == 1);
      for (int i = 0; i < im.n; ++i, ++g) {
        const int s = g & 1, qs = g % 3;
        const uint32_t ph = (uint32_t)(g & 1);
        const bool more = i + 1 < im.n;
        // P^T(g) sits packed in the S^T columns: dV += P^T dO, then S^T(g+1) behind it
        APROF_ADD(6);
        APROF_COUNT(7);
        if (!dead) dead = !mbar_wait(bar(B_PREADY), ph, abort_flag, p.err, ERR_WAIT_AUX);
        APROF_ADD(3);
        // the previous item's dK / dV must have been drained
        if (i == 0 && it >= 1 && !dead) dead = !mbar_wait(bar(B_ACCFREE), (uint32_t)((it - 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
        APROF_ADD(4);
        tc_fence_after();
        if (elect_one() && !dead) {
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16_ts(tdV, tS + packed_col(k), sdesc_mn(sdO(s), k), id_km, (i | k) ? 1u : 0u);
        }
        if (more) issue_s(g + 1);
        // dS^T(g) sits packed in the dP^T columns: dK += dS^T Qh, then dP^T(g+1) behind it
        APROF_ADD(6);
        if (!dead) dead = !mbar_wait(bar(B_DSREADY), ph, abort_flag, p.err, ERR_WAIT_AUX);
        APROF_ADD(5);
        tc_fence_after();
        if (elect_one() && !dead) {
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16_ts(tdK, tdP + packed_col(k), sdesc_mn(sQ(qs), k), id_km, (i | k) ? 1u : 0u);
          tc_commit(bar(B_QFREE0 + qs));
          tc_commit(bar(B_DOFREE0 + s));     // dO(g) was read by dV(g); its statistics were in use until dS(g) was stored
          if (!more) tc_commit(bar(B_DONE));
        }
        if (more) issue_dp(g + 1, i + 2 == im.n);
      }
    }
    APROF_ADD(6);
    if (lane == 0) {
      for (int i = 0; i < 7; ++i) APROF_STORE(i, i);
      APROF_TOTAL(7);
      APROF_STORE(8, 7);
    }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2;
    const int r = q * 32 + lane;                       // key row of this thread
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const int c0 = part * 32;                          // first query column of this thread
    bool ok = true;
    int g = 0, it = 0;
    APROF_DECL(8);
    for (;; ++it) {
      const int w = ok ? item_take(ring_bars, ring_slots, it, abort_flag, p.err) : -1;
      if (w < 0) break;
      const DkvItem im = dkv_item(p, w, n_tiles);
      const int k0 = im.kt * ST, kpos = k0 + r;
      const long long row0 = (long long)im.b * p.T;
      int nx_lo_last = p.doc_start ? p.doc_start[row0 + min(k0 + ST, p.T) - 1] : 0;
      for (int i = 0; i < im.n; ++i, ++g) {
        const int s = g & 1;
        const uint32_t ph = (uint32_t)(g & 1);
        APROF_ADD(2);
        bool got = mbar_wait(bar(B_DO0 + s), (uint32_t)((g >> 1) & 1), abort_flag, p.err, ERR_WAIT_FULL);   // this tile's statistics
        APROF_ADD(0);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        const float4* st4 = reinterpret_cast<const float4*>(gen + STILE * 7 + s * 1024) + c0 / 2;   // two queries per float4
        // document starts of this tile's queries (global, cached): only the tile that straddles a document start past
        // this key tile needs them element by element, and its last query decides that
        const int q0 = (im.kt + i) * ST;
        const int* slo = p.doc_start ? p.doc_start + row0 + q0 : nullptr;
        const bool need_doc = slo && nx_lo_last > k0;
        if (slo && i + 1 < im.n) nx_lo_last = slo[min(2 * ST, p.T - q0) - 1];
        float pr[32];
        got = mbar_wait(bar(B_SFULL), ph, abort_flag, p.err, ERR_WAIT_TMEM_FULL);
        APROF_ADD(1);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t v0[32];
          __syncwarp();
          BONES_TMEM_LD32(tS + lane_addr + (uint32_t)c0, v0);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float4 a = st4[j];
            pr[2 * j] = ex2_fast(fmaf(__uint_as_float(v0[2 * j]), p.c1, a.x));
            pr[2 * j + 1] = ex2_fast(fmaf(__uint_as_float(v0[2 * j + 1]), p.c1, a.z));
          }
        }
        if (i == 0) {                                    // diagonal tile: a key sees only queries at or after it
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (r > c0 + j) pr[j] = 0.f;
        }
        if (need_doc) {                                  // a query sees only keys of its own document
          if (q0 + ST <= p.T) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (kpos < slo[c0 + j]) pr[j] = 0.f;
          } else {                                       // last tile of a ragged sequence: P is already 0 past its end
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (q0 + c0 + j < p.T && kpos < slo[c0 + j]) pr[j] = 0.f;
          }
        }
        store_packed32(tS + lane_addr + (uint32_t)c0, pr);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(B_PREADY));
        APROF_ADD(2);
        got = mbar_wait(bar(B_DPFULL), ph, abort_flag, p.err, ERR_WAIT_TMEM_FULL);
        APROF_ADD(3);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t v0[32];
          __syncwarp();
          BONES_TMEM_LD32(tdP + lane_addr + (uint32_t)c0, v0);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float4 a = st4[j];
            pr[2 * j] *= (__uint_as_float(v0[2 * j]) - a.y) * p.scale;
            pr[2 * j + 1] *= (__uint_as_float(v0[2 * j + 1]) - a.w) * p.scale;
          }
        }
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) pk[j] = pack_bf16(pr[2 * j], pr[2 * j + 1]);
        BONES_TMEM_ST16(tdP + lane_addr + (uint32_t)c0, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(B_DSREADY));
        // behind the hand-over: four strips of 8 queries, where the 32 key rows of a warp are neighbours (512 B contiguous a
        // store; as rows of 128 queries, 32 lines a store, this cost 44 us of 287)
        if (p.ds) {
          uint4* dst = reinterpret_cast<uint4*>(p.ds + ds_slot(p, im.b, im.h, im.kt + i, im.kt) * 16384) + part * 4 * 128 + r;
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[j * 128] = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
        }
        APROF_ADD(4);
      }
      if (!ok) break;
      const bool got = mbar_wait(bar(B_DONE), (uint32_t)(it & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
      APROF_ADD(5);
      if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
      tc_fence_after();
      const long long hcol = (long long)im.h * D + part * DT;
      drain_row<DT>(tdK + lane_addr + (uint32_t)(part * DT), kpos < p.T ? p.dqk + (row0 + kpos) * 2 * A + A + hcol : nullptr);
      drain_row<DT>(tdV + lane_addr + (uint32_t)(part * DT), kpos < p.T ? p.dv + (row0 + kpos) * p.dv_ld + hcol : nullptr);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_ACCFREE));
      APROF_ADD(6);
    }
    if (warp == 2 && lane == 0) {
      APROF_STORE(10, 0); APROF_STORE(11, 1); APROF_STORE(12, 2); APROF_STORE(13, 3); APROF_STORE(14, 4); APROF_STORE(15, 5); APROF_STORE(16, 6);
      APROF_TOTAL(17);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// dQ  (TMEM lanes are queries, columns are keys; dP double-buffered so the MMAs of tile j+1 run under the
//      exponentiation of tile j).  K tiles live from S(j) to dQ(j), V tiles only until dP(j): a K ring of three and a V
//      ring of two keep every load a full tile ahead of its first use.
//      One "dS ready" barrier per dP buffer: S(j+1) and dP(j+1) are issued before dS(j) is awaited, so a compute warp
//      can finish tile j+1 while a slower one is still on tile j; with one barrier for both buffers its second
//      arrival completed the slower warp's phase and the dQ MMAs read that warp's columns before it had stored them
//      (a few non-finite rows of dq once in a few hundred calls, more often with sixteen compute warps whose masking
//      work differs).  dP(j+2) is only issued after dQ(j), so nobody can be two tiles ahead.
//      Persistent: one CTA per SM walks (query tile, head, batch) items in the forward kernel's order (the query tiles
//      of one (head, batch) run at the same time and share K/V through L2).  Barrier phases, the K/V rings and the dP
//      buffers run on across items; Q and dO are single-buffered and reloaded as soon as the item's last S and dP MMAs
//      have been issued, so the next item's first tiles are computed while the compute warps drain dQ.
// ---------------------------------------------------------------------------------------------------------------
__host__ __device__ constexpr uint32_t dq_bars(int D) { return (uint32_t)(D / 64) * SATOM * 7; }

struct DqItem {
  int qt, h, b, kt0, n;
};
__device__ __forceinline__ DqItem dq_item(const SplitParams& p, int w, int n_tiles) {
  DqItem it;
  const int grp = w / n_tiles;
  it.qt = n_tiles - 1 - (w % n_tiles + grp) % n_tiles;
  it.h = grp % p.H;
  it.b = grp / p.H;
  it.kt0 = split_first_tile(p, it.b, it.qt);
  it.n = it.qt - it.kt0 + 1;
  return it;
}

template <int D>
__global__ void __launch_bounds__(STHREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_qk, const __grid_constant__ CUtensorMap tm_v,
                   const __grid_constant__ CUtensorMap tm_dy, const SplitParams p) {
  constexpr uint32_t STILE = (D / 64) * SATOM;
  constexpr int DT = D / 4;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  const uint32_t sQ = base, sdO = base + STILE;
  auto sK = [&](int s) { return base + STILE * (2 + s); };      // three stages
  auto sV = [&](int s) { return base + STILE * (5 + s); };      // two stages
  const uint32_t bars = base + dq_bars(D);
  enum { B_QDO = 0, B_QDOFREE, B_K0, B_K1, B_K2, B_KFREE0, B_KFREE1, B_KFREE2, B_V0, B_V1, B_VFREE0, B_VFREE1, B_SFULL, B_SFREE,
         B_DPFULL0, B_DPFULL1, B_DSREADY0, B_DSREADY1, B_DONE, B_DQFREE, B_COUNT };
  auto bar = [&](int i) { return bars + 8u * i; };
  const uint32_t tmem_slot = bars + 8u * B_COUNT;
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(gen + dq_bars(D) + 8 * B_COUNT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + dq_bars(D) + 8 * B_COUNT + 8);
  const uint32_t ring_bars = bars + 176u;
  volatile int* ring_slots = reinterpret_cast<volatile int*>(gen + dq_bars(D) + 208);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int A = p.H * D;
  const int n_tiles = p.Tp / ST;
  const int total = n_tiles * p.H * p.B;

  if (threadIdx.x == 0) {
    mbar_init(bar(B_QDO), 1);
    mbar_init(bar(B_QDOFREE), 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(bar(B_K0 + s), 1);
      mbar_init(bar(B_KFREE0 + s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(B_V0 + s), 1);
      mbar_init(bar(B_VFREE0 + s), 1);
      mbar_init(bar(B_DPFULL0 + s), 1);
    }
    mbar_init(bar(B_SFULL), 1);
    mbar_init(bar(B_SFREE), SCW);
    mbar_init(bar(B_DSREADY0), SCW);
    mbar_init(bar(B_DSREADY1), SCW);
    mbar_init(bar(B_DONE), 1);
    mbar_init(bar(B_DQFREE), SCW);
    for (int s = 0; s < 4; ++s) mbar_init(ring_bars + 8u * s, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_qk);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_dy);
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_g;
  const uint32_t tS = tmem, tdQ = tmem + 384;
  auto tdP = [&](int s) { return tmem + 128u + (uint32_t)s * 128u; };

  // producer and MMA roles: warp-uniform loops issuing from the elected lane, as in the dK / dV kernel above
  if (warp == 0) {
    int g = 0, it = 0;
    bool dead = false;
    for (;; ++it) {
      int w = -1;
      if (lane == 0 && !dead) w = item_publish(ring_bars, ring_slots, it, p.items, total);
      w = warp_uniform(w);
      if (w < 0) break;
      DqItem im = dq_item(p, w, n_tiles);
      im.kt0 = warp_uniform(im.kt0);
      im.n = im.qt - im.kt0 + 1;
      if (it >= 1 && !dead) dead = !mbar_wait(bar(B_QDOFREE), (uint32_t)((it - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
      if (elect_one() && !dead) {
        mbar_arrive_expect_tx(bar(B_QDO), 2 * STILE);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_3d(sQ + c * SATOM, &tm_qk, bar(B_QDO), im.h * D + c * 64, im.qt * ST, im.b);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_3d(sdO + c * SATOM, &tm_dy, bar(B_QDO), im.h * D + c * 64, im.qt * ST, im.b);
      }
      for (int j = 0; j < im.n; ++j, ++g) {
        const int ks = g % 3, vs = g & 1;
        const int r = (im.kt0 + j) * ST;
        if (g >= 3 && !dead) dead = !mbar_wait(bar(B_KFREE0 + ks), (uint32_t)(((g - 3) / 3) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(bar(B_K0 + ks), STILE);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sK(ks) + c * SATOM, &tm_qk, bar(B_K0 + ks), A + im.h * D + c * 64, r, im.b);
        }
        if (g >= 2 && !dead) dead = !mbar_wait(bar(B_VFREE0 + vs), (uint32_t)(((g - 2) >> 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(bar(B_V0 + vs), STILE);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sV(vs) + c * SATOM, &tm_v, bar(B_V0 + vs), 2 * A + im.h * D + c * 64, r, im.b);
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t id_kk = umma_idesc_f16(128, 128, 1, 0, 0);
    const uint32_t id_km = umma_idesc_f16(128, D, 1, 0, 1);
    bool dead = false;
    // S(t) and dP(t) of running tile t; `last`: t is the last tile of its item, after which Q and dO may be reloaded
    auto issue_sdp = [&](int t, bool last) {
      if (!dead) dead = !mbar_wait(bar(B_K0 + t % 3), (uint32_t)((t / 3) & 1), abort_flag, p.err, ERR_WAIT_FULL);
      if (t >= 1 && !dead) dead = !mbar_wait(bar(B_SFREE), (uint32_t)((t - 1) & 1), abort_flag, p.err, ERR_WAIT_AUX);
      tc_fence_after();
      if (elect_one() && !dead) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tS, sdesc_k(sQ, k), sdesc_k(sK(t % 3), k), id_kk, k ? 1u : 0u);
        tc_commit(bar(B_SFULL));
      }
      if (!dead) dead = !mbar_wait(bar(B_V0 + (t & 1)), (uint32_t)((t >> 1) & 1), abort_flag, p.err, ERR_WAIT_FULL);
      tc_fence_after();
      // dP(t) goes into the buffer whose packed dS(t-2) the dQ MMAs of tile t-2 (issued earlier, same pipe) have read
      if (elect_one() && !dead) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tdP(t & 1), sdesc_k(sdO, k), sdesc_k(sV(t & 1), k), id_kk, k ? 1u : 0u);
        tc_commit(bar(B_DPFULL0 + (t & 1)));
        tc_commit(bar(B_VFREE0 + (t & 1)));
        if (last) tc_commit(bar(B_QDOFREE));
      }
    };
    int g = 0, it = 0;
    for (;; ++it) {
      int w = -1;
      if (!dead) w = item_take(ring_bars, ring_slots, it, abort_flag, p.err);
      w = warp_uniform(w);
      if (w < 0) break;
      DqItem im = dq_item(p, w, n_tiles);
      im.kt0 = warp_uniform(im.kt0);
      im.n = im.qt - im.kt0 + 1;
      if (!dead) dead = !mbar_wait(bar(B_QDO), (uint32_t)(it & 1), abort_flag, p.err, ERR_WAIT_FULL);
      for (int j = 0; j < im.n; ++j, ++g) {
        if (j == 0) issue_sdp(g, im.n == 1);
        if (j + 1 < im.n) issue_sdp(g + 1, j + 2 == im.n);
        // dS(g) sits packed in the dP(g) columns: dQ += dS Kh(g), which also frees that K stage
        if (!dead) dead = !mbar_wait(bar(B_DSREADY0 + (g & 1)), (uint32_t)((g >> 1) & 1), abort_flag, p.err, ERR_WAIT_AUX);
        if (j == 0 && it >= 1 && !dead) dead = !mbar_wait(bar(B_DQFREE), (uint32_t)((it - 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after();
        if (elect_one() && !dead) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_f16_ts(tdQ, tdP(g & 1) + packed_col(k), sdesc_mn(sK(g % 3), k), id_km, (j | k) ? 1u : 0u);
          tc_commit(bar(B_KFREE0 + g % 3));
          if (j + 1 == im.n) tc_commit(bar(B_DONE));
        }
      }
    }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2;
    const int r = q * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const int c0 = part * 32;
    bool ok = true;
    int g = 0, it = 0;
    for (;; ++it) {
      const int w = ok ? item_take(ring_bars, ring_slots, it, abort_flag, p.err) : -1;
      if (w < 0) break;
      const DqItem im = dq_item(p, w, n_tiles);
      const int qpos = im.qt * ST + r;
      const long long row0 = (long long)im.b * p.T;
      const float2 st = p.stats[((long long)im.b * p.H + im.h) * p.Tp + qpos];
      int lo = 0;
      if (p.doc_start && qpos < p.T) lo = p.doc_start[row0 + qpos];
      for (int j = 0; j < im.n; ++j, ++g) {
        const int s = g & 1;
        bool got = mbar_wait(bar(B_SFULL), (uint32_t)(g & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
        const int k0 = (im.kt0 + j) * ST + c0;
        const bool need_mask = __any_sync(0xffffffffu, (k0 + 31 > qpos) || (k0 < lo));
        float pr[32];
        {
          uint32_t v0[32];
          __syncwarp();
          BONES_TMEM_LD32(tS + lane_addr + (uint32_t)c0, v0);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(B_SFREE));
#pragma unroll
          for (int i = 0; i < 32; ++i) pr[i] = ex2_fast(fmaf(__uint_as_float(v0[i]), p.c1, st.x));
        }
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int kp = k0 + i;
            if (kp > qpos || kp < lo) pr[i] = 0.f;
          }
        }
        got = mbar_wait(bar(B_DPFULL0 + s), (uint32_t)((g >> 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t v0[32];
          __syncwarp();
          BONES_TMEM_LD32(tdP(s) + lane_addr + (uint32_t)c0, v0);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) pr[i] *= (__uint_as_float(v0[i]) - st.y) * p.scale;
        }
        store_packed32(tdP(s) + lane_addr + (uint32_t)c0, pr);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(B_DSREADY0 + s));
      }
      if (!ok) break;
      const bool got = mbar_wait(bar(B_DONE), (uint32_t)(it & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
      tc_fence_after();
      drain_row<DT>(tdQ + lane_addr + (uint32_t)(part * DT),
                    qpos < p.T ? p.dqk + (row0 + qpos) * 2 * A + (long long)im.h * D + part * DT : nullptr);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_DQFREE));
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// dQ from stored dS: dQ = sum over key tiles of dS Kh, with dS^T as the dK / dV kernel left it (bf16, what its own MMAs consumed).
// The kernel above computes S, the exponentials and dP a second time for this; a tile pair costs it 3 300 clocks, most of them
// exponentials and TMEM traffic, where the dQ MMAs themselves take 512.  Reading 32 KB of dS^T per tile pair instead is bound by
// memory.  16 x 2048 tokens, 10 heads (0.71 GB of dS): dQ 198 -> 101 us, 7.1 TB/s, for 288 -> 297 us of the dK / dV kernel that
// stores it.
// A tile's strips of 8 queries x 128 keys are the unswizzled MN-major operand layout as they stand (8 keys of a strip are one
// 128-byte core matrix), so a tile arrives as one 32 KB bulk copy; Kh is an MN-major operand in the usual swizzled atoms.  (Rows of
// 128 queries would load as swizzled boxes in 101 us, but cost the dK / dV kernel 44 us of scattered stores; strips of 16 with
// copying warps that swizzle took 121.)  Warp 0: item draws and loads, warp 1: MMAs, eight epilogue warps; two accumulators, so an
// item's drain hides behind the next one's MMAs.
// ---------------------------------------------------------------------------------------------------------------
constexpr int DQG_SA = 4, DQG_SB = 3, DQG_EW = 8, DQG_THREADS = 64 + 32 * DQG_EW;
constexpr int DQG_NBARS = 2 * DQG_SA + 2 * DQG_SB + 12;
__host__ __device__ constexpr uint32_t dqg_bars(int D) { return DQG_SA * 2 * SATOM + DQG_SB * (uint32_t)(D / 64) * SATOM; }

template <int D>
__global__ void __launch_bounds__(DQG_THREADS, 1)
attn_bwd_dq_gemm_kernel(const __grid_constant__ CUtensorMap tm_qk, const SplitParams p) {
  constexpr uint32_t KT = (D / 64) * SATOM, BARS = dqg_bars(D);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  auto sA = [&](int s) { return base + (uint32_t)s * 2 * SATOM; };
  auto sB = [&](int s) { return base + DQG_SA * 2 * SATOM + (uint32_t)s * KT; };
  const uint32_t bars = base + BARS;
  auto a_full = [&](int s) { return bars + 8u * s; };
  auto a_free = [&](int s) { return bars + 8u * (DQG_SA + s); };
  auto b_full = [&](int s) { return bars + 8u * (2 * DQG_SA + s); };
  auto b_free = [&](int s) { return bars + 8u * (2 * DQG_SA + DQG_SB + s); };
  auto tfull = [&](int a) { return bars + 8u * (2 * DQG_SA + 2 * DQG_SB + a); };
  auto tempty = [&](int a) { return bars + 8u * (2 * DQG_SA + 2 * DQG_SB + 2 + a); };
  const uint32_t ring_bars = bars + 8u * (2 * DQG_SA + 2 * DQG_SB + 4), ring_free = ring_bars + 32u;
  volatile int* ring_slots = reinterpret_cast<volatile int*>(gen + BARS + 8 * DQG_NBARS);
  const uint32_t tmem_slot = bars + 8u * (DQG_NBARS + 2);
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(gen + BARS + 8 * (DQG_NBARS + 2));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + BARS + 8 * (DQG_NBARS + 2) + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int A = p.H * D, n_tiles = p.Tp / ST, total = n_tiles * p.H * p.B;
  if (threadIdx.x == 0) {
    for (int s = 0; s < DQG_SA; ++s) {
      mbar_init(a_full(s), 1);
      mbar_init(a_free(s), 1);
    }
    for (int s = 0; s < DQG_SB; ++s) {
      mbar_init(b_full(s), 1);
      mbar_init(b_free(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull(a), 1);
      mbar_init(tempty(a), DQG_EW);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(ring_bars + 8u * s, 1);
      mbar_init(ring_free + 8u * s, DQG_EW + 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_qk);
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_g;
  auto take = [&](int it) {                    // a consumer takes item `it` and gives its ring slot back
    const int w = warp_uniform(item_take(ring_bars, ring_slots, it, abort_flag, p.err));
    if (lane == 0) mbar_arrive(ring_free + 8u * (it & 3));
    return w;
  };
  if (warp == 0) {
    int g = 0;
    bool dead = false;
    for (int it = 0;; ++it) {
      if (it >= 4 && !dead) dead = !mbar_wait(ring_free + 8u * (it & 3), (uint32_t)(((it >> 2) - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
      int w = -1;
      if (lane == 0 && !dead) w = item_publish(ring_bars, ring_slots, it, p.items, total);
      w = warp_uniform(w);
      if (w < 0) break;
      DqItem im = dq_item(p, w, n_tiles);
      im.kt0 = warp_uniform(im.kt0);
      im.n = im.qt - im.kt0 + 1;
      const __nv_bfloat16* ds = p.ds + ds_slot(p, im.b, im.h, im.qt, im.kt0) * 16384;
      for (int j = 0; j < im.n; ++j, ++g) {
        const int as = g % DQG_SA, s = g % DQG_SB;
        if (g >= DQG_SA && !dead) dead = !mbar_wait(a_free(as), (uint32_t)((g / DQG_SA - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(a_full(as), 2 * SATOM);
          bulk_load(sA(as), ds + (long long)j * 16384, 2 * SATOM, a_full(as));
        }
        if (g >= DQG_SB && !dead) dead = !mbar_wait(b_free(s), (uint32_t)((g / DQG_SB - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(b_full(s), KT);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sB(s) + c * SATOM, &tm_qk, b_full(s), A + im.h * D + c * 64, (im.kt0 + j) * ST, im.b);
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(128, D, 1, 1, 1);
    int g = 0;
    bool dead = false;
    for (int it = 0;; ++it) {
      const int w = dead ? -1 : take(it);
      if (w < 0) break;
      DqItem im = dq_item(p, w, n_tiles);
      im.kt0 = warp_uniform(im.kt0);
      im.n = im.qt - im.kt0 + 1;
      const int acc = it & 1;
      if (it >= 2 && !dead) dead = !mbar_wait(tempty(acc), (uint32_t)(((it - 2) >> 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
      for (int j = 0; j < im.n; ++j, ++g) {
        const int as = g % DQG_SA, bs = g % DQG_SB;
        if (!dead) dead = !mbar_wait(b_full(bs), (uint32_t)((g / DQG_SB) & 1), abort_flag, p.err, ERR_WAIT_FULL);
        if (!dead) dead = !mbar_wait(a_full(as), (uint32_t)((g / DQG_SA) & 1), abort_flag, p.err, ERR_WAIT_FULL);
        tc_fence_after();
        if (elect_one() && !dead) {
#pragma unroll
          for (int k = 0; k < 8; ++k)              // 16 keys a step: two core matrices of a strip
            umma_f16(tmem + acc * 128, umma_smem_desc(sA(as), 128, 2048, kLayoutNone) + (uint64_t)((k * 256) >> 4), sdesc_mn(sB(bs), k), idesc,
                     (j | k) ? 1u : 0u);
          tc_commit(a_free(as));
          tc_commit(b_free(bs));
          if (j == im.n - 1) tc_commit(tfull(acc));
        }
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    for (int it = 0;; ++it) {
      const int w = take(it);
      if (w < 0) break;
      const DqItem im = dq_item(p, w, n_tiles);
      const int acc = it & 1, qpos = im.qt * ST + q * 32 + lane;
      const bool got = mbar_wait(tfull(acc), (uint32_t)((it >> 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, got)) break;
      tc_fence_after();
      __nv_bfloat16* dst = qpos < p.T ? p.dqk + ((long long)im.b * p.T + qpos) * 2 * A + (long long)im.h * D : nullptr;
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        const int col = half * (D / 2) + c;
        drain_row<32>(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 128 + col), dst ? dst + col : nullptr);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty(acc));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// [B, T, cols] bf16 rows, boxes of 64 columns x 128 rows of one sequence; rows past T read as zeros
static int tmap_rows_3d_s(CUtensorMap* out, const void* ptr, int B, int T, long long cols) {
  uint64_t dims[3] = {(uint64_t)cols, (uint64_t)T, (uint64_t)B};
  uint64_t strides[2] = {(uint64_t)cols * 2, (uint64_t)cols * 2 * (uint64_t)T};
  uint32_t box[3] = {64, 128, 1};
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int D>
static int launch_split(const CUtensorMap& tq, const CUtensorMap& tv, const CUtensorMap& td, SplitParams p, int* counters, int sms, cudaStream_t s) {
  constexpr size_t smem_dkv = (size_t)dkv_bars(D) + 256 + DKV_SLACK;
  constexpr size_t smem_dq = (size_t)dq_bars(D) + 256 + 1024;
  static OncePerDevice limit;
  BONES_ONCE(limit, {
    BONES_CHECK(cudaFuncSetAttribute(attn_bwd_dkv_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_dkv));
    BONES_CHECK(cudaFuncSetAttribute(attn_bwd_dq_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_dq));
  });
  const long long items = (long long)(p.Tp / ST) * p.H * p.B;
  const unsigned grid = (unsigned)(items < sms ? items : sms);          // persistent: one CTA per SM in both kernels
  p.items = counters;
  attn_bwd_dkv_kernel<D><<<grid, STHREADS, smem_dkv, s>>>(tq, tv, td, p);
  BONES_CHECK(cudaGetLastError());
  p.items = counters + 1;
  if (p.ds) {
    constexpr size_t smem_g = (size_t)dqg_bars(D) + 8 * (DQG_NBARS + 2) + 16 + 1024;
    static OncePerDevice limit;
    BONES_ONCE(limit, {
      BONES_CHECK(cudaFuncSetAttribute(attn_bwd_dq_gemm_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_g));
    });
    attn_bwd_dq_gemm_kernel<D><<<grid, DQG_THREADS, smem_g, s>>>(tq, p);
  } else {
    attn_bwd_dq_kernel<D><<<grid, STHREADS, smem_dq, s>>>(tq, tv, td, p);
  }
  return (int)cudaGetLastError();
}

}  // namespace bones

extern "C" {
using namespace bones;

int bones_rope_qknorm_bwd_bf16(const void* qkv, const float* cosT, const float* sinT, const void* dqk, void* dqkv, long long M, int T, int H,
                               int D, void* stream);

// stats: [B, H, Tp] float2 scratch (Tp: T rounded up to a multiple of 128); counters: two ints, zeroed here
int bones_attn_bwd_stats(const void* dy, const void* y, const float* lse, void* stats, int* counters, int B, int T, int H, int D, void* stream) {
  if (misaligned16(dy, y, stats)) return -3;
  const int Tp = (T + ST - 1) / ST * ST;
  const long long threads = (long long)B * H * Tp / 2 * (D / 8);
  const unsigned grid = (unsigned)((threads + 255) / 256);
  const auto *g = (const __nv_bfloat16*)dy, *o = (const __nv_bfloat16*)y;
  if (D == 128) attn_bwd_stats_kernel<128><<<grid, 256, 0, (cudaStream_t)stream>>>(g, o, lse, (float2*)stats, counters, B, T, Tp, H);
  else if (D == 64) attn_bwd_stats_kernel<64><<<grid, 256, 0, (cudaStream_t)stream>>>(g, o, lse, (float2*)stats, counters, B, T, Tp, H);
  else return -2;
  return (int)cudaGetLastError();
}

// qk: [B*T, 2A] rotated, normalised q | k;  qkv: [B*T, 3A] (values read in place);  dy: [B*T, A];  stats and counters from the
// pre-pass.  Outputs (bf16, every element overwritten): dqk [B*T, 2A];  dv rows of dv_ld elements (e.g. the last third of dqkv).
// ds: scratch, 32 KB for each of the B * H * ds_before(tiles, window_tiles) tile pairs, 32-byte aligned; or null: dQ computes S and dP again.
int bones_attn_bwd_split(const void* qk, const void* qkv, const void* dy, const void* stats, int* counters, void* dqk, void* dv,
                         long long dv_ld, void* ds, const int* doc_start, int B, int T, int H, int D, float scale, int window_tiles, void* stream) {
  if (D != 128 && D != 64) return -2;
  if ((dv_ld % 16) || ((uintptr_t)dv & 31) || ((uintptr_t)dqk & 31) || ((uintptr_t)stats & 15)) return -3;
  const long long A = (long long)H * D;
  CUtensorMap tq, tv, td;
  int rc = tmap_rows_3d_s(&tq, qk, B, T, 2 * A);
  if (rc) return rc;
  rc = tmap_rows_3d_s(&tv, qkv, B, T, 3 * A);
  if (rc) return rc;
  rc = tmap_rows_3d_s(&td, dy, B, T, A);
  if (rc) return rc;
  SplitParams p;
  p.B = B; p.T = T; p.H = H;
  p.Tp = (T + ST - 1) / ST * ST;
  p.c1 = scale * kLog2e;
  p.scale = scale;
  p.window_tiles = window_tiles;
  p.doc_start = doc_start;
  p.stats = (const float2*)stats;
  p.dqk = (__nv_bfloat16*)dqk;
  p.dv = (__nv_bfloat16*)dv;
  p.dv_ld = dv_ld;
  p.ds = (__nv_bfloat16*)ds;
  p.slots = ds_before(p.Tp / ST, window_tiles);
  if (ds && (((uintptr_t)ds & 31) || (long long)B * H * p.slots >= (1LL << 31))) return -3;
  p.err = error_word();
  int dev = 0, sms = 0;
  BONES_CHECK(cudaGetDevice(&dev));
  BONES_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return D == 128 ? launch_split<128>(tq, tv, td, p, counters, sms, (cudaStream_t)stream)
                  : launch_split<64>(tq, tv, td, p, counters, sms, (cudaStream_t)stream);
}

// The whole backward: statistics (which zeroes the counters), dK / dV and dQ, RoPE / QK-norm backward into dqkv [B*T, 3A].
int bones_attention_bwd(const void* dy, const void* qkv, const void* qk, const void* y, const float* lse, const float* cosT, const float* sinT,
                        const int* doc_start, void* stats, int* counters, void* ds, void* dqk, void* dqkv, int B, int T, int H, int D, float scale,
                        int window_tiles, void* stream) {
  const long long A = (long long)H * D;
  int rc = bones_attn_bwd_stats(dy, y, lse, stats, counters, B, T, H, D, stream);
  if (rc) return rc;
  rc = bones_attn_bwd_split(qk, qkv, dy, stats, counters, dqk, (__nv_bfloat16*)dqkv + 2 * A, 3 * A, ds, doc_start, B, T, H, D, scale, window_tiles, stream);
  if (rc) return rc;
  return bones_rope_qknorm_bwd_bf16(qkv, cosT, sinT, dqk, dqkv, (long long)B * T, T, H, D, stream);
}

#ifdef BONES_ATTN_PROF
// measuring build: device buffer of 32 counters per CTA that the next dK / dV launches fill (null switches it off)
void bones_attn_set_prof(void* buf) {
  long long* b = (long long*)buf;
  cudaMemcpyToSymbol(bones::g_attn_prof, &b, sizeof(b));
}
#endif
}  // extern "C"
