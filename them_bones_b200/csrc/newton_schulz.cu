// Muon's Newton-Schulz iteration over a stack of matrices as one persistent kernel.
//
// Per iteration and matrix X [r, c] (s = min(r, c)):  G = X^T X or X X^T [s, s];  B = b G + c G G;  X' = a X + X B or a X + B X.
// As three batched GEMM launches an iteration this left the tensor cores idle for two reasons.  A launch of 5 matrices of
// 5120 x 1280 is 125, 125 and 500 tiles of 256 x 256 on 74 CTA pairs, so the waves are 1.7, 1.7 and 6.8 full and cost 2, 2 and 7;
// and G and B are symmetric, so nearly half of their tiles were computed twice.  Here
//   * only the tiles that reach into the lower triangle are computed, and written to both sides;
//   * the work of all iterations is one ordered list of 256 x 256 tiles that CTA pairs draw from a device counter.  A product waits
//     for the product it reads (a counter per product and matrix), and the list runs the products of different matrices side
//     by side -- G of one matrix, B of an earlier one, X' of one earlier still -- so that a matrix's own chain of three hides
//     behind the others' work.  CTAs draw items in order, and an item depends only on earlier ones: whatever part of the grid
//     is resident makes progress.
// Tile loop, operand views and roles are those of gemm_bf16.cu, with eight epilogue warps.
// Figures: ops/muon_native.py.  Per item of K = 1280 (5 x 5120 x 1280): 10 240 clocks of MMAs, 460 a K block for the loads of 256
// rows, about 4 000 waiting for a product that is not complete yet.
#include "common.cuh"

namespace bones {

constexpr int NT = 256, NK = 64, NSTAGES = 6;       // pair tile (each CTA: 128 rows of A, 128 of B), K block, stages
constexpr uint32_t NA_BYTES = 128 * NK * 2, NB_BYTES = 128 * NK * 2, NSTAGE_BYTES = NA_BYTES + NB_BYTES;
constexpr int NS_MAX_STEPS = 8;
// Epilogue warps of a CTA: four per 32-lane quadrant, two 32-column chunks each.  With eight warps of four chunks an item's
// epilogue (residual, stores to both sides, fence and count) took 11 800 clocks against 10 240 of MMAs at K = 1280.
constexpr int NS_EW = 16;
constexpr int NS_THREADS = 96 + 32 * NS_EW;     // and the producer, MMA and drawing warps

enum NsOp : int { NS_G = 0, NS_B = 1, NS_X = 2 };

struct NsMaps {
  CUtensorMap xk[3], xm[3];   // X buffers (input, two work buffers): contraction along the columns / along the rows
  CUtensorMap g, b;
};
struct NsParams {
  int n, r, c, s, steps, tall;
  int tri, rect;              // tiles of a symmetric product, of X'
  int lag_b, lag_x;           // B and X' of a (step, matrix) slot are listed so many slots after its G
  int total;
  float ca[NS_MAX_STEPS], cb[NS_MAX_STEPS], cc[NS_MAX_STEPS];
  __nv_bfloat16* x[3];
  __nv_bfloat16 *g, *b;
  int* items;                 // draws; zero at launch
  int* done;                  // [steps * n][3] finished epilogue warps (2 NS_EW a tile); zero at launch
  int* err;
};
struct NsItem {
  int op, slot, step, m, mb, nb;
};

// Walks the list: slot k's G, then B of slot k - lag_b, then X' of slot k - lag_x.  `k`: a lower bound kept by the caller.
__device__ __forceinline__ NsItem ns_item(const NsParams& p, int w, int& k) {
  const int S = p.steps * p.n;
  auto before = [&](int q) { return p.tri * (min(q, S) + min(max(q - p.lag_b, 0), S)) + p.rect * min(max(q - p.lag_x, 0), S); };
  while (w >= before(k + 1)) ++k;
  int t = w - before(k);
  NsItem it;
  it.op = NS_G;
  it.slot = k;
  bool placed = false;
  if (k < S) {
    if (t < p.tri) placed = true;
    else t -= p.tri;
  }
  if (!placed && k >= p.lag_b && k - p.lag_b < S) {
    if (t < p.tri) { it.op = NS_B; it.slot = k - p.lag_b; placed = true; }
    else t -= p.tri;
  }
  if (!placed) { it.op = NS_X; it.slot = k - p.lag_x; }
  it.step = it.slot / p.n;
  it.m = it.slot - it.step * p.n;
  if (it.op == NS_X) {
    const int tn = (p.c + NT - 1) / NT;
    it.mb = t / tn;
    it.nb = t - it.mb * tn;
  } else {                                     // lower triangle: row block mb has the column blocks 0 .. mb
    int q = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((q + 1) * (q + 2) / 2 <= t) ++q;
    while (q * (q + 1) / 2 > t) --q;
    it.mb = q;
    it.nb = t - q * (q + 1) / 2;
  }
  return it;
}
__device__ __forceinline__ int ns_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Pair helpers: this CTA's rank, arrival on the barrier at the same offset in another CTA of the cluster (releasing at cluster
// scope), the wait that goes with it, TMA loads and MMAs of a pair, a commit that arrives in both CTAs.
__device__ __forceinline__ uint32_t ns_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void ns_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t ns_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void ns_arrive(uint32_t bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(ns_map(bar, rank)) : "memory");
}
// The arrival that publishes a ring slot: releases at cluster scope.  Not for the per-stage arrivals, which hand over no data of
// this thread: there the release cost as much as a K block's MMAs (the whole iteration took twice as long).
__device__ __forceinline__ void ns_arrive_release(uint32_t bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(ns_map(bar, rank)) : "memory");
}
__device__ __forceinline__ bool ns_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kWaitHintNs)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool ns_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err, int code) {
  const long long t0 = clock64();
  while (!ns_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitLimitCycles) {
      *abort_flag = 1;
      atomicCAS(err, 0, code);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void ns_tma(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar & 0xFEFFFFFFu), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void ns_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ns_commit(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask)
               : "memory");
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
// The counter of the product that this item reads, and what it says when that product is complete.
__device__ __forceinline__ const int* ns_inputs(const NsParams& p, const NsItem& it, int& need) {
  if (it.op == NS_G) {
    need = p.rect * 2 * NS_EW;
    return it.step > 0 ? p.done + ((it.slot - p.n) * 3 + NS_X) : nullptr;
  }
  need = p.tri * 2 * NS_EW;
  return p.done + (it.slot * 3 + it.op - 1);
}
__device__ __forceinline__ bool ns_inputs_ready(const NsParams& p, int w, int k, int lane) {
  const NsItem it = ns_item(p, w, k);
  int need, ok = 1;
  const int* flag = ns_inputs(p, it, need);
  if (flag && lane == 0) ok = ns_acquire(flag) >= need;
  __syncwarp();
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
// Lane 0 waits until the product this item reads is complete (bounded); the warp leaves together.
__device__ __forceinline__ bool ns_wait_inputs(const NsParams& p, const NsItem& it, volatile int* abort_flag, int lane) {
  int need, ok = 1;
  const int* flag = ns_inputs(p, it, need);
  if (flag && lane == 0) {
    const long long t0 = clock64();
    while (ns_acquire(flag) < need) {
      if (*abort_flag || clock64() - t0 > kWaitLimitCycles) {
        *abort_flag = 1;
        atomicCAS(p.err, 0, ERR_WAIT_AUX);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NS_THREADS, 1) newton_schulz_kernel(const __grid_constant__ NsMaps maps, const __grid_constant__ NsParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  constexpr uint32_t kBars = NSTAGES * NSTAGE_BYTES;
  const uint32_t bars = base + kBars;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (NSTAGES + s); };
  auto tfull = [&](int a) { return bars + 8u * (2 * NSTAGES + a); };
  auto tempty = [&](int a) { return bars + 8u * (2 * NSTAGES + 2 + a); };
  const uint32_t ring_bars = bars + 8u * (2 * NSTAGES + 4);
  volatile int* ring_slots = reinterpret_cast<volatile int*>(gen + kBars + 8 * (2 * NSTAGES + 8));
  const uint32_t ring_free = bars + 8u * (2 * NSTAGES + 10);
  const uint32_t want = bars + 8u * (2 * NSTAGES + 14);
  const uint32_t tmem_slot = bars + 8u * (2 * NSTAGES + 15);
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(gen + kBars + 8 * (2 * NSTAGES + 15));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + kBars + 8 * (2 * NSTAGES + 15) + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ns_rank();
  const bool leader = rank == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGES; ++s) {
      mbar_init(full(s), 2);                   // leader: its own arrive.expect_tx and the peer's arrive
      mbar_init(empty(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull(a), 1);
      mbar_init(tempty(a), 2 * NS_EW);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(ring_bars + 8u * s, 1);
      mbar_init(ring_free + 8u * s, 2 * NS_EW + 3);       // leader: every epilogue warp, its MMA warp, both producers
    }
    mbar_init(want, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  ns_cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  ns_cluster_sync();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_g;
  // what every consumer of the ring does: lane 0 waits for slot i, everybody reads it
  auto take = [&](int i) {
    int w = -1;
    if (ns_wait(ring_bars + 8u * (uint32_t)(i & 3), (uint32_t)((i >> 2) & 1), abort_flag, p.err, ERR_WAIT_AUX)) w = ring_slots[i & 3];
    w = warp_uniform(w);
    if (lane == 0) ns_arrive(ring_free + 8u * (uint32_t)(i & 3), 0);
    return w;
  };
  // operand layouts by product (0: contraction contiguous, 1: rows contiguous) and contraction length
  auto a_major = [&](int op) { return op == NS_G && p.tall ? 1 : 0; };
  auto b_major = [&](int op) { return (op == NS_G && p.tall) || (op == NS_X && !p.tall) ? 1 : 0; };
  auto k_blocks = [&](int op) { return ((op == NS_G ? (p.tall ? p.r : p.c) : p.s) + NK - 1) / NK; };

  if (warp == 2 + NS_EW) {
    // The leader's last warp draws items and hands them to both CTAs' roles through a four-slot ring in each CTA's shared memory:
    // the next one when the producer begins an item (a draw, a round trip to L2 and a release, cost the producer warp itself
    // 2 500 clocks; drawing as far ahead as the ring allows parks items behind long ones: 639 -> 813 us).
    if (leader) {
      bool dead = false;
      for (int i = 0;; ++i) {
        if (i >= 4 && !dead) dead = !ns_wait(ring_free + 8u * (uint32_t)(i & 3), (uint32_t)(((i >> 2) - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        if (i >= 1 && !dead) dead = !mbar_wait(want, (uint32_t)((i - 1) & 1), abort_flag, p.err, ERR_WAIT_AUX);
        int w = -1;
        if (lane == 0 && !dead) {
          const int d = atomicAdd(p.items, 1);
          w = d < p.total ? d : -1;
          const uint32_t slot = smem_u32((const void*)(ring_slots + (i & 3)));
#pragma unroll
          for (uint32_t r = 0; r < 2; ++r) {
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ns_map(slot, r)), "r"(w) : "memory");
            ns_arrive_release(ring_bars + 8u * (uint32_t)(i & 3), r);
          }
        }
        if (warp_uniform(w) < 0) break;
      }
    }
  } else if (warp == 0) {
    int stage = 0, it = 0, k = 0;
    uint32_t phase = 0;
    bool dead = false;
    int w = take(0), w_next = -1;
    bool ready = false;
    for (; w >= 0; ++it, w = w_next) {
      if (leader && lane == 0) mbar_arrive(want);
      NsItem im = ns_item(p, w, k);
      // (the shuffles tell the compiler that what the TMA instructions take is warp-uniform)
      im.op = warp_uniform(im.op); im.m = warp_uniform(im.m); im.mb = warp_uniform(im.mb); im.nb = warp_uniform(im.nb);
      im.step = warp_uniform(im.step);
      if (!ready && !dead) dead = !ns_wait_inputs(p, im, abort_flag, lane);
      fence_proxy_async_all();                 // what other SMs wrote with ordinary stores is read by TMA below
      const int cur = im.step == 0 ? 0 : 1 + ((im.step - 1) & 1);
      const CUtensorMap *ma, *mb;
      if (im.op == NS_G) ma = mb = p.tall ? &maps.xm[cur] : &maps.xk[cur];
      else if (im.op == NS_B) ma = mb = &maps.g;
      else { ma = p.tall ? &maps.xk[cur] : &maps.b; mb = p.tall ? &maps.b : &maps.xm[cur]; }
      const int am = a_major(im.op), bm = b_major(im.op), KB = k_blocks(im.op);
      const int m0 = im.mb * NT + (int)rank * 128, n0 = im.nb * NT + (int)rank * 128;
      for (int kb = 0; kb < KB; ++kb) {
        if (kb == KB / 2) w_next = dead ? -1 : take(it + 1);
        // the next item's inputs are looked at before the last loads of this one are issued
        if (kb == KB - 1) ready = w_next >= 0 && !dead && ns_inputs_ready(p, w_next, k, lane);
        if (!dead) dead = !mbar_wait(empty(stage), phase ^ 1u, abort_flag, p.err, ERR_WAIT_EMPTY);
        const uint32_t sa = base + stage * NSTAGE_BYTES, sb = sa + NA_BYTES;
        if (elect_one() && !dead) {
          if (leader) mbar_arrive_expect_tx(full(stage), 2 * NSTAGE_BYTES);
          if (am == 0) {
            ns_tma(sa, ma, full(stage), kb * NK, m0, im.m);
          } else {
            ns_tma(sa, ma, full(stage), m0, kb * NK, im.m);
            ns_tma(sa + NK * 128, ma, full(stage), m0 + 64, kb * NK, im.m);
          }
          if (bm == 0) {
            ns_tma(sb, mb, full(stage), kb * NK, n0, im.m);
          } else {
            ns_tma(sb, mb, full(stage), n0, kb * NK, im.m);
            ns_tma(sb + NK * 128, mb, full(stage), n0 + 64, kb * NK, im.m);
          }
          if (!leader) ns_arrive(full(stage), 0);
        }
        if (++stage == NSTAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (leader) {
      int stage = 0, it = 0, k = 0;
      uint32_t phase = 0;
      bool dead = false;
      const uint64_t ad[2] = {umma_smem_desc(base, 0, 1024, kLayoutSw128), umma_smem_desc(base, NK * 128, 1024, kLayoutSw128)};
      const uint64_t bd[2] = {umma_smem_desc(base + NA_BYTES, 0, 1024, kLayoutSw128), umma_smem_desc(base + NA_BYTES, NK * 128, 1024, kLayoutSw128)};
      for (;; ++it) {
        const int w = dead ? -1 : take(it);
        if (w < 0) break;
        const NsItem im = ns_item(p, w, k);
        const int op = warp_uniform(im.op), acc = it & 1;
        const int am = a_major(op), bm = b_major(op), KB = k_blocks(op);
        if (it >= 2 && !dead) dead = !ns_wait(tempty(acc), (uint32_t)(((it - 2) >> 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after();
        const uint32_t idesc = umma_idesc_f16(NT, NT, 1, (uint32_t)am, (uint32_t)bm);
        const uint32_t a_step = am ? (16 * 128) >> 4 : 32 >> 4, b_step = bm ? (16 * 128) >> 4 : 32 >> 4;
        const uint64_t ad0 = am ? ad[1] : ad[0], bd0 = bm ? bd[1] : bd[0];
        for (int kb = 0; kb < KB; ++kb) {
          if (!dead) dead = !mbar_wait(full(stage), phase, abort_flag, p.err, ERR_WAIT_FULL);
          tc_fence_after();
          const uint64_t soff = (uint64_t)(stage * (NSTAGE_BYTES >> 4));
          if (elect_one() && !dead) {
#pragma unroll
            for (int q = 0; q < NK / 16; ++q)
              ns_umma(tmem + acc * NT, ad0 + soff + (uint64_t)(q * a_step), bd0 + soff + (uint64_t)(q * b_step), idesc, (kb | q) ? 1u : 0u);
            ns_commit(empty(stage));
            if (kb == KB - 1) ns_commit(tfull(acc));
          }
          if (++stage == NSTAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2;
    int it = 0, k = 0;
    bool ok = true;
    for (;; ++it) {
      const int w = ok ? take(it) : -1;
      if (w < 0) break;
      const NsItem im = ns_item(p, w, k);
      const int acc = it & 1, cur = im.step == 0 ? 0 : 1 + ((im.step - 1) & 1), nxt = 1 + (im.step & 1);
      const bool sym = im.op != NS_X, with_r = im.op != NS_G;
      const int M = sym ? p.s : p.r, N = sym ? p.s : p.c, ld = N;
      const long long mat = (long long)im.m * M * N;
      __nv_bfloat16* D = (im.op == NS_G ? p.g : im.op == NS_B ? p.b : p.x[nxt]) + mat;
      const __nv_bfloat16* R = (im.op == NS_B ? p.g : p.x[cur]) + mat;
      const float alpha = im.op == NS_B ? p.cc[im.step] : 1.0f, beta = im.op == NS_B ? p.cb[im.step] : p.ca[im.step];
      const int row = im.mb * NT + (int)rank * 128 + q * 32 + lane, c0 = im.nb * NT + part * 64;
      const bool row_ok = row < M, mirror = sym && im.nb < im.mb;      // tiles below the diagonal are written to both sides
      uint4 rp[2][4];
      if (with_r) {
        // R was written by other SMs: this warp's own look at the counter orders its loads behind those stores
        if (!ns_wait_inputs(p, im, abort_flag, lane)) { ok = false; break; }
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 2; ++j)
            if (c0 + j * 32 + 32 <= N) {
              const __nv_bfloat16* src = R + (long long)row * ld + c0 + j * 32;
              ld_global_v8(src, rp[j][0], rp[j][1]);
              ld_global_v8(src + 16, rp[j][2], rp[j][3]);
            }
        }
      }
      const bool got = mbar_wait(tfull(acc), (uint32_t)((it >> 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
      tc_fence_after();
      {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint32_t v[32];
          __syncwarp();
          BONES_TMEM_LD32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * NT + part * 64 + j * 32), v);
          tmem_ld_wait();
          if (j == 1) {                        // the accumulator is free from here on
            tc_fence_before();
            __syncwarp();
            if (lane == 0) ns_arrive(tempty(acc), 0);
          }
          const int col0 = c0 + j * 32;
          if (!row_ok || col0 >= N) continue;
          __nv_bfloat16* dst = D + (long long)row * ld + col0;
          if (col0 + 32 <= N) {
            uint4 u[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint32_t o[4];
              const uint32_t rr[4] = {rp[j][g].x, rp[j][g].y, rp[j][g].z, rp[j][g].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float a0 = alpha * __uint_as_float(v[g * 8 + 2 * e]), a1 = alpha * __uint_as_float(v[g * 8 + 2 * e + 1]);
                if (with_r) {
                  a0 = fmaf(beta, __uint_as_float(rr[e] << 16), a0);
                  a1 = fmaf(beta, __uint_as_float(rr[e] & 0xffff0000u), a1);
                }
                o[e] = pack_bf16(a0, a1);
              }
              u[g] = make_uint4(o[0], o[1], o[2], o[3]);
            }
            st_global_v8(dst, u[0], u[1]);
            st_global_v8(dst + 16, u[2], u[3]);
            if (mirror) {
              // lanes are consecutive rows, so each of these stores is 64 contiguous bytes of a mirrored row
              unsigned short* md = reinterpret_cast<unsigned short*>(D + (long long)col0 * ld + row);
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const uint32_t o[4] = {u[g].x, u[g].y, u[g].z, u[g].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  md[(long long)(g * 8 + 2 * e) * ld] = (unsigned short)(o[e] & 0xffffu);
                  md[(long long)(g * 8 + 2 * e + 1) * ld] = (unsigned short)(o[e] >> 16);
                }
              }
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (col0 + e < N) {
                float a = alpha * __uint_as_float(v[e]);
                if (with_r) a = fmaf(beta, __bfloat162float(R[(long long)row * ld + col0 + e]), a);
                const __nv_bfloat16 h = __float2bfloat16(a);
                dst[e] = h;
                if (mirror) D[(long long)(col0 + e) * ld + row] = h;
              }
            }
          }
        }
      }
      // this warp's stores before its count: they are ordered by the warp barrier and lane 0's fence, and before the TMA reads of
      // whoever waits for the count by that reader's own proxy fence (fences in every lane took 6 300 clocks of an item)
      __syncwarp();
      if (lane == 0) {
        __threadfence();
        atomicAdd(p.done + im.slot * 3 + im.op, 1);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  ns_cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

static int ns_tmap(CUtensorMap* out, const void* ptr, int rows, int cols, int n, int box_rows) {
  uint64_t dims[3] = {(uint64_t)cols, (uint64_t)rows, (uint64_t)n};
  uint64_t strides[2] = {(uint64_t)cols * 2, (uint64_t)cols * 2 * (uint64_t)rows};
  uint32_t box[3] = {64, (uint32_t)box_rows, 1};
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace bones

extern "C" {
using namespace bones;

// x0 [n, r, c] bf16 (left as it is); x1, x2: work buffers of the same size (the result is in x1 after an odd number of steps,
// in x2 after an even one); g, b: [n, s, s]; coeffs: host array of 3 * steps floats; scratch: 1 + 3 * steps * n ints, zeroed here.
// r and c multiples of 16, every pointer 32-byte aligned.
int bones_newton_schulz(const void* x0, void* x1, void* x2, void* g, void* b, int n, int r, int c, int steps, const float* coeffs, int* scratch,
                        void* stream) {
  if (n < 1 || r < 1 || c < 1 || steps < 1 || steps > NS_MAX_STEPS || (r % 16) || (c % 16)) return -2;
  if (((uintptr_t)x0 | (uintptr_t)x1 | (uintptr_t)x2 | (uintptr_t)g | (uintptr_t)b) & 31) return -2;
  NsParams p;
  p.n = n; p.r = r; p.c = c; p.steps = steps;
  p.tall = r > c;
  p.s = r > c ? c : r;
  const int rb = (p.s + NT - 1) / NT;
  p.tri = rb * (rb + 1) / 2;
  p.rect = ((r + NT - 1) / NT) * ((c + NT - 1) / NT);
  // Distances in the list, in slots: long enough that a product is complete when its reader's turn comes.  In units of a tile with
  // a contraction of s, a tile takes its contraction and about one more until its result can be read, and a slot's tiles take
  // `slot`.  X' must also be complete when the matrix's next G comes, n slots after the last one, so with few matrices the lags
  // are what fits (5 matrices of 5120 x 1280: 2 and 3 slots 673 us, 3 and 4 slots 797, 1 and 2 slots 715, none 1697).
  int dev = 0, sms = 0;
  BONES_CHECK(cudaGetDevice(&dev));
  BONES_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const float kg = (float)(p.tall ? r : c) / (float)p.s, slot = ((float)p.tri * (kg + 1.0f) + (float)p.rect) / (float)(sms / 2);
  auto up = [](float v) { const int i = (int)v; return i + ((float)i < v ? 1 : 0); };
  p.lag_b = up((kg + 1.0f) / slot);
  p.lag_x = p.lag_b + up(2.0f / slot);
  if (p.lag_x > n - 1 - up(2.0f / slot)) {
    p.lag_x = n > 3 ? n - 2 : n - 1;
    p.lag_b = p.lag_x > 1 ? p.lag_x - 1 : p.lag_x;
  }
  const long long total = (long long)steps * n * (2 * p.tri + p.rect);
  if (total > (1LL << 30)) return -2;
  p.total = (int)total;
  for (int i = 0; i < steps; ++i) { p.ca[i] = coeffs[3 * i]; p.cb[i] = coeffs[3 * i + 1]; p.cc[i] = coeffs[3 * i + 2]; }
  p.x[0] = (__nv_bfloat16*)x0; p.x[1] = (__nv_bfloat16*)x1; p.x[2] = (__nv_bfloat16*)x2;
  p.g = (__nv_bfloat16*)g; p.b = (__nv_bfloat16*)b;
  p.items = scratch;
  p.done = scratch + 1;
  p.err = error_word();
  NsMaps maps;
  for (int i = 0; i < 3; ++i) {
    int rc = ns_tmap(&maps.xk[i], p.x[i], r, c, n, 128);
    if (rc) return rc;
    rc = ns_tmap(&maps.xm[i], p.x[i], r, c, n, 64);
    if (rc) return rc;
  }
  int rc = ns_tmap(&maps.g, g, p.s, p.s, n, 128);
  if (rc) return rc;
  rc = ns_tmap(&maps.b, b, p.s, p.s, n, 128);
  if (rc) return rc;
  constexpr size_t smem = (size_t)NSTAGES * NSTAGE_BYTES + 8 * (2 * NSTAGES + 15) + 16 + 1024;
  static OncePerDevice limit;
  BONES_ONCE(limit, {
    BONES_CHECK(cudaFuncSetAttribute(newton_schulz_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  });
  BONES_CHECK(cudaMemsetAsync(scratch, 0, sizeof(int) * (1 + 3 * (size_t)steps * n), (cudaStream_t)stream));
  const int pairs = p.total < sms / 2 ? p.total : sms / 2;
  newton_schulz_kernel<<<2 * pairs, NS_THREADS, smem, (cudaStream_t)stream>>>(maps, p);
  return (int)cudaGetLastError();
}
}  // extern "C"
