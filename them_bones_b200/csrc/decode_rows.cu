// Projections of one decode step of up to 64 sequences: the sequences are the rows of the MMA, the weights its narrow columns.
//
//   out[t, n] = epilogue( r_t * sum_k X[t, k] W[n, k] )          X bf16 [b, K], W bf16 [N, K], b <= 64
//
// Every weight is read once from HBM (10 to 13 MB a projection, 1.5 to 2 us at the copy rate), so the work goes to as many SMs as
// there are, and what counts beside the bytes is the chain from the previous kernel's end: one read of X, one accumulator, one store.
//   * A CTA owns `nt` output columns (16 to 64) of all sequences over the whole contraction: no partial sums are exchanged.  X is
//     read by every CTA from L2 (160 KB at 64 sequences and K = 1280), which costs less than the exchange it replaces: with
//     128-column tiles and the contraction split over a cluster (decode_gemm.cu) the accumulator was complete 4 us after the wait and
//     the exchange took another 1.3 to 2.9 us.  The CTAs walk the contraction from different places, so they do not ask the same
//     lines of L2 at the same time.
//   * Long contractions (c_proj, K = 4 C) are still shared by a cluster, each CTA over its K range; the partial sums of 64 x nt are
//     small (10 KB a CTA at nt = 40), and a CTA finishes 64 / S sequences, adding in the order of the ranks.
//   * Weights depend on nothing in the step: their producer fills its ring before the wait for the previous kernel, and the idle
//     epilogue warps bring the next projection's weights to L2.  X has a ring and a producer of its own behind the wait.  Both rings
//     are deep: 48 KB of X in flight (two CTAs on an SM) fed a CTA at 47 KB/us, and a step took 700 us instead of 640.
//   * M = 64: a sequence is a TMEM lane (16 of each warp's 32), a thread owns consecutive columns of one sequence: 16-byte
//     loads of the residual and stores, squares' sums without shuffles.
//   * With many tiles the CTAs are persistent with two accumulators, and the rings run on across tiles.
// 20 layers, 1280 wide, head of 65536, us a step at position 64, with decode_gemm.cu's kernel for all projections and with this one: batch 64
// 810 -> 640, 40 804 -> 605, 16 603 -> 545, 4 562 -> 520 (two runs within 1 %).  A layer takes 33 us at batch 64: qkv 6.2, attention 10 (21 MB of
// keys and values, 3.2 us at the copy rate: its chain of waits, rounds of keys and sums is what takes the time there), out 4.2, c_fc 5.7, c_proj
// 7.3; of each about 1.1 us lie between one kernel's last store and the next one's start, 0.8 us until the first rows of X arrive, and the
// MMAs of K = 1280 take 1.7 us at least (35 clocks each, 64 x nt x 16).  All CTAs together read X 13 to 20 MB worth from L2, more than the
// weights of qkv and c_proj.
#include "decode_common.cuh"

namespace bones {

struct DecRowsParams {
  int N, b, KS;               // KS: K / 128
  int nt, tiles;              // output columns of a tile, tiles
  int xs, ws, rb;             // ring slots of X and W, rows of an X slot (b rounded up to 8)
  const float* ssq_in;        // [n_ssq, b] partial sums of squares of X's rows (null: r = 1)
  int n_ssq;
  float inv_k;                // 1 / K
  const __nv_bfloat16* res;   // [b, N]
  const __nv_bfloat16* x0;    // [b, N] or null
  const float *mix_a, *mix_b;
  float* ssq_out;             // [tiles, b] or null
  __nv_bfloat16* out;         // [b, N]
  float cap;
  int* err;
  const uint8_t* next_w;      // the weights that the step reads after these, to bring to L2 (null: none)
  long long next_bytes;
};

constexpr int DR_EW = 8;                              // epilogue warps: two per 32-lane quadrant of TMEM
constexpr int DR_THREADS = 32 * (3 + DR_EW);          // X loads, MMAs, W loads, epilogue
constexpr int DR_MAX_SLOTS = 24;
constexpr uint32_t DR_BARS = 8 * (4 * DR_MAX_SLOTS + 4) + 16;
constexpr int DR_SUMS = 4 * 64 * 4;                   // squares' sums, four parts

#define BONES_TMEM_LD8(taddr, r)                                                                                            \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"                              \
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])             \
               : "r"(taddr)                                                                                                 \
               : "memory")

constexpr int DR_AHEAD = 4096;
__device__ __forceinline__ void l2_prefetch_bulk(const void* a, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint4 dr_ld16(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint2 dr_ld8(const __nv_bfloat16* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void dr_bf16x8(const uint4& u, float* f) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 g = unpack_bf16(w[i]);
    f[2 * i] = g.x;
    f[2 * i + 1] = g.y;
  }
}

// shared memory: [X ring][W ring][partial sums of the cluster][barriers][squares' sums]; a slot of X is 128 of K of `rb` rows, and
// the MMA reads 64 rows from it: behind `rb` they are whatever follows in shared memory, and only rows without a sequence see them
template <int EPI, bool SPLIT>
__global__ void __launch_bounds__(DR_THREADS)
decode_rows_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const DecRowsParams p) {
  extern __shared__ uint8_t dr_raw[];
  const uint32_t raw = smem_u32(dr_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* gen = dr_raw + (base - raw);
  const uint32_t x_slot = (uint32_t)p.rb * 256u, w_slot = (uint32_t)p.nt * 256u;
  const uint32_t w_base = base + (uint32_t)p.xs * x_slot, red_off = (uint32_t)p.xs * x_slot + (uint32_t)p.ws * w_slot;
  const uint32_t red_bytes = SPLIT ? 64u * (uint32_t)(p.nt + 4) * 4u : 0u, bars = base + red_off + red_bytes;
  auto xfull = [&](int s) { return bars + 8u * s; };
  auto xempty = [&](int s) { return bars + 8u * (DR_MAX_SLOTS + s); };
  auto wfull = [&](int s) { return bars + 8u * (2 * DR_MAX_SLOTS + s); };
  auto wempty = [&](int s) { return bars + 8u * (3 * DR_MAX_SLOTS + s); };
  auto tfull = [&](int a) { return bars + 8u * (4 * DR_MAX_SLOTS + a); };
  auto tempty = [&](int a) { return bars + 8u * (4 * DR_MAX_SLOTS + 2 + a); };
  const uint32_t tmem_slot = bars + 8u * (4 * DR_MAX_SLOTS + 4);
  uint8_t* bars_g = gen + red_off + red_bytes;
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(bars_g + 8 * (4 * DR_MAX_SLOTS + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars_g + 8 * (4 * DR_MAX_SLOTS + 4) + 8);
  float* wsq = reinterpret_cast<float*>(bars_g + DR_BARS);                // [4][64]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = SPLIT ? (int)cluster_rank() : 0, S = SPLIT ? (int)cluster_size() : 1;
  const int first = blockIdx.x / S, step = gridDim.x / S;
  const int k0 = p.KS * rank / S, k1 = p.KS * (rank + 1) / S;
  // The CTAs begin at different places of the contraction and wrap around: they all read the same X, and in step they would all ask
  // the same few lines of L2 at a time.  A column's place follows its CTA, so where CTAs walk several tiles (the head) the order of
  // its sum, and with it the last bits, depends on the number of SMs; on one device every call gives the same bits.
  const int turn = first % (k1 - k0);
  auto at_k = [&](int k) { return k + turn < k1 ? k + turn : k + turn - (k1 - k0); };
  const uint32_t tcols = p.nt > 32 ? 64u : 32u;                          // columns between the two accumulators

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.xs; ++s) {
      mbar_init(xfull(s), 1);
      mbar_init(xempty(s), 1);
    }
    for (int s = 0; s < p.ws; ++s) {
      mbar_init(wfull(s), 1);
      mbar_init(wempty(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull(a), 1);
      mbar_init(tempty(a), DR_EW);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  pdl_launch();
  if (SPLIT) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // waited for before the exchange

  if (warp == 2) {
    int s = 0;
    uint32_t ph = 1;                                         // the first pass over the ring finds it empty: a wait takes 150 clocks even so
    bool dead = false, again = false;
    for (int tile = first; tile < p.tiles; tile += step)
      for (int k = k0; k < k1; ++k) {
        if (again && !dead) dead = !mbar_wait(wempty(s), ph, abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(wfull(s), w_slot);
          tma_load_3d(w_base + (uint32_t)s * w_slot, &tm_w, wfull(s), 0, tile * p.nt, at_k(k) * 2);
        }
        if (++s == p.ws) { s = 0; ph ^= 1u; again = true; }
      }
    __syncwarp();
  } else if (warp == 0) {
    pdl_wait();
    int s = 0;
    uint32_t ph = 1;
    bool dead = false, again = false;
    for (int tile = first; tile < p.tiles; tile += step)
      for (int k = k0; k < k1; ++k) {
        if (again && !dead) dead = !mbar_wait(xempty(s), ph, abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(xfull(s), x_slot);
          tma_load_3d(base + (uint32_t)s * x_slot, &tm_x, xfull(s), 0, 0, at_k(k) * 2);
        }
        if (++s == p.xs) { s = 0; ph ^= 1u; again = true; }
      }
    __syncwarp();
  } else if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * tcols);
    tmem_relinquish();
    tc_fence_before();
    asm volatile("bar.sync 2, 288;" ::: "memory");           // the epilogue warps read the address behind it
    tc_fence_after();
    // everything an MMA takes is warp-uniform, and known to be: an MMA of this size takes 35 clocks where its operands come from
    // uniform registers and 80 where each is moved there first, and the chain of K / 16 of them is what a tile waits for
    constexpr uint32_t kHi = umma_desc_hi(1024, kLayoutSw128);
    const uint32_t tmem = (uint32_t)warp_uniform((int)*tmem_slot_g), idesc = (uint32_t)warp_uniform((int)umma_idesc_f16(64, (uint32_t)p.nt, 1, 0, 0));
    const uint32_t x_lo = (uint32_t)warp_uniform((int)umma_desc_lo(base, 0)), w_lo = (uint32_t)warp_uniform((int)umma_desc_lo(w_base, 0));
    const uint32_t x_step = (uint32_t)p.rb * 16u, w_step = (uint32_t)p.nt * 16u;          // of a slot, in 16-byte units; half of it a block of 64
    const int stages = (k1 - k0) * ((p.tiles - first + step - 1) / step);
    const bool refill_x = stages > p.xs, refill_w = stages > p.ws;
    int xsl = 0, wsl = 0, it = 0;
    uint32_t xph = 0, wph = 0;
    bool dead = false, ready = false;
    // Two waits are as long as a stage's eight MMAs: whether the next stage is there is asked before this one's are issued (`mbar_test`).
    for (int tile = first; tile < p.tiles; tile += step, ++it) {
      const int a = it & 1;
      if (it > 1 && !dead) dead = !mbar_wait(tempty(a), ((uint32_t)(it >> 1) & 1u) ^ 1u, abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
      tc_fence_after();
      const uint32_t d = tmem + (uint32_t)a * tcols;
      for (int k = k0; k < k1; ++k) {
        if (!ready) {
          if (!dead) dead = !mbar_wait(wfull(wsl), wph, abort_flag, p.err, ERR_WAIT_FULL);
          if (!dead) dead = !mbar_wait(xfull(xsl), xph, abort_flag, p.err, ERR_WAIT_FULL);
        }
        tc_fence_after();
        const int xn = xsl + 1 == p.xs ? 0 : xsl + 1, wn = wsl + 1 == p.ws ? 0 : wsl + 1;
        const uint32_t xpn = xn ? xph : xph ^ 1u, wpn = wn ? wph : wph ^ 1u;
        const uint32_t w_there = mbar_test(wfull(wn), wpn), x_there = mbar_test(xfull(xn), xpn);
        const uint32_t xa = x_lo + (uint32_t)xsl * x_step, wa = w_lo + (uint32_t)wsl * w_step, xb = xa + x_step / 2, wb = wa + w_step / 2;
        if (elect_one() && !dead) {                          // two swizzled blocks of 64, four steps of 16 each
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lh(d, xa + (uint32_t)(2 * j), kHi, wa + (uint32_t)(2 * j), kHi, idesc, (k > k0 || j > 0) ? 1u : 0u);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lh(d, xb + (uint32_t)(2 * j), kHi, wb + (uint32_t)(2 * j), kHi, idesc, 1u);
          if (refill_x) tc_commit(xempty(xsl));
          if (refill_w) tc_commit(wempty(wsl));
          if (k == k1 - 1) tc_commit(tfull(a));
        }
        ready = __all_sync(0xffffffffu, (w_there & x_there) != 0u);
        xsl = xn; xph = xpn;
        wsl = wn; wph = wpn;
      }
    }
    __syncwarp();
  } else {
    asm volatile("bar.sync 2, 288;" ::: "memory");
    tc_fence_after();
    const uint32_t tmem = *tmem_slot_g;
    const int q = warp & 3, half = (warp - 3) >> 2, t = q * 16 + lane, e = threadIdx.x - 96;
    const bool live = lane < 16 && t < p.b;
    const int chunks = p.nt >> 3;
    for (long long o = ((long long)e * gridDim.x + blockIdx.x) * DR_AHEAD; o < p.next_bytes; o += 32ll * DR_EW * gridDim.x * DR_AHEAD)
      l2_prefetch_bulk(p.next_w + o, (uint32_t)min((long long)DR_AHEAD, p.next_bytes - o));
    pdl_wait();
    float ma = 0.f, mb = 0.f;
    if (EPI == DEC_RES && p.x0) { ma = *p.mix_a; mb = *p.mix_b; }
    const long long row = (long long)t * p.N;
    // of the cluster's sequences this CTA finishes `mine`, four columns a thread
    const int own = 64 / S, groups = p.nt >> 2, mine = max(0, min(own, p.b - rank * own));
    // a thread's first residual (and second, without a split), requested before the accumulator is complete
    uint4 rs0 = make_uint4(0u, 0u, 0u, 0u), rs1 = rs0, zs0 = rs0, zs1 = rs0;
    uint2 rq = make_uint2(0u, 0u), zq = rq;
    if (EPI == DEC_RES && !SPLIT && live && first < p.tiles) {
      const long long at = row + first * p.nt + half * 8;
      if (half < chunks) {
        rs0 = dr_ld16(p.res + at);
        if (p.x0) zs0 = dr_ld16(p.x0 + at);
      }
      if (half + 2 < chunks) {
        rs1 = dr_ld16(p.res + at + 16);
        if (p.x0) zs1 = dr_ld16(p.x0 + at + 16);
      }
    }
    auto split_at = [&](int item) { return (long long)(rank * own + item / groups) * p.N + first * p.nt + (item % groups) * 4; };
    if (EPI == DEC_RES && SPLIT && e < mine * groups) {
      rq = dr_ld8(p.res + split_at(e));
      if (p.x0) zq = dr_ld8(p.x0 + split_at(e));
    }
    if (p.ssq_in) {
      const int tt = e & 63;
      float ss = 0.f;
      if (tt < p.b) {
#pragma unroll 5
        for (int j = e >> 6; j < p.n_ssq; j += 4) ss += p.ssq_in[j * p.b + tt];
      }
      wsq[e] = ss;
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    auto factor = [&](int tt) {
      return p.ssq_in ? rsqrtf(((wsq[tt] + wsq[64 + tt]) + (wsq[128 + tt] + wsq[192 + tt])) * p.inv_k + 1.1920928955078125e-07f) : 1.0f;
    };
    auto finish = [&](float v, float r, float x, float z) {
      float y = v * r;
      if (EPI == DEC_RELU2) {
        y = fmaxf(y, 0.f);
        y *= y;
      } else if (EPI == DEC_SOFTCAP) {
        float th;
        asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(y / p.cap));
        y = p.cap * th;
      } else if (EPI == DEC_RES) {
        y = __bfloat162float(__float2bfloat16(y + x));
        if (p.x0) y = ma * y + mb * z;
      }
      return y;
    };
    if (!SPLIT) {
      const float r = live ? factor(t) : 0.f;
      int it = 0;
      for (int tile = first; tile < p.tiles; tile += step, ++it) {
        const int a = it & 1;
        const bool got = mbar_wait(tfull(a), (uint32_t)(it >> 1) & 1u, abort_flag, p.err, ERR_WAIT_TMEM_FULL);
        const int upto = __all_sync(0xffffffffu, got) ? chunks : 0;      // a wait that ran out: the barriers below are still met
        tc_fence_after();
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)a * tcols;
        float ss = 0.f;
#pragma unroll 1
        for (int c = half; c < upto; c += 2) {
          uint32_t v[8];
          __syncwarp();
          BONES_TMEM_LD8(at + (uint32_t)(c * 8), v);
          tmem_ld_wait();
          if (live) {
            const long long o_at = row + tile * p.nt + c * 8;
            float x[8], z[8];
            if (EPI == DEC_RES) {
              if (c >= 4 || it > 0) {
                rs0 = dr_ld16(p.res + o_at);
                if (p.x0) zs0 = dr_ld16(p.x0 + o_at);
              }
              dr_bf16x8(rs0, x);
              dr_bf16x8(zs0, z);
              rs0 = rs1;                                   // the second chunk's, if it is the first tile
              zs0 = zs1;
            }
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              o[j] = pack_bf16(finish(__uint_as_float(v[2 * j]), r, x[2 * j], z[2 * j]), finish(__uint_as_float(v[2 * j + 1]), r, x[2 * j + 1], z[2 * j + 1]));
              const float2 f = unpack_bf16(o[j]);
              ss += f.x * f.x + f.y * f.y;
            }
            *reinterpret_cast<uint4*>(p.out + o_at) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty(a));
        if (EPI == DEC_RES && p.ssq_out) {                 // the two halves of a sequence's columns
          asm volatile("bar.sync 1, 256;" ::: "memory");   // everybody has read what stood there
          if (lane < 16) wsq[half * 64 + t] = ss;
          asm volatile("bar.sync 1, 256;" ::: "memory");
          if (e < p.b) p.ssq_out[tile * p.b + e] = wsq[e] + wsq[64 + e];
        }
      }
    } else {
      const bool got = mbar_wait(tfull(0), 0u, abort_flag, p.err, ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      cluster_wait();                                      // every CTA of the cluster runs: its shared memory may be written
      // to the sequence's owner: rows of nt + 4 floats, so that lanes write to different banks
      if (__all_sync(0xffffffffu, got)) {
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16);
        const int to = (t & 63) / own;
        const uint32_t dst = map_to_rank(base + red_off + (uint32_t)(((rank * own + ((t & 63) - to * own)) * (p.nt + 4)) * 4), (uint32_t)to);
#pragma unroll 1
        for (int c = half; c < chunks; c += 2) {
          uint32_t v[8];
          __syncwarp();
          BONES_TMEM_LD8(at + (uint32_t)(c * 8), v);
          tmem_ld_wait();
          if (live) {
            st_cluster_v4(dst + (uint32_t)(c * 32), v[0], v[1], v[2], v[3]);
            st_cluster_v4(dst + (uint32_t)(c * 32 + 16), v[4], v[5], v[6], v[7]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      cluster_barrier();                                   // every partial sum of the cluster is in its owner's memory
      float* redg = reinterpret_cast<float*>(gen + red_off);
      if (!*abort_flag) {
        for (int item = e; item < mine * groups; item += 256) {
          const int tl = item / groups, g = item - tl * groups;
          const long long o_at = split_at(item);
          float* src = redg + tl * (p.nt + 4) + g * 4;
          float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
          for (int s = 0; s < S; ++s) {
            const float4 w = *reinterpret_cast<const float4*>(src + s * own * (p.nt + 4));
            v[0] += w.x; v[1] += w.y; v[2] += w.z; v[3] += w.w;
          }
          if (EPI == DEC_RES && item != e) {
            rq = dr_ld8(p.res + o_at);
            if (p.x0) zq = dr_ld8(p.x0 + o_at);
          }
          const float r = factor(rank * own + tl);
          const float2 x0 = unpack_bf16(rq.x), x1 = unpack_bf16(rq.y), z0 = unpack_bf16(zq.x), z1 = unpack_bf16(zq.y);
          const uint32_t o0 = pack_bf16(finish(v[0], r, x0.x, z0.x), finish(v[1], r, x0.y, z0.y));
          const uint32_t o1 = pack_bf16(finish(v[2], r, x1.x, z1.x), finish(v[3], r, x1.y, z1.y));
          *reinterpret_cast<uint2*>(p.out + o_at) = make_uint2(o0, o1);
          if (EPI == DEC_RES && p.ssq_out) {               // into a place that only this thread has read
            const float2 f0 = unpack_bf16(o0), f1 = unpack_bf16(o1);
            *src = (f0.x * f0.x + f0.y * f0.y) + (f1.x * f1.x + f1.y * f1.y);
          }
        }
        if (EPI == DEC_RES && p.ssq_out) {
          asm volatile("bar.sync 1, 256;" ::: "memory");
          if (e < mine) {
            float ss = 0.f;
            for (int g = 0; g < groups; ++g) ss += redg[e * (p.nt + 4) + g * 4];
            p.ssq_out[first * p.b + rank * own + e] = ss;
          }
        }
      }
    }
  }
  if (SPLIT && warp < 3) {
    cluster_wait();
    cluster_barrier();
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);         // copies in flight land before the memory is given up
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(*tmem_slot_g, 2 * tcols);
  }
}

constexpr int DR_SMEM_MAX = 200 * 1024;
// Shared memory of a CTA: the SM's, less room for the attention's CTAs (5 KB each), so that they start while a projection runs.
constexpr int DR_SMEM_AIM = 190 * 1024;

template <int EPI, bool SPLIT>
static int launch_rows(const CUtensorMap& tw, const CUtensorMap& tx, const DecRowsParams& p, int S, int ctas, int smem, int pdl, cudaStream_t stream) {
  static OncePerDevice limit;
  BONES_ONCE(limit, {
    BONES_CHECK(cudaFuncSetAttribute(decode_rows_kernel<EPI, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, DR_SMEM_MAX));
  });
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(DR_THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = (unsigned)dec_launch_attrs(at, S, pdl);
  return (int)cudaLaunchKernelEx(&cfg, decode_rows_kernel<EPI, SPLIT>, tw, tx, p);
}

}  // namespace bones

extern "C" {
using namespace bones;

// As bones_decode_gemm for b <= 64 and K a multiple of 128, in tiles of `nt` columns (a multiple of 8 from 16 to 64 that divides N);
// ssq_out is [N / nt, b].  `splits` (1, 2, 4 or 8, at most K / 128): CTAs of a cluster that share a tile's contraction.  `ctas`: without a split,
// how many CTAs walk the tiles (0: one for each).  The soft-cap comes without a split only.
int bones_decode_rows(const void* X, const void* W, void* out, int b, int N, int K, int nt, int splits, int ctas, int epi, const float* ssq_in, int n_ssq,
                      const void* res, const void* x0, const float* mix_a, const float* mix_b, float* ssq_out, float cap, const void* next_w, long long next_bytes, int pdl, void* stream) {
  if (b < 1 || b > 64 || N <= 0 || K <= 0 || (K % 128) || nt < 16 || nt > 64 || (nt % 8) || (N % nt)) return -2;
  if ((splits != 1 && splits != 2 && splits != 4 && splits != 8) || splits > K / 128 || ctas < 0 || (splits > 1 && ctas)) return -2;
  if (misaligned16(X, W, out, res, x0, next_w) || (epi == DEC_RES && !res)) return -2;
  DecRowsParams p;
  p.N = N; p.b = b; p.KS = K / 128;
  p.nt = nt; p.tiles = N / nt;
  p.rb = (b + 7) & ~7;
  const int grid = splits > 1 || ctas == 0 || ctas > p.tiles ? p.tiles * splits : ctas;
  // slots: X the bytes that keep its loads going at L2 speed (96 KB), W what is left; none holds more than the CTA will load
  const int stages = (p.KS + splits - 1) / splits * (splits > 1 ? 1 : (p.tiles + grid - 1) / grid);
  const int xb = p.rb * 256, wb = nt * 256, fixed = (splits > 1 ? 64 * (nt + 4) * 4 : 0) + (int)DR_BARS + DR_SUMS + 1024;
  // the MMA reads 64 rows of a slot: behind the last X slot stands the W ring, at least two slots of 4 KB (a block's rows end 8 KB after
  // its start at most)
  int room = DR_SMEM_AIM - fixed;
  p.xs = 96 * 1024 / xb;
  if (p.xs > stages) p.xs = stages;
  if (p.xs > DR_MAX_SLOTS) p.xs = DR_MAX_SLOTS;
  p.ws = (room - p.xs * xb) / wb;
  if (p.ws > stages) p.ws = stages;
  if (p.ws > DR_MAX_SLOTS) p.ws = DR_MAX_SLOTS;
  if (p.ws < 2) p.ws = 2;
  const int smem = p.xs * xb + p.ws * wb + fixed;
  if (smem > DR_SMEM_MAX) return -2;
  p.ssq_in = ssq_in; p.n_ssq = n_ssq; p.inv_k = 1.0f / (float)K;
  p.res = (const __nv_bfloat16*)res;
  p.x0 = (const __nv_bfloat16*)x0;
  p.mix_a = mix_a; p.mix_b = mix_b;
  p.ssq_out = ssq_out;
  p.out = (__nv_bfloat16*)out;
  p.cap = cap;
  p.err = error_word();
  p.next_w = (const uint8_t*)next_w;
  p.next_bytes = next_w ? next_bytes & ~15ll : 0;
  CUtensorMap tw, tx;
  const uint64_t wd[3] = {64, (uint64_t)N, (uint64_t)K / 64}, xd[3] = {64, (uint64_t)b, (uint64_t)K / 64}, st[2] = {(uint64_t)K * 2, 128};
  const uint32_t wbox[3] = {64, (uint32_t)nt, 2}, xbox[3] = {64, (uint32_t)p.rb, 2};
  int rc = make_tmap(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, W, wd, st, wbox, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  rc = make_tmap(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, X, xd, st, xbox, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
#define BONES_ROWS(E) (splits > 1 ? launch_rows<E, true>(tw, tx, p, splits, grid, smem, pdl, s) : launch_rows<E, false>(tw, tx, p, 1, grid, smem, pdl, s))
  switch (epi) {
    case DEC_SCALE: return BONES_ROWS(DEC_SCALE);
    case DEC_RELU2: return BONES_ROWS(DEC_RELU2);
    case DEC_RES: return BONES_ROWS(DEC_RES);
    case DEC_SOFTCAP: return splits > 1 ? -2 : launch_rows<DEC_SOFTCAP, false>(tw, tx, p, 1, grid, smem, pdl, s);      // a head has tiles enough
  }
#undef BONES_ROWS
  return -2;
}
}  // extern "C"
