// Projections of one decode step: few rows (up to 128 sequences), every weight read once.
//
//   out[t, n] = epilogue( r_t * sum_k X[t, k] W[n, k] )          X bf16 [b, K], W bf16 [N, K]
//
// Bound by the weights' bytes and by latency: 10 to 13 MB per projection are 1.5 to 2 us at the copy rate, about what one
// load round trip, one barrier and one launch cost each.  So:
//   * the weights are the 128-row operand (M) and the sequences the narrow one (N = 16 .. 128): no padded token rows are
//     loaded, and the accumulator's lanes are output columns, so stores of a sequence are contiguous;
//   * the contraction of a 128-column tile is split over the CTAs of a cluster, which exchange their fp32 partial sums through
//     distributed shared memory and add them in a fixed order: no slices in global memory, no finishing kernel, and a step is
//     reproducible bit for bit (the slices and their finishing kernels were 26 of 158 ms of 128 steps at batch 64);
//   * RMSNorm has no gain, so it is one factor per sequence: norm(x) W^T = r (x W^T).  The epilogue that produces x leaves the
//     squares' sums per 128-column tile, the epilogue that consumes it multiplies by r: no norm kernel, and x enters the MMA
//     as it is instead of rounded once more;
//   * launched with programmatic dependence, and every kernel lets its successor start as soon as it runs itself: the weight tiles
//     of the first stages (weights depend on nothing in the step) and the cache rows of the attention are requested before the wait
//     for the previous kernel, so their latency hides behind it.  Only that wait orders data: nothing is written before it, and
//     nothing that a kernel of this step writes is used before it.  (The attention looks at the document start ahead of the wait only
//     to choose what it requests early, and reads it again behind the wait.)
// Warp 0 issues the TMA loads, warp 1 the MMAs, the others run the epilogue.
//
// Up to 64 sequences most layers' projections, and most heads of more than 32, run on decode_rows.cu, whose tiles exchange no partial sums or small
// ones (`use_rows` and `head_on_rows` in utils/decode.py); this kernel has the rest: more sequences, other heads, models wider than 1536 and
// narrow ones with few sequences.  What bounds it is a chain of latencies: per projection about 1.1 us from the previous kernel's end to this
// one's start, 1.5 to 4 us until the accumulator is complete, 1.3 to 2.9 us for the exchange, 0.7 to 1.3 us of epilogue.
#include "decode_common.cuh"

namespace bones {

struct DecGemmParams {
  int N, b, KB;
  const float* ssq_in;        // [n_ssq, b] partial sums of squares of X's rows (null: r = 1)
  int n_ssq;
  float inv_k;                // 1 / K
  const __nv_bfloat16* res;   // [b, N]
  const __nv_bfloat16* x0;    // [b, N] or null
  const float *mix_a, *mix_b;
  float* ssq_out;             // [N / 128, b] or null
  __nv_bfloat16* out;         // [b, N]
  float cap;
  int* err;
};

// Where the partial sums of output column n, tokens 4 u .. 4 u + 3 of `1 << lc`, of cluster rank s stand in their owner's buffer
// (16-byte units; the unit index is turned by the row so that eight lanes of a warp hit different banks).
__device__ __forceinline__ uint32_t red_unit(int s, int n, int u, int lc) {
  const int lu = lc - 2;
  const int turn = lu >= 3 ? (n & 7) : ((n >> (3 - lu)) & ((1 << lu) - 1));
  return (uint32_t)((((s << 7) + n) << lu) + (u ^ turn));
}

// Sixteen epilogue warps, four per 32-lane quadrant of the accumulator: each handles few columns, because a lone warp per
// scheduler runs its instructions one latency after the other (with four warps the two phases of the epilogue took 2.2 us, with
// everything unrolled 5.5).
constexpr int DG_EW = 16;
constexpr int DG_THREADS = 64 + 32 * DG_EW;
constexpr uint32_t DG_W_BYTES = 128 * 64 * 2;
// Stages: as many as leave room for two CTAs on an SM (the next kernel's CTAs move in while this one runs), at 128 sequences
// for one.
template <int NB>
struct DgGeom {
  static constexpr uint32_t kX = NB * 64 * 2, kStage = DG_W_BYTES + kX, kRed = 128 * NB * 4;
  static constexpr int kStages = NB == 128 ? 4 : NB == 64 ? 3 : NB == 32 ? 4 : 5;
  static constexpr uint32_t kBars = kStages * kStage + kRed;
  static constexpr uint32_t kSmem = kBars + 128 + 5 * NB * 4 + 1024;      // barriers, squares' sums of four warps, norm factors, alignment slack
};

template <int NB, int EPI>
__global__ void __launch_bounds__(DG_THREADS)
decode_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const DecGemmParams p) {
  using G = DgGeom<NB>;
  constexpr int ST = G::kStages;
  constexpr uint32_t TCOLS = NB < 32 ? 32 : NB;
  extern __shared__ uint8_t dg_raw[];
  const uint32_t raw = smem_u32(dg_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* gen = dg_raw + (base - raw);
  const uint32_t red = base + ST * G::kStage, bars = base + G::kBars;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (ST + s); };
  const uint32_t tfull = bars + 8u * (2 * ST), tmem_slot = bars + 8u * (2 * ST + 1);
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(gen + G::kBars + 8 * (2 * ST + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + G::kBars + 8 * (2 * ST + 1) + 8);
  float* wsq = reinterpret_cast<float*>(gen + G::kBars + 128);            // [4 warps][tokens of this CTA]
  float* rowr = wsq + 4 * NB;                                             // norm factors of this CTA's tokens
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank(), S = (int)cluster_size();
  const int tile = blockIdx.x / S, n0 = tile * 128;
  const int kb0 = p.KB * rank / S, kb1 = p.KB * (rank + 1) / S;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  __syncthreads();
  if (warp == 0) {
    // weights of the first stages: independent of the previous kernel
    if (elect_one()) {
      for (int kb = kb0; kb < min(kb1, kb0 + ST); ++kb) {
        const int s = kb - kb0;
        mbar_arrive_expect_tx(full(s), G::kStage);
        tma_load_2d(base + s * G::kStage, &tm_w, full(s), kb * 64, n0);
      }
    }
    __syncwarp();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  cluster_barrier();                           // also: every CTA of the cluster runs, so its shared memory may be written
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_g;
  const int cols = NB / S, lc = 31 - __clz(cols);        // tokens this CTA finishes (a power of two), and how many of them exist
  const int mine = max(0, min(cols, p.b - rank * cols));
  pdl_launch();
  pdl_wait();
  // residual, x0 and mix factors of an epilogue thread's first four tokens, requested before the wait for the accumulator
  __nv_bfloat16 rs[4], x0[4];
  float ma = 0.f, mb = 0.f;
  auto residual = [&](int c0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long at = (long long)(rank * cols + min(c0 + i, mine - 1)) * p.N + n0 + (warp & 3) * 32 + lane;
      rs[i] = p.res[at];
      if (p.x0) x0[i] = p.x0[at];
    }
  };

  if (warp == 0) {
    bool dead = false;
    for (int kb = kb0; kb < kb1; ++kb) {
      const int i = kb - kb0, s = i % ST;
      if (i >= ST && !dead) dead = !mbar_wait(empty(s), (uint32_t)((i / ST - 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
      if (elect_one() && !dead) {
        if (i >= ST) {
          mbar_arrive_expect_tx(full(s), G::kStage);
          tma_load_2d(base + s * G::kStage, &tm_w, full(s), kb * 64, n0);
        }
        tma_load_2d(base + s * G::kStage + DG_W_BYTES, &tm_x, full(s), kb * 64, 0);
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(128, NB, 1, 0, 0);
    bool dead = false;
    for (int kb = kb0; kb < kb1; ++kb) {
      const int i = kb - kb0, s = i % ST;
      if (!dead) dead = !mbar_wait(full(s), (uint32_t)((i / ST) & 1), abort_flag, p.err, ERR_WAIT_FULL);
      tc_fence_after();
      const uint64_t wd = umma_smem_desc(base + s * G::kStage, 0, 1024, kLayoutSw128);
      const uint64_t xd = umma_smem_desc(base + s * G::kStage + DG_W_BYTES, 0, 1024, kLayoutSw128);
      if (elect_one() && !dead) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f16(tmem, wd + (uint64_t)(k * 2), xd + (uint64_t)(k * 2), idesc, (i | k) ? 1u : 0u);
        tc_commit(empty(s));
        if (kb == kb1 - 1) tc_commit(tfull);
      }
    }
  } else {
    // while the weights are on their way: the norm factors of this CTA's tokens
    const int q = warp & 3, nl = q * 32 + lane;
    if (EPI == DEC_RES && ((warp - 2) >> 2) * 4 < mine) {
      residual(((warp - 2) >> 2) * 4);
      if (p.x0) { ma = *p.mix_a; mb = *p.mix_b; }
    }
    {
      const int e = threadIdx.x - 64, t = rank * cols + e;
      if (e < cols) {
        float ss = 0.f;
        if (p.ssq_in && t < p.b) {
#pragma unroll 5
          for (int j = 0; j < p.n_ssq; ++j) ss += p.ssq_in[j * p.b + t];
        }
        rowr[e] = p.ssq_in ? rsqrtf(ss * p.inv_k + 1.1920928955078125e-07f) : 1.0f;
      }
    }
    const bool got = mbar_wait(tfull, 0, abort_flag, p.err, ERR_WAIT_TMEM_FULL);
    // partial sums to their owners: CTA o of the cluster finishes tokens o * cols .. of the tile
    if (__all_sync(0xffffffffu, got)) {
      tc_fence_after();
#pragma unroll 1
      for (int c0 = ((warp - 2) >> 2) * 16; c0 < NB; c0 += DG_EW * 4) {
        uint32_t v[16];
        __syncwarp();
        BONES_TMEM_LD16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const int c = c0 + i;
          st_cluster_v4(map_to_rank(red + 16u * red_unit(rank, nl, (c & (cols - 1)) >> 2, lc), (uint32_t)(c >> lc)), v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  cluster_barrier();                           // every partial sum of the cluster is in its owner's memory
  if (warp >= 2) {
    // four tokens at a time
    const int q = warp & 3, nl = q * 32 + lane, warp_group = (warp - 2) >> 2;
    if (!*abort_flag) {
#pragma unroll 1
      for (int c0 = warp_group * 4; c0 < mine; c0 += DG_EW) {
        const long long at0 = (long long)(rank * cols + c0) * p.N + n0 + nl;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (EPI == DEC_RES && c0 != warp_group * 4) residual(c0);
#pragma unroll 2
        for (int s = 0; s < S; ++s) {
          const float4 w = *reinterpret_cast<const float4*>(gen + ST * G::kStage + 16u * red_unit(s, nl, c0 >> 2, lc));
          v[0] += w.x; v[1] += w.y; v[2] += w.z; v[3] += w.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float y = v[i] * rowr[c0 + i];
          if (EPI == DEC_RELU2) {
            y = fmaxf(y, 0.f);
            y *= y;
          } else if (EPI == DEC_SOFTCAP) {
            float th;
            asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(y / p.cap));
            y = p.cap * th;
          } else if (EPI == DEC_RES) {
            y = __bfloat162float(__float2bfloat16(y + __bfloat162float(rs[i])));
            if (p.x0) y = ma * y + mb * __bfloat162float(x0[i]);
          }
          const __nv_bfloat16 o = __float2bfloat16(y);
          if (c0 + i < mine) p.out[at0 + (long long)i * p.N] = o;
          v[i] = __bfloat162float(o);
        }
        if (EPI == DEC_RES && p.ssq_out) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float w = warp_sum(v[i] * v[i]);
            if (lane == 0) wsq[q * NB + c0 + i] = w;
          }
        }
      }
    }
    if (EPI == DEC_RES && p.ssq_out) {
      asm volatile("bar.sync 1, 512;" ::: "memory");
      const int e = threadIdx.x - 64;
      if (e < mine) p.ssq_out[tile * p.b + rank * cols + e] = (wsq[e] + wsq[NB + e]) + (wsq[2 * NB + e] + wsq[3 * NB + e]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TCOLS);
  }
}

template <int NB, int EPI>
static int launch_dec_gemm(const CUtensorMap& tw, const CUtensorMap& tx, const DecGemmParams& p, int S, int pdl, cudaStream_t stream) {
  using G = DgGeom<NB>;
  static OncePerDevice limit;
  BONES_ONCE(limit, {
    BONES_CHECK(cudaFuncSetAttribute(decode_gemm_kernel<NB, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::kSmem));
    BONES_CHECK(cudaFuncSetAttribute(decode_gemm_kernel<NB, EPI>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  });
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  cfg.gridDim = dim3((unsigned)(p.N / 128 * S));
  cfg.blockDim = dim3(DG_THREADS);
  cfg.dynamicSmemBytes = G::kSmem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = (unsigned)dec_launch_attrs(at, S, pdl);
  if (S > 8) {                                 // more than the portable cluster size: a device may have no room for one
    static OncePerDevice asked;
    static int rooms[OncePerDevice::kDevices] = {0};
    int dev = 0, room = 0;
    BONES_CHECK(cudaGetDevice(&dev));
    BONES_ONCE(asked, {
      BONES_CHECK(cudaOccupancyMaxActiveClusters(&room, decode_gemm_kernel<NB, EPI>, &cfg));
      if (dev < OncePerDevice::kDevices) rooms[dev] = room;
    });
    if (dev < OncePerDevice::kDevices) room = rooms[dev];
    if (room == 0) return launch_dec_gemm<NB, EPI>(tw, tx, p, 8, pdl, stream);
  }
  return (int)cudaLaunchKernelEx(&cfg, decode_gemm_kernel<NB, EPI>, tw, tx, p);
}
template <int NB>
static int launch_dec_gemm_epi(int epi, const CUtensorMap& tw, const CUtensorMap& tx, const DecGemmParams& p, int S, int pdl, cudaStream_t stream) {
  switch (epi) {
    case DEC_SCALE: return launch_dec_gemm<NB, DEC_SCALE>(tw, tx, p, S, pdl, stream);
    case DEC_RELU2: return launch_dec_gemm<NB, DEC_RELU2>(tw, tx, p, S, pdl, stream);
    case DEC_RES: return launch_dec_gemm<NB, DEC_RES>(tw, tx, p, S, pdl, stream);
    case DEC_SOFTCAP: return launch_dec_gemm<NB, DEC_SOFTCAP>(tw, tx, p, S, pdl, stream);
  }
  return -2;
}

// ---------------------------------------------------------------------------------------------------------------
// Between the projections: RoPE + QK-norm of the new token, cache append and attention over the cache, one CTA per
// (head, sequence).  Sixteen lanes share a key (8 dims each), a lane has U keys a round: the keys' loads of the next round go out as soon
// as this round's scores are computed, the values' as soon as its sums are, so 2 U loads a thread are in flight nearly all the time.  The
// scores of a lane's keys are folded across the sixteen lanes together (four keys: five shuffles, and four to hand the weights back;
// one key after the other takes sixteen), and a weight is computed by 16 / U lanes instead of sixteen.
// U = 4 keeps 64 keys and values a CTA in flight and takes 64 registers, so an SM holds four CTAs; above that U = 2 (48 registers, five
// CTAs), for 640 CTAs of 64 sequences x 10 heads in one wave.  Six layers, 1280 wide, us a step at position 64 / 256 / 1000, with one key a
// lane in flight and with these: batch 4 194 / 239 / 422 -> 190 / 213 / 292; batch 32 (U = 4) 208 / 263 / 465 -> 205 / 239 / 352, with U = 2
// 207 / 250 / 400; batch 64 (U = 2) 225 / 295 / 525 -> 222 / 277 / 466, with U = 4 231 / 277 / 465.
// The fixed soft-max shift of the training kernels applies (q and k are RMS-normalised).
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ int ld_relaxed(const int* p) {      // from L2: an earlier look may have left the line in L1
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(int* p, int v) { asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }
constexpr int kDaWarps = 8;
template <int U, int CTAS>
__global__ void __launch_bounds__(32 * kDaWarps, CTAS) decode_attn_step_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ cosT,
                                                                  const float* __restrict__ sinT, __nv_bfloat16* kcache, __nv_bfloat16* vcache,
                                                                  const int* pos_ptr, const int* doc_start, __nv_bfloat16* __restrict__ y, int H,
                                                                  int Tmax, float scale, int window_tiles) {
  static_assert(U == 2 || U == 4, "the fold of the scores");
  constexpr int NW = kDaWarps, ROUND = 2 * U * NW;            // keys of the CTA in a round
  __shared__ __align__(16) __nv_bfloat16 s_new[3][128];
  __shared__ __align__(16) float s_acc[NW][128];
  __shared__ float s_l[NW];
  pdl_launch();
  const int h = blockIdx.x, b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l16 = lane & 15;
  const int pos = *pos_ptr;
  if (pos < 0 || pos >= Tmax) {
    pdl_wait();
    return;
  }
  const int band = window_tiles > 0 ? max((pos / 128 - (window_tiles - 1)) * 128, 0) : 0;
  // The first kernel of this step may be storing a new document start: until the wait this is where the first key probably is,
  // and any value only moves requests that stay below `pos`.
  int lo = doc_start ? max(ld_relaxed(doc_start + b), band) : band;
  const int A = H * 128;
  const __nv_bfloat16 *kp = kcache + ((long long)b * Tmax * H + h) * 128 + l16 * 8, *vp = vcache + ((long long)b * Tmax * H + h) * 128 + l16 * 8;
  uint4 k[U], v[U];
  // key u of this lane in the round that begins at j: j + 2 u; keys before the new one come from the cache
  auto fetch = [&](uint4* to, const __nv_bfloat16* from, int j) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (j + 2 * u < pos) to[u] = *reinterpret_cast<const uint4*>(from + (long long)(j + 2 * u) * A);
  };
  int j = lo + warp * 2 * U + (lane >> 4);
  fetch(k, kp, j);
  fetch(v, vp, j);
  // the cache holds earlier steps' keys: the next ones come to L2 while the projection before this kernel still runs
  if ((l16 & 3) == 0) {
    for (int n = j + ROUND; n < min(pos, lo + 128); n += ROUND) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (n + 2 * u < pos) prefetch_l2(((l16 & 4) ? vp : kp) - l16 * 8 + (l16 >> 3) * 64 + (long long)(n + 2 * u) * A);
    }
  }
  pdl_wait();
  const int now = doc_start ? max(ld_relaxed(doc_start + b), band) : band;      // on its way while q, k and v are handled
  if (warp < 3) {
    const __nv_bfloat16* src = qkv + (long long)b * 3 * A + warp * A + h * 128;
    float2 x1 = unpack_bf16(*reinterpret_cast<const uint32_t*>(src + 2 * lane));
    float2 x2 = unpack_bf16(*reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane));
    if (warp < 2) {
      const float2 cs = *reinterpret_cast<const float2*>(cosT + (long long)pos * 64 + 2 * lane);
      const float2 sn = *reinterpret_cast<const float2*>(sinT + (long long)pos * 64 + 2 * lane);
      float2 y1, y2;
      y1.x = x1.x * cs.x + x2.x * sn.x; y1.y = x1.y * cs.y + x2.y * sn.y;
      y2.x = -x1.x * sn.x + x2.x * cs.x; y2.y = -x1.y * sn.y + x2.y * cs.y;
      const float ss = warp_sum(y1.x * y1.x + y1.y * y1.y + y2.x * y2.x + y2.y * y2.y);
      const float r = rsqrtf(ss * (1.0f / 128.0f) + 1.1920928955078125e-07f);
      x1 = make_float2(y1.x * r, y1.y * r);
      x2 = make_float2(y2.x * r, y2.y * r);
    }
    const uint32_t w1 = pack_bf16(x1.x, x1.y), w2 = pack_bf16(x2.x, x2.y);
    *reinterpret_cast<uint32_t*>(&s_new[warp][2 * lane]) = w1;
    *reinterpret_cast<uint32_t*>(&s_new[warp][64 + 2 * lane]) = w2;
    if (warp > 0) {
      __nv_bfloat16* dst = (warp == 1 ? kcache : vcache) + (((long long)b * Tmax + pos) * H + h) * 128;
      *reinterpret_cast<uint32_t*>(dst + 2 * lane) = w1;
      *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = w2;
    }
  }
  if (now != lo) {                             // a document begins here
    lo = now;
    j = lo + warp * 2 * U + (lane >> 4);
    fetch(k, kp, j);
    fetch(v, vp, j);
  }
  __syncthreads();
  float q[8], acc[8], l = 0.f;
  unpack8(*reinterpret_cast<const uint4*>(&s_new[0][l16 * 8]), q);
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  const float c1 = scale * 1.4426950408889634f, c2 = scale * 128.0f * 1.4426950408889634f;
  const bool up = (lane & 8) != 0, right = (lane & 4) != 0;
  const int mine = U == 4 ? 2 * ((up ? 2 : 0) + (right ? 1 : 0)) : (up ? 2 : 0);      // after the fold this lane has the score of key j + mine
#pragma unroll 1
  for (int j0 = lo + warp * 2 * U; j0 <= pos; j0 += ROUND, j += ROUND) {
    float s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (j + 2 * u >= pos) {                  // the new token's own key and value; past it nothing
        k[u] = *reinterpret_cast<const uint4*>(&s_new[1][l16 * 8]);
        v[u] = *reinterpret_cast<const uint4*>(&s_new[2][l16 * 8]);
      }
      float kf[8];
      unpack8(k[u], kf);
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i += 2) { s0 += q[i] * kf[i]; s1 += q[i + 1] * kf[i + 1]; }
      s[u] = s0 + s1;
    }
    fetch(k, kp, j + ROUND);
    float r;
    if (U == 4) {
      const float t0 = __shfl_xor_sync(0xffffffffu, up ? s[0] : s[U - 2], 8), t1 = __shfl_xor_sync(0xffffffffu, up ? s[1] : s[U - 1], 8);
      const float r0 = (up ? s[U - 2] : s[0]) + t0, r1 = (up ? s[U - 1] : s[1]) + t1;
      r = (right ? r1 : r0) + __shfl_xor_sync(0xffffffffu, right ? r0 : r1, 4);
    } else {
      r = (up ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, up ? s[0] : s[1], 8);
      r += __shfl_xor_sync(0xffffffffu, r, 4);
    }
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    const float w = j + mine <= pos ? exp2f(r * c1 - c2) : 0.f;
    l += w;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float pu = __shfl_sync(0xffffffffu, w, (lane & 16) | (u * (16 / U)));
      float vf[8];
      unpack8(v[u], vf);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += pu * vf[i];
    }
    fetch(v, vp, j + ROUND);
  }
  if (U == 4) l += __shfl_xor_sync(0xffffffffu, l, 4);
  l += __shfl_xor_sync(0xffffffffu, l, 8);
  l += __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
  if (lane < 16) {
    *reinterpret_cast<float4*>(&s_acc[warp][l16 * 8]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<float4*>(&s_acc[warp][l16 * 8 + 4]) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    if (l16 == 0) s_l[warp] = l;
  }
  __syncthreads();
  if (threadIdx.x < 128) {
    float o = 0.f, lt = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) { o += s_acc[w][threadIdx.x]; lt += s_l[w]; }
    y[((long long)b * H + h) * 128 + threadIdx.x] = __float2bfloat16(lt > 0.f ? o / lt : 0.f);
  }
}

// First kernel of a step, one CTA per sequence: document start, x0 = norm(embedding), x = a x0 + b x0 and its squares' sum.
__global__ void __launch_bounds__(256) decode_begin_kernel(const long long* tok, const int* pos_ptr, int* doc_start, long long bos,
                                                           const __nv_bfloat16* __restrict__ wte, long long rows, int C,
                                                           const float* __restrict__ mix_a, const float* __restrict__ mix_b,
                                                           __nv_bfloat16* __restrict__ x0, __nv_bfloat16* __restrict__ x, float* __restrict__ ssq) {
  __shared__ float red[8];
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long t = tok[b];
  if (doc_start && threadIdx.x == 0 && t == bos) st_relaxed(doc_start + b, *pos_ptr);
  auto sum = [&](float v) {
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[i];
    return s;
  };
  const bool known = t >= 0 && t < rows;       // any other id has a zero row, as in the embedding gather
  const __nv_bfloat16* e = wte + (known ? t : 0) * C;
  auto at = [&](int c) { return known ? __bfloat162float(e[c]) : 0.f; };
  float s = 0.f;
  for (int c = threadIdx.x; c < C; c += 256) { const float f = at(c); s += f * f; }
  const float r = rsqrtf(sum(s) / C + 1.1920928955078125e-07f), ma = *mix_a, mb = *mix_b;
  s = 0.f;
  for (int c = threadIdx.x; c < C; c += 256) {
    const __nv_bfloat16 z = __float2bfloat16(at(c) * r);
    const float f = __bfloat162float(z);
    const __nv_bfloat16 m = __float2bfloat16(ma * f + mb * f);
    x0[(long long)b * C + c] = z;
    x[(long long)b * C + c] = m;
    s += __bfloat162float(m) * __bfloat162float(m);
  }
  s = sum(s);
  if (threadIdx.x == 0) ssq[b] = s;
}

// Last kernel of a step, one CTA per sequence: arg-max of the logits (lowest index of equal values, a NaN above everything),
// the forced token while the prompt lasts, and the position's advance by the last CTA to finish.
__global__ void __launch_bounds__(1024) decode_end_kernel(const __nv_bfloat16* __restrict__ logits, long long ldl, int V, int* pos_ptr,
                                                          const int* __restrict__ prompt_len, long long* out, long long ldo, int L, long long* tok,
                                                          int* ticket) {
  __shared__ float sv[32];
  __shared__ int si[32];
  pdl_wait();
  pdl_launch();
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float best = 0.f;
  int at = -1;
  auto better = [](float v, int i, float w, int k) {       // (v, i) before (w, k)
    if (i < 0) return false;
    if (k < 0) return true;
    const bool vn = v != v, wn = w != w;
    if (vn || wn) return vn && (!wn || i < k);
    return v > w || (v == w && i < k);
  };
  const __nv_bfloat16* row = logits + (long long)b * ldl;
  for (int c = threadIdx.x * 8; c < V; c += 8192) {
    const uint4 u = *reinterpret_cast<const uint4*>(row + c);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 f = unpack_bf16(w[i >> 1]);
      const float v = (i & 1) ? f.y : f.x;
      if (c + i < V && better(v, c + i, best, at)) { best = v; at = c + i; }
    }
  }
  auto fold = [&](float& v, int& i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float w = __shfl_xor_sync(0xffffffffu, v, o);
      const int k = __shfl_xor_sync(0xffffffffu, i, o);
      if (better(w, k, v, i)) { v = w; i = k; }
    }
  };
  fold(best, at);
  if (lane == 0) { sv[warp] = best; si[warp] = at; }
  __syncthreads();
  if (warp == 0) {
    best = sv[lane];
    at = si[lane];
    fold(best, at);
    if (lane == 0) {
      const int pos = *pos_ptr + 1;
      long long nxt = at;
      if (pos < L) {
        if (pos < *prompt_len) nxt = out[b * ldo + pos];
        else out[b * ldo + pos] = nxt;
      }
      tok[b] = nxt;
      __threadfence();
      if (atomicAdd(ticket, 1) == (int)gridDim.x - 1) {     // everybody has read the position
        *ticket = 0;
        *pos_ptr = pos;
      }
    }
  }
}

}  // namespace bones

extern "C" {
using namespace bones;

// X [b, K], W [N, K], out [b, N], all bf16 and contiguous; N a multiple of 128, K of 64, b <= 128.  `splits`: CTAs of a cluster
// that share a tile's contraction (1, 2, 4, 8 or 16; a CTA finishes four tokens or more, so few
// sequences are padded to 4 * splits).  `pdl`: the previous kernel on the stream is one of this file's.
int bones_decode_gemm(const void* X, const void* W, void* out, int b, int N, int K, int splits, int epi, const float* ssq_in, int n_ssq,
                      const void* res, const void* x0, const float* mix_a, const float* mix_b, float* ssq_out, float cap, int pdl, void* stream) {
  if (b < 1 || b > 128 || (N % 128) || (K % 64) || N <= 0 || K <= 0 || (splits != 1 && splits != 2 && splits != 4 && splits != 8 && splits != 16) || splits > K / 64)
    return -2;
  if (((uintptr_t)X & 15) || ((uintptr_t)W & 15) || (epi == DEC_RES && !res)) return -2;
  const int rows = b > 4 * splits ? b : 4 * splits, nb = rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
  DecGemmParams p;
  p.N = N; p.b = b; p.KB = K / 64;
  p.ssq_in = ssq_in; p.n_ssq = n_ssq; p.inv_k = 1.0f / (float)K;
  p.res = (const __nv_bfloat16*)res;
  p.x0 = (const __nv_bfloat16*)x0;
  p.mix_a = mix_a; p.mix_b = mix_b;
  p.ssq_out = ssq_out;
  p.out = (__nv_bfloat16*)out;
  p.cap = cap;
  p.err = error_word();
  CUtensorMap tw, tx;
  const uint64_t wd[2] = {(uint64_t)K, (uint64_t)N}, xd[2] = {(uint64_t)K, (uint64_t)b}, st[1] = {(uint64_t)K * 2};
  const uint32_t wb[2] = {64, 128}, xb[2] = {64, (uint32_t)nb};
  int rc = make_tmap(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, wd, st, wb, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  rc = make_tmap(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, xd, st, xb, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  if (nb == 16) return launch_dec_gemm_epi<16>(epi, tw, tx, p, splits, pdl, s);
  if (nb == 32) return launch_dec_gemm_epi<32>(epi, tw, tx, p, splits, pdl, s);
  if (nb == 64) return launch_dec_gemm_epi<64>(epi, tw, tx, p, splits, pdl, s);
  return launch_dec_gemm_epi<128>(epi, tw, tx, p, splits, pdl, s);
}

int bones_decode_attn_step(const void* qkv, const float* cosT, const float* sinT, void* kcache, void* vcache, const int* pos, const int* doc_start,
                           void* y, int B, int H, int Tmax, float scale, int window_tiles, void* stream) {
  static int sms[64] = {0};
  int dev = 0;
  BONES_CHECK(cudaGetDevice(&dev));
  if (dev < 64 && !sms[dev]) BONES_CHECK(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  const bool four = dev < 64 && (long long)H * B <= 4ll * sms[dev];        // the CTAs of one wave with four keys a lane
  cfg.gridDim = dim3((unsigned)H, (unsigned)B);
  cfg.blockDim = dim3(32 * kDaWarps);
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = at;
  cfg.numAttrs = (unsigned)dec_launch_attrs(at, 1, 1);
  return (int)cudaLaunchKernelEx(&cfg, four ? decode_attn_step_kernel<4, 4> : decode_attn_step_kernel<2, 5>, (const __nv_bfloat16*)qkv, cosT, sinT,
                                 (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, pos, doc_start, (__nv_bfloat16*)y, H, Tmax, scale, window_tiles);
}

int bones_decode_begin(const long long* tok, const int* pos, int* doc_start, long long bos, const void* wte, long long rows, int C,
                       const float* mix_a, const float* mix_b, void* x0, void* x, float* ssq, int B, void* stream) {
  decode_begin_kernel<<<B, 256, 0, (cudaStream_t)stream>>>(tok, pos, doc_start, bos, (const __nv_bfloat16*)wte, rows, C, mix_a, mix_b,
                                                           (__nv_bfloat16*)x0, (__nv_bfloat16*)x, ssq);
  return (int)cudaGetLastError();
}

// out: rows of L tokens, ldo apart; ticket: one int, zero before the first step
int bones_decode_end(const void* logits, long long ldl, int V, int* pos, const int* prompt_len, long long* out, long long ldo, int L, long long* tok,
                     int* ticket, int B, void* stream) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3((unsigned)B);
  cfg.blockDim = dim3(1024);
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = at;
  cfg.numAttrs = (unsigned)dec_launch_attrs(at, 1, 1);
  return (int)cudaLaunchKernelEx(&cfg, decode_end_kernel, (const __nv_bfloat16*)logits, ldl, V, pos, prompt_len, out, ldo, L, tok, ticket);
}
}  // extern "C"
