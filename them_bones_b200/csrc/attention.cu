// Causal flash attention for the decoder, forward pass, on tcgen05 tensor cores with TMEM accumulators and TMA loads,
// plus the RoPE + QK-RMSNorm pre/post passes.
//
// Semantics (reference: fused RoPE + QK-norm + causal attention, round2/source/kernels/nki_attn_bandpro.py:686-978; eager
// form round2/source/train.py:10209-10252): q and k are rotated (rotate-half RoPE), RMS-normalised per head, and
// attention is causal softmax(scale * q k^T) v.  Added here: keys are limited to the query's document
// (`doc_start[b, t]` = position of the most recent BOS) and, for banded layers, to the query's 128-token tile and the
// `window_tiles - 1` tiles before it (the reference's tile band, round2/source/train.py:4740-4745).
//
// Because q and k are RMS-normalised, |q.k| <= head_dim, so the softmax uses the fixed shift `scale * head_dim` instead
// of a running maximum (the reference kernels do the same): P = exp(scale*s - scale*D) never overflows and no rescale of
// the output accumulator is ever needed.  The row sum is kept in registers and `lse = log(sum) + scale*D` is saved.
//
// The roles of the persistent forward kernel stand with it below.
#include "common.cuh"

namespace bones {

constexpr float kQkEps = 1.1920928955078125e-07f;   // 2^-23

// ---------------------------------------------------------------------------------------------------------------
// RoPE + QK-norm pre-pass: qkv [M, 3A] -> qk [M, 2A]  (A = H * D; q-hat then k-hat), and its backward
// (u = rope(x), r = rsqrt(mean(u^2)+eps), xhat = u r;  du = r (dxhat - xhat mean(dxhat xhat));  dx = rope^T(du)).
// ---------------------------------------------------------------------------------------------------------------
// D / 16 lanes per head vector (16-byte accesses: elements [8 l, 8 l + 8) of the first half and their rotate-half partners
// in the second half), reductions over that group of lanes.
__device__ __forceinline__ void ld8_bf16(const __nv_bfloat16* p, float* f) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float2 v = unpack_bf16(w[t]);
    f[2 * t] = v.x;
    f[2 * t + 1] = v.y;
  }
}
__device__ __forceinline__ void st8_bf16(__nv_bfloat16* p, const float* f) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]); u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}
__device__ __forceinline__ void ld8_f32(const float* p, float* f) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <int LANES>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// D / 16 threads per (row, head); a thread takes its 16 elements of the query head and of the key head, which share the
// rotation tables, so that 64 bytes of loads per thread are in flight (with 32 the kernel sat at 0.7 of the copy rate).
// `counter`: the work-item counter of the attention launch that follows on the stream, zeroed here (a memset of its own is
// one more launch on calls whose kernels take a few microseconds).
template <int D>
__global__ void rope_qknorm_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ cosT, const float* __restrict__ sinT,
                                       __nv_bfloat16* __restrict__ qk, int* counter, long long M, int T, int H) {
  constexpr int LANES = D / 16, HALF = D / 2;
  if (counter && blockIdx.x == 0 && threadIdx.x == 0) *counter = 0;
  const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;     // (row, head)
  const int l8 = threadIdx.x & (LANES - 1);
  const long long total = M * H;
  const bool live = item < total;
  const long long it = live ? item : total - 1;
  const int h = (int)(it % H);
  const long long row = it / H;
  const int t = (int)(row % T);
  const long long A = (long long)H * D;
  const __nv_bfloat16* src = qkv + row * 3 * A + (long long)h * D + l8 * 8;
  float x1[2][8], x2[2][8], cs[8], sn[8];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    ld8_bf16(src + w * A, x1[w]);
    ld8_bf16(src + w * A + HALF, x2[w]);
  }
  ld8_f32(cosT + (long long)t * HALF + l8 * 8, cs);
  ld8_f32(sinT + (long long)t * HALF + l8 * 8, sn);
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    float y1[8], y2[8];
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      y1[e] = x1[w][e] * cs[e] + x2[w][e] * sn[e];
      y2[e] = -x1[w][e] * sn[e] + x2[w][e] * cs[e];
      ss += y1[e] * y1[e] + y2[e] * y2[e];
    }
    ss = group_sum<LANES>(ss);
    const float r = rsqrtf(ss * (1.0f / D) + kQkEps);
#pragma unroll
    for (int e = 0; e < 8; ++e) { y1[e] *= r; y2[e] *= r; }
    if (live) {
      __nv_bfloat16* dst = qk + row * 2 * A + w * A + (long long)h * D + l8 * 8;
      st8_bf16(dst, y1);
      st8_bf16(dst + HALF, y2);
    }
  }
}

__global__ void rope_qknorm_bwd128_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ cosT,
                                          const float* __restrict__ sinT, const float* __restrict__ dqk,
                                          const __nv_bfloat16* __restrict__ dv, __nv_bfloat16* __restrict__ dqkv, long long M, int T,
                                          int H) {
  const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;     // (row, q|k|v, head)
  const int l8 = threadIdx.x & 7;
  const long long total = M * 3 * H;
  const bool live = item < total;
  const long long it = live ? item : total - 1;
  const int h = (int)(it % H), which = (int)((it / H) % 3);
  const long long row = it / (3 * H);
  const long long A = (long long)H * 128;
  __nv_bfloat16* out = dqkv + row * 3 * A + which * A + (long long)h * 128 + l8 * 8;
  // `which` is uniform over each 8-lane group but may differ inside a warp; the shuffles below are executed by all lanes
  const int t = (int)(row % T);
  const bool is_v = which == 2;
  const int wq = is_v ? 0 : which;
  const __nv_bfloat16* src = qkv + row * 3 * A + wq * A + (long long)h * 128 + l8 * 8;
  const float* g = dqk + row * 2 * A + wq * A + (long long)h * 128 + l8 * 8;
  float x1[8], x2[8], cs[8], sn[8], g1[8], g2[8], y1[8], y2[8];
  ld8_bf16(src, x1);
  ld8_bf16(src + 64, x2);
  ld8_f32(cosT + (long long)t * 64 + l8 * 8, cs);
  ld8_f32(sinT + (long long)t * 64 + l8 * 8, sn);
  ld8_f32(g, g1);
  ld8_f32(g + 64, g2);
  float ss = 0.f, dot = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    y1[e] = x1[e] * cs[e] + x2[e] * sn[e];
    y2[e] = -x1[e] * sn[e] + x2[e] * cs[e];
    ss += y1[e] * y1[e] + y2[e] * y2[e];
    dot += y1[e] * g1[e] + y2[e] * g2[e];
  }
  ss = group_sum<8>(ss);
  dot = group_sum<8>(dot);
  const float r = rsqrtf(ss * (1.0f / 128.0f) + kQkEps);
  const float m = dot * r * r * (1.0f / 128.0f);
  float o1[8], o2[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float du1 = r * (g1[e] - y1[e] * m), du2 = r * (g2[e] - y2[e] * m);
    o1[e] = du1 * cs[e] - du2 * sn[e];
    o2[e] = du1 * sn[e] + du2 * cs[e];
  }
  if (!live) return;
  if (is_v) {
    const __nv_bfloat16* gv = dv + row * A + (long long)h * 128 + l8 * 8;
    *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(gv);
    *reinterpret_cast<uint4*>(out + 64) = *reinterpret_cast<const uint4*>(gv + 64);
  } else {
    st8_bf16(out, o1);
    st8_bf16(out + 64, o2);
  }
}

// Same backward for bf16 dq-hat | dk-hat (the two-kernel attention backward writes them in bf16 and puts dV straight into
// its third of dqkv): only the q and k thirds are produced here.
template <int D>
__global__ void rope_qknorm_bwd_bf16_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ cosT,
                                               const float* __restrict__ sinT, const __nv_bfloat16* __restrict__ dqk,
                                               __nv_bfloat16* __restrict__ dqkv, long long M, int T, int H) {
  constexpr int LANES = D / 16, HALF = D / 2;
  const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;     // (row, head): query and key head
  const int l8 = threadIdx.x & (LANES - 1);
  const long long total = M * H;
  const bool live = item < total;
  const long long it = live ? item : total - 1;
  const int h = (int)(it % H);
  const long long row = it / H;
  const long long A = (long long)H * D;
  const long long col = (long long)h * D + l8 * 8;
  const __nv_bfloat16* src = qkv + row * 3 * A + col;
  const __nv_bfloat16* g = dqk + row * 2 * A + col;
  const int t = (int)(row % T);
  float x1[2][8], x2[2][8], g1[2][8], g2[2][8], cs[8], sn[8];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    ld8_bf16(src + w * A, x1[w]);
    ld8_bf16(src + w * A + HALF, x2[w]);
    ld8_bf16(g + w * A, g1[w]);
    ld8_bf16(g + w * A + HALF, g2[w]);
  }
  ld8_f32(cosT + (long long)t * HALF + l8 * 8, cs);
  ld8_f32(sinT + (long long)t * HALF + l8 * 8, sn);
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    float y1[8], y2[8];
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      y1[e] = x1[w][e] * cs[e] + x2[w][e] * sn[e];
      y2[e] = -x1[w][e] * sn[e] + x2[w][e] * cs[e];
      ss += y1[e] * y1[e] + y2[e] * y2[e];
      dot += y1[e] * g1[w][e] + y2[e] * g2[w][e];
    }
    ss = group_sum<LANES>(ss);
    dot = group_sum<LANES>(dot);
    const float r = rsqrtf(ss * (1.0f / D) + kQkEps);
    const float m = dot * r * r * (1.0f / D);
    float o1[8], o2[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float du1 = r * (g1[w][e] - y1[e] * m), du2 = r * (g2[w][e] - y2[e] * m);
      o1[e] = du1 * cs[e] - du2 * sn[e];
      o2[e] = du1 * sn[e] + du2 * cs[e];
    }
    if (live) {
      __nv_bfloat16* out = dqkv + row * 3 * A + w * A + col;
      st8_bf16(out, o1);
      st8_bf16(out + HALF, o2);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// forward attention, head_dim 128 or 64
// ---------------------------------------------------------------------------------------------------------------
struct AttnParams {
  int B, T, H;
  float c1;          // scale * log2(e)
  float c2;          // scale * D * log2(e)   (fixed softmax shift, in base-2 units)
  float shift_ln;    // scale * D
  int window_tiles;  // 0: full causal
  const int* doc_start;
  __nv_bfloat16* y;  // [B*T, H*128]
  float* lse;        // [B, H, T]
  int* err;
  int* items;        // device counter the persistent CTAs draw their work items from (zero at launch)
};

constexpr int AT = 128;                         // tile edge (queries and keys)
constexpr uint32_t ATOM_BYTES = AT * 64 * 2;    // 16 KB: one 128-byte-swizzled atom of [128 rows][64 cols]; a tile has D / 64

// first key tile of query tile `qt`, whose first query's document begins at `doc`
__device__ __forceinline__ int attn_first_tile(const AttnParams& p, int doc, int qt) {
  return p.window_tiles > 0 ? max(doc / AT, qt - p.window_tiles + 1) : doc / AT;
}

// Persistent forward: one CTA per SM walks (query tile, head, batch) items.  Consecutive items are the query tiles of one
// (head, batch), so the CTAs that run at one time share their K/V tiles through L2 (dealing the heaviest tiles of all
// heads first made every CTA stream its own K/V from DRAM at once); the tile order is rotated from one (head, batch) to
// the next so that every CTA sees a mix of lengths.  All barrier phases run on across items: the producer loads the next
// item's Q and K/V while the current item computes, the S warp issues the next item's first tiles while the softmax
// warps finish the current one, and four warps of their own drain the output, so the softmax warps do nothing but exponentials.
//   TMEM: S/P buffers at columns 0, 128 and 256 (running tile count mod 3), O at 384.  The scores run two tiles ahead of the
//   exponentials, so S(g + 1) and its latency (PV, S and their hand-overs are 1 400 clocks) lie under two tiles of exponentials.
// What bounds it now is the special-function units: a 128 x 128 tile's exponentials are 1 024 clocks, with sixteen warps 1 300 of the
// 1 830 that a tile takes (2 770 with both products issued by one warp, the items drawn behind the last load and the output
// drained by the softmax warps).  us: 16 x 2048 tokens in documents, 10 heads of 128, 133 -> 114; 8 x 2048 causal 104 -> 89; 4 x 2048 in
// documents 44.7 -> 37.0; a window of 256 at 16 x 2048 67 -> 58.
// With a tile or two a CTA the longer chain of roles cost 0.3 to 0.7 us; what took it back: a CTA's first item is its own number (no
// counter, no ring), its Q is requested before its document start is known, and an item's coordinates are divided out once, not again before its
// loads.  us with the counter's zero fill, one warp for both products / drawn first item / now: 4 x 256, 4 heads of 64 8.5 / 9.2 / 8.6; 8 x 100
// 7.4 / 8.1 / 7.3; 10 heads of 128: 1 x 128 8.4 / 8.8 / 7.9, 8 x 128 8.8 / 9.2 / 8.5, 16 x 512 in documents 28.3 / 25.8 / 22.0.
// Tried and slower: two query tiles at a time with four warps each and shared K/V (8 x 2048 causal 129: the two fall in step, both
// in their exponentials and then both waiting for MMAs), two groups of eight warps with items of their own (127).
//   smem: Q x 2 (item parity), K x 2 and V x 3 stages (running tile count): a K stage is free again once its S tile is
//   done, a V stage only after its O MMAs, so K and V rings of different depth keep the loads a full tile ahead.
struct FwdItem {
  int qt, h, b;
};
__device__ __forceinline__ FwdItem fwd_item(const AttnParams& p, int w, int n_tiles) {
  FwdItem it;
  const int grp = w / n_tiles;
  it.qt = n_tiles - 1 - (w % n_tiles + grp) % n_tiles;
  it.h = grp % p.H;
  it.b = grp / p.H;
  return it;
}

// Threads: Q and K loads, S warp, sixteen softmax warps (four per 32-lane TMEM quadrant, 32 keys a thread), four drain warps, PV warp, V loads.
constexpr int FWD_SW = 16;
constexpr uint32_t FWD_BARS = 384;            // barriers, item ring, TMEM address, abort flag
constexpr uint32_t FWD_SLACK = 640;           // room for aligning the tiles to 1024 bytes (the seven tiles, the barriers and
                                             // the scratch fill the rest of the 227 KB)
constexpr int FWD_DW = 4;
constexpr int FWD_PV = 2 + FWD_SW + FWD_DW;
constexpr int FWD_VW = FWD_PV + 1;
constexpr int FWD_THREADS = 32 * (FWD_VW + 1);

// The producer hands items to the other roles through a ring of eight (`item_take` in common.cuh has four): with items of a single tile
// the drain warps may be six behind it, since S(t) needs the buffer of PV(t - 3), whose accumulator the drain before had to leave.
constexpr int FWD_RING = 8;
__device__ __forceinline__ int fwd_take(uint32_t bars, volatile int* slots, int it, volatile int* abort_flag, int* err) {
  if (!mbar_wait(bars + 8u * (uint32_t)(it % FWD_RING), (uint32_t)((it / FWD_RING) & 1), abort_flag, err, ERR_WAIT_AUX)) return -1;
  return slots[it % FWD_RING];
}

// D: head dim (64-wide heads on 128-wide tiles with zero halves did twice the MMAs and ten PyTorch passes of padding: a
// forward and backward of 4 x 256 tokens, 4 heads took 314 us, 155 us natively).  T may have any value (padding the sequences
// to whole tiles in PyTorch took 157 of the 271 us of 8 x 1777 tokens, 10 heads; 100 us without): the tensor maps are three-dimensional ([B, T, columns]), so the rows of a last tile
// past the sequence's end arrive as zeros instead of the next sequence's values; their keys lie behind every real query and
// are masked by causality, their queries are computed and not stored.
template <int D>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_qk, const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
  constexpr uint32_t TILE_BYTES = (D / 64) * ATOM_BYTES;
  if (threadIdx.x == 32 * FWD_VW) {
    tma_prefetch_desc(&tm_qk);
    tma_prefetch_desc(&tm_v);
  }
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  if (base - raw > FWD_SLACK) {                       // the tiles would not fit behind the alignment gap
    if (threadIdx.x == 0) atomicCAS(p.err, 0, ERR_WAIT_AUX);
    return;
  }
  uint8_t* gen = smem_raw + (base - raw);
  auto sQ = [&](int s) { return base + TILE_BYTES * s; };
  auto sK = [&](int s) { return base + TILE_BYTES * (2 + s); };
  auto sV = [&](int s) { return base + TILE_BYTES * (4 + s); };
  constexpr uint32_t kBars = TILE_BYTES * 7;
  const uint32_t bars = base + kBars;
  auto q_full = [&](int s) { return bars + 8u * (0 + s); };
  auto q_free = [&](int s) { return bars + 8u * (2 + s); };
  auto k_full = [&](int s) { return bars + 8u * (4 + s); };
  auto k_free = [&](int s) { return bars + 8u * (6 + s); };
  auto v_full = [&](int s) { return bars + 8u * (8 + s); };
  auto v_free = [&](int s) { return bars + 8u * (11 + s); };
  auto s_full = [&](int s) { return bars + 8u * (14 + s); };
  auto p_full = [&](int s) { return bars + 8u * (17 + s); };
  auto s_free = [&](int s) { return bars + 336u + 8u * s; };
  const uint32_t o_full = bars + 8u * 20, o_free = bars + 8u * 21, l_full = bars + 8u * 22, l_free = bars + 8u * 23, ring_bars = bars + 8u * 24;
  volatile int* ring_slots = reinterpret_cast<volatile int*>(gen + kBars + 256);      // item numbers, and behind them first key tiles
  const uint32_t tmem_slot = bars + 320u;
  volatile uint32_t* tmem_slot_g = reinterpret_cast<volatile uint32_t*>(gen + kBars + 320);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + kBars + 328);
  float* lsum = reinterpret_cast<float*>(gen + kBars + FWD_BARS);           // [4 column parts][128 rows]

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int A = p.H * D;
  const int n_tiles = (p.T + AT - 1) / AT;
  const int total = n_tiles * p.H * p.B;

  if (warp == 0) {                                     // a barrier a lane, in the order of the list above
    const bool by_softmax = (lane >= 17 && lane < 20) || lane == 22, by_drain = lane == 21 || lane == 23;
    mbar_init(bars + 8u * (uint32_t)lane, by_softmax ? FWD_SW : by_drain ? FWD_DW : 1);
    if (lane < 3) mbar_init(s_free(lane), 1);
    if (lane == 0) *abort_flag = 0;
    fence_barrier_init();
  } else if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)warp_uniform((int)*tmem_slot_g);
  // the first item, whose keys every role looks up itself
  const FwdItem first = fwd_item(p, (int)blockIdx.x, n_tiles);
  const int doc_first = p.doc_start ? p.doc_start[(long long)first.b * p.T + first.qt * AT] : 0;
  const int kt_first = warp_uniform(attn_first_tile(p, doc_first, first.qt));
  // item `it` of this CTA and its first key tile; -1 behind the last one
  auto take = [&](int it, int* kt0) {
    *kt0 = kt_first;
    if (it == 0) return (int)blockIdx.x;
    const int w = fwd_take(ring_bars, ring_slots, it - 1, abort_flag, p.err);
    *kt0 = ring_slots[FWD_RING + (it - 1) % FWD_RING];
    return w;
  };
  auto tS = [&](int s) { return tmem + (uint32_t)s * 128u; };
  const uint32_t tO = tmem + 384u;

  // The producer and MMA roles run on all 32 lanes of their warp with warp-uniform state and issue from the elected lane
  // (`elect_one` in common.cuh: operands computed under a `lane == 0` branch cost about 80 clocks per `tcgen05.mma`, more
  // than the 64 clocks a 128 x 128 x 16 MMA executes).  Work items are drawn by lane 0 and handed round with a shuffle.
  // A lane whose bounded wait ran out turns `dead`: it walks on without waiting or issuing; when lane 0 is dead no
  // further item is drawn and the warp leaves together.
  if (warp == 0) {
    // Q and K loads, and the items: the next one is drawn, its document start read, and it is handed round and its Q requested one step
    // a tile over the last tiles of the item before, so nobody waits for either latency (drawn and published behind the last
    // load, it held the scores up for about 3 500 clocks an item).
    // From two tiles ahead on.  One / two / three, us: 16 x 2048 tokens in documents 114.6 / 113.8 / 114.2, with a window of 256 59.2 / 58.3 / 58.4;
    // calls of few items the same.
    constexpr int ahead = 2;
    int g = 0, it = 0, w = (int)blockIdx.x, kt0 = kt_first;
    bool dead = false;
    FwdItem after = first;
    auto load_q = [&](const FwdItem& im, int qb) {
      if (elect_one() && !dead) {
        mbar_arrive_expect_tx(q_full(qb), TILE_BYTES);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_3d(sQ(qb) + c * ATOM_BYTES, &tm_qk, q_full(qb), im.h * D + c * 64, im.qt * AT, im.b);
      }
    };
    auto draw = [&](int step, int i) {
      if (step == 0) {
        if (lane == 0) w = (int)gridDim.x + atomicAdd(p.items, 1);
      } else if (step == 1) {
        w = warp_uniform(lane == 0 && !dead && w < total ? w : -1);
        if (w >= 0) after = fwd_item(p, w, n_tiles);
        if (lane == 0 && w >= 0) {
          kt0 = attn_first_tile(p, p.doc_start ? p.doc_start[(long long)after.b * p.T + after.qt * AT] : 0, after.qt);
        }
      } else {
        if (lane == 0 && !dead) {
          const int s = (i - 1) % FWD_RING;
          ring_slots[FWD_RING + s] = kt0;
          ring_slots[s] = w;
          mbar_arrive(ring_bars + 8u * (uint32_t)s);
        }
        kt0 = warp_uniform(kt0);
        if (w < 0) return;
        const int qb = i & 1;
        if (i >= 2 && !dead) dead = !mbar_wait(q_free(qb), (uint32_t)(((i - 2) >> 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        load_q(after, qb);
      }
    };
    FwdItem im = first;
    load_q(first, 0);
    for (; w >= 0; ++it, im = after) {
      const int k_first = kt0, n = im.qt - kt0 + 1;
      int step = 0;
      for (int j = 0; j < n; ++j, ++g) {
        const int ks = g & 1;
        if (g >= 2 && !dead) dead = !mbar_wait(k_free(ks), (uint32_t)(((g - 2) >> 1) & 1), abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(k_full(ks), TILE_BYTES);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sK(ks) + c * ATOM_BYTES, &tm_qk, k_full(ks), A + im.h * D + c * 64, (k_first + j) * AT, im.b);
        }
        if (j >= n - ahead) draw(step++, it + 1);
      }
      for (; step < 3; ++step) draw(step, it + 1);
    }
  } else if (warp == FWD_VW) {
    // V loads
    int g = 0, it = 0, vs = 0;
    uint32_t vph = 1;
    bool dead = false;
    for (;; ++it) {
      int w = -1, kt0 = 0;
      if (!dead) w = take(it, &kt0);
      kt0 = warp_uniform(kt0);
      w = warp_uniform(w);
      if (w < 0) break;
      const FwdItem im = fwd_item(p, w, n_tiles);
      for (int kt = kt0; kt <= im.qt; ++kt, ++g) {
        if (g >= 3 && !dead) dead = !mbar_wait(v_free(vs), vph, abort_flag, p.err, ERR_WAIT_EMPTY);
        if (elect_one() && !dead) {
          mbar_arrive_expect_tx(v_full(vs), TILE_BYTES);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sV(vs) + c * ATOM_BYTES, &tm_v, v_full(vs), 2 * A + im.h * D + c * 64, kt * AT, im.b);
        }
        if (++vs == 3) { vs = 0; vph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // S = Q K^T of each tile, into the buffer whose O += P V (three tiles before) is done.  The products have a warp each: a wait takes
    // 100 to 160 clocks even where it finds its barrier complete, and with three or four of them between the MMAs of one warp
    // the tensor pipe stood still for as long as it worked (2 250 clocks a tile for 1 024 of MMAs).
    // Everything an MMA takes is in uniform registers and known to be (`warp_uniform`): moved there one by one they cost about
    // 100 clocks an MMA of 64.
    constexpr uint32_t kHi = umma_desc_hi(1024, kLayoutSw128);
    const uint32_t idesc_s = umma_idesc_f16(128, 128, 1, 0, 0);   // Q (K-major) x K (K-major)
    const uint32_t q_lo = (uint32_t)warp_uniform((int)umma_desc_lo(sQ(0), 0)), k_lo = (uint32_t)warp_uniform((int)umma_desc_lo(sK(0), 0));
    bool dead = false;
    int g = 0, gs = 0, it = 0;
    uint32_t fph = 1;
    for (;; ++it) {
      int w = -1, kt0 = 0;
      if (!dead) w = take(it, &kt0);
      kt0 = warp_uniform(kt0);
      w = warp_uniform(w);
      if (w < 0) break;
      const int n = fwd_item(p, w, n_tiles).qt - kt0 + 1, qb = it & 1;
      if (!dead) dead = !mbar_wait(q_full(qb), (uint32_t)((it >> 1) & 1), abort_flag, p.err, ERR_WAIT_FULL);
      for (int j = 0; j < n; ++j, ++g) {
        const int kb = g & 1;
        if (!dead) dead = !mbar_wait(k_full(kb), (uint32_t)((g >> 1) & 1), abort_flag, p.err, ERR_WAIT_FULL);
        if (g >= 3 && !dead) dead = !mbar_wait(s_free(gs), fph, abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after();
        const uint32_t qd = q_lo + (uint32_t)qb * (TILE_BYTES >> 4), kd = k_lo + (uint32_t)kb * (TILE_BYTES >> 4), sd = tS(gs);
        if (elect_one() && !dead) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t off = ((k >> 2) * ATOM_BYTES + (k & 3) * 32) >> 4;
            umma_f16_lh(sd, qd + off, kHi, kd + off, kHi, idesc_s, k ? 1u : 0u);
          }
          tc_commit(s_full(gs));
          tc_commit(k_free(kb));
          if (j == n - 1) tc_commit(q_free(qb));
        }
        if (++gs == 3) { gs = 0; fph ^= 1u; }
      }
    }
  } else if (warp == FWD_PV) {
    // O += P V.  P(g) sits in TMEM as packed bf16 pairs over the S(g) columns it was computed from (each softmax warp packs its 32
    // columns into the first 16 of its own range).
    constexpr uint32_t kHi = umma_desc_hi(1024, kLayoutSw128);
    const uint32_t idesc_o = umma_idesc_f16(128, D, 1, 0, 1);   // P (TMEM) x V (MN-major)
    const uint32_t v_lo = (uint32_t)warp_uniform((int)umma_desc_lo(sV(0), ATOM_BYTES));
    bool dead = false;
    int ps = 0, it = 0;                      // P buffer and V stage
    uint32_t pph = 0;
    for (;; ++it) {
      int w = -1, kt0 = 0;
      if (!dead) w = take(it, &kt0);
      kt0 = warp_uniform(kt0);
      w = warp_uniform(w);
      if (w < 0) break;
      const int n = fwd_item(p, w, n_tiles).qt - kt0 + 1;
      for (int j = 0; j < n; ++j) {
        if (!dead) dead = !mbar_wait(v_full(ps), pph, abort_flag, p.err, ERR_WAIT_FULL);
        if (j == 0 && it >= 1 && !dead) dead = !mbar_wait(o_free, (uint32_t)((it - 1) & 1), abort_flag, p.err, ERR_WAIT_TMEM_EMPTY);
        if (!dead) dead = !mbar_wait(p_full(ps), pph, abort_flag, p.err, ERR_WAIT_AUX);
        tc_fence_after();
        const uint32_t vd = v_lo + (uint32_t)ps * (TILE_BYTES >> 4), pd = tS(ps);
        if (elect_one() && !dead) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_f16_ts_lh(tO, pd + (uint32_t)((k >> 1) * 32 + (k & 1) * 8), vd + (uint32_t)((k * 2048) >> 4), kHi, idesc_o, (j == 0 && k == 0) ? 0u : 1u);
          tc_commit(s_free(ps));
          tc_commit(v_free(ps));
          if (j == n - 1) tc_commit(o_full);
        }
        if (++ps == 3) { ps = 0; pph ^= 1u; }
      }
    }
  } else if (warp < 2 + FWD_SW) {
    // Softmax: sixteen warps, four per 32-lane TMEM quadrant; each thread owns one query row and 32 of the tile's 128 keys.
    // (Two groups of warps on tiles or items of their own were no faster: they fall in step and wait for the MMAs together.)
    const int q = warp & 3, part = (warp - 2) >> 2;
    const int r = q * 32 + lane;            // row within the tile == TMEM lane
    const int c0 = part * 32;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    int gs = 0;
    uint32_t sph = 0;
    bool ok = true;
    for (int it = 0; ok; ++it) {
      int kt0;
      const int w = take(it, &kt0);
      if (w < 0) break;
      const FwdItem im = fwd_item(p, w, n_tiles);
      const int qpos = im.qt * AT + r;
      int lo = 0;                                // on its way while the first scores are waited for and exponentiated
      if (p.doc_start && qpos < p.T) lo = p.doc_start[(long long)im.b * p.T + qpos];
      float l = 0.f;
      for (int kt = kt0; kt <= im.qt; ++kt) {
        const bool got = mbar_wait(s_full(gs), sph, abort_flag, p.err, ERR_WAIT_TMEM_FULL);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
        const int k0 = kt * AT + c0;
        uint32_t v0[32], pk[16];
        __syncwarp();
        BONES_TMEM_LD32(tS(gs) + lane_addr + (uint32_t)c0, v0);
        tmem_ld_wait();
        {
          float e[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float x = fmaf(__uint_as_float(v0[i]), p.c1, -p.c2);
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e[i]) : "f"(x));
          }
          // warp-uniform: does any row of this warp need the element mask for these 32 keys (diagonal or document start)?
          if (__any_sync(0xffffffffu, (k0 + 31 > qpos) || (k0 < lo))) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const int kpos = k0 + i;
              if (kpos > qpos || kpos < lo) e[i] = 0.f;
            }
          }
          float l4[4] = {0.f, 0.f, 0.f, 0.f};              // four chains: one of 32 additions takes as long as a quarter of the exponentials
#pragma unroll
          for (int i = 0; i < 32; ++i) l4[i & 3] += e[i];
          l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = pack_bf16(e[2 * i], e[2 * i + 1]);
        }
        BONES_TMEM_ST16(tS(gs) + lane_addr + (uint32_t)c0, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(gs));
        if (++gs == 3) { gs = 0; sph ^= 1u; }
      }
      if (!ok) break;
      // the partial row sums of the four threads of a row go to the drain warps
      if (it >= 1 && !__all_sync(0xffffffffu, mbar_wait(l_free, (uint32_t)((it - 1) & 1), abort_flag, p.err, ERR_WAIT_AUX))) break;
      lsum[part * AT + r] = l;
      __syncwarp();
      if (lane == 0) mbar_arrive(l_full);
    }
  } else {
    // Drain: a thread per query row.
    const int q = warp & 3, r = q * 32 + lane;
    const uint32_t tOr = tO + ((uint32_t)(q * 32) << 16);
    for (int it = 0;; ++it) {
      int kt0;
      const int w = take(it, &kt0);
      if (w < 0) break;
      const FwdItem im = fwd_item(p, w, n_tiles);
      const int qpos = im.qt * AT + r;
      const bool real = qpos < p.T;
      bool got = mbar_wait(l_full, (uint32_t)(it & 1), abort_flag, p.err, ERR_WAIT_AUX);
      if (!__all_sync(0xffffffffu, got)) break;
      const float l = (lsum[r] + lsum[AT + r]) + (lsum[2 * AT + r] + lsum[3 * AT + r]);
      __syncwarp();
      if (lane == 0) mbar_arrive(l_free);
      if (real) p.lse[((long long)im.b * p.H + im.h) * p.T + qpos] = logf(l) + p.shift_ln;
      const float inv = 1.0f / l;
      __nv_bfloat16* y = p.y + ((long long)im.b * p.T + qpos) * A + (long long)im.h * D;
      got = mbar_wait(o_full, (uint32_t)(it & 1), abort_flag, p.err, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, got)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        __syncwarp();
        BONES_TMEM_LD32(tOr + (uint32_t)c, v);
        tmem_ld_wait();
        if (c + 32 >= D) {                             // the next item's products may have the accumulator
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(o_free);
        }
        uint4 u[4];
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          u[gq].x = pack_bf16(__uint_as_float(v[gq * 8 + 0]) * inv, __uint_as_float(v[gq * 8 + 1]) * inv);
          u[gq].y = pack_bf16(__uint_as_float(v[gq * 8 + 2]) * inv, __uint_as_float(v[gq * 8 + 3]) * inv);
          u[gq].z = pack_bf16(__uint_as_float(v[gq * 8 + 4]) * inv, __uint_as_float(v[gq * 8 + 5]) * inv);
          u[gq].w = pack_bf16(__uint_as_float(v[gq * 8 + 6]) * inv, __uint_as_float(v[gq * 8 + 7]) * inv);
        }
        if (real) {                                    // full 32-byte sectors
          st_global_v8(y + c, u[0], u[1]);
          st_global_v8(y + c + 16, u[2], u[3]);
        }
      }
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

// [B, T, cols] bf16 rows, boxes of 64 columns x 128 rows of one sequence; rows past T read as zeros
static int tmap_rows_3d(CUtensorMap* out, const void* ptr, int B, int T, long long cols) {
  uint64_t dims[3] = {(uint64_t)cols, (uint64_t)T, (uint64_t)B};
  uint64_t strides[2] = {(uint64_t)cols * 2, (uint64_t)cols * 2 * (uint64_t)T};
  uint32_t box[3] = {64, 128, 1};
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int D>
static int launch_attn_fwd(const CUtensorMap& tq, const CUtensorMap& tv, const AttnParams& p, int sms, cudaStream_t s) {
  constexpr size_t smem = (size_t)(D / 64) * ATOM_BYTES * 7 + FWD_BARS + 2048 + FWD_SLACK;   // tiles, barriers, row-sum scratch, alignment slack
  static OncePerDevice limit;
  BONES_ONCE(limit, {
    BONES_CHECK(cudaFuncSetAttribute(attn_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  });
  const long long items = (long long)((p.T + AT - 1) / AT) * p.H * p.B;
  const unsigned grid = (unsigned)(items < sms ? items : sms);       // persistent: one CTA per SM
  attn_fwd_kernel<D><<<grid, FWD_THREADS, smem, s>>>(tq, tv, p);
  return (int)cudaGetLastError();
}

template <int D>
static int launch_rope_fwd(const void* qkv, const float* cosT, const float* sinT, void* qk, int* counter, long long M, int T, int H,
                           cudaStream_t s) {
  const long long threads = M * H * (D / 16);
  rope_qknorm_fwd_kernel<D><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>((const __nv_bfloat16*)qkv, cosT, sinT, (__nv_bfloat16*)qk,
                                                                              counter, M, T, H);
  return (int)cudaGetLastError();
}

}  // namespace bones

extern "C" {
using namespace bones;

int bones_rope_qknorm_fwd(const void* qkv, const float* cosT, const float* sinT, void* qk, int* counter, long long M, int T, int H, int D,
                          void* stream) {
  if (misaligned16(qkv, qk, cosT, sinT)) return -3;
  if (D == 128) return launch_rope_fwd<128>(qkv, cosT, sinT, qk, counter, M, T, H, (cudaStream_t)stream);
  if (D == 64) return launch_rope_fwd<64>(qkv, cosT, sinT, qk, counter, M, T, H, (cudaStream_t)stream);
  return -2;
}

// fp32 dq-hat | dk-hat (the single-kernel backward), head_dim 128 only
int bones_rope_qknorm_bwd(const void* qkv, const float* cosT, const float* sinT, const float* dqk, const void* dv, void* dqkv, long long M,
                          int T, int H, int D, void* stream) {
  if (D != 128) return -2;
  if (misaligned16(qkv, dqk, cosT, sinT, dv, dqkv)) return -3;
  const long long threads = M * 3 * H * 8;
  rope_qknorm_bwd128_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)qkv, cosT, sinT, dqk, (const __nv_bfloat16*)dv, (__nv_bfloat16*)dqkv, M, T, H);
  return (int)cudaGetLastError();
}

// dqk: bf16 [M, 2*H*D]; writes the q and k thirds of dqkv [M, 3*H*D]
int bones_rope_qknorm_bwd_bf16(const void* qkv, const float* cosT, const float* sinT, const void* dqk, void* dqkv, long long M, int T, int H,
                               int D, void* stream) {
  if (misaligned16(qkv, dqk, cosT, sinT, dqkv)) return -3;
  const long long threads = M * H * (D / 16);
  const unsigned grid = (unsigned)((threads + 255) / 256);
  const auto *x = (const __nv_bfloat16*)qkv, *g = (const __nv_bfloat16*)dqk;
  if (D == 128) rope_qknorm_bwd_bf16_kernel<128><<<grid, 256, 0, (cudaStream_t)stream>>>(x, cosT, sinT, g, (__nv_bfloat16*)dqkv, M, T, H);
  else if (D == 64) rope_qknorm_bwd_bf16_kernel<64><<<grid, 256, 0, (cudaStream_t)stream>>>(x, cosT, sinT, g, (__nv_bfloat16*)dqkv, M, T, H);
  else return -2;
  return (int)cudaGetLastError();
}

// qk: [B*T, 2*H*D] (rotated, normalised q and k); qkv: [B*T, 3*H*D] (values read in place); y: [B*T, H*D]; lse: [B,H,T];
// counter: one int that is zero when the kernel starts
int bones_attn_fwd(const void* qk, const void* qkv, void* y, float* lse, const int* doc_start, int* counter, int B, int T, int H, int D,
                   float scale, int window_tiles, void* stream) {
  if (D != 128 && D != 64) return -2;
  if ((uintptr_t)y & 31) return -3;
  CUtensorMap tq, tv;
  const long long A = (long long)H * D;
  int rc = tmap_rows_3d(&tq, qk, B, T, 2 * A);
  if (rc) return rc;
  rc = tmap_rows_3d(&tv, qkv, B, T, 3 * A);
  if (rc) return rc;
  AttnParams p;
  p.B = B; p.T = T; p.H = H;
  p.c1 = scale * 1.4426950408889634f;
  p.c2 = scale * D * 1.4426950408889634f;
  p.shift_ln = scale * D;
  p.window_tiles = window_tiles;
  p.doc_start = doc_start;
  p.y = (__nv_bfloat16*)y;
  p.lse = lse;
  p.err = error_word();
  p.items = counter;
  int dev = 0, sms = 0;
  BONES_CHECK(cudaGetDevice(&dev));
  BONES_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return D == 128 ? launch_attn_fwd<128>(tq, tv, p, sms, (cudaStream_t)stream) : launch_attn_fwd<64>(tq, tv, p, sms, (cudaStream_t)stream);
}

// The whole forward: RoPE + QK-norm (which zeroes the counter), then attention.
int bones_attention_fwd(const void* qkv, const float* cosT, const float* sinT, void* qk, void* y, float* lse, const int* doc_start,
                        int* counter, int B, int T, int H, int D, float scale, int window_tiles, void* stream) {
  const int rc = bones_rope_qknorm_fwd(qkv, cosT, sinT, qk, counter, (long long)B * T, T, H, D, stream);
  return rc ? rc : bones_attn_fwd(qk, qkv, y, lse, doc_start, counter, B, T, H, D, scale, window_tiles, stream);
}
}  // extern "C"
