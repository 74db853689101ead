// Cross-entropy on logits whose statistics the logits GEMM already left (`bones_logits_stats`): per row the sums of exp(z - cap)
// by half tile.  What remains is the rows' log-sum-exp and loss (8 MB of partial sums for 4096 rows of 65536 logits) and,
// for training, one element-wise pass that turns the logits into their gradient in place.
//
// Bound by the pass over the logits: 0.54 GB read and 0.54 GB written per 4096 rows of 65536, 164 us at the copy rate.  Measured 164 us
// with L2 flushed before and 160 right behind the GEMM, whose last logits are still in L2; and 12 us for the rows.  Two passes over a
// row kept in shared memory (sum of exponentials, then gradient: `softcap_ce_row_kernel`, still used with label smoothing) took 327 us,
// because a row's read, its two exponential passes and its write followed one another in the one CTA an SM has room for.  The
// element-wise pass has no dependence on the rest of the row: small CTAs, many to an SM.
#include "common.cuh"

namespace bones {

struct CeAux {
  const long long* tg[2];      // further targets of the row (multi-token prediction), null where absent
  const float* w[2];           // their absolute weights
  float* nll_aux;              // [M] or null
};

constexpr int CF_ROWS = 32, CF_WARPS = 16;

// nll[row]; with `info` also what the gradient pass needs: (log2 of sum over |weight|, target weight, auxiliary weights).
// 32 rows per CTA, one per lane; the warps share the P partial sums and add them in a fixed order.
__global__ void __launch_bounds__(CF_WARPS * 32) ce_finish_kernel(const float* __restrict__ part, int P, int M, const __nv_bfloat16* __restrict__ logits,
                                                                  long long ldl, const float* __restrict__ z_target, const long long* __restrict__ targets,
                                                                  int V, float cap, float* __restrict__ nll, float4* __restrict__ info,
                                                                  const float* __restrict__ row_w, const float* __restrict__ n_valid, float inv_loss_div,
                                                                  CeAux aux) {
  __shared__ float red[CF_WARPS][CF_ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * CF_ROWS + lane;
  float s = 0.f;
  if (row < M) {
#pragma unroll 8
    for (int j = warp; j < P; j += CF_WARPS) s += part[(long long)j * M + row];
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp || row >= M) return;
  s = 0.f;
#pragma unroll
  for (int w = 0; w < CF_WARPS; ++w) s += red[w][lane];
  const float lse2 = log2f(s) + cap * 1.4426950408889634f, lse = lse2 * 0.6931471805599453f;
  const long long t = targets[row];
  const bool valid = t >= 0 && t < V;
  const __nv_bfloat16* l = logits ? logits + (long long)row * ldl : nullptr;
  nll[row] = valid ? lse - (l ? __bfloat162float(l[t]) : z_target[row]) : 0.f;
  if (!info) return;
  float a[2] = {0.f, 0.f}, oa = 0.f;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (!aux.tg[j]) continue;
    const long long k = aux.tg[j][row];
    if (k < 0 || k >= V) continue;
    a[j] = aux.w[j][row];
    if (a[j] != 0.f) oa += a[j] * (lse - __bfloat162float(l[k]));
  }
  if (aux.nll_aux) aux.nll_aux[row] = oa;
  const float w = valid ? (row_w ? row_w[row] : inv_loss_div / fmaxf(1.0f, *n_valid)) : 0.f;
  const float sum = w + a[0] + a[1];
  // weights may be negative (the gradient pass takes the sign from their sum); a row without any live target: +inf makes every
  // probability term exactly 0
  info[row] = make_float4(sum != 0.f ? lse2 - log2f(fabsf(sum)) : __int_as_float(0x7f800000), w, a[0], a[1]);
}

// In place: z -> (w_sum softmax(z) - sum of target weights at their columns) (1 - (z / cap)^2); columns V .. ldl - 1 become 0.
// A CTA takes 8192 columns of one row, 32 a thread in four 16-byte accesses that are all in flight together.
constexpr int CG_COLS = 8192;
__global__ void __launch_bounds__(256) ce_grad_kernel(__nv_bfloat16* __restrict__ logits, long long ldl, const float4* __restrict__ info,
                                                      const long long* __restrict__ targets, const long long* __restrict__ tg2,
                                                      const long long* __restrict__ tg3, int V, float nic2) {
  const long long row = blockIdx.y;
  const int c0 = blockIdx.x * CG_COLS + threadIdx.x * 8;
  __nv_bfloat16* l = logits + row * ldl;
  uint4 u[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = c0 + i * 2048;
    if (c < V) u[i] = *reinterpret_cast<const uint4*>(l + c);
  }
  const float4 f = info[row];
  const bool neg = f.y + f.z + f.w < 0.f;
  const int t1 = f.y != 0.f ? (int)targets[row] : -8, t2 = f.z != 0.f ? (int)tg2[row] : -8, t3 = f.w != 0.f ? (int)tg3[row] : -8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = c0 + i * 2048;
    if (c >= ldl) break;
    uint32_t w[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
    if (c >= V) {
      *reinterpret_cast<uint4*>(l + c) = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const bool own = (unsigned)(t1 - c) < 8u || (unsigned)(t2 - c) < 8u || (unsigned)(t3 - c) < 8u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float z0 = __uint_as_float(w[j] << 16), z1 = __uint_as_float(w[j] & 0xffff0000u);
      float p0, p1;
      asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p0) : "f"(fmaf(z0, 1.4426950408889634f, -f.x)));
      asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p1) : "f"(fmaf(z1, 1.4426950408889634f, -f.x)));
      if (neg) { p0 = -p0; p1 = -p1; }
      if (own) {
        const int k = c + 2 * j;
        if (k == t1) p0 -= f.y;
        if (k + 1 == t1) p1 -= f.y;
        if (k == t2) p0 -= f.z;
        if (k + 1 == t2) p1 -= f.z;
        if (k == t3) p0 -= f.w;
        if (k + 1 == t3) p1 -= f.w;
      }
      w[j] = pack_bf16(p0 * fmaf(z0 * nic2, z0, 1.0f), p1 * fmaf(z1 * nic2, z1, 1.0f));
    }
    *reinterpret_cast<uint4*>(l + c) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// out = bf16( bf16(in) * bf16(*scale) ): a gradient kept in fp32, handed to autograd times the loss's own gradient.
// One pass where a cast and a multiply by a zero-dimensional tensor were two (99 against 366 us for 65536 + 16384 rows of 1280).
__global__ void __launch_bounds__(256) scale_cast_kernel(const float* __restrict__ in, const float* __restrict__ scale, __nv_bfloat16* __restrict__ out,
                                                         long long n) {
  const float s = __bfloat162float(__float2bfloat16(*scale));
  const long long stride = (long long)gridDim.x * 256 * 8;
  for (long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 8; i < n; i += stride) {
    const float4 a = *reinterpret_cast<const float4*>(in + i), b = *reinterpret_cast<const float4*>(in + i + 4);
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = pack_bf16(__bfloat162float(__float2bfloat16(v[2 * j])) * s, __bfloat162float(__float2bfloat16(v[2 * j + 1])) * s);
    *reinterpret_cast<uint4*>(out + i) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace bones

extern "C" {
using namespace bones;

// part [P, M] from bones_logits_stats; logits [M, ldl] (soft-capped, bf16) or null with z_target [M].  info [M] float4 or null
// (no gradient follows).
int bones_ce_finish(const float* part, int P, int M, const void* logits, long long ldl, const float* z_target, const long long* targets, int V, float cap,
                    float* nll, void* info, const float* row_w, const float* n_valid, float inv_loss_div, const long long* tg2, const float* w2,
                    const long long* tg3, const float* w3, float* nll_aux, void* stream) {
  if (M <= 0) return 0;
  if ((!logits && !z_target) || (info && (!logits || (!row_w && !n_valid) || ((uintptr_t)info & 15)))) return -2;
  CeAux aux;
  aux.tg[0] = tg2; aux.w[0] = w2; aux.tg[1] = tg3; aux.w[1] = w3; aux.nll_aux = nll_aux;
  ce_finish_kernel<<<(M + CF_ROWS - 1) / CF_ROWS, CF_WARPS * 32, 0, (cudaStream_t)stream>>>(part, P, M, (const __nv_bfloat16*)logits, ldl, z_target,
                                                                                            targets, V, cap, nll, (float4*)info, row_w, n_valid,
                                                                                            inv_loss_div, aux);
  return (int)cudaGetLastError();
}

int bones_ce_grad(void* logits, long long ldl, const void* info, const long long* targets, const long long* tg2, const long long* tg3, int V, float cap,
                  int M, void* stream) {
  if (M <= 0) return 0;
  if ((V % 8) || (ldl % 8) || ((uintptr_t)logits & 15) || M > 65535) return -2;
  const dim3 grid((unsigned)((ldl + CG_COLS - 1) / CG_COLS), (unsigned)M);
  ce_grad_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)logits, ldl, (const float4*)info, targets, tg2, tg3, V, -1.0f / (cap * cap));
  return (int)cudaGetLastError();
}

// n a multiple of 8, both tensors 16-byte aligned
int bones_scale_cast(const float* in, const float* scale, void* out, long long n, void* stream) {
  if ((n % 8) || ((uintptr_t)in & 15) || ((uintptr_t)out & 15)) return -2;
  if (n <= 0) return 0;
  const long long blocks = (n / 8 + 255) / 256;
  scale_cast_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(in, scale, (__nv_bfloat16*)out, n);
  return (int)cudaGetLastError();
}
}  // extern "C"
