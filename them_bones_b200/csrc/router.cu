// MoE router after its logits GEMM: soft-max over the experts, top-k choice, gates and the load-balance / z statistics in one
// pass over the logits, and the gradient of all of it in another.
//
// Bound by launches, not by bytes: at 16384 tokens and 16 experts the logits are 1 MB, and the same arithmetic as PyTorch
// operators was about 50 kernels forward and backward of 2 to 10 us each (about 200 us of 2050, and 800 us of host time); the two
// passes take 17 us.  One thread per token; a CTA stages its 128 tokens' logits in shared memory (rows of E + 1 floats: no bank
// conflicts by row or by column).  Sums over tokens are per-CTA partials added in a fixed order by a second small kernel: results
// are the same on every run.
#include "common.cuh"

namespace bones {

constexpr int RT = 128;            // tokens (and threads) per CTA
constexpr int RMAXE = 64;

// this thread's row of logits in shared memory -> probabilities; returns log-sum-exp
__device__ __forceinline__ float row_softmax(float* row, int E) {
  float m = row[0];
  for (int e = 1; e < E; ++e) m = fmaxf(m, row[e]);
  float s = 0.f;
  for (int e = 0; e < E; ++e) {
    const float x = expf(row[e] - m);
    row[e] = x;
    s += x;
  }
  for (int e = 0; e < E; ++e) row[e] = row[e] / s;
  return m + logf(s);
}
// first maximum of the row, skipping `skip`.  A row without a number (NaN) chooses experts 0 and 1.
__device__ __forceinline__ int row_argmax(const float* row, int E, int skip) {
  int best = skip == 0 ? 1 : 0;
  float v = row[best];
  for (int e = best + 1; e < E; ++e)
    if (e != skip && row[e] > v) { v = row[e]; best = e; }
  return best;
}
__device__ __forceinline__ void stage_logits(float* sm, const float* logits, long long ldl, long long n0, int here, int E) {
  for (int i = threadIdx.x; i < here * E; i += RT) {
    const int r = i / E, e = i - r * E;
    sm[r * (E + 1) + e] = logits[(n0 + r) * ldl + e];
  }
}

// part [CTAs][2 E + 1]: sums of probabilities, counts of choices, sum of squared log-sum-exp; null: no statistics wanted
__global__ void __launch_bounds__(RT) moe_route_fwd_kernel(const float* __restrict__ logits, long long ldl, long long N, int E, int k,
                                                           long long* __restrict__ idx, float* __restrict__ gates, float* __restrict__ part) {
  extern __shared__ float rsm[];
  int* top = reinterpret_cast<int*>(rsm + RT * (E + 1));
  __shared__ float zred[RT / 32];
  const long long n0 = (long long)blockIdx.x * RT;
  const int here = (int)min((long long)RT, N - n0), r = threadIdx.x;
  stage_logits(rsm, logits, ldl, n0, here, E);
  __syncthreads();
  float z2 = 0.f;
  if (r < here) {
    float* row = rsm + r * (E + 1);
    const float lse = row_softmax(row, E);
    z2 = lse * lse;
    const int i1 = row_argmax(row, E, -1);
    const long long n = n0 + r;
    top[r * 2] = i1;
    top[r * 2 + 1] = -1;
    idx[n * k] = i1;
    if (k == 1) {
      gates[n] = row[i1];
    } else {
      const int i2 = row_argmax(row, E, i1);
      top[r * 2 + 1] = i2;
      idx[n * 2 + 1] = i2;
      const float v1 = row[i1], v2 = row[i2], den = v1 + v2;
      gates[n * 2] = v1 / den;
      gates[n * 2 + 1] = v2 / den;
    }
  }
  if (!part) return;
  z2 = warp_sum(z2);
  if ((r & 31) == 0) zred[r >> 5] = z2;
  __syncthreads();
  float* out = part + (long long)blockIdx.x * (2 * E + 1);
  if (r < E) {
    float ps = 0.f;
    int c = 0;
    for (int j = 0; j < here; ++j) {
      ps += rsm[j * (E + 1) + r];
      c += (top[j * 2] == r) + (top[j * 2 + 1] == r);
    }
    out[r] = ps;
    out[E + r] = (float)c;
  }
  if (r == RT - 1) out[2 * E] = (zred[0] + zred[1]) + (zred[2] + zred[3]);
}

// aux = aux_w * lb + z_w * z with lb = E sum_e f_e P_e, z = mean squared log-sum-exp; stats = [lb, z, f_0 .. f_{E-1}]
__global__ void __launch_bounds__(1024) moe_route_stats_kernel(const float* __restrict__ part, int ctas, long long N, int E, int k, float aux_w,
                                                               float z_w, float* __restrict__ aux, float* __restrict__ stats) {
  __shared__ float tot[2 * RMAXE + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cols = 2 * E + 1;
  for (int c = warp; c < cols; c += 32) {
    float s = 0.f;
    for (int j = lane; j < ctas; j += 32) s += part[(long long)j * cols + c];
    s = warp_sum(s);
    if (lane == 0) tot[c] = s;
  }
  __syncthreads();
  if (warp == 0) {
    const float inv = 1.0f / (float)N, finv = inv / (float)k;
    float lb = 0.f;
    for (int e = lane; e < E; e += 32) {
      const float f = tot[E + e] * finv;
      stats[2 + e] = f;
      lb += f * (tot[e] * inv);
    }
    lb = warp_sum(lb) * (float)E;
    if (lane == 0) {
      const float z = tot[2 * E] * inv;
      stats[0] = lb;
      stats[1] = z;
      *aux = aux_w * lb + z_w * z;
    }
  }
}

// Gradient of the logits as bf16 rows of 128 columns (the padded operand of the router's two gradient GEMMs; columns from E
// on are zero), from the gates' gradient and the auxiliary loss's (either may be null).
__global__ void __launch_bounds__(RT) moe_route_bwd_kernel(const float* __restrict__ logits, long long ldl, long long N, int E, int k,
                                                           const long long* __restrict__ idx, const float* __restrict__ dgates,
                                                           const float* __restrict__ daux, const float* __restrict__ f, float aux_w, float z_w,
                                                           __nv_bfloat16* __restrict__ dl) {
  extern __shared__ float rsm[];
  __shared__ float sf[RMAXE];
  const long long n0 = (long long)blockIdx.x * RT;
  const int here = (int)min((long long)RT, N - n0), r = threadIdx.x;
  stage_logits(rsm, logits, ldl, n0, here, E);
  const float da = daux ? *daux : 0.f;
  if (r < E) sf[r] = daux ? da * aux_w * (float)E / (float)N * f[r] : 0.f;
  __syncthreads();
  if (r < here) {
    float* row = rsm + r * (E + 1);
    const float lse = row_softmax(row, E);
    const long long n = n0 + r;
    int i1 = -1, i2 = -1;
    float d1 = 0.f, d2 = 0.f;
    if (dgates) {
      i1 = (int)idx[n * k];
      if (k == 1) {
        d1 = dgates[n];
      } else {
        i2 = (int)idx[n * 2 + 1];
        const float v1 = row[i1], v2 = row[i2], den = v1 + v2, g1 = dgates[n * 2], g2 = dgates[n * 2 + 1];
        const float mean = (g1 * v1 + g2 * v2) / den;
        d1 = (g1 - mean) / den;
        d2 = (g2 - mean) / den;
      }
    }
    float dot = 0.f;
    for (int e = 0; e < E; ++e) dot += row[e] * (sf[e] + (e == i1 ? d1 : 0.f) + (e == i2 ? d2 : 0.f));
    const float dz = daux ? da * z_w * 2.0f * lse / (float)N : 0.f;
    for (int e = 0; e < E; ++e) row[e] *= (sf[e] + (e == i1 ? d1 : 0.f) + (e == i2 ? d2 : 0.f)) - dot + dz;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < here * 16; i += RT) {
    const int j = i >> 4, c = (i & 15) * 8;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = c + q < E ? rsm[j * (E + 1) + c + q] : 0.f;
    *reinterpret_cast<uint4*>(dl + (n0 + j) * 128 + c) =
        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  }
}

}  // namespace bones

extern "C" {
using namespace bones;

// logits: fp32 [N, >= E], rows of ldl floats; idx, gates [N, k]; part: [ceil(N / 128), 2 E + 1] scratch or null (then no aux, stats)
int bones_moe_route_fwd(const float* logits, long long ldl, long long N, int E, int k, long long* idx, float* gates, float* part, float aux_w,
                        float z_w, float* aux, float* stats, void* stream) {
  if (E < 1 || E > RMAXE || (k != 1 && k != 2) || k > E) return -2;
  if (N <= 0) return N == 0 ? 0 : -2;
  const int ctas = (int)((N + RT - 1) / RT);
  const size_t smem = (size_t)RT * (E + 1) * 4 + RT * 2 * 4;
  moe_route_fwd_kernel<<<ctas, RT, smem, (cudaStream_t)stream>>>(logits, ldl, N, E, k, idx, gates, part);
  BONES_CHECK(cudaGetLastError());
  if (part) moe_route_stats_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(part, ctas, N, E, k, aux_w, z_w, aux, stats);
  return (int)cudaGetLastError();
}

// dl: bf16 [N, 128]; f: the choice frequencies of the forward's stats
int bones_moe_route_bwd(const float* logits, long long ldl, long long N, int E, int k, const long long* idx, const float* dgates, const float* daux,
                        const float* f, float aux_w, float z_w, void* dl, void* stream) {
  if (E < 1 || E > RMAXE || (k != 1 && k != 2) || k > E) return -2;
  if (N <= 0) return N == 0 ? 0 : -2;
  const size_t smem = (size_t)RT * (E + 1) * 4;
  moe_route_bwd_kernel<<<(unsigned)((N + RT - 1) / RT), RT, smem, (cudaStream_t)stream>>>(logits, ldl, N, E, k, idx, dgates, daux, f, aux_w, z_w,
                                                                                       (__nv_bfloat16*)dl);
  return (int)cudaGetLastError();
}
}  // extern "C"
