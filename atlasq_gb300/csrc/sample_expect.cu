// Sampling and expectation helper kernels (sm_103a).
//
// Sampling (replaces _batch_sweep_sample, src/atlas_q/mps_pytorch.py:247-355):
// per site the host computes temp = L @ T.reshape(chiL, 2 chiR) with the GEMM;
// agb_sample_site then, per shot (one warp each),
//   p_s = sum |temp[shot, s*chiR : (s+1)*chiR]|^2 (double accumulation),
//   p_s += 1e-15 (the reference's floor, :313), pz = p0 / (p0 + p1),
//   u = Philox4x32-10((shot, shot>>32, site, 0), seed) word0 >> 8 * 2^-24,
//   outcome = u >= pz; bits = bits << 1 | outcome (qubit 0 = MSB, :321),
//   L_new = temp[shot, outcome*chiR : ...]  (left state kept unnormalised, :342-352).
//
// Expectations (replaces the einsum of expectation_value, src/atlas_q/mpo_ops.py:1145):
// E'[r,B] = sum E[a,b] conj(A[a,t,r]) W[L,s,t,R] A[b,s,B] is evaluated as
//   M_L = E_L @ A.reshape(chiA, 2 chiB)               (GEMM)
//   N_R[(a,t),B] = sum_{L,s} W[L,s,t,R] M_L[a,(s,B)]  (agb_mpo_mix, this file)
//   E'_R = A.reshape(2 chiA, chiB)^H @ N_R            (GEMM)
#include "common.cuh"

namespace {

// A warp per shot, kSampleShots shots per CTA.  The row is read once, into registers,
// all of its loads in flight, where a lane's share is at most K elements a half (K = 0:
// any length, read again for the output).  The decisions of a CTA's shots (two dozen
// FP64 instructions, whatever the number of active lanes, at 16 cycles of the SM's
// pipe) are taken together by one warp: by each shot's own warp they were 20 us for
// 16 384 shots, more than the traffic.  16 384 shots: chi 256
// 25 -> 20 us (5.1 TB/s, from L2), chi 64 22.5 -> 7.4.
constexpr int kSampleShots = 16;
template <typename CX, int K>
__global__ void __launch_bounds__(32 * kSampleShots) sample_site_kernel(const CX* __restrict__ temp, int shots, int chiR, int site,
                                                          uint64_t seed, uint64_t shot_offset,
                                                          int64_t* __restrict__ bits, CX* __restrict__ Lnew,
                                                          double* __restrict__ pz_out) {
  typedef typename cx_traits<CX>::R R;
  __shared__ __align__(16) unsigned char sum_raw[2 * kSampleShots * sizeof(SumAcc<R>)];
  SumAcc<R>* sums = (SumAcc<R>*)sum_raw;  // [2][kSampleShots]
  __shared__ int outcome[kSampleShots];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int s0 = blockIdx.x * kSampleShots, s = s0 + wid;
  const bool on = s < shots;
  const CX* row = temp + (int64_t)(on ? s : 0) * 2 * chiR;
  // both probabilities to double accuracy on the FP32 pipe
  SumAcc<R> a0, a1;
  CX v0[K ? K : 1], v1[K ? K : 1];
  if (K) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = lane + 32 * k;
      v0[k] = c < chiR ? row[c] : czero<CX>();
      v1[k] = c < chiR ? row[chiR + c] : czero<CX>();
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (lane + 32 * k < chiR) {
        a0.add(cabs2(v0[k]));
        a1.add(cabs2(v1[k]));
      }
  } else {
    for (int c = lane; c < chiR; c += 32) {
      a0.add(cabs2(row[c]));
      a1.add(cabs2(row[chiR + c]));
    }
  }
  a0.warp_reduce();
  a1.warp_reduce();
  if (lane == 0) {
    sums[wid] = a0;
    sums[kSampleShots + wid] = a1;
  }
  __syncthreads();
  if (wid == 0 && lane < kSampleShots && s0 + lane < shots) {
    const int t = s0 + lane;
    const double p0 = sums[lane].value() + 1e-15, p1 = sums[kSampleShots + lane].value() + 1e-15;
    const double pz = p0 / (p0 + p1);
    const uint64_t shot = shot_offset + (uint64_t)t;
    const philox_out o = philox4x32_10((uint32_t)shot, (uint32_t)(shot >> 32), (uint32_t)site, 0u,
                                       (uint32_t)seed, (uint32_t)(seed >> 32));
    const double u = (double)(o.x >> 8) * (1.0 / 16777216.0);
    const int outc = (u >= pz) ? 1 : 0;
    bits[t] = (bits[t] << 1) | outc;
    if (pz_out) pz_out[t] = pz;
    outcome[lane] = outc;
  }
  __syncthreads();
  const int outc = outcome[wid];
  if (Lnew && on) {
    CX* dst = Lnew + (int64_t)s * chiR;
    if (K) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (lane + 32 * k < chiR) dst[lane + 32 * k] = outc ? v1[k] : v0[k];
    } else {
      const CX* src = row + outc * chiR;
      for (int c = lane; c < chiR; c += 32) dst[c] = src[c];
    }
  }
}

template <typename CX>
__global__ void mpo_mix_kernel(const CX* __restrict__ M, const CX* __restrict__ W, CX* __restrict__ N,
                               int Lw, int Rw, int chiA, int chiB) {
  const int64_t per = (int64_t)chiA * 2 * chiB;
  const int64_t total = per * Rw;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int R = (int)(i / per);
    const int64_t rem = i % per;
    const int a = (int)(rem / (2 * chiB));
    const int t = (int)((rem / chiB) % 2);
    const int B = (int)(rem % chiB);
    CX acc = czero<CX>();
    for (int L = 0; L < Lw; ++L)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const CX w = W[((L * 2 + s) * 2 + t) * Rw + R];
        if (w.x != 0 || w.y != 0)
          cfma(acc, w, M[(int64_t)L * per + ((int64_t)a * 2 + s) * chiB + B]);
      }
    N[i] = acc;
  }
}

// N[g][a][t][b] = sum_s W[g][s][t] M[g][a][s][b]   (W: one 2x2 operator per item);
// items (if given): a list of {M, W, N, chiA, chiB} instead of a uniform batch
template <typename CX>
__global__ void site_mix_kernel(const CX* __restrict__ M, const CX* __restrict__ W, CX* __restrict__ N, int chiA,
                                int chiB, const int64_t* __restrict__ items) {
  const int g = blockIdx.y;
  const CX* Mg;
  const CX* Wg;
  CX* Ng;
  if (items) {
    const int64_t* it = items + 5 * (int64_t)g;
    Mg = (const CX*)it[0];
    Wg = (const CX*)it[1];
    Ng = (CX*)it[2];
    chiA = (int)it[3];
    chiB = (int)it[4];
  } else {
    const int64_t per = (int64_t)chiA * 2 * chiB;
    Mg = M + (int64_t)g * per;
    Wg = W + (int64_t)g * 4;
    Ng = N + (int64_t)g * per;
  }
  const CX w00 = Wg[0], w01 = Wg[1], w10 = Wg[2], w11 = Wg[3];
  const int64_t half = (int64_t)chiA * chiB;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(i / chiB), b = (int)(i % chiB);
    const CX m0 = Mg[((int64_t)a * 2 + 0) * chiB + b], m1 = Mg[((int64_t)a * 2 + 1) * chiB + b];
    CX n0 = czero<CX>(), n1 = czero<CX>();
    cfma(n0, w00, m0);  // t = 0: W[0][0] M[s=0] + W[1][0] M[s=1]
    cfma(n0, w10, m1);
    cfma(n1, w01, m0);  // t = 1
    cfma(n1, w11, m1);
    Ng[((int64_t)a * 2 + 0) * chiB + b] = n0;
    Ng[((int64_t)a * 2 + 1) * chiB + b] = n1;
  }
}

// out = sum_{r,c} E[r,c] * Q[c,r]   (one block of 32 x 32 threads per item, double
// accuracy; items (if given): a list of {E, Q, n}).  A block takes 54 us for n =
// 256 whatever else runs, so the traces of a set of observables share a launch
// (99 of them: 62 us, 5.4 ms one by one).  32 x 32 tiles, two in flight per barrier: thread (ty, tx) takes
// E[r0 + ty][c0 + tx] (coalesced) and Q[c0 + tx][r0 + ty] from a tile of Q
// staged row-wise (coalesced) in shared memory.
template <typename CX>
__global__ void __launch_bounds__(1024) trace_prod_kernel(const CX* __restrict__ E, const CX* __restrict__ Q,
                                                          int n, double* out, const int64_t* __restrict__ items) {
  typedef typename cx_traits<CX>::R R;
  if (items) {
    const int64_t* it = items + 3 * (int64_t)blockIdx.x;
    E = (const CX*)it[0];
    Q = (const CX*)it[1];
    n = (int)it[2];
    out += 2 * (int64_t)blockIdx.x;
  }
  __shared__ CX qs[2][32][33];
  __shared__ double red[32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int nb = (n + 31) / 32, ntile = nb * nb;
  SumAcc<R> re, im;
  for (int t0 = 0; t0 < ntile; t0 += 2) {
    CX ev[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = t0 + u;
      CX qv = czero<CX>();
      ev[u] = czero<CX>();
      if (t < ntile) {
        const int r0 = (t / nb) * 32, c0 = (t % nb) * 32;
        if (c0 + ty < n && r0 + tx < n) qv = Q[(int64_t)(c0 + ty) * n + r0 + tx];
        if (r0 + ty < n && c0 + tx < n) ev[u] = E[(int64_t)(r0 + ty) * n + c0 + tx];
      }
      qs[u][ty][tx] = qv;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const CX a = ev[u], b = qs[u][tx][ty];
      re.add_prod(a.x, b.x);
      re.add_prod(-a.y, b.y);
      im.add_prod(a.x, b.y);
      im.add_prod(a.y, b.x);
    }
    __syncthreads();
  }
  const double sre = block_sum(re.value(), red);
  const double sim = block_sum(im.value(), red);
  if (threadIdx.x == 0) {
    out[0] = sre;
    out[1] = sim;
  }
}

}  // namespace

extern "C" int agb_sample_site(int dtype, const void* temp, int shots, int chiR, int site, uint64_t seed,
                               uint64_t shot_offset, int64_t* bits, void* Lnew, double* pz_out,
                               void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (shots < 0 || chiR <= 0 || !temp || !bits) return AGB_ERR_ARG;
  if (shots == 0) return AGB_OK;
  const dim3 grid((shots + kSampleShots - 1) / kSampleShots);
  cudaStream_t s = (cudaStream_t)stream;
  auto run = [&](auto kern, auto cx) {
    typedef decltype(cx) CX;
    kern<<<grid, 32 * kSampleShots, 0, s>>>((const CX*)temp, shots, chiR, site, seed, shot_offset, bits, (CX*)Lnew, pz_out);
  };
  if (dtype == AGB_C64) {
    if (chiR <= 64) run(sample_site_kernel<float2, 2>, float2());
    else if (chiR <= 128) run(sample_site_kernel<float2, 4>, float2());
    else if (chiR <= 256) run(sample_site_kernel<float2, 8>, float2());
    else run(sample_site_kernel<float2, 0>, float2());
  } else {
    if (chiR <= 128) run(sample_site_kernel<double2, 4>, double2());
    else run(sample_site_kernel<double2, 0>, double2());
  }
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

extern "C" int agb_mpo_mix(int dtype, const void* M, const void* W, void* N, int Lw, int Rw, int chiA,
                           int chiB, void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (!M || !W || !N || Lw <= 0 || Rw <= 0 || chiA <= 0 || chiB <= 0) return AGB_ERR_ARG;
  const int64_t total = (int64_t)Rw * chiA * 2 * chiB;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 4096) blocks = 4096;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == AGB_C64)
    mpo_mix_kernel<float2><<<blocks, 256, 0, s>>>((const float2*)M, (const float2*)W, (float2*)N, Lw, Rw, chiA, chiB);
  else
    mpo_mix_kernel<double2><<<blocks, 256, 0, s>>>((const double2*)M, (const double2*)W, (double2*)N, Lw, Rw, chiA, chiB);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

extern "C" int agb_site_mix(int dtype, const void* M, const void* W, void* N, int count, int chiA, int chiB,
                            void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (!M || !W || !N || count < 0 || count > 65535 || chiA <= 0 || chiB <= 0) return AGB_ERR_ARG;
  if (count == 0) return AGB_OK;
  const int64_t half = (int64_t)chiA * chiB;
  int bx = (int)((half + 255) / 256);
  if (bx > 256) bx = 256;
  const dim3 grid(bx, count);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == AGB_C64)
    site_mix_kernel<float2><<<grid, 256, 0, s>>>((const float2*)M, (const float2*)W, (float2*)N, chiA, chiB, nullptr);
  else
    site_mix_kernel<double2><<<grid, 256, 0, s>>>((const double2*)M, (const double2*)W, (double2*)N, chiA, chiB,
                                                  nullptr);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

extern "C" int agb_trace_prod(int dtype, const void* E, const void* Q, int n, double* out2, void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (!E || !Q || !out2 || n <= 0) return AGB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == AGB_C64) trace_prod_kernel<float2><<<1, 1024, 0, s>>>((const float2*)E, (const float2*)Q, n, out2, nullptr);
  else trace_prod_kernel<double2><<<1, 1024, 0, s>>>((const double2*)E, (const double2*)Q, n, out2, nullptr);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

extern "C" int agb_site_mix_list(int dtype, const int64_t* items, int count, int64_t max_elems, void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (count < 0 || count > 65535 || max_elems < 0) return AGB_ERR_ARG;
  if (count == 0 || max_elems == 0) return AGB_OK;
  if (!items) return AGB_ERR_ARG;
  int64_t bx = (max_elems + 255) / 256;
  if (bx > 256) bx = 256;
  const dim3 grid((unsigned)bx, count);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == AGB_C64) site_mix_kernel<float2><<<grid, 256, 0, s>>>(nullptr, nullptr, nullptr, 0, 0, items);
  else site_mix_kernel<double2><<<grid, 256, 0, s>>>(nullptr, nullptr, nullptr, 0, 0, items);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

extern "C" int agb_trace_prod_list(int dtype, const int64_t* items, int count, double* out2, void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (count < 0) return AGB_ERR_ARG;
  if (count == 0) return AGB_OK;
  if (!items || !out2) return AGB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == AGB_C64) trace_prod_kernel<float2><<<count, 1024, 0, s>>>(nullptr, nullptr, 0, out2, items);
  else trace_prod_kernel<double2><<<count, 1024, 0, s>>>(nullptr, nullptr, 0, out2, items);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}
