// SIMT batched complex GEMM for sm_103a, 256 threads.  complex64: 64 x 64 or
// 32 x 32 output tiles (launch_simt), for small and ragged shapes.  complex128:
// 16 x 16 tiles, one output per thread (32 x 32 for many whole ones): the FP64 pipe does 2 lanes per clock and SM
// whatever the tile, so what counts is how many SMs a product spreads over and how
// little of a ragged tile is padding (a 10-gate layer at chi 48: 189 us over its 19 launches, 2043 us with
// 64 x 64 tiles, 40 CTAs a launch and a third of their area padding).
#include "gemm.cuh"
#include "gemm_tc.cuh"

namespace {

struct StridedBatch {
  GemmProb base;
  int64_t sA, sB, sC;  // element strides between batch entries
};

template <typename CX>
AGB_DEV GemmProb get_prob(const GemmProb* probs, const StridedBatch& sb) {
  if (probs) return probs[blockIdx.z];
  GemmProb p = sb.base;
  const int64_t z = blockIdx.z;
  p.A = (const CX*)sb.base.A + z * sb.sA;
  p.B = (const CX*)sb.base.B + z * sb.sB;
  p.D = (CX*)sb.base.D + z * sb.sC;
  p.Csrc = (const CX*)sb.base.Csrc + z * sb.sC;
  return p;
}

// BT x BT tile, K-step BK, T x T outputs per thread (BT = 16 T).
template <typename CX, int BT, int BK, int T>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const GemmProb* __restrict__ probs, StridedBatch sb,
                                                        int tiles_n) {
  constexpr int BM = BT, BN = BT;
  const GemmProb p = get_prob<CX>(probs, sb);
  const int m0 = (int)(blockIdx.x / tiles_n) * BM, n0 = (int)(blockIdx.x % tiles_n) * BN;
  if (m0 >= p.M || n0 >= p.N) return;
  typedef typename cx_traits<CX>::R R;
  __shared__ CX As[2][BK][BM + 1];
  __shared__ CX Bs[2][BK][BN + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const CX* A = (const CX*)p.A;
  const CX* B = (const CX*)p.B;
  CX acc[T][T];
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) acc[i][j] = czero<CX>();

  // A tile: BM x BK of op(A); B tile: BK x BN of op(B).  The next two K steps are
  // read into registers while one is multiplied (a step is shorter than the
  // latency of L2), and the two shared-memory buffers leave one barrier per step.
  constexpr int NE = BM * BK / 256;
  const bool an = p.opA == 0 || p.opA == 3, bn = p.opB == 0 || p.opB == 3;  // K along a row / down a column
  const bool conja = p.opA >= 2, conjb = p.opB >= 2;
  const CX *pa[NE], *pb[NE];  // this thread's elements of the next step to read
  int ka[NE], kb[NE];         // their K index, past K for rows and columns outside
  const int64_t stepa = an ? BK : BK * p.lda, stepb = bn ? BK * p.ldb : BK;
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int idx = tid + e * 256;
    const int r = an ? idx / BK : idx % BM, c = an ? idx % BK : idx / BM;
    pa[e] = A + (an ? (int64_t)(m0 + r) * p.lda + c : (int64_t)c * p.lda + m0 + r);
    ka[e] = m0 + r < p.M ? c : p.K;
    const int kr = bn ? idx / BN : idx % BK, nc = bn ? idx % BN : idx / BK;
    pb[e] = B + (bn ? (int64_t)kr * p.ldb + n0 + nc : (int64_t)(n0 + nc) * p.ldb + kr);
    kb[e] = n0 + nc < p.N ? kr : p.K;
  }
  CX va[2][NE], vb[2][NE];
  auto fetch = [&](int k0, CX (&xa)[NE], CX (&xb)[NE]) {
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      xa[e] = k0 + ka[e] < p.K ? *pa[e] : czero<CX>();
      xb[e] = k0 + kb[e] < p.K ? *pb[e] : czero<CX>();
      pa[e] += stepa;
      pb[e] += stepb;
    }
  };
  auto step = [&](int k0, int buf, CX (&xa)[NE], CX (&xb)[NE]) {
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int idx = tid + e * 256;
      const int r = an ? idx / BK : idx % BM, c = an ? idx % BK : idx / BM;
      As[buf][c][r] = conja ? cconj(xa[e]) : xa[e];
      const int kr = bn ? idx / BN : idx % BK, nc = bn ? idx % BN : idx / BK;
      Bs[buf][kr][nc] = conjb ? cconj(xb[e]) : xb[e];
    }
    __syncthreads();
    if (k0 + 2 * BK < p.K) fetch(k0 + 2 * BK, xa, xb);
    const int kn = min(BK, p.K - k0);
    auto product = [&](int k) {
      CX a[T], b[T];
#pragma unroll
      for (int i = 0; i < T; ++i) a[i] = As[buf][k][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < T; ++j) b[j] = Bs[buf][k][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) cfma(acc[i][j], a[i], b[j]);
    };
    if (kn == BK) {
#pragma unroll
      for (int k = 0; k < BK; ++k) product(k);
    } else {
      // a last step in eighths of products; on the FP64 pipe none is padding
      int k = 0;
#pragma unroll 1
      for (; k + (T == 1 ? 8 : 1) <= kn; k += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) product(k + u);
      }
      if (T == 1)
#pragma unroll 1
        for (; k < kn; ++k) product(k);
    }
  };
  fetch(0, va[0], vb[0]);
  if (BK < p.K) fetch(BK, va[1], vb[1]);
  for (int k0 = 0; k0 < p.K; k0 += 2 * BK) {
    step(k0, 0, va[0], vb[0]);
    if (k0 + BK < p.K) step(k0 + BK, 1, va[1], vb[1]);
  }
  const CX alpha = mk<CX>((R)p.alpha_re, (R)p.alpha_im);
  const CX beta = mk<CX>((R)p.beta_re, (R)p.beta_im);
  const bool use_beta = (p.beta_re != 0.0 || p.beta_im != 0.0);
  CX* D = (CX*)p.D;
  const CX* C = (const CX*)p.Csrc;
#pragma unroll
  for (int i = 0; i < T; ++i) {
    const int r = m0 + ty + 16 * i;
    if (r >= p.M) continue;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      const int c = n0 + tx + 16 * j;
      if (c >= p.N) continue;
      CX v = cmul(alpha, acc[i][j]);
      if (use_beta) v = cadd(v, cmul(beta, C[(int64_t)r * p.ldc + c]));
      if (r == c) v.x += (R)p.eye;
      D[(int64_t)r * p.ldd + c] = v;
    }
  }
}

}  // namespace

// complex64: 64 x 64 tiles where they give every SM one and pad less than half as much
// again as 32 x 32 ones (1000 products of 33^3: 37 us, 43 on 32 x 32; 152 of 65^3,
// three quarters more area: 36 and 27; 4096 of 8^3: 42 and 16).  K-step 8: with 16 the
// short products (K = 8 to 20) load and add up to a whole step of padding.
// 32 x 32 tiles: up to two CTAs an SM they are bound by the latency of a step, so it is
// long (K-step 32), and two are read ahead from addresses formed once: a 256 x 512 x 256
// product takes 12.4 us (16.1 with K-step 16; 23 reading one step ahead, 27 with a
// transposed operand; 32 CTAs of 64 x 64 took 40), 1 x 1000 x 1000 43 (K-step 8: 45).
// Beyond that, and for short K, K-step 8: 20 of 200 x 400 x 200 84 (94), 200 of 32^3
// 5.2 (5.9), 300 of 8^3 3.4 (4.8).
// complex128: 32 x 32 tiles (K-step 8) where the bounds are multiples of 32 and there are
// ten CTAs an SM, so that a last wave costs little: 152 products of 128^3 2136 us
// (16 x 16: 2190), 1000 of 64 x 64 x 8 315 (343); 160 of 64^3, 640 CTAs, 344 (302).
template <typename CX>
static int launch_simt(const GemmProb* probs, const StridedBatch& sb, int count, int64_t M, int64_t N, int64_t K,
                       cudaStream_t s) {
  auto tiles = [&](int b) { return ((N + b - 1) / b) * ((M + b - 1) / b); };
  int b = 16;
  if (sizeof(CX) == 8) b = tiles(64) * count >= 152 && 8 * tiles(64) < 3 * tiles(32) ? 64 : 32;
  else if (M % 32 == 0 && N % 32 == 0 && tiles(32) * count >= 1520) b = 32;
  const int64_t t = tiles(b), tn = (N + b - 1) / b;
  if (t > 0x7fffffff) return AGB_ERR_UNSUPPORTED;
  const dim3 grid((unsigned)t, 1, count);
  if constexpr (sizeof(CX) == 16) {
    if (b == 32) gemm_simt_kernel<CX, 32, 8, 2><<<grid, 256, 0, s>>>(probs, sb, (int)tn);
    else gemm_simt_kernel<CX, 16, 16, 1><<<grid, 256, 0, s>>>(probs, sb, (int)tn);
  } else {
    if (b == 64) gemm_simt_kernel<CX, 64, 8, 4><<<grid, 256, 0, s>>>(probs, sb, (int)tn);
    else if (K > 32 && t * count <= 304) gemm_simt_kernel<CX, 32, 32, 2><<<grid, 256, 0, s>>>(probs, sb, (int)tn);
    else gemm_simt_kernel<CX, 32, 8, 2><<<grid, 256, 0, s>>>(probs, sb, (int)tn);
  }
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

template <typename CX>
int launch_gemm_probs(const GemmProb* probs, int count, int maxM, int maxN, cudaStream_t s, const GemmCtx* ctx,
                      int maxK) {
  if (count <= 0 || maxM <= 0 || maxN <= 0) return AGB_OK;
  if (sizeof(CX) == 8 && ctx && ctx->tc_scratch && maxM >= 64 && maxN >= 64 && maxK >= 32 &&
      ctx->tc_bytes >= tc_gemm_scratch_bytes(count, maxM, maxN, maxK))
    return launch_gemm_tc(probs, count, maxM, maxN, maxK, ctx->tc_scratch, ctx->tc_bytes, ctx->status, s);
  return launch_simt<CX>(probs, StridedBatch{}, count, maxM, maxN, maxK, s);
}

template int launch_gemm_probs<float2>(const GemmProb*, int, int, int, cudaStream_t, const GemmCtx*, int);
template int launch_gemm_probs<double2>(const GemmProb*, int, int, int, cudaStream_t, const GemmCtx*, int);

namespace {
// 'N' as stored, 'T' transposed, 'C' conjugate-transposed, 'R' conjugated (not transposed)
int op_code(char c) {
  return (c == 'N' || c == 'n') ? 0 : (c == 'T' || c == 't') ? 1 : (c == 'C' || c == 'c') ? 2 : (c == 'R' || c == 'r') ? 3 : -1;
}
}  // namespace

// Strided-batch host entry (no allocation: the kernel derives each batch
// entry's pointers from the base problem and the element strides).
extern "C" int agb_cgemm_batched(int dtype, char opA, char opB, int batch, int M, int N, int K,
                                 const void* A, int64_t lda, int64_t strideA, const void* B,
                                 int64_t ldb, int64_t strideB, void* C, int64_t ldc, int64_t strideC,
                                 double alpha_re, double alpha_im, double beta_re, double beta_im,
                                 void* stream) {
  const int oa = op_code(opA), ob = op_code(opB);
  if (oa < 0 || ob < 0 || batch < 0 || M < 0 || N < 0 || K < 0) return AGB_ERR_ARG;
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (batch == 0 || M == 0 || N == 0) return AGB_OK;
  if (batch > 65535) return AGB_ERR_UNSUPPORTED;
  StridedBatch sb;
  GemmProb& b = sb.base;
  b.A = A;
  b.B = B;
  b.D = C;
  b.Csrc = C;
  b.lda = lda;
  b.ldb = ldb;
  b.ldd = ldc;
  b.ldc = ldc;
  b.M = M;
  b.N = N;
  b.K = K;
  b.opA = oa;
  b.opB = ob;
  b.alpha_re = alpha_re;
  b.alpha_im = alpha_im;
  b.beta_re = beta_re;
  b.beta_im = beta_im;
  b.eye = 0;
  sb.sA = strideA;
  sb.sB = strideB;
  sb.sC = strideC;
  cudaStream_t s = (cudaStream_t)stream;
  return dtype == AGB_C64 ? launch_simt<float2>(nullptr, sb, batch, M, N, K, s)
                          : launch_simt<double2>(nullptr, sb, batch, M, N, K, s);
}
