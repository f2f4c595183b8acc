// SIMT batched complex GEMM for sm_103a, 256 threads.  complex64: 64 x 64 output
// tiles, K-step 8, 4 x 4 complex accumulators per thread (small and ragged
// shapes).  complex128: 16 x 16 tiles, K-step 16, one output per thread: the
// FP64 pipe does 2 lanes per clock and SM whatever the tile, so what counts is
// how many SMs a product spreads over and how little of a ragged tile is
// padding (a 10-gate layer at chi 48: 189 us over its 19 launches, 2043 us with
// 64 x 64 tiles, 40 CTAs a launch and a third of their area padding).
#include "gemm.cuh"
#include "gemm_tc.cuh"

namespace {

template <typename CX> struct Tile;
template <> struct Tile<float2> { static constexpr int B = 64, K = 8, T = 4; };
template <> struct Tile<double2> { static constexpr int B = 16, K = 16, T = 1; };

template <typename CX>
AGB_DEV CX load_op(const CX* P, int64_t ld, int op, int row, int col, int rows, int cols) {
  // element (row, col) of op(P), where op(P) is rows x cols
  if (row >= rows || col >= cols) return czero<CX>();
  if (op == 0) return P[(int64_t)row * ld + col];
  if (op == 3) return cconj(P[(int64_t)row * ld + col]);
  CX v = P[(int64_t)col * ld + row];
  return op == 2 ? cconj(v) : v;
}

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

template <typename CX>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const GemmProb* __restrict__ probs, StridedBatch sb,
                                                        int tiles_n) {
  constexpr int BM = Tile<CX>::B, BN = Tile<CX>::B, BK = Tile<CX>::K, T = Tile<CX>::T;
  const GemmProb p = get_prob<CX>(probs, sb);
  const int m0 = (int)(blockIdx.x / tiles_n) * BM, n0 = (int)(blockIdx.x % tiles_n) * BN;
  if (m0 >= p.M || n0 >= p.N) return;
  typedef typename cx_traits<CX>::R R;
  __shared__ CX As[BK][BM + 1];
  __shared__ CX Bs[BK][BN + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const CX* A = (const CX*)p.A;
  const CX* B = (const CX*)p.B;
  CX acc[T][T];
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) acc[i][j] = czero<CX>();

  for (int k0 = 0; k0 < p.K; k0 += BK) {
    // A tile: BM x BK of op(A); B tile: BK x BN of op(B)
#pragma unroll
    for (int e = 0; e < BM * BK / 256; ++e) {
      const int idx = tid + e * 256;
      int r, c;
      if (p.opA == 0 || p.opA == 3) { r = idx / BK; c = idx % BK; } else { r = idx % BM; c = idx / BM; }
      As[c][r] = load_op(A, p.lda, p.opA, m0 + r, k0 + c, p.M, p.K);
      int kr, nc;
      if (p.opB == 0 || p.opB == 3) { kr = idx / BN; nc = idx % BN; } else { kr = idx % BK; nc = idx / BK; }
      Bs[kr][nc] = load_op(B, p.ldb, p.opB, k0 + kr, n0 + nc, p.K, p.N);
    }
    __syncthreads();
    const int kn = min(BK, p.K - k0);
    if (T == 1 && kn < BK) {  // no padding products on the FP64 pipe
      for (int k = 0; k < kn; ++k) cfma(acc[0][0], As[k][ty], Bs[k][tx]);
    } else {
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        CX a[T], b[T];
#pragma unroll
        for (int i = 0; i < T; ++i) a[i] = As[k][ty + 16 * i];
#pragma unroll
        for (int j = 0; j < T; ++j) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) cfma(acc[i][j], a[i], b[j]);
      }
    }
    __syncthreads();
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

template <typename CX>
int launch_gemm_probs(const GemmProb* probs, int count, int maxM, int maxN, cudaStream_t s, const GemmCtx* ctx,
                      int maxK) {
  if (count <= 0 || maxM <= 0 || maxN <= 0) return AGB_OK;
  if (sizeof(CX) == 8 && ctx && ctx->tc_scratch && maxM >= 64 && maxN >= 64 && maxK >= 32 &&
      ctx->tc_bytes >= tc_gemm_scratch_bytes(count, maxM, maxN, maxK))
    return launch_gemm_tc(probs, count, maxM, maxN, maxK, ctx->tc_scratch, ctx->tc_bytes, ctx->status, s);
  constexpr int B = Tile<CX>::B;
  const int tn = (maxN + B - 1) / B, tm = (maxM + B - 1) / B;
  if ((int64_t)tn * tm > 0x7fffffff) return AGB_ERR_UNSUPPORTED;
  StridedBatch sb = {};
  gemm_simt_kernel<CX><<<dim3(tn * tm, 1, count), 256, 0, s>>>(probs, sb, tn);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
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
  const int B_ = dtype == AGB_C64 ? Tile<float2>::B : Tile<double2>::B;
  const int64_t tn = ((int64_t)N + B_ - 1) / B_, tm = ((int64_t)M + B_ - 1) / B_;
  if (tn * tm > 0x7fffffff) return AGB_ERR_UNSUPPORTED;
  const dim3 grid((unsigned)(tn * tm), 1, batch);
  if (dtype == AGB_C64)
    gemm_simt_kernel<float2><<<grid, 256, 0, s>>>(nullptr, sb, (int)tn);
  else
    gemm_simt_kernel<double2><<<grid, 256, 0, s>>>(nullptr, sb, (int)tn);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}
