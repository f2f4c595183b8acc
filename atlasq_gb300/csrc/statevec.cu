// Dense state of a short chain in one launch: psi = T_0 T_1 ... T_{n-1}.
//
// As one matrix product per site a 10-qubit read-out is nine launches of a few
// thousand multiply-adds each, and what it costs is the nine calls.  Here each
// CTA holds the first h qubits fixed (its index gives their values), carries the
// remaining rows 2^(s-h) x chi_s in shared memory from site to site and writes
// its contiguous 2^(n-h) amplitudes.  The tensors are read once per CTA, from L2
// after the first.  Sums run over the bond in order, as in the SIMT GEMM, so the
// amplitudes are bit for bit those of the product-per-site path.
//
// Bound by latency (one barrier and one L2 round trip per site).  Measured
// (GB300, complex64, Haar brickwork): 10 qubits, bonds up to 32, 9 launches and
// 28 us before, one of 8 us now; 24 states of 6 to 10 qubits 168 launches, 530 us
// on the device and 7.8 ms of host calls, now 24, 162 us and 2 ms.
//
// Rule: n <= 20, the rows of every site fit 24 KB, and the CTAs together read at
// most 4 M elements (2^h times the chain).  Beyond that the re-reading of the
// wide middle tensors would cost more than the launches, and the products fill
// the chip by themselves.
#include "common.cuh"

namespace {

constexpr int kSvSites = 20;
constexpr size_t kSvBufBytes = 24 * 1024;   // one of the two row buffers
constexpr int64_t kSvReads = (int64_t)1 << 22;

struct SvChain {
  const void* T[kSvSites];
  int chi[kSvSites + 1];
};

// out[r, j] = sum_k v[r, k] T[k, j0 + j] for `rows` rows; RT rows per thread share the loads of T
template <typename CX, int RT>
AGB_DEV void sv_site(const CX* v, const CX* __restrict__ T, CX* out, int rows, int K, int cols, int ld) {
  const int groups = (rows + RT - 1) / RT;
  for (int item = threadIdx.x; item < groups * cols; item += blockDim.x) {
    const int r0 = item / cols * RT, j = item % cols;
    CX acc[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) acc[i] = czero<CX>();
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
      const CX t = T[(int64_t)k * ld + j];
#pragma unroll
      for (int i = 0; i < RT; ++i) cfma(acc[i], v[min(r0 + i, rows - 1) * K + k], t);
    }
#pragma unroll
    for (int i = 0; i < RT; ++i)
      if (r0 + i < rows) out[(int64_t)(r0 + i) * cols + j] = acc[i];
  }
}

template <typename CX>
__global__ void __launch_bounds__(256) statevector_kernel(SvChain c, int n, int h, CX* __restrict__ out) {
  __shared__ __align__(16) unsigned char smem_raw[2 * kSvBufBytes];
  CX* v = (CX*)smem_raw;
  CX* w = (CX*)(smem_raw + kSvBufBytes);
  const unsigned p = blockIdx.x;
  int rows = 1;
  for (int s = 0; s < n; ++s) {
    const int K = c.chi[s], cn = c.chi[s + 1];
    const bool fixed = s < h;
    const int cols = fixed ? cn : 2 * cn;
    const CX* T = (const CX*)c.T[s] + (fixed ? (int)((p >> (h - 1 - s)) & 1u) * cn : 0);
    CX* o = s == n - 1 ? out + ((size_t)p << (n - h)) : w;
    if (s == 0) {
      for (int j = threadIdx.x; j < cols; j += blockDim.x) o[j] = T[j];  // one row, K = 1
    } else if (rows * cols <= 4 * (int)blockDim.x) {
      sv_site<CX, 1>(v, T, o, rows, K, cols, 2 * cn);
    } else {
      sv_site<CX, 4>(v, T, o, rows, K, cols, 2 * cn);
    }
    __syncthreads();
    CX* t = v;
    v = w;
    w = t;
    if (!fixed) rows *= 2;
  }
}

}  // namespace

extern "C" int agb_statevector(int dtype, int n, const int64_t* tensors, const int32_t* chi, void* out,
                               void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (!tensors || !chi || !out || n < 1) return AGB_ERR_ARG;
  if (n > kSvSites) return AGB_ERR_UNSUPPORTED;
  if (chi[0] != 1 || chi[n] != 1) return AGB_ERR_ARG;
  SvChain c = {};
  int64_t total = 0;
  for (int s = 0; s < n; ++s) {
    if (!tensors[s] || chi[s + 1] < 1) return AGB_ERR_ARG;
    if (chi[s + 1] > (1 << 20)) return AGB_ERR_UNSUPPORTED;
    c.T[s] = (const void*)tensors[s];
    total += 2 * (int64_t)chi[s] * chi[s + 1];
  }
  for (int s = 0; s <= n; ++s) c.chi[s] = chi[s];
  const int64_t cap = (int64_t)(kSvBufBytes / (dtype == AGB_C64 ? 8 : 16));
  // fewest fixed qubits, from 5 (32 CTAs) up, for which every site's rows fit
  for (int h = n - 1 < 5 ? n - 1 : 5; h < n && (total << h) <= kSvReads; ++h) {
    bool fits = true;
    for (int s = 1; s < n; ++s) fits = fits && ((int64_t)chi[s] << (s > h ? s - h : 0)) <= cap;
    if (!fits) continue;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == AGB_C64) statevector_kernel<float2><<<1 << h, 256, 0, st>>>(c, n, h, (float2*)out);
    else statevector_kernel<double2><<<1 << h, 256, 0, st>>>(c, n, h, (double2*)out);
    AGB_CHECK_LAUNCH();
    return AGB_OK;
  }
  return AGB_ERR_UNSUPPORTED;
}
