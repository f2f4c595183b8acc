// Householder tridiagonalisation of a complex64 Hermitian matrix held in
// registers (and the shared memory behind them) of a thread-block cluster
// (sm_103a).
//
// Row owners.  A cluster of C CTAs reduces one matrix; the 256 threads of a CTA
// form G groups (G = 1 unless the matrix is small), and owner o = q G + g of
// the V = C G owners holds the rows r = o + V i.  Both triangles are kept, so a
// thread owns whole columns (CPT adjacent ones) of every row of its group.  The
// last RR rows of an owner stay in registers (they are the ones that live
// longest), the rows before them in shared memory, and what fits neither in
// the problem's scratch in L2.
//
// Step j (zhetd2 formulation), with v, w of the previous step pending:
//   A. every CTA has row j, the previous p = tau A v and the previous v^H A v:
//      it forms w = p + K v (K = -|tau|^2 v^H A v / 2, real) for the columns its
//      threads own, updates row j and builds the reflector (redundantly in
//      every CTA: no exchange);
//   B. one pass over the own rows: A -= v w^H + w v^H, then p_c += conj(A[r][c])
//      v_r with the new v.  With whole columns per thread this is 14 instructions per
//      element on registers, the row's factors broadcast from shared memory, no
//      index arithmetic and no reduction across lanes.  The partial p's go to
//      the CTA that reduces their columns, with row j + 1 from its owner;
//   C. that CTA adds the V partials, scales by tau and sends its slice of p and
//      of row j + 1 to every CTA.
// The exchanges are remote stores that count their bytes on the receiver's
// mbarrier (st.async), so a step has no cluster barrier and no fence; every CTA
// waits for a word of every other on both barriers (tridiag_exchange.cuh).  A matrix
// whose rows fit one CTA (n <= 128) exchanges through its own shared memory.
//
// What bounds it: the FP32 pipe in pass B (a third of 14 n^2 / C operations per step on
// average) and the dependent chain around it (the norm's reduction, the
// reflector, two exchanges).  Storing both triangles doubles the update's
// arithmetic against the packed rows of tridiag_cluster.cu, whose second
// (column) pass, per-element addressing and C remote vector reads per step
// cost more than that.
// Only the lower triangle of H is read.  Outputs as in tridiag_cluster.cu: d, e
// (real), tau, reflector v_j in row j of H (columns j+2 .., v_j[j+1] = 1
// implicit), scale.
#include "heevd.cuh"
#include "householder.cuh"
#include "prof.cuh"
#include "tridiag_exchange.cuh"

namespace {

constexpr int NT = 256;
constexpr int NW = NT / 32;
static_assert(NW == exchange::kWarps, "words of the exchange");
constexpr int UB = 4;        // register rows per branch of the pass
constexpr int PAD = UB - 1;  // row-factor entries in front (the slots below an owner's first row)

AGB_DEV uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
AGB_DEV uint32_t peer_addr(uint32_t local, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// Remote stores that count their bytes on the receiver's mbarrier: the data is
// its own signal (a cluster barrier's release would also wait for the stored
// reflector's global writes).
AGB_DEV void send(uint32_t a, uint32_t bar, float v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
AGB_DEV void send(uint32_t a, uint32_t bar, float2 u, float2 v) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
      "r"(__float_as_uint(u.x)), "r"(__float_as_uint(u.y)), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)),
      "r"(bar)
      : "memory");
}
AGB_DEV void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded (2^20 waits of about a microsecond): false when the phase did not complete.
AGB_DEV bool bar_wait(uint32_t bar, uint32_t parity) {
  for (unsigned it = 0; it < (1u << 20); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(1000u)
        : "memory");
    if (ok) return true;
  }
  return false;
}
AGB_DEV void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// CTAs that reduce an n x n matrix in a launch of C-CTA clusters: a matrix whose
// rows fit the registers of fewer CTAs uses fewer (the others leave at once):
// 128 columns are one CTA's registers, 256 columns four CTAs' (C256 of them are used).
AGB_HD int active_ctas(int n, int C, int C256) { return n <= 128 ? 1 : (n <= 256 && C > C256 ? C256 : C); }

// Row-factor entries of one CTA: per group its row slots and PAD in front (the
// slots below an owner's first row, read as zeros).
AGB_HD int rowc_entries(int nmax, int C, int C256) {
  int best = 0;
  const int lim[3] = {nmax < 128 ? nmax : 128, nmax < 256 ? nmax : 256, nmax};
  for (int k = 0; k < 3; ++k) {
    const int e = lim[k] / active_ctas(lim[k], C, C256) + 8 * (PAD + 1) + 1;  // the last one takes unused stores
    if (e > best) best = e;
  }
  return best;
}

// Row groups of a CTA: as many as leave every column a thread.
AGB_HD int row_groups(int n, int cpt) {
  int G = 1;
  while (G < 8 && cpt * (NT / (2 * G)) >= n) G *= 2;
  return G;
}

struct Layout {
  size_t part, pr, rowsl, dots, red, bars, f4, f2, rows;  // byte offsets
};
AGB_HD Layout layout(int cpt, int rce) {
  const size_t nc = (size_t)NT * cpt;
  Layout L;
  size_t o = 0;
  L.part = o;  o += (nc + 256) * 8;
  L.pr = o;    o += nc * 16;
  L.rowsl = o; o += nc * 8;
  L.dots = o;  o += 48 * 4;
  L.red = o;   o += 16 * 4;
  L.bars = o;  o += 32;
  L.f4 = o;    o += (size_t)rce * 16;
  L.f2 = o;    o += ((size_t)rce * 8 + 15) & ~(size_t)15;
  L.rows = o;
  return L;
}

// y = a[s] for a run-time s: a jump table, as register arrays take constant
// indices only (a chain of RR selects costs more than the row's update).
template <int CPT, int RR>
AGB_DEV void pick_row(const float2 (&a)[RR][CPT], int s, float2 (&y)[CPT]) {
#define AGB_PICK(i)                                                               \
  case i:                                                                         \
    if constexpr (i < RR) {                                                       \
      _Pragma("unroll") for (int k = 0; k < CPT; ++k) y[k] = a[i < RR ? i : 0][k]; \
    }                                                                             \
    break;
#define AGB_PICK8(i)                                                                               \
  AGB_PICK(i) AGB_PICK(i + 1) AGB_PICK(i + 2) AGB_PICK(i + 3) AGB_PICK(i + 4) AGB_PICK(i + 5) AGB_PICK(i + 6) \
      AGB_PICK(i + 7)
  switch (s) {
    AGB_PICK8(0)
    AGB_PICK8(8)
    AGB_PICK8(16)
    AGB_PICK8(24)
    AGB_PICK8(32)
    default:
      break;
  }
#undef AGB_PICK8
#undef AGB_PICK
}

template <int CPT, int RR>
__global__ void __launch_bounds__(NT, 1)
    tridiag_reg_kernel(HeevdProb* __restrict__ probs, int C, int C256, int rce, int row_elems) {
  constexpr int NC = NT * CPT;
  const HeevdProb P = probs[blockIdx.x / C];
  const int q = blockIdx.x % C;
  const int n = P.n;
  if (n <= 0) return;
  const int Ce = active_ctas(n, C, C256);
  if (q >= Ce) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int G = row_groups(n, CPT);
  const int ct = NT / G, g = tid / ct, c0 = CPT * (tid - g * ct);  // own columns c0 .. c0 + CPT - 1
  const int V = Ce * G, o = q * G + g;
  const int nr = (n + V - 1) / V;  // row slots per owner
  extern __shared__ __align__(16) unsigned char smem[];
  const Layout L = layout(CPT, rce);
  float2* part = (float2*)(smem + L.part);    // [V][S] partial p of this CTA's column slice
  float2* pr = (float2*)(smem + L.pr);        // [NC][2] p and row j + 1, side by side
  float2* rowsl = (float2*)(smem + L.rowsl);  // [S] row j + 1 over the own slice
  float* wdots = (float*)(smem + L.dots);     // [2][16] v^H A v shares of the warps that report here, by step
  float* dots = wdots + 32;                   // [16] shares of the CTAs
  float* red = (float*)(smem + L.red);        // [NW] norm partials, then alpha at red[8..9] (red[10..11] takes the others' stores)
  const uint32_t bar1 = smem_u32(smem + L.bars), bar2 = bar1 + 8;  // partials; their sums
  volatile int* stop = (volatile int*)(smem + L.bars + 16);
  float4* f4 = (float4*)(smem + L.f4);  // [G][PAD + nr] row factors v, w of step j-1
  float2* f2 = (float2*)(smem + L.f2);  // [G][PAD + nr] row factors v of step j
  float2* rows = (float2*)(smem + L.rows);
  float2* H = (float2*)P.H;
  const int64_t ld = P.ldh;
  float2* spill = (float2*)P.band;  // [n][n] rows that fit neither registers nor shared memory
  // own rows: slots [0, ngm) in L2, [ngm, nr - RR) in shared memory, the last RR in registers
  const int ns = (n + CPT - 1) / CPT * CPT;  // stride of the rows kept in shared memory
  int nsm = nr - RR > 0 ? nr - RR : 0;
  {
    const int cap = row_elems / (G * ns);
    if (nsm > cap) nsm = cap;
  }
  const int base = nr - RR;  // slot of register row 0 (may be negative)
  const int ngm = (base > 0 ? base : 0) - nsm;
  const int S = ((n + Ce - 1) / Ce + CPT - 1) / CPT * CPT;  // columns of a CTA's slice

  // ---- scale by the largest diagonal magnitude (every CTA reads the diagonal)
  float mx = 0;
  for (int i = tid; i < n; i += NT) mx = fmaxf(mx, fabsf(H[(int64_t)i * ld + i].x));
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
  if (lane == 0) red[wid] = mx;
  const float2 zero = make_float2(0.f, 0.f);
  for (int i = tid; i < rce; i += NT) {
    f4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    f2[i] = zero;
  }
  for (int i = tid; i < 2 * NC; i += NT) pr[i] = zero;
  for (int i = tid; i < NC + 256; i += NT) part[i] = zero;
  for (int i = tid; i < NC; i += NT) rowsl[i] = zero;
  if (tid < 48) wdots[tid] = 0.f;
  if (tid == 0) {
    *stop = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar1));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar2));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) mx = fmaxf(mx, red[w]);
  if (mx == 0.f) {  // no diagonal to scale by: the largest entry (no Gram matrix comes here)
    __syncthreads();
    for (int i = tid; i < n * n; i += NT) {
      const int r = i / n, c = i - r * n;
      if (c < r) mx = fmaxf(mx, fmaxf(fabsf(H[(int64_t)r * ld + c].x), fabsf(H[(int64_t)r * ld + c].y)));
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
    if (lane == 0) red[wid] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int w = 1; w < NW; ++w) mx = fmaxf(mx, red[w]);
    if (mx == 0.f) mx = 1.f;
  }
  if (q == 0 && tid == 0) *((float*)P.scale) = mx;
  const float inv = 1.f / mx;

  // ---- load (lower triangle, mirrored)
  auto elem = [&](int r, int c) -> float2 {
    if (r >= n || c >= n) return zero;
    float2 h = (c <= r) ? H[(int64_t)r * ld + c] : cconj(H[(int64_t)c * ld + r]);
    if (r == c) h.y = 0.f;
    return cscale(h, inv);
  };
  float2 a[RR][CPT];
#pragma unroll
  for (int s = 0; s < RR; ++s)
#pragma unroll
    for (int k = 0; k < CPT; ++k) a[s][k] = (base + s >= 0) ? elem(o + V * (base + s), c0 + k) : zero;
  for (int i = 0; i < ngm + nsm; ++i)
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int c = c0 + k, r = o + V * i;
      if (c0 >= n || r >= n) continue;
      if (i >= ngm) rows[(int64_t)((i - ngm) * G + g) * ns + c] = elem(r, c);
      else if (c < n) spill[(int64_t)r * n + c] = elem(r, c);
    }
  if (n == 1) {
    if (tid == 0) {
      ((float*)P.d)[0] = elem(0, 0).x;
      ((float*)P.e)[0] = 0.f;
      ((float2*)P.tau)[0] = zero;
    }
    return;
  }

  // ---- per-thread column constants
  // where this owner's partial p of the own columns, and its rows, go (CTA c0 / S)
  const int dq = c0 < n ? c0 / S : 0;
  const uint32_t part_addr = peer_addr(smem_u32(part + (size_t)o * S + (c0 - dq * S)), dq);
  const uint32_t row_addr = peer_addr(smem_u32(rowsl + (c0 - dq * S)), dq);
  const uint32_t part_bar = peer_addr(bar1, dq);
  // the warp's share of v^H A v
  const int dd = exchange::dot_dest(wid, Ce);
  const uint32_t dot_addr = peer_addr(smem_u32(wdots + q * exchange::dot_pitch(Ce) + wid / Ce), dd);
  const uint32_t dot_bar = peer_addr(bar1, dd);
  const int ndot = exchange::dot_words(q, Ce) * Ce;  // words of it that arrive here
  const int nslice = min(n, q * S + S);               // end of the own slice
  int fac[CPT];   // row-factor entry of row c when this owner holds it, else an unused one
  float2 v[CPT];  // own columns of v (step j-1 until A, then step j)
  float2 w[CPT];  // own columns of w of step j-1
  float2 y[CPT];  // own columns of row j + 1, updated through step j-2, in its owner
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const int c = c0 + k;
    fac[k] = (c < n && c % V == o) ? g * (PAD + nr) + PAD + c / V : rce - 1;
    v[k] = w[k] = zero;
    y[k] = elem(1, c);
  }
  const float4* rf4 = f4 + g * (PAD + nr) + PAD;
  const float2* rf2 = f2 + g * (PAD + nr) + PAD;
  float* dg = (float*)P.d;
  float* eg = (float*)P.e;
  float2* tau = (float2*)P.tau;
  // row 0 (each CTA reads it itself); the zeroed p belongs to no step
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (g == 0 && c0 + k < n) {
      pr[2 * (c0 + k) + 1] = elem(0, c0 + k);
      if (Ce == 1) rowsl[c0 + k] = elem(0, c0 + k);
    }
  if (Ce > 1) cluster_barrier();  // every CTA is running and its buffers and barriers are initialised
  else __syncthreads();

  float2 t = zero;              // tau of the previous step
  float kt = 0.f;               // -|tau|^2 / 2
  int turn = 0;                 // CTA that stores reflector j
  int i0 = 0, nexto = o;        // first own slot with row > j, and its row
  bool hasy = o == 1 % V;       // y holds row j + 1
  int yslot = 1 / V;
  float2* hrow = H;
  bool ok = true;
  for (int j = 0; j < n; ++j, hrow += ld) {
    // ---------------- A: w of step j-1 for the own columns, row j, reflector j
    // (columns below j carry stale values: nothing reads what they produce)
    float2 x[CPT], wj;
    if (Ce == 1) {
      const float4 d0 = *(const float4*)wdots, d1 = *(const float4*)(wdots + 4);
      const float Kc = kt * (((d0.x + d0.y) + (d0.z + d0.w)) + ((d1.x + d1.y) + (d1.z + d1.w)));
      float2 sj = zero;
#pragma unroll
      for (int k = 0; k < CPT; ++k) w[k] = zero;
      const float2* pp = part;
      if (c0 < n) {  // S covers the columns below n only
#pragma unroll 4
        for (int i = 0; i < V; ++i, pp += S) {
          sj = cadd(sj, pp[j]);
#pragma unroll
          for (int k = 0; k < CPT; ++k) w[k] = cadd(w[k], pp[c0 + k]);
        }
      }
      wj = cmul(t, sj);
      wj.x += Kc;  // v_{j-1}[j] = 1
#pragma unroll
      for (int k = 0; k < CPT; ++k) {
        w[k] = cmul(t, w[k]);
        w[k].x = fmaf(Kc, v[k].x, w[k].x);
        w[k].y = fmaf(Kc, v[k].y, w[k].y);
        x[k] = c0 < n ? rowsl[c0 + k] : zero;
      }
    } else {
      const float4 d0 = *(const float4*)dots, d1 = *(const float4*)(dots + 4);
      float s = ((d0.x + d0.y) + (d0.z + d0.w)) + ((d1.x + d1.y) + (d1.z + d1.w));
      if (Ce > 8) {
        const float4 d2 = *(const float4*)(dots + 8), d3 = *(const float4*)(dots + 12);
        s += ((d2.x + d2.y) + (d2.z + d2.w)) + ((d3.x + d3.y) + (d3.z + d3.w));
      }
      const float Kc = kt * s;
      wj = pr[2 * j];
      wj.x += Kc;
#pragma unroll
      for (int k = 0; k < CPT; ++k) {
        const float4 z = *(const float4*)(pr + 2 * (c0 + k));
        w[k] = make_float2(fmaf(Kc, v[k].x, z.x), fmaf(Kc, v[k].y, z.y));
        x[k] = make_float2(z.z, z.w);
      }
    }
    float pn = 0.f, dj = 0.f;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int c = c0 + k;
      f4[fac[k]] = make_float4(v[k].x, v[k].y, w[k].x, w[k].y);
      // x = row - v[j] conj(w) - w[j] conj(v), v[j] = 1
      x[k].x = fmaf(-wj.x, v[k].x, fmaf(-wj.y, v[k].y, x[k].x - w[k].x));
      x[k].y = fmaf(-wj.y, v[k].x, fmaf(wj.x, v[k].y, x[k].y + w[k].y));
      *(float2*)(red + (c == j + 1 ? 8 : 10)) = cconj(x[k]);
      dj = c == j ? x[k].x : dj;
      if (c >= j + 2) pn = fmaf(x[k].x, x[k].x, fmaf(x[k].y, x[k].y, pn));
    }
    if (j == n - 1) {
      if (o == 0 && j - c0 >= 0 && j - c0 < CPT) {
        dg[j] = dj;
        eg[j] = 0.f;
      }
      break;
    }
    pn = warp_sum(pn);
    if (lane == 0) red[wid] = g == 0 ? pn : 0.f;  // every group holds the whole row
    __syncthreads();
    const int halt = *stop;  // a wait of the previous step expired: the whole CTA stops
    const float4 z0 = *(const float4*)red, z1 = *(const float4*)(red + 4);
    const float xn2 = ((z0.x + z0.y) + (z0.z + z0.w)) + ((z1.x + z1.y) + (z1.z + z1.w));
    float2 sc;
    float beta;
    reflector(*(const float2*)(red + 8), xn2, beta, t, sc);
    float2 vp[CPT];  // v of step j-1
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int c = c0 + k;
      vp[k] = v[k];
      const float2 u = cmul(cconj(x[k]), sc);
      v[k] = (c == j + 1) ? make_float2(1.f, 0.f) : c >= j + 2 ? u : zero;
      f2[fac[k]] = v[k];
    }
    __syncthreads();
    if (halt) break;
    // ---------------- B: update with step j-1, partial matvec with v, over own rows > j
    if (nexto <= j) {
      ++i0;
      nexto += V;
    }
    auto update = [&](float2& e, int k, const float4& f) {
      // the four products are summed first: one rounding at the size of e (as a chain of
      // FMAs into e, two instructions fewer and 2 to 6% faster, its four roundings made the
      // eigenvalue error 0.59 instead of 0.52 u lambda_0 at n = 100)
      float tx = f.x * w[k].x, ty = f.y * w[k].x;
      tx = fmaf(f.y, w[k].y, tx);
      ty = fmaf(-f.x, w[k].y, ty);
      tx = fmaf(f.z, vp[k].x, tx);
      ty = fmaf(f.w, vp[k].x, ty);
      tx = fmaf(f.w, vp[k].y, tx);
      ty = fmaf(-f.z, vp[k].y, ty);
      e.x -= tx;
      e.y -= ty;
    };
    float sd = 0.f;
    if (c0 + CPT - 1 > j && c0 < n) {  // own columns still in use
      // row j + 1 (updated through step j-1), in column slices
      if (hasy) {
        const float4 f = rf4[yslot];
#pragma unroll
        for (int k = 0; k < CPT; ++k) update(y[k], k, f);
#pragma unroll
        for (int k = 0; k < CPT; k += 2) {
          if (Ce == 1) *(float4*)(rowsl + c0 + k) = make_float4(y[k].x, y[k].y, y[k + 1].x, y[k + 1].y);
          else send(row_addr + 8u * k, part_bar, y[k], y[k + 1]);
        }
      }
      float2 p[CPT];
#pragma unroll
      for (int k = 0; k < CPT; ++k) p[k] = zero;
      auto matvec = [&](const float2& e, int k, const float2& f) {  // conj(e) f
        p[k].x = fmaf(e.x, f.x, p[k].x);
        p[k].y = fmaf(e.x, f.y, p[k].y);
        p[k].x = fmaf(e.y, f.y, p[k].x);
        p[k].y = fmaf(-e.y, f.x, p[k].y);
      };
      {
        // rows in L2: GB at a time, their loads ahead of any store (a slot past
        // the last row reads the first again and is dropped)
        constexpr int GB = 16 / CPT;
        const bool full = c0 + CPT <= n;
        for (int i = i0; i < ngm; i += GB) {
          float2 e[GB][CPT];
#pragma unroll
          for (int u = 0; u < GB; ++u) {
            const float2* row = spill + (int64_t)(o + V * (i + u < ngm ? i + u : i)) * n + c0;
#pragma unroll
            for (int k = 0; k < CPT; ++k) e[u][k] = full || c0 + k < n ? row[k] : zero;
          }
#pragma unroll
          for (int u = 0; u < GB; ++u) {
            if (i + u >= ngm) break;
            const float4 f = rf4[i + u];
            const float2 fx = rf2[i + u];
            float2* row = spill + (int64_t)(o + V * (i + u)) * n + c0;
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
              update(e[u][k], k, f);
              if (full || c0 + k < n) row[k] = e[u][k];
              matvec(e[u][k], k, fx);
            }
          }
        }
      }
      {
        const int ib = i0 > ngm ? i0 : ngm;
        float4* row = (float4*)(rows + (int64_t)((ib - ngm) * G + g) * ns + c0);
        const int step = G * ns / 2;
        // SB rows at a time: their loads ahead of any store
        constexpr int SB = 8 / CPT;
        int i = ib;
        for (; i + SB <= ngm + nsm; i += SB, row += SB * step) {
          float4 f[SB], z[SB][CPT / 2];
          float2 fx[SB];
#pragma unroll
          for (int u = 0; u < SB; ++u) {
            f[u] = rf4[i + u];
            fx[u] = rf2[i + u];
#pragma unroll
            for (int k = 0; k < CPT / 2; ++k) z[u][k] = row[u * step + k];
          }
#pragma unroll
          for (int u = 0; u < SB; ++u)
#pragma unroll
            for (int k = 0; k < CPT; k += 2) {
              float2 e0 = make_float2(z[u][k / 2].x, z[u][k / 2].y), e1 = make_float2(z[u][k / 2].z, z[u][k / 2].w);
              update(e0, k, f[u]);
              update(e1, k + 1, f[u]);
              row[u * step + k / 2] = make_float4(e0.x, e0.y, e1.x, e1.y);
              matvec(e0, k, fx[u]);
              matvec(e1, k + 1, fx[u]);
            }
        }
        for (; i < ngm + nsm; ++i, row += step) {
          const float4 f = rf4[i];
          const float2 fx = rf2[i];
#pragma unroll
          for (int k = 0; k < CPT; k += 2) {
            const float4 z = row[k / 2];
            float2 e0 = make_float2(z.x, z.y), e1 = make_float2(z.z, z.w);
            update(e0, k, f);
            update(e1, k + 1, f);
            row[k / 2] = make_float4(e0.x, e0.y, e1.x, e1.y);
            matvec(e0, k, fx);
            matvec(e1, k + 1, fx);
          }
        }
      }
      // register rows in blocks (used-up rows of a block have v = 0: they add nothing)
      static_assert(RR % UB == 0, "register rows in blocks");
      const float4* b4 = rf4 + base;
      const float2* b2 = rf2 + base;
      const int sb = i0 > base ? (i0 - base) & ~(UB - 1) : 0;
#pragma unroll
      for (int s = 0; s < RR; s += UB) {
        if (s >= sb) {
          float4 f[UB];
          float2 fx[UB];
#pragma unroll
          for (int u = 0; u < UB; ++u) {
            f[u] = b4[s + u];
            fx[u] = b2[s + u];
          }
#pragma unroll
          for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
              update(a[s + u][k], k, f[u]);
              matvec(a[s + u][k], k, fx[u]);
            }
        }
      }
#pragma unroll
      for (int k = 0; k < CPT; k += 2) {
        if (Ce == 1) *(float4*)(part + (size_t)o * S + c0 + k) = make_float4(p[k].x, p[k].y, p[k + 1].x, p[k + 1].y);
        else send(part_addr + 8u * k, part_bar, p[k], p[k + 1]);
      }
#pragma unroll
      for (int k = 0; k < CPT; ++k) sd = fmaf(v[k].x, p[k].x, fmaf(v[k].y, p[k].y, sd));
    }
    // v^H A v (real), by warps
    sd = warp_sum(sd);
    if (lane == 0) {
      if (Ce == 1) wdots[wid] = sd;
      else send(dot_addr + 64u * (j & 1), dot_bar, sd);
      if (Ce > NW && wid < exchange::zeros(Ce))
        send(peer_addr(smem_u32(wdots + 16 * (j & 1) + q), NW + wid), peer_addr(bar1, NW + wid), 0.f);
    }
    // off the exchange's critical path: bytes to expect, the stored reflector, the next row
    if (tid == 0 && Ce > 1) {
      // pairs of columns of the own slice still in use (CPT at a time)
      const int f0 = max(q * S, (j + 1) / CPT * CPT);
      const int sl = nslice > f0 ? (nslice - f0 + CPT - 1) / CPT : 0;
      bar_expect(bar1, (uint32_t)(sl * (V + 1) * CPT * 8 + ndot * 4));
      bar_expect(bar2, (uint32_t)((n - 1 - j) * 16 + Ce * 4));
    }
    if (o == 0 && j - c0 >= 0 && j - c0 < CPT) dg[j] = dj;
    if (turn == q && g == 0) {
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (c0 + k >= j + 2 && c0 + k < n) hrow[c0 + k] = v[k];
      if (tid == 0) {
        eg[j] = beta;
        tau[j] = t;
      }
    }
    if (++turn == Ce) turn = 0;
    kt = -0.5f * cabs2(t);
    {
      const int own = nexto == j + 1 ? 1 : 0;  // first own row > j + 1
      yslot = i0 + own;
      hasy = nexto + own * V == j + 2 && j + 2 < n;
      if (hasy) {
        if (yslot >= base) {
          pick_row<CPT, RR>(a, yslot - base, y);
        } else if (yslot >= ngm) {
          const float2* row = rows + (int64_t)((yslot - ngm) * G + g) * ns + c0;
#pragma unroll
          for (int k = 0; k < CPT; ++k) y[k] = c0 < n ? row[k] : zero;
        } else {
#pragma unroll
          for (int k = 0; k < CPT; ++k) y[k] = c0 + k < n ? spill[(int64_t)(j + 2) * n + c0 + k] : zero;
        }
      }
    }
    if (Ce == 1) {
      __syncthreads();
      continue;
    }
    if (!bar_wait(bar1, j & 1)) ok = false;
    // ---------------- C: reduce the own column slice; p and row j+1 of it to every CTA
    // (each lane reads the shares for itself: a peer that has its word may write the next
    // step's, into the other half, before the last lane has read these)
    if (wid == NW - 1 && lane < Ce) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 z = *(const float4*)(wdots + 16 * (j & 1) + i);
        s += (z.x + z.y) + (z.z + z.w);
      }
      send(peer_addr(smem_u32(dots + q), lane), peer_addr(bar2, lane), s);
    }
    for (int cl = tid; cl < S; cl += NT) {
      const int c = q * S + cl;
      if (c < n && c > j) {
        float2 acc = zero, ac1 = zero;
        const float2* pp = part + cl;
#pragma unroll 4
        for (int i = 0; i + 1 < V; i += 2) {
          acc = cadd(acc, pp[(size_t)i * S]);
          ac1 = cadd(ac1, pp[(size_t)(i + 1) * S]);
        }
        if (V & 1) acc = cadd(acc, pp[(size_t)(V - 1) * S]);
        const float2 rv = rowsl[cl];
        acc = cmul(t, cadd(acc, ac1));
        const uint32_t da = smem_u32(pr + 2 * c);
#pragma unroll 4
        for (int d = 0; d < Ce; ++d) send(peer_addr(da, d), peer_addr(bar2, d), acc, rv);
      }
    }
    if (!bar_wait(bar2, j & 1)) ok = false;
    if (!ok) *stop = 1;
  }
  if (Ce > 1 && __syncthreads_or(!ok || *stop)) {
    // an exchange did not arrive (cannot happen unless a peer stopped): report it,
    // and let sends in flight land before this CTA's shared memory goes away
    probs[blockIdx.x / C].fail = 1;
    cluster_barrier();
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
}

typedef void (*RegKernel)(HeevdProb*, int, int, int, int);
struct Form {
  RegKernel kern;
  int cpt, rr;
};
// Columns per thread and register rows: 128 registers of matrix per thread in
// every form but the smallest, whose short code and fewer rows suit n <= 64.
Form form_for(int maxn) {
  if (maxn <= 64) return {tridiag_reg_kernel<2, 8>, 2, 8};
  if (maxn <= 512) return {tridiag_reg_kernel<2, 32>, 2, 32};
  return {tridiag_reg_kernel<4, 16>, 4, 16};
}
constexpr size_t kRegSmem = 224 * 1024;

cudaLaunchConfig_t config(int grid, int C, size_t smem, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(NT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace



int launch_tridiag_reg(const HeevdProb* probs, int count, int maxn, int C, cudaStream_t s) {
  if (C < 1 || C > 16 || maxn > 1024) return AGB_ERR_UNSUPPORTED;
  const Form f = form_for(maxn);
  const int C256 = 8 * count <= 152 ? 8 : 4;  // 0.62 ms on 4 SMs or 0.54 on 8 (n = 256)
  const int rce = rowc_entries(maxn, C, C256);
  const size_t off = layout(f.cpt, rce).rows;
  if (off > kRegSmem) return AGB_ERR_UNSUPPORTED;
  // shared-memory rows: as many as a matrix of this batch can use
  size_t want = 0;
  const int lim[3] = {maxn < 128 ? maxn : 128, maxn < 256 ? maxn : 256, maxn};
  for (int k = 0; k < 3; ++k) {
    const int nn = lim[k], Ce = active_ctas(nn, C, C256), G = row_groups(nn, f.cpt);
    const int nr = (nn + Ce * G - 1) / (Ce * G);
    const size_t e = nr > f.rr ? (size_t)(nr - f.rr) * G * (nn + f.cpt - 1) * sizeof(float2) : 0;
    if (e > want) want = e;
  }
  const size_t smem = off + want < kRegSmem ? off + want : kRegSmem;
  if (C > 8) cudaFuncSetAttribute(f.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaFuncSetAttribute(f.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegSmem);
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = config(count * C, C, smem, attr);
  cfg.stream = s;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, f.kern, const_cast<HeevdProb*>(probs), C, C256, rce,
                                             (int)((smem - off) / sizeof(float2)));
  agb_note_launch();
  if (err != cudaSuccess) {
    agb_note_error(__FILE__, __LINE__, err);
    return AGB_ERR_CUDA;
  }
  return AGB_OK;
}

// Clusters of C CTAs of the kernel for this size that the device holds at once
// (0 where it schedules none; sizes above 8 are not portable).
int tridiag_reg_clusters(int maxn, int C) {
  static int cached[3][17];  // + 1
  if (C < 1 || C > 16) return 0;
  int& c = cached[maxn <= 64 ? 0 : maxn <= 512 ? 1 : 2][C];
  if (c) return c - 1;
  int ncl = 0;
  const RegKernel kern = form_for(maxn).kern;
  if ((C <= 8 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegSmem) == cudaSuccess) {
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = config(C, C, kRegSmem, attr);
    if (cudaOccupancyMaxActiveClusters(&ncl, kern, &cfg) != cudaSuccess) ncl = 0;
  }
  cudaGetLastError();
  c = ncl + 1;
  return ncl;
}

// CTAs per matrix for `count` matrices of up to maxn columns.  Up to 128 columns
// are one CTA's registers; up to 256 columns take 8 CTAs while every matrix
// gets its own SMs (0.54 against 0.62 ms at n = 256) and 4 beyond that.
// Between 256 and 512 the fewest waves decide: a matrix of n = 512 takes 1.27,
// 1.40 and 1.52 ms on 16, 10 and 8 CTAs (counted as 0.72 + 5.6 / C), and a cluster
// needs its SMs in one GPC.  The rule knows the count and the largest n only: 20
// equal matrices of 512 take 2.80 ms on 10 CTAs and would take 1.80 on 6, but a
// chain's layer of 20 gates, whose end gates are small, runs all its full-size
// ones at once on 10 (1.6 ms; 6% more on 6).  Above 512 rows spill to L2 below 16 CTAs
// (n = 1024: 6.8 against 14.4 ms on 8).
int tridiag_reg_ctas(int maxn, int count) {
  if (maxn <= 128) return 1;
  if (maxn <= 256) return 8 * count <= 152 ? 8 : 4;
  if (maxn > 512) return tridiag_reg_clusters(maxn, 16) > 0 ? 16 : 8;
  int best = 8;
  float cost = 1e30f;
  for (int C : {16, 10, 8}) {
    const int held = tridiag_reg_clusters(maxn, C);
    if (held <= 0) continue;
    const float t = (float)((count + held - 1) / held) * (0.72f + 5.6f / (float)C);
    if (t < cost) {
      cost = t;
      best = C;
    }
  }
  return best;
}
