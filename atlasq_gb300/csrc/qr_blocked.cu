// Blocked Householder QR on a thread-block cluster (sm_103a), for the
// canonicalisation sweeps (QR of a site tensor, up to ~1000 x 512).
//
// Same factorisation as qr_kernel (zgeqr2 reflectors H_i = I - tau_i v_i v_i^H,
// beta = -sign(Re alpha) ||x||, thin Q = H_0 H_1 ... applied to [I; 0]),
// reorganised in panels of QB columns (zgeqrf / zlarft / zlarfb):
//
// * Columns are dealt to the C CTAs of one cluster in panels, block-cyclically
//   (panel p -> CTA p mod C); each CTA keeps its panels column-major in shared
//   memory.
// * Panel p is factored by its owner alone: warp w holds panel column w; per
//   column the owner warp forms the reflector and one block barrier publishes
//   it.  The later warps apply it to their columns; the earlier ones, whose
//   columns are done, form its products with their reflectors, from which warp
//   0 builds the next column of the triangular factor T_p of H_pb ... H_pb+QB-1 =
//   I - V T V^H (forward, columnwise) one column behind; and the whole CTA
//   writes it to global memory (L2; explicit zeros above the unit diagonal).
//   When the last column is done, V_p and T_p are complete.
// * One cluster barrier per panel; every CTA then applies Q_p^H = I - V T^H V^H
//   to its later panels from a shared-memory copy of V_p:
//   W = V^H Y, W = T^H W, Y -= V W.
// * The thin Q is formed backwards, Z = Q_p Z from Z = [I; 0], each CTA on its
//   own columns with V_p, T_p read back from L2: no barrier between CTAs.
//
// One cluster barrier per QB columns (the unblocked cluster kernel needs two
// per column), and the trailing updates are QB-wide instead of rank-1.
//
// What bounds it: the chain owner's panel -> barrier -> next owner's update -> its
// panel, on one SM at a time: the panel is a chain of QB columns (norm, reflector,
// barrier, product, update), the update of QB columns by QB reflectors is bound by
// that SM's FP32 pipe (2 QB^2 M complex multiply-adds).
// Inside a panel 15 warps issue ~15 instructions a row for product and update of
// each column (1400 of its 2800 cycles; the reflector 1200): the reflector is read
// once, into registers, and in complex64 up to 512 rows padded with zeros to the
// registers' rows, so that no access is predicated.  512 x 256 on 16 CTAs: 0.58 ms
// (0.65 with predicated reads, twice a column); updates 8 us, the thin Q 6 us a
// panel.
#include <cooperative_groups.h>

#include "householder.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int QBT = 512;  // threads per CTA (16 warps)
constexpr size_t kQrbSmemBudget = 220 * 1024;
constexpr int kQrbMaxCols = 256;  // own columns per CTA (npo * QB)

template <typename CX> struct QrbCfg;
template <> struct QrbCfg<float2> { static constexpr int QB = 16; };
template <> struct QrbCfg<double2> { static constexpr int QB = 8; };

struct QrbLayout {
  int QB, C, P, PF, npo, ld;
  size_t panels, vloc, vloc2, w, w2, t, vb, total;  // byte offsets (vloc2 == vloc: one buffer of V)
};

// vrows: rows of the two reflector buffers
AGB_HD QrbLayout qrb_layout(int esz, int QB, int M, int N, int C, int vrows) {
  QrbLayout L;
  L.QB = QB;
  L.C = C;
  const int kk = M < N ? M : N;
  L.P = (N + QB - 1) / QB;
  L.PF = (kk + QB - 1) / QB;
  L.npo = (L.P + C - 1) / C;
  L.ld = M + 1;  // odd column stride: lanes reading one row of different columns hit different banks
  size_t o = 0;
  L.panels = o; o += (size_t)L.npo * QB * L.ld * esz;
  L.vloc = o;   o += (size_t)QB * L.ld * esz;
  L.vloc2 = L.vloc;
  L.w = o;      o += (size_t)QB * L.npo * QB * esz;
  L.w2 = o;     o += (size_t)QB * L.npo * QB * esz;
  L.t = o;      o += (size_t)QB * QB * esz;
  L.vb = o;     o += (size_t)2 * vrows * esz;
  // a second V buffer where it fits: the thin Q's panels are then read ahead
  if (o + (size_t)QB * L.ld * esz <= kQrbSmemBudget) {
    L.vloc2 = o;
    o += (size_t)QB * L.ld * esz;
  }
  L.total = o;
  return L;
}

// Y <- (I - V op(T) V^H) Y on rows [r0, M) of ncol local columns (column j of
// Y at Y + ycols[j] * ld).  op(T) = T^H when herm (Q_p^H), T otherwise (Q_p).
// V (QB columns, stride ld, rows r0..M-1 valid) and T are in shared memory;
// QB and ncol are multiples of 4.  Register tiles of 4 x 4 keep the
// shared-memory traffic at two loads per four complex FMAs.
template <typename CX, int QB>
AGB_DEV void qrb_apply(CX* Y, const int* ycols, int ncol, const CX* V, const CX* T, CX* W, CX* W2, int r0, int M,
                       int ld, bool herm) {
  typedef typename cx_traits<CX>::R Rt;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int NW = QBT / 32;
  if (ncol == 0) return;
  // W = V^H Y: a warp per 4 x 4 tile of W, lanes split the rows; the 32 partial
  // sums (16 complex) are reduced so that lane l ends with sum number l
  const int ti_n = QB / 4, tj_n = ncol / 4;
  for (int tile = wid; tile < ti_n * tj_n; tile += NW) {
    const int i0 = (tile / tj_n) * 4, y0 = (tile % tj_n) * 4;
    const CX* vc[4];
    const CX* yc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      vc[k] = V + (size_t)(i0 + k) * ld;
      yc[k] = Y + (size_t)ycols[y0 + k] * ld;
    }
    Rt a[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) a[k] = 0;
    for (int r = r0 + lane; r < M; r += 32) {
      CX v[4], y[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k] = vc[k][r];
        y[k] = yc[k][r];
      }
#pragma unroll
      for (int ii = 0; ii < 4; ++ii)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          // conj(v) * y
          a[(ii * 4 + jj) * 2] = fma(v[ii].x, y[jj].x, fma(v[ii].y, y[jj].y, a[(ii * 4 + jj) * 2]));
          a[(ii * 4 + jj) * 2 + 1] = fma(v[ii].x, y[jj].y, fma(-v[ii].y, y[jj].x, a[(ii * 4 + jj) * 2 + 1]));
        }
    }
#pragma unroll
    for (int o = 16, n = 32; o >= 1; o >>= 1, n >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < n / 2; ++k) {
        const Rt send = up ? a[k] : a[k + n / 2];
        const Rt keep = up ? a[k + n / 2] : a[k];
        a[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    // lane l holds value l = ((ii * 4 + jj) * 2 + component)
    const int comp = lane & 1, jj = (lane >> 1) & 3, ii = lane >> 3;
    Rt* wp = (Rt*)&W[(i0 + ii) * ncol + y0 + jj];
    wp[comp] = a[0];
  }
  __syncthreads();
  // W2 = op(T) W   (T upper triangular)
  for (int pr = tid; pr < QB * ncol; pr += QBT) {
    const int i = pr / ncol, y = pr % ncol;
    CX acc = czero<CX>();  // T's other triangle is stored as zeros: no bound on k
    if (herm) {
#pragma unroll
      for (int k = 0; k < QB; ++k) cfmac(acc, T[k * QB + i], W[k * ncol + y]);  // conj(T[k][i]) W[k][y]
    } else {
#pragma unroll
      for (int k = 0; k < QB; ++k) cfma(acc, T[i * QB + k], W[k * ncol + y]);
    }
    W2[pr] = acc;
  }
  __syncthreads();
  // Y -= V W2: a warp per block of 128 rows x 4 columns, lane rows r, r+32, r+64, r+96
  const int L = M - r0;
  const int rb_n = (L + 127) / 128;
  for (int task = wid; task < rb_n * tj_n; task += NW) {
    const int rbase = r0 + (task / tj_n) * 128 + lane, y0 = (task % tj_n) * 4;
    CX acc[4][4];
#pragma unroll
    for (int jr = 0; jr < 4; ++jr)
#pragma unroll
      for (int jc = 0; jc < 4; ++jc) acc[jr][jc] = czero<CX>();
#pragma unroll 4
    for (int i = 0; i < QB; ++i) {
      CX v[4], w[4];
#pragma unroll
      for (int jr = 0; jr < 4; ++jr) {
        const int r = rbase + 32 * jr;
        v[jr] = (r < M) ? V[(size_t)i * ld + r] : czero<CX>();
      }
#pragma unroll
      for (int jc = 0; jc < 4; ++jc) w[jc] = W2[i * ncol + y0 + jc];
#pragma unroll
      for (int jr = 0; jr < 4; ++jr)
#pragma unroll
        for (int jc = 0; jc < 4; ++jc) cfma(acc[jr][jc], v[jr], w[jc]);
    }
#pragma unroll
    for (int jc = 0; jc < 4; ++jc) {
      CX* yc = Y + (size_t)ycols[y0 + jc] * ld;
#pragma unroll
      for (int jr = 0; jr < 4; ++jr) {
        const int r = rbase + 32 * jr;
        if (r < M) yc[r] = csub(yc[r], acc[jr][jc]);
      }
    }
  }
  __syncthreads();
}

// One factorisation; a launch holds one, or two on a cluster each (the sweeps
// from the two ends of a chain, each a sequence of dependent factorisations on 16
// of the 152 SMs).
template <typename CX>
struct QrbProb {
  const CX* A;
  CX *Q, *R, *Vg, *Tg;
  int M, N, transA, trans_out;
};

template <typename CX, int NK, bool PAD>
__global__ void __launch_bounds__(QBT, 1) qr_blocked_kernel(QrbProb<CX> pr0, QrbProb<CX> pr1, int C) {
  const QrbProb<CX> pr = (int)blockIdx.x < C ? pr0 : pr1;
  const CX* __restrict__ Ain = pr.A;
  CX *Q = pr.Q, *R = pr.R, *Vg = pr.Vg, *Tg = pr.Tg;
  const int M = pr.M, N = pr.N, transA = pr.transA, trans_out = pr.trans_out;
  typedef typename cx_traits<CX>::R Rt;
  constexpr int QB = QrbCfg<CX>::QB;
  cg::cluster_group cluster = cg::this_cluster();
  const int q = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int kk = M < N ? M : N;
  const int vrows = PAD ? 32 * NK : M;
  const QrbLayout Lo = qrb_layout(sizeof(CX), QB, M, N, C, vrows);
  const int ld = Lo.ld;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CX* pan = (CX*)(smem_raw + Lo.panels);  // own panels: local column s * QB + jj
  CX* Vl = (CX*)(smem_raw + Lo.vloc);
  CX* V2 = (CX*)(smem_raw + Lo.vloc2);
  CX* W = (CX*)(smem_raw + Lo.w);
  CX* W2 = (CX*)(smem_raw + Lo.w2);
  CX* Tl = (CX*)(smem_raw + Lo.t);
  CX* vbuf = (CX*)(smem_raw + Lo.vb);  // [2][vrows] the current reflector, double-buffered
  __shared__ int ycols[kQrbMaxCols];
  __shared__ int ycount;
  __shared__ CX taus[QB];
  constexpr int TP = QB + 1;
  constexpr bool HOLD = NK * sizeof(CX) <= 128;  // the reflector stays in registers between product and update
  __shared__ CX Ssh[QB * TP], Tsh[QB * TP];
  // own panels: p = q + s * C
  const int nown = (q < Lo.P) ? (Lo.P - q + C - 1) / C : 0;
  // ---- load own columns of op(A)
  for (int s = 0; s < nown; ++s) {
    const int p = q + s * C;
    for (int jj = wid; jj < QB; jj += QBT / 32) {
      const int c = p * QB + jj;
      CX* col = pan + (size_t)(s * QB + jj) * ld;
      for (int r = lane; r < M; r += 32)
        col[r] = (c < N) ? (transA ? Ain[(int64_t)c * M + r] : Ain[(int64_t)r * N + c]) : czero<CX>();
    }
  }
  __syncthreads();
  // ---- factorisation, panel by panel
  for (int p = 0; p < Lo.PF; ++p) {
    const int pb = p * QB;
    const int owner = p % C;
    if (q == owner) {
      const int s = p / C;
      CX* P0 = pan + (size_t)(s * QB) * ld;
      const int pw = min(QB, N - pb);  // columns in the panel
      const int bw = min(QB, kk - pb);  // columns factored
      // The panel in registers: warp w holds column w, lane `lane` its rows
      // lane + 32 k.  Per column the owner warp forms the reflector and writes
      // v to a shared vector (double-buffered by column parity: the next
      // owner cannot overwrite it before every warp has passed the barrier of
      // the column in between); one block barrier; the later warps apply it.
      CX x[NK];
      if (wid < pw) {
        const CX* col = P0 + (size_t)wid * ld;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const int r = lane + 32 * k;
          x[k] = (r < M) ? col[r] : czero<CX>();
        }
      }
      CX* Vp = Vg + (size_t)p * QB * M;
      // T[k][i] = -tau_i sum_{k <= m < i} T[k][m] S[m][i] (lane k of warp 0), T[i][i] = tau_i
      auto t_column = [&](int i) {
        if (lane < i) {
          CX acc = czero<CX>();
          for (int m = lane; m < i; ++m) cfma(acc, Tsh[lane * TP + m], Ssh[m * TP + i]);
          const CX ti = taus[i];
          Tsh[lane * TP + i] = cmul(mk<CX>(-ti.x, -ti.y), acc);
        } else if (lane < QB) {
          Tsh[lane * TP + i] = lane == i ? taus[i] : czero<CX>();
        }
        __syncwarp();
      };
      for (int jj = 0; jj < bw; ++jj) {
        const int c = pb + jj;
        CX* vb = vbuf + (size_t)(jj & 1) * vrows;
        if (wid == jj) {
          Rt p0 = 0, p1 = 0;
          CX am = czero<CX>();
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            const int r = lane + 32 * k;
            const Rt z = cabs2(x[k]);  // rows past M hold zeros
            if (k & 1) p1 += r > c ? z : Rt(0);
            else p0 += r > c ? z : Rt(0);
            if (r == c) am = x[k];
          }
          const Rt xn2 = warp_sum(p0 + p1);
          CX alpha;
          alpha.x = __shfl_sync(0xffffffffu, am.x, c & 31);
          alpha.y = __shfl_sync(0xffffffffu, am.y, c & 31);
          CX t, sc;
          Rt beta;
          reflector_unscaled(alpha, xn2, beta, t, sc);
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            const int r = lane + 32 * k;
            const CX u = cmul(x[k], sc);
            const CX v = r > c ? u : r == c ? mk<CX>(1, 0) : czero<CX>();
            if (PAD || r < M) vb[r] = v;
            x[k] = r > c ? u : r == c ? mk<CX>(beta, 0) : x[k];  // v below the diagonal
          }
          if (lane == 0) taus[jj] = t;
        }
        __syncthreads();
        // v_c^H x: for the later columns H_c^H = I - conj(tau) v v^H is applied, for
        // the earlier ones (x = v_w below its diagonal) it is conj(S[w][jj])
        if (wid != jj && wid < pw) {
          CX a0 = czero<CX>(), a1 = czero<CX>();
          CX v[HOLD ? NK : 1];
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            const int r = lane + 32 * k;
            const CX vr = PAD || r < M ? vb[r] : czero<CX>();  // zero above row c and past M
            if (HOLD) v[HOLD ? k : 0] = vr;
            if (k & 1) cfmac(a1, vr, x[k]);
            else cfmac(a0, vr, x[k]);
          }
          const CX acc = warp_csum(cadd(a0, a1));
          if (wid > jj) {
            const CX tw = cmul(cconj(taus[jj]), acc);
#pragma unroll
            for (int k = 0; k < NK; ++k) {
              const int r = lane + 32 * k;
              if (HOLD) x[k] = csub(x[k], cmul(v[HOLD ? k : 0], tw));
              else if (PAD || r < M) x[k] = csub(x[k], cmul(vb[r], tw));
            }
          } else if (lane == 0) {
            Ssh[wid * TP + jj] = cconj(acc);
          }
        }
        for (int r = tid; r < M; r += QBT) Vp[(size_t)jj * M + r] = vb[r];
        if (wid == 0 && jj > 0) t_column(jj - 1);  // S[.][jj-1] is complete since the barrier
      }
      if (wid < pw) {
        CX* col = P0 + (size_t)wid * ld;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const int r = lane + 32 * k;
          if (r < M) col[r] = x[k];
        }
      }
      __syncthreads();
      if (wid == 0) {
        if (bw > 0) t_column(bw - 1);
        CX* Tp = Tg + (size_t)p * QB * QB;
        for (int e = lane; e < QB * QB; e += 32)
          Tp[e] = e % QB < bw && e / QB < bw ? Tsh[(e / QB) * TP + e % QB] : czero<CX>();
      }
      for (int e = tid; e < (QB - bw) * M; e += QBT) Vp[(size_t)bw * M + e] = czero<CX>();  // past bw
      __threadfence();  // V_p, T_p visible to the cluster before the barrier
    }
    cluster.sync();
    // Q_p^H on own later panels (p' > p)
    if (tid == 0) {
      int nc = 0;
      for (int s = 0; s < nown; ++s) {
        const int pp = q + s * C;
        if (pp > p)
          for (int jj = 0; jj < QB; ++jj) ycols[nc++] = s * QB + jj;
      }
      ycount = nc;
    }
    __syncthreads();
    const int ncol = ycount;
    if (ncol > 0) {
      const CX* Vp = Vg + (size_t)p * QB * M;
      for (int jj = wid; jj < QB; jj += QBT / 32) {
#pragma unroll 8
        for (int r = pb + lane; r < M; r += 32) Vl[(size_t)jj * ld + r] = __ldcg(Vp + (size_t)jj * M + r);
      }
      for (int e = tid; e < QB * QB; e += QBT) Tl[e] = __ldcg(Tg + (size_t)p * QB * QB + e);
      __syncthreads();
      qrb_apply<CX, QB>(pan, ycols, ncol, Vl, Tl, W, W2, pb, M, ld, true);
    }
  }
  // ---- R = upper triangle of the factored columns (kk x N)
  for (int s = 0; s < nown; ++s) {
    const int p = q + s * C;
    for (int jj = wid; jj < QB; jj += QBT / 32) {
      const int c = p * QB + jj;
      if (c >= N) continue;
      const CX* col = pan + (size_t)(s * QB + jj) * ld;
      for (int r = lane; r < kk; r += 32) {
        const CX val = (r <= c) ? col[r] : czero<CX>();
        if (trans_out) R[(int64_t)c * kk + r] = val;
        else R[(int64_t)r * N + c] = val;
      }
    }
  }
  __syncthreads();
  // ---- thin Q: Z = [I; 0] in the panel storage, Z <- Q_p Z backwards.  The columns
  // are dealt to the CTAs one by one (column q + m C in slot m), so that each
  // panel's work, on the columns from its first on, is spread evenly: by panels,
  // the last CTA had every panel to apply to all its columns.
  const int nq = q < kk ? (kk - q + C - 1) / C : 0;      // own columns of Q
  const int nq4 = (nq + 3) & ~3;                    // slots in use (the update takes fours) <= npo QB
  for (int m = wid; m < nq4; m += QBT / 32) {
    const int c = m < nq ? q + m * C : -1;
    CX* col = pan + (size_t)m * ld;
    for (int r = lane; r < M; r += 32) col[r] = (r == c) ? mk<CX>(1, 0) : czero<CX>();
  }
  __syncthreads();
  // V_p to buffer buf by asynchronous copies (its rows >= pb), T_p with it
  auto read_panel = [&](int p, CX* Vd) {
    const int pb = p * QB;
    const CX* Vp = Vg + (size_t)p * QB * M;
    for (int jj = wid; jj < QB; jj += QBT / 32)
      for (int r = pb + lane; r < M; r += 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(Vd + (size_t)jj * ld + r)),
                     "l"(Vp + (size_t)jj * M + r), "n"((int)sizeof(CX))
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const bool ahead = Lo.vloc2 != Lo.vloc;
  const int plast = nq4 > 0 ? Lo.PF - 1 : -1;
  if (ahead && plast >= 0) read_panel(plast, Vl);
  for (int p = plast; p >= 0; --p) {
    const int pb = p * QB;
    // slots of the columns >= pb (columns below pb are e_c, which Q_p leaves alone)
    const int m0 = (pb > q ? (pb - q + C - 1) / C : 0) & ~3;
    const int ncol = nq4 > m0 ? nq4 - m0 : 0;
    for (int m = tid; m < ncol; m += QBT) ycols[m] = m0 + m;
    CX* Vd = ahead && ((plast - p) & 1) ? V2 : Vl;
    for (int e = tid; e < QB * QB; e += QBT) Tl[e] = __ldcg(Tg + (size_t)p * QB * QB + e);
    if (!ahead) read_panel(p, Vd);
    if (ahead && p > 0) {
      read_panel(p - 1, Vd == Vl ? V2 : Vl);  // that buffer's panel was applied before the last barrier
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    qrb_apply<CX, QB>(pan, ycols, ncol, Vd, Tl, W, W2, pb, M, ld, false);
    if (ncol == 0) __syncthreads();  // the update's last barrier frees the buffers
  }
  // ---- write Q (M x kk, or its transpose)
  if (trans_out) {
    for (int m = wid; m < nq; m += QBT / 32) {
      const CX* col = pan + (size_t)m * ld;
      for (int r = lane; r < M; r += 32) Q[(int64_t)(q + m * C) * M + r] = col[r];
    }
  } else {
    for (int m = wid; m < nq; m += QBT / 32) {
      const CX* col = pan + (size_t)m * ld;
      for (int r = lane; r < M; r += 32) Q[(int64_t)r * kk + q + m * C] = col[r];
    }
  }
  cluster.sync();
}

template <typename CX>
using QrbKernel = void (*)(QrbProb<CX>, QrbProb<CX>, int);

// The instance whose per-lane register column (NK rows per lane) covers M rows;
// nullptr above 1024 rows (512 for complex128, whose columns would spill).
template <typename CX>
QrbKernel<CX> qrb_kernel_for(int M, bool pad) {
  if constexpr (sizeof(CX) == 8) {
    if (pad && M <= 128) return qr_blocked_kernel<CX, 4, true>;
    if (pad && M <= 256) return qr_blocked_kernel<CX, 8, true>;
    if (pad && M <= 512) return qr_blocked_kernel<CX, 16, true>;
  }
  if (M <= 128) return qr_blocked_kernel<CX, 4, false>;
  if (M <= 256) return qr_blocked_kernel<CX, 8, false>;
  if (M <= 512) return qr_blocked_kernel<CX, 16, false>;
  if constexpr (sizeof(CX) == 8) {
    if (M <= 1024) return qr_blocked_kernel<CX, 32, false>;
  }
  return nullptr;
}

// Cluster size for the blocked kernel: the largest of 16, 8, 4, 2 CTAs not
// above the panel count whose shared memory fits; 0 if none.
template <typename CX>
int qrb_cluster_size(int M, int N) {
  const QrbKernel<CX> kern = qrb_kernel_for<CX>(M, true);
  if (!kern) return 0;
  constexpr int QB = QrbCfg<CX>::QB;
  const int P = (N + QB - 1) / QB;
  static int allow16 = -1;
  for (int C : {16, 8, 4, 2}) {
    if (C > P) continue;
    const QrbLayout L = qrb_layout(sizeof(CX), QB, M, N, C, M);
    if (L.total > kQrbSmemBudget || L.npo * QB > kQrbMaxCols) continue;
    if (C == 16) {
      if (allow16 < 0) {
        allow16 = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                cudaSuccess &&
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kQrbSmemBudget) == cudaSuccess) {
          cudaLaunchConfig_t cfg = {};
          cfg.gridDim = dim3(16, 1, 1);
          cfg.blockDim = dim3(QBT, 1, 1);
          cfg.dynamicSmemBytes = kQrbSmemBudget;
          cudaLaunchAttribute attr[1];
          attr[0].id = cudaLaunchAttributeClusterDimension;
          attr[0].val.clusterDim.x = 16;
          attr[0].val.clusterDim.y = 1;
          attr[0].val.clusterDim.z = 1;
          cfg.attrs = attr;
          cfg.numAttrs = 1;
          int ncl = 0;
          if (cudaOccupancyMaxActiveClusters(&ncl, kern, &cfg) == cudaSuccess && ncl > 0)
            allow16 = 1;
        }
        cudaGetLastError();
      }
      if (!allow16) continue;
    }
    return C;
  }
  return 0;
}

}  // namespace

// Workspace of the blocked kernel: reflector panels (M x QB each) and T factors.
size_t qr_blocked_workspace(int esz, int M, int N) {
  const int QB = esz == 8 ? QrbCfg<float2>::QB : QrbCfg<double2>::QB;
  const int kk = M < N ? M : N;
  const int PF = (kk + QB - 1) / QB;
  return agb_align((size_t)PF * QB * M * esz) + agb_align((size_t)PF * QB * QB * esz);
}

// probs[0 .. count), count 1 or 2, ws as large as their workspaces together; two
// take one launch only if they split over the same number of CTAs.
template <typename CX>
static int launch_qrb(QrbProb<CX>* probs, int count, void* ws, size_t ws_bytes, cudaStream_t s) {
  constexpr int QB = QrbCfg<CX>::QB;
  size_t at = 0;
  int C = 0, maxM = 0;
  for (int i = 0; i < count; ++i) {
    QrbProb<CX>& p = probs[i];
    const int c = qrb_cluster_size<CX>(p.M, p.N);
    if (c == 0 || (i > 0 && c != C)) return AGB_ERR_UNSUPPORTED;
    C = c;
    maxM = p.M > maxM ? p.M : maxM;
    const int kk = p.M < p.N ? p.M : p.N, PF = (kk + QB - 1) / QB;
    p.Vg = (CX*)((char*)ws + at);
    p.Tg = (CX*)((char*)ws + at + agb_align((size_t)PF * QB * p.M * sizeof(CX)));
    at += qr_blocked_workspace(sizeof(CX), p.M, p.N);
  }
  if (ws_bytes < at) return AGB_ERR_WORKSPACE;
  auto shared = [&](bool padded) {
    size_t most = 0;
    for (int i = 0; i < count; ++i) {
      const int vrows = padded ? (maxM <= 128 ? 128 : maxM <= 256 ? 256 : 512) : probs[i].M;
      const size_t sm = qrb_layout(sizeof(CX), QB, probs[i].M, probs[i].N, C, vrows).total;
      most = sm > most ? sm : most;
    }
    return most;
  };
  // padded where there is such an instance and its buffers fit
  const bool pad = sizeof(CX) == 8 && maxM <= 512 && shared(true) <= kQrbSmemBudget;
  const size_t smem = shared(pad);
  const QrbKernel<CX> kern = qrb_kernel_for<CX>(maxM, pad);
  if (C > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return AGB_ERR_UNSUPPORTED;
  }
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return AGB_ERR_UNSUPPORTED;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(count * C, 1, 1);
  cfg.blockDim = dim3(QBT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, probs[0], probs[count - 1], C);
  agb_note_launch();
  if (err != cudaSuccess) {
    cudaGetLastError();
    return AGB_ERR_UNSUPPORTED;
  }
  return AGB_OK;
}

template <typename CX>
int launch_qr_blocked(const CX* A, int M, int N, int transA, CX* Q, CX* R, int trans_out, void* ws, size_t ws_bytes,
                      cudaStream_t s) {
  QrbProb<CX> p = {A, Q, R, nullptr, nullptr, M, N, transA, trans_out};
  return launch_qrb<CX>(&p, 1, ws, ws_bytes, s);
}

template int launch_qr_blocked<float2>(const float2*, int, int, int, float2*, float2*, int, void*, size_t,
                                       cudaStream_t);
template int launch_qr_blocked<double2>(const double2*, int, int, int, double2*, double2*, int, void*, size_t,
                                        cudaStream_t);

template <typename CX>
static int qr_pair(const int64_t* probs, void* ws, size_t ws_bytes, cudaStream_t s) {
  QrbProb<CX> p[2];
  for (int i = 0; i < 2; ++i) {
    const int64_t* d = probs + 7 * i;
    if (d[1] * d[2] < 64 * 64) return AGB_ERR_UNSUPPORTED;  // these take the unblocked kernel
    p[i] = {(const CX*)d[0], (CX*)d[4], (CX*)d[5], nullptr, nullptr, (int)d[1], (int)d[2], (int)d[3], (int)d[6]};
  }
  return launch_qrb<CX>(p, 2, ws, ws_bytes, s);
}

// Two factorisations in one launch where both take the blocked kernel with the
// same cluster size, one after the other otherwise.  512 x 256, then its mirror image:
// 1164 us one after the other, 582 us side by side (a chain of 40 sites at chi 256 to
// its mixed form: 16.9 -> 9.8 ms at 657 us each).
extern "C" int agb_qr_pair(int dtype, const int64_t* probs, void* ws, size_t ws_bytes, void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (!probs || !ws) return AGB_ERR_ARG;
  size_t need[2];
  for (int i = 0; i < 2; ++i) {
    const int64_t* d = probs + 7 * i;
    if (!d[0] || !d[4] || !d[5] || d[1] <= 0 || d[2] <= 0) return AGB_ERR_ARG;
    if (d[1] > 8192 || d[2] > 0x7fffffff) return AGB_ERR_UNSUPPORTED;
    need[i] = agb_qr_workspace(dtype, (int)d[1], (int)d[2]);
  }
  if (ws_bytes < need[0] + need[1]) return AGB_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  const int rc = dtype == AGB_C64 ? qr_pair<float2>(probs, ws, ws_bytes, s) : qr_pair<double2>(probs, ws, ws_bytes, s);
  if (rc == AGB_OK) return AGB_OK;
  for (int i = 0; i < 2; ++i) {
    const int64_t* d = probs + 7 * i;
    const int r = agb_qr(dtype, (const void*)d[0], (int)d[1], (int)d[2], (int)d[3], (void*)d[4], (void*)d[5],
                         (int)d[6], (char*)ws + (i ? need[0] : 0), need[i], stream);
    if (r != AGB_OK) return r;
  }
  return AGB_OK;
}
