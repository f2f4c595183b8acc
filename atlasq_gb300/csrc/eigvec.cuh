// Device pieces of the eigenvector phase shared by the batched kernels (heevd.cu)
// and the one-kernel form for small gates (two_site.cu).
#pragma once
#include <float.h>

#include "heevd.cuh"

template <typename R> struct rlim;

// Reciprocal of an LU pivot, the pivot first floored at piv in magnitude (a
// zero pivot takes +piv).  The factors store reciprocals so that the back
// substitution's dependent chain is multiply-adds only.
template <typename R>
__device__ __forceinline__ R inv_pivot(R u, R piv) {
  if (fabs(u) < piv) u = copysign(piv, u == R(0) ? R(1) : u);
  return R(1) / u;
}
template <> struct rlim<float> {
  static AGB_HD float eps() { return FLT_EPSILON; }
  static AGB_HD float pivmin() { return 1e-30f; }
  static AGB_HD float huge() { return FLT_MAX; }
};
template <> struct rlim<double> {
  static AGB_HD double eps() { return DBL_EPSILON; }
  static AGB_HD double pivmin() { return 1e-290; }
  static AGB_HD double huge() { return DBL_MAX; }
};

template <typename R>
AGB_DEV R cluster_tol(const R* lam, int ell, double tolrel) {
  const R scale = fmax(fabs(lam[0]), fabs(lam[ell - 1]));
  return (R)tolrel * fmax(scale, rlim<R>::pivmin());
}

template <typename R>
AGB_DEV bool in_cluster(const R* lam, int ell, int t, R tol) {
  const bool left = (t > 0) && (lam[t - 1] - lam[t]) <= tol;
  const bool right = (t + 1 < ell) && (lam[t] - lam[t + 1]) <= tol;
  return left || right;
}

// Shift of cluster member j: its own eigenvalue.  LAPACK's stein walks the
// shifts of near-equal members apart by 10 eps |lambda| each, which is
// harmless in double precision but in float32 moves the last members of a
// cluster by ~1e-6 |lambda| per member, toward the first eigenvalue below
// the cluster.  Measured on 64-qubit HEA gates (chi 512): eight members within
// 6.6e-6 lambda_0 of each other and the next eigenvalue 1.2e-5 below; the
// walked shift of the eighth member amplified that outside eigenvector about
// a sixth as much as its own, and after the Gram-Schmidt pass had removed the
// directions of the first seven members, what remained was 92% the outside
// eigenvector.  With unwalked shifts the outside component is suppressed by
// (bisection error / gap) per solve; members with equal shifts still get
// independent iterates from their own random starts, which Gram-Schmidt
// separates.  The shift is also kept above the midpoint to the eigenvalue
// below the cluster.
template <typename R>
AGB_DEV R member_shift(const R* lam, int ell, int j, int t1) {
  const R sh = lam[j];
  if (t1 >= ell) return sh;
  return fmax(sh, R(0.5) * (lam[t1 - 1] + lam[t1]));
}

// LU with partial pivoting of T - lam I into the interleaved factor arrays
// (column t of each), as in invit_kernel.
template <typename R>
AGB_DEV void tri_lu(const R* d, const R* e, int n, R lam, R piv, R* U0, R* U1, R* U2, R* Lm, R* Pv,
                    int64_t L, int t) {
  R u0 = d[0] - lam, u1 = (n > 1) ? e[0] : R(0), u2 = 0;
  for (int i = 0; i < n - 1; ++i) {
    const R sub = e[i], nd = d[i + 1] - lam, ns = (i + 1 < n - 1) ? e[i + 1] : R(0);
    const bool keep = fabs(u0) >= fabs(sub);  // selects: one division serves both cases
    if (keep && u0 == R(0)) u0 = piv;
    const R a0 = keep ? u0 : sub, a1 = keep ? u1 : nd, a2 = keep ? u2 : ns, pv = keep ? R(0) : R(1);
    const R m = (keep ? sub : u0) / a0;
    u0 = (keep ? nd : u1) - m * a1;
    u1 = (keep ? ns : u2) - m * a2;
    u2 = 0;
    U0[i * L + t] = inv_pivot(a0, piv);
    U1[i * L + t] = a1;
    U2[i * L + t] = a2;
    Lm[i * L + t] = m;
    Pv[i * L + t] = pv;
  }
  U0[(int64_t)(n - 1) * L + t] = inv_pivot(u0, piv);
  U1[(int64_t)(n - 1) * L + t] = 0;
  U2[(int64_t)(n - 1) * L + t] = 0;
}

// y <- (T - lam I)^{-1} (s * y) for column t of Y (stride L) with the stored
// factors of column t; returns ||y||^2.  Factor and iterate loads do not depend
// on the recurrence, so each chunk of IB steps loads them into registers first
// (IB loads in flight instead of one dependent load per step).
template <typename R>
AGB_DEV R tri_solve_pf(R* Y, int n, const R* U0, const R* U1, const R* U2, const R* Lm, const R* Pv, int64_t L,
                       int t, R piv, R s) {
  constexpr int IB = 16;
  R bi = Y[t] * s;
  for (int i0 = 0; i0 < n - 1; i0 += IB) {
    R yb[IB], pv[IB], lm[IB];
#pragma unroll
    for (int k = 0; k < IB; ++k) {
      const int i = i0 + k;
      if (i < n - 1) {
        yb[k] = Y[(int64_t)(i + 1) * L + t];
        pv[k] = Pv[(int64_t)i * L + t];
        lm[k] = Lm[(int64_t)i * L + t];
      }
    }
#pragma unroll
    for (int k = 0; k < IB; ++k) {
      const int i = i0 + k;
      if (i < n - 1) {
        R bn = yb[k] * s;
        if (pv[k] != R(0)) {
          const R tmp = bi;
          bi = bn;
          bn = tmp;
        }
        Y[(int64_t)i * L + t] = bi;
        bi = bn - lm[k] * bi;
      }
    }
  }
  Y[(int64_t)(n - 1) * L + t] = bi;
  R x1 = 0, x2 = 0, nrm = 0;
  for (int i0 = n - 1; i0 >= 0; i0 -= IB) {
    R u0[IB], u1[IB], u2[IB], yb[IB];
#pragma unroll
    for (int k = 0; k < IB; ++k) {
      const int i = i0 - k;
      if (i >= 0) {
        u0[k] = U0[(int64_t)i * L + t];
        u1[k] = U1[(int64_t)i * L + t];
        u2[k] = U2[(int64_t)i * L + t];
        yb[k] = Y[(int64_t)i * L + t];
      }
    }
#pragma unroll
    for (int k = 0; k < IB; ++k) {
      const int i = i0 - k;
      if (i >= 0) {
        const R x = (yb[k] - u1[k] * x1 - u2[k] * x2) * u0[k];  // u0: reciprocal pivot
        Y[(int64_t)i * L + t] = x;
        nrm += x * x;
        x2 = x1;
        x1 = x;
      }
    }
  }
  return nrm;
}

// CGS2 of column jj of the staged cluster block Z (n x c in shared
// memory, row stride ld) against its columns [0, jj), then normalisation (block-wide).
template <typename R>
AGB_DEV void cgs2_block_smem(R* Z, int n, int ld, int jj, R* coef, R* red, R* part) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  for (int pass = 0; pass < 2 && jj > 0; ++pass) {
    for (int c0 = 0; c0 < jj; c0 += 32) {
      const int i = c0 + lane;
      R a = 0;
      if (i < jj)
        for (int r = wid; r < n; r += nw) a += Z[(int64_t)r * ld + i] * Z[(int64_t)r * ld + jj];
      part[wid * 32 + lane] = a;
      __syncthreads();
      if (wid == 0 && i < jj) {
        R sum = 0;
        for (int w = 0; w < nw; ++w) sum += part[w * 32 + lane];
        coef[i] = sum;
      }
      __syncthreads();
    }
    for (int r = wid; r < n; r += nw) {
      R* row = Z + (int64_t)r * ld;
      R acc = 0;
      for (int i = lane; i < jj; i += 32) acc += coef[i] * row[i];
      acc = warp_sum(acc);
      if (lane == 0) row[jj] -= acc;
    }
    __syncthreads();
  }
  R psum = 0;
  for (int r = tid; r < n; r += nt) psum += Z[(int64_t)r * ld + jj] * Z[(int64_t)r * ld + jj];
  const R nrm = block_sum(psum, red);
  const R sc = R(1) / sqrt(fmax(nrm, rlim<R>::pivmin()));
  for (int r = tid; r < n; r += nt) Z[(int64_t)r * ld + jj] *= sc;
  __syncthreads();
}

