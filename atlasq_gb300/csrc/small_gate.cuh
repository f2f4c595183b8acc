// The eigenvector phase, X V, rank selection and the repair pass of a small
// complex64 gate (m, n, ell <= 64) in one CTA, included by two_site.cu.
//
// As separate kernels these are 15 launches of 2-30 us for the vector phase and
// as many again, idle, for the repair pass; for a 10-qubit circuit at chi 32 the
// launches alone took half of the time.  Here everything between the
// eigenvalues and the scatter stays in shared memory: inverse iteration (one
// thread per vector), clusters (the whole CTA, one after another),
// back-transformation (a warp per two columns), Newton-Schulz polish and X V
// (4 x 4 outputs per thread), rank rule; and a gate that needs the repair goes
// round again.  The arithmetic is that of the batched kernels, sum by sum.
//
// What bounds it: the serial chains of the solves and of the reflectors (latency
// of one CTA per gate), not throughput.  Measured (GB300): one gate of a 10-qubit
// chain at chi 16, 33 launches and 200 us of device time before, 14 and 147 us
// now, 513 -> 430 us a call; ten layers of a device-resident 10-qubit circuit
// (the idle repair pass goes too) 5.4 -> 4.2 ms.  The limit is shared memory: the
// LU factors (5 n ell floats) and the iterates of 64 vectors take 96 KB, those of
// 128 would not fit, and the batched kernels fill the chip there.

constexpr int kSmallMax = 64;   // largest m, n and ell
constexpr int kSmallThreads = 256;

struct SmallLayout {
  size_t y, a0, a1, a2, total;  // float [n ell]; complex [64 64] areas (the LU factors lie over a0..a2)
};
AGB_HD SmallLayout small_layout() {
  SmallLayout L;
  const size_t area = (size_t)kSmallMax * kSmallMax * sizeof(float2);
  L.y = 0;
  L.a0 = (size_t)kSmallMax * kSmallMax * sizeof(float);
  L.a1 = L.a0 + area;
  L.a2 = L.a1 + area;
  L.total = L.a2 + area;
  return L;
}

// out(i, j) = sum_k a(i, k) b(k, j), k in order, for i < M, j < N: the SIMT GEMM's sum.
template <typename FA, typename FB, typename FS>
AGB_DEV void small_product(int M, int N, int K, FA a, FB b, FS store) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int i0 = 0; i0 < M; i0 += 64)
    for (int j0 = 0; j0 < N; j0 += 64) {
      float2 acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = czero<float2>();
      const int ni = (M - i0 + 15) / 16, nj = (N - j0 + 15) / 16;  // 16-wide strips in use
      for (int k = 0; k < K; ++k) {
        float2 av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          av[i] = (i < ni && i0 + ty + 16 * i < M) ? a(i0 + ty + 16 * i, k) : czero<float2>();
#pragma unroll
        for (int j = 0; j < 4; ++j)
          bv[j] = (j < nj && j0 + tx + 16 * j < N) ? b(k, j0 + tx + 16 * j) : czero<float2>();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < ni)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (j < nj) cfma(acc[i][j], av[i], bv[j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i0 + ty + 16 * i < M && j0 + tx + 16 * j < N) store(i0 + ty + 16 * i, j0 + tx + 16 * j, acc[i][j]);
    }
}

__global__ void __launch_bounds__(kSmallThreads) small_gate_kernel(int64_t* __restrict__ desc, int ng, char* ws,
                                                                    int guard, int repair) {
  typedef float2 CX;
  const int g = blockIdx.x;
  int64_t* D = desc + (int64_t)g * AGB_D_NFIELDS;
  HeevdProb* hp = (HeevdProb*)ws + g;
  const int chiL = (int)D[AGB_D_CHIL], chiR = (int)D[AGB_D_CHIR];
  const int m = 2 * chiL, n = 2 * chiR, ell = (int)D[AGB_D_ELL], cap = (int)D[AGB_D_CAP];
  const double eps = dbits(D[AGB_D_EPS]);
  char* slab = ws + D[AGB_D_WS];
  const Slab Ls = slab_layout(m, n, ell, sizeof(CX));
  const CX* X = (const CX*)(slab + Ls.X);
  CX* AV = (CX*)(slab + Ls.AV);
  CX* Vg = (CX*)(slab + Ls.V);
  double* sig2 = (double*)(slab + Ls.sig2);
  int* perm = (int*)(slab + Ls.perm);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int NT = kSmallThreads, NWP = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SmallLayout L = small_layout();
  float* Y = (float*)(smem_raw + L.y);
  float* lu = (float*)(smem_raw + L.a0);
  CX* a0 = (CX*)(smem_raw + L.a0);
  CX* a1 = (CX*)(smem_raw + L.a1);
  CX* a2 = (CX*)(smem_raw + L.a2);
  __shared__ float d[kSmallMax], e[kSmallMax], lam[kSmallMax], coef[kSmallMax], shs[kSmallMax];
  __shared__ CX tau[kSmallMax], pairc[kSmallMax / 2];
  __shared__ int cl[kSmallMax + 2];
  __shared__ float redf[32], part[256], tnorm_s;
  __shared__ unsigned omax, owmax;
  __shared__ double red[32], s_raw[kSmallMax], s_sorted[2 * kSmallMax];
  __shared__ float s_key[kSmallMax];
  __shared__ double partd[NT];
  __shared__ int nonfinite;
  const int mode0 = (int)D[AGB_D_MODE];
  for (int i = tid; i < n; i += NT) {
    d[i] = ((const float*)hp->d)[i];
    e[i] = (i < n - 1) ? ((const float*)hp->e)[i] : 0.f;
    tau[i] = (i < n - 1) ? ((const CX*)hp->tau)[i] : czero<CX>();
  }
  for (int i = tid; i < ell; i += NT) lam[i] = ((const float*)hp->lam)[i];
  // total = ||X||_F^2 to double accuracy
  SumAcc<float> xa;
  for (int i = tid; i < m * n; i += NT) xa.add(cabs2(X[i]));
  const double total_d = block_sum(xa.value(), red);
  const uint64_t seed = hp->seed;
  double ctol = hp->ctol;
  int nv = mode0 == 1 ? ell : min(hp->nvec, ell);
  int repaired = 0;
  for (int attempt = 0;; ++attempt) {
    if (tid == 0) {
      nonfinite = !isfinite(total_d);
      omax = owmax = 0u;
    }
    if (mode0 != 1) {
      // ---------------- inverse iteration, one thread per eigenvector
      const CX* H = (const CX*)hp->H;
      const int64_t ldh = hp->ldh;
      float *U0 = lu, *U1 = lu + n * ell, *U2 = lu + 2 * n * ell, *Lm = lu + 3 * n * ell, *Pv = lu + 4 * n * ell;
      const float tol = cluster_tol(lam, ell, ctol);
      if (tid == 0) {
        float tn = 0.f;
        for (int i = 0; i < n; ++i) tn = fmaxf(tn, fabsf(d[i]) + fabsf(e[i]) + (i ? fabsf(e[i - 1]) : 0.f));
        tnorm_s = tn;
        // clusters of the leading nv eigenvalues: count, then (t0, t1) pairs
        int found = 0, s = 0;
        for (int t = 1; t <= nv; ++t)
          if (t == nv || (lam[t - 1] - lam[t]) > tol) {
            if (t - s > 1) {
              cl[1 + 2 * found] = s;
              cl[2 + 2 * found] = t;
              ++found;
            }
            s = t;
          }
        cl[0] = nv < 2 ? 0 : found;
      }
      __syncthreads();
      const float piv = rlim<float>::eps() * fmaxf(tnorm_s, rlim<float>::pivmin());
      if (tid < nv && !in_cluster(lam, nv, tid, tol)) {
        const int t = tid;
        tri_lu(d, e, n, lam[t], piv, U0, U1, U2, Lm, Pv, (int64_t)ell, t);
        float nrm = 0.f;
        const uint64_t per = (uint64_t)((n + 3) / 4);
        for (int i0 = 0; i0 < n; i0 += 4) {
          const uint64_t idx = (uint64_t)t * per + (uint64_t)(i0 >> 2);
          const philox_out o = philox4x32_10((uint32_t)idx, (uint32_t)(idx >> 32), 0x11u, 0x5EEDu, (uint32_t)seed,
                                             (uint32_t)(seed >> 32));
          const uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (i0 + k < n) {
              const float b = (float)(int32_t)w[k] * 4.656612873077393e-10f;  // 2^-31
              Y[(i0 + k) * ell + t] = b;
              nrm += b * b;
            }
        }
        for (int it = 0; it < 3; ++it) {
          const float s = 1.f / sqrtf(fmaxf(nrm, rlim<float>::pivmin()));
          float bi = Y[t] * s;
#pragma unroll 4
          for (int i = 0; i < n - 1; ++i) {
            float bn = Y[(i + 1) * ell + t] * s;
            if (Pv[i * ell + t] != 0.f) {
              const float tmp = bi;
              bi = bn;
              bn = tmp;
            }
            Y[i * ell + t] = bi;
            bi = bn - Lm[i * ell + t] * bi;
          }
          Y[(n - 1) * ell + t] = bi;
          float x1 = 0.f, x2 = 0.f;
          nrm = 0.f;
#pragma unroll 4
          for (int i = n - 1; i >= 0; --i) {
            const float x = (Y[i * ell + t] - U1[i * ell + t] * x1 - U2[i * ell + t] * x2) * U0[i * ell + t];
            Y[i * ell + t] = x;
            nrm += x * x;
            x2 = x1;
            x1 = x;
          }
          if (!(nrm < 1e300) || !(nrm > 0.f)) {  // overflow / breakdown: restart from a unit vector
            for (int i = 0; i < n; ++i) Y[i * ell + t] = (i == (t % n)) ? 1.f : 0.f;
            nrm = 1.f;
          }
        }
        const float sc = 1.f / sqrtf(fmaxf(nrm, rlim<float>::pivmin()));
        for (int i = 0; i < n; ++i) Y[i * ell + t] *= sc;
      }
      __syncthreads();
      // ---------------- clusters: members in parallel, two rounds of [solve; Gram-Schmidt]
      for (int q = 0; q < cl[0]; ++q) {
        const int t0 = cl[1 + 2 * q], t1 = cl[2 + 2 * q], c = t1 - t0;
        if (tid < c) {
          shs[tid] = member_shift(lam, ell, t0 + tid, t1);
          tri_lu(d, e, n, shs[tid], piv, U0, U1, U2, Lm, Pv, (int64_t)ell, t0 + tid);
        }
        for (int idx = tid; idx < n * c; idx += NT) {
          const int r = idx / c, j = t0 + idx % c;
          Y[r * ell + j] = philox_normal(seed, (uint64_t)j * (uint64_t)n + r, 0x11u);
        }
        __syncthreads();
        for (int it = 0; it < 2; ++it) {
          if (tid < c) {
            const int j = t0 + tid;
            const float nrm = tri_solve_pf(Y, n, U0, U1, U2, Lm, Pv, (int64_t)ell, j, piv, 1.f);
            if (!(nrm < 1e300) || !(nrm > 0.f)) {  // overflow / breakdown: restart from a new random vector
              for (int r = 0; r < n; ++r)
                Y[r * ell + j] = philox_normal(seed ^ 0xABCDEFull, (uint64_t)(j + it + 1) * (uint64_t)n + r, 0x13u);
            } else {
              const float sc = 1.f / sqrtf(nrm);
              for (int r = 0; r < n; ++r) Y[r * ell + j] *= sc;
            }
          }
          __syncthreads();
          for (int jj = 0; jj < c; ++jj) cgs2_block_smem(Y + t0, n, ell, jj, coef, redf, part);
        }
      }
      // ---------------- back-transformation (reflectors in pairs), a warp per two columns
      for (int i = tid; i < n * n; i += NT) {
        const int r = i / n, c = i % n;
        a0[i] = c > r + 1 ? H[(int64_t)r * ldh + c] : c == r + 1 ? mk<CX>(1, 0) : czero<CX>();  // v_r
      }
      __syncthreads();
      for (int pi = wid; n - 2 - 2 * pi >= 1; pi += NWP) {  // v_{j-1}^H v_j, j = n - 2 - 2 pi
        const int j = n - 2 - 2 * pi;
        CX c = czero<CX>();
        for (int r = j + 1 + lane; r < n; r += 32) cfmac(c, a0[(j - 1) * n + r], a0[j * n + r]);
        c = warp_csum(c);
        if (lane == 0) pairc[pi] = c;
      }
      __syncthreads();
      for (int t0 = 2 * wid; t0 < nv; t0 += 2 * NWP) {
        const int t1 = t0 + 1;
        const bool h1 = t1 < nv;
        CX z0[2], z1[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int r = lane + 32 * k;
          z0[k] = r < n ? mk<CX>(Y[r * ell + t0], 0) : czero<CX>();
          z1[k] = (r < n && h1) ? mk<CX>(Y[r * ell + t1], 0) : czero<CX>();
        }
        for (int j = n - 2; j >= 0; j -= 2) {
          const CX tj = tau[j], tk = j >= 1 ? tau[j - 1] : czero<CX>();
          const bool on1 = tj.x != 0.f || tj.y != 0.f, on2 = tk.x != 0.f || tk.y != 0.f;
          if (!on1 && !on2) continue;
          const CX c = j >= 1 ? pairc[(n - 2 - j) >> 1] : czero<CX>();
          CX d10 = czero<CX>(), d11 = czero<CX>(), d20 = czero<CX>(), d21 = czero<CX>();
          CX v1[2], v2[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int r = lane + 32 * k;
            v1[k] = r < n ? a0[j * n + r] : czero<CX>();
            v2[k] = (j >= 1 && r < n) ? a0[(j - 1) * n + r] : czero<CX>();
            if (32 * k + 31 >= j && r < n) {
              cfmac(d10, v1[k], z0[k]);
              cfmac(d11, v1[k], z1[k]);
              cfmac(d20, v2[k], z0[k]);
              cfmac(d21, v2[k], z1[k]);
            }
          }
          d10 = warp_csum(d10);
          d11 = warp_csum(d11);
          d20 = warp_csum(d20);
          d21 = warp_csum(d21);
          const CX s10 = cmul(tj, d10), s11 = cmul(tj, d11);
          const CX s20 = cmul(tk, csub(d20, cmul(c, s10))), s21 = cmul(tk, csub(d21, cmul(c, s11)));
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int r = lane + 32 * k;
            if (32 * k + 31 >= j && r < n) {
              z0[k] = csub(z0[k], cadd(cmul(v1[k], s10), cmul(v2[k], s20)));
              z1[k] = csub(z1[k], cadd(cmul(v1[k], s11), cmul(v2[k], s21)));
            }
          }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int r = lane + 32 * k;
          if (r < n) {
            a1[r * ell + t0] = z0[k];
            if (h1) a1[r * ell + t1] = z1[k];
          }
        }
      }
      __syncthreads();
      // ---------------- polish: M = I - V^H V in a0, V + V M / 2 from a1 to a2 and back
      for (int step = 0; step < 4; ++step) {
        if (step >= 2 && !orth_above(omax, kOrthPolish)) break;
        CX* Vs = (step & 1) ? a2 : a1;
        CX* Vd = (step & 1) ? a1 : a2;
        small_product(
            nv, nv, n, [&](int i, int k) { return cconj(Vs[k * ell + i]); },
            [&](int k, int j) { return Vs[k * ell + j]; },
            [&](int i, int j, CX acc) {
              CX v = cmul(mk<CX>(-1, 0), acc);
              if (i == j) v.x += 1.f;
              a0[i * ell + j] = v;
            });
        __syncthreads();
        if (step == 0) {
          // orthogonality guard (orth_guard_kernel)
          const float l0 = lam[0];
          if (l0 > 0.f) {
            const float floor_ = l0 * 64.f * 5.96e-8f;
            int kl = 0;
            while (kl < nv && lam[kl] > floor_) ++kl;
            float worst = 0.f, wworst = 0.f;
            for (int i = 1 + wid; i < kl; i += NWP) {
              const float wi = lam[i] / l0;
              for (int j = lane; j < i; j += 32) {
                const CX z = a0[i * ell + j];
                const float v2 = cabs2(z);
                const bool fin = isfinite(z.x) && isfinite(z.y);
                worst = fin ? fmaxf(worst, v2) : __int_as_float(0x7f800000);
                wworst = fin ? fmaxf(wworst, v2 * wi) : __int_as_float(0x7f800000);
              }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
              wworst = fmaxf(wworst, __shfl_xor_sync(0xffffffffu, wworst, o));
            }
            if (lane == 0 && worst > 0.f) atomicMax(&omax, __float_as_uint(worst));
            if (lane == 0 && wworst > 0.f) atomicMax(&owmax, __float_as_uint(wworst));
          }
        }
        small_product(
            n, nv, nv, [&](int i, int k) { return Vs[i * ell + k]; }, [&](int k, int j) { return a0[k * ell + j]; },
            [&](int i, int j, CX acc) {
              Vd[i * ell + j] = cadd(cmul(mk<CX>(0.5f, 0), acc), cmul(mk<CX>(1, 0), Vs[i * ell + j]));
            });
        __syncthreads();
      }
      // ---------------- X V and the squared column norms
      for (int i = tid; i < m * n; i += NT) a0[i] = X[i];
      for (int i = tid; i < n * ell; i += NT)
        if (i % ell < nv) Vg[i] = a1[i];
      __syncthreads();
      small_product(
          m, nv, n, [&](int i, int k) { return a0[i * n + k]; }, [&](int k, int j) { return a1[k * ell + j]; },
          [&](int i, int j, CX acc) {
            const CX v = cmul(mk<CX>(1, 0), acc);
            AV[(int64_t)i * ell + j] = v;
            a2[i * ell + j] = v;
          });
      __syncthreads();
      const int cw = min(max(32, ((nv + 31) / 32) * 32), NT), G = NT / cw;
      const int lt = tid % cw, grp = tid / cw;
      SumAcc<float> ca;
      if (grp < G && lt < nv)
        for (int r = grp; r < m; r += G) ca.add(cabs2(a2[r * ell + lt]));
      partd[tid] = ca.value();
      __syncthreads();
      if (grp == 0 && lt < nv) {
        double acc = 0;
        for (int q = 0; q < G; ++q) acc += partd[q * cw + lt];
        s_raw[lt] = acc;
      }
    }
    __syncthreads();
    // ---------------- rank selection (rank_kernel)
    for (int t = tid; t < nv; t += NT) {
      double acc = s_raw[t];
      if (mode0 == 1) {
        const float v = lam[t] * *((const float*)hp->scale);
        acc = v > 0.f ? (double)v : 0.0;
      }
      if (!isfinite(acc)) {
        nonfinite = 1;
        acc = -1.0;
      }
      s_raw[t] = (double)(float)acc;
      s_key[t] = (float)s_raw[t];
    }
    __syncthreads();
    for (int t = tid; t < nv; t += NT) {
      int rk = t;
      if (mode0 != 1) {
        const float vk = s_key[t];
        rk = 0;
        for (int u = 0; u < nv; ++u) rk += (s_key[u] > vk) || (s_key[u] == vk && u < t);
      }
      s_sorted[rk] = s_raw[t];
      perm[rk] = t;
    }
    __syncthreads();
    for (int t = tid; t < nv; t += NT) sig2[t] = s_sorted[t];
    int k, status, needed;
    double eps_local, entropy, condS;
    rank_rule_block(s_sorted, s_sorted + ell, nv, min(m, n), cap, eps, true, total_d, k, eps_local, entropy, condS,
                    status, needed);
    if (nonfinite) {
      status = AGB_ERR_NOCONV;
      k = 0;
    }
    const int bits = repair_bits(status, nv, ell, mode0, omax, guard);
    if (attempt == 0 && repair && bits) {
      repaired = bits;
      if (bits & 2) ctol = kClusterTolWide;
      nv = ell;
      __syncthreads();
      continue;
    }
    if (tid == 0) {
      if (guard && orth_exceeds(omax) && mode0 != 1) {  // not orthonormal, no repair left
        status = AGB_ERR_NOCONV;
        k = 0;
      }
      if (hp->fail) {
        status = AGB_ERR_TIMEOUT;
        k = 0;
      }
      if (*status_word(ws, ng) != 0) {  // a bounded wait in a tensor-core GEMM expired
        status = *status_word(ws, ng);
        k = 0;
      }
      if (D[AGB_D_STATUS] != AGB_OK) {  // shapes rejected in setup
        status = (int)D[AGB_D_STATUS];
        k = 0;
      }
      hp->nvec = nv;
      D[AGB_D_REPAIR] = repaired;
      D[AGB_D_K] = k;
      D[AGB_D_EPSLOC] = bitsd(eps_local);
      D[AGB_D_ENTROPY] = bitsd(entropy);
      D[AGB_D_CONDS] = bitsd(condS);
      D[AGB_D_STATUS] = status;
      D[AGB_D_TOTAL] = bitsd(total_d);
      D[AGB_D_NEEDED] = needed;
      D[AGB_D_ORTH] = bitsd(mode0 == 1 ? 0.0 : (double)__uint_as_float(omax));
      D[AGB_D_ORTHW] = bitsd(mode0 == 1 ? 0.0 : (double)__uint_as_float(owmax));
    }
    return;
  }
}
