// Batched complex GEMM on the 5th-generation tensor cores (sm_103a):
// D = alpha * op(A) op(B) + beta * Csrc, complex64, split precision 3xTF32.
//
// One CTA (9 warps) per 128 x 64 output tile, K in slices of 32:
//  * warps 0-7 (the converters) read the complex64 slice of op(A) (128 x 32)
//    and op(B)^T (64 x 32) straight from the operands with coalesced loads
//    (along k when k is contiguous in memory, along the rows otherwise), split
//    each value into TF32 hi = x rounded to TF32 (11-bit significand) and
//    lo = x - hi, fold conjugation into the imaginary parts, and store them
//    into a shared-memory stage in the K-major 128-byte-swizzled layout the
//    tensor core reads (the layout a TMA SWIZZLE_128B copy of 32-float rows
//    produces): A as four planes {Re_hi, Re_lo, Im_hi, Im_lo}, B as two
//    planes {hi, lo} of 192 rows [-Im | Re | Im]; out-of-range rows and k are
//    stored as zeros;
//  * warp 8 lane 0 issues tcgen05.mma.kind::tf32 (M=128, N=128, K=8) per stage,
//    the real and imaginary accumulators of the tile being adjacent TMEM
//    columns written by one MMA: with B rows 64..191 = [Re | Im] and rows
//    0..127 = [-Im | Re],
//       [Re | Im] += Ar_h [Br|Bi]_h + Ar_h [Br|Bi]_l + Ar_l [Br|Bi]_h
//                  + Ai_h [-Bi|Br]_h + Ai_h [-Bi|Br]_l + Ai_l [-Bi|Br]_h
//    (six MMAs per K=8 step, each accumulator receiving the same products in
//    the same order as twelve N=64 MMAs would), k slices rotating over four
//    accumulator pairs; a commit per stage frees the stage for the converters;
//  * warps 0-7 then read the accumulators with tcgen05.ld (warp w reads TMEM
//    lanes 32(w%4)..+31 = tile rows, columns 32(w/4)..+31), turn their blocks
//    in shared memory and write alpha*C + beta*Csrc in whole row pieces.
// What bounds it: shared-memory bandwidth.  A slice moves 112 KiB of converter
// stores, 192 KiB of operand reads by its 24 MMAs and 96 KiB of global loads
// through the SM's 128 B/clk: 3100 cycles, as measured (24 MMAs alone: 1900).
// 16384 x 512 x 256 (one site of 16 384 shots at chi 256): 118 us a launch, 152
// before the epilogue's turn, the once-formed addresses and the one-slice read-ahead.
// The operands are read once per tile and never written back in split form:
// no packing pass and no packed copy in global memory.  The converters'
// shared-memory stores reach the tensor core through fence.proxy.async and the
// stage's full barrier.  Every mbarrier wait is bounded; on expiry the kernel
// records AGB_ERR_TIMEOUT in a device status word, waits (bounded) for the
// issued MMAs and frees its tensor memory.
#include "gemm.cuh"
#include "gemm_tc.cuh"

namespace {

constexpr int BM = 128, BN = 64, BK = 32, STAGES = 2;
constexpr int TILE_A = BM * BK * 4;                    // 16 KiB per plane
constexpr int B_ROWS = 3 * BN;                         // B plane rows: -Im | Re | Im
constexpr int TILE_B = B_ROWS * BK * 4;                // 24 KiB per plane (hi, lo)
constexpr int STAGE_BYTES = 4 * TILE_A + 2 * TILE_B;   // 112 KiB
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int NACC = 4;                                // k-tiles rotate over 4 accumulator pairs
constexpr int TMEM_COLS = 2 * BN * NACC;               // 512 columns: (Re, Im) x 4
constexpr int CONV_WARPS = 8;
constexpr int NCONV = 32 * CONV_WARPS;                 // converter / epilogue threads (warps 0-7)
constexpr int NTHREADS = NCONV + 32;                   // + warp 8: tensor memory and MMA issue
constexpr int MMA_WARP = CONV_WARPS;
constexpr int QA = BM * BK / 4 / NCONV, QB = BN * BK / 4 / NCONV;  // quads (4 consecutive k) per thread per k slice
constexpr unsigned WAIT_LIMIT = 1u << 26;              // bounded spin (~seconds)

AGB_DEV uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

AGB_DEV void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
AGB_DEV void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// true when phase `parity` of the barrier completed; false after `limit` polls
AGB_DEV bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned limit = WAIT_LIMIT) {
  const uint32_t a = smem_u32(bar);
  for (unsigned it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row atoms of
// 1024 B (stride byte offset), descriptor version 1.
AGB_DEV uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset
  d |= (uint64_t)1 << 46;             // version
  d |= (uint64_t)2 << 61;             // SWIZZLE_128B
  return d;
}
// Instruction descriptor, kind::tf32: D f32, A/B tf32, K-major, M=128, N=128
// (the real and imaginary accumulators of a tile are adjacent TMEM columns,
// written by one MMA).
constexpr uint32_t IDESC =
    (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)((2 * BN) >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);

AGB_DEV void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
AGB_DEV void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// 16 columns of the warp's 32 lanes; valid after the next wait::ld.
AGB_DEV void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
        "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}

// x rounded to TF32 (10 explicit mantissa bits), round to nearest even.
AGB_DEV float tf32_hi(float x) {
  uint32_t b;
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(b) : "f"(x));
  return __uint_as_float(b & 0xFFFFE000u);
}

// Byte offset of element (row r, k) in a plane tile of 128-byte rows (32 fp32)
// with the 128-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ (r % 8)
// (the tile starts on a 1024-byte boundary).
AGB_DEV uint32_t sw128(int r, int k) { return (uint32_t)(r * 128 + (((k >> 2) ^ (r & 7)) << 4) + ((k & 3) << 2)); }

AGB_DEV void st_shared_v4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// A converter thread handles quads: 4 consecutive k of one row, which are
// one 16-byte chunk of the swizzled tile (one vector store per plane).  The
// j-th quad of thread ct:
//  * k contiguous in memory: a warp takes 4 rows x 32 k (lanes: row
//    lane / 8, quad lane % 8), rows 4 (w + 8 j) ..; each row is one 256-byte
//    read;
//  * otherwise: a warp takes 32 consecutive rows x one quad (lanes: row),
//    blocks b = w + 8 j with quad b % 8 and 32-row chunk b / 8; each k of the
//    quad is one 256-byte read.
// Either way each 8-lane phase of a vector store covers the 8 chunk positions
// of the 128-byte swizzle (chunk (k/4) ^ (row % 8)): no bank conflicts.
AGB_DEV void quad_coord(bool k_contig, int ct, int j, int& r, int& k4) {
  const int lane = ct & 31, w = ct >> 5;
  if (k_contig) {
    r = 4 * (w + CONV_WARPS * j) + (lane >> 3);
    k4 = 4 * (lane & 7);
  } else {
    const int b = w + CONV_WARPS * j;
    k4 = 4 * (b & 7);
    r = 32 * (b >> 3) + lane;
  }
}

// Element (row, k) of the operand as the MMA sees it:
//   A (which 0): op(A)[row][k];  B (which 1): op(B)[k][row]
// stored form: A op N/R -> A[row][k]; op T/C -> A[k][row]
//              B op N/R -> B[k][row]; op T/C -> B[row][k]
// A converter thread reads NQ quads of every k slice.  Their addresses are
// formed once and advance by a constant per slice: with the address
// arithmetic and the bounds checks of each element inside the loop, a slice cost
// ~40 instructions per element and the tensor pipe was 31% active.
template <int NQ>
struct Operand {
  const float2* q[NQ];  // quad j of the next slice
  int64_t kstride, step;  // elements between consecutive k, and between slices
  int K;
  bool row_ok[NQ], k_contig, vec, conj;
};
template <int NQ>
AGB_DEV Operand<NQ> operand(const GemmProb& P, int which, int r0, int ct) {
  Operand<NQ> o;
  const int op = which == 0 ? P.opA : P.opB;
  const float2* p = (const float2*)(which == 0 ? P.A : P.B);
  const int64_t ld = which == 0 ? P.lda : P.ldb;
  const int rows = which == 0 ? P.M : P.N;
  const bool transposed = (op == 1 || op == 2);
  o.K = P.K;
  o.k_contig = (which == 0) ? !transposed : transposed;
  o.conj = (op == 2 || op == 3);
  o.kstride = o.k_contig ? 1 : ld;
  o.step = BK * o.kstride;
  // a quad of consecutive k is two 16-byte loads where every row starts on 16 bytes
  o.vec = o.k_contig && ((uintptr_t)p & 15) == 0 && (ld & 1) == 0;
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    int r, k4;
    quad_coord(o.k_contig, ct, j, r, k4);
    o.row_ok[j] = r0 + r < rows;
    const int rr = o.row_ok[j] ? r0 + r : 0;
    o.q[j] = o.k_contig ? p + (int64_t)rr * ld + k4 : p + (int64_t)k4 * ld + rr;
  }
  return o;
}
template <int NQ>
AGB_DEV void load_slice(Operand<NQ>& o, int k0, int ct, float2* v) {
  const float2 zero = make_float2(0.f, 0.f);
  const bool full = k0 + BK <= o.K;
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    float2* d = v + 4 * j;
    const float2* q = o.q[j];
#pragma unroll
    for (int t = 0; t < 4; ++t) d[t] = zero;
    if (o.row_ok[j]) {
      if (full) {
        if (o.vec) {
          const float4 a = *(const float4*)q, b = *(const float4*)(q + 2);
          d[0] = make_float2(a.x, a.y);
          d[1] = make_float2(a.z, a.w);
          d[2] = make_float2(b.x, b.y);
          d[3] = make_float2(b.z, b.w);
        } else {
#pragma unroll
          for (int t = 0; t < 4; ++t) d[t] = q[t * o.kstride];
        }
      } else {
        int r, k4;
        quad_coord(o.k_contig, ct, j, r, k4);
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (k0 + k4 + t < o.K) d[t] = q[t * o.kstride];
      }
    }
    o.q[j] = q + o.step;
  }
}
// B quads: the hi and lo planes hold rows [-Im | Re | Im] (BN rows each), so
// rows BN..3BN-1 are the operand [Re | Im] of an A_re product and rows
// 0..2BN-1 the operand [-Im | Re] of an A_im product: one N = 2 BN MMA then
// accumulates both the real and the imaginary part of the tile.
template <int NQ>
AGB_DEV void store_slice_b(const Operand<NQ>& o, uint32_t tile, int ct, const float2* v) {
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    int r, k4;
    quad_coord(o.k_contig, ct, j, r, k4);
    float rh[4], rl[4], ih[4], il[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float re = v[4 * j + t].x, im = o.conj ? -v[4 * j + t].y : v[4 * j + t].y;
      rh[t] = tf32_hi(re);
      ih[t] = tf32_hi(im);
      rl[t] = re - rh[t];
      il[t] = im - ih[t];
    }
    const uint32_t a = tile + sw128(r, k4);  // rows r, r + BN, r + 2 BN share the swizzle phase
    constexpr uint32_t RB = BN * 128;
    st_shared_v4(a, -ih[0], -ih[1], -ih[2], -ih[3]);
    st_shared_v4(a + RB, rh[0], rh[1], rh[2], rh[3]);
    st_shared_v4(a + 2 * RB, ih[0], ih[1], ih[2], ih[3]);
    st_shared_v4(a + TILE_B, -il[0], -il[1], -il[2], -il[3]);
    st_shared_v4(a + TILE_B + RB, rl[0], rl[1], rl[2], rl[3]);
    st_shared_v4(a + TILE_B + 2 * RB, il[0], il[1], il[2], il[3]);
  }
}
template <int NQ>
AGB_DEV void store_slice(const Operand<NQ>& o, uint32_t tile, int plane_bytes, int ct, const float2* v) {
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    int r, k4;
    quad_coord(o.k_contig, ct, j, r, k4);
    float rh[4], rl[4], ih[4], il[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float re = v[4 * j + t].x, im = o.conj ? -v[4 * j + t].y : v[4 * j + t].y;
      rh[t] = tf32_hi(re);
      ih[t] = tf32_hi(im);
      rl[t] = re - rh[t];
      il[t] = im - ih[t];
    }
    const uint32_t a = tile + sw128(r, k4);
    st_shared_v4(a, rh[0], rh[1], rh[2], rh[3]);
    st_shared_v4(a + plane_bytes, rl[0], rl[1], rl[2], rl[3]);
    st_shared_v4(a + 2 * plane_bytes, ih[0], ih[1], ih[2], ih[3]);
    st_shared_v4(a + 3 * plane_bytes, il[0], il[1], il[2], il[3]);
  }
}

// ------------------------------------------------------------------ GEMM
// Problems from device memory, or (probs null) a strided batch passed by value.
struct StridedProbs {
  GemmProb base;
  int64_t sA, sB, sC;  // element strides between batch entries
};
AGB_DEV GemmProb get_prob(const GemmProb* probs, const StridedProbs& sp) {
  if (probs) return probs[blockIdx.z];
  GemmProb p = sp.base;
  const int64_t z = blockIdx.z;
  p.A = (const float2*)p.A + z * sp.sA;
  p.B = (const float2*)p.B + z * sp.sB;
  p.D = (float2*)p.D + z * sp.sC;
  p.Csrc = (const float2*)p.Csrc + z * sp.sC;
  return p;
}

__global__ void __launch_bounds__(NTHREADS, 1)
    tc_gemm_kernel(const GemmProb* __restrict__ probs, const __grid_constant__ StridedProbs sp,
                   int* __restrict__ status, unsigned pipe_limit) {
  const GemmProb P = get_prob(probs, sp);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (m0 >= P.M || n0 >= P.N) return;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = (P.K + BK - 1) / BK;
  // the first slice's loads are in flight while the barriers and TMEM are set up
  const int ct = threadIdx.x;
  Operand<QA> oa;
  Operand<QB> ob;
  float2 va[2][4 * QA], vb[2][4 * QB];
  if (warp < CONV_WARPS) {
    oa = operand<QA>(P, 0, m0, ct);
    ob = operand<QB>(P, 1, n0, ct);
    if (nk > 0) {
      load_slice<QA>(oa, 0, ct, va[0]);
      load_slice<QB>(ob, 0, ct, vb[0]);
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], CONV_WARPS);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  if (warp < CONV_WARPS) {
    // ---------------- converters: global complex64 -> split TF32 planes in shared memory
    // slice kt + 1 is read from global memory while slice kt is converted
    bool stopped = false;
    for (int kt0 = 0; kt0 < nk && !stopped; kt0 += 2) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int kt = kt0 + u, s = u;  // STAGES == 2: slice kt uses stage kt % 2
        if (kt >= nk || stopped) break;
        if (kt + 1 < nk) {
          load_slice<QA>(oa, (kt + 1) * BK, ct, va[u ^ 1]);
          load_slice<QB>(ob, (kt + 1) * BK, ct, vb[u ^ 1]);
        }
        // one decision per warp: its lanes meet again at the __syncwarp below
        bool go = kt < STAGES || mbar_wait(&empty[s], ((kt / STAGES) - 1) & 1, pipe_limit);
        if (!go) *abort_flag = 1;
        go = go && !*abort_flag;
        if (!__all_sync(0xffffffffu, go)) {
          stopped = true;
          break;
        }
        const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
        store_slice<QA>(oa, st, TILE_A, ct, va[u]);
        store_slice_b<QB>(ob, st + 4 * TILE_A, ct, vb[u]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the tensor core
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
      }
    }
  } else if (lane == 0) {
    // ---------------- MMA issuer
    // k-tile kt accumulates into pair kt % NACC: four chains of length K/4 instead
    // of one of length K (the tensor core's fp32 accumulation error grows with
    // the chain length); the epilogue sums the pairs in fp32.
    // Shared-memory descriptors: the address field is (address / 16) in the low
    // 14 bits, so a descriptor at a 16-byte multiple `off` past a stage base is
    // the base's descriptor + off / 16 (every operand lies below 256 KiB); the
    // two stage bases are formed once.
    static_assert(STAGES == 2, "two stage descriptors");
    const uint64_t dstage0 = sdesc(smem_u32(smem)), dstage1 = sdesc(smem_u32(smem + STAGE_BYTES));
    constexpr uint64_t A_PL = TILE_A >> 4, B0 = (4 * TILE_A) >> 4, B_LO = TILE_B >> 4, B_RE = (BN * 128) >> 4;
    for (int kt = 0; kt < nk; ++kt) {
      const int s = kt % STAGES;
      const uint32_t d = tmem + (uint32_t)(2 * BN * (kt % NACC));  // [re | im] columns of pair kt % NACC
      if (!mbar_wait(&full[s], (kt / STAGES) & 1, pipe_limit)) {
        *abort_flag = 1;
        break;
      }
      if (*abort_flag) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t ds = s ? dstage1 : dstage0;
#pragma unroll
      for (int ks = 0; ks < BK / 8; ++ks) {
        const uint64_t dk = ds + (uint64_t)(ks * 2);  // +32 bytes per K=8 step
        // A planes Re_hi, Re_lo, Im_hi, Im_lo; the [Re | Im] and [-Im | Re]
        // windows of the hi and lo B planes
        const uint64_t a0 = dk, a1 = dk + A_PL, a2 = dk + 2 * A_PL, a3 = dk + 3 * A_PL;
        const uint64_t bre_hi = dk + B0 + B_RE, bre_lo = dk + B0 + B_LO + B_RE;
        const uint64_t bim_hi = dk + B0, bim_lo = dk + B0 + B_LO;
        const uint32_t first = (kt < NACC && ks == 0) ? 0u : 1u;
        // re += Are Bre - Aim Bim,  im += Are Bim + Aim Bre  (3xTF32: hi hi, hi lo, lo hi)
        umma(d, a0, bre_hi, IDESC, first);
        umma(d, a0, bre_lo, IDESC, 1);
        umma(d, a1, bre_hi, IDESC, 1);
        umma(d, a2, bim_hi, IDESC, 1);
        umma(d, a2, bim_lo, IDESC, 1);
        umma(d, a3, bim_hi, IDESC, 1);
      }
      umma_commit(&empty[s]);  // stage s may be refilled once these MMAs retire
    }
    umma_commit(done);  // every MMA issued above has completed when this arrives
  }
  __syncwarp();
  // ---------------- epilogue (warps 0-7); the MMA warp waits for the MMAs before freeing TMEM.
  // This wait keeps the full limit even when the pipeline's is lowered, so an
  // aborted tile still retires every MMA it issued before TMEM is freed.
  const bool ok = mbar_wait(done, 0);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp < CONV_WARPS && ok && !*abort_flag) {
    // Warp (quarter, half) reads TMEM lanes 32 quarter.. and columns 32 half..,
    // one tile row per lane, and turns its 32 x 32 block in shared memory (the
    // stages are free), so that the global accesses are whole 256-byte row pieces.
    // Stored straight from the TMEM layout, a store touched 32 rows with 8 bytes
    // each: 13 800 of a 16 384 x 512 x 256 tile's 44 800 cycles, and the loads of
    // the other CTAs waited behind it.
    const int quarter = warp & 3, half = warp >> 2;
    const int row0 = m0 + quarter * 32, col = n0 + half * (BN / 2) + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    float2* D = (float2*)P.D;
    const float2* C = (const float2*)P.Csrc;
    const float ar = (float)P.alpha_re, ai = (float)P.alpha_im, br = (float)P.beta_re, bi = (float)P.beta_im;
    const float eye = (float)P.eye;
    const bool use_beta = (br != 0.f || bi != 0.f);
    const int nacc = nk < NACC ? nk : NACC;
    constexpr int PITCH = BN / 2 + 1;
    float2* buf = (float2*)smem + warp * 32 * PITCH;
#pragma unroll 1
    for (int c0 = 0; c0 < BN / 2; c0 += 16) {
      const uint32_t tc = tmem + lane_base + (uint32_t)(half * (BN / 2) + c0);
      float re[NACC][16], im[NACC][16];
#pragma unroll
      for (int a = 0; a < NACC; ++a)
        if (a < nacc) {
          tmem_ld16(tc + (uint32_t)(2 * BN * a), re[a]);
          tmem_ld16(tc + (uint32_t)(2 * BN * a) + BN, im[a]);
        }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // the values count as written here: no use of them moves ahead of the wait
#pragma unroll
      for (int a = 0; a < NACC; ++a)
#pragma unroll
        for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(re[a][i]), "+f"(im[a][i]));
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float x = 0.f, y = 0.f;  // empty inner dimension: product is zero
#pragma unroll
        for (int a = 0; a < NACC; ++a)
          if (a < nacc) {
            x = a ? x + re[a][i] : re[a][i];
            y = a ? y + im[a][i] : im[a][i];
          }
        buf[lane * PITCH + c0 + i] = make_float2(ar * x - ai * y, ar * y + ai * x);
      }
    }
    __syncwarp();
    const int nrow = min(32, P.M - row0);
    if (col < P.N) {
      float2* d = D + (int64_t)row0 * P.ldd + col;
      const float2* c = C + (int64_t)row0 * P.ldc + col;
      const float2* b = buf + lane;
      if (use_beta || eye != 0.f) {
#pragma unroll 4
        for (int r = 0; r < nrow; ++r, d += P.ldd, c += P.ldc, b += PITCH) {
          float2 v = *b;
          if (use_beta) {
            const float2 z = *c;
            v.x += br * z.x - bi * z.y;
            v.y += br * z.y + bi * z.x;
          }
          if (row0 + r == col) v.x += eye;
          *d = v;
        }
      } else {
#pragma unroll 8
        for (int r = 0; r < nrow; ++r, d += P.ldd, b += PITCH) *d = *b;
      }
    }
  } else if (threadIdx.x == 0 && (!ok || *abort_flag)) {
    atomicExch(status, AGB_ERR_TIMEOUT);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

int round_up(int x, int m) { return (x + m - 1) / m * m; }

unsigned g_pipe_limit = WAIT_LIMIT;

}  // namespace

// Poll limit of the GEMM's pipeline waits (stage full / empty); a negative value
// restores the default.  Lets a test make those waits expire: the kernel then
// reports AGB_ERR_TIMEOUT and skips its epilogue.
extern "C" int agb_set_gemm_wait_limit(long long polls) {
  g_pipe_limit = polls < 0 ? WAIT_LIMIT : (unsigned)(polls < (long long)WAIT_LIMIT ? polls : (long long)WAIT_LIMIT);
  return AGB_OK;
}

// The split operands live only in shared memory: the tensor-core path needs
// no global scratch beyond a token the dispatcher checks for.
size_t tc_gemm_scratch_bytes(int count, int maxM, int maxN, int maxK) {
  (void)count;
  (void)maxM;
  (void)maxN;
  (void)maxK;
  return 256;
}

static int launch_tc(const GemmProb* probs, const StridedProbs& sp, int count, int maxM, int maxN, int maxK,
                     void* scratch, size_t scratch_bytes, int* status, cudaStream_t s) {
  if (count <= 0 || maxM <= 0 || maxN <= 0) return AGB_OK;
  if (maxK <= 0) return AGB_ERR_ARG;
  if (count > 65535) return AGB_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < tc_gemm_scratch_bytes(count, maxM, maxN, maxK)) return AGB_ERR_WORKSPACE;
  const int Mp = round_up(maxM, BM), Np = round_up(maxN, BN);
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(tc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
      return AGB_ERR_CUDA;
    attr = true;
  }
  tc_gemm_kernel<<<dim3(Np / BN, Mp / BM, count), NTHREADS, SMEM_BYTES, s>>>(probs, sp, status, g_pipe_limit);
  AGB_CHECK_LAUNCH();
  return AGB_OK;
}

int launch_gemm_tc(const GemmProb* probs, int count, int maxM, int maxN, int maxK, void* scratch,
                   size_t scratch_bytes, int* status, cudaStream_t s) {
  if (!probs) return AGB_ERR_ARG;
  const StridedProbs none = {};
  return launch_tc(probs, none, count, maxM, maxN, maxK, scratch, scratch_bytes, status, s);
}

// Products listed in device memory, any shapes, one launch.
extern "C" size_t agb_gemm_prob_bytes(void) { return sizeof(GemmProb); }

extern "C" int agb_gemm_list(int dtype, int tensor_cores, const void* probs, int count, int maxM, int maxN, int maxK,
                             int* status_dev, void* stream) {
  if (dtype != AGB_C64 && dtype != AGB_C128) return AGB_ERR_ARG;
  if (count < 0 || maxM < 0 || maxN < 0 || maxK < 0 || count > 65535) return AGB_ERR_ARG;
  if (count == 0 || maxM == 0 || maxN == 0) return AGB_OK;
  if (!probs) return AGB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const GemmProb* p = (const GemmProb*)probs;
  if (tensor_cores) {
    if (dtype != AGB_C64 || !status_dev) return AGB_ERR_ARG;
    // the split operands live in shared memory: the scratch is a token
    return launch_gemm_tc(p, count, maxM, maxN, maxK, status_dev, tc_gemm_scratch_bytes(count, maxM, maxN, maxK),
                          status_dev, s);
  }
  return dtype == AGB_C64 ? launch_gemm_probs<float2>(p, count, maxM, maxN, s, nullptr, maxK)
                          : launch_gemm_probs<double2>(p, count, maxM, maxN, s, nullptr, maxK);
}

// Strided-batch host entry for the tensor-core GEMM (complex64).
namespace {
int opc(char c) {
  return (c == 'N' || c == 'n') ? 0 : (c == 'T' || c == 't') ? 1 : (c == 'C' || c == 'c') ? 2 : (c == 'R' || c == 'r') ? 3 : -1;
}
}  // namespace

extern "C" size_t agb_cgemm_tc_workspace(int batch, int M, int N, int K) {
  return agb_align((size_t)batch * sizeof(GemmProb)) + agb_align(sizeof(int)) + tc_gemm_scratch_bytes(batch, M, N, K);
}

// status_dev == NULL: the status word lives in the workspace, is cleared first,
// and (if status_host) is read back after a stream synchronisation.
// status_dev != NULL: the kernels record a timeout in *status_dev, which is
// never cleared here (sticky across calls), and nothing synchronises.
static int cgemm_tc_impl(char opA, char opB, int batch, int M, int N, int K, const void* A, int64_t lda,
                         int64_t strideA, const void* B, int64_t ldb, int64_t strideB, void* C, int64_t ldc,
                         int64_t strideC, float alpha_re, float alpha_im, float beta_re, float beta_im, void* ws,
                         size_t ws_bytes, int* status_host, int* status_dev, void* stream) {
  const int oa = opc(opA), ob = opc(opB);
  if (oa < 0 || ob < 0 || batch < 0 || M < 0 || N < 0 || K <= 0 || !ws) return AGB_ERR_ARG;
  if (batch == 0 || M == 0 || N == 0) return AGB_OK;
  if (ws_bytes < agb_cgemm_tc_workspace(batch, M, N, K)) return AGB_ERR_WORKSPACE;
  StridedProbs sp;
  GemmProb& base = sp.base;
  base.A = A;
  base.B = B;
  base.D = C;
  base.Csrc = C;
  base.lda = lda;
  base.ldb = ldb;
  base.ldd = ldc;
  base.ldc = ldc;
  base.M = M;
  base.N = N;
  base.K = K;
  base.opA = oa;
  base.opB = ob;
  base.alpha_re = alpha_re;
  base.alpha_im = alpha_im;
  base.beta_re = beta_re;
  base.beta_im = beta_im;
  base.eye = 0;
  char* w = (char*)ws;
  sp.sA = strideA;
  sp.sB = strideB;
  sp.sC = strideC;
  int* status = (int*)(w + agb_align((size_t)batch * sizeof(GemmProb)));
  void* scratch = w + agb_align((size_t)batch * sizeof(GemmProb)) + agb_align(sizeof(int));
  cudaStream_t s = (cudaStream_t)stream;
  if (status_dev) status = status_dev;
  else if (cudaMemsetAsync(status, 0, sizeof(int), s) != cudaSuccess) return AGB_ERR_CUDA;
  int rc = launch_tc(nullptr, sp, batch, M, N, K, scratch, ws_bytes - (size_t)((char*)scratch - w), status, s);
  if (rc) return rc;
  if (status_host && !status_dev) {
    if (cudaMemcpyAsync(status_host, status, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return AGB_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return AGB_ERR_CUDA;
    if (*status_host) return *status_host;
  }
  return AGB_OK;
}

extern "C" int agb_cgemm_tc(char opA, char opB, int batch, int M, int N, int K, const void* A, int64_t lda,
                            int64_t strideA, const void* B, int64_t ldb, int64_t strideB, void* C, int64_t ldc,
                            int64_t strideC, float alpha_re, float alpha_im, float beta_re, float beta_im, void* ws,
                            size_t ws_bytes, int* status_host, void* stream) {
  return cgemm_tc_impl(opA, opB, batch, M, N, K, A, lda, strideA, B, ldb, strideB, C, ldc, strideC, alpha_re,
                       alpha_im, beta_re, beta_im, ws, ws_bytes, status_host, nullptr, stream);
}

extern "C" int agb_cgemm_tc_async(char opA, char opB, int batch, int M, int N, int K, const void* A, int64_t lda,
                                  int64_t strideA, const void* B, int64_t ldb, int64_t strideB, void* C,
                                  int64_t ldc, int64_t strideC, float alpha_re, float alpha_im, float beta_re,
                                  float beta_im, void* ws, size_t ws_bytes, int* status_dev, void* stream) {
  if (!status_dev) return AGB_ERR_ARG;
  return cgemm_tc_impl(opA, opB, batch, M, N, K, A, lda, strideA, B, ldb, strideB, C, ldc, strideC, alpha_re,
                       alpha_im, beta_re, beta_im, ws, ws_bytes, nullptr, status_dev, stream);
}
