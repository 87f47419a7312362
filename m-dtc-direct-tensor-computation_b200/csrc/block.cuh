// block.cuh -- block CG of the multigrid-preconditioned FP32 inner solve: the 24 load cases of a
// domain share one Krylov space.
//
// Not a step of the reference, which runs one KSPCG per load case (f-src/mod_dtc_main_subroutines.f90:
// 1072-1078): like the V-cycle it only changes how fast the inner solve of the iterative refinement
// reaches its tolerance, never the FP64 outer residual or the tensor it converges to.
//
// Per domain the block P of 24 directions is made K-conjugate as a whole (O'Leary's block CG).  The
// residual block is kept as R sigma, R a basis and sigma a 24 x 24 matrix: while the columns lose
// independence (weakly connected bone gives every load case the same slow modes), R is made
// orthonormal in the preconditioner's inner product again and sigma takes the factor, which is
// Dubrulle's remedy against the breakdown of the plain recurrence.  With V the V-cycle,
//   S = V R,  C = R^T S
//   beta = C_old^-1 C                      (if C is ill conditioned: R <- R tau, S <- S tau,
//   P <- S + P beta                         beta <- beta tau, sigma <- tau^T C sigma, C <- I)
//   W = K P,  G = P^T W,  alpha = G^-1 C   (after R <- R tau: alpha = G^-1 P^T R, see k_blk_gram)
//   x <- x + P alpha sigma,  R <- R - W alpha
// The natural norm sqrt(r^T V r) of load case j is sqrt(sigma_j^T C sigma_j), the stopping measure.
//
// On 384 trabecular domains of 32^3 (bone fraction 0.1 to 0.4, rtol 1e-7) the load cases need 79
// iterations (median; 340 at most) one by one and 40 (81) as a block: 1451 -> 745 ms.  The domains with the
// weakest connections, which set the length of a batch, gain most: 32 domains of 15^3 to 56^3 807 -> 333 ms.
#pragma once

namespace dtc {

// Up to kChunkMax nodes of one domain, first .. first + count of the list of active interior nodes.
struct Chunk {
  int32_t dom, count;
  int64_t first;
};
constexpr int kChunkMax = 256;    // nodes of a chunk at most
constexpr int kBlkTile = 32;      // nodes staged at a time by the 24 x 24 updates
constexpr int kBlkM = kNLC * kNLC;
constexpr int kGramPart = 6 * 64; // upper triangle of 8 x 8 tiles of a 24 x 24 Gram matrix

// A basis is made orthonormal again when a pivot of its scaled Gram matrix falls below this; 1e2 needs
// 1 to 5 of these per solve, 1e4 lets rounding errors cost iterations.
constexpr double kBlkRenorm = 1e-2;
// Scaled pivots below these count as dependent columns.  C: the rounding of an FP32 V-cycle leaves pivots of
// dependent columns at up to +-3.5e-6 instead of 0, and a column of noise spoils those eliminated after it; the columns
// left out stay in the residual, for the next refinement step.  G: below the rounding noise of FP32 directions.
// H, the measured p.r of columns just made orthonormal, is the identity up to noise: what is not near 1 is noise.
// Over 4608 domains of 15^3 to 56^3, bone fraction 0.05 to 0.45: at 1e-10 for C and 1e-7 for H two small bones in
// a corner of their domain, whose load cases span 18 dimensions, took 3313 and 4625 iterations (now 27 and 24);
// 1e-10 and 0.1 27.8 on average and 126 at most, 1e-6 and 0.1 27.2 and 126, 1e-5 27.3 with more refinement steps.
constexpr double kBlkDropC = 1e-6, kBlkDropG = 1e-7, kBlkDropH = 0.1;
// A column made orthonormal whose measured p.r is below this (it should be 1) is rounding noise.
constexpr double kBlkNoise = 0.25;

// Recurrence state of one domain (FP64, small) and the coefficients of the current step (FP32).
struct BlkState {
  double C[kBlkM], Cinv[kBlkM], sig[kBlkM];   // row-major
  double n0[kNLC];
  double first, best;       // ratio of a residual norm to its target (largest over the columns): initial, smallest so far
  int32_t its, reason, active, renorm, best_it, pad;
};
struct BlkCoef {
  float alpha[kBlkM], gamma[kBlkM], beta[kBlkM], tau[kBlkM];   // row-major: out_j = sum_i in_i M[i][j]
};

// When an inner solve gives up and leaves the rest to the FP64 refinement.  Voxels that share an edge or a corner only
// are hinges: K has null vectors, no direction reduces what FP32 rounding puts along them, and once the rest of a
// residual has shrunk to it these directions are all that the basis holds.  Their curvature is rounding, their steps
// blow up (without the two rules below sparse random domains of 5^3 to 17^3 ended at residuals of 1e22 to 1e38).
//  * A residual that has come down to kBlkFar of the first one and rises to kBlkRise times its smallest (4: 6658
//    iterations on 300 such domains, 10: 6906, none of it: 13886 and one domain lost).
//  * A scaled pivot of G below -kBlkNegative: curvature that a positive semidefinite operator does not have.
//  * No new smallest residual for kBlkPatience iterations, and for as many as had been taken by then: where moduli span
//    8 decades the natural norm stays level for hundreds while the error falls (of 300 such domains 268 converge load
//    case by load case, 291 with 48, 297 with 512, 296 with 1024 or no such rule).
constexpr int kBlkPatience = 512;
constexpr double kBlkFar = 1e-3, kBlkRise = 4.0, kBlkNegative = 1e-3;

enum { kBlkInit = 0, kBlkCurv = 1, kBlkRes = 2 };

// 24 x 24 products in shared memory, 256 threads: c = op(a) b
template <bool TRANS>
__device__ __forceinline__ void blk_mul(const double* a, const double* b, double* c) {
  for (int e = threadIdx.x; e < kBlkM; e += 256) {
    const int i = e / kNLC, j = e % kNLC;
    double s = 0.0;
#pragma unroll 8
    for (int k = 0; k < kNLC; ++k) s = fma(TRANS ? a[k * kNLC + i] : a[i * kNLC + k], b[k * kNLC + j], s);
    c[e] = s;
  }
  __syncthreads();
}

// Elimination of the scaled symmetric matrix: on return t holds T with T^T A T = 1 on the columns kept
// (upper triangular, a column left out is zero).  u (scratch) is overwritten.  minp: smallest scaled
// pivot of a column with a positive diagonal entry; kept: columns kept.
__device__ __forceinline__ void blk_factor(const double* a, double* u, double* li, double* t, double eps,
                                           double& minp, int& kept) {
  __shared__ double sc[kNLC], rs[kNLC];
  if (threadIdx.x < kNLC) {
    const double d = a[threadIdx.x * (kNLC + 1)];
    sc[threadIdx.x] = d > 0.0 ? rsqrt(d) : 0.0;
  }
  __syncthreads();
  kept = 0;
  for (int e = threadIdx.x; e < kBlkM; e += 256) {
    const int i = e / kNLC, j = e % kNLC;
    u[e] = a[e] * sc[i] * sc[j];
    li[e] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  minp = 1.0;
  for (int k = 0; k < kNLC; ++k) {
    const double v = u[k * (kNLC + 1)];
    if (sc[k] > 0.0) minp = fmin(minp, v);
    const bool keep = sc[k] > 0.0 && v > eps;
    kept += keep;
    if (threadIdx.x == 0) rs[k] = keep ? rsqrt(v) : 0.0;
    if (keep) {
      const double rv = 1.0 / v;
      for (int e = threadIdx.x; e < (kNLC - 1 - k) * kNLC; e += 256) {
        const int i = k + 1 + e / kNLC, j = e % kNLC;
        const double f = u[i * kNLC + k] * rv;
        if (j > k) u[i * kNLC + j] = fma(-f, u[k * kNLC + j], u[i * kNLC + j]);
        else li[i * kNLC + j] = fma(-f, li[k * kNLC + j], li[i * kNLC + j]);
      }
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < kBlkM; e += 256) {
    const int i = e / kNLC, k = e % kNLC;
    t[e] = i <= k ? sc[i] * li[k * kNLC + i] * rs[k] : 0.0;
  }
  __syncthreads();
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Gram matrix a^T b of every listed domain (FP64 accumulation on the tensor cores: the FP32 entries are
// converted exactly, a warp takes 4 rows = (node, component) per step, whose 8-load-case pieces are whole
// 32-byte sectors), and, in the CTA that finishes a domain, the 24 x 24 algebra of the step:
//   kBlkCurv: G = P^T W -> alpha, gamma = alpha sigma
//   kBlkInit / kBlkRes: C = R^T S -> norms and convergence, beta, tau
// Both matrices are symmetric in exact arithmetic; the upper triangle of 8 x 8 tiles is computed.  In the
// step after R <- R tau, kBlkCurv also computes H = P^T R tau and takes it in place of C = 1: tau magnifies
// the rounding of nearly dependent columns, some of which are then nothing else.  With H the step is the
// projection on the directions as they are, and columns whose diagonal entry or pivot shows them to be noise are
// left out of it.
// Bound by the FP64 tensor pipe and by reading the two blocks: 201 us on 384 domains of 32^3 (3.2 TB/s
// while all are active).  8 warps and pieces of 256 nodes keep the atomic traffic below a tenth of
// the reads; smaller pieces are cut when the batch would not fill the card.
template <int STEP>
__global__ void __launch_bounds__(256) k_blk_gram(const Chunk* __restrict__ chunks, const int64_t* __restrict__ list,
                                                  const float* __restrict__ a, const float* __restrict__ b,
                                                  const float* __restrict__ r, double* __restrict__ gram,
                                                  double* __restrict__ gram_h, int* __restrict__ done,
                                                  const int* __restrict__ nchunk, BlkState* __restrict__ state,
                                                  BlkCoef* __restrict__ coef, const double* __restrict__ target,
                                                  double inner_rtol, int64_t max_it, int* dom_active) {
  __shared__ double sh[6 * kBlkM];   // the warps' partial sums, then the matrices of the finishing CTA
  __shared__ int64_t base[kChunkMax];
  __shared__ int last;
  __shared__ double worst;
  const Chunk ch = chunks[blockIdx.x];
  if (!dom_active[ch.dom]) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < ch.count; i += 256) base[i] = (list[ch.first + i] & kListNodeMask) * (3 * kNLC);
  __syncthreads();
  double acc[6][2];
#pragma unroll
  for (int t = 0; t < 6; ++t) acc[t][0] = acc[t][1] = 0.0;
  const int rows = 3 * ch.count, rk = lane & 3, lq = lane >> 2;
#pragma unroll 4
  for (int r0 = 4 * warp; r0 < rows; r0 += 32) {
    const int row = r0 + rk;
    float va[3] = {0.f, 0.f, 0.f}, vb[3] = {0.f, 0.f, 0.f};
    if (row < rows) {
      const int64_t k = base[row / 3] + (row % 3) * kNLC + lq;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        va[i] = __ldg(a + k + 8 * i);
        vb[i] = __ldg(b + k + 8 * i);
      }
    }
    double da[3], db[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) { da[i] = (double)va[i]; db[i] = (double)vb[i]; }
    dmma884(acc[0], da[0], db[0]);
    dmma884(acc[1], da[0], db[1]);
    dmma884(acc[2], da[0], db[2]);
    dmma884(acc[3], da[1], db[1]);
    dmma884(acc[4], da[1], db[2]);
    dmma884(acc[5], da[2], db[2]);
  }
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    sh[warp * kGramPart + t * 64 + lq * 8 + 2 * rk] = acc[t][0];
    sh[warp * kGramPart + t * 64 + lq * 8 + 2 * rk + 1] = acc[t][1];
  }
  __syncthreads();
  double* g = gram + (int64_t)ch.dom * kGramPart;
  for (int e = tid; e < kGramPart; e += 256) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += sh[w * kGramPart + e];
    atomicAdd(g + e, s);
  }
  const bool renorm = STEP == kBlkCurv && state[ch.dom].renorm != 0;
  double* gh = gram_h + (int64_t)ch.dom * kBlkM;
  if (renorm) {   // P^T R (all 9 tiles)
    double h[9][2];
#pragma unroll
    for (int t = 0; t < 9; ++t) h[t][0] = h[t][1] = 0.0;
#pragma unroll 2
    for (int r0 = 4 * warp; r0 < rows; r0 += 32) {
      const int row = r0 + rk;
      double da[3] = {0, 0, 0}, db[3] = {0, 0, 0};
      if (row < rows) {
        const int64_t k = base[row / 3] + (row % 3) * kNLC + lq;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          da[i] = (double)__ldg(a + k + 8 * i);
          db[i] = (double)__ldg(r + k + 8 * i);
        }
      }
#pragma unroll
      for (int t = 0; t < 9; ++t) dmma884(h[t], da[t / 3], db[t % 3]);
    }
    for (int w = 0; w < 8; ++w) {
      __syncthreads();
      if (warp != w) continue;
#pragma unroll
      for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          double& q = sh[t * 64 + lq * 8 + 2 * rk + c];
          q = w == 0 ? h[t][c] : q + h[t][c];
        }
    }
    __syncthreads();
    for (int e = tid; e < kBlkM; e += 256) atomicAdd(gh + e, sh[e]);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(done + ch.dom, 1) == nchunk[ch.dom] - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (tid == 0) done[ch.dom] = 0;
  BlkState& st = state[ch.dom];
  BlkCoef& cf = coef[ch.dom];
  static_assert(6 * kBlkM >= 8 * kGramPart, "the partial sums of 8 warps");
  double *A = sh, *U = sh + kBlkM, *L = sh + 2 * kBlkM, *T = sh + 3 * kBlkM, *M = sh + 4 * kBlkM;
  int bad = 0;
  for (int e = tid; e < kGramPart; e += 256) {
    const double v = __ldcg(g + e);
    g[e] = 0.0;
    bad |= !isfinite(v);
    const int t = e >> 6, m = (e >> 3) & 7, n = e & 7;
    const int ti = t < 3 ? 0 : t < 5 ? 1 : 2, tj = t < 3 ? t : t < 5 ? t - 2 : 2;
    const int i = 8 * ti + m, j = 8 * tj + n;
    if (ti != tj || i <= j) { A[i * kNLC + j] = v; A[j * kNLC + i] = v; }
  }
  bad = __syncthreads_or(bad);
  double minp;
  int kept;
  if (STEP == kBlkCurv) {
    if (renorm) {   // M = H = P^T R tau
      for (int e = tid; e < kBlkM; e += 256) {
        const int t = e >> 6, m = (e >> 3) & 7, n = e & 7;
        const double v = __ldcg(gh + e);
        gh[e] = 0.0;
        bad |= !isfinite(v);
        U[(8 * (t / 3) + m) * kNLC + 8 * (t % 3) + n] = v;
        L[e] = (double)cf.tau[e];
      }
      bad = __syncthreads_or(bad);
      blk_mul<false>(U, L, M);
      double* Hs = sh + 5 * kBlkM;
      for (int e = tid; e < kBlkM; e += 256) {
        const int i = e / kNLC, j = e % kNLC;
        const bool good = M[i * (kNLC + 1)] > kBlkNoise && M[j * (kNLC + 1)] > kBlkNoise;
        Hs[e] = good ? 0.5 * (M[e] + M[j * kNLC + i]) : 0.0;
        if (!good) A[e] = 0.0;
      }
      __syncthreads();
      blk_factor(Hs, U, L, T, kBlkDropH, minp, kept);
      for (int e = tid; e < kBlkM; e += 256) {
        const int i = e / kNLC, j = e % kNLC;
        if (T[i * (kNLC + 1)] == 0.0 || T[j * (kNLC + 1)] == 0.0) A[e] = 0.0;
        double s = 0.0;
        for (int k = 0; k < kNLC; ++k) s = fma(T[i * kNLC + k], T[j * kNLC + k], s);
        st.Cinv[e] = s;
      }
      __syncthreads();
    } else {
      for (int e = tid; e < kBlkM; e += 256) M[e] = st.C[e];
    }
    blk_factor(A, U, L, T, kBlkDropG, minp, kept);
    if (bad || kept == 0 || minp < -kBlkNegative) {   // non-finite, no direction of positive curvature, or rounding
      for (int e = tid; e < kBlkM; e += 256) cf.alpha[e] = cf.gamma[e] = 0.f;
      if (tid == 0) {
        st.its += 1;
        st.reason = bad ? kNanOrInf : kept == 0 ? kIndefinite : kDivergedIts;
        st.active = 0;
        dom_active[ch.dom] = 0;
      }
      return;
    }
    blk_mul<true>(T, M, U);      // T^T C
    blk_mul<false>(T, U, L);     // alpha = T T^T C
    for (int e = tid; e < kBlkM; e += 256) { A[e] = st.sig[e]; cf.alpha[e] = (float)L[e]; }
    __syncthreads();
    blk_mul<false>(L, A, M);
    for (int e = tid; e < kBlkM; e += 256) cf.gamma[e] = (float)M[e];
    if (tid == 0) st.its += 1;
    return;
  }
  // C step: norms of the residuals of the load cases in the preconditioner's inner product
  double* S = U;   // sigma
  for (int e = tid; e < kBlkM; e += 256) S[e] = STEP == kBlkInit ? (e % (kNLC + 1) == 0 ? 1.0 : 0.0) : st.sig[e];
  __syncthreads();
  blk_mul<false>(A, S, M);       // C sigma
  int diverged = 0;
  double ratio = 0.0;
  if (tid < kNLC) {
    double q = 0.0;
    for (int i = 0; i < kNLC; ++i) q = fma(S[i * kNLC + tid], M[i * kNLC + tid], q);
    const double nrm = sqrt(fmax(q, 0.0));
    const double n0 = STEP == kBlkInit ? nrm : st.n0[tid];
    if (STEP == kBlkInit) st.n0[tid] = nrm;
    if (n0 > 0.0) {
      ratio = nrm / (fmax(inner_rtol, target[(int64_t)ch.dom * kNLC + tid]) * n0);
      diverged = nrm >= 1e5 * n0;
    }
  }
  if (tid < 32) {
#pragma unroll
    for (int o = 16; o; o >>= 1) ratio = fmax(ratio, __shfl_xor_sync(0xffffffffu, ratio, o));
    if (tid == 0) worst = ratio;
  }
  diverged = __syncthreads_or(diverged);
  const int its = STEP == kBlkInit ? 0 : st.its;
  int reason = kIterating;
  if (bad) reason = kNanOrInf;
  else if (diverged) reason = kDivergedDtol;
  else if (worst <= 1.0) reason = kConverged;
  else if (its >= max_it) reason = kDivergedIts;
  else if (STEP == kBlkRes && worst >= st.best && its - st.best_it >= max(kBlkPatience, st.best_it)) reason = kDivergedIts;
  else if (STEP == kBlkRes && st.best < kBlkFar * st.first && worst > kBlkRise * st.best) reason = kDivergedIts;
  if (reason == kIterating) {
    for (int e = tid; e < kBlkM; e += 256) st.sig[e] = S[e];
    __syncthreads();
    blk_factor(A, U, L, T, kBlkDropC, minp, kept);   // S is overwritten, M stays
    if (kept == 0) reason = kIndefinite;
  }
  if (reason != kIterating) {
    if (tid == 0) {
      st.its = its;
      st.reason = reason;
      st.active = 0;
      dom_active[ch.dom] = 0;
    }
    return;
  }
  const bool tilt = minp < kBlkRenorm;
  if (STEP == kBlkInit) {
    for (int e = tid; e < kBlkM; e += 256) U[e] = 0.0;
    __syncthreads();
  } else {
    for (int e = tid; e < kBlkM; e += 256) L[e] = st.Cinv[e];
    __syncthreads();
    blk_mul<false>(L, A, U);     // beta = C_old^-1 C
  }
  if (tilt) {
    blk_mul<true>(T, M, L);      // sigma = tau^T C sigma
    for (int e = tid; e < kBlkM; e += 256) { st.sig[e] = L[e]; cf.tau[e] = (float)T[e]; }
    blk_mul<false>(U, T, M);     // beta tau (ends with a barrier; reads U and T only)
    for (int e = tid; e < kBlkM; e += 256) {
      const int i = e / kNLC, j = e % kNLC;
      const double one = i == j && T[e] != 0.0 ? 1.0 : 0.0;
      st.C[e] = one;
      st.Cinv[e] = one;
      cf.beta[e] = (float)M[e];
    }
  } else {
    for (int e = tid; e < kBlkM; e += 256) {
      const int i = e / kNLC, j = e % kNLC;
      double s = 0.0;
#pragma unroll 8
      for (int k = 0; k < kNLC; ++k) s = fma(T[i * kNLC + k], T[j * kNLC + k], s);
      st.C[e] = A[e];
      st.Cinv[e] = s;
      cf.beta[e] = (float)U[e];
    }
  }
  if (tid == 0) {
    st.its = its;
    if (STEP == kBlkInit) st.first = worst;
    if (STEP == kBlkInit || worst < st.best) {
      st.best = worst;
      st.best_it = its;
    }
    st.reason = kIterating;
    st.active = 1;
    st.renorm = tilt;
  }
}

// One node, 4 load cases: acc[c] += sum_i in[c][i] m[i][4 q ..]; in: the node's 3 staged rows of 24 values
// (kBlkRow apart, so that the 16-byte reads of neighbouring nodes fall into different banks).
constexpr int kBlkRow = 28;
__device__ __forceinline__ void blk_rows(const float* in, const float* m, int q, float2 (&acc)[3][2]) {
#pragma unroll
  for (int i4 = 0; i4 < kNLC; i4 += 4) {
    float v[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 x = *reinterpret_cast<const float4*>(in + c * kBlkRow + i4);
      v[c][0] = x.x; v[c][1] = x.y; v[c][2] = x.z; v[c][3] = x.w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 w = *reinterpret_cast<const float4*>(m + (i4 + i) * kNLC + 4 * q);
      const float2 w0 = make_float2(w.x, w.y), w1 = make_float2(w.z, w.w);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float2 vv = make_float2(v[c][i], v[c][i]);
        acc[c][0] = __ffma2_rn(vv, w0, acc[c][0]);
        acc[c][1] = __ffma2_rn(vv, w1, acc[c][1]);
      }
    }
  }
}
// n staged nodes (3 rows of 24 floats each) of a block, in 16-byte pieces
__device__ __forceinline__ void blk_stage(const float* __restrict__ src, const int64_t* base, int n, float* dst) {
  for (int i = threadIdx.x; i < n * 18; i += 192) {
    const int node = i / 18, part = i % 18;
    *reinterpret_cast<float4*>(dst + (node * 3 + part / 6) * kBlkRow + 4 * (part % 6)) =
        __ldg(reinterpret_cast<const float4*>(src + base[node] + 4 * part));
  }
}
__device__ __forceinline__ void blk_load(const float* p, float2 (&v)[3][2]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float4 x = *reinterpret_cast<const float4*>(p + c * kNLC);
    v[c][0] = make_float2(x.x, x.y);
    v[c][1] = make_float2(x.z, x.w);
  }
}
__device__ __forceinline__ void blk_store(float* p, const float2 (&v)[3][2]) {
#pragma unroll
  for (int c = 0; c < 3; ++c)
    *reinterpret_cast<float4*>(p + c * kNLC) = make_float4(v[c][0].x, v[c][0].y, v[c][1].x, v[c][1].y);
}

// x += P gamma; R = R [tau] - W alpha; t = omega D^-1 R (the first step of the next V-cycle).  A thread owns
// one node and 4 load cases; the rows it multiplies and the 24 x 24 coefficients come from shared memory.
// Bound by the FP32 FMAs (24 per value, twice) and the 7 vectors it moves: 507 us on 384 domains of 32^3
// (4.4 TB/s); the column-by-column update it replaces moved the same vectors at 6.3 TB/s in 2.2 times as
// many iterations.
__global__ void __launch_bounds__(192) k_blk_update(const Chunk* __restrict__ chunks, const int64_t* __restrict__ list,
                                                    float* __restrict__ x, float* __restrict__ r,
                                                    const float* __restrict__ p, const float* __restrict__ w,
                                                    const BlkState* __restrict__ state,
                                                    const BlkCoef* __restrict__ coef, const float* __restrict__ binv,
                                                    float omega, float* __restrict__ t_out,
                                                    const int* __restrict__ dom_active) {
  __shared__ __align__(16) float sp[kBlkTile * 3 * kBlkRow], sw[kBlkTile * 3 * kBlkRow];
  __shared__ __align__(16) float mg[kBlkM], ma[kBlkM], mt[kBlkM];
  __shared__ int64_t base[kBlkTile];
  const Chunk ch = chunks[blockIdx.x];
  if (!dom_active[ch.dom]) return;
  const BlkCoef& cf = coef[ch.dom];
  const bool renorm = state[ch.dom].renorm != 0;
  const int tid = threadIdx.x, q = tid % kQuads, slot = tid / kQuads;
  for (int e = tid; e < kBlkM; e += 192) {
    mg[e] = cf.gamma[e];
    ma[e] = -cf.alpha[e];
    mt[e] = renorm ? cf.tau[e] : 0.f;
  }
  for (int n0 = 0; n0 < ch.count; n0 += kBlkTile) {
    const int n = min(kBlkTile, ch.count - n0);
    if (tid < n) base[tid] = (list[ch.first + n0 + tid] & kListNodeMask) * (3 * kNLC);
    __syncthreads();
    const bool on = slot < n;
    const int64_t k = on ? base[slot] + 4 * q : 0;
    float2 xv[3][2], rv[3][2];
    if (on) {
      blk_load(x + k, xv);
      blk_load(r + k, rv);
    }
    blk_stage(p, base, n, sp);
    blk_stage(w, base, n, sw);
    __syncthreads();
    if (on) {
      blk_rows(sp + slot * 3 * kBlkRow, mg, q, xv);
      blk_store(x + k, xv);
    }
    if (renorm) {
      __syncthreads();
      blk_stage(r, base, n, sp);
      __syncthreads();
      if (on) {
#pragma unroll
        for (int c = 0; c < 3; ++c) rv[c][0] = rv[c][1] = make_float2(0.f, 0.f);
        blk_rows(sp + slot * 3 * kBlkRow, mt, q, rv);
      }
      __syncthreads();   // every row of r is staged before any is written
    }
    if (on) {
      blk_rows(sw + slot * 3 * kBlkRow, ma, q, rv);
      blk_store(r + k, rv);
      const float2* bq = reinterpret_cast<const float2*>(binv + base[slot] / 12);   // 6 per node
      const float2 q0 = __ldg(bq), q1 = __ldg(bq + 1), q2 = __ldg(bq + 2);
      const float b0 = q0.x, b1 = q0.y, b2 = q1.x, b3 = q1.y, b4 = q2.x, b5 = q2.y;
      float2 tv[3][2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 r0 = rv[0][h], r1 = rv[1][h], r2 = rv[2][h];
        tv[0][h] = make_float2(omega * (b0 * r0.x + b3 * r1.x + b4 * r2.x), omega * (b0 * r0.y + b3 * r1.y + b4 * r2.y));
        tv[1][h] = make_float2(omega * (b3 * r0.x + b1 * r1.x + b5 * r2.x), omega * (b3 * r0.y + b1 * r1.y + b5 * r2.y));
        tv[2][h] = make_float2(omega * (b4 * r0.x + b5 * r1.x + b2 * r2.x), omega * (b4 * r0.y + b5 * r1.y + b2 * r2.y));
      }
      blk_store(t_out + k, tv);
    }
    __syncthreads();
  }
}

// P = S [tau] + P beta, as k_blk_update: 216 us on 384 domains of 32^3 (4.4 TB/s, 3 vectors).
__global__ void __launch_bounds__(192) k_blk_direction(const Chunk* __restrict__ chunks,
                                                       const int64_t* __restrict__ list, const float* __restrict__ s,
                                                       float* __restrict__ p, const BlkState* __restrict__ state,
                                                       const BlkCoef* __restrict__ coef,
                                                       const int* __restrict__ dom_active) {
  __shared__ __align__(16) float sp[kBlkTile * 3 * kBlkRow], ss[kBlkTile * 3 * kBlkRow];
  __shared__ __align__(16) float mb[kBlkM], mt[kBlkM];
  __shared__ int64_t base[kBlkTile];
  const Chunk ch = chunks[blockIdx.x];
  if (!dom_active[ch.dom]) return;
  const BlkCoef& cf = coef[ch.dom];
  const bool renorm = state[ch.dom].renorm != 0;
  const int tid = threadIdx.x, q = tid % kQuads, slot = tid / kQuads;
  for (int e = tid; e < kBlkM; e += 192) {
    mb[e] = cf.beta[e];
    mt[e] = renorm ? cf.tau[e] : 0.f;
  }
  for (int n0 = 0; n0 < ch.count; n0 += kBlkTile) {
    const int n = min(kBlkTile, ch.count - n0);
    if (tid < n) base[tid] = (list[ch.first + n0 + tid] & kListNodeMask) * (3 * kNLC);
    __syncthreads();
    const bool on = slot < n;
    const int64_t k = on ? base[slot] + 4 * q : 0;
    float2 v[3][2];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c][0] = v[c][1] = make_float2(0.f, 0.f);
    if (renorm) blk_stage(s, base, n, ss);
    else if (on) blk_load(s + k, v);
    blk_stage(p, base, n, sp);
    __syncthreads();
    if (on) {
      if (renorm) blk_rows(ss + slot * 3 * kBlkRow, mt, q, v);
      blk_rows(sp + slot * 3 * kBlkRow, mb, q, v);
      blk_store(p + k, v);
    }
    __syncthreads();
  }
}

// Iterations and failures of an inner block solve in the outer state of its load cases.
__global__ void k_blk_finish(ColState* __restrict__ ost, const BlkState* __restrict__ state, int64_t ncol) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= ncol || !ost[i].active) return;
  const BlkState& b = state[i / kNLC];
  ost[i].its += b.its;
  ost[i].pad += 1;   // refinement steps taken
  if (b.reason == kIndefinite || b.reason == kNanOrInf || b.reason == kDivergedDtol)
    ost[i].betaold = 1.0;   // remembers an inner failure
}

}  // namespace dtc
