// rotation.cu -- parallel rotation search of the 6x6 effective tensor (sm_100a, FP64).
//
// mod_struct_calcmat.f90:533-1603 evaluates, for every candidate rotation (alpha about the
// axis n(phi, eta)) on a 1-degree grid alpha, phi in [0,180], eta in [0,90], the
// off-diagonal energy of B^T E B (CR1: rows 1-4 x cols 5-6; CR2: all 12 upper off-diagonal
// entries), takes the first minimum in column-major order (MINLOC), then refines in a
// +-1 step window at 10x finer resolution until the minimum changes by < 1e-9 or 16 rounds.
// Here one thread evaluates the candidates about one axis; the argmin reductions keep MINLOC's tie rule
// (smallest linear index, alpha fastest).  This file is compiled with --fmad=false so every
// criterion is evaluated with the same rounding steps as the written expression.
//
// Sines and cosines: the 1-degree sweep reads two tables built on the host, each refinement
// level builds its 3 x 21 values in shared memory; all of them are the correctly rounded
// values (ddmath.h), the same on the host and the device, so the argmin indices do not
// depend on which math library evaluated them.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "ddmath.h"
#include "fe.h"
#include "kernels.cuh"
#include "solver.h"

namespace cg = cooperative_groups;

namespace dtc {

__constant__ double c_cosd[181], c_sind[181];

namespace {

constexpr int kSweepA = 181, kSweepP = 181, kSweepE = 91;
constexpr int kAxes = kSweepP * kSweepE;
constexpr int kSegments = 8;            // the sweep's work item: one axis, an eighth of the angles about it
constexpr int kSegLen = (kSweepA + kSegments - 1) / kSegments;
constexpr int kSweepBlocks = 64;        // per tensor, when there are many
constexpr int kSweepFill = 888;         // CTAs that fill the card twice (3 on each of 148 SMs)
constexpr int kSweepThreadsRot = 128;
// refinement of one (tensor, criterion): a cluster of 7 CTAs, an item is one of 21 x 21 axes and a part of the angles
constexpr int kRefineCtas = 7, kRefineAxes = 21 * 21 / kRefineCtas, kRefineThreads = 64;   // per part
static_assert(kRefineAxes * kRefineCtas == 21 * 21 && kRefineAxes <= kRefineThreads, "an item per thread");

// The axis of a candidate rotation and the products of its components.
struct Axis {
  double n0, n1, n2, n00, n11, n22, n12, n13, n23;
  __device__ __forceinline__ Axis(double cp, double sp, double ce, double se) {
    n0 = cp * se; n1 = sp * se; n2 = ce;
    const double nr = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
    n0 = n0 / nr; n1 = n1 / nr; n2 = n2 / nr;
    n00 = n0 * n0; n11 = n1 * n1; n22 = n2 * n2;
    n12 = n0 * n1; n13 = n0 * n2; n23 = n1 * n2;
  }
};

// Criteria of the rotation by (ca, sa) about an axis (WHICH bit 0: CR1, bit 1: CR2), every expression in the
// reference's order.  Both criteria contain the squares of t15, t25, t35 and t45, and CR2 all terms of CR1:
// once such a sum alone is above what some candidate is known to reach (most1, most2: with a margin far above
// the rounding of a dozen terms), the candidate cannot be the first minimum, and the criterion is returned as
// infinity.  Of rotated orthotropic tensors with noise 46 to 89 of 100 candidates end before the
// second column of the product and 2 to 12 reach the last.
template <int WHICH>
__device__ __forceinline__ void criteria(const volatile double* E, const Axis& x, double ca, double sa, double most1,
                                         double most2, double& c1, double& c2) {
  const double omc = 1.0 - ca;
  double a11 = ca + x.n00 * omc, a22 = ca + x.n11 * omc, a33 = ca + x.n22 * omc;
  double a12 = x.n12 * omc - x.n2 * sa, a21 = x.n12 * omc + x.n2 * sa;
  double a13 = x.n13 * omc + x.n1 * sa, a31 = x.n13 * omc - x.n1 * sa;
  double a23 = x.n23 * omc - x.n0 * sa, a32 = x.n23 * omc + x.n0 * sa;
  // the columns of B are formed again for each column j of the product instead of kept: 72 registers less
  auto again = [&]() {
    asm volatile("" : "+d"(a11), "+d"(a12), "+d"(a13), "+d"(a21), "+d"(a22), "+d"(a23), "+d"(a31), "+d"(a32),
                      "+d"(a33)::"memory");
  };
  const double s2 = 1.4142135623730951;  // sqrt(2), the value std::sqrt(2.0) rounds to
  auto square = [&](double p, double q, double r, double (&B)[6]) {   // columns 1 to 3 from (p, q, r)
    B[0] = p * p; B[1] = q * q; B[2] = r * r;
    B[3] = s2 * q * p; B[4] = s2 * p * r; B[5] = s2 * q * r;
  };
  auto mixed = [&](double p1, double q1, double r1, double p2, double q2, double r2, double (&B)[6]) {   // 4 to 6
    B[0] = s2 * p1 * p2; B[1] = s2 * q1 * q2; B[2] = s2 * r1 * r2;
    B[3] = q1 * p2 + q2 * p1; B[4] = p1 * r2 + p2 * r1; B[5] = q1 * r2 + q2 * r1;
  };
  // S_j(r) = sum_{c=6..1} B(c,j) E(r,c), then T(i,j) = sum_{r=6..1} B(r,i) S_j(r)
  double S[6];
  auto column = [&](const double (&B)[6]) {
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      double s = B[5] * E[r + 6 * 5];
#pragma unroll
      for (int c = 4; c >= 0; --c) s = s + B[c] * E[r + 6 * c];
      S[r] = s;
    }
  };
  auto T = [&](const double (&B)[6]) {
    double t = B[5] * S[5];
#pragma unroll
    for (int r = 4; r >= 0; --r) t = t + B[r] * S[r];
    return t;
  };
  c1 = c2 = INFINITY;
  const double most = fmax(most1, most2);
  double B[6];
  mixed(a11, a21, a31, a13, a23, a33, B);
  column(B);
  square(a11, a21, a31, B);
  const double t15 = T(B);
  square(a12, a22, a32, B);
  const double t25 = T(B);
  if (t15 * t15 + t25 * t25 > most) return;
  square(a13, a23, a33, B);
  const double t35 = T(B);
  mixed(a11, a21, a31, a12, a22, a32, B);
  const double t45 = T(B);
  const double part5 = t15 * t15 + t25 * t25 + t35 * t35 + t45 * t45;
  if (part5 > most) return;
  again();
  mixed(a12, a22, a32, a13, a23, a33, B);
  column(B);
  square(a11, a21, a31, B);
  const double t16 = T(B);
  square(a12, a22, a32, B);
  const double t26 = T(B);
  if (part5 + (t16 * t16 + t26 * t26) > most) return;
  square(a13, a23, a33, B);
  const double t36 = T(B);
  mixed(a11, a21, a31, a12, a22, a32, B);
  const double t46 = T(B);
  if (WHICH & 1) {
    c1 = t15 * t15 + t16 * t16 + t25 * t25 + t26 * t26 + t35 * t35 + t36 * t36 + t45 * t45 + t46 * t46;
    if (!(c1 == c1)) c1 = INFINITY;
  }
  if ((WHICH & 2) && !(part5 + (t16 * t16 + t26 * t26 + t36 * t36 + t46 * t46) > most2)) {
    again();
    mixed(a11, a21, a31, a13, a23, a33, B);
    const double t56 = T(B);
    mixed(a11, a21, a31, a12, a22, a32, B);
    column(B);
    square(a11, a21, a31, B);
    const double t14 = T(B);
    square(a12, a22, a32, B);
    const double t24 = T(B);
    square(a13, a23, a33, B);
    const double t34 = T(B);
    c2 = t14 * t14 + t15 * t15 + t16 * t16 + t24 * t24 + t25 * t25 + t26 * t26 + t34 * t34 + t35 * t35 + t36 * t36 +
         t45 * t45 + t46 * t46 + t56 * t56;
    if (!(c2 == c2)) c2 = INFINITY;
  }
}

struct ArgMin {
  double v;
  int64_t i;
};
__device__ __forceinline__ bool better(const ArgMin& a, const ArgMin& b) {
  return a.v < b.v || (a.v == b.v && a.i < b.i);
}

// The best of all threads of the CTA, in every thread.
__device__ __forceinline__ ArgMin block_argmin(ArgMin m, ArgMin* sh) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    ArgMin q;
    q.v = __shfl_xor_sync(0xffffffffu, m.v, o);
    q.i = __shfl_xor_sync(0xffffffffu, m.i, o);
    if (better(q, m)) m = q;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
    if (better(sh[w], m)) m = sh[w];
  return m;
}

// 1-degree sweep: a thread evaluates the angles of one segment about one axis, whose normalisation (a square
// root and three divisions) it does once.  The CTA first evaluates a coarse subset of the same grid: the
// smallest values there bound what a candidate may reach, and the bounds shrink as its threads find better ones.
// Bound by the FP64 pipe (80 % busy at 12 warps an SM; the register file holds no more): 62 us a tensor when there
// are many, 4.00 ms for 64; one CTA row of angles per thread without the bounds took 6.32.  A single tensor is
// spread over every SM twice over: 0.10 ms, 0.24 with 64 CTAs.
__global__ void __launch_bounds__(kSweepThreadsRot, 3) k_rot_sweep(const double* __restrict__ ee,
                                                                ArgMin* __restrict__ part) {
  __shared__ double E[36];
  __shared__ ArgMin sh[kSweepThreadsRot / 32];
  const int dom = blockIdx.y;
  if (threadIdx.x < 36) E[threadIdx.x] = ee[(int64_t)dom * 36 + threadIdx.x];
  __syncthreads();
  __shared__ long long most[2];   // bits of the bounds, which are not negative: their order is that of the numbers
  {
    ArgMin b1{INFINITY, INT64_MAX}, b2{INFINITY, INT64_MAX};
    if (threadIdx.x < 6 * 6 * 3) {
      const int ia = 30 * (threadIdx.x % 6), ip = 30 * (threadIdx.x / 6 % 6), ie = 45 * (threadIdx.x / 36);
      criteria<3>(E, Axis(c_cosd[ip], c_sind[ip], c_cosd[ie], c_sind[ie]), c_cosd[ia], c_sind[ia], INFINITY,
                  INFINITY, b1.v, b2.v);
    }
    b1 = block_argmin(b1, sh);
    b2 = block_argmin(b2, sh);
    if (threadIdx.x == 0) {
      most[0] = __double_as_longlong(b1.v * (1.0 + 1e-9));
      most[1] = __double_as_longlong(b2.v * (1.0 + 1e-9));
    }
    __syncthreads();
  }
  ArgMin b1{INFINITY, INT64_MAX}, b2{INFINITY, INT64_MAX};
  for (int item = blockIdx.x * kSweepThreadsRot + threadIdx.x; item < kAxes * kSegments;
       item += gridDim.x * kSweepThreadsRot) {
    const int axis = item % kAxes, a0 = item / kAxes * kSegLen, a1 = min(a0 + kSegLen, kSweepA);
    const int ip = axis % kSweepP, ie = axis / kSweepP;
    const Axis x(c_cosd[ip], c_sind[ip], c_cosd[ie], c_sind[ie]);
    const double most1 = __longlong_as_double(*(volatile long long*)&most[0]);
    const double most2 = __longlong_as_double(*(volatile long long*)&most[1]);
    for (int ia = a0; ia < a1; ++ia) {
      double c1, c2;
      criteria<3>(E, x, c_cosd[ia], c_sind[ia], most1, most2, c1, c2);
      const int64_t idx = ia + (int64_t)kSweepA * axis;
      // a thread's items do not come in index order: ties go to the smaller index
      if (c1 < b1.v || (c1 == b1.v && idx < b1.i && c1 < INFINITY)) { b1.v = c1; b1.i = idx; }
      if (c2 < b2.v || (c2 == b2.v && idx < b2.i && c2 < INFINITY)) { b2.v = c2; b2.i = idx; }
    }
    const double own1 = b1.v * (1.0 + 1e-9), own2 = b2.v * (1.0 + 1e-9);
    if (own1 < most1) atomicMin(&most[0], __double_as_longlong(own1));
    if (own2 < most2) atomicMin(&most[1], __double_as_longlong(own2));
  }
  const ArgMin r1 = block_argmin(b1, sh);
  const ArgMin r2 = block_argmin(b2, sh);
  if (threadIdx.x == 0) {
    part[((int64_t)dom * gridDim.x + blockIdx.x) * 2 + 0] = r1;
    part[((int64_t)dom * gridDim.x + blockIdx.x) * 2 + 1] = r2;
  }
}

// CTAs per tensor of the sweep: enough to fill the card, at least kSweepBlocks.
int sweep_blocks(int64_t n) { return (int)std::max<int64_t>(kSweepBlocks, kSweepFill / std::max<int64_t>(n, 1)); }

// One cluster per (domain, criterion): reduce the sweep, then the x10 refinement loop, the best of a level
// exchanged through the cluster's shared memories.  Bound by the serial chain of a level: its sines and cosines, 11 or 21
// candidates one after the other, the reduction.  One tensor 0.28 ms, 0.51 with one CTA per search; 64 tensors
// 0.77 ms (0.79).
template <int PARTS>
__global__ void __cluster_dims__(kRefineCtas, 1, 1) __launch_bounds__(kRefineThreads * PARTS, 6 / PARTS)
    k_rot_refine(const double* __restrict__ ee, const ArgMin* __restrict__ part, int nblocks, double pi_div_180,
                 int64_t* __restrict__ ang_out, int* __restrict__ jj_out, double* __restrict__ crit_out) {
  __shared__ double E[36];
  __shared__ ArgMin sh[kRefineThreads * PARTS / 32];
  __shared__ ArgMin level_best[2];   // of this CTA; written for alternate levels
  __shared__ double tsin[3][21], tcos[3][21];
  cg::cluster_group cluster = cg::this_cluster();
  const int dom = blockIdx.x / kRefineCtas, rank = (int)cluster.block_rank();
  const int which = 1 - (int)blockIdx.y;   // CR2, the longer one, first
  if (threadIdx.x < 36) E[threadIdx.x] = ee[(int64_t)dom * 36 + threadIdx.x];
  ArgMin m{INFINITY, INT64_MAX};
  for (int b = threadIdx.x; b < nblocks; b += kRefineThreads * PARTS) {
    const ArgMin q = part[((int64_t)dom * nblocks + b) * 2 + which];
    if (better(q, m)) m = q;
  }
  const ArgMin s0 = block_argmin(m, sh);
  int64_t a[3];
  if (s0.i == INT64_MAX) { a[0] = a[1] = a[2] = 0; }
  else { a[0] = s0.i % kSweepA; a[1] = (s0.i / kSweepA) % kSweepP; a[2] = s0.i / (kSweepA * kSweepP); }
  double prev = s0.v, cur = s0.v;
  double div = pi_div_180;
  int jj = 1;
  const int slot = (int)threadIdx.x % kRefineThreads, part_of = (int)threadIdx.x / kRefineThreads;
  const int axis = rank * kRefineAxes + slot;
  constexpr int kEach = (21 + PARTS - 1) / PARTS;
  for (;;) {   // every CTA of the cluster takes the same decisions
    const int64_t lo[3] = {(a[0] - 1) * 10, (a[1] - 1) * 10, (a[2] - 1) * 10};
    div = div * 0.1;
    if (threadIdx.x < 63) {
      const int d = threadIdx.x / 21, i = threadIdx.x % 21;
      double sv, cv;
      dd::sincos_cr((double)(lo[d] + i) * div, &sv, &cv);
      tsin[d][i] = sv;
      tcos[d][i] = cv;
    }
    __syncthreads();
    ArgMin w{INFINITY, INT64_MAX};
    if (slot < kRefineAxes) {
      const int i1 = axis % 21, i2 = axis / 21;
      const Axis x(tcos[1][i1], tsin[1][i1], tcos[2][i2], tsin[2][i2]);
      for (int i0 = kEach * part_of; i0 < min(kEach * part_of + kEach, 21); ++i0) {
        double c1, c2;
        const double most = w.v * (1.0 + 1e-9);
        if (which == 0) criteria<1>(E, x, tcos[0][i0], tsin[0][i0], most, -INFINITY, c1, c2);
        else criteria<2>(E, x, tcos[0][i0], tsin[0][i0], -INFINITY, most, c1, c2);
        const double c = which == 0 ? c1 : c2;
        if (c < w.v) { w.v = c; w.i = i0 + 21 * (int64_t)axis; }
      }
    }
    const ArgMin mine = block_argmin(w, sh);
    if (threadIdx.x == 0) level_best[jj & 1] = mine;
    cluster.sync();
    ArgMin r{INFINITY, INT64_MAX};
    for (int q = 0; q < kRefineCtas; ++q) {
      const ArgMin o = *cluster.map_shared_rank(&level_best[jj & 1], q);
      if (better(o, r)) r = o;
    }
    cur = r.v;
    if (r.i != INT64_MAX) { a[0] = lo[0] + r.i % 21; a[1] = lo[1] + (r.i / 21) % 21; a[2] = lo[2] + r.i / 441; }
    if (fabs(prev - cur) < 1.0e-9 || jj >= 16) break;
    prev = cur;
    jj += 1;
  }
  cluster.sync();   // no CTA leaves while another reads its best
  if (threadIdx.x == 0 && rank == 0) {
    int64_t* o = ang_out + ((int64_t)dom * 2 + which) * 3;
    o[0] = a[0]; o[1] = a[1]; o[2] = a[2];
    jj_out[dom * 2 + which] = jj;
    crit_out[dom * 2 + which] = cur;
  }
}

// Two threads per axis while all clusters are resident at once (3 CTAs of 128 threads on each of 148 SMs), where
// the serial chain of a level counts; one beyond that, where the FP64 pipe does (64 tensors: 1.08 ms
// with two, 0.77 with one; a single tensor 0.28 with two).
void launch_refine(const double* ee, const ArgMin* part, int64_t n, int nb, int64_t* ang, int* jj, double* crit,
                   cudaStream_t s) {
  const double deg = std::acos(-1.0) / 180.0;
  const dim3 grid((unsigned)(kRefineCtas * n), 2);
  if (2 * kRefineCtas * n <= kSweepFill / 2) k_rot_refine<2><<<grid, 2 * kRefineThreads, 0, s>>>(ee, part, nb, deg, ang, jj, crit);
  else k_rot_refine<1><<<grid, kRefineThreads, 0, s>>>(ee, part, nb, deg, ang, jj, crit);
}

}  // namespace

namespace {
std::mutex g_tables_mu;
bool g_tables_loaded[256] = {false};   // c_cosd / c_sind written on this device ordinal
}  // namespace

// Loads the sweep's degree tables into the current device's constant memory once per device
// and process.  Waits until the copy has landed (a later kernel may run on any stream), so
// the first call must not come inside a stream capture.  Later calls do nothing, so calls
// already in flight on other streams never see the tables being rewritten.
int ensure_degree_tables(std::string& msg) {
  int dev = -1;
  DTC_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) { msg = "device ordinal out of range"; return DTC_ERR_CUDA; }
  std::lock_guard<std::mutex> lock(g_tables_mu);
  if (g_tables_loaded[dev]) return DTC_OK;
  double c[181], sn[181];
  degree_tables(c, sn);
  DTC_CUDA(cudaMemcpyToSymbol(c_cosd, c, sizeof(c)));
  DTC_CUDA(cudaMemcpyToSymbol(c_sind, sn, sizeof(sn)));
  DTC_CUDA(cudaDeviceSynchronize());
  g_tables_loaded[dev] = true;
  return DTC_OK;
}

// Sweep and refinement of every tensor on the device; ms (optional) receives their CUDA-event
// time on stream s.
int rotation_search_device(const std::vector<const double*>& ees, std::vector<int64_t>& ang, std::vector<int>& jj,
                           std::vector<double>& crit, cudaStream_t s, int64_t& launches, std::string& msg,
                           double* ms) {
  const int ndom = (int)ees.size();
  if (ndom == 0) return DTC_OK;
  if (int rc = ensure_degree_tables(msg)) return rc;
  std::vector<double> hee((size_t)36 * ndom);
  for (int d = 0; d < ndom; ++d) std::memcpy(&hee[(size_t)36 * d], ees[d], 36 * sizeof(double));
  double* dee = nullptr;
  ArgMin* dpart = nullptr;
  int64_t* dang = nullptr;
  int* djj = nullptr;
  double* dcrit = nullptr;
  auto cleanup = [&]() {
    cudaFree(dee); cudaFree(dpart); cudaFree(dang); cudaFree(djj); cudaFree(dcrit);
  };
  auto fail = [&](cudaError_t e, const char* what) {
    msg = std::string(what) + ": " + cudaGetErrorString(e);
    cleanup();
    return e == cudaErrorMemoryAllocation ? DTC_ERR_OUT_OF_MEMORY : DTC_ERR_CUDA;
  };
  cudaError_t e;
  if ((e = cudaMalloc(&dee, sizeof(double) * 36 * ndom))) return fail(e, "cudaMalloc");
  const int nb = sweep_blocks(ndom);
  if ((e = cudaMalloc(&dpart, sizeof(ArgMin) * 2 * nb * ndom))) return fail(e, "cudaMalloc");
  if ((e = cudaMalloc(&dang, sizeof(int64_t) * 6 * ndom))) return fail(e, "cudaMalloc");
  if ((e = cudaMalloc(&djj, sizeof(int) * 2 * ndom))) return fail(e, "cudaMalloc");
  if ((e = cudaMalloc(&dcrit, sizeof(double) * 2 * ndom))) return fail(e, "cudaMalloc");
  if ((e = cudaMemcpyAsync(dee, hee.data(), sizeof(double) * 36 * ndom, cudaMemcpyHostToDevice, s)))
    return fail(e, "cudaMemcpyAsync");
  cudaEvent_t ev[2] = {nullptr, nullptr};
  if (ms && (cudaEventCreate(&ev[0]) != cudaSuccess || cudaEventCreate(&ev[1]) != cudaSuccess)) ms = nullptr;
  if (ms) cudaEventRecord(ev[0], s);
  k_rot_sweep<<<dim3(nb, ndom), kSweepThreadsRot, 0, s>>>(dee, dpart);
  launch_refine(dee, dpart, ndom, nb, dang, djj, dcrit, s);
  if (ms) cudaEventRecord(ev[1], s);
  launches += 2;
  if ((e = cudaGetLastError())) {
    for (cudaEvent_t q : ev) if (q) cudaEventDestroy(q);
    return fail(e, "rotation kernels");
  }
  ang.resize(6 * ndom); jj.resize(2 * ndom); crit.resize(2 * ndom);
  if ((e = cudaMemcpyAsync(ang.data(), dang, sizeof(int64_t) * 6 * ndom, cudaMemcpyDeviceToHost, s)) ||
      (e = cudaMemcpyAsync(jj.data(), djj, sizeof(int) * 2 * ndom, cudaMemcpyDeviceToHost, s)) ||
      (e = cudaMemcpyAsync(crit.data(), dcrit, sizeof(double) * 2 * ndom, cudaMemcpyDeviceToHost, s)) ||
      (e = cudaStreamSynchronize(s))) {
    for (cudaEvent_t q : ev) if (q) cudaEventDestroy(q);
    return fail(e, "rotation results");
  }
  if (ms) {
    float t = 0.f;
    *ms = cudaEventElapsedTime(&t, ev[0], ev[1]) == cudaSuccess ? (double)t : 0.0;
  }
  for (cudaEvent_t q : ev) if (q) cudaEventDestroy(q);
  cleanup();
  return DTC_OK;
}

// -------------------------------------------------------------------------------------
// Allocation-free variant of the rotation search.  Its only scratch, the per-block sweep
// minima, lives in a file-scope device array sized for kNoAllocMaxDomains domains
// (1024 x 64 blocks x 2 criteria x 16 B = 2 MiB, held by every device that loads the
// library until the process exits).
constexpr int64_t kNoAllocMaxDomains = 1024;
static __device__ __align__(256) ArgMin g_noalloc_part[kNoAllocMaxDomains * kSweepBlocks * 2];

namespace {
std::mutex g_noalloc_mu;
ArgMin* g_noalloc_ptr[256] = {nullptr};   // device address of g_noalloc_part, per device ordinal
}  // namespace

}  // namespace dtc

extern "C" dtc_status dtc_rotation_search_noalloc(const double* ee, int64_t n, int64_t* ang, int32_t* jj,
                                                  double* crit, void* stream) {
  using namespace dtc;
  if (n < 0 || n > kNoAllocMaxDomains) return DTC_ERR_INVALID_ARGUMENT;
  if (n == 0) return DTC_OK;
  if (!ee || !ang || !jj || !crit) return DTC_ERR_INVALID_ARGUMENT;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return DTC_ERR_CUDA;
  ArgMin* part = nullptr;
  {
    // first call on a device: resolve the scratch array's device address and load the
    // degree tables of the sweep, with that device current
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_noalloc_part) != cudaSuccess || !p) return DTC_ERR_CUDA;
      std::string msg;
      if (ensure_degree_tables(msg) != DTC_OK) return DTC_ERR_CUDA;   // uploads and waits for them
      g_noalloc_ptr[dev] = static_cast<ArgMin*>(p);
    }
    part = g_noalloc_ptr[dev];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // every block of the sweep writes its own two minima, so no clearing is needed
  const int nb = sweep_blocks(n);   // n * nb <= kNoAllocMaxDomains * kSweepBlocks
  k_rot_sweep<<<dim3(nb, (unsigned)n), kSweepThreadsRot, 0, s>>>(ee, part);
  launch_refine(ee, part, n, nb, ang, jj, crit, s);
  return cudaGetLastError() == cudaSuccess ? DTC_OK : DTC_ERR_CUDA;
}
