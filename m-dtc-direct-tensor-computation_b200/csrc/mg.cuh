// mg.cuh -- multigrid V-cycle that preconditions the FP32 inner solve (HEX08 grids; a HEX20
// fine level is first coarsened to the HEX08 mesh of the same voxels).
//
// Not a step of the reference (its KSP uses PCJACOBI, f-src/mod_dtc_main_subroutines.f90:
// 995-1078); it only changes how fast the inner FP32 solve of the iterative refinement
// reaches its tolerance, never the FP64 outer residual or the tensor it converges to.
//
// Hierarchy: level l+1 halves the voxel grid of level l (ceil(L/2) voxels per edge); a coarse
// voxel carries the mean of the moduli of its <= 8 children (void and missing children count
// as 0) and twice the edge, so its element matrix is 2 * mean(E) * a * Khat.  For moduli that
// are constant inside each coarse voxel this equals the Galerkin product P^T K P of the
// trilinear prolongation P, because the coarse trilinear space is nested in the fine one.
// Every level keeps all nodes on its domain box fixed (zero correction).  The coarsest level
// (at most 4 voxels per edge, at most 27 interior nodes) is solved with a dense inverse.
//
// Smoother: one damped node-block-Jacobi sweep x = omega D^-1 r, D the 3x3 diagonal blocks
// (Chebyshev of degree 1 on [lambda*/30, 1.1 lambda*]; lambda* = the largest eigenvalue of
// Khat v = lambda De v for the unit voxel, De its node-block diagonal, bounds
// lambda_max(D^-1 K) for any assembly of scaled voxels), the same before and after the coarse
// correction, so the V-cycle is a fixed SPD operator.
//
// One V-cycle per CG iteration, per level l that is not a domain's coarsest:
//   t_l = omega D_l^-1 b_l                        k_mg_jacobi_flat (fine level: k_blk_update)
//   r_l = b_l - K_l t_l                           k_sweep<kSwRes>
//   b_{l+1} = P^T r_l                             k_mg_restrict_flat
//   (level l+1: recurse, or z_{l+1} = K^-1 b)     ...  / k_mg_coarse
//   t_l += P z_{l+1}                              k_mg_prolong_flat
//   z_l = t_l + omega D_l^-1 (b_l - K_l t_l)      k_sweep<kSwPost>
// Levels >= 2 apply the smoothing step twice before and twice after the coarse correction.  In small batches
// k_mg_tail does all of this for the last two levels of a domain.
#pragma once

namespace dtc {

constexpr int kMgMaxCoarse = 4;                  // voxels per edge on the coarsest level
constexpr int kMgDenseN = 81;                    // 3 * 3^3 interior DOFs at most
enum { kMgRes = 0, kMgPost = 1 };
// node-list entries: (domain << kListShift) | node
constexpr int kListShift = 40;
constexpr int64_t kListNodeMask = (int64_t(1) << kListShift) - 1;

// Node-local second half of the residual / smoother when K t was applied on its own
// (HEX20 fine level), z holding -K t on entry:
//   kMgRes : z = b + z
//   kMgPost: z = t + omega D^-1 (b + z)
template <int MODE>
__global__ void __launch_bounds__(kThreads) k_mg_combine(const Tile* __restrict__ tiles, const DomDev* __restrict__ doms,
                                                         const uint8_t* __restrict__ flags,
                                                         const float* __restrict__ binv, const float* __restrict__ b,
                                                         const float* __restrict__ t_in, float* __restrict__ z,
                                                         float omega, const int* __restrict__ dom_active) {
  const Tile t = tiles[blockIdx.x / 3];
  if (dom_active && !dom_active[t.dom]) return;
  const DomDev D = doms[t.dom];
  const int lc = (blockIdx.x % 3) * kLcGroup + (threadIdx.x & 7);
  const int row = threadIdx.x >> 3;
  const int yy = t.y0 + (row & 3), zz = t.z0 + (row >> 2);
  if (yy >= 1 && yy <= D.n[1] - 2 && zz >= 1 && zz <= D.n[2] - 2) {
    for (int i = 0; i < kTileX; ++i) {
      const int x = t.x0 + i;
      if (x > D.n[0] - 2) break;
      const int64_t n = node_index(D, x, yy, zz);
      if (!(flags[n] & kNodeActive)) continue;
      const int64_t k0 = vec_index(n, 0, lc);
      float bc[3], res[3], v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        bc[c] = b[k0 + c * kNLC];
        res[c] = bc[c] + z[k0 + c * kNLC];
      }
      if (MODE == kMgRes) {
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = res[c];
      } else {
        float dz[3];
        block_jacobi(binv, n, omega, res, dz);
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = t_in[k0 + c * kNLC] + dz[c];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) z[k0 + c * kNLC] = v[c];
    }
  }
}

// -------------------------------------------------------------------------------------
// Grid transfers over node lists: one thread per (active interior node, 4 load cases) with
// 16-byte loads and stores, all threads independent.  (A tile walk, one thread per node row and
// load case, visits a tile's nodes one after the other including its inactive ones, and ran at
// 27-38 % of the HBM bandwidth; these lists carry only the active nodes.)
constexpr int kQuads = kNLC / 4;

__device__ __forceinline__ float4 ldq(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void fmaq(float w, float4 v, float4& s) {
  s.x = fmaf(w, v.x, s.x);
  s.y = fmaf(w, v.y, s.y);
  s.z = fmaf(w, v.z, s.z);
  s.w = fmaf(w, v.w, s.w);
}

// t_f += P z_c (trilinear) over a fine level's node list; domains without a coarser level
// (their coarse record is empty) are skipped.
__global__ void __launch_bounds__(256) k_mg_prolong_flat(const int64_t* __restrict__ list, int64_t nitems,
                                                         const DomDev* __restrict__ doms_f,
                                                         const DomDev* __restrict__ doms_c,
                                                         const float* __restrict__ z_c, float* __restrict__ t_f,
                                                         const int* __restrict__ dom_active) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nitems) return;
  const int64_t e = __ldg(list + i / kQuads);
  const int dom = (int)(e >> kListShift);
  if (dom_active && !dom_active[dom]) return;
  const DomDev C = doms_c[dom];
  if (C.n[0] == 0) return;
  const DomDev F = doms_f[dom];
  const int64_t nf = e & kListNodeMask;
  const int loc = (int)(nf - F.node_off);
  const int x = loc % F.n[0], yz = loc / F.n[0];
  const int y = yz % F.n[1], z = yz / F.n[1];
  const int lc0 = 4 * (int)(i % kQuads);
  const int cx0 = x >> 1, cx1 = (x + 1) >> 1, cy0 = y >> 1, cy1 = (y + 1) >> 1, cz0 = z >> 1, cz1 = (z + 1) >> 1;
  float4 s[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) s[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int kz = 0; kz < 2; ++kz)
#pragma unroll
    for (int ky = 0; ky < 2; ++ky)
#pragma unroll
      for (int kx = 0; kx < 2; ++kx) {
        const int64_t k = vec_index(node_index(C, kx ? cx1 : cx0, ky ? cy1 : cy0, kz ? cz1 : cz0), 0, lc0);
#pragma unroll
        for (int c = 0; c < 3; ++c) fmaq(0.125f, ldq(z_c + k + c * kNLC), s[c]);
      }
  const int64_t k0 = vec_index(nf, 0, lc0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float4* q = reinterpret_cast<float4*>(t_f + k0 + c * kNLC);
    float4 v = *q;
    v.x += s[c].x;
    v.y += s[c].y;
    v.z += s[c].z;
    v.w += s[c].w;
    *q = v;
  }
}

// b_c = P^T r_f (full weighting) over a coarse level's node list.  Branch-free, so that the loads of a z plane
// are in flight together (coarse levels of 24 domains of 32^3: 21 -> 16 us).
__global__ void __launch_bounds__(256) k_mg_restrict_flat(const int64_t* __restrict__ list, int64_t nitems,
                                                          const DomDev* __restrict__ doms_c,
                                                          const DomDev* __restrict__ doms_f,
                                                          const float* __restrict__ r_f, float* __restrict__ b_c,
                                                          const int* __restrict__ dom_active) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nitems) return;
  const int64_t e = __ldg(list + i / kQuads);
  const int dom = (int)(e >> kListShift);
  if (dom_active && !dom_active[dom]) return;
  const DomDev C = doms_c[dom];
  const DomDev F = doms_f[dom];
  const int64_t nc = e & kListNodeMask;
  const int loc = (int)(nc - C.node_off);
  const int x = loc % C.n[0], yz = loc / C.n[0];
  const int y = yz % C.n[1], z = yz / C.n[1];
  const int lc0 = 4 * (int)(i % kQuads);
  float4 s[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) s[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  // the 27 fine nodes; one past the grid's far side (odd voxel count) has weight 0, its neighbour's address
#pragma unroll 1
  for (int dz = -1; dz <= 1; ++dz) {
    const int fz = 2 * z + dz;
    const float wz = fz > F.n[2] - 1 ? 0.f : dz ? 0.5f : 1.f;
    const int64_t pz = node_index(F, 0, 0, min(fz, F.n[2] - 1));
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      const int fy = 2 * y + dy;
      const float wy = fy > F.n[1] - 1 ? 0.f : dy ? 0.5f * wz : wz;
      const int64_t py = pz + (int64_t)F.n[0] * min(fy, F.n[1] - 1);
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        const int fx = 2 * x + dx;
        const float wgt = fx > F.n[0] - 1 ? 0.f : dx ? 0.5f * wy : wy;
        const int64_t k = vec_index(py + min(fx, F.n[0] - 1), 0, lc0);
#pragma unroll
        for (int c = 0; c < 3; ++c) fmaq(wgt, ldq(r_f + k + c * kNLC), s[c]);
      }
    }
  }
  const int64_t k0 = vec_index(nc, 0, lc0);
#pragma unroll
  for (int c = 0; c < 3; ++c) *reinterpret_cast<float4*>(b_c + k0 + c * kNLC) = s[c];
}

// t = omega D^-1 b (pre-smoothing from a zero guess) over a level's node list, for the domains
// that have a coarser level (the record of the next level is not empty).
__global__ void __launch_bounds__(256) k_mg_jacobi_flat(const int64_t* __restrict__ list, int64_t nitems,
                                                        const DomDev* __restrict__ doms_next,
                                                        const float* __restrict__ binv, const float* __restrict__ b,
                                                        float omega, float* __restrict__ t_out,
                                                        const int* __restrict__ dom_active) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nitems) return;
  const int64_t e = __ldg(list + i / kQuads);
  const int dom = (int)(e >> kListShift);
  if (dom_active && !dom_active[dom]) return;
  if (doms_next[dom].n[0] == 0) return;
  const int64_t n = e & kListNodeMask;
  const int64_t k0 = vec_index(n, 0, 4 * (int)(i % kQuads));
  const float4 r0 = ldq(b + k0), r1 = ldq(b + k0 + kNLC), r2 = ldq(b + k0 + 2 * kNLC);
  const float* bp = binv + n * 6;
  const float b0 = __ldg(bp), b1 = __ldg(bp + 1), b2 = __ldg(bp + 2), b3 = __ldg(bp + 3), b4 = __ldg(bp + 4),
              b5 = __ldg(bp + 5);
  float4 z0, z1, z2;
  z0.x = omega * (b0 * r0.x + b3 * r1.x + b4 * r2.x);
  z1.x = omega * (b3 * r0.x + b1 * r1.x + b5 * r2.x);
  z2.x = omega * (b4 * r0.x + b5 * r1.x + b2 * r2.x);
  z0.y = omega * (b0 * r0.y + b3 * r1.y + b4 * r2.y);
  z1.y = omega * (b3 * r0.y + b1 * r1.y + b5 * r2.y);
  z2.y = omega * (b4 * r0.y + b5 * r1.y + b2 * r2.y);
  z0.z = omega * (b0 * r0.z + b3 * r1.z + b4 * r2.z);
  z1.z = omega * (b3 * r0.z + b1 * r1.z + b5 * r2.z);
  z2.z = omega * (b4 * r0.z + b5 * r1.z + b2 * r2.z);
  z0.w = omega * (b0 * r0.w + b3 * r1.w + b4 * r2.w);
  z1.w = omega * (b3 * r0.w + b1 * r1.w + b5 * r2.w);
  z2.w = omega * (b4 * r0.w + b5 * r1.w + b2 * r2.w);
  *reinterpret_cast<float4*>(t_out + k0) = z0;
  *reinterpret_cast<float4*>(t_out + k0 + kNLC) = z1;
  *reinterpret_cast<float4*>(t_out + k0 + 2 * kNLC) = z2;
}

// Coarsest level: z = Minv b over the <= 27 interior nodes of each listed domain (one CTA per
// domain, Minv 81 x 81 symmetric on the DOFs 3 * ((x-1) + 3 (y-1) + 9 (z-1)) + c).  A thread owns one DOF and
// 8 load cases; the symmetric matrix is read by columns, so that a warp reads consecutive entries.  Bound by
// the latency of its 81 steps: 36 -> 21 us (24 domains; one thread per output read a row of the matrix).
constexpr int kMgCoarseThreads = 3 * 96;
__global__ void __launch_bounds__(kMgCoarseThreads) k_mg_coarse(const int* __restrict__ list,
                                                                const DomDev* __restrict__ doms,
                                                                const float* __restrict__ minv,
                                                                const float* __restrict__ b, float* __restrict__ z,
                                                                const int* __restrict__ dom_active) {
  __shared__ __align__(16) float sb[kMgDenseN * kNLC];
  const int d = list[blockIdx.x];
  if (dom_active && !dom_active[d]) return;
  const DomDev D = doms[d];
  const int ix = D.n[0] - 2, iy = D.n[1] - 2, iz = D.n[2] - 2;   // interior nodes per axis (<= 3)
  for (int i = threadIdx.x; i < kMgDenseN * kNLC; i += kMgCoarseThreads) {
    const int lc = i % kNLC, dof = i / kNLC, node = dof / 3, c = dof % 3;
    const int x = node % 3, y = (node / 3) % 3, zc = node / 9;
    float v = 0.f;
    if (x < ix && y < iy && zc < iz) v = b[vec_index(node_index(D, x + 1, y + 1, zc + 1), c, lc)];
    sb[i] = v;
  }
  __syncthreads();
  const int dof = threadIdx.x % 96, lc0 = 8 * (threadIdx.x / 96);
  const int node = dof / 3, c = dof % 3, x = node % 3, y = (node / 3) % 3, zc = node / 9;
  if (dof >= kMgDenseN || x >= ix || y >= iy || zc >= iz) return;
  const float* M = minv + (int64_t)d * kMgDenseN * kMgDenseN + dof;
  float s[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) s[q] = 0.f;
#pragma unroll 9
  for (int k = 0; k < kMgDenseN; ++k) {
    const float m = __ldg(M + k * kMgDenseN);
    const float4 v0 = *reinterpret_cast<const float4*>(sb + k * kNLC + lc0);
    const float4 v1 = *reinterpret_cast<const float4*>(sb + k * kNLC + lc0 + 4);
    s[0] = fmaf(m, v0.x, s[0]); s[1] = fmaf(m, v0.y, s[1]); s[2] = fmaf(m, v0.z, s[2]); s[3] = fmaf(m, v0.w, s[3]);
    s[4] = fmaf(m, v1.x, s[4]); s[5] = fmaf(m, v1.y, s[5]); s[6] = fmaf(m, v1.z, s[6]); s[7] = fmaf(m, v1.w, s[7]);
  }
  float* zp = z + vec_index(node_index(D, x + 1, y + 1, zc + 1), c, lc0);
  *reinterpret_cast<float4*>(zp) = make_float4(s[0], s[1], s[2], s[3]);
  *reinterpret_cast<float4*>(zp + 4) = make_float4(s[4], s[5], s[6], s[7]);
}

// The last two levels of the domains whose coarsest level the list holds (level l of at most 8^3 voxels, level
// l + 1 of at most 4^3): pre-smoothing, residual, restriction, dense solve, prolongation and post-smoothing of 4
// load cases of one domain in one CTA, in shared memory.  As kernels of their own these steps are 6 (8 where the
// level smooths twice) launches of a few microseconds, each a serial chain over a grid too small for the card.
// A thread applies K to one node and load case from the differences to its 26 neighbours, which keeps
// rigid translations exact null vectors.  Bound by shared-memory reads (81 a node and load case) and the
// latency between its 7 (9) barriers.  One domain of 16^3: coarse levels 1.34 -> 0.71 ms of a solve, the solve
// 4.7 -> 3.6 ms; 16 domains of 32^3 with 60 load cases 32 -> 23 ms, the solve 148 -> 115.
constexpr int kTailThreads = 512, kTailLc = 4, kTailN = 9, kTailIn = 7;   // nodes per edge, interior ones
constexpr int kTailVec = kTailN * kTailN * kTailN * 3 * kTailLc;
constexpr int kTailItems = kTailIn * kTailIn * kTailIn * kTailLc;
constexpr int kTailCoarse = 5 * 5 * 5 * 3 * kTailLc;
constexpr int kTailFloats = 2 * kTailVec + 3 * kTailItems + 6 * kTailItems / kTailLc + 512 + kMgDenseN * kMgDenseN +
                            kMgDenseN * kTailLc + kTailCoarse;
constexpr int kTailSmem = 4 * kTailFloats + kTailItems / kTailLc;

// sum over the 8 voxels around a node of s_v Khat (u - u(node)); u: the node's load case in the staged
// vector, sv: its voxel on the low sides (stride 8)
__device__ __forceinline__ void tail_apply(const VoxelMatrix<float>& kh, const float* u, const float* sv,
                                           float (&r)[3]) {
  constexpr int X = 3 * kTailLc, Y = kTailN * X, Z = kTailN * Y;
  float d[27][3];
#pragma unroll
  for (int n = 0; n < 27; ++n)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      d[n][c] = u[(n % 3 - 1) * X + (n / 3 % 3 - 1) * Y + (n / 9 - 1) * Z + c * kTailLc];
#pragma unroll
  for (int n = 0; n < 27; ++n)
    if (n != 13)
#pragma unroll
      for (int c = 0; c < 3; ++c) d[n][c] -= d[13][c];
  r[0] = r[1] = r[2] = 0.f;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int vx = v & 1, vy = v >> 1 & 1, vz = v >> 2;   // 0: the voxel on the low side
    const int a = corner_local(1 - vx, 1 - vy, 1 - vz);
    float k[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int qx = q & 1, qy = q >> 1 & 1, qz = q >> 2, e = corner_local(qx, qy, qz);
      const int n = (vx + qx) + 3 * (vy + qy) + 9 * (vz + qz);
      if (e == a) continue;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) k[i] = fmaf(kh.v[3 * a + i + 24 * (3 * e + j)], d[n][j], k[i]);
    }
    const float s = sv[vx + 8 * vy + 64 * vz];
#pragma unroll
    for (int i = 0; i < 3; ++i) r[i] = fmaf(s, k[i], r[i]);
  }
}

__global__ void __launch_bounds__(kTailThreads, 1)
    k_mg_tail(const int* __restrict__ list, const DomDev* __restrict__ doms_f, const DomDev* __restrict__ doms_c,
              const float* __restrict__ svox, const __grid_constant__ VoxelMatrix<float> kh,
              const uint8_t* __restrict__ flags, const float* __restrict__ binv, const float* __restrict__ minv,
              const float* __restrict__ b, float* __restrict__ z, float omega, int steps,
              const int* __restrict__ dom_active) {
  extern __shared__ __align__(16) unsigned char tail_smem[];
  constexpr int kNodes = kTailItems / kTailLc, NT = kTailThreads;
  float* src = reinterpret_cast<float*>(tail_smem);
  float* dst = src + kTailVec;
  float* sb = dst + kTailVec;                       // b, [item][3]
  float* sd = sb + 3 * kTailItems;                  // D^-1, [node][6]
  float* sv = sd + 6 * kNodes;                      // voxel factors, 8^3
  float* sm = sv + 512;                             // dense inverse
  float* bc = sm + kMgDenseN * kMgDenseN;           // [81][4]
  float* zc = bc + kMgDenseN * kTailLc;             // [5^3][3][4], zero on the box
  unsigned char* on = reinterpret_cast<unsigned char*>(zc + kTailCoarse);   // the node is an unknown
  const int dom = list[blockIdx.x / (kNLC / kTailLc)], lc0 = (int)(blockIdx.x % (kNLC / kTailLc)) * kTailLc;
  if (dom_active && !dom_active[dom]) return;
  const DomDev& F = doms_f[dom];
  const DomDev& C = doms_c[dom];
  const int tid = threadIdx.x, n0 = F.n[0], n1 = F.n[1], n2 = F.n[2];
  const int64_t node_off = F.node_off;
  const double scale = F.scale;
  auto at = [](int x, int y, int zz) { return (x + kTailN * (y + kTailN * zz)) * 3 * kTailLc; };
  for (int i = tid; i < 2 * kTailVec; i += NT) src[i] = 0.f;
  for (int i = tid; i < kTailCoarse; i += NT) zc[i] = 0.f;
  for (int i = tid; i < 512; i += NT) {
    const int x = i % 8, y = i / 8 % 8, zz = i / 64;
    sv[i] = x < n0 - 1 && y < n1 - 1 && zz < n2 - 1
                ? __ldg(svox + F.vox_off + x + (int64_t)(n0 - 1) * (y + (int64_t)(n1 - 1) * zz)) : 0.f;
  }
  for (int i = tid; i < kMgDenseN * kMgDenseN; i += NT) sm[i] = __ldg(minv + (int64_t)dom * kMgDenseN * kMgDenseN + i);
  for (int i = tid; i < kNodes; i += NT) {
    const int x = i % kTailIn + 1, y = i / kTailIn % kTailIn + 1, zz = i / (kTailIn * kTailIn) + 1;
    const int64_t n = node_off + x + (int64_t)n0 * (y + (int64_t)n1 * zz);
    const bool use = x <= n0 - 2 && y <= n1 - 2 && zz <= n2 - 2 && (flags[n] & kNodeActive);
    on[i] = use;
    if (use)
      for (int q = 0; q < 6; ++q) sd[6 * i + q] = omega * __ldg(binv + 6 * n + q);
  }
  __syncthreads();
  // the thread's nodes, load case tid % 4; f(index of the node, its position in a vector)
  auto nodes = [&](auto&& f) {
#pragma unroll 1
    for (int i = tid; i < kTailItems; i += NT) {
      const int n = i / kTailLc;
      if (!on[n]) continue;
      const int x = n % kTailIn + 1, y = n / kTailIn % kTailIn + 1, zz = n / (kTailIn * kTailIn) + 1;
      f(n, i, x, y, zz, at(x, y, zz) + tid % kTailLc);
    }
  };
  auto smooth = [&](int n, const float (&r)[3], float (&v)[3]) {
    const float* q = sd + 6 * n;
    v[0] = q[0] * r[0] + q[3] * r[1] + q[4] * r[2];
    v[1] = q[3] * r[0] + q[1] * r[1] + q[5] * r[2];
    v[2] = q[4] * r[0] + q[5] * r[1] + q[2] * r[2];
  };
  nodes([&](int n, int i, int x, int y, int zz, int k) {
    const int64_t g = vec_index(node_off + x + (int64_t)n0 * (y + (int64_t)n1 * zz), 0, lc0 + tid % kTailLc);
    float r[3], v[3];
    for (int c = 0; c < 3; ++c) sb[3 * i + c] = r[c] = __ldg(b + g + c * kNLC);
    smooth(n, r, v);
    for (int c = 0; c < 3; ++c) src[k + c * kTailLc] = v[c];
  });
  __syncthreads();
  const int turn = steps / 2 - 1;   // the step that leaves the residual for the coarse level
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    nodes([&](int n, int i, int x, int y, int zz, int k) {
      float r[3], v[3];
      tail_apply(kh, src + k, sv + (x - 1) + 8 * (y - 1) + 64 * (zz - 1), r);
      for (int c = 0; c < 3; ++c) r[c] = sb[3 * i + c] - (float)(scale * (double)r[c]);   // the scale in FP64, as the sweeps
      if (step == turn) {
        for (int c = 0; c < 3; ++c) dst[k + c * kTailLc] = r[c];
        return;
      }
      smooth(n, r, v);
      for (int c = 0; c < 3; ++c) v[c] += src[k + c * kTailLc];
      if (step < steps - 1) {
        for (int c = 0; c < 3; ++c) dst[k + c * kTailLc] = v[c];
      } else {
        const int64_t g = vec_index(node_off + x + (int64_t)n0 * (y + (int64_t)n1 * zz), 0, lc0 + tid % kTailLc);
        for (int c = 0; c < 3; ++c) z[g + c * kNLC] = v[c];
      }
    });
    __syncthreads();
    if (step != turn) {
      float* q = src;
      src = dst;
      dst = q;
      continue;
    }
    // full weighting, the dense solve on at most 27 nodes, trilinear interpolation
    const int item = tid, lc = item % kTailLc, dof = item / kTailLc, cn = dof / 3, c = dof % 3;
    const int cx = cn % 3 + 1, cy = cn / 3 % 3 + 1, cz = cn / 9 + 1;
    if (dof < kMgDenseN) {
      float s = 0.f;
#pragma unroll
      for (int q = 0; q < 27; ++q) {
        const int dx = q % 3 - 1, dy = q / 3 % 3 - 1, dz = q / 9 - 1;
        const float w = (dx ? 0.5f : 1.f) * (dy ? 0.5f : 1.f) * (dz ? 0.5f : 1.f);
        s = fmaf(w, dst[at(2 * cx + dx, 2 * cy + dy, 2 * cz + dz) + c * kTailLc + lc], s);
      }
      bc[item] = cx <= C.n[0] - 2 && cy <= C.n[1] - 2 && cz <= C.n[2] - 2 ? s : 0.f;
    }
    __syncthreads();
    if (dof < kMgDenseN && cx <= C.n[0] - 2 && cy <= C.n[1] - 2 && cz <= C.n[2] - 2) {
      float s = 0.f;
#pragma unroll 9
      for (int k = 0; k < kMgDenseN; ++k) s = fmaf(sm[k * kMgDenseN + dof], bc[k * kTailLc + lc], s);
      zc[((cx + 5 * (cy + 5 * cz)) * 3 + c) * kTailLc + lc] = s;
    }
    __syncthreads();
    nodes([&](int, int, int x, int y, int zz, int k) {
      float s[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int px = (x + (q & 1)) >> 1, py = (y + (q >> 1 & 1)) >> 1, pz = (zz + (q >> 2)) >> 1;
        for (int c2 = 0; c2 < 3; ++c2)
          s[c2] = fmaf(0.125f, zc[((px + 5 * (py + 5 * pz)) * 3 + c2) * kTailLc + tid % kTailLc], s[c2]);
      }
      for (int c2 = 0; c2 < 3; ++c2) src[k + c2 * kTailLc] += s[c2];
    });
    __syncthreads();
  }
}

}  // namespace dtc
