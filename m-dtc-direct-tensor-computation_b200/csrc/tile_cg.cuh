// tile_cg.cuh -- the plain FP64 CG of HEX08 domains on node tiles: the operator with the dense voxel matrix and
// the vector kernels, one thread per node row and load case.
//
// At a loose tolerance (the reference's default is rtol 1e-3) the CG stops far from the solution, and where it stops
// depends on the order in which an application and a dot product are summed: rounding, amplified by the loss of
// conjugacy, moves a column's stop by an iteration or more, and the tensor by up to 6 rtol.  These kernels keep the
// order that the results of the reference's default setting have always had here: per node the 24 columns of the
// kept voxels' matrices corner by corner, per dot product rows of a tile, then the tile.  On domains of two tiles or
// fewer the results are the same bit for bit from run to run.
//
// The price, against the sweeps and the list kernels (sweep.cuh, k_update): 8 domains of 23^3 at rtol 1e-3
// 12.7 -> 22.9 ms (operator 32 -> 60 us, update 13 -> 23, direction 10 -> 13).  At kTightRtol and below the stop no
// longer shows (two runs differ by less than 1e-9 of the tensor), and the faster kernels are used.
#pragma once

namespace dtc {

// Tolerance up to which the summation order decides nothing: runs, and the two sets of kernels, differ by 0.1 to
// 6 rtol of the tensor, which is below 1e-9 from here on.
constexpr double kTightRtol = 1e-10;

// Voxel-outer FP64 slab of a node row: the kept voxel (b, c) of the row between planes x and x+1 reads its 8
// corners' values from u, kb being the index of the row's value at plane x for its load case, and adds to node x
// (corner offset 0 in x) and node x+1 (offset 1).  FIRST: only node x+1 belongs to the tile.
template <bool FIRST>
__device__ __forceinline__ void voxel_rd(const VoxelMatrix<double>& kh, const double* __restrict__ u, int64_t kb,
                                         int sy, int sz, int b, int c, float s, double (&cur)[3], double (&nxt)[3]) {
  const int l0 = corner_local(0, 1 - b, 1 - c), l1 = corner_local(1, 1 - b, 1 - c);
  double t0 = 0, t1 = 0, t2 = 0, q0 = 0, q1 = 0, q2 = 0;
#pragma unroll 1
  for (int mz = 0; mz < 2; ++mz)
#pragma unroll
    for (int my = 0; my < 2; ++my)
#pragma unroll
      for (int mx = 0; mx < 2; ++mx) {
        const int lm = corner_local(mx, my, mz);
        const int64_t k = kb + mx * (3 * kNLC) + (b - 1 + my) * sy + (c - 1 + mz) * sz;
#pragma unroll
        for (int cj = 0; cj < 3; ++cj) {
          const double v = __ldg(u + k + cj * kNLC);
          const int col = 24 * (3 * lm + cj);
          if (!FIRST) {
            t0 = fma(kh.v[col + 3 * l0 + 0], v, t0);
            t1 = fma(kh.v[col + 3 * l0 + 1], v, t1);
            t2 = fma(kh.v[col + 3 * l0 + 2], v, t2);
          }
          q0 = fma(kh.v[col + 3 * l1 + 0], v, q0);
          q1 = fma(kh.v[col + 3 * l1 + 1], v, q1);
          q2 = fma(kh.v[col + 3 * l1 + 2], v, q2);
        }
      }
  const double ts = (double)s;
  if (!FIRST) {
    cur[0] = fma(ts, t0, cur[0]);
    cur[1] = fma(ts, t1, cur[1]);
    cur[2] = fma(ts, t2, cur[2]);
  }
  nxt[0] = fma(ts, q0, nxt[0]);
  nxt[1] = fma(ts, q1, nxt[1]);
  nxt[2] = fma(ts, q2, nxt[2]);
}

// y = scale * K u on the interior nodes of tiles of kSweepX x kTileY x kTileZ nodes; DOT: acc[col] += u . y.
// bnd_only: u vanishes off the domain box (the right-hand side) and y is zero on entry; a row whose neighbour rows
// lie inside the box then has values at x = 1 and x = n0 - 2 only.  4 CTAs per SM (128 registers).
template <bool DOT>
__global__ void __launch_bounds__(kThreads, 4) k_tile_matvec(const Tile* __restrict__ tiles,
                                                             const DomDev* __restrict__ doms,
                                                             const float* __restrict__ svox,
                                                             const __grid_constant__ VoxelMatrix<double> kh,
                                                             const double* __restrict__ u, double* __restrict__ y,
                                                             double scale, double* __restrict__ acc,
                                                             const int* __restrict__ dom_active, int bnd_only) {
  __shared__ double red[32];
  const Tile t = tiles[blockIdx.x / 3];
  if (dom_active && !dom_active[t.dom]) return;
  const DomDev D = doms[t.dom];
  const int lc = (blockIdx.x % 3) * kLcGroup + (threadIdx.x & 7);
  const int row = threadIdx.x >> 3;
  const int yy = t.y0 + (row & 3), zz = t.z0 + (row >> 2);
  int x0 = t.x0, xe = min(D.n[0] - 2, t.x0 + kSweepX - 1);   // nodes of the row
  if (bnd_only && yy >= 2 && yy <= D.n[1] - 3 && zz >= 2 && zz <= D.n[2] - 3) {
    const bool has_lo = x0 <= 1 && 1 <= xe, has_hi = x0 <= D.n[0] - 2 && D.n[0] - 2 <= xe;
    if (has_lo && !has_hi) xe = 1;
    else if (has_hi && !has_lo) x0 = D.n[0] - 2;
    else if (!has_lo) xe = x0 - 1;   // neither: nothing to compute on this row
  }
  double dot = 0.0;
  if (yy >= 1 && yy <= D.n[1] - 2 && zz >= 1 && zz <= D.n[2] - 2 && x0 <= xe) {
    const int sy = D.n[0] * (3 * kNLC), sz = D.n[0] * D.n[1] * (3 * kNLC);
    int64_t kx = vec_index(node_index(D, x0 - 1, yy, zz), 0, lc);   // plane x0 - 1 of the row
    const float* vp = svox + D.vox_off + (x0 - 1) + (int64_t)D.L[0] * ((yy - 1) + (int64_t)D.L[1] * (zz - 1));
    const int vsy = D.L[0], vsz = D.L[0] * D.L[1];
    float sv[2][2];   // the 4 voxels of the row between planes x and x + 1
    auto voxels = [&]() {
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c) sv[b][c] = __ldg(vp + b * vsy + c * vsz);
      return (sv[0][0] != 0.f) | (sv[0][1] != 0.f) | (sv[1][0] != 0.f) | (sv[1][1] != 0.f);
    };
    double cur[3] = {0, 0, 0}, nxt[3] = {0, 0, 0};
    bool anyp = voxels();
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (sv[b][c] != 0.f) voxel_rd<true>(kh, u, kx, sy, sz, b, c, sv[b][c], cur, nxt);
#pragma unroll 1
    for (int x = x0; x <= xe; ++x) {
      kx += 3 * kNLC;   // plane x
      ++vp;
      const bool anyc = voxels();
#pragma unroll
      for (int c = 0; c < 3; ++c) { cur[c] = nxt[c]; nxt[c] = 0.0; }
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          if (sv[b][c] != 0.f) voxel_rd<false>(kh, u, kx, sy, sz, b, c, sv[b][c], cur, nxt);
      if (anyp | anyc) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double v = scale * D.scale * cur[c];
          y[kx + c * kNLC] = v;
          if (DOT) dot += __ldg(u + kx + c * kNLC) * v;
        }
      }
      anyp = anyc;
    }
  }
  if (DOT) {
    const double s = block_sum_lc<double>(dot, red);
    if (threadIdx.x < 8) atomicAdd(acc + (int64_t)t.dom * kNLC + lc, s);
  }
}

// p = D^-1 r + bfac * p for the iterating columns
__global__ void __launch_bounds__(kThreads) k_tile_direction(const Tile* __restrict__ tiles,
                                                             const DomDev* __restrict__ doms,
                                                             const uint8_t* __restrict__ flags,
                                                             const double* __restrict__ dinv,
                                                             const double* __restrict__ r, double* __restrict__ p,
                                                             const ColState* __restrict__ st,
                                                             const int* __restrict__ dom_active) {
  DTC_TILE_PROLOGUE
  if (!rowok || !st[col].active) return;
  const double bf = st[col].bfac;
  for (int i = 0; i < kTileX; ++i) {
    const int x = t.x0 + i;
    if (x > D.n[0] - 2) break;
    const int64_t n = node_index(D, x, yy, zz);
    if (!(flags[n] & kNodeActive)) continue;
    const int64_t k0 = vec_index(n, 0, lc);
    double rr[3], z[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) rr[c] = r[k0 + c * kNLC];
    precond<double, false>(dinv, n, rr, z);
#pragma unroll
    for (int c = 0; c < 3; ++c) p[k0 + c * kNLC] = z[c] + bf * p[k0 + c * kNLC];
  }
}

// x += alpha p ; r -= alpha w ; z = D^-1 r ; acc_zz += z.z ; acc_zr += z.r, with alpha as in k_update
__global__ void __launch_bounds__(kThreads) k_tile_update(const Tile* __restrict__ tiles,
                                                          const DomDev* __restrict__ doms,
                                                          const uint8_t* __restrict__ flags,
                                                          const double* __restrict__ dinv, double* __restrict__ x,
                                                          double* __restrict__ r, const double* __restrict__ p,
                                                          const double* __restrict__ w,
                                                          const ColState* __restrict__ st,
                                                          const double* __restrict__ acc_pw,
                                                          double* __restrict__ acc_zz, double* __restrict__ acc_zr,
                                                          const int* __restrict__ dom_active) {
  __shared__ double red[32];
  DTC_TILE_PROLOGUE
  double zz2 = 0.0, zr = 0.0;
  const ColState s = st[col];
  const double pw = acc_pw[col];
  const bool flip = s.its > 0 && ((pw > 0) != (s.dpi > 0) || pw == 0.0);
  const bool valid = s.active && pw != 0.0 && !flip;
  if (rowok && valid) {
    const double a = s.beta / pw;
    for (int i = 0; i < kTileX; ++i) {
      const int xx = t.x0 + i;
      if (xx > D.n[0] - 2) break;
      const int64_t n = node_index(D, xx, yy, zz);
      if (!(flags[n] & kNodeActive)) continue;
      const int64_t k0 = vec_index(n, 0, lc);
      double rn[3], z[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t k = k0 + c * kNLC;
        x[k] = x[k] + a * p[k];
        rn[c] = r[k] - a * w[k];
        r[k] = rn[c];
      }
      precond<double, false>(dinv, n, rn, z);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        zz2 += z[c] * z[c];
        zr += z[c] * rn[c];
      }
    }
  }
  const double s1 = block_sum_lc<double>(zz2, red);
  __syncthreads();
  const double s2 = block_sum_lc<double>(zr, red);
  if (threadIdx.x < 8 && valid) {
    atomicAdd(acc_zz + col, s1);
    atomicAdd(acc_zr + col, s2);
  }
}

}  // namespace dtc
