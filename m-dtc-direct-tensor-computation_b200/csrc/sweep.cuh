// sweep.cuh -- HEX08 matrix-free K*u in the Hadamard basis of the voxel (the SIMT sweeps, FP32 and FP64).
//
// The sums and differences of a voxel's corner values along x, y and z split its 24 x 24 stiffness: the
// cube is mirror symmetric, so a displacement component couples only to those of the same parity under the
// three reflections, in eight classes of three.  Per class the matrix has one or two distinct entries,
// 8 numbers in all for any Poisson ratio (hadamard_entries), and the three translations drop out, which
// also makes them exact.  72 additions each way and 31 products replace 576 multiply-adds per voxel and
// load case, and most of the additions are shared: along x by a thread that walks a voxel row (the
// y/z-transformed node plane between two voxels serves both), and the transform back in y and z is done
// once per node plane.
//
// A thread walks one voxel row for 8 bytes of load cases: two of them packed in FP32 (sm_100's packed
// add and FMA), one in FP64.  The 8 x 6 node rows of a tile need the 9 x 7 voxel rows around them; each
// step the threads exchange their shares of the node plane through shared memory, and the thread of
// voxel row (j, k) finishes node row (j, k): its own share and those of three neighbours.  Node-centric
// sweeps without an exchange do every voxel's work four times.
#pragma once

namespace dtc {

constexpr int kVoxRowsY = kSweepY + 1, kVoxRowsZ = kSweepZ + 1;
constexpr int kVoxRows = kVoxRowsY * kVoxRowsZ;   // 63 rows x 4 threads
constexpr int kSweepThreads = 256;
static_assert(kVoxRows * 4 <= kSweepThreads, "one thread per voxel row and 8 bytes of load cases");

// Entries of the transformed unit voxel matrix: axial diagonal - off-diagonal and off-diagonal (the class of
// the normal strains), shear, the corner mode, the same two for the classes that are odd in one axis,
// and for the class that is odd in all three.
enum { kWhAxD, kWhAxO, kWhSh, kWhCo, kWhOneD, kWhOneO, kWhAllD, kWhAllO, kWhNum };
template <typename T> struct Hadamard { T w[kWhNum]; };
template <> struct Hadamard<float> { float2 w[kWhNum]; };   // twice: an operand of packed arithmetic

// The entries from the voxel matrix (column-major 24 x 24): g_b^T K g_a / 64 with g the +-1 corner patterns.
inline void hadamard_entries(const double* khat, double (&w)[kWhNum]) {
  auto entry = [&](int cr, int ar, int cc, int ac) {   // component and pattern (bits x, y, z: difference) of row, column
    auto sign = [](int pat, int x, int y, int z) {
      return ((pat & 1) && !x ? -1 : 1) * ((pat & 2) && !y ? -1 : 1) * ((pat & 4) && !z ? -1 : 1);
    };
    double s = 0.0;
    for (int p = 0; p < 8; ++p)
      for (int q = 0; q < 8; ++q) {
        const int px = p & 1, py = (p >> 1) & 1, pz = p >> 2, qx = q & 1, qy = (q >> 1) & 1, qz = q >> 2;
        s += sign(ar, px, py, pz) * sign(ac, qx, qy, qz) *
             khat[(3 * corner_local(px, py, pz) + cr) + 24 * (3 * corner_local(qx, qy, qz) + cc)];
      }
    return s / 64.0;
  };
  w[kWhAxO] = entry(0, 1, 1, 2);
  w[kWhAxD] = entry(0, 1, 0, 1) - w[kWhAxO];
  w[kWhSh] = entry(0, 2, 1, 1);
  w[kWhCo] = entry(2, 7, 2, 7);
  w[kWhOneO] = entry(1, 3, 2, 5);
  w[kWhOneD] = entry(1, 3, 1, 3) - w[kWhOneO];
  w[kWhAllO] = entry(0, 6, 1, 5);
  w[kWhAllD] = entry(0, 6, 0, 6) - w[kWhAllO];
}

// 8 bytes of load cases
template <typename T> struct Lane;
template <> struct Lane<float> {
  using V = float2;
  static constexpr int kCols = 2;   // load cases per thread
  static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul2_rn(a, b); }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
  static __device__ __forceinline__ V coef(V w, float s) { return __fmul2_rn(w, make_float2(s, s)); }
  static __device__ __forceinline__ V load(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
  static __device__ __forceinline__ void store(float* p, V v) { *reinterpret_cast<float2*>(p) = v; }
  // v * scale with the FP64 scale as two floats: the float that the product in FP64 rounds to (4 million pairs)
  struct Scale {
    float2 hi, lo;
    __device__ __forceinline__ explicit Scale(double s) {
      const float h = (float)s, l = (float)(s - (double)h);
      hi = make_float2(h, h);
      lo = make_float2(l, l);
    }
    __device__ __forceinline__ V operator()(V v) const { return __ffma2_rn(v, hi, __fmul2_rn(v, lo)); }
  };
};
template <> struct Lane<double> {
  using V = double;
  static constexpr int kCols = 1;
  static __device__ __forceinline__ V zero() { return 0.0; }
  static __device__ __forceinline__ V add(V a, V b) { return a + b; }
  static __device__ __forceinline__ V sub(V a, V b) { return a - b; }
  static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ V coef(V w, float s) { return w * (double)s; }
  static __device__ __forceinline__ V load(const double* p) { return __ldg(p); }
  static __device__ __forceinline__ void store(double* p, V v) { *p = v; }
  struct Scale {
    double s;
    __device__ __forceinline__ explicit Scale(double v) : s(v) {}
    __device__ __forceinline__ V operator()(V v) const { return v * s; }
  };
};

// A staged node plane: the node rows around the tile's voxel rows, 3 components x 4 threads' elements each.
constexpr int kPlaneY = kSweepY + 2, kPlaneZ = kSweepZ + 2;
constexpr int kPlaneRows = kPlaneY * kPlaneZ, kPlaneElems = kPlaneRows * 12;
constexpr int kRing = 5;   // planes x .. x + 2 in use, x + 3 and x + 4 on their way

// Sums and differences p[b][c] of the voxel row's four corner values at one staged plane (q: its corner
// (0, 0)): b = 0 sum, 1 difference in y, 2 in z, 3 in both; component c.
template <typename T>
__device__ __forceinline__ void wh_plane(const typename Lane<T>::V* q, typename Lane<T>::V (&p)[4][3]) {
  using L = Lane<T>;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const auto r00 = q[4 * c], r10 = q[4 * c + 12], r01 = q[4 * c + 12 * kPlaneY], r11 = q[4 * c + 12 * kPlaneY + 12];
    const auto s0 = L::add(r10, r00), d0 = L::sub(r10, r00);
    const auto s1 = L::add(r11, r01), d1 = L::sub(r11, r01);
    p[0][c] = L::add(s1, s0);
    p[1][c] = L::add(d1, d0);
    p[2][c] = L::sub(s1, s0);
    p[3][c] = L::sub(d1, d0);
  }
}

// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The voxel between planes p and q (factor s): f holds the transformed force on plane p from the voxel before
// and becomes the whole force on plane p; g becomes this voxel's share of plane q.  A part of a class that
// is even in x (from p + q) pushes both planes alike, an odd one (from q - p) against each other.  Class by
// class, so that few of the 21 sums and differences live at a time.
template <typename T>
__device__ __forceinline__ void wh_voxel(const typename Lane<T>::V (&p)[4][3], const typename Lane<T>::V (&q)[4][3],
                                         const Hadamard<T>& W, float s, typename Lane<T>::V (&f)[4][3],
                                         typename Lane<T>::V (&g)[4][3]) {
  using L = Lane<T>;
  using V = typename L::V;
  auto sum = [&](int b, int c) { return L::add(q[b][c], p[b][c]); };
  auto dif = [&](int b, int c) { return L::sub(q[b][c], p[b][c]); };
  // first and second part of a channel of plane q; the translations (b = 0) have one
  auto even1 = [&](int b, int c, V v) { f[b][c] = L::add(f[b][c], v); g[b][c] = v; };
  auto even2 = [&](int b, int c, V v) { f[b][c] = L::add(f[b][c], v); g[b][c] = L::add(g[b][c], v); };
  auto odd1 = [&](int b, int c, V v) { f[b][c] = L::sub(f[b][c], v); g[b][c] = v; };
  auto odd2 = [&](int b, int c, V v) { f[b][c] = L::sub(f[b][c], v); g[b][c] = L::add(g[b][c], v); };
  const V one_d = L::coef(W.w[kWhOneD], s), one_o = L::coef(W.w[kWhOneO], s), sh = L::coef(W.w[kWhSh], s);
  {   // normal strains
    const V a = dif(0, 0), b = sum(1, 1), c = sum(2, 2);
    const V d = L::coef(W.w[kWhAxD], s), t = L::mul(L::coef(W.w[kWhAxO], s), L::add(L::add(a, b), c));
    odd1(0, 0, L::fma(d, a, t));
    even1(1, 1, L::fma(d, b, t));
    even1(2, 2, L::fma(d, c, t));
  }
  {   // odd in x
    const V a = dif(1, 1), b = dif(2, 2), t = L::mul(one_o, L::add(a, b));
    odd2(1, 1, L::fma(one_d, a, t));
    odd2(2, 2, L::fma(one_d, b, t));
  }
  {   // shear xy, odd in y
    const V m = L::mul(sh, L::add(sum(1, 0), dif(0, 1)));
    even1(1, 0, m);
    odd1(0, 1, m);
    const V a = dif(1, 0), b = sum(3, 2), t = L::mul(one_o, L::add(a, b));
    odd2(1, 0, L::fma(one_d, a, t));
    even1(3, 2, L::fma(one_d, b, t));
  }
  {   // shear xz, odd in z
    const V m = L::mul(sh, L::add(sum(2, 0), dif(0, 2)));
    even1(2, 0, m);
    odd1(0, 2, m);
    const V a = dif(2, 0), b = sum(3, 1), t = L::mul(one_o, L::add(a, b));
    odd2(2, 0, L::fma(one_d, a, t));
    even1(3, 1, L::fma(one_d, b, t));
  }
  {   // shear yz, odd in all
    const V m = L::mul(sh, L::add(sum(2, 1), sum(1, 2)));
    even1(2, 1, m);
    even1(1, 2, m);
    const V a = sum(3, 0), b = dif(2, 1), c = dif(1, 2);
    const V d = L::coef(W.w[kWhAllD], s), t = L::mul(L::coef(W.w[kWhAllO], s), L::add(L::add(a, b), c));
    even1(3, 0, L::fma(d, a, t));
    odd2(2, 1, L::fma(d, b, t));
    odd2(1, 2, L::fma(d, c, t));
  }
  {   // corner modes
    const V e = L::coef(W.w[kWhCo], s);
#pragma unroll
    for (int c = 0; c < 3; ++c) odd2(3, c, L::mul(e, dif(3, c)));
  }
}

// Voxel rows are dealt to the threads in blocks of 4 x 2, so that the 8 rows of a warp lie close together and
// more often are void at the same plane: rows j < 8, k < kSweepZ in blocks, then row k = kSweepZ, then
// column j = 8.
__device__ __forceinline__ int row_slot(int j, int k) {
  return j < 8 && k < kSweepZ ? 16 * (k >> 1) + 8 * (j >> 2) + 4 * (k & 1) + (j & 3)
                              : j < 8 ? 8 * kSweepZ + j : 8 * kSweepZ + 8 + k;
}
__device__ __forceinline__ void slot_row(int s, int& j, int& k) {
  if (s < 8 * kSweepZ) {
    j = (s & 3) + 4 * ((s >> 3) & 1);
    k = ((s >> 2) & 1) + 2 * (s >> 4);
  } else if (s < 8 * kSweepZ + 8) {
    j = s - 8 * kSweepZ;
    k = kSweepZ;
  } else {
    j = 8;
    k = s - 8 * kSweepZ - 8;
  }
}
static_assert(kSweepY == 8 && kSweepZ % 2 == 0, "the dealing of rows to threads");

enum { kSwApply = 0, kSwApplyDot = 1, kSwRes = 2, kSwPost = 3 };

// On the node rows of the listed tiles, len <= kSweepX nodes in x (interior nodes; ALL: every node of the grid):
//   kSwApply: y = scale K u;  kSwApplyDot: acc[dom][load case] += u . y as well
//   kSwRes  : y = b - K u
//   kSwPost : y = u + omega D^-1 (b - K u)
// Voxels outside the grid read as void, and only the corners of kept voxels are read.  Grid: (tile, group of 32
// bytes of load cases).  Node planes are staged through a ring in shared memory two steps ahead of
// their use (each value once per CTA, from four voxel rows), the voxel factors for the whole tile at the
// start, with a bit mask of the kept voxels per row that says who has work, what to stage and whose share
// a node row gets.  16 warps per SM (122 to 128 registers, none spilled).  A first form with register budgets for 18
// warps spilled, ended in an illegal memory access twice, for a cause not found, and was left out.
// Bound by instruction issue (49 %) and the barrier per plane, DRAM at 13 %.  Average over the launches of a
// solve of 64 domains of 32^3, against the node-centric sweeps that applied the 24 x 24 matrix: residual
// 361 -> 249 us, post-smoothing 375 -> 298, CG application 319 -> 224; FP64 application, 27 x 20^3,
// 116 -> 85.  Loading the planes into registers one step ahead took 278, 331 and 255 us.
template <typename T, bool ALL, int MODE>
__global__ void __launch_bounds__(kSweepThreads, 2) k_sweep(const Tile* __restrict__ tiles, int len,
                                                            const DomDev* __restrict__ doms,
                                                            const float* __restrict__ svox,
                                                            const __grid_constant__ Hadamard<T> W,
                                                            const T* __restrict__ u, T* __restrict__ y,
                                                            double scale, const float* __restrict__ binv,
                                                            const T* __restrict__ b, float omega,
                                                            double* __restrict__ acc,
                                                            const int* __restrict__ dom_active) {
  using L = Lane<T>;
  using V = typename L::V;
  constexpr int kGroups = kNLC / (4 * L::kCols);
  constexpr int kStep = kSweepX + 1;            // voxels of a row: x0 - 1 .. x0 + kSweepX - 1
  constexpr int kCopies = (kPlaneRows * 6 + kSweepThreads - 1) / kSweepThreads;   // 16-byte pieces of a plane
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  V* ring = reinterpret_cast<V*>(sweep_smem);   // kRing planes
  V* xch = ring + kRing * kPlaneElems;          // 2 x 9 x kSweepThreads: shares of the neighbours' node rows
  float* fac = reinterpret_cast<float*>(xch + 2 * 9 * kSweepThreads);   // [row][step]
  unsigned* kept_of = reinterpret_cast<unsigned*>(fac + kVoxRows * kStep);
  __shared__ unsigned kept_any;
  const Tile t = tiles[blockIdx.x / kGroups];
  if (dom_active && !dom_active[t.dom]) return;
  const DomDev D = doms[t.dom];
  const int tid = threadIdx.x, row = tid >> 2;
  int j, k;
  slot_row(row, j, k);
  const int lc0 = (blockIdx.x % kGroups) * (4 * L::kCols), lc = lc0 + (tid & 3) * L::kCols;
  const int vy = t.y0 - 1 + j, vz = t.z0 - 1 + k;   // voxel row; node row (vy, vz) is finished here
  const int hi = ALL ? 1 : 2;
  const int xe = min(D.n[0] - hi, t.x0 + len - 1);
  if (tid == 0) kept_any = 0;
  for (int e = tid; e < kVoxRows * kStep; e += kSweepThreads) {
    const int q = e / kStep, i = e % kStep;
    int jq, kq;
    slot_row(q, jq, kq);
    const int x = t.x0 - 1 + i, yy = t.y0 - 1 + jq, zz = t.z0 - 1 + kq;
    const bool in = i <= len && x >= 0 && yy >= 0 && zz >= 0 && x < D.L[0] && yy < D.L[1] && zz < D.L[2];
    const int64_t at = in ? x + (int64_t)D.L[0] * (yy + (int64_t)D.L[1] * zz) : 0;
    const float s = __ldg(svox + D.vox_off + at);
    fac[e] = in ? s : 0.f;
  }
  __syncthreads();
  unsigned kept = 0;   // bit i: voxel x0 - 1 + i of the row
  if (row < kVoxRows) {
#pragma unroll
    for (int i = 0; i < kStep; ++i) kept |= fac[row * kStep + i] != 0.f ? 1u << i : 0u;
    if ((tid & 3) == 0) {
      kept_of[row] = kept;
      if (kept) atomicOr(&kept_any, kept);
    }
  }
  __syncthreads();
  if (kept_any == 0) return;
  const bool node_row = row < kVoxRows && j > 0 && k > 0 && vy <= D.n[1] - hi && vz <= D.n[2] - hi;
  // voxel rows whose shares complete the node row: their exchange places (a byte each) and kept voxels
  const int ny = node_row ? row_slot(j - 1, k) : 0, nz = node_row ? row_slot(j, k - 1) : 0,
            nyz = node_row ? row_slot(j - 1, k - 1) : 0;
  const unsigned from = (4 * ny + (tid & 3)) | (4 * nz + (tid & 3)) << 8 | (4 * nyz + (tid & 3)) << 16;
  const unsigned ky = node_row ? kept_of[ny] : 0, kz = node_row ? kept_of[nz] : 0, kyz = node_row ? kept_of[nyz] : 0;
  // node of the row at plane x0 - 1 inside the domain, and the domain's first value of the load case
  const int node0 = t.x0 - 1 + (node_row ? D.n[0] * (vy + D.n[1] * vz) : 0);
  const int64_t first = vec_index(D.node_off, 0, lc);
  const int steps = xe - t.x0 + 2;
  // this thread's 16-byte pieces of every staged plane, and the planes at which a kept voxel reads them
  const T* csrc[kCopies];
  unsigned cneed[kCopies];
#pragma unroll
  for (int m = 0; m < kCopies; ++m) {
    const int e = tid + m * kSweepThreads, r = e / 6, part = e % 6, jn = r % kPlaneY, kn = r / kPlaneY;
    cneed[m] = 0;
    csrc[m] = u;
    if (r < kPlaneRows) {
      unsigned n = 0;   // the voxel rows (jn - 1 .. jn, kn - 1 .. kn) around node row (jn, kn)
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int jv = jn - (a & 1), kv = kn - (a >> 1);
        if (jv >= 0 && kv >= 0 && jv < kVoxRowsY && kv < kVoxRowsZ) n |= kept_of[row_slot(jv, kv)];
      }
      cneed[m] = n | n << 1;
      if (n) {
        const int node = t.x0 - 1 + D.n[0] * (t.y0 - 1 + jn + D.n[1] * (t.z0 - 1 + kn));
        csrc[m] = u + vec_index(D.node_off + node, part >> 1, lc0) + (part & 1) * (2 * L::kCols);
      }
    }
  }
  auto stage = [&](int plane) {   // plane x0 - 1 + plane into its place of the ring
#pragma unroll
    for (int m = 0; m < kCopies; ++m)
      if ((cneed[m] >> plane) & 1)
        copy16(ring + (plane % kRing) * kPlaneElems + 2 * (tid + m * kSweepThreads), csrc[m] + (int64_t)plane * (3 * kNLC));
    copy_commit();
  };
#pragma unroll
  for (int i = 0; i < kRing - 1; ++i) stage(i);
  copy_wait<kRing - 3>();
  __syncthreads();
  // corner (0, 0) of the voxel row, which is node row (vy, vz), inside a staged plane
  const int corner = (j + kPlaneY * k) * 12 + (tid & 3);
  V p[4][3], f[4][3];   // transformed plane x, force on it from the voxel before
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 3; ++c) p[a][c] = f[a][c] = L::zero();
  if (kept & 1) wh_plane<T>(ring + corner, p);
  double dot[L::kCols] = {};
  int slot = 0;         // of plane x in the ring
#pragma unroll 2
  for (int i = 0; i < steps; ++i) {             // plane x = x0 - 1 + i
    const int64_t k0 = first + (int64_t)(node0 + i) * (3 * kNLC);   // the node row at plane x
    const bool done = node_row && i > 0 && (((kept | ky | kz | kyz) >> (i - 1)) & 3);
    V bv[3];
    if (done && (MODE == kSwRes || MODE == kSwPost)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) bv[c] = L::load(b + k0 + c * kNLC);
    }
    const int next = slot + 1 == kRing ? 0 : slot + 1;
    V q[4][3], g[4][3];                         // q holds nothing where no voxel needs it
    if ((kept >> i) & 3) wh_plane<T>(ring + next * kPlaneElems + corner, q);   // plane x + 1
    if ((kept >> i) & 1) {
      wh_voxel<T>(p, q, W, fac[row * kStep + i], f, g);
    } else {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) g[a][c] = L::zero();
    }
    V v[3];
    V* xc = xch + (i & 1) * (9 * kSweepThreads);
    if (i > 0 && ((kept >> (i - 1)) & 3)) {     // back to the four node rows
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const V u0 = L::sub(f[0][c], f[2][c]), u1 = L::add(f[0][c], f[2][c]);
        const V w0 = L::sub(f[1][c], f[3][c]), w1 = L::add(f[1][c], f[3][c]);
        v[c] = L::sub(u0, w0);
        xc[c * kSweepThreads + tid] = L::add(u0, w0);
        xc[(3 + c) * kSweepThreads + tid] = L::sub(u1, w1);
        xc[(6 + c) * kSweepThreads + tid] = L::add(u1, w1);
      }
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = L::zero();
    }
    copy_wait<1>();                             // plane x + 2 has landed
    __syncthreads();
    if (i + kRing - 1 <= steps) stage(i + kRing - 1);
    else copy_commit();
    if (done) {
      V uv[3];
      if constexpr (MODE == kSwPost || MODE == kSwApplyDot) {
#pragma unroll
        for (int c = 0; c < 3; ++c) uv[c] = ring[slot * kPlaneElems + corner + 4 * c];
      }
      const typename L::Scale sc(scale * D.scale);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if ((ky >> (i - 1)) & 3) v[c] = L::add(v[c], xc[c * kSweepThreads + (from & 255)]);
        if ((kz >> (i - 1)) & 3) v[c] = L::add(v[c], xc[(3 + c) * kSweepThreads + ((from >> 8) & 255)]);
        if ((kyz >> (i - 1)) & 3) v[c] = L::add(v[c], xc[(6 + c) * kSweepThreads + (from >> 16)]);
        v[c] = sc(v[c]);
      }
      if constexpr (MODE == kSwRes || MODE == kSwPost) {
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = L::sub(bv[c], v[c]);
      }
      if constexpr (MODE == kSwPost) {
        const float* bi = binv + (D.node_off + node0 + i) * 6;
        const float b0 = omega * __ldg(bi), b1 = omega * __ldg(bi + 1), b2 = omega * __ldg(bi + 2);
        const float b3 = omega * __ldg(bi + 3), b4 = omega * __ldg(bi + 4), b5 = omega * __ldg(bi + 5);
        const V c00 = make_float2(b0, b0), c11 = make_float2(b1, b1), c22 = make_float2(b2, b2);
        const V c01 = make_float2(b3, b3), c02 = make_float2(b4, b4), c12 = make_float2(b5, b5);
        const V z0 = L::fma(c00, v[0], L::fma(c01, v[1], L::fma(c02, v[2], uv[0])));
        const V z1 = L::fma(c01, v[0], L::fma(c11, v[1], L::fma(c12, v[2], uv[1])));
        const V z2 = L::fma(c02, v[0], L::fma(c12, v[1], L::fma(c22, v[2], uv[2])));
        v[0] = z0;
        v[1] = z1;
        v[2] = z2;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) L::store(y + k0 + c * kNLC, v[c]);
      if constexpr (MODE == kSwApplyDot) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if constexpr (L::kCols == 2) {
            dot[0] += (double)uv[c].x * (double)v[c].x;
            dot[1] += (double)uv[c].y * (double)v[c].y;
          } else {
            dot[0] = fma(uv[c], v[c], dot[0]);
          }
        }
      }
    }
    slot = next;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 3; ++c) { p[a][c] = q[a][c]; f[a][c] = g[a][c]; }
  }
  if constexpr (MODE == kSwApplyDot) {
    // lanes with equal (lane & 3) carry the same load cases
    __shared__ double red[kSweepThreads / 32][4][L::kCols];
#pragma unroll
    for (int i = 0; i < L::kCols; ++i) {
      double v = dot[i];
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if ((tid & 31) < 4) red[tid >> 5][tid & 3][i] = v;
    }
    __syncthreads();
    if (tid < 4)
#pragma unroll
      for (int i = 0; i < L::kCols; ++i) {
        double v = 0.0;
        for (int w = 0; w < kSweepThreads / 32; ++w) v += red[w][tid][i];
        atomicAdd(acc + (int64_t)t.dom * kNLC + lc + i, v);
      }
  }
}

constexpr int kSweepSmem = (kRing * kPlaneElems + 2 * 9 * kSweepThreads) * 8 +
                           (kVoxRows * (kSweepX + 1) + kVoxRows) * 4;

}  // namespace dtc
