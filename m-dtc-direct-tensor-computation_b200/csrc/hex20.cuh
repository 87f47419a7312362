// hex20.cuh -- HEX20 stiffness application in the voxel's reflection classes.
//
// A cubic voxel's element matrix commutes with the reflections of the three axes.  Signed sums of the
// displacements over the 8 corners and over the 4 mid-edge nodes of each direction, which transforms of
// 2 x 2 x 2 and 2 x 2 points give, therefore split the 60 x 60 matrix into blocks of 9, 8, 8, 8, 7, 7, 7 and 6:
// 456 products and 288 additions in place of 3600 products per voxel and load case.
//
// One CTA owns a column of kColX x kColY voxels' worth of nodes (the nodes whose coordinate divided by 2 is in
// the column) for 32 bytes of load cases and walks it along z.  A thread keeps one voxel of the layer, halo on
// the low sides included, and 8 bytes of load cases.  Per layer it reads the voxel's 20 nodes from
// shared memory, where the nodes of the next layer arrive meanwhile (a ring of three layers filled by
// cp.async), applies the matrix in registers, and puts what its lower and middle nodes receive into shared
// memory; what the upper nodes receive stays in registers for the next layer.  Then every owned node is summed
// over its voxels and written once, without atomics.
#pragma once
#include <algorithm>
#include <cmath>

namespace dtc {

// HEX20 ring-order node offsets on the doubled grid (mod_gen_quadmesh.f90:244-265)
__host__ __device__ constexpr int ring_off(int a, int d) {
  return "000100200210220120020010001201"
         "221021002102202212222122022012"[3 * a + d] - '0';
}

template <int NEN> struct Elem;
template <> struct Elem<8> {
  static constexpr int M = 1, ND = 24;
  __host__ __device__ static constexpr int off(int a, int d) {
    return d == 0 ? ((a & 3) == 1 || (a & 3) == 2) : (d == 1 ? ((a & 3) >= 2) : (a >= 4));
  }
};
template <> struct Elem<20> {
  static constexpr int M = 2, ND = 60;
  __host__ __device__ static constexpr int off(int a, int d) { return ring_off(a, d); }
};

// A voxel's 60 values, before the transforms by position (bit d of a corner: its side along axis d), after them
// by parity: corners c * 8 + (x + 2 y + 4 z), x-edges 24 + c * 4 + (y + 2 z), y-edges 36 + c * 4 + (x + 2 z),
// z-edges 48 + c * 4 + (x + 2 y).  Class p holds the component c at parity p ^ (1 << c).
__host__ __device__ constexpr int class_size(int p) { return 9 - ((p & 1) + (p >> 1 & 1) + (p >> 2 & 1)); }
__host__ __device__ constexpr int class_offset(int p) {   // of its packed lower triangle
  int o = 0;
  for (int q = 0; q < p; ++q) o += class_size(q) * (class_size(q) + 1) / 2;
  return o;
}
constexpr int kClassEntries = class_offset(8);
__host__ __device__ constexpr int class_mode(int p, int i) {
  int k = 0;
  for (int c = 0; c < 3; ++c) {
    const int h = p ^ (1 << c), x = h & 1, y = h >> 1 & 1, z = h >> 2;
    if (k++ == i) return c * 8 + h;
    if (!x && k++ == i) return 24 + c * 4 + y + 2 * z;
    if (!y && k++ == i) return 36 + c * 4 + x + 2 * z;
    if (!z && k++ == i) return 48 + c * 4 + x + 2 * y;
  }
  return -1;
}

// The class blocks of a unit element matrix, divided by the squared lengths of the signed sums.  A translation along c
// is the vector (2, 1, 1, 1) on the four modes of class 1 << c that hold the component c (2 c on: the corners, then
// the edges along x, y and z), and the blocks hold exactly 0 for it: the entries of these columns are rounded to
// a grid of half their last place, coarse enough for the corner column to follow from the edges' without rounding.
// An entry off by one rounding acts as a spring to the ground whose energy is counted in every voxel with the square of
// the voxel's distance from the middle of the domain: on 24^3 the macro stiffness of rigid translations was 4e-12 of
// its largest entry, tensors were 2.8e-12 off, and FP32 solves of weakly connected bone stopped 1.1e-9 off.
template <typename T> struct ClassBlocks { T k[kClassEntries]; };
template <> struct ClassBlocks<float> { float2 k[kClassEntries]; };   // twice: an operand of packed arithmetic
inline void set_entry(double& e, long double v) { e = (double)v; }
inline void set_entry(float2& e, long double v) { e = make_float2((float)v, (float)v); }

template <typename T>
ClassBlocks<T> class_blocks(const double* k20) {
  double sign[60][60] = {};   // mode, DOF 3 * node + c
  double inv[60];
  for (int m = 0; m < 60; ++m) {
    const int set = m < 24 ? 0 : m < 36 ? 1 : m < 48 ? 2 : 3;
    const int c = set == 0 ? m / 8 : (m - 24) % 12 / 4, h = set == 0 ? m % 8 : (m - 24) % 4;
    inv[m] = set == 0 ? 0.125 : 0.25;
    for (int a = 0; a < 20; ++a) {
      const int o[3] = {ring_off(a, 0), ring_off(a, 1), ring_off(a, 2)};
      const int odd = (o[0] == 1) + (o[1] == 1) + (o[2] == 1);
      if (set == 0 ? odd != 0 : o[set - 1] != 1) continue;
      int bits = 0, k = 0;
      for (int d = 0; d < 3; ++d)
        if (d != set - 1) bits |= (o[d] / 2) << k++;
      int par = bits & h;
      par ^= par >> 2;
      par ^= par >> 1;
      sign[m][3 * a + c] = par & 1 ? -1.0 : 1.0;
    }
  }
  ClassBlocks<T> B;
  constexpr int kBits = sizeof(T) == 8 ? 53 : 24;
  for (int p = 0; p < 8; ++p) {
    const int n = class_size(p);
    long double m[9][9];
    for (int i = 0; i < n; ++i)
      for (int j = 0; j <= i; ++j) {
        const int mi = class_mode(p, i), mj = class_mode(p, j);
        long double v = 0;
        for (int a = 0; a < 60; ++a)
          if (sign[mi][a] != 0)
            for (int b = 0; b < 60; ++b) v += (long double)(sign[mi][a] * sign[mj][b]) * k20[a + 60 * b];
        m[i][j] = m[j][i] = v * inv[mi] * inv[mj];
      }
    const int c = p == 1 ? 0 : p == 2 ? 1 : p == 4 ? 2 : -1, q = 2 * c;
    if (c >= 0) {   // the class holds a translation
      auto last_place = [](long double v) { return std::ldexp(1.0L, std::ilogb(v) + 1 - kBits); };
      // the edges' own block first, on one grid: its sums give the corner's row and column, their sum its diagonal entry
      long double most = std::fabs(m[q][q]);
      for (int i = q; i <= q + 3; ++i)
        for (int k = q; k <= q + 3; ++k) most = std::max(most, std::fabs(m[i][k]));
      const long double grid = 4 * last_place(most);
      long double total = 0;
      for (int i = q + 1; i <= q + 3; ++i) {
        long double sum = 0;
        for (int k = q + 1; k <= q + 3; ++k) sum += m[i][k] = std::nearbyint(m[i][k] / grid) * grid;
        m[i][q] = m[q][i] = -sum / 2;
        total += sum;
      }
      m[q][q] = total / 4;
      for (int i = 0; i < n; ++i) {
        if (i >= q && i <= q + 3) continue;
        most = std::fabs(m[i][q]);
        for (int k = q + 1; k <= q + 3; ++k) most = std::max(most, std::fabs(m[i][k]));
        if (!(most > 0)) continue;
        const long double g = 2 * last_place(most);
        long double sum = 0;
        for (int k = q + 1; k <= q + 3; ++k) sum += m[k][i] = m[i][k] = std::nearbyint(m[i][k] / g) * g;
        m[i][q] = m[q][i] = -sum / 2;
      }
    }
    for (int i = 0; i < n; ++i)
      for (int j = 0; j <= i; ++j) set_entry(B.k[class_offset(p) + i * (i + 1) / 2 + j], m[i][j]);
  }
  return B;
}

constexpr int kColX = 8, kColY = 6;                        // voxels of a column
constexpr int kColVox = (kColX + 1) * (kColY + 1);         // with the halo on the low sides
constexpr int kColPos = (kColX + 2) * (kColY + 2);         // corner positions of these voxels
constexpr int kColWords = 4;                               // threads per voxel
constexpr int kColThreads = 256;
constexpr int kColIn = 12 * kColPos * kColWords;           // 8-byte words of a layer of nodes
constexpr int kColOut = 36 * kColVox * kColWords;
constexpr int kColSmem = 8 * (3 * kColIn + kColOut);
static_assert(kColVox * kColWords <= kColThreads, "a thread per voxel and word");
static_assert(12 * kColX * kColY * kColWords % kColThreads == 0, "the owned nodes divide evenly");

// 8 bytes of load cases
template <typename T> struct ColLane;
template <> struct ColLane<float> {
  using V = float2;
  static constexpr int kCols = 2;
  static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
  static __device__ __forceinline__ V mul(V k, V a) { return __fmul2_rn(k, a); }
  static __device__ __forceinline__ V fma(V k, V a, V c) { return __ffma2_rn(k, a, c); }
  static __device__ __forceinline__ V all(float s) { return make_float2(s, s); }
  static __device__ __forceinline__ void pin(V& a) { asm volatile("" : "+f"(a.x), "+f"(a.y)); }
  static __device__ __forceinline__ V scaled(double s, V a) {
    return make_float2((float)(s * (double)a.x), (float)(s * (double)a.y));
  }
  static __device__ __forceinline__ void dot(V a, V b, double (&d)[2]) {
    d[0] += (double)a.x * (double)b.x;
    d[1] += (double)a.y * (double)b.y;
  }
};
template <> struct ColLane<double> {
  using V = double;
  static constexpr int kCols = 1;
  static __device__ __forceinline__ V zero() { return 0.0; }
  static __device__ __forceinline__ V add(V a, V b) { return a + b; }
  static __device__ __forceinline__ V sub(V a, V b) { return a - b; }
  static __device__ __forceinline__ V mul(double k, V a) { return k * a; }
  static __device__ __forceinline__ V all(float s) { return (double)s; }
  static __device__ __forceinline__ V fma(double k, V a, V c) { return ::fma(k, a, c); }
  static __device__ __forceinline__ void pin(V& a) { asm volatile("" : "+d"(a)); }
  static __device__ __forceinline__ V scaled(double s, V a) { return s * a; }
  static __device__ __forceinline__ void dot(V a, V b, double (&d)[1]) { d[0] += a * b; }
};

// Sums and differences along each axis, in place; the inverse up to the factor in the blocks.
template <typename T>
__device__ __forceinline__ void col_transform(typename ColLane<T>::V (&v)[60]) {
  using Op = ColLane<T>;
  auto pair = [](typename Op::V& a, typename Op::V& b) {
    const typename Op::V s = Op::add(a, b);
    b = Op::sub(a, b);
    a = s;
  };
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & 1)) pair(v[c * 8 + i], v[c * 8 + i + 1]);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & 2)) pair(v[c * 8 + i], v[c * 8 + i + 2]);
#pragma unroll
    for (int i = 0; i < 4; ++i) pair(v[c * 8 + i], v[c * 8 + i + 4]);
#pragma unroll
    for (int e = 24 + 4 * c; e < 60; e += 12) {
      pair(v[e], v[e + 1]);
      pair(v[e + 2], v[e + 3]);
      pair(v[e], v[e + 2]);
      pair(v[e + 1], v[e + 3]);
    }
  }
}

template <typename T, int P>
__device__ __forceinline__ void col_class(const ClassBlocks<T>& B, typename ColLane<T>::V s, typename ColLane<T>::V (&v)[60]) {
  using Op = ColLane<T>;
  constexpr int N = class_size(P), O = class_offset(P);
  typename Op::V r[N];
#pragma unroll
  for (int i = 0; i < N; ++i) Op::pin(v[class_mode(P, i)]);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    r[i] = Op::mul(B.k[O + i * (i + 1) / 2], v[class_mode(P, 0)]);
#pragma unroll
    for (int j = 1; j < N; ++j)
      r[i] = Op::fma(B.k[O + (i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i)], v[class_mode(P, j)], r[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    v[class_mode(P, i)] = Op::mul(s, r[i]);
    Op::pin(v[class_mode(P, i)]);
  }
}

// y = scale * K u on the owned nodes of a column of `layers` voxel layers from (t.x0, t.y0, t.z0); ALL: every
// grid node, else the interior nodes (the unknowns); DOT: acc[col] += u . y.
// Bound in turn by the FP32 pipe (1608 of 7000 cycles a layer and warp, two warps a scheduler), shared memory
// (2800) and the latency between the two barriers of a layer: the registers (all 255) leave one CTA to an SM.
// 16 domains of 24^3 at BV/TV 0.25, FP32: 374 us, 15 to 17 TFLOP/s of the dense matrix's operations; an
// element-by-element kernel with the 60 x 60 matrix in shared memory and shared atomics took 940.  One load case
// per thread (512 threads of 128 registers) took 418.
template <typename T, bool ALL, bool DOT>
__global__ void __launch_bounds__(kColThreads, 1)
    k_hex20(const Tile* __restrict__ tiles, int layers, const DomDev* __restrict__ doms,
            const float* __restrict__ svox, const uint8_t* __restrict__ flags,
            const __grid_constant__ ClassBlocks<T> B, const T* __restrict__ u, T* __restrict__ y, double scale,
            double* __restrict__ acc, const int* __restrict__ dom_active) {
  using Op = ColLane<T>;
  using V = typename Op::V;
  constexpr int W = kColWords, LC = W * Op::kCols, GROUPS = kNLC / LC, NT = kColThreads;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* in = reinterpret_cast<V*>(smem_raw);          // [3][12][kColPos][W]
  V* out = in + 3 * kColIn;                        // [36][kColVox][W]
  __shared__ uint8_t write[4 * kColX * kColY];     // the node is written
  __shared__ double red[LC];

  const Tile t = tiles[blockIdx.x / GROUPS];
  if (dom_active && !dom_active[t.dom]) return;
  const DomDev& D = doms[t.dom];
  const int n0 = D.n[0], n1 = D.n[1], n2 = D.n[2], lc0 = (int)(blockIdx.x % GROUPS) * LC;
  const int64_t node_off = D.node_off;
  const int lo = ALL ? 0 : 1, hx = n0 - 1 - lo, hy = n1 - 1 - lo, hz = n2 - 1 - lo;
  const int k0 = t.z0 > 0 ? t.z0 - 1 : 0;
  const int k1 = min(t.z0 + layers, hz / 2 + 1);   // owned layers end here
  const int tid = threadIdx.x;
  const double total = scale * D.scale;
  if (DOT && tid < LC) red[tid] = 0.0;

  // the nodes 2 k and 2 k + 1 of the column's positions, zero outside the grid
  auto fetch = [&](int k) {
    unsigned char* dst = reinterpret_cast<unsigned char*>(in + k % 3 * kColIn);
    int me = tid;
    asm volatile("" : "+r"(me));
#pragma unroll 4
    for (int i = me; i < kColIn / 2; i += NT) {   // 16 bytes each
      const int half = i % 2, pos = i / 2 % kColPos, nc = i / (2 * kColPos), type = nc / 3, c = nc % 3;
      const int gx = 2 * (t.x0 - 1 + pos % (kColX + 2)) + (type == 1);
      const int gy = 2 * (t.y0 - 1 + pos / (kColX + 2)) + (type == 2), gz = 2 * k + (type == 3);
      if (gx >= 0 && gy >= 0 && gx < n0 && gy < n1 && gz < n2)
        copy16(dst + 16 * i, u + vec_index(node_off + gx + (int64_t)n0 * (gy + (int64_t)n1 * gz), c, lc0 + half * LC / 2));
      else
        *reinterpret_cast<float4*>(dst + 16 * i) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  // the thread's voxel
  const int word = tid % W, vox = tid / W, px = vox % (kColX + 1), py = vox / (kColX + 1);
  const int vx = t.x0 - 1 + px, vy = t.y0 - 1 + py;
  const bool column = vox < kColVox && vx >= 0 && vy >= 0 && vx < D.L[0] && vy < D.L[1];
  const float* sv = svox + D.vox_off + vx + (int64_t)D.L[0] * vy;
  const int64_t sz = (int64_t)D.L[0] * D.L[1];
  auto factor = [&](int k) { return column && k < D.L[2] ? __ldg(sv + sz * k) : 0.f; };
  // the node whose flag the thread looks up
  const int ftype = tid % 4, fcol = tid / 4;
  const int fx = 2 * (t.x0 + fcol % kColX) + (ftype == 1), fy = 2 * (t.y0 + fcol / kColX) + (ftype == 2);
  const bool fin = fcol < kColX * kColY && fx >= lo && fx <= hx && fy >= lo && fy <= hy;

  V carry[24];
#pragma unroll
  for (int i = 0; i < 24; ++i) carry[i] = Op::zero();
  double dots[Op::kCols] = {};
  fetch(k0);
  fetch(k0 + 1);
  copy_commit();
  float s = factor(k0);
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    copy_wait<0>();
    __syncthreads();
    if (k + 1 < k1) fetch(k + 2);
    copy_commit();
    const float s_next = factor(k + 1);
    const int fz = 2 * k + (ftype == 3);
    uint8_t flag = 0;
    if (fin && fz >= lo && fz <= hz) flag = __ldg(flags + node_off + fx + (int64_t)n0 * (fy + (int64_t)n1 * fz)) & kNodeActive;
    if (vox < kColVox) {
      V* o = out + tid;
      if (s != 0.f) {
        V v[60];
        const V* a = in + k % 3 * kColIn + (px + (kColX + 2) * py) * W + word;
        const V* b = in + (k + 1) % 3 * kColIn + (px + (kColX + 2) * py) * W + word;
        auto at = [&](const V* q, int type, int c, int x, int yy) {
          return q[((type * 3 + c) * kColPos + x + (kColX + 2) * yy) * W];
        };
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[c * 8 + i] = at(i & 4 ? b : a, 0, c, i & 1, i >> 1 & 1);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            v[24 + c * 4 + i] = at(i & 2 ? b : a, 1, c, 0, i & 1);
            v[36 + c * 4 + i] = at(i & 2 ? b : a, 2, c, i & 1, 0);
            v[48 + c * 4 + i] = at(a, 3, c, i & 1, i >> 1);
          }
        }
        col_transform<T>(v);
        const V sv2 = Op::all(s);
        col_class<T, 0>(B, sv2, v);
        col_class<T, 1>(B, sv2, v);
        col_class<T, 2>(B, sv2, v);
        col_class<T, 3>(B, sv2, v);
        col_class<T, 4>(B, sv2, v);
        col_class<T, 5>(B, sv2, v);
        col_class<T, 6>(B, sv2, v);
        col_class<T, 7>(B, sv2, v);
        col_transform<T>(v);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            o[(c * 4 + i) * kColVox * W] = Op::add(carry[c * 4 + i], v[c * 8 + i]);
            carry[c * 4 + i] = v[c * 8 + 4 + i];
            o[(24 + c * 4 + i) * kColVox * W] = v[48 + c * 4 + i];
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            o[(12 + c * 2 + i) * kColVox * W] = Op::add(carry[12 + c * 2 + i], v[24 + c * 4 + i]);
            carry[12 + c * 2 + i] = v[24 + c * 4 + 2 + i];
            o[(18 + c * 2 + i) * kColVox * W] = Op::add(carry[18 + c * 2 + i], v[36 + c * 4 + i]);
            carry[18 + c * 2 + i] = v[36 + c * 4 + 2 + i];
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 24; ++i) {
          o[i * kColVox * W] = carry[i];
          carry[i] = Op::zero();
        }
#pragma unroll
        for (int i = 24; i < 36; ++i) o[i * kColVox * W] = Op::zero();
      }
    }
    s = s_next;
    if (tid < 4 * kColX * kColY) write[tid] = flag;
    __syncthreads();
    if (k < t.z0) continue;
    // sum every owned node over its voxels and write it
    int me = tid;
    asm volatile("" : "+r"(me));   // what follows from the thread's number is formed again per layer, not kept
    const V* from = in + k % 3 * kColIn;
#pragma unroll 3
    for (int j = 0; j < 12 * kColX * kColY * W / NT; ++j) {
      const int i = me + j * NT, nc = i / (W * kColX * kColY), type = nc / 3, c = nc % 3;
      const int col = i / W % (kColX * kColY), cx = col % kColX, cy = col / kColX;
      if (!write[4 * col + type]) continue;
      const V* q = out + ((cx + 1) + (kColX + 1) * (cy + 1)) * W + word;   // the voxel on the node's high sides
      constexpr int X = W, Y = (kColX + 1) * W, O = kColVox * W;
      V r;
      if (type == 0 || type == 3) {
        const V* e = q + ((type == 0 ? 0 : 24) + c * 4) * O;
        r = Op::add(Op::add(e[0], e[O - X]), Op::add(e[2 * O - Y], e[3 * O - X - Y]));
      } else if (type == 1) {
        const V* e = q + (12 + c * 2) * O;
        r = Op::add(e[0], e[O - Y]);
      } else {
        const V* e = q + (18 + c * 2) * O;
        r = Op::add(e[0], e[O - X]);
      }
      const V v = Op::scaled(total, r);
      const int gx = 2 * (t.x0 + cx) + (type == 1), gy = 2 * (t.y0 + cy) + (type == 2), gz = 2 * k + (type == 3);
      *reinterpret_cast<V*>(y + vec_index(node_off + gx + (int64_t)n0 * (gy + (int64_t)n1 * gz), c,
                                          lc0 + word * Op::kCols)) = v;
      if (DOT) Op::dot(from[(nc * kColPos + (cx + 1) + (kColX + 2) * (cy + 1)) * W + word], v, dots);
    }
  }
  copy_wait<0>();
  if (DOT) {
    __syncthreads();
#pragma unroll
    for (int l = 0; l < Op::kCols; ++l) atomicAdd(&red[word * Op::kCols + l], dots[l]);
    __syncthreads();
    if (tid < LC) atomicAdd(acc + (int64_t)t.dom * kNLC + lc0 + tid, red[tid]);
  }
}

}  // namespace dtc
