// Finite-difference stencils on complex and padded real grids.
//
// Boundary values follow the reference's value_outside functions
// (src/cgrid_bc.c:21-86, src/rgrid_bc.c:19-74): Dirichlet returns a constant
// (the grid's outside parameter, 0 by default), Neumann mirrors i -> -i and
// i -> 2n - i - 2, periodic wraps.  On an axis of length 1 the Neumann mirror
// lands outside the grid again (the reference recurses without end there);
// this implementation uses the single plane instead.
//
// Stencils read their neighbours directly, two or four output elements per thread
// with their loads issued together (k_fd below).  Laplacian sums keep the reference's left-to-right
// order
//   (-6 c + z+ + z- + y+ + y- + x+ + x-) / h^2     (src/cgrid_diff.c:330-335).
#include <string.h>

#include <algorithm>

#include "gb_common.cuh"
#include "gb_internal_cuda.h"

namespace {

template <typename T, bool REAL> struct Elem;
template <typename T> struct Elem<T, false> {
  using V = C2<T>;
  static __device__ __forceinline__ V zero() { return V{(T) 0, (T) 0}; }
  static __device__ __forceinline__ V outside(double re, double im) { return V{(T) re, (T) im}; }
  static __device__ __forceinline__ V add(V a, V b) { return cadd(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return csub(a, b); }
  static __device__ __forceinline__ V scale(V a, T s) { return cscale(a, s); }
};
template <typename T> struct Elem<T, true> {
  using V = T;
  static __device__ __forceinline__ V zero() { return (T) 0; }
  static __device__ __forceinline__ V outside(double re, double) { return (T) re; }
  static __device__ __forceinline__ V add(V a, V b) { return a + b; }
  static __device__ __forceinline__ V sub(V a, V b) { return a - b; }
  static __device__ __forceinline__ V scale(V a, T s) { return a * s; }
};

struct FdArgs {
  long nx, ny, nz, row;  // row = elements per (i, j) row of the storage
  int bc;
  double out_re, out_im;
  double coef;
};

// Map a possibly out-of-range index on one axis; returns false for
// "Dirichlet outside".
__device__ __forceinline__ bool map_index(long &i, long n, int bc) {
  if (i >= 0 && i < n) return true;
  if (bc == GB_BC_DIRICHLET) return false;
  if (bc == GB_BC_PERIODIC) {
    i %= n;
    if (i < 0) i += n;
    return true;
  }
  // Neumann mirror (src/cgrid_bc.c:45-57)
  if (i < 0) i = -i;
  if (i > n - 1) i = 2 * n - i - 2;
  if (i < 0 || i >= n) i = 0;  // axis of length 1
  return true;
}

template <typename T>
__device__ __forceinline__ C2<T> fetch(const C2<T> *src, long i, long j, long k, const FdArgs &a) {
  using E = Elem<T, false>;
  if (i < 0 || i >= a.nx || j < 0 || j >= a.ny || k < 0 || k >= a.nz) {
    if (a.bc == GB_BC_DIRICHLET) return E::outside(a.out_re, a.out_im);
    // Neumann/periodic remap all three indices like the reference does
    if (!map_index(i, a.nx, a.bc) || !map_index(j, a.ny, a.bc) || !map_index(k, a.nz, a.bc))
      return E::outside(a.out_re, a.out_im);
  }
  return src[(i * a.ny + j) * a.row + k];
}

// Direct stencils.  Bound by memory: a CTA takes kFdThreads * U consecutive
// elements, a thread U of them kFdThreads apart with their loads issued
// together.  A chunk's row and plane neighbours are the chunk itself, its edge
// rows and two planes nearby, so DRAM sees each element about once.  Halo tiles
// marched along x (k_fd_kinetic below keeps them) hold two planes of a column
// in flight and meet at a CTA barrier once per plane.  Tiles / direct, FP64, in
// microseconds: complex gradients 150 / 81 at 256^3, 46 / 17 at 200 x 150 x
// 101, 16.7 / 5.4 at 64^3; complex Laplacian 152 / 135, 48.7 / 28.3, 17.5 /
// 5.5; real Laplacian 118 / 83, 37 / 19, 14.6 / 5.1.  Not kept: the boundary as
// an index select instead of a branch (complex Laplacian at 256^3 167), chunks
// of two planes (138, real 117).
constexpr int kFdThreads = 256;

// The axis neighbour of element idx at coordinate c of an axis of n points
// with element stride s: in range at once, else by the boundary rule
// (src/cgrid_bc.c:21-86).  A Neumann axis of length 1 uses its single plane.
template <int DIR, typename T, bool REAL, typename I>
__device__ __forceinline__ typename Elem<T, REAL>::V neighbour(const typename Elem<T, REAL>::V *__restrict__ src, I idx,
                                                               I c, I n, I s, const FdArgs &a) {
  const bool in = DIR > 0 ? c + 1 < n : c > 0;
  if (in) return src[DIR > 0 ? idx + s : idx - s];
  if (a.bc == GB_BC_DIRICHLET) return Elem<T, REAL>::outside(a.out_re, a.out_im);
  I m;  // the coordinate that stands for the outside one
  if (a.bc == GB_BC_PERIODIC) m = DIR > 0 ? 0 : n - 1;
  else m = n == 1 ? 0 : DIR > 0 ? n - 2 : 1;
  return src[idx - c * s + m * s];
}

// Element e of the grid's nx * ny * nz points: its storage index (both below
// 2^31) and its neighbours along the axes that MODE takes (0, 1, 2: x, y, z; 3: all, in the
// order z+, z-, y+, y-, x+, x-).
template <typename T, bool REAL, int MODE, typename I>
__device__ __forceinline__ I fd_load(typename Elem<T, REAL>::V (&nb)[MODE == 3 ? 6 : 2],
                                     const typename Elem<T, REAL>::V *__restrict__ src, I e, const FdArgs &a) {
  constexpr int Y = MODE == 3 ? 2 : 0, X = MODE == 3 ? 4 : 0;
  const I nz = (I) a.nz, ny = (I) a.ny, r = e / nz, k = e - r * nz, i = r / ny, j = r - i * ny;
  const I sy = (I) a.row, sx = (I) a.ny * (I) a.row, idx = r * sy + k;
  if constexpr (MODE >= 2) {
    nb[0] = neighbour<1, T, REAL, I>(src, idx, k, nz, (I) 1, a);
    nb[1] = neighbour<-1, T, REAL, I>(src, idx, k, nz, (I) 1, a);
  }
  if constexpr (MODE == 1 || MODE == 3) {
    nb[Y] = neighbour<1, T, REAL, I>(src, idx, j, ny, sy, a);
    nb[Y + 1] = neighbour<-1, T, REAL, I>(src, idx, j, ny, sy, a);
  }
  if constexpr (MODE == 0 || MODE == 3) {
    nb[X] = neighbour<1, T, REAL, I>(src, idx, i, (I) a.nx, sx, a);
    nb[X + 1] = neighbour<-1, T, REAL, I>(src, idx, i, (I) a.nx, sx, a);
  }
  return idx;
}

__host__ __device__ constexpr int fd_unroll(int mode) { return mode == 3 ? 2 : 4; }

// MODE 0, 1, 2: second difference (lap) or central difference along x, y, z;
// MODE 3: the seven-point Laplacian.
template <typename T, bool REAL, int MODE>
__global__ void __launch_bounds__(kFdThreads) k_fd(bool lap, typename Elem<T, REAL>::V *__restrict__ dst,
                                                   const typename Elem<T, REAL>::V *__restrict__ src, FdArgs a) {
  using E = Elem<T, REAL>;
  using V = typename E::V;
  using I = unsigned;
  constexpr int U = fd_unroll(MODE), NB = MODE == 3 ? 6 : 2;
  const I total = (I) a.nx * (I) a.ny * (I) a.nz;
  const I e0 = (I) blockIdx.x * (I) (kFdThreads * U) + (I) threadIdx.x;
  const bool centre = MODE == 3 || lap;
  V c[U], nb[U][NB];
  I idx[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const I e = e0 + (I) (u * kFdThreads);
    if (e < total) {
      idx[u] = fd_load<T, REAL, MODE, I>(nb[u], src, e, a);
      if (centre) c[u] = src[idx[u]];
    }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (e0 + (I) (u * kFdThreads) < total) {
      V r;
      if (centre) {
        r = E::scale(c[u], (T) (MODE == 3 ? -6.0 : -2.0));
#pragma unroll
        for (int q = 0; q < NB; q++) r = E::add(r, nb[u][q]);
      } else {
        r = E::sub(nb[u][0], nb[u][1]);
      }
      dst[idx[u]] = E::scale(r, (T) a.coef);
    }
  }
}

// The same over bands of rows: a CTA takes consecutive elements of the band j0 ..
// j0 + rows - 1 of plane i, the CTAs go along x within a band.  Offsets within
// the band and coordinates are of type N; the plane's x neighbours and the row and
// column shifts are pointers of the whole CTA.
struct FdBands {
  unsigned rows, cpb;  // rows of a band, CTAs of a band of one plane
};

// The neighbour below (DIR < 0) or above along y or z at p[off]; outside the axis
// by the boundary rule, as an offset of c, n, s (coordinate, points, stride).
template <int DIR, typename T, bool REAL, typename N>
__device__ __forceinline__ typename Elem<T, REAL>::V band_neighbour(const typename Elem<T, REAL>::V *__restrict__ p,
                                                                    N off, N c, N n, long s, const FdArgs &a) {
  if (DIR > 0 ? c + 1 < n : c > 0) return p[off];
  if (a.bc == GB_BC_DIRICHLET) return Elem<T, REAL>::outside(a.out_re, a.out_im);
  N m;  // the coordinate that stands for the outside one
  if (a.bc == GB_BC_PERIODIC) m = DIR > 0 ? 0 : n - 1;
  else m = n == 1 ? 0 : DIR > 0 ? n - 2 : 1;
  return (p + ((long) m - (long) c - DIR) * s)[off];
}

template <typename T, bool REAL, int MODE, typename N>
__global__ void __launch_bounds__(kFdThreads) k_fd_bands(bool lap, typename Elem<T, REAL>::V *__restrict__ dst,
                                                         const typename Elem<T, REAL>::V *__restrict__ src, FdArgs a,
                                                         FdBands b) {
  using E = Elem<T, REAL>;
  using V = typename E::V;
  constexpr int U = fd_unroll(MODE), NB = MODE == 3 ? 6 : 2, Y = MODE == 3 ? 2 : 0, X = MODE == 3 ? 4 : 0;
  const unsigned q = blockIdx.x / b.cpb, band = q / (unsigned) a.nx, i = q - band * (unsigned) a.nx;
  const N nz = (N) a.nz, ny = (N) a.ny, row = (N) a.row, j0 = (N) band * b.rows;
  const N total = min((N) b.rows, ny - j0) * nz;
  const N e0 = (N) (blockIdx.x - q * b.cpb) * (N) (kFdThreads * U) + threadIdx.x;
  const long plane = a.ny * a.row, base = (long) i * plane + (long) j0 * a.row;
  const V *s = src + base;
  V *d = dst + base;
  // planes i + 1 and i - 1, or the ones that stand for them
  const V *xp = s + plane, *xm = s - plane;
  bool xp_out = false, xm_out = false;
  if (MODE == 0 || MODE == 3) {
    const long nx = a.nx;
    if (i + 1 == nx) {
      xp_out = a.bc == GB_BC_DIRICHLET;
      xp = s + ((a.bc == GB_BC_PERIODIC || nx == 1 ? 0 : nx - 2) - (long) i) * plane;
    }
    if (i == 0) {
      xm_out = a.bc == GB_BC_DIRICHLET;
      xm = s + (a.bc == GB_BC_PERIODIC ? nx - 1 : nx == 1 ? 0 : 1) * plane;
    }
  }
  const bool centre = MODE == 3 || lap;
  V c[U], nb[U][NB];
  N off[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const N e = e0 + (N) (u * kFdThreads);
    if (e < total) {
      const N r = e / nz, k = e - r * nz;
      const N o = r * row + k;
      off[u] = o;
      if constexpr (MODE >= 2) {
        nb[u][0] = band_neighbour<1, T, REAL, N>(s + 1, o, k, nz, 1, a);
        nb[u][1] = band_neighbour<-1, T, REAL, N>(s - 1, o, k, nz, 1, a);
      }
      if constexpr (MODE == 1 || MODE == 3) {
        nb[u][Y] = band_neighbour<1, T, REAL, N>(s + a.row, o, j0 + r, ny, a.row, a);
        nb[u][Y + 1] = band_neighbour<-1, T, REAL, N>(s - a.row, o, j0 + r, ny, a.row, a);
      }
      if constexpr (MODE == 0 || MODE == 3) {
        nb[u][X] = xp_out ? E::outside(a.out_re, a.out_im) : xp[o];
        nb[u][X + 1] = xm_out ? E::outside(a.out_re, a.out_im) : xm[o];
      }
      if (centre) c[u] = s[o];
    }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (e0 + (N) (u * kFdThreads) < total) {
      V r;
      if (centre) {
        r = E::scale(c[u], (T) (MODE == 3 ? -6.0 : -2.0));
#pragma unroll
        for (int w = 0; w < NB; w++) r = E::add(r, nb[u][w]);
      } else {
        r = E::sub(nb[u][0], nb[u][1]);
      }
      d[off[u]] = E::scale(r, (T) a.coef);
    }
  }
}

// Tiles: a CTA of 256 threads owns a (kFdTY x kFdTZ) = (8 x 32) tile of
// (y, z) over kFdXC consecutive x planes and marches along x.  Each thread
// keeps its own column's x-1, x and x+1 values in registers and loads the
// x+2 plane two steps ahead; the current plane's tile and its one-point y/z
// halo sit in a double-buffered shared-memory plane, so the y/z neighbours
// come from shared memory and every element is read from HBM about once
// ((kFdXC + 2) / kFdXC planes per chunk, plus the halo rows from L2).  The
// halo points are loaded two steps ahead as well: warp 0 the row y-1,
// warp 1 the row y+8, warp 2 the columns z-1 (lanes 0-7) and z+32 (lanes
// 8-15).  Measured at 256^3: two planes ahead at four CTAs per SM beat four
// planes ahead at three.
constexpr int kFdTY = 8, kFdTZ = 32, kFdXC = 16;
static_assert(kFdTY * kFdTZ == kFdThreads, "one thread per tile column");

template <typename T> struct FdTile {
  using E = Elem<T, false>;
  using V = C2<T>;
  V xm, c, xp, xq;  // this thread's column, planes i-1, i, i+1, i+2
  V h, hn;          // its halo point (if it owns one), planes i and i+1
  long hj, hk;      // halo point (y, z); may lie outside the grid
  int hy, hz;       // its place in the shared plane
  bool has_h;       // whether this thread owns a halo point

  __device__ void init(const V *src, const FdArgs &a, long i0, long j, long k, int ty, int tz) {
    const long j0 = j - ty, k0 = k - tz;
    hj = hk = 0;
    hy = hz = 0;
    has_h = ty < 2 || (ty == 2 && tz < 2 * kFdTY);
    if (ty == 0) {
      hj = j0 - 1, hk = k, hy = 0, hz = tz + 1;
    } else if (ty == 1) {
      hj = j0 + kFdTY, hk = k, hy = kFdTY + 1, hz = tz + 1;
    } else if (ty == 2 && tz < 2 * kFdTY) {
      const int r = tz & (kFdTY - 1);
      hj = j0 + r, hk = tz < kFdTY ? k0 - 1 : k0 + kFdTZ, hy = r + 1, hz = tz < kFdTY ? 0 : kFdTZ + 1;
    }
    // every thread of the tile loads its column, also past the far edge of
    // the grid (a partial tile): there fetch returns the boundary value the
    // last row/column needs as its neighbour
    xm = fetch<T>(src, i0 - 1, j, k, a);
    c = fetch<T>(src, i0, j, k, a);
    xp = fetch<T>(src, i0 + 1, j, k, a);
    xq = E::zero();
    h = has_h ? fetch<T>(src, i0, hj, hk, a) : E::zero();
    hn = has_h ? fetch<T>(src, i0 + 1, hj, hk, a) : E::zero();
  }

  // loads of plane i + 2 (column and halo), issued at the top of step i;
  // returns the halo value for the shift
  __device__ __forceinline__ V prefetch(const V *src, const FdArgs &a, long i, long i1, long j, long k) {
    if (i + 2 <= i1) xq = fetch<T>(src, i + 2, j, k, a);
    return (has_h && i + 2 < i1) ? fetch<T>(src, i + 2, hj, hk, a) : E::zero();
  }

  __device__ __forceinline__ void shift(V hq) {
    xm = c;
    c = xp;
    xp = xq;
    h = hn;
    hn = hq;
  }
};

// sum of a CTA's (sx, sy) by a fixed shuffle tree and warp order
__device__ __forceinline__ void fd_block_sum(double sx, double sy, double2 *out) {
  __shared__ double sb[2 * kFdThreads / 32];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    sx += __shfl_down_sync(0xffffffffu, sx, off);
    sy += __shfl_down_sync(0xffffffffu, sy, off);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    sb[2 * w] = sx;
    sb[2 * w + 1] = sy;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tx = 0.0, tyy = 0.0;
    for (int q = 0; q < kFdThreads / 32; q++) {
      tx += sb[2 * q];
      tyy += sb[2 * q + 1];
    }
    *out = make_double2(tx, tyy);
  }
}

// sum conj(psi) * Laplacian(psi) over the grid, the Laplacian summed in the
// stencil kernel's order and scaled by 1/h^2 (a.coef) before the product.
// Each CTA writes one partial (x, y) sum,
// reduced in a fixed order, so the result is the same from run to run.
template <typename T>
__global__ void __launch_bounds__(kFdThreads) k_fd_kinetic(const C2<T> *__restrict__ src, FdArgs a,
                                                           double2 *__restrict__ partial) {
  using E = Elem<T, false>;
  using V = C2<T>;
  __shared__ V sm[2][kFdTY + 2][kFdTZ + 2];
  const int tz = threadIdx.x % kFdTZ, ty = threadIdx.x / kFdTZ;
  const long k = blockIdx.x * (long) kFdTZ + tz, j = blockIdx.y * (long) kFdTY + ty;
  const long i0 = blockIdx.z * (long) kFdXC;
  const long i1 = i0 + kFdXC < a.nx ? i0 + kFdXC : a.nx;
  const bool in = k < a.nz && j < a.ny;
  FdTile<T> t;
  t.init(src, a, i0, j, k, ty, tz);
  double sx = 0.0, sy = 0.0;
  for (long i = i0; i < i1; i++) {
    const V hq = t.prefetch(src, a, i, i1, j, k);
    const int b = (int) ((i - i0) & 1);
    const V c = t.c;
    sm[b][ty + 1][tz + 1] = c;
    if (t.has_h) sm[b][t.hy][t.hz] = t.h;
    __syncthreads();
    if (in) {
      const V nb[6] = {sm[b][ty + 1][tz + 2], sm[b][ty + 1][tz], sm[b][ty + 2][tz + 1], sm[b][ty][tz + 1], t.xp, t.xm};
      double sr = -6.0 * (double) c.x, si = -6.0 * (double) c.y;
#pragma unroll
      for (int q = 0; q < 6; q++) {
        sr += (double) nb[q].x;
        si += (double) nb[q].y;
      }
      sr *= a.coef;
      si *= a.coef;
      // conj(c) * (sr + i si)
      sx += (double) c.x * sr + (double) c.y * si;
      sy += (double) c.x * si - (double) c.y * sr;
    }
    t.shift(hq);
  }
  fd_block_sum(sx, sy, partial + ((long) blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
}

// The same sum with direct neighbour reads: CTAs walk the chunks with a stride of
// the launch, faster until L2 no longer holds what is read again.  One sum, tiles
// / direct, us: FP64 150^3 (54 MB of psi) 63 / 47, 180 x 181 x 183 (95 MB) 84 /
// 71, 200^3 (128 MB) 95 / 87, 230 x 231 x 229 (195 MB) 129 / 118, 256^3 (268 MB)
// 154 / 170; FP32, where the arithmetic is a larger part, 200^3 (64 MB) 91 / 80,
// 205 x 205 x 203 (68 MB) 93 / 91, 220^3 (85 MB) 106 / 116.
constexpr int kFdKinPerSm = 6;
constexpr long fd_kin_direct_bytes(int prec) { return prec == GB_FP32 ? 64L << 20 : 192L << 20; }

template <typename T>
__global__ void __launch_bounds__(kFdThreads) k_fd_kinetic_direct(const C2<T> *__restrict__ src, FdArgs a,
                                                                  double2 *__restrict__ partial) {
  constexpr unsigned U = 2;
  const unsigned total = (unsigned) (a.nx * a.ny * a.nz);
  double sx = 0.0, sy = 0.0;
  for (unsigned e0 = blockIdx.x * (kFdThreads * U) + threadIdx.x; e0 < total; e0 += gridDim.x * (kFdThreads * U)) {
    C2<T> c[U], nb[U][6];
#pragma unroll
    for (unsigned u = 0; u < U; u++) {
      const unsigned e = e0 + u * kFdThreads;
      if (e < total) c[u] = src[fd_load<T, false, 3, unsigned>(nb[u], src, e, a)];
    }
#pragma unroll
    for (unsigned u = 0; u < U; u++) {
      if (e0 + u * kFdThreads < total) {
        double sr = -6.0 * (double) c[u].x, si = -6.0 * (double) c[u].y;
#pragma unroll
        for (int q = 0; q < 6; q++) {
          sr += (double) nb[u][q].x;
          si += (double) nb[u][q].y;
        }
        sr *= a.coef;
        si *= a.coef;
        // conj(c) * (sr + i si)
        sx += (double) c[u].x * sr + (double) c[u].y * si;
        sy += (double) c[u].x * si - (double) c[u].y * sr;
      }
    }
  }
  fd_block_sum(sx, sy, partial + blockIdx.x);
}

// Sum of n partials by one CTA of 256 threads: strided per-thread sums,
// then a fixed shuffle tree (deterministic).
__global__ void __launch_bounds__(256) k_finish_fd(const double2 *__restrict__ p, long n, double2 *out) {
  __shared__ double sb[16];
  double sx = 0.0, sy = 0.0;
  for (long i = threadIdx.x; i < n; i += 256) {
    sx += p[i].x;
    sy += p[i].y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    sx += __shfl_down_sync(0xffffffffu, sx, off);
    sy += __shfl_down_sync(0xffffffffu, sy, off);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    sb[2 * w] = sx;
    sb[2 * w + 1] = sy;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tx = 0.0, ty = 0.0;
    for (int q = 0; q < 8; q++) {
      tx += sb[2 * q];
      ty += sb[2 * q + 1];
    }
    *out = make_double2(tx, ty);
  }
}

// Launch grid of the tiled kinetic sum: (z tiles, y tiles, x chunks).  Extents
// beyond it are refused by the stencils too: one limit for all calls.
int fd_grid(const gb_geom *g, dim3 *grid) {
  const long gz = (g->nz + kFdTZ - 1) / kFdTZ, gy = (g->ny + kFdTY - 1) / kFdTY, gx = (g->nx + kFdXC - 1) / kFdXC;
  if (gy > 65535 || gx > 65535) return gb__set_error(1005, "fd: grid too large for the stencil tiling");
  *grid = dim3((unsigned) gz, (unsigned) gy, (unsigned) gx);
  return 0;
}

// Flat order up to 2^31 stored elements less the overhang of a launch: the two
// divisions of a point cost several times as much in 64 bits.  Beyond, and where
// the planes that an x neighbour takes are too large for L2 to hold three of, in
// bands: at 1300^3 (2.2e9 points) flat with 64-bit indices / bands, ms: Laplacian
// 31.0 / 15.3 complex, 17.4 / 11.2 real FP32; x gradient 16.2 / 10.7, 10.6 / 5.1;
// z gradient 11.7 / 10.3, 7.2 / 5.3 (halo tiles 17.7 and 11.6 throughout).  Complex
// FP64 Laplacian, flat / bands, us: 96 x 1024 x 1024 (planes of 17 MB) 669 / 705;
// 80 x 1150 x 1150 (21 MB) 781 / 773; 64 x 1300 x 1300 (27 MB) 947 / 764; 32 x
// 2048 x 2048 (67 MB) 1181 / 947; x gradient there 914 / 666, y 625 / 652.
// Elements of 8 bytes: Laplacian 690 / 732 at 32 x 2048 x 2048.  Bands of 8 MB in
// place of 2: 825 at 64 x 1300 x 1300; where three planes fit, whole planes (1300^3
// real FP32 Laplacian 11.2 ms against 12.5 in bands of 2 MB).
constexpr long kFdBandPlane = 20L << 20, kFdBandBytes = 2L << 20;

template <typename T, bool REAL, int MODE>
int fd_launch(bool lap, void *dst, const void *src, const FdArgs &a) {
  using V = typename Elem<T, REAL>::V;
  constexpr long CH = (long) kFdThreads * fd_unroll(MODE), kMost = (1L << 31) - (1L << 20);
  const long plane = a.ny * a.row, row_bytes = a.row * (long) sizeof(V);
  V *d = (V *) dst;
  const V *s = (const V *) src;
  cudaStream_t st = gb__stream();
  const bool along_x = (MODE == 0 || MODE == 3) && sizeof(V) == 16;
  if (a.nx * plane < kMost && !(along_x && plane * (long) sizeof(V) > kFdBandPlane)) {
    const long nb = (a.nx * a.ny * a.nz + CH - 1) / CH;
    k_fd<T, REAL, MODE><<<(unsigned) nb, kFdThreads, 0, st>>>(lap, d, s, a);
  } else {
    FdBands b;
    const long want = plane * (long) sizeof(V) <= kFdBandPlane ? a.ny : std::max(8L, kFdBandBytes / row_bytes);
    const long rows = std::max(1L, std::min(std::min(a.ny, want), kMost / a.row));
    b.rows = (unsigned) rows;
    b.cpb = (unsigned) ((rows * a.nz + CH - 1) / CH);
    const unsigned nb = (unsigned) ((a.ny + rows - 1) / rows * a.nx * b.cpb);
    if (a.row < kMost) k_fd_bands<T, REAL, MODE, unsigned><<<nb, kFdThreads, 0, st>>>(lap, d, s, a, b);
    else k_fd_bands<T, REAL, MODE, unsigned long><<<nb, kFdThreads, 0, st>>>(lap, d, s, a, b);
  }
  GB_CHECK_LAUNCH("fd stencil");
  return 0;
}

template <typename T, bool REAL> int fd_op(int op, void *dst, const void *src, const FdArgs &a) {
  switch (op) {
    case GB_FD_LAPLACE: return fd_launch<T, REAL, 3>(true, dst, src, a);
    case GB_FD_LAPLACE_X: return fd_launch<T, REAL, 0>(true, dst, src, a);
    case GB_FD_LAPLACE_Y: return fd_launch<T, REAL, 1>(true, dst, src, a);
    case GB_FD_LAPLACE_Z: return fd_launch<T, REAL, 2>(true, dst, src, a);
    case GB_FD_GRADIENT_X: return fd_launch<T, REAL, 0>(false, dst, src, a);
    case GB_FD_GRADIENT_Y: return fd_launch<T, REAL, 1>(false, dst, src, a);
    default: return fd_launch<T, REAL, 2>(false, dst, src, a);
  }
}

}  // namespace

extern "C" int gb_fd(int op, void *dst, const void *src, const gb_geom *g, int bc, double out_re, double out_im, double coef,
                     int is_real, long row) {
  FdArgs a;
  a.nx = g->nx;
  a.ny = g->ny;
  a.nz = g->nz;
  a.row = row;
  a.bc = bc;
  a.out_re = out_re;
  a.out_im = out_im;
  a.coef = coef;
  dim3 grid;
  if (fd_grid(g, &grid)) return gb_last_error();
  if (is_real) return g->prec == GB_FP32 ? fd_op<float, true>(op, dst, src, a) : fd_op<double, true>(op, dst, src, a);
  return g->prec == GB_FP32 ? fd_op<float, false>(op, dst, src, a) : fd_op<double, false>(op, dst, src, a);
}

extern "C" int gb_fd_kinetic_sum(const void *psi, const gb_geom *g, int bc, double out_re, double out_im, double inv_h2,
                                 double *out) {
  FdArgs a;
  a.nx = g->nx;
  a.ny = g->ny;
  a.nz = g->nz;
  a.row = g->nz;
  a.bc = bc;
  a.out_re = out_re;
  a.out_im = out_im;
  a.coef = inv_h2;
  dim3 grid;
  if (fd_grid(g, &grid)) return gb_last_error();
  const long n = g->nx * g->ny * g->nz, chunks = (n + 2 * kFdThreads - 1) / (2 * kFdThreads);
  const bool direct = n * (g->prec == GB_FP32 ? 8 : 16) <= fd_kin_direct_bytes(g->prec);
  const long nb = direct ? std::min(chunks, (long) kFdKinPerSm * gb__num_sms()) : (long) grid.x * grid.y * grid.z;
  double2 *partial = (double2 *) gb__scratch(GB_SCR_PARTIAL, sizeof(double2) * (size_t) nb);
  double2 *res = (double2 *) gb__result_slot();
  if (!partial || !res) return gb_last_error();
  cudaStream_t st = gb__stream();
  if (direct) {
    if (g->prec == GB_FP32) k_fd_kinetic_direct<float><<<(unsigned) nb, kFdThreads, 0, st>>>((const float2 *) psi, a, partial);
    else k_fd_kinetic_direct<double><<<(unsigned) nb, kFdThreads, 0, st>>>((const double2 *) psi, a, partial);
  } else if (g->prec == GB_FP32) k_fd_kinetic<float><<<grid, kFdThreads, 0, st>>>((const float2 *) psi, a, partial);
  else k_fd_kinetic<double><<<grid, kFdThreads, 0, st>>>((const double2 *) psi, a, partial);
  GB_CHECK_LAUNCH("fd kinetic");
  k_finish_fd<<<1, 256, 0, st>>>(partial, nb, res);
  GB_CHECK_LAUNCH("fd kinetic finish");
  double2 h;
  int rc = gb__read_result(&h, sizeof(double2));
  out[0] = h.x;
  out[1] = h.y;
  return rc;
}
