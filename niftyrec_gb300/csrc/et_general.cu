// General-orientation path: cameras with any (theta_x, theta_y, theta_z),
// any background values, any grid.  Volumes in nifti layout.  Each stage is a
// separate kernel following the reference's float operation order (products
// and sums rounded separately), so this path reproduces the reference CPU
// path up to the last bit of expf.  A launch covers a group of cameras (their
// matrices are launch parameters, the work volumes sit one after another), so
// the per-ray scans of one camera -- a few thousand threads -- do not leave the
// GPU idle.  The fused kernels of et_yg_*.cu cover the common gantry case;
// this path covers everything else.
#include "et_kernels.h"
#include "et_profile.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace nrgb {

namespace {

template <class T>
struct Affine34T {
  T m[12];
};
using Affine34 = Affine34T<float>;

// Separately rounded arithmetic in the working type (float: the reference's
// type; double: the float64 reference path).
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double fm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fa(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double fs(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float flo(float v) { return floorf(v); }
__device__ __forceinline__ double flo(double v) { return floor(v); }
__device__ __forceinline__ float ex(float v) { return expf(v); }
__device__ __forceinline__ double ex(double v) { return exp(v); }

// Matrices of a group of cameras, a kernel parameter.
template <class T>
struct AffineSetT {
  T m[kGeneralGroup][12];
};

// Grid and layout of the work volumes: planes [y][x] (x fastest, the caller's
// order) or, with col, [x][y].
struct Grid {
  int nx, ny, nz, col;
  __device__ __forceinline__ int sx() const { return col ? ny : 1; }
  __device__ __forceinline__ int sy() const { return col ? 1 : nx; }
  __device__ __forceinline__ size_t at(int x, int y, int z) const {
    return static_cast<size_t>(z) * ny * nx + static_cast<size_t>(y) * sy() + static_cast<size_t>(x) * sx();
  }
  // index of element i of a work plane in the caller's [y][x] plane
  __device__ __forceinline__ size_t caller(size_t i) const { return col ? i % ny * nx + i / ny : i; }
};

// Footprint of one voxel: floor positions and the two weights per axis
// (reg-lib/_reg_affineTransformation.cpp:116-132 with an identity
// voxel-to-world matrix, reg-lib/_reg_resampling.cpp:334-364).
template <class T>
struct Foot {
  int prev[3];
  T b0[3], b1[3];
};

template <class T>
__device__ __forceinline__ Foot<T> footprint(const T* m, int x, int y, int z) {
  const T fx = static_cast<T>(x), fy = static_cast<T>(y), fz = static_cast<T>(z);
  Foot<T> f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T pos = fa(fa(fa(fm(m[4 * i + 0], fx), fm(m[4 * i + 1], fy)), fm(m[4 * i + 2], fz)), m[4 * i + 3]);
    f.prev[i] = static_cast<int>(flo(pos));
    T rel = fs(pos, static_cast<T>(f.prev[i]));
    if (rel < T(0)) rel = T(0);
    f.b0[i] = fs(T(1), rel);
    f.b1[i] = rel;
  }
  return f;
}

// Trilinear value of a footprint, reg-lib/_reg_resampling.cpp:365-450.  With
// bg != 0 every neighbour outside the grid adds bg * xBasis[.] to a separate
// background weight, as the reference does (:366-396).  A footprint inside
// the grid -- nearly all -- takes the same sums without the tests.  Under a
// caller's affine matrix the floor may saturate: no neighbour's index is formed
// before it is known to lie in the grid, so that it cannot wrap into it.
template <class T>
__device__ __forceinline__ T trilinear_ref(const T* __restrict__ src, const Grid& n, const Foot<T>& f, T bg) {
  const int nx = n.nx, ny = n.ny, nz = n.nz;
  const int px = f.prev[0], py = f.prev[1], pz = f.prev[2];
  if (px >= 0 && px < nx - 1 && py >= 0 && py < ny - 1 && pz >= 0 && pz < nz - 1) {
    const T* p = src + n.at(px, py, pz);
    const T* q = p + static_cast<size_t>(ny) * nx;
    const int sx = n.sx(), sy = n.sy();
    auto line = [&](const T* r) { return fa(fm(__ldg(r), f.b0[0]), fm(__ldg(r + sx), f.b1[0])); };
    auto plane = [&](const T* r) { return fa(fm(line(r), f.b0[1]), fm(line(r + sy), f.b1[1])); };
    return fa(fm(plane(p), f.b0[2]), fm(plane(q), f.b1[2]));
  }
  const T bx[2] = {f.b0[0], f.b1[0]};
  const T by[2] = {f.b0[1], f.b1[1]};
  const T bz[2] = {f.b0[2], f.b1[2]};
  T val = T(0), bgw = T(0);
  const bool use_bg = (bg != T(0));
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (pz >= -c && pz < nz - c) {
      T ysum = T(0);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (py >= -b && py < ny - b) {
          T xsum = T(0);
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            if (px >= -a && px < nx - a)
              xsum = fa(xsum, fm(__ldg(src + n.at(px + a, py + b, pz + c)), bx[a]));
            else if (use_bg)
              bgw = fa(bgw, fm(bg, bx[a]));
          }
          ysum = fa(ysum, fm(xsum, by[b]));
        } else if (use_bg) {
          bgw = fa(bgw, fm(bg, bx[b]));
        }
      }
      val = fa(val, fm(ysum, bz[c]));
    } else if (use_bg) {
      bgw = fa(bgw, fm(bg, bx[c]));
    }
  }
  if (use_bg) val = fa(val, bgw);
  return val;
}

// Voxel of this thread in a launch of 32 x 8-voxel blocks (32 along the fast
// axis) over (fast tile, slow tile, z, camera of the group); one set of 32-bit
// divisions per block.
struct Voxel {
  int x, y, z, g;
};

__device__ __forceinline__ Voxel block_voxel(const Grid& n) {
  const int tf = ((n.col ? n.ny : n.nx) + 31) / 32, ts = ((n.col ? n.nx : n.ny) + 7) / 8;
  int b = blockIdx.x;
  Voxel v;
  const int fast = b % tf * 32 + threadIdx.x;
  b /= tf;
  const int slow = b % ts * 8 + threadIdx.y;
  b /= ts;
  v.x = n.col ? slow : fast;
  v.y = n.col ? fast : slow;
  v.z = b % n.nz;
  v.g = b / n.nz;
  return v;
}

// dst[g] = src resampled at the positions of camera g; with src2 the same for
// a second volume (activity and mu share their footprints).
template <class T>
__global__ void __launch_bounds__(256)
    k_resample(const T* __restrict__ src, T* __restrict__ dst, T bg, const T* __restrict__ src2, T* __restrict__ dst2,
               T bg2, const Grid n, const __grid_constant__ AffineSetT<T> A) {
  const Voxel v = block_voxel(n);
  if (v.x >= n.nx || v.y >= n.ny) return;
  const Foot<T> f = footprint(A.m[v.g], v.x, v.y, v.z);
  const size_t o = static_cast<size_t>(v.g) * n.nz * n.ny * n.nx + n.at(v.x, v.y, v.z);
  if (src) dst[o] = trilinear_ref(src, n, f, bg);
  if (src2) dst2[o] = trilinear_ref(src2, n, f, bg2);
}

// dst (the caller's layout) (+)= sum over the group's cameras, in camera order,
// of src[g] resampled at camera g's positions; first: assign; clamp: store
// negative sums as zero.
template <class T>
__global__ void __launch_bounds__(256)
    k_resample_sum(const T* __restrict__ src, T* __restrict__ dst, int count, int first, int clamp, T bg, const Grid n,
                   const __grid_constant__ AffineSetT<T> A) {
  const Voxel v = block_voxel(n);
  if (v.x >= n.nx || v.y >= n.ny) return;
  const size_t nvox = static_cast<size_t>(n.nx) * n.ny * n.nz;
  const size_t o = (static_cast<size_t>(v.z) * n.ny + v.y) * n.nx + v.x;
  T acc = first ? T(0) : dst[o];
  for (int g = 0; g < count; ++g)
    acc = fa(acc, trilinear_ref(src + nvox * g, n, footprint(A.m[g], v.x, v.y, v.z), bg));
  dst[o] = clamp && acc < T(0) ? T(0) : acc;
}

// Planes [y][x] to [x][y] through a 32 x 32 tile.
template <class T>
__global__ void __launch_bounds__(256) k_transpose(const T* __restrict__ src, T* __restrict__ dst, int nx, int ny) {
  __shared__ T tile[32][33];
  const int tx = (nx + 31) / 32, ty = (ny + 31) / 32;
  int b = blockIdx.x;
  const int x0 = b % tx * 32;
  b /= tx;
  const int y0 = b % ty * 32;
  b /= ty;
  const size_t plane = static_cast<size_t>(b) * ny * nx;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (x0 + threadIdx.x < nx && y0 + r < ny)
      tile[r][threadIdx.x] = src[plane + static_cast<size_t>(y0 + r) * nx + x0 + threadIdx.x];
  __syncthreads();
  for (int c = threadIdx.y; c < 32; c += 8)
    if (x0 + c < nx && y0 + threadIdx.x < ny)
      dst[plane + static_cast<size_t>(x0 + c) * ny + y0 + threadIdx.x] = tile[threadIdx.x][c];
}

// Transpose of trilinear_ref with bg = 0: add v * weight to each in-grid
// corner of the footprint (atomics: footprints overlap).
__device__ __forceinline__ void trilinear_scatter(float* __restrict__ dst, int nx, int ny, int nz,
                                                  const Foot<float>& f, float v) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (f.prev[2] < -c || f.prev[2] >= nz - c) continue;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (f.prev[1] < -b || f.prev[1] >= ny - b) continue;
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        if (f.prev[0] < -a || f.prev[0] >= nx - a) continue;
        const float w = (a ? f.b1[0] : f.b0[0]) * (b ? f.b1[1] : f.b0[1]) * (c ? f.b1[2] : f.b0[2]);
        if (w != 0.0f)
          atomicAdd(dst + (static_cast<size_t>(f.prev[2] + c) * ny + f.prev[1] + b) * nx + f.prev[0] + a, v * w);
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_scatter(const float* __restrict__ src, float* __restrict__ dst, int nx, int ny,
                                                 int nz, const __grid_constant__ AffineSetT<float> A) {
  const Voxel v = block_voxel(Grid{nx, ny, nz, 0});
  if (v.x >= nx || v.y >= ny) return;
  const float s = src[((static_cast<size_t>(v.g) * nz + v.z) * ny + v.y) * nx + v.x];
  if (s == 0.0f) return;
  trilinear_scatter(dst, nx, ny, nz, footprint(A.m[v.g], v.x, v.y, v.z), s);
}

// Row (x) then column (y) pass of emission-lib/_et_convolveSeparable2D.cpp:13-40:
// true convolution (kernel index R-k), zero outside the plane, plane z uses
// kernel plane z.  sep layout [plane][row k | column k].  FLIP: correlation
// (kernel index R+k), the transpose of the convolution.
template <bool ROWS, bool FLIP = false, class T = float>
__global__ void k_conv(const T* __restrict__ in, T* __restrict__ out, int nx, int ny, int nz, const T* __restrict__ sep,
                       int k) {
  const size_t nvox = static_cast<size_t>(nx) * ny * nz;
  const int R = (k - 1) / 2;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nvox;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int x = static_cast<int>(i % nx);
    const int y = static_cast<int>((i / nx) % ny);
    const int z = static_cast<int>(i / (static_cast<size_t>(nx) * ny));
    const T* K = sep + static_cast<size_t>(2 * k) * z + (ROWS ? 0 : k);
    T s = T(0);
    for (int kk = -R; kk <= R; ++kk) {
      if (ROWS) {
        const int d = x + kk;
        if (d >= 0 && d < nx) s = fa(s, fm(__ldg(in + i + kk), __ldg(K + (FLIP ? R + kk : R - kk))));
      } else {
        const int d = y + kk;
        if (d >= 0 && d < ny)
          s = fa(s, fm(__ldg(in + i + static_cast<ptrdiff_t>(kk) * nx), __ldg(K + (FLIP ? R + kk : R - kk))));
      }
    }
    out[i] = s;
  }
}

// Both passes of one 32 x 32 tile of a plane through shared memory, PSF radius
// R <= 7: the tile and its halo are read once (zeros outside the plane), a
// thread then sums four consecutive outputs of a row, and of a column, from
// 4 + 2R values.  Same products and order as k_conv<ROWS> then k_conv<columns>
// (a zero outside the plane adds nothing), which read every tap from L1/L2 and
// took two passes over the volume.  With FLIP both are correlations.
// The row kernel index advances with the plane of the volume: plane z of
// camera g of the group.
template <int R, bool FLIP, class T>
__global__ void __launch_bounds__(256)
    k_conv2(const T* __restrict__ in, T* __restrict__ out, int nx, int ny, int nz, const T* __restrict__ sep, int col) {
  constexpr int K = 2 * R + 1, W = 32 + 2 * R, N = 4;
  __shared__ T s_in[W][W + 1];
  __shared__ T s_row[W][33];
  const int tx = (nx + 31) / 32, ty = (ny + 31) / 32;
  int b = blockIdx.x;
  const int x0 = b % tx * 32;
  b /= tx;
  const int y0 = b % ty * 32;
  b /= ty;  // plane of the group: camera * nz + z
  const T* src = in + static_cast<size_t>(b) * ny * nx;
  const T* k = sep + static_cast<size_t>(2 * K) * (b % nz);
  for (int e = threadIdx.x; e < W * W; e += 256) {
    const int r = col ? e % W : e / W, c = col ? e / W : e % W;  // lanes along the fast axis
    const int x = x0 - R + c, y = y0 - R + r;
    const size_t o = col ? static_cast<size_t>(x) * ny + y : static_cast<size_t>(y) * nx + x;
    s_in[r][c] = x >= 0 && x < nx && y >= 0 && y < ny ? __ldg(src + o) : T(0);
  }
  T kr[K], kc[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    kr[j] = __ldg(k + (FLIP ? j : 2 * R - j));
    kc[j] = __ldg(k + K + (FLIP ? j : 2 * R - j));
  }
  __syncthreads();
  // a coefficient that is not finite must not meet the zeros outside the plane
  bool finite = true;
#pragma unroll
  for (int j = 0; j < K; ++j) finite = finite && isfinite(kr[j]) && isfinite(kc[j]);
  // this thread's outputs of the column pass: lanes along the fast axis
  const int c = col ? threadIdx.x / 8 : threadIdx.x % 32, r = (col ? threadIdx.x % 8 : threadIdx.x / 32) * N;
  T s[N];
  auto both = [&](auto check) {
    constexpr bool CHECK = decltype(check)::value;
    for (int e = threadIdx.x; e < W * (32 / N); e += 256) {
      const int er = e % W, ec = e / W * N;
#pragma unroll
      for (int i = 0; i < N; ++i) s[i] = T(0);
#pragma unroll
      for (int j = 0; j < N + 2 * R; ++j) {
        const T v = s_in[er][ec + j];
        const int x = x0 - R + ec + j;
        if (CHECK && (x < 0 || x >= nx)) continue;
#pragma unroll
        for (int i = 0; i < N; ++i)
          if (j - i >= 0 && j - i < K) s[i] = fa(s[i], fm(v, kr[j - i]));
      }
#pragma unroll
      for (int i = 0; i < N; ++i) s_row[er][ec + i] = s[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = T(0);
#pragma unroll
    for (int j = 0; j < N + 2 * R; ++j) {
      const T v = s_row[r + j][c];
      const int y = y0 - R + r + j;
      if (CHECK && (y < 0 || y >= ny)) continue;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (j - i >= 0 && j - i < K) s[i] = fa(s[i], fm(v, kc[j - i]));
    }
  };
  if (finite) both(std::false_type());
  else both(std::true_type());  // uniform over the block: one plane's coefficients
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (x0 + c < nx && y0 + r + i < ny)
      out[static_cast<size_t>(b) * ny * nx + (col ? static_cast<size_t>(x0 + c) * ny + y0 + r + i
                                                  : static_cast<size_t>(y0 + r + i) * nx + x0 + c)] = s[i];
}

constexpr int kScanDepth = 8;  // depth planes whose loads a ray scan has in flight

// Attenuated line integral along z, emission-lib/_et_line_integral_attenuated.cpp:14-68;
// blockIdx.y: camera of the group.
template <class R = float>
__global__ void k_line_integral(const R* __restrict__ act, const R* __restrict__ att, R* __restrict__ out,
                                const Grid n, R bg, int truncate) {
  const int nz = n.nz;
  const size_t nxy = static_cast<size_t>(n.nx) * n.ny;
  const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= nxy) return;
  const size_t vol = nxy * nz * blockIdx.y;
  if (act) act += vol + i;
  if (att) att += vol + i;
  R p = R(0), T = R(0);
  for (int z0 = 0; z0 < nz; z0 += kScanDepth) {
    R a[kScanDepth], m[kScanDepth];
#pragma unroll
    for (int d = 0; d < kScanDepth; ++d) {
      const bool in = z0 + d < nz;
      a[d] = act && in ? __ldg(act + nxy * (z0 + d)) : R(0);
      m[d] = att && in ? __ldg(att + nxy * (z0 + d)) : R(0);
    }
#pragma unroll
    for (int d = 0; d < kScanDepth; ++d) {
      if (z0 + d >= nz) break;
      if (att) T = fa(T, m[d]);
      if (act) p = fa(p, att ? fm(a[d], ex(-T)) : a[d]);
    }
  }
  if (act && att) p = fa(p, fm(bg, ex(-T)));
  else if (act) p = fa(p, bg);
  else p = fm(bg, ex(-T));
  if (truncate && p < R(0)) p = R(0);
  out[nxy * blockIdx.y + n.caller(i)] = p;
}

// Spread along z, emission-lib/_et_line_backproject_attenuated.cpp:17-36 and
// emission-lib/_et_line_backproject.cpp:17-30; blockIdx.y: camera of the group.
template <class R = float>
__global__ void k_spread(const R* __restrict__ plane, const R* __restrict__ att, R* __restrict__ vol, const Grid n) {
  const int nz = n.nz;
  const size_t nxy = static_cast<size_t>(n.nx) * n.ny;
  const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= nxy) return;
  const size_t off = nxy * nz * blockIdx.y + i;
  const R s = __ldg(plane + nxy * blockIdx.y + n.caller(i));
  R T = R(0);
  for (int z0 = 0; z0 < nz; z0 += kScanDepth) {
    R m[kScanDepth];
#pragma unroll
    for (int d = 0; d < kScanDepth; ++d) m[d] = att && z0 + d < nz ? __ldg(att + off + nxy * (z0 + d)) : R(0);
#pragma unroll
    for (int d = 0; d < kScanDepth; ++d) {
      if (z0 + d >= nz) break;
      T = fa(T, m[d]);
      vol[off + nxy * (z0 + d)] = att ? fm(s, ex(-T)) : s;
    }
  }
}

// Partial-sum line integral, the partial-sum branch of
// emission-lib_gpu/_et_line_integral_attenuated_gpu_kernels.cu:57-103: walk
// depth from the far end, partial[z] = s before voxel z is added and
// attenuated; s starts at bg (times bg_image[x, y]); the projection is the
// final s.
__global__ void k_line_partial(const float* __restrict__ act, const float* __restrict__ att,
                               const float* __restrict__ bg_image, float* __restrict__ out,
                               float* __restrict__ partial, int nx, int ny, int nz, float bg) {
  const int nxy = nx * ny;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nxy) return;
  const size_t off = static_cast<size_t>(nxy) * nz * blockIdx.y, off2 = static_cast<size_t>(nxy) * blockIdx.y;
  if (act) act += off;
  if (att) att += off;
  partial += off;
  out += off2;
  float s = bg;
  if (bg_image) s = fm(s, __ldg(bg_image + i));
  for (int z = nz - 1; z >= 0; --z) {
    const size_t j = static_cast<size_t>(z) * nxy + i;
    partial[j] = s;
    if (act && att)
      s = fm(fa(s, __ldg(act + j)), expf(-__ldg(att + j)));
    else if (att)
      s = fm(s, expf(-__ldg(att + j)));
    else
      s = fa(s, __ldg(act + j));
  }
  out[i] = s;
}

// Attenuation-gradient scan, emission-lib_gpu/_et_attenuation_gradient_gpu_kernels.cu:24-39:
// pass 1 stores the inclusive prefix T_z, pass 2 (far to near) accumulates
// a_z * exp(-T_z) and stores s * acc.
__global__ void k_grad_scan(const float* __restrict__ act, const float* __restrict__ att,
                            const float* __restrict__ plane, float* __restrict__ vol, int nx, int ny, int nz) {
  const int nxy = nx * ny;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nxy) return;
  const size_t off = static_cast<size_t>(nxy) * nz * blockIdx.y, off2 = static_cast<size_t>(nxy) * blockIdx.y;
  if (act) act += off;
  if (att) att += off;
  vol += off;
  plane += off2;
  float T = 0.0f;
  for (int z = 0; z < nz; ++z) {
    const size_t j = static_cast<size_t>(z) * nxy + i;
    T = fa(T, __ldg(att + j));
    vol[j] = T;
  }
  const float s = __ldg(plane + i);
  float acc = 0.0f;
  for (int z = nz - 1; z >= 0; --z) {
    const size_t j = static_cast<size_t>(z) * nxy + i;
    acc = fa(acc, fm(__ldg(act + j), expf(-vol[j])));
    vol[j] = fm(s, acc);
  }
}

// Gradient of a projection plane with respect to the rotated mu.  With
// p = sum_z v_z exp(-T_z) + bg exp(-T_N) (v: PSF-convolved rotated activity,
// T inclusive prefix of the rotated mu m), dp/dm_z' = -(S_z' + bg exp(-T_N)),
// S_z' = sum_{z >= z'} v_z exp(-T_z) = P_v - (prefix of v exp(-T) before z').
// out[z'] = g * dp/dm_z'.  Not in the reference (whose gradient,
// emission-lib_gpu/_et_attenuation_gradient_gpu_kernels.cu:15-42, ignores the
// PSF coupling, the sign and the background).
__global__ void k_dmu_scan(const float* __restrict__ v, const float* __restrict__ m, const float* __restrict__ g_plane,
                           float* __restrict__ out, int nx, int ny, int nz, float bg) {
  const int nxy = nx * ny;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nxy) return;
  const size_t off = static_cast<size_t>(nxy) * nz * blockIdx.y, off2 = static_cast<size_t>(nxy) * blockIdx.y;
  v += off;
  m += off;
  out += off;
  g_plane += off2;
  float T = 0.0f, Pv = 0.0f;
  for (int z = 0; z < nz; ++z) {
    const size_t j = static_cast<size_t>(z) * nxy + i;
    T += __ldg(m + j);
    Pv = fmaf(__ldg(v + j), __expf(-T), Pv);
  }
  const float tail = bg * __expf(-T);
  const float g = __ldg(g_plane + i);
  float prefix = 0.0f;
  T = 0.0f;
  for (int z = 0; z < nz; ++z) {
    const size_t j = static_cast<size_t>(z) * nxy + i;
    T += __ldg(m + j);
    const float e = __expf(-T);
    out[j] = -g * ((Pv - prefix) + tail);
    prefix = fmaf(__ldg(v + j), e, prefix);
  }
}

int grid_for(size_t n, int block) {
  const size_t g = (n + block - 1) / block;
  const int cap = sm_count() * 64;
  return static_cast<int>(g < cap ? g : cap);
}

// Launches of one call's stages over groups of cameras.
template <class T>
struct General {
  const GeneralArgsT<T>& a;
  cudaStream_t st;
  size_t nvox, nxy;
  int cam0 = 0, n = 0;  // the current group
  Grid grid;

  General(const GeneralArgsT<T>& args, cudaStream_t stream) : a(args), st(stream) {
    nxy = static_cast<size_t>(a.nx) * a.ny;
    nvox = nxy * a.nz;
    grid = {a.nx, a.ny, a.nz, 0};
  }

  // Work volumes as planes [x][y] where that is the better order: the lanes of
  // a resampling step along the fast axis, and a load is coalesced as far as
  // that step stays on the axis.  Cameras turned about y (tilted heads) keep y:
  // 96^3 x 30 cameras tilted by 7 degrees, projection + backprojection 1.53 ms
  // along x, 1.43 along y.  Needs the fused convolution, and two volumes for
  // the sources.
  void choose_layout() {
    if (!a.ws_src || a.ncam < 2 || (a.psf_sep && a.psf_k > 15)) return;
    T off_x = 0, off_y = 0;  // how far steps along x and y leave their axis
    for (int c = 0; c < a.ncam; ++c) {
      const T* m = a.geom_host[c].fwd;
      off_x += std::abs(m[4]) + std::abs(m[8]);
      off_y += std::abs(m[1]) + std::abs(m[9]);
    }
    grid.col = off_y < T(0.7) * off_x;
  }

  // A source volume in the work layout (slot 0 or 1 of a.ws_src).
  const T* source(const T* src, int slot) {
    if (!src || !grid.col) return src;
    T* dst = a.ws_src + nvox * slot;
    NRGB_LAUNCH_SCOPE("k_transpose", st);
    k_transpose<T><<<static_cast<unsigned>((a.nx + 31) / 32) * ((a.ny + 31) / 32) * a.nz, dim3(32, 8), 0, st>>>(
        src, dst, a.nx, a.ny);
    return dst;
  }

  template <class Body>
  int groups(Body body) {
    const int group = std::max(1, std::min(a.group, kGeneralGroup));
    for (cam0 = 0; cam0 < a.ncam; cam0 += group) {
      n = std::min(group, a.ncam - cam0);
      body();
    }
    return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
  }

  bool last() const { return cam0 + n == a.ncam; }

  AffineSetT<T> matrices(bool back) const {
    AffineSetT<T> s = {};
    for (int g = 0; g < n; ++g) {
      const T* m = back ? a.geom_host[cam0 + g].bwd : a.geom_host[cam0 + g].fwd;
      std::copy(m, m + 12, s.m[g]);
    }
    return s;
  }

  // blocks of 32 (fast axis) x rows voxels over `volumes` volumes
  unsigned blocks(int rows, int volumes) const {
    const int fast = grid.col ? a.ny : a.nx, slow = grid.col ? a.nx : a.ny;
    return static_cast<unsigned>((fast + 31) / 32) * ((slow + rows - 1) / rows) * a.nz * volumes;
  }
  dim3 rays() const { return dim3(static_cast<unsigned>((nxy + 127) / 128), n); }

  // rotate one or two volumes (either may be null) into work volumes
  void rotate(const T* src, T* dst, T bg, const T* src2, T* dst2, T bg2) {
    if (!src && !src2) return;
    NRGB_LAUNCH_SCOPE("k_resample", st);
    k_resample<T><<<blocks(8, n), dim3(32, 8), 0, st>>>(src, dst, bg, src2, dst2, bg2, grid, matrices(false));
  }

  // PSF of the group's volumes; returns where the result is (tmp, or vol for
  // radii beyond the fused kernel, whose two passes go through tmp)
  template <bool FLIP = false>
  T* convolve(T* vol, T* tmp) {
    if (!a.psf_sep) return vol;
    auto go = [&](auto k) {
      NRGB_LAUNCH_SCOPE("k_conv2", st);
      k<<<blocks(32, n), 256, 0, st>>>(vol, tmp, a.nx, a.ny, a.nz, a.psf_sep, grid.col);
    };
    switch ((a.psf_k - 1) / 2) {
      case 0: go(k_conv2<0, FLIP, T>); return tmp;
      case 1: go(k_conv2<1, FLIP, T>); return tmp;
      case 2: go(k_conv2<2, FLIP, T>); return tmp;
      case 3: go(k_conv2<3, FLIP, T>); return tmp;
      case 4: go(k_conv2<4, FLIP, T>); return tmp;
      case 5: go(k_conv2<5, FLIP, T>); return tmp;
      case 6: go(k_conv2<6, FLIP, T>); return tmp;
      case 7: go(k_conv2<7, FLIP, T>); return tmp;
      default: break;
    }
    for (int g = 0; g < n; ++g) {
      T *v = vol + nvox * g, *t = tmp + nvox * g;
      NRGB_LAUNCH_SCOPE("k_conv", st);
      k_conv<true, FLIP, T><<<grid_for(nvox, 256), 256, 0, st>>>(v, t, a.nx, a.ny, a.nz, a.psf_sep, a.psf_k);
      k_conv<false, FLIP, T><<<grid_for(nvox, 256), 256, 0, st>>>(t, v, a.nx, a.ny, a.nz, a.psf_sep, a.psf_k);
    }
    return vol;
  }

  void spread(const T* att, T* vol) {
    NRGB_LAUNCH_SCOPE("k_spread", st);
    k_spread<T><<<rays(), 128, 0, st>>>(a.sino + nxy * cam0, att, vol, grid);
  }

  // rotate the group's volumes back and add them to the output
  void gather(const T* src, T bg) {
    NRGB_LAUNCH_SCOPE("k_resample_sum", st);
    k_resample_sum<T><<<blocks(8, 1), dim3(32, 8), 0, st>>>(src, a.out, n, cam0 == 0, a.truncate && last(), bg, grid,
                                                            matrices(true));
  }
};

// et_project (emission-lib/_et.cpp:218-281): per camera rotate activity and
// mu, PSF, attenuated line integral, truncation (:283-292).
template <class T>
int general_project_t(const GeneralArgsT<T>& a, cudaStream_t st) {
  General<T> p(a, st);
  p.choose_layout();
  const T *act = p.source(a.act, 0), *att = p.source(a.att, 1);
  return p.groups([&] {
    p.rotate(act, a.ws_act, a.bg, att, a.ws_att, a.bg_att);
    const T* v = a.act ? p.convolve(a.ws_act, a.ws_tmp) : nullptr;
    NRGB_LAUNCH_SCOPE("k_line_integral", st);
    k_line_integral<T><<<p.rays(), 128, 0, st>>>(v, a.att ? a.ws_att : nullptr, a.out + p.nxy * p.cam0, p.grid, a.bg,
                                                 a.truncate);
  });
}

// et_backproject (emission-lib/_et.cpp:415-499): per camera rotate mu, spread
// the attenuated plane, PSF, rotate back with the inverse matrix, accumulate.
template <class T>
int general_backproject_t(const GeneralArgsT<T>& a, cudaStream_t st) {
  General<T> p(a, st);
  p.choose_layout();
  const T* att = p.source(a.att, 0);
  return p.groups([&] {
    p.rotate(nullptr, nullptr, T(0), att, a.ws_att, a.bg_att);
    p.spread(a.att ? a.ws_att : nullptr, a.ws_act);
    p.gather(p.convolve(a.ws_act, a.ws_tmp), a.bg);
  });
}

}  // namespace

int general_group(size_t nvox, size_t element, int ncam) {
  const size_t most = kGeneralScratch / (3 * element * std::max<size_t>(nvox, 1));
  return static_cast<int>(std::max<size_t>(1, std::min<size_t>({most, static_cast<size_t>(kGeneralGroup),
                                                                static_cast<size_t>(std::max(1, ncam))})));
}

// et_project_partial_gpu (emission-lib/_et.cpp:2106-2436): per camera rotate
// activity (bg) and mu (bg_att), PSF, partial-sum line integral; with
// do_rotate the camera's partial-sum volume is rotated back to the image frame
// (-theta, ZYX, background bg, :2373-2404).  partial: [ncam][nz][ny][nx].
int general_project_partial(const GeneralArgs& a, const float* bg_image, float* partial, int do_rotate,
                            cudaStream_t st) {
  General<float> p(a, st);
  const int s = p.groups([&] {
    p.rotate(a.act, a.ws_act, a.bg, a.att, a.ws_att, a.bg_att);
    const float* v = a.act ? p.convolve(a.ws_act, a.ws_tmp) : nullptr;
    float* dst = partial + p.nvox * p.cam0;
    // the sums to rotate back go where the scan no longer reads
    float* sums = v == a.ws_tmp ? a.ws_act : a.ws_tmp;
    {
      NRGB_LAUNCH_SCOPE("k_line_partial", st);
      k_line_partial<<<p.rays(), 128, 0, st>>>(v, a.att ? a.ws_att : nullptr, bg_image, a.out + p.nxy * p.cam0,
                                               do_rotate ? sums : dst, a.nx, a.ny, a.nz, a.bg);
    }
    for (int g = 0; do_rotate && g < p.n; ++g) {
      AffineSetT<float> m = {};
      std::copy(a.geom_host[p.cam0 + g].bwd, a.geom_host[p.cam0 + g].bwd + 12, m.m[0]);
      NRGB_LAUNCH_SCOPE("k_resample", st);
      k_resample<float><<<p.blocks(8, 1), dim3(32, 8), 0, st>>>(sums + p.nvox * g, dst + p.nvox * g, a.bg, nullptr,
                                                                nullptr, 0.0f, p.grid, m);
    }
  });
  if (s == kOk && a.truncate) launch_truncate(a.out, p.nxy * a.ncam, st);
  return cudaGetLastError() == cudaSuccess ? s : kErrKernel;
}

int general_project(const GeneralArgs& a, cudaStream_t st) { return general_project_t<float>(a, st); }
int general_backproject(const GeneralArgs& a, cudaStream_t st) { return general_backproject_t<float>(a, st); }
int general_project64(const GeneralArgs64& a, cudaStream_t st) { return general_project_t<double>(a, st); }
int general_backproject64(const GeneralArgs64& a, cudaStream_t st) { return general_backproject_t<double>(a, st); }

namespace {

void scatter(const General<float>& p, const float* src) {
  NRGB_LAUNCH_SCOPE("k_scatter", p.st);
  k_scatter<<<p.blocks(8, p.n), dim3(32, 8), 0, p.st>>>(src, p.a.out, p.a.nx, p.a.ny, p.a.nz, p.matrices(false));
}

}  // namespace

// Exact transpose of general_project for fixed mu (bg terms dropped: the
// transpose of the projector's linear part): spread, transposed PSF
// (correlation), transposed trilinear scatter.
int general_adjoint(const GeneralArgs& a, cudaStream_t st) {
  General<float> p(a, st);
  cudaMemsetAsync(a.out, 0, p.nvox * sizeof(float), st);
  return p.groups([&] {
    p.rotate(nullptr, nullptr, 0.0f, a.att, a.ws_att, a.bg_att);
    p.spread(a.att ? a.ws_att : nullptr, a.ws_act);
    scatter(p, p.convolve<true>(a.ws_act, a.ws_tmp));
  });
}

// Gradient of sum(g * project(act, mu)) with respect to mu (a.sino = g),
// into a.out.  Per camera: rotate activity and mu, PSF on the activity,
// k_dmu_scan, transposed trilinear scatter of the rotated-frame gradient.
int general_dmu(const GeneralArgs& a, cudaStream_t st) {
  General<float> p(a, st);
  cudaMemsetAsync(a.out, 0, p.nvox * sizeof(float), st);
  return p.groups([&] {
    p.rotate(a.act, a.ws_act, a.bg, a.att, a.ws_att, a.bg_att);
    const float* v = p.convolve(a.ws_act, a.ws_tmp);
    float* d = v == a.ws_tmp ? a.ws_act : a.ws_tmp;
    {
      NRGB_LAUNCH_SCOPE("k_dmu_scan", st);
      k_dmu_scan<<<p.rays(), 128, 0, st>>>(v, a.ws_att, a.sino + p.nxy * p.cam0, d, a.nx, a.ny, a.nz, a.bg);
    }
    scatter(p, d);
  });
}

int general_gradient(const GeneralArgs& a, cudaStream_t st) {
  General<float> p(a, st);
  return p.groups([&] {
    p.rotate(a.act, a.ws_act, a.bg, a.att, a.ws_att, a.bg_att);
    {
      NRGB_LAUNCH_SCOPE("k_grad_scan", st);
      k_grad_scan<<<p.rays(), 128, 0, st>>>(a.ws_act, a.ws_att, a.sino + p.nxy * p.cam0, a.ws_tmp, a.nx, a.ny, a.nz);
    }
    p.gather(p.convolve(a.ws_tmp, a.ws_act), a.bg);
  });
}

namespace {

// Per-slice 2D true convolution with kernel slice z (centre ((kx-1)/2,
// (ky-1)/2)), the image clamped to its border outside; terms in (j, i) order,
// multiply and add rounded separately (the oracle's order and rounding).
__global__ void k_convolve2d(const float* __restrict__ src, float* __restrict__ dst, int nx, int ny,
                             const float* __restrict__ psf, int kx, int ky) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int z = blockIdx.z;
  if (x >= nx || y >= ny) return;
  const int cx = (kx - 1) / 2, cy = (ky - 1) / 2;
  const float* k = psf + static_cast<size_t>(z) * kx * ky;
  const float* img = src + static_cast<size_t>(z) * nx * ny;
  float acc = 0.0f;
  for (int j = 0; j < ky; ++j) {
    const int yy = min(max(y + cy - j, 0), ny - 1);
    const float* row = img + static_cast<size_t>(yy) * nx;
    for (int i = 0; i < kx; ++i) {
      const int xx = min(max(x + cx - i, 0), nx - 1);
      acc = __fadd_rn(acc, __fmul_rn(__ldg(k + i + kx * j), __ldg(row + xx)));
    }
  }
  dst[(static_cast<size_t>(z) * ny + y) * nx + x] = acc;
}

}  // namespace

int general_convolve2d(const float* src, float* dst, int nx, int ny, int nz, const float* psf, int kx, int ky,
                       cudaStream_t st) {
  const dim3 block(32, 8), grid((nx + 31) / 32, (ny + 7) / 8, nz);
  { NRGB_LAUNCH_SCOPE("k_convolve2d", st); k_convolve2d<<<grid, block, 0, st>>>(src, dst, nx, ny, psf, kx, ky); }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

int general_rotate(const float* src, float* dst, int nx, int ny, int nz, const float* m12, float bg, cudaStream_t st) {
  GeneralArgs a;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  AffineSetT<float> m = {};
  std::copy(m12, m12 + 12, m.m[0]);
  NRGB_LAUNCH_SCOPE("k_resample", st);
  k_resample<float><<<General<float>(a, st).blocks(8, 1), dim3(32, 8), 0, st>>>(src, dst, bg, nullptr, nullptr, 0.0f,
                                                                                Grid{nx, ny, nz, 0}, m);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

}  // namespace nrgb
