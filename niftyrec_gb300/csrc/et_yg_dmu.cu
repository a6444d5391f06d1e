// Fused y-gantry gradient with respect to mu: the scatter of the rays'
// gradients, and the dispatch by PSF radius, row windows and camera groups
// (first kernel in et_yg_dmu_kernels.cuh).
#include "et_yg_device.cuh"

namespace nrgb {

template <int R>
int launch_dmu_R(const YgArgs& a, int n, int* slabs, cudaStream_t st);  // et_yg_dmu_kernels.cuh

namespace {

// One lane group per (camera, depth slab, column): the column's terms summed in
// depth order give -g S(z) = A + B * Pre(z), scattered with the projector's
// bilinear weights of that camera (a mirror camera's terms lie in its unit's
// frame; they are scattered at its own positions, whose rounding the scatter
// of a noisy g would show).  Consecutive planes of a column step through the (x, z)
// grid by at most one cell either way, so the four nodes of the current cell
// are summed in registers and leave with one vector reduction each when the
// walk moves off them (about 2.3 reductions a plane instead of 4).  With a.det
// the gradient replaces the term for the transposed gather.
// Bound by the reductions and by reading the terms, hence as many warps as fit.
template <int L>
__global__ void __launch_bounds__(256, 3) k_dmu_scatter_yg(const YgArgs a, int n) {
  const int lane = threadIdx.x % L;
  const long long item = blockIdx.x * static_cast<long long>(256 / L) + threadIdx.x / L;
  if (item >= static_cast<long long>(a.units ? 2 * n : n) * a.pslabs * a.nx) return;  // whole lane groups
  const unsigned group_mask = L == 32 ? kFull : ((1u << (L & 31)) - 1u) << (threadIdx.x % 32 / L * L);
  const int x = static_cast<int>(item % a.nx);
  const int slab = static_cast<int>(item / a.nx % a.pslabs);
  int g = static_cast<int>(item / a.nx / a.pslabs);  // the mates' volumes after the first cameras'
  const bool mate = g >= n;
  if (mate) g -= n;
  const int2 uc = a.units ? a.units[a.cam0 + g] : make_int2(a.cam0 + g, -1);
  const int cam = mate ? uc.y : uc.x;
  if (cam < 0) return;
  if (mate) g += a.group;
  const int yb = lane * 4;
  const bool ok = lane_rows_ok(a, yb) && lane_writes(a, yb);
  const int zper = (a.nz + a.pslabs - 1) / a.pslabs;
  const int zbeg = slab * zper, zend = min(a.nz, zbeg + zper);
  const CamRows cr = cam_rows(a.geom[cam].fwd);
  float* term = a.temp + (static_cast<size_t>(g) * a.nz * a.nx + x) * a.cs + yb;
  float* out = a.out + a.row0 + yb;
  const size_t plane = static_cast<size_t>(a.nx) * a.cs;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 A = zero, B = zero;
  if (ok) {
    const float* cf = a.coef + ((static_cast<size_t>(g) * a.pslabs + slab) * a.nx + x) * 2 * a.cs + yb;
    A = *reinterpret_cast<const float4*>(cf);
    B = *reinterpret_cast<const float4*>(cf + a.cs);
  }
  // nodes of the current cell: n00 = (X, Z), n10 = (X + 1, Z), n01, n11
  float4 pre = zero, n00 = zero, n10 = zero, n01 = zero, n11 = zero;
  int X = 0, Z = 0;
  auto flush = [&](const float4& v, int nx, int nz) {
    if (ok && nx >= 0 && nx < a.nx && nz >= 0 && nz < a.nz)
      red4(out + (static_cast<size_t>(nz) * a.nx + nx) * a.cy, v);
  };
  for (int zc = zbeg; zc < zend; zc += L) {
    // lane q: position of plane zc + q (make_tap's arithmetic)
    const float fx = static_cast<float>(mate ? a.nx - 1 - x : x);
    const float fz = static_cast<float>(mate ? a.nz - 1 - zc - lane : zc + lane);
    const float px = fa(fa(fm(cr.m00, fx), fm(cr.m02, fz)), cr.m03);
    const float pz = fa(fa(fm(cr.m20, fx), fm(cr.m22, fz)), cr.m23);
    const int pxs = static_cast<int>(floorf(px)), pzs = static_cast<int>(floorf(pz));
    float prx = __fsub_rn(px, static_cast<float>(pxs)), prz = __fsub_rn(pz, static_cast<float>(pzs));
    if (prx < 0.0f) prx = 0.0f;
    if (prz < 0.0f) prz = 0.0f;
    const int m = min(L, zend - zc);
    for (int h = 0; h < m; h += 4) {
      float4 w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        w[q] = ok && h + q < m ? *reinterpret_cast<const float4*>(term + plane * (zc + h + q)) : zero;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (h + q >= m) break;
        float4 d = A, upto = pre;
        add4p(pre, w[q]);
        if (mate) upto = pre;
        fma4p(d, B, upto);
        if (a.det) {  // uniform over the launch
          if (ok) *reinterpret_cast<float4*>(term + plane * (zc + h + q)) = d;
          continue;
        }
        const int xs = __shfl_sync(group_mask, pxs, h + q, L), zs = __shfl_sync(group_mask, pzs, h + q, L);
        const float rx = __shfl_sync(group_mask, prx, h + q, L), rz = __shfl_sync(group_mask, prz, h + q, L);
        if (xs != X || zs != Z) {  // uniform over the lane group
          const int dx = xs - X, dz = zs - Z;
          if (zc + h + q == zbeg) {
            // nothing summed yet
          } else if (dx > 1 || dx < -1 || dz > 1 || dz < -1) {
            flush(n00, X, Z);
            flush(n10, X + 1, Z);
            flush(n01, X, Z + 1);
            flush(n11, X + 1, Z + 1);
            n00 = n10 = n01 = n11 = zero;
          } else {
            // in x first: the nodes left behind go out, the shared ones move over
            if (dx == 1) {
              flush(n00, X, Z);
              flush(n01, X, Z + 1);
              n00 = n10;
              n01 = n11;
              n10 = n11 = zero;
            } else if (dx == -1) {
              flush(n10, X + 1, Z);
              flush(n11, X + 1, Z + 1);
              n10 = n00;
              n11 = n01;
              n00 = n01 = zero;
            }
            // then in z; a node that came in empty with the step in x (x + 1
            // after dx = 1, x after dx = -1) has nothing to send
            if (dz == 1) {
              if (dx != -1) flush(n00, xs, Z);
              if (dx != 1) flush(n10, xs + 1, Z);
              n00 = n01;
              n10 = n11;
              n01 = n11 = zero;
            } else if (dz == -1) {
              if (dx != -1) flush(n01, xs, Z + 1);
              if (dx != 1) flush(n11, xs + 1, Z + 1);
              n01 = n00;
              n11 = n10;
              n00 = n10 = zero;
            }
          }
          X = xs;
          Z = zs;
        }
        const float wx0 = __fsub_rn(1.0f, rx), wz0 = __fsub_rn(1.0f, rz);
        // a corner without weight takes nothing: d may be infinite (uniform tests,
        // 128^3 x 120: 0.259 -> 0.266 ms a launch)
        const float w00 = wx0 * wz0, w10 = rx * wz0, w01 = wx0 * rz, w11 = rx * rz;
        if (w00 != 0.0f) axpy4(n00, w00, d);
        if (w10 != 0.0f) axpy4(n10, w10, d);
        if (w01 != 0.0f) axpy4(n01, w01, d);
        if (w11 != 0.0f) axpy4(n11, w11, d);
      }
    }
  }
  if (!a.det && zbeg < zend) {
    flush(n00, X, Z);
    flush(n10, X + 1, Z);
    flush(n01, X, Z + 1);
    flush(n11, X + 1, Z + 1);
  }
}

int launch_scatter(const YgArgs& a, int n, cudaStream_t st) {
  const long long columns = static_cast<long long>(a.units ? 2 * n : n) * a.pslabs * a.nx;
  auto go = [&](auto lanes) {
    constexpr int L = decltype(lanes)::value;
    NRGB_LAUNCH_SCOPE("k_dmu_scatter_yg", st);
    k_dmu_scatter_yg<L><<<static_cast<unsigned>((columns * L + 255) / 256), 256, 0, st>>>(a, n);
  };
  const int lanes = column_lanes(a.ny);
  if (lanes == 8) go(std::integral_constant<int, 8>());
  else if (lanes == 16) go(std::integral_constant<int, 16>());
  else go(std::integral_constant<int, 32>());
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

int dmu_by_radius(int R, const YgArgs& a, int n, int* slabs, cudaStream_t st) {
  switch (R) {
    case 0: return launch_dmu_R<0>(a, n, slabs, st);
    case 1: return launch_dmu_R<1>(a, n, slabs, st);
    case 2: return launch_dmu_R<2>(a, n, slabs, st);
    case 3: return launch_dmu_R<3>(a, n, slabs, st);
    case 4: return launch_dmu_R<4>(a, n, slabs, st);
    case 5: return launch_dmu_R<5>(a, n, slabs, st);
    case 6: return launch_dmu_R<6>(a, n, slabs, st);
    case 7: return launch_dmu_R<7>(a, n, slabs, st);
    default: return kErrParameters;
  }
}

// Units (or cameras) per launch: as many as fit two scratch slots of the
// backprojector (its work space for the same cameras is larger), with mirror
// units two volumes each.
int dmu_group(int n, int ncam, int group, bool pair) {
  const int slot = std::max(1, std::min(group, ncam));
  return yg_even_group(n, pair ? slot : 2 * slot);
}

}  // namespace

int yg_dmu(const YgArgs& a_in, cudaStream_t st) {
  YgArgs a = a_in;
  if (!a.mu || !a.act || !a.sino || !a.out || !a.work) return kErrParameters;
  const int R = a.psf ? (a.psf_k - 1) / 2 : 0;
  // the transposed gather of the deterministic form reads one volume per
  // camera in the camera's own frame: no mirror units there
  const bool pair = !a.det && a.units && a.nunits > 0;
  if (!pair) a.units = nullptr;
  const int units = pair ? a.nunits : a.ncam;
  const int group = dmu_group(units, a.ncam, a.group, pair);
  a.coef = a.work + static_cast<size_t>(pair ? 2 * group : group) * a.nz * a.nx * scratch_rows(a.ny);
  a.group = group;
  if (!a.det) {
    const size_t full = static_cast<size_t>(a.nz) * a.nx * a.cy;
    if (cudaMemsetAsync(a.out, 0, sizeof(float) * full, st) != cudaSuccess) return kErrKernel;
  }
  for (const Window& w : call_windows(a, R)) {
    YgArgs b = windowed(a, w);
    b.temp = a.work;
    for (int c0 = 0; c0 < units; c0 += group) {
      const int n = std::min(group, units - c0);
      b.cam0 = c0;
      int s = dmu_by_radius(R, b, n, &b.pslabs, st);
      if (s == kOk) s = launch_scatter(b, n, st);
      if (s != kOk) return s;
      if (a.det) yg_tgather(b, c0, n, 0, st);
    }
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

size_t yg_dmu_workspace(int nx, int ny, int nz, int ncam, int group) {
  const size_t column = sizeof(float) * static_cast<size_t>(nx) * scratch_rows(ny);
  return column * 2 * std::max(1, std::min(group, ncam)) * (static_cast<size_t>(nz) + 2 * kDmuSlabs);
}

}  // namespace nrgb
