// Fused y-gantry gradient of L = sum(g * project(activity, mu)) with respect
// to mu (the d/dmu of the differentiable projector; the reference's own
// attenuation gradient, emission-lib/_et.cpp:1679-1924, is a different
// quantity and stays in et_yg_grad.cu).
//
// For one ray of camera c, p = sum_z v_z exp(-T_z) with v the PSF-convolved
// rotated activity and T_z the inclusive sum of the rotated mu, so
//   dL/dmu_rot(z) = -g * S(z),  S(z) = sum_{z' >= z} v_z' exp(-T_z'),
// and dL/dmu is its transposed bilinear scatter into the volume.  Two kernels
// per group of units:
//   k_dmu_terms_yg: the projector's walk (a camera and its mirror camera from
//     one set of samples), leaving the rays' terms in the group scratch and two
//     coefficients per ray and depth slab (project_item, TERMS);
//   k_dmu_scatter_yg: the terms summed along the ray and -g S(z) scattered at
//     each camera's own positions.
// 128^3 x 120, PSF 11: 1.36 ms (terms 2 x 0.40, scatter 2 x 0.27), against 1.96 ms
// of one kernel whose second walk recomputed samples and PSF of every camera
// alone.  The terms (4 bytes per voxel and camera, 1 GB written and read) cost
// less than that walk.  Reading them back in the first kernel's own CTAs
// took 1.27 ms with one scatter per unit at the first camera's positions, but
// the error of a noisy g's gradient rose from 8.1e-6 to 1.0e-5; every camera
// alone with both kernels: 1.54 ms.
#pragma once

#include "et_yg_project_kernels.cuh"

namespace nrgb {
namespace {

template <int R, bool PSF, bool PAIR, int CTAS, int L>
__global__ void __launch_bounds__(32 * kW, CTAS) k_dmu_terms_yg(const YgArgs a_in) {
  extern __shared__ __align__(16) unsigned char smem[];
  YgArgs a = a_in;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int item = blockIdx.x / a.pslabs;
  a.vol0 = item / ntile;
  const int2 uc = PAIR ? a.units[a.cam0 + a.vol0] : make_int2(a.cam0 + a.vol0, -1);
  project_item<R, PSF, true, float, PAIR, false, L, L, true>(a, uc.x, uc.y, (item % ntile) * kTX<L>, smem);
}

template <int R, bool PAIR, int CTAS, int L>
__global__ void __launch_bounds__(32 * kW, CTAS)
    k_dmu_terms_ptab_yg(const YgArgs a_in, const __grid_constant__ PsfTable t) {
  extern __shared__ __align__(16) unsigned char smem[];
  YgArgs a = a_in;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int item = blockIdx.x / a.pslabs;
  a.vol0 = item / ntile;
  const int2 uc = PAIR ? a.units[a.cam0 + a.vol0] : make_int2(a.cam0 + a.vol0, -1);
  project_item<R, true, true, float, PAIR, true, L, L, true>(a, uc.x, uc.y, (item % ntile) * kTX<L>, smem, t.c);
}

// Terms of units (or cameras) [a.cam0, a.cam0 + n); *slabs: the depth slabs of a.coef.
template <int R, int L>
int launch_dmu_terms(const YgArgs& a_in, int n, int* slabs, cudaStream_t st) {
  YgArgs a = a_in;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const bool psf = a.psf != nullptr;
  const bool ptab = psf_in_parameters<R>(a);
  const bool pair = a.units != nullptr;
  const size_t smem = project_smem_bytes<R, L>(psf && !ptab ? a.nz : 0, pair, false);
  const bool three = !pair && 3 * (smem + kYBufBytes<L> + 1024) <= 228 * 1024;
  bool launch_err = false;
  auto launch = [&](auto k, auto&&... extra) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    auto clusters = [&](int s) {
      return s > kDmuSlabs ? 0 : max_active_clusters(reinterpret_cast<const void*>(k), s, 32 * kW, smem);
    };
    a.pslabs = std::min(project_slabs(n * ntile, a.nz, three ? 3 : 2, pair, clusters), kDmuSlabs);
    *slabs = a.pslabs;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n * ntile * a.pslabs);
    cfg.blockDim = dim3(32 * kW);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.pslabs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NRGB_LAUNCH_SCOPE("k_dmu_terms_yg", st);
    if (cudaLaunchKernelEx(&cfg, k, a, extra...) != cudaSuccess) launch_err = true;
  };
  auto pick = [&](auto paired, auto ctas) {
    constexpr bool P = decltype(paired)::value;
    constexpr int C = decltype(ctas)::value;
    if (ptab) {
      static thread_local PsfTable table;
      std::memcpy(table.c, a.psf_host, sizeof(float) * a.nz * 2 * (2 * R + 1));
      launch(k_dmu_terms_ptab_yg<R, P, C, L>, table);
    } else if (psf) {
      if constexpr (L == 32) launch(k_dmu_terms_yg<R, true, P, C, L>);
    } else if constexpr (R == 0) {
      launch(k_dmu_terms_yg<0, false, P, C, L>);
    }
  };
  if (pair) pick(std::true_type(), std::integral_constant<int, 2>());
  else if (three) pick(std::false_type(), std::integral_constant<int, 3>());
  else pick(std::false_type(), std::integral_constant<int, 2>());
  return cudaGetLastError() == cudaSuccess && !launch_err ? kOk : kErrKernel;
}

}  // namespace

// With the window's lane count; explicitly instantiated in et_yg_dmu_r*.cu.
template <int R>
int launch_dmu_R(const YgArgs& a, int n, int* slabs, cudaStream_t st) {
  if (!a.psf || psf_in_parameters<R>(a)) {
    if (a.lanes == 8) return launch_dmu_terms<R, 8>(a, n, slabs, st);
    if (a.lanes == 16) return launch_dmu_terms<R, 16>(a, n, slabs, st);
  }
  return launch_dmu_terms<R, 32>(a, n, slabs, st);
}

}  // namespace nrgb
