// Per-call projector kernels and their launcher, instantiated per PSF
// radius in separate translation units (et_yg_proj_r*.cu) so that the
// projector's many instantiations compile in parallel.
#pragma once

#include "et_yg_device.cuh"

#include <functional>

namespace nrgb {

// Depth slabs (cluster size 2, 4, 6, 8 or 16) of the projector for `items`
// cluster work items of nz depth planes: the least planes per slab times the
// rounds of resident clusters (clusters(s): how many of size s fit at once,
// cudaOccupancyMaxActiveClusters).  A round is weighted by the CTAs that share
// an SM -- a plane step of 2 (3) of them takes 1.28 (1.7) times as long as of
// one alone, 1.5 times with mirror units; measured at 128^3 -- and two planes
// stand for a slab's start and merge.  Against the count for three waves of
// CTAs: 128^3 x 30 cameras of a half-turn 258 -> 196 us (6 slabs), x 15 125 ->
// 114, 256^3 x 18 PSF 15 1.66 -> 1.25 ms, 64^3 x 60 plain 25 -> 19 us (8),
// 32^3 x 8 27 -> 19 us (8; 16: 15 us, but its slabs of two planes cost accuracy,
// 1.0e-7 -> 1.3e-7, so 16 needs 128 planes); 128^3 x 120 keeps 4 (0.504 ms; 8: 0.519).
// Left out: 5 and 7 (128^3 x 15: 131 and 136 us although they fit one round),
// with mirror units 6 (96 x 96 x 80 x 90: 206 us, 8: 200), and fewer than the
// three-wave count (6 or 8 at least): longer float sums for nothing more than
// 7 % (96 x 96 x 80 x 90 with 2 slabs, error 2.4e-7 -> 3.2e-7).
int project_slabs(int items, int nz, int ctas_per_sm, bool pair, const std::function<int(int)>& clusters);
// Clusters of `cluster` CTAs of a kernel that are resident at once (0: none);
// asked of the driver once per device, kernel and shape.
int max_active_clusters(const void* kernel, int cluster, int threads, size_t smem);

namespace {

// One work item per cluster of a.pslabs CTAs (the cluster size is set at
// launch): blockIdx.x / a.pslabs = (unit, x-tile); a unit is a camera and,
// with a.units, its mirror camera.  CTAS: CTAs per SM the kernel is compiled
// for -- 3 (80 registers, more warps to hide the gathers' latency) where
// three tiles fit in shared memory and the storage is float32, else 2 (128
// registers; bfloat16 needs them for its Kahan compensations).
template <int R, bool PSF, bool ATT, class V, int CTAS, bool PAIR, int L>
__global__ void __launch_bounds__(32 * kW, CTAS) k_project_yg(const YgArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int item = blockIdx.x / a.pslabs;
  const int u = item / ntile;
  const int2 uc = PAIR ? a.units[u] : make_int2(u, -1);
  project_item<R, PSF, ATT, V, PAIR, false, L>(a, uc.x, uc.y, (item % ntile) * kTX<L>, smem);
}

// The same with the separated PSF in the kernel parameters (PsfTable).
template <int R, bool ATT, class V, int CTAS, bool PAIR, int L>
__global__ void __launch_bounds__(32 * kW, CTAS) k_project_ptab_yg(const YgArgs a, const __grid_constant__ PsfTable t) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int item = blockIdx.x / a.pslabs;
  const int u = item / ntile;
  const int2 uc = PAIR ? a.units[u] : make_int2(u, -1);
  project_item<R, true, ATT, V, PAIR, true, L>(a, uc.x, uc.y, (item % ntile) * kTX<L>, smem, t.c);
}

// L lanes per column (L < 32: narrow row windows; no PSF, or the PSF in the
// kernel parameters).
template <int R, int L>
int launch_project_lanes(const YgArgs& a_in, cudaStream_t st, int* slabs_used) {
  YgArgs a = a_in;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const bool psf = a.psf != nullptr;
  const bool bf16 = a.storage == kStorageBF16;
  const bool ptab = psf_in_parameters<R>(a);
  // mirror cameras: float32 always; bfloat16 (Kahan compensations in shared
  // memory) where two CTAs per SM still fit
  bool pair = a.units != nullptr && a.nunits > 0;
  size_t smem = project_smem_bytes<R, L>(psf && !ptab ? a.nz : 0, pair, bf16);
  if (pair && bf16 && 2 * (smem + kYBufBytes<L> + 1024) > 228 * 1024) {
    pair = false;
    smem = project_smem_bytes<R, L>(psf && !ptab ? a.nz : 0, false, true);
  }
  const int nunits = pair ? a.nunits : a.ncam;
  // three CTAs per SM need three tiles (plus 1 KB reserved each) in the 228 KB
  const bool three = 3 * (smem + kYBufBytes<L> + 1024) <= 228 * 1024;
  // carry split: the slab's halves must be the backprojector's slabs of twice
  // the count, with at most 8 of them
  auto split_ok = [&](int p) {
    return a.carry_out && a.mu && a.carry_split && 2 * p <= 8 &&
           (a.nz + p - 1) / p == 2 * ((a.nz + 2 * p - 1) / (2 * p));
  };
  // one cluster of a.pslabs CTAs per (unit, x-tile); 16 is a non-portable
  // cluster size: it falls back to 8 where the kernel cannot be resident so
  bool launch_err = false;
  auto launch = [&](auto k, auto&&... extra) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(32 * kW);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto clusters = [&](int s) {
      return max_active_clusters(reinterpret_cast<const void*>(k), s, 32 * kW, smem);
    };
    if (a.pslabs < 2 || (a.pslabs > 8 && a.pslabs != 16))
      a.pslabs = project_slabs(nunits * ntile, a.nz, three && !bf16 && !pair ? 3 : 2, pair || a.carry_out, clusters);
    else if (a.pslabs == 16 && clusters(16) < 1)
      a.pslabs = 8;
    a.carry_split = split_ok(a.pslabs) ? 1 : 0;
    cfg.gridDim = dim3(nunits * ntile * a.pslabs);
    attr[0].val.clusterDim.x = a.pslabs;
    if (slabs_used) {
      slabs_used[0] = a.carry_split ? 2 * a.pslabs : a.pslabs;
      slabs_used[1] = a.pslabs;
    }
    NRGB_LAUNCH_SCOPE("k_project_yg", st);
    if (cudaLaunchKernelEx(&cfg, k, a, extra...) != cudaSuccess) launch_err = true;
  };
  auto go = [&](auto k) { launch(k); };
  auto go_tab = [&](auto k) {
    static thread_local PsfTable table;
    std::memcpy(table.c, a.psf_host, sizeof(float) * a.nz * 2 * (2 * R + 1));
    launch(k, table);
  };
  auto pick = [&](auto v, auto ctas, auto paired) {
    using V = decltype(v);
    constexpr int C = decltype(ctas)::value;
    constexpr bool P = decltype(paired)::value;
    if (psf && ptab) {
      if (a.mu) go_tab(k_project_ptab_yg<R, true, V, C, P, L>);
      else go_tab(k_project_ptab_yg<R, false, V, C, P, L>);
    } else if (psf) {
      if constexpr (L == 32) {
        if (a.mu) go(k_project_yg<R, true, true, V, C, P, L>);
        else go(k_project_yg<R, true, false, V, C, P, L>);
      }
    } else if constexpr (R == 0) {
      if (a.mu) go(k_project_yg<0, false, true, V, C, P, L>);
      else go(k_project_yg<0, false, false, V, C, P, L>);
    }
  };
  using Off = std::false_type;
  using On = std::true_type;
  // the mirror-camera item needs the 128-register budget of two CTAs per SM
  if (bf16 && pair)
    pick(__nv_bfloat16(), std::integral_constant<int, 2>(), On());
  else if (bf16)
    pick(__nv_bfloat16(), std::integral_constant<int, 2>(), Off());
  else if (pair)
    pick(0.0f, std::integral_constant<int, 2>(), On());
  else if (three)
    pick(0.0f, std::integral_constant<int, 3>(), Off());
  else
    pick(0.0f, std::integral_constant<int, 2>(), Off());
  return cudaGetLastError() == cudaSuccess && !launch_err ? kOk : kErrKernel;
}

}  // namespace

// Launch the per-call projector of PSF radius R (R = 0: no PSF) for one row
// window; explicitly instantiated in et_yg_proj_r*.cu.  slabs_used (if
// non-null) receives the slab count of the carries written to a.carry_out and
// the depth-slab count of the launch.
template <int R>
int launch_project_R(const YgArgs& a, cudaStream_t st, int* slabs_used) {
  if (!a.psf || psf_in_parameters<R>(a)) {
    if (a.lanes == 8) return launch_project_lanes<R, 8>(a, st, slabs_used);
    if (a.lanes == 16) return launch_project_lanes<R, 16>(a, st, slabs_used);
  }
  return launch_project_lanes<R, 32>(a, st, slabs_used);
}

}  // namespace nrgb
