// Fused y-gantry projector: dispatch of the per-call kernels by PSF radius,
// the persistent batched projector, and the public entry points.
#include "et_yg_device.cuh"

#include <cmath>
#include <functional>
#include <tuple>

namespace nrgb {

template <int R>
int launch_project_R(const YgArgs& a, cudaStream_t st, int* slabs_used);  // et_yg_project_kernels.cuh

// ------------------------------------------------------------- dispatch
double slab_rounds(double rounds, double ctas, int ctas_per_sm) {
  static const double step[2][3] = {{1.0, 1.5, 1.5}, {1.0, 1.28, 1.7}};
  const double* t = step[ctas_per_sm > 2 ? 1 : 0];
  const int most = ctas_per_sm > 2 ? 3 : 2;
  const double full = std::floor(rounds), rest = rounds - full;
  double cost = full * t[most - 1];
  if (rest > 0) {
    const int per_sm = static_cast<int>(std::ceil(ctas * rest / rounds / sm_count()));
    cost += t[std::min(std::max(per_sm, 1), most) - 1];
  }
  return cost;
}

namespace {

// The fewest of 2, 4, 8 (16 with 128 planes) slabs that give three waves of
// CTAs; four where one round of them holds every item.
int three_wave_slabs(int items, int nz, int ctas_per_sm) {
  const int slots = sm_count() * ctas_per_sm;
  if (items * 4 <= slots) return 4;
  const int most = nz >= 128 ? 16 : 8;
  for (int s = 2; s < most; s *= 2)
    if (items * s >= 3 * slots) return s;
  return most;
}

}  // namespace

int project_slabs(int items, int nz, int ctas_per_sm, bool pair, const std::function<int(int)>& clusters) {
  const int waves = three_wave_slabs(items, nz, ctas_per_sm);
  const int least = std::min(waves, pair ? 8 : 6);
  int best = least;
  double cost = 0.0;
  for (int s : {2, 4, 6, 8, 16}) {
    if (s < least || (pair && s == 6) || (s == 16 && nz < 128)) continue;
    const int resident = clusters(s);
    if (resident < 1) continue;
    const double c = ((nz + s - 1) / s + 2) *
                     slab_rounds(static_cast<double>(items) / resident, static_cast<double>(items) * s, ctas_per_sm);
    if (cost == 0.0 || c < cost) {
      best = s;
      cost = c;
    }
  }
  return best;
}

int yg_spread_slabs(int items, int nz, int ctas_per_sm) {
  int best = kSlabsB;
  double cost = 0.0;
  for (int s = kSlabsB; s > 12; --s) {
    const double ctas = static_cast<double>(items) * s;
    const double c =
        ((nz + s - 1) / s + 1) * slab_rounds(ctas / (sm_count() * ctas_per_sm), ctas, ctas_per_sm);
    if (cost == 0.0 || c < cost) {
      best = s;
      cost = c;
    }
  }
  return best;
}

int max_active_clusters(const void* kernel, int cluster, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, int, size_t>, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  const auto key = std::make_tuple(dev, kernel, cluster, threads, smem);
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if ((cluster > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  return known[key] = n;
}

namespace {

// Persistent projector over a batch of volumes: each cluster takes work items
// (volume, row window, camera, x-tile) from a global counter until none are
// left, so volumes of any size share the GPU in one launch.  The item number
// is drawn by the cluster's first thread and read by the other CTAs from its
// shared memory (double-buffered: the slot of item i is rewritten at item i+2,
// after the barriers of item i+1).
// CTAS: CTAs per SM the kernel is built for.  With mu 2 (128 registers): the
// three bodies of the lane counts spill 796 bytes at the 80 registers of 3 CTAs, and
// a step of 24 volumes takes 4.98 ms against 5.50.  Without mu nothing spills at
// 3 CTAs, taken where more of them are resident.
template <int R, bool PSF, bool ATT, int CTAS>
__global__ void __cluster_dims__(kSlabsP, 1, 1) __launch_bounds__(32 * kW, CTAS)
    k_project_batch_yg(const BatchStepDesc* __restrict__ descs, const BatchSel sel, int* __restrict__ counter) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_item[2];
  cg::cluster_group cluster = cg::this_cluster();
  const bool leader = cluster.block_rank() == 0 && threadIdx.x == 0;
  for (int it = 0;; ++it) {
    int* slot = &s_item[it & 1];
    if (leader) *slot = atomicAdd(counter, 1);
    cluster.sync();
    const int item = *cluster.map_shared_rank(slot, 0);
    if (item >= sel.total) {
      cluster.sync();  // rank 0's shared memory stays alive until every CTA has read it
      return;
    }
    int v = 0;
    while (v + 1 < sel.n && item >= sel.begin[v + 1]) ++v;
    const BatchStepDesc& d = descs[sel.desc[v]];
    int r = item - sel.begin[v], w = 0;
    while (w + 1 < d.nwin && r >= d.tiles[w] * d.proj.ncam) r -= d.tiles[w++] * d.proj.ncam;
    const int ntile = d.tiles[w];
    YgArgs a = d.proj;
    a.row0 = d.win[w][0];
    a.ny = d.win[w][1];
    a.out_lo = d.win[w][2];
    a.out_hi = d.win[w][3];
    const int cam = r / ntile, t = r % ntile;
    switch (d.lanes[w]) {  // uniform over the cluster
      case 8: project_item<R, PSF, ATT, float, false, false, 8, 8>(a, cam, -1, t * kTX<8>, smem); break;
      case 16: project_item<R, PSF, ATT, float, false, false, 16, 8>(a, cam, -1, t * kTX<16>, smem); break;
      default: project_item<R, PSF, ATT, float, false, false, 32, 8>(a, cam, -1, t * kTX<32>, smem);
    }
  }
}

int project_by_radius(int R, const YgArgs& a, cudaStream_t st, int* slabs_used) {
  switch (R) {
    case 0: return launch_project_R<0>(a, st, slabs_used);
    case 1: return launch_project_R<1>(a, st, slabs_used);
    case 2: return launch_project_R<2>(a, st, slabs_used);
    case 3: return launch_project_R<3>(a, st, slabs_used);
    case 4: return launch_project_R<4>(a, st, slabs_used);
    case 5: return launch_project_R<5>(a, st, slabs_used);
    case 6: return launch_project_R<6>(a, st, slabs_used);
    case 7: return launch_project_R<7>(a, st, slabs_used);
    default: return kErrParameters;
  }
}

// One launch of the batched projector, or with info only what that launch
// would be: {CTAs per SM the kernel is built for, its static shared memory and
// its local memory per thread in bytes, clusters launched}.
template <int R, bool PSF>
int launch_project_batch_R(const BatchStepDesc* d, const BatchSel& sel, bool att, int max_nz, int* counter,
                           cudaStream_t st, int* info) {
  // one launch runs windows of any lane count: the largest tile of the three
  const int planes = PSF ? max_nz : 0;
  const size_t smem =
      std::max({tile_smem_bytes<R, 32>(planes), tile_smem_bytes<R, 16>(planes), tile_smem_bytes<R, 8>(planes)});
  // persistent grid: the clusters that are resident at once
  auto clusters = [&](auto k) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    return max_active_clusters(reinterpret_cast<const void*>(k), kSlabsP, 32 * kW, smem);
  };
  auto go = [&](auto k, int ctas, int resident) {
    const int grid = resident > 0 ? resident : sm_count() * ctas / kSlabsP;
    if (info) {
      cudaFuncAttributes attr = {};
      if (cudaFuncGetAttributes(&attr, k) != cudaSuccess) return;
      info[0] = ctas;
      info[1] = static_cast<int>(attr.sharedSizeBytes);
      info[2] = static_cast<int>(attr.localSizeBytes);
      info[3] = grid;
      return;
    }
    NRGB_LAUNCH_SCOPE("k_project_batch_yg", st);
    k<<<grid * kSlabsP, 32 * kW, smem, st>>>(d, sel, counter);
  };
  if (att) {
    auto k = k_project_batch_yg<R, PSF, true, 2>;
    go(k, 2, clusters(k));
  } else {
    auto two = k_project_batch_yg<R, PSF, false, 2>;
    auto three = k_project_batch_yg<R, PSF, false, 3>;
    const int n2 = clusters(two), n3 = clusters(three);
    if (n3 > n2) go(three, 3, n3);
    else go(two, 2, n2);
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

int project_batch_by_radius(int psf_k, const BatchStepDesc* d, const BatchSel& sel, bool att, int max_nz,
                            int* counter, cudaStream_t st, int* info) {
  if (psf_k == 0) return launch_project_batch_R<0, false>(d, sel, att, max_nz, counter, st, info);
  switch ((psf_k - 1) / 2) {
    case 0: return launch_project_batch_R<0, true>(d, sel, att, max_nz, counter, st, info);
    case 1: return launch_project_batch_R<1, true>(d, sel, att, max_nz, counter, st, info);
    case 2: return launch_project_batch_R<2, true>(d, sel, att, max_nz, counter, st, info);
    case 3: return launch_project_batch_R<3, true>(d, sel, att, max_nz, counter, st, info);
    case 4: return launch_project_batch_R<4, true>(d, sel, att, max_nz, counter, st, info);
    case 5: return launch_project_batch_R<5, true>(d, sel, att, max_nz, counter, st, info);
    case 6: return launch_project_batch_R<6, true>(d, sel, att, max_nz, counter, st, info);
    case 7: return launch_project_batch_R<7, true>(d, sel, att, max_nz, counter, st, info);
    default: return kErrParameters;
  }
}

}  // namespace

int yg_project_batch(const BatchStepDesc* d_desc, const BatchSel& sel, int psf_k, bool att, int max_nz,
                     int* d_counter, cudaStream_t st) {
  if (sel.n <= 0 || sel.total <= 0) return kOk;
  return project_batch_by_radius(psf_k, d_desc, sel, att, max_nz, d_counter, st, nullptr);
}

int yg_project_batch_info(int psf_k, bool att, int max_nz, int* info) {
  return project_batch_by_radius(psf_k, nullptr, BatchSel(), att, max_nz, nullptr, nullptr, info);
}

int yg_project(const YgArgs& a, cudaStream_t st, int* slabs_used) {
  const int R = a.psf ? (a.psf_k - 1) / 2 : 0;
  const std::vector<Window> wins = call_windows(a, R);
  int pslabs = a.pslabs;
  for (size_t i = 0; i < wins.size(); ++i) {
    int used[2] = {0, 0};
    YgArgs b = windowed(a, wins[i]);
    b.pslabs = pslabs;
    const int s = project_by_radius(R, b, st, used);
    if (s != kOk) return s;
    if (a.carry_out) {
      // the carries of every window have the slabs of the first; a window
      // whose kernel fell back from 16 takes the others with it
      if (i > 0 && used[1] != pslabs) i = static_cast<size_t>(-1);
      pslabs = used[1];
    }
    if (slabs_used) *slabs_used = used[0];
  }
  return kOk;
}

}  // namespace nrgb
