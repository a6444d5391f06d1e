// Fused y-gantry backprojector: transmission carries, spread (reference and
// exact-transpose forms, mirror units), inverse-rotation gather and the
// two-stream pipeline over camera groups.
#include "et_yg_device.cuh"

namespace nrgb {

// et_yg_spread_kernels.cuh
template <int R, bool ADJ>
int launch_spread_R(const YgArgs& a, int c0, int gcount, cudaStream_t st);
template <int R, bool ADJ>
int launch_spread_pair_R(const YgArgs& a, int u0, int gcount, cudaStream_t st);

namespace {

// ------------------------------------------------ backprojector: slab carry
// carry[c][s][x][y] (s < a.bslabs) = sum of the rotated mu over the depth
// slabs before s (exclusive prefix): the transmission a depth slab starts
// from; carry[c][a.bslabs][x][y] = the whole column's sum.  One block row per
// camera c, or with a.units per unit (its first camera c; a mirror camera's
// transmissions are c's read from the other end); one warp per depth slab.
// L lanes per column: a warp walks 32 / L times kCarryCols columns.
template <class V, int L>
__global__ void __launch_bounds__(32 * kSlabsB) k_mu_carry_yg(const YgArgs a, int u0) {
  constexpr int C = kCarryCols, GW = 32 / L;
  constexpr bool KAHAN = StorageTraits<V>::kKahan;
  const V* __restrict__ mu = reinterpret_cast<const V*>(a.mu) + a.row0;
  __shared__ Tap s_tap[kSlabsB][GW][C];
  __shared__ float4 s_sum[kSlabsB][C][32];
  const int warp = threadIdx.x >> 5, wlane = threadIdx.x & 31, sub = wlane / L, lane = wlane % L;
  const int nchunk = (a.nx + C * GW - 1) / (C * GW);
  const int unit = u0 + blockIdx.x / nchunk;
  const int cam = a.units ? a.units[unit].x : unit;
  const int x0 = ((blockIdx.x % nchunk) * GW + sub) * C;
  const int yb = lane * 4;
  const bool yok = lane_rows_ok(a, yb);
  const CamRows cr = cam_rows(a.geom[cam].fwd);
  const int nsl = a.bslabs, slots = nsl + 1;
  const int zper = (a.nz + nsl - 1) / nsl;
  const int zbeg = warp * zper, zend = min(a.nz, zbeg + zper);
  float4 S[C], cS[C];
#pragma unroll
  for (int i = 0; i < C; ++i) {
    S[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    cS[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int z = zbeg; z < zend; ++z) {
    if (lane < C) {
      const int xp = x0 + lane;
      s_tap[warp][sub][lane] = make_tap(xp, z, cr.m00, cr.m02, cr.m03, cr.m20, cr.m22, cr.m23, a.nx, a.nz, a.cy, xp < a.nx);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < C; ++i) depth_add4<KAHAN>(S[i], cS[i], sample4(mu, s_tap[warp][sub][i], yb, yok));
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < C; ++i) s_sum[warp][i][wlane] = depth_value4<KAHAN>(S[i], cS[i]);
  __syncthreads();
  if (!yok || !lane_writes(a, yb)) return;
#pragma unroll
  for (int i = 0; i < C; ++i) {
    const int x = x0 + i;
    if (x >= a.nx) continue;
    float4 pre = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < warp; ++s) add4(pre, s_sum[s][i][wlane]);
    float* dst = a.slab_T + ((static_cast<size_t>(cam) * slots + warp) * a.nx + x) * a.cy + a.row0 + yb;
    *reinterpret_cast<float4*>(dst) = pre;
    if (warp == nsl - 1) {  // the column total, one slot further
      add4(pre, s_sum[warp][i][wlane]);
      *reinterpret_cast<float4*>(dst + static_cast<size_t>(a.nx) * a.cy) = pre;
    }
  }
}

// ------------------------------------ backprojector: inverse-rotation gather
// out[Z][X][y] (+)= sum_g bilinear(temp[g], B_g * (X, y, Z)) with B_g the
// camera's inverse matrix (ZYX order, -theta), emission-lib/_et.cpp:474-497.
// With a.units, g runs over units and B_g is the unit's first camera's.
// first: assign instead of adding to a.out; clamp: the last group of the
// window with a.truncate -- negative sums become zero as they are stored.
// L lanes hold one column, 32 / L lane groups per warp; footprints of
// kGatherTaps units at a time sit in shared memory.  One column and four units
// in flight per group: 60 us a 30-unit group at 128^3 (two columns and two
// units, the same loads in flight from half the warps, 66 us; three units 72).
template <int U, int L>
__global__ void __launch_bounds__(32 * kGatherWarps) k_gather_yg(const YgArgs a, int c0, int gcount, int first,
                                                                int clamp) {
  constexpr int GROUPS = 32 * kGatherWarps / L;
  __shared__ Tap s_gtap[GROUPS][kGatherTaps];
  const int grp = threadIdx.x / L, lane = threadIdx.x % L;
  const int item = blockIdx.x * GROUPS + grp;
  const int Z = item / a.nx, X = item % a.nx;
  const int yb = lane * 4;
  const bool rows = Z < a.nz && lane_rows_ok(a, yb) && lane_writes(a, yb);
  Tap* tap = s_gtap[grp];
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * a.cs;
  // the loads of U units' volumes in flight at once (every footprint offset is
  // inside its volume, see make_tap), added in unit order
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int g0 = 0; g0 < gcount; g0 += kGatherTaps) {
    const int n = min(kGatherTaps, gcount - g0);
    if (Z < a.nz)
      for (int e = lane; e < n; e += L) {
        const int g = c0 + g0 + e;
        const int cam = !a.units ? g : a.mates ? a.units[g].y : a.units[g].x;
        // footprints in the scratch (column stride cs); none without a camera
        const CamRows cr = cam_rows(a.geom[max(cam, 0)].bwd);
        tap[e] = make_tap(X, Z, cr.m00, cr.m02, cr.m03, cr.m20, cr.m22, cr.m23, a.nx, a.nz, a.cs, cam >= 0);
      }
    __syncwarp();
    if (rows) {
      const float* src = a.temp + vol * g0;
      int g = 0;
      for (; g + U <= n; g += U) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = sample4_loaded(src + vol * (g + u), tap[g + u], yb);
#pragma unroll
        for (int u = 0; u < U; ++u) add4(acc, v[u]);
      }
      for (; g < n; ++g) add4(acc, sample4(src + vol * g, tap[g], yb, true));
    }
    __syncwarp();
  }
  if (!rows) return;
  float4* dst = reinterpret_cast<float4*>(a.out + (static_cast<size_t>(Z) * a.nx + X) * a.cy + a.row0 + yb);
  if (!first) add4(acc, *dst);
  if (clamp) acc = clamp0(acc);
  *dst = acc;
}

// Forward bilinear weight of corner (X, Z) in the footprint of rotated column
// (xp, zp) (0 when (X, Z) is not one of its corners): make_tap's position,
// floor, relative and basis arithmetic, and its product for that corner, so
// the weight equals the one the scatter of the atomic form applies.
__device__ __forceinline__ float corner_weight(int xp, int zp, const CamRows& cr, int X, int Z) {
  const float fx = static_cast<float>(xp), fz = static_cast<float>(zp);
  const float px = fa(fa(fm(cr.m00, fx), fm(cr.m02, fz)), cr.m03);
  const float pz = fa(fa(fm(cr.m20, fx), fm(cr.m22, fz)), cr.m23);
  const int xs = static_cast<int>(floorf(px));
  const int zs = static_cast<int>(floorf(pz));
  if ((X != xs && X != xs + 1) || (Z != zs && Z != zs + 1)) return 0.0f;
  float rx = __fsub_rn(px, static_cast<float>(xs));
  float rz = __fsub_rn(pz, static_cast<float>(zs));
  if (rx < 0.0f) rx = 0.0f;
  if (rz < 0.0f) rz = 0.0f;
  const float wx = X == xs ? __fsub_rn(1.0f, rx) : rx;
  const float wz = Z == zs ? __fsub_rn(1.0f, rz) : rz;
  return wx * wz;
}

// Deterministic transposed gather: out[Z][X][y] (+)= sum over the group's
// units g (camera order) and over the rotated columns (x', z') whose forward
// footprint has (X, Z) as a corner, of that corner's weight times
// scratch_g[z'][x'][y] -- the transpose of the projector's bilinear sampling
// without vector reductions.  The forward rows are a rotation, so those
// columns lie within sqrt(2) of the inverse image of (X, Z): inside the 4 x 4
// integer box around it.  Lane l evaluates box candidate l % 16 of output
// column X0 + l / 16; the nonzero weights are then added in lane order.
__global__ void __launch_bounds__(32 * kGatherWarps) k_tgather_yg(const YgArgs a, int c0, int gcount, int first,
                                                                  int clamp) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nchunk = (a.nx + 1) / 2;
  const int item = blockIdx.x * kGatherWarps + warp;
  if (item >= nchunk * a.nz) return;
  const int Z = item / nchunk;
  const int X0 = (item % nchunk) * 2;
  const int yb = lane * 4;
  const bool rows = lane_rows_ok(a, yb) && lane_writes(a, yb);
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * a.cs;
  const int X = X0 + (lane >> 4);
  const int bx = (lane & 3) - 1, bz = ((lane >> 2) & 3) - 1;
  float4 acc[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  for (int g = 0; g < gcount; ++g) {
    const CamRows cr = cam_rows(a.geom[a.units ? a.units[c0 + g].x : c0 + g].fwd);
    float w = 0.0f;
    int off = 0;
    if (X < a.nx) {
      const float det = cr.m00 * cr.m22 - cr.m02 * cr.m20;
      const float dx = static_cast<float>(X) - cr.m03, dz = static_cast<float>(Z) - cr.m23;
      const int xp = static_cast<int>(floorf((cr.m22 * dx - cr.m02 * dz) / det)) + bx;
      const int zp = static_cast<int>(floorf((cr.m00 * dz - cr.m20 * dx) / det)) + bz;
      if (xp >= 0 && xp < a.nx && zp >= 0 && zp < a.nz) {
        w = corner_weight(xp, zp, cr, X, Z);
        off = (zp * a.nx + xp) * a.cs;
      }
    }
    const float* src = a.temp + vol * g + (rows ? yb : 0);
    // the nonzero weights four at a time: their loads in flight together,
    // then the terms added in lane order
    for (unsigned m = __ballot_sync(kFull, w != 0.0f); m;) {
      int l[4];
      float wl[4];
      float4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        l[q] = m ? __ffs(m) - 1 : -1;  // uniform: from the ballot
        m &= m ? m - 1 : 0u;
        const int src_lane = l[q] < 0 ? 0 : l[q];
        wl[q] = __shfl_sync(kFull, w, src_lane);
        const int ol = __shfl_sync(kFull, off, src_lane);  // an offset inside the volume
        v[q] = ldg4(src + ol);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (l[q] < 0) break;
        const float4 wv = make_float4(wl[q] * v[q].x, wl[q] * v[q].y, wl[q] * v[q].z, wl[q] * v[q].w);
        if (l[q] < 16)
          add4(acc[0], wv);
        else
          add4(acc[1], wv);
      }
    }
  }
  if (!rows) return;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int Xo = X0 + i;
    if (Xo >= a.nx) continue;
    float4* dst = reinterpret_cast<float4*>(a.out + (static_cast<size_t>(Z) * a.nx + Xo) * a.cy + a.row0 + yb);
    if (!first) add4(acc[i], *dst);
    if (clamp) acc[i] = clamp0(acc[i]);
    *dst = acc[i];
  }
}

// clamp: this is the window's last group and the result is truncated
void launch_tgather(const YgArgs& b, int c0, int gcount, int clamp, cudaStream_t st) {
  const int blocks = ((b.nx + 1) / 2 * b.nz + kGatherWarps - 1) / kGatherWarps;
  NRGB_LAUNCH_SCOPE("k_tgather_yg", st);
  k_tgather_yg<<<blocks, 32 * kGatherWarps, 0, st>>>(b, c0, gcount, c0 == 0 ? 1 : 0, clamp);
}

template <int L>
void launch_gather_as(const YgArgs& b, int c0, int gcount, int first, int clamp, cudaStream_t st) {
  constexpr int GROUPS = 32 * kGatherWarps / L;
  const int items = b.nx * b.nz;
  NRGB_LAUNCH_SCOPE("k_gather_yg", st);
  k_gather_yg<kGatherUnits, L>
      <<<(items + GROUPS - 1) / GROUPS, 32 * kGatherWarps, 0, st>>>(b, c0, gcount, first, clamp);
}

}  // namespace

void yg_gather(const YgArgs& b, int c0, int gcount, int first, int clamp, cudaStream_t st) {
  const int lanes = column_lanes(b.ny);
  if (lanes == 8) launch_gather_as<8>(b, c0, gcount, first, clamp, st);
  else if (lanes == 16) launch_gather_as<16>(b, c0, gcount, first, clamp, st);
  else launch_gather_as<32>(b, c0, gcount, first, clamp, st);
}

namespace {

template <bool ADJ>
int spread_pair_by_radius(int R, const YgArgs& a, int u0, int gcount, cudaStream_t st) {
  switch (R) {
    case 0: return launch_spread_pair_R<0, ADJ>(a, u0, gcount, st);
    case 1: return launch_spread_pair_R<1, ADJ>(a, u0, gcount, st);
    case 2: return launch_spread_pair_R<2, ADJ>(a, u0, gcount, st);
    case 3: return launch_spread_pair_R<3, ADJ>(a, u0, gcount, st);
    case 4: return launch_spread_pair_R<4, ADJ>(a, u0, gcount, st);
    case 5: return launch_spread_pair_R<5, ADJ>(a, u0, gcount, st);
    case 6: return launch_spread_pair_R<6, ADJ>(a, u0, gcount, st);
    case 7: return launch_spread_pair_R<7, ADJ>(a, u0, gcount, st);
    default: return kErrParameters;
  }
}

template <bool ADJ>
int spread_by_radius_t(int R, const YgArgs& a, int c0, int gcount, cudaStream_t st) {
  switch (R) {
    case 0: return launch_spread_R<0, ADJ>(a, c0, gcount, st);
    case 1: return launch_spread_R<1, ADJ>(a, c0, gcount, st);
    case 2: return launch_spread_R<2, ADJ>(a, c0, gcount, st);
    case 3: return launch_spread_R<3, ADJ>(a, c0, gcount, st);
    case 4: return launch_spread_R<4, ADJ>(a, c0, gcount, st);
    case 5: return launch_spread_R<5, ADJ>(a, c0, gcount, st);
    case 6: return launch_spread_R<6, ADJ>(a, c0, gcount, st);
    case 7: return launch_spread_R<7, ADJ>(a, c0, gcount, st);
    default: return kErrParameters;
  }
}

int spread_by_radius(int R, const YgArgs& a, int c0, int gcount, cudaStream_t st) {
  return spread_by_radius_t<false>(R, a, c0, gcount, st);
}

}  // namespace

int yg_even_group(int n, int group) {
  group = std::max(1, std::min(group, n));
  const int ngroups = (n + group - 1) / group;
  return (n + ngroups - 1) / ngroups;
}

size_t yg_backproject_workspace(int nx, int ny, int nz, int ncam, int group, int slots) {
  const size_t cy = round_up(ny, 4);
  const size_t vol = static_cast<size_t>(nz) * nx * scratch_rows(ny);  // one window's scratch volume
  const size_t slabs = static_cast<size_t>(ncam) * kCarrySlots * nx * cy;  // at most kSlabsB slabs
  // with two slots the spread of group g+1 overlaps the gather of group g
  return sizeof(float) * (slabs + static_cast<size_t>(slots) * vol * std::max(1, std::min(group, ncam)));
}

int yg_carry_slabs() { return kCarrySlots; }

int yg_backproject_slabs(int nx, int ny, int nz, int n, int ctas_per_sm) {
  const int columns = 1024 / window_lanes(std::min(ny, kWindowRows), nx);
  return yg_spread_slabs(n * ((nx + columns - 1) / columns), nz, ctas_per_sm);
}

namespace {

// Carries of units (or cameras) [u0, u0 + n).
int mu_carry_range(const YgArgs& a_in, float* out, int u0, int n, cudaStream_t st) {
  for (const Window& w : row_windows(a_in.ny, 0, a_in.nx)) {  // carries need no halo
    YgArgs a = windowed(a_in, w);
    a.slab_T = out;
    auto go = [&](auto v, auto lanes) {
      using V = decltype(v);
      constexpr int L = decltype(lanes)::value, C = kCarryCols * (32 / L);
      NRGB_LAUNCH_SCOPE("k_mu_carry_yg", st);
      k_mu_carry_yg<V, L><<<n * ((a.nx + C - 1) / C), 32 * a.bslabs, 0, st>>>(a, u0);
    };
    auto pick = [&](auto v) {
      const int lanes = column_lanes(a.ny);
      if (lanes == 8) go(v, std::integral_constant<int, 8>());
      else if (lanes == 16) go(v, std::integral_constant<int, 16>());
      else go(v, std::integral_constant<int, 32>());
    };
    if (a.storage == kStorageBF16) pick(__nv_bfloat16());
    else pick(0.0f);
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

}  // namespace

int yg_mu_carry(const YgArgs& a, float* out, cudaStream_t st) {
  return mu_carry_range(a, out, 0, a.units ? a.nunits : a.ncam, st);
}

namespace {

// Second stream and events of the backprojection pipeline, one set per
// device; `mu` makes each call's event records and waits one sequence (calls
// from several host threads, e.g. plans on their own streams).
struct Pipe {
  std::mutex mu;
  cudaStream_t aux = nullptr, aux2 = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr, spread_done[2] = {nullptr, nullptr},
              gather_done[2] = {nullptr, nullptr};
};

Pipe* pipe_for_current_device() {
  static std::mutex mu;
  static std::map<int, Pipe> pipes;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  Pipe& p = pipes[dev];
  if (!p.aux) {
    if (cudaStreamCreateWithFlags(&p.aux, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&p.aux2, cudaStreamNonBlocking) != cudaSuccess)
      return nullptr;
    cudaEvent_t* evs[] = {&p.fork, &p.join, &p.spread_done[0], &p.spread_done[1], &p.gather_done[0],
                          &p.gather_done[1]};
    for (cudaEvent_t* e : evs)
      if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return nullptr;
  }
  return &p;
}

}  // namespace

void yg_tgather(const YgArgs& a, int c0, int gcount, int clamp, cudaStream_t st) {
  launch_tgather(a, c0, gcount, clamp, st);
}

// Per row window and camera group: step g (over all windows' groups) uses
// scratch slot g % 2 and spreads on the caller's stream (even g) or a second
// spread stream (odd g), its gather following on a gather stream.  The
// spread of step g+1 thus starts while step g's last wave of CTAs drains (a
// 30-unit spread at 128^3 is 3.2 waves on 152 SMs) and runs beside the
// gather of step g; a slot is spread again only after its gather.
int yg_backproject(const YgArgs& a_in, cudaStream_t st) {
  YgArgs a = a_in;
  if (a.bslabs < 0 || a.bslabs > kSlabsB) return kErrParameters;
  const int R = a.psf ? (a.psf_k - 1) / 2 : 0;
  // mirror units: float32 mu, or bfloat16 mu in reference mode
  const bool pair = a.units && a.nunits > 0 &&
                    (a.storage != kStorageBF16 || a.back_mode != kBackAdjoint);
  if (!pair) {
    a.units = nullptr;
    a.nunits = 0;
  }
  const int nunits = pair ? a.nunits : a.ncam;  // scratch volumes to spread and gather
  // even groups of at most a.group units
  int group = yg_even_group(nunits, a.group);
  if (a.bslabs == 0) {
    const bool scatter = a.back_mode == kBackAdjoint && !a.det;  // every unit in one launch
    const bool three = !pair && a.mu && a.storage != kStorageBF16 && a.back_mode != kBackAdjoint;
    a.bslabs = yg_backproject_slabs(a.nx, a.ny, a.nz, scatter ? nunits : group, three ? 3 : 2);
  }
  const std::vector<Window> wins = call_windows(a, R);
  // work space: slab carries first (unless given), then the scratch slot(s)
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * scratch_rows(a.ny);
  float* slot0;
  // carries of every unit first (computing group g+1's carries on the gather
  // stream while group g spreads measured no faster on GB300)
  if (a.carry || !a.mu) {  // carries given, or not needed
    a.slab_T = const_cast<float*>(a.carry);
    slot0 = a.work;
  } else {
    a.slab_T = a.work;
    slot0 = a.work + static_cast<size_t>(a.ncam) * (a.bslabs + 1) * a.nx * a.cy;
    int s = yg_mu_carry(a, a.slab_T, st);
    if (s != kOk) return s;
  }
  if (a.sino_ready) cudaStreamWaitEvent(st, static_cast<cudaEvent_t>(a.sino_ready), 0);
  a.group = group;
  // the exact transpose in its deterministic form: group scratch + transposed gather
  const bool tgather = a.back_mode == kBackAdjoint && a.det;
  auto spread_on = [&](const YgArgs& b, int c0, int gcount, cudaStream_t ss) {
    if (tgather)
      return pair ? spread_pair_by_radius<true>(R, b, c0, gcount, ss) : spread_by_radius_t<true>(R, b, c0, gcount, ss);
    return pair ? spread_pair_by_radius<false>(R, b, c0, gcount, ss) : spread_by_radius(R, b, c0, gcount, ss);
  };
  // with a.truncate the window's last group clamps the result as it stores it
  auto gather_on = [&](const YgArgs& b, int c0, int gcount, cudaStream_t gs) {
    const int clamp = a.truncate && c0 + gcount == nunits ? 1 : 0;
    if (tgather)
      launch_tgather(b, c0, gcount, clamp, gs);
    else
      yg_gather(b, c0, gcount, c0 == 0 ? 1 : 0, clamp, gs);
  };
  auto spread = [&](const YgArgs& b, int c0, int gcount) { return spread_on(b, c0, gcount, st); };
  if (a.back_mode == kBackAdjoint && !a.det) {
    // transpose of the projector: one launch per window over all cameras,
    // scattered straight into the zeroed accumulator
    const size_t full = static_cast<size_t>(a.nz) * a.nx * a.cy;
    if (cudaMemsetAsync(a.out, 0, sizeof(float) * full, st) != cudaSuccess) return kErrKernel;
    for (const Window& w : wins) {
      const int s = pair ? spread_pair_by_radius<true>(R, windowed(a, w), 0, nunits, st)
                         : spread_by_radius_t<true>(R, windowed(a, w), 0, a.ncam, st);
      if (s != kOk) return s;
    }
    return kOk;
  }
  if (!a.pipelined) {
    for (const Window& w : wins) {
      YgArgs b = windowed(a, w);
      b.temp = slot0;
      for (int c0 = 0; c0 < nunits; c0 += group) {
        const int gcount = std::min(group, nunits - c0);
        int st_ = spread(b, c0, gcount);
        if (st_ != kOk) return st_;
        gather_on(b, c0, gcount, st);
      }
    }
    return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
  }
  Pipe* pp = pipe_for_current_device();
  if (!pp) return kErrUnspecified;
  std::lock_guard<std::mutex> pipe_lock(pp->mu);
  cudaEventRecord(pp->fork, st);
  cudaStreamWaitEvent(pp->aux, pp->fork, 0);
  cudaStreamWaitEvent(pp->aux2, pp->fork, 0);
  int gi = 0;
  for (const Window& w : wins) {
    YgArgs b = windowed(a, w);
    for (int c0 = 0; c0 < nunits; c0 += group, ++gi) {
      const int gcount = std::min(group, nunits - c0);
      const int slot = gi & 1;
      cudaStream_t ss = slot ? pp->aux2 : st;
      b.temp = slot0 + vol * group * slot;
      if (gi >= 2) cudaStreamWaitEvent(ss, pp->gather_done[slot], 0);
      int st_ = spread_on(b, c0, gcount, ss);
      if (st_ != kOk) return st_;
      cudaEventRecord(pp->spread_done[slot], ss);
      cudaStreamWaitEvent(pp->aux, pp->spread_done[slot], 0);
      gather_on(b, c0, gcount, pp->aux);
      cudaEventRecord(pp->gather_done[slot], pp->aux);
    }
  }
  cudaEventRecord(pp->join, pp->aux);
  cudaStreamWaitEvent(st, pp->join, 0);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

}  // namespace nrgb
