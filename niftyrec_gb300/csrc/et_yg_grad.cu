// Fused y-gantry form of the reference's attenuation gradient
// (et_array_gradient_attenuation; emission-lib/_et.cpp:1679-1924 with the
// scan of emission-lib_gpu/_et_attenuation_gradient_gpu_kernels.cu:15-42).
// Per camera, in the rotated frame (a, m: rotated activity and mu, T_z the
// inclusive depth sum of m, s the sinogram plane):
//   w(x, y, z) = s(x, y) * sum_{z' >= z} a_z' exp(-T_z'),
// then the per-plane PSF (as in the projector) and the inverse-rotation
// gather into the accumulator.  Three kernels per group of cameras:
//   k_grad_weights_yg: w of a camera and its mirror camera from one set of
//     samples (no PSF halo: every column once), each in its own frame;
//   k_grad_conv_yg: the PSF of the w volumes into the scratch volumes;
//   the backprojector's gather, each volume at its own camera's positions.
// Every sum over depth adds its terms (none is taken as a difference): the
// camera's suffix and the mirror camera's, which is a prefix in this frame,
// run over terms that the first walk left in the volume itself.
// 128^3 x 120, PSF 11: 1.26 ms, against 2.10 ms of one spread kernel per camera
// that sampled activity and mu twice, halo columns included.
#include "et_yg_device.cuh"

namespace nrgb {
namespace {

constexpr int kGradCols = 2;    // columns per lane group of k_grad_weights_yg
constexpr int kGradPlanes = 8;  // planes whose terms its second walk has in flight

// One warp per depth slab (kSlabsB of them), 32 / L lane groups of kGradCols
// columns each; a block holds its columns' whole depth, so the slabs exchange
// through shared memory.  Volume g of a.temp: w of the unit's camera (walk 1
// leaves the terms a exp(-T) there, T local to the slab); volume a.group + g,
// in the mirror camera's frame: the mate's (walk 1: the running sum of
// a exp(E), E the slab's mu before the plane; a slab whose mu exceeds kMateMaxT
// is summed again with the direct weights exp(E - slab)).
// Bound by gather latency and by the volumes' traffic.  One block per SM with
// the registers it wants: 1.24 ms a call at 128^3 x 120, 1.37 ms with two blocks
// of 64 registers, which spill.
template <int L>
__global__ void __launch_bounds__(32 * kSlabsB) k_grad_weights_yg(const YgArgs a, int u0) {
  constexpr int C = kGradCols, GW = 32 / L;
  const float* __restrict__ act = a.act + a.row0;
  const float* __restrict__ mu = a.mu + a.row0;
  extern __shared__ __align__(16) unsigned char smem[];
  float4(*sT)[C][32] = reinterpret_cast<float4(*)[C][32]>(smem);  // [kSlabsB][C][32], then P, Q
  float4(*sP)[C][32] = sT + kSlabsB;
  float4(*sQ)[C][32] = sP + kSlabsB;
  __shared__ Tap s_tap[kSlabsB][GW][C];
  const int slab = threadIdx.x >> 5, wlane = threadIdx.x & 31, sub = wlane / L, lane = wlane % L;
  const int nchunk = (a.nx + C * GW - 1) / (C * GW);
  const int g = blockIdx.x / nchunk;
  const int2 uc = a.units ? a.units[u0 + g] : make_int2(u0 + g, -1);
  const bool paired = uc.y >= 0;  // uniform over the block
  const int x0 = ((blockIdx.x % nchunk) * GW + sub) * C;
  const int yb = lane * 4;
  const bool yok = lane_rows_ok(a, yb);
  const CamRows cr = cam_rows(a.geom[uc.x].fwd);
  const int zper = (a.nz + kSlabsB - 1) / kSlabsB;
  const int zbeg = slab * zper, zend = min(a.nz, zbeg + zper);
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * a.cs;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto mine = [&](int z, int x) {  // the camera's w at (z, x)
    return reinterpret_cast<float4*>(a.temp + vol * g + (static_cast<size_t>(z) * a.nx + x) * a.cs + yb);
  };
  auto mates = [&](int z, int x) {  // the mate's, in its own frame
    return reinterpret_cast<float4*>(a.temp + vol * (a.group + g) +
                                     (static_cast<size_t>(a.nz - 1 - z) * a.nx + a.nx - 1 - x) * a.cs + yb);
  };
  auto footprints = [&](int z) {
    if (lane < C)
      s_tap[slab][sub][lane] = make_tap(x0 + lane, z, cr.m00, cr.m02, cr.m03, cr.m20, cr.m22, cr.m23, a.nx, a.nz,
                                        a.cy, x0 + lane < a.nx);
    __syncwarp();
  };

  // walk 1: terms, and the slab's transmission and partials
  float4 T[C], P[C], Q[C];
#pragma unroll
  for (int i = 0; i < C; ++i) T[i] = P[i] = Q[i] = zero;
  for (int z = zbeg; z < zend; ++z) {
    footprints(z);
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const Tap& t = s_tap[slab][sub][i];
      const float4 m = sample4(mu, t, yb, yok), x = sample4(act, t, yb, yok);
      const bool ok = x0 + i < a.nx && yok;
      if (paired) {
        add4p(Q[i], mul4p(x, exp_neg4(make_float4(-T[i].x, -T[i].y, -T[i].z, -T[i].w))));
        if (ok) *mates(z, x0 + i) = Q[i];
      }
      add4p(T[i], m);
      const float4 e = mul4p(x, exp_neg4(T[i]));
      add4p(P[i], e);
      if (ok) *mine(z, x0 + i) = e;
    }
    __syncwarp();
  }
  bool direct = false;  // uniform over the warp: the mate's sums carry the direct weights
  if (paired) {
    bool redo = false;
#pragma unroll
    for (int i = 0; i < C; ++i) {
      redo |= !(T[i].x <= kMateMaxT && T[i].y <= kMateMaxT && T[i].z <= kMateMaxT && T[i].w <= kMateMaxT);
      redo |= !(isfinite(Q[i].x) && isfinite(Q[i].y) && isfinite(Q[i].z) && isfinite(Q[i].w));
    }
    direct = __any_sync(kFull, redo);
    if (direct) {
      float4 E[C];
#pragma unroll
      for (int i = 0; i < C; ++i) E[i] = Q[i] = zero;
      for (int z = zbeg; z < zend; ++z) {
        footprints(z);
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const Tap& t = s_tap[slab][sub][i];
          const float4 after = make_float4(T[i].x - E[i].x, T[i].y - E[i].y, T[i].z - E[i].z, T[i].w - E[i].w);
          fma4(Q[i], sample4(act, t, yb, yok), exp_neg4(after));
          if (x0 + i < a.nx && yok) *mates(z, x0 + i) = Q[i];
          add4(E[i], sample4(mu, t, yb, yok));
        }
        __syncwarp();
      }
    }
  }

  // slabs: w = exp(-mu before), later = the weighted partials after this slab;
  // the mate's from the other end
#pragma unroll
  for (int i = 0; i < C; ++i) sT[slab][i][wlane] = T[i];
  __syncthreads();
  float4 w[C], wm[C];
#pragma unroll
  for (int i = 0; i < C; ++i) {
    float4 before = zero, after = direct ? zero : T[i];
    for (int s = 0; s < slab; ++s) add4(before, sT[s][i][wlane]);
    for (int s = kSlabsB - 1; s > slab; --s) add4(after, sT[s][i][wlane]);
    w[i] = exp_neg4(before);
    wm[i] = exp_neg4(after);
    sP[slab][i][wlane] = mul4(w[i], P[i]);
    sQ[slab][i][wlane] = mul4(wm[i], Q[i]);
  }
  __syncthreads();
  // walk 2: w = s * (later + weight * running sum), in place
#pragma unroll
  for (int i = 0; i < C; ++i) {
    const int x = x0 + i;
    if (x >= a.nx || !yok) continue;
    float4 later = zero, run = zero;
    for (int s = kSlabsB - 1; s > slab; --s) add4(later, sP[s][i][wlane]);
    const float4 sc = ldg4(a.sino + (static_cast<size_t>(uc.x) * a.nx + x) * a.cy + a.row0 + yb);
    for (int z = zend - 1; z >= zbeg; z -= kGradPlanes) {
      float4 e[kGradPlanes];  // loaded before the stores below, which the compiler cannot move them over
#pragma unroll
      for (int q = 0; q < kGradPlanes; ++q) e[q] = z - q >= zbeg ? *mine(z - q, x) : zero;
#pragma unroll
      for (int q = 0; q < kGradPlanes; ++q) {
        if (z - q < zbeg) break;
        float4 v = later;
        add4p(run, e[q]);
        fma4p(v, w[i], run);
        *mine(z - q, x) = mul4p(sc, v);
      }
    }
    if (paired) {
      float4 earlier = zero;
      for (int s = 0; s < slab; ++s) add4(earlier, sQ[s][i][wlane]);
      const float4 sm = ldg4(a.sino + (static_cast<size_t>(uc.y) * a.nx + a.nx - 1 - x) * a.cy + a.row0 + yb);
      for (int z = zbeg; z < zend; z += kGradPlanes) {
        float4 e[kGradPlanes];
#pragma unroll
        for (int q = 0; q < kGradPlanes; ++q) e[q] = z + q < zend ? *mates(z + q, x) : zero;
#pragma unroll
        for (int q = 0; q < kGradPlanes; ++q) {
          if (z + q >= zend) break;
          float4 v = earlier;
          fma4p(v, wm[i], e[q]);
          *mates(z + q, x) = mul4p(sm, v);
        }
      }
    }
  }
}

// PSF of the w volumes: volume v of the launch from a.temp to a.out (both
// [v][nz][nx][cs]); with a.units the volumes from a.nunits on are the mirror
// cameras' (skipped where a unit has none).  CTA = (volume, x-tile, depth slab).
template <int R, bool PTAB, int L>
__device__ __forceinline__ void grad_conv_body(const YgArgs& a, int u0, int n, const float* ptab) {
  using TS = TileShape<R, L>;
  constexpr int NS = TS::NS, K = 2 * R + 1;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* sb = reinterpret_cast<float4*>(smem);                       // [2][NS][L]
  float* s_psf = reinterpret_cast<float*>(smem + TS::kSbBytes);        // [nz][2K]
  const int grp = threadIdx.x / L, lane = threadIdx.x % L;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int slab = blockIdx.x % a.bslabs, item = blockIdx.x / a.bslabs;
  const int x0 = (item % ntile) * kTX<L>;
  int v = item / ntile;
  if (v >= n) {
    if (a.units[u0 + v - n].y < 0) return;  // uniform over the CTA
    v += a.group - n;
  }
  const int yb = lane * 4;
  const bool yok = lane_rows_ok(a, yb);
  const int zper = (a.nz + a.bslabs - 1) / a.bslabs;
  const int zbeg = slab * zper, zend = min(a.nz, zbeg + zper);
  if (!PTAB)
    for (int i = zbeg * 2 * K + threadIdx.x; i < zend * 2 * K; i += blockDim.x) s_psf[i] = __ldg(a.psf + i);
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * a.cs;
  const float* __restrict__ src = a.temp + vol * v + yb;
  float* __restrict__ dst = a.out + vol * v + yb;
  ybuf_zero_pads<L>();
  __syncthreads();
  auto load = [&](int z, float4 (&r)[TS::kOwn]) {
#pragma unroll
    for (int k = 0; k < TS::kOwn; ++k) {
      const int c = grp + TS::G * k, xp = x0 - R + c;
      r[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < NS && xp >= 0 && xp < a.nx && yok) r[k] = ldg4(src + (static_cast<size_t>(z) * a.nx + xp) * a.cs);
    }
  };
  float4 next[TS::kOwn];  // the next plane's columns, in flight during this plane's passes
  if (zbeg < zend) load(zbeg, next);
  for (int z = zbeg; z < zend; ++z) {
    float4* sbuf = sb + (z & 1) * NS * L;
#pragma unroll
    for (int k = 0; k < TS::kOwn; ++k) {
      const int c = grp + TS::G * k;
      if (c < NS) sbuf[c * L + lane] = next[k];
    }
    __syncthreads();
    if (z + 1 < zend) load(z + 1, next);
    const float* kr = (PTAB ? ptab : s_psf) + z * 2 * K;
    rowpass_from_tile_p<R, L, L>(
        sbuf, grp * kTXW,
        [&](int i, const float4& o) {
          const int x = x0 + grp * kTXW + i;
          if (x < a.nx && yok) *reinterpret_cast<float4*>(dst + (static_cast<size_t>(z) * a.nx + x) * a.cs) = o;
        },
        kr, kr + K, lane, a.ny);
  }
}

template <int R, int L>
__global__ void __launch_bounds__(32 * kW, 3) k_grad_conv_yg(const YgArgs a, int u0, int n) {
  grad_conv_body<R, false, L>(a, u0, n, nullptr);
}

template <int R, int L>
__global__ void __launch_bounds__(32 * kW, 3)
    k_grad_conv_ptab_yg(const YgArgs a, int u0, int n, const __grid_constant__ PsfTable t) {
  grad_conv_body<R, true, L>(a, u0, n, t.c);
}

template <int R, int L>
int launch_grad_conv(const YgArgs& a_in, int u0, int n, cudaStream_t st) {
  YgArgs a = a_in;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int volumes = a.units ? 2 * n : n;
  a.bslabs = yg_spread_slabs(volumes * ntile, a.nz, 3);
  const bool ptab = psf_in_parameters<R>(a);
  const size_t smem = TileShape<R, L>::kSbBytes + (ptab ? 0 : sizeof(float) * a.nz * 2 * (2 * R + 1));
  const dim3 grid(volumes * ntile * a.bslabs), block(32 * kW);
  if (ptab) {
    static thread_local PsfTable table;
    std::memcpy(table.c, a.psf_host, sizeof(float) * a.nz * 2 * (2 * R + 1));
    auto k = k_grad_conv_ptab_yg<R, L>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE("k_grad_conv_yg", st);
    k<<<grid, block, smem, st>>>(a, u0, n, table);
  } else if constexpr (L == 32) {
    auto k = k_grad_conv_yg<R, L>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE("k_grad_conv_yg", st);
    k<<<grid, block, smem, st>>>(a, u0, n);
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

template <int R>
int grad_conv_R(const YgArgs& a, int u0, int n, cudaStream_t st) {
  if (psf_in_parameters<R>(a)) {
    if (a.lanes == 8) return launch_grad_conv<R, 8>(a, u0, n, st);
    if (a.lanes == 16) return launch_grad_conv<R, 16>(a, u0, n, st);
  }
  return launch_grad_conv<R, 32>(a, u0, n, st);
}

int grad_conv_by_radius(int R, const YgArgs& a, int u0, int n, cudaStream_t st) {
  switch (R) {
    case 0: return grad_conv_R<0>(a, u0, n, st);
    case 1: return grad_conv_R<1>(a, u0, n, st);
    case 2: return grad_conv_R<2>(a, u0, n, st);
    case 3: return grad_conv_R<3>(a, u0, n, st);
    case 4: return grad_conv_R<4>(a, u0, n, st);
    case 5: return grad_conv_R<5>(a, u0, n, st);
    case 6: return grad_conv_R<6>(a, u0, n, st);
    case 7: return grad_conv_R<7>(a, u0, n, st);
    default: return kErrParameters;
  }
}

int launch_weights(const YgArgs& a, int u0, int n, cudaStream_t st) {
  constexpr size_t smem = sizeof(float4) * 3 * kSlabsB * kGradCols * 32;
  auto go = [&](auto lanes) {
    constexpr int L = decltype(lanes)::value, C = kGradCols * (32 / L);
    auto k = k_grad_weights_yg<L>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE("k_grad_weights_yg", st);
    k<<<n * ((a.nx + C - 1) / C), 32 * kSlabsB, smem, st>>>(a, u0);
  };
  const int lanes = column_lanes(a.ny);
  if (lanes == 8) go(std::integral_constant<int, 8>());
  else if (lanes == 16) go(std::integral_constant<int, 16>());
  else go(std::integral_constant<int, 32>());
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

}  // namespace

int yg_gradient(const YgArgs& a_in, cudaStream_t st) {
  YgArgs a = a_in;
  if (!a.mu || !a.act || !a.sino || !a.out || !a.work || a.group < 2) return kErrParameters;
  const int R = a.psf ? (a.psf_k - 1) / 2 : 0;
  // units (or cameras) per group: w and PSF volumes, two of each per mirror unit
  const bool pair = a.units && a.nunits > 0 && a.group >= 4;
  if (!pair) a.units = nullptr;
  const int units = pair ? a.nunits : a.ncam;
  const int group = yg_even_group(units, a.group / (pair ? 4 : 2));
  const int slots = pair ? 2 * group : group;  // volumes of a group
  a.group = group;
  for (const Window& w : call_windows(a, R)) {
    YgArgs b = windowed(a, w);
    const size_t vol = static_cast<size_t>(b.nz) * b.nx * b.cs;
    float* weights = a.work;
    float* blurred = a.psf ? a.work + vol * slots : weights;
    for (int u0 = 0; u0 < units; u0 += group) {
      const int n = std::min(group, units - u0);
      b.temp = weights;
      int s = launch_weights(b, u0, n, st);
      if (s == kOk && a.psf) {
        YgArgs c = b;
        c.out = blurred;
        s = grad_conv_by_radius(R, c, u0, n, st);
      }
      if (s != kOk) return s;
      const bool last = u0 + n == units;
      b.temp = blurred;
      yg_gather(b, u0, n, u0 == 0, a.truncate && last && !pair, st);
      if (pair) {
        b.temp = blurred + vol * group;
        b.mates = 1;
        yg_gather(b, u0, n, 0, a.truncate && last, st);
        b.mates = 0;
      }
    }
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

size_t yg_gradient_workspace(int nx, int ny, int nz, int volumes) {
  return sizeof(float) * static_cast<size_t>(nz) * nx * scratch_rows(ny) * volumes;
}

}  // namespace nrgb
