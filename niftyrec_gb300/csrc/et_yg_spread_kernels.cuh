// Spread kernels of the backprojector (reference and exact-transpose forms,
// mirror units) and their launchers, instantiated per PSF radius in separate
// translation units (et_yg_spread_r*.cu) that compile in parallel.
#pragma once

#include "et_yg_device.cuh"

namespace nrgb {
namespace {

// Row pass of a single camera: packed, but scalar at radius 4, where the packed
// form spills 16 bytes at the 80 registers of three CTAs per SM and the scalar one
// none (111 x 93 x 111 x 72, PSF 9: backprojection 555 us, packed 559; 96^3 x 72: 402,
// 405).  Radii 3 and 5 spill 4 and 8 bytes packed and still gain.
template <int R, int L, class EmitFn, class KR, class KC>
__device__ __forceinline__ void rowpass_single(const float4* __restrict__ sbuf, int base, EmitFn emit, KR kr, KC kc,
                                               int lane, int ny) {
  if constexpr (R == 4) rowpass_from_tile<R, L, L>(sbuf, base, emit, kr, kc, lane, ny);
  else rowpass_from_tile_p<R, L, L>(sbuf, base, emit, kr, kc, lane, ny);
}

// ---------------------------------------- backprojector: spread + PSF
// temp[g][z][x][y] = PSF_z( s(x', y) * exp(-T_z(x', y)) ) for camera c0+g,
// T inclusive (emission-lib/_et_line_backproject_attenuated.cpp:24-34), PSF
// as in the projector.  CTA = (camera, x-tile, depth slab); every sampled
// column starts its transmission from the slab carry.
// ADJ: the exact transpose of the projector instead (not in the reference):
// the PSF taps are flipped (correlation) and each output column is scattered
// with the projector's own bilinear weights into the accumulator a.out
// (vector reductions; all cameras in one launch, no scratch), or, with
// a.det, written to the group scratch like the reference form for the
// transposed gather k_tgather_yg (a fixed summation order).
// CTAS: CTAs per SM the kernel is compiled for (3 where three tiles fit in
// shared memory, for the float32 reference spread; else 2).
// PTAB: the separated PSF comes from the kernel-parameter table `ptab`
// ([nz][2K]) instead of a shared-memory copy of the slab's planes.
template <int R, bool PSF, bool ATT, bool ADJ, class V, bool PTAB, int L>
__device__ __forceinline__ void spread_body(const YgArgs& a, int c0, const float* ptab) {
  using TS = TileShape<R, L>;
  constexpr bool KAHAN = StorageTraits<V>::kKahan;
  const V* __restrict__ mu = reinterpret_cast<const V*>(a.mu) + a.row0;
  constexpr int NS = TS::NS;
  constexpr int K = 2 * R + 1;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* sb = reinterpret_cast<float4*>(smem);
  Tap* taps = reinterpret_cast<Tap*>(smem + TS::kSbBytes);
  float* s_psf = reinterpret_cast<float*>(smem + TS::kSbBytes + TS::kTapBytes);

  const int grp = threadIdx.x / L, lane = threadIdx.x % L;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int nsl = a.bslabs, slots = nsl + 1;
  const int slab = blockIdx.x % nsl;
  const int item = blockIdx.x / nsl;
  const int g = item / ntile;
  const int cam = c0 + g;
  const int x0 = (item % ntile) * kTX<L>;
  const int yb = lane * 4;
  const bool yok = lane_rows_ok(a, yb);
  const int zper = (a.nz + nsl - 1) / nsl;
  const int zbeg = slab * zper, zend = min(a.nz, zbeg + zper);
  if (zbeg >= zend) return;  // uniform over the CTA
  if (PSF && !PTAB) {  // this slab's planes only
    for (int i = zbeg * 2 * K + threadIdx.x; i < zend * 2 * K; i += blockDim.x) {
      const int j = i % (2 * K), base = i - j;
      // transpose of a convolution = correlation: reverse each kernel
      const int src = !ADJ ? i : (j < K ? base + (K - 1 - j) : base + K + (2 * K - 1 - j));
      s_psf[i] = __ldg(a.psf + src);
    }
  }
  const CamRows cr = cam_rows(a.geom[cam].fwd);
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * a.cs;  // one scratch volume
  const bool scatter = ADJ && !a.det;  // uniform over the launch
  float* __restrict__ tmp = scatter ? a.out + a.row0 : a.temp + vol * g;
  const float* __restrict__ srow = a.sino + static_cast<size_t>(cam) * a.nx * a.cy + a.row0;

  float4 Tc[TS::kOwn], cTc[TS::kOwn];  // transmission per sampled column (+ Kahan compensation)
#pragma unroll
  for (int k = 0; k < TS::kOwn; ++k) {
    Tc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    cTc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int xp = x0 - R + grp + TS::G * k;
    if (ATT && grp + TS::G * k < NS && xp >= 0 && xp < a.nx && yok)
      Tc[k] = ldg4(a.slab_T + ((static_cast<size_t>(cam) * slots + slab) * a.nx + xp) * a.cy + a.row0 + yb);
  }
  ybuf_zero_pads<L>();
  __syncthreads();

  for (int z = zbeg; z < zend; ++z) {
    const int b = z & 1;
    float4* sbuf = sb + b * NS * L;
    Tap* tb = taps + b * TS::kTapSlots;
    if ((ATT || ADJ) && lane < TS::kOwn) {
      const int c = grp + TS::G * lane;
      if (c < NS) {
        const int xp = x0 - R + c;
        tb[tap_slot<R, L>(c)] = make_tap(xp, z, cr.m00, cr.m02, cr.m03, cr.m20, cr.m22, cr.m23, a.nx, a.nz, a.cy,
                         xp >= 0 && xp < a.nx);
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < TS::kOwn; ++k) {
      const int c = grp + TS::G * k;
      if (c < NS) {
        const int xp = x0 - R + c;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (xp >= 0 && xp < a.nx && yok) s = ldg4(srow + static_cast<size_t>(xp) * a.cy + yb);
        if (ATT) {
          depth_add4<KAHAN>(Tc[k], cTc[k], sample4(mu, tb[tap_slot<R, L>(c)], yb, yok));
          s = mul4(s, exp_neg4(depth_value4<KAHAN>(Tc[k], cTc[k])));
        }
        sbuf[c * L + lane] = s;
      }
    }
    __syncthreads();
    auto emit = [&](int i, const float4& v) {
      const int x = x0 + grp * kTXW + i;
      if (x >= a.nx || !yok) return;
      if (scatter) {
        // halo rows lack part of their PSF support: their owner window adds them
        if (lane_writes(a, yb)) scatter4(tmp, tb[tap_slot<R, L>(grp * kTXW + i + R)], yb, v);
      } else {
        *reinterpret_cast<float4*>(tmp + (static_cast<size_t>(z) * a.nx + x) * a.cs + yb) = v;
      }
    };
    if (PSF) {
      if constexpr (PTAB && ADJ) {  // transpose of a convolution = correlation: both kernels reversed
        const float* kr = ptab + z * 2 * K;
        rowpass_single<R, L>(sbuf, grp * kTXW, emit, Reversed<R>{kr}, Reversed<R>{kr + K}, lane, a.ny);
      } else {
        const float* kr = (PTAB ? ptab : s_psf) + z * 2 * K;
        rowpass_single<R, L>(sbuf, grp * kTXW, emit, kr, kr + K, lane, a.ny);
      }
    } else {
#pragma unroll
      for (int i = 0; i < kTXW; ++i) emit(i, sbuf[(grp * kTXW + i) * L + lane]);
    }
  }
}

template <int R, bool PSF, bool ATT, bool ADJ, class V, int CTAS, int L>
__global__ void __launch_bounds__(32 * kW, CTAS) k_spread_yg(const YgArgs a, int c0) {
  spread_body<R, PSF, ATT, ADJ, V, false, L>(a, c0, nullptr);
}

template <int R, bool ATT, bool ADJ, class V, int CTAS, int L>
__global__ void __launch_bounds__(32 * kW, CTAS)
    k_spread_ptab_yg(const YgArgs a, int c0, const __grid_constant__ PsfTable t) {
  spread_body<R, true, ATT, ADJ, V, true, L>(a, c0, t.c);
}

// Reference-mode spread of a mirror unit -- camera c and its mate m at the
// opposite angle about the grid centre -- into ONE scratch volume in c's
// rotated frame:
//   U(x', y, z') = PSF_z'[s_c e^{-T}](x') + PSF'_{nz-1-z'}[s_m(nx-1-x') e^{-T'}](x')
// with T the inclusive mu sum along c's column from its detector side, T'
// the inclusive sum from the other end (the mate's detector side), and PSF'
// the mate's plane nz-1-z' with the row kernel reversed.  The mate's inverse
// matrix is c's mirrored in x and z, so gathering U with c's inverse matrix
// adds both cameras' terms: one mu scan, one scratch volume and one gather
// per pair.  A unit without a mate spreads its camera alone.  CTA = (unit,
// x-tile, depth slab); the PSF planes of the slab only sit in shared memory.
//
// ADJ: the exact transpose of the mirror-unit projector instead: both terms in
// c's frame go through the transposed PSF (camera: both kernels reversed;
// mate: row kernel forward, column kernel reversed) and, summed, are
// scattered with c's bilinear weights into the accumulator a.out (the mate's
// footprint of its mirrored column is c's), or with a.det written to the
// group scratch for k_tgather_yg.
//
// V = bfloat16 (mu stored in bfloat16): the forward transmission is summed
// with Kahan compensation (the compensation of each sampled column in shared
// memory), the mate's transmission is the column total minus the compensated
// forward sum (no second running sum), and the tiles are single-buffered (a
// second barrier per plane) so that two CTAs per SM still fit.
//
// float32 reference mode of radius 6 and 7 is single-buffered too: the smaller
// tiles leave more L1 for the gathers (256^3 x 60, PSF 15: pair 6.11 -> 6.06 ms;
// 128^3 x 120, PSF 13: backprojection 0.855 -> 0.839; PSF 11 0.828 -> 0.833).
template <int R, bool ADJ, class V>
constexpr bool kSingleTile = StorageTraits<V>::kKahan || (R >= 6 && !ADJ);

template <int R, int L, bool ADJ, class V>
__host__ __device__ constexpr size_t spread_pair_fixed_smem() {
  using TS = TileShape<R, L>;
  constexpr bool KAHAN = StorageTraits<V>::kKahan;
  return (kSingleTile<R, ADJ, V> ? 1 : 2) * TS::kSbBytes + TS::kTapBytes + (KAHAN ? sizeof(float4) * TS::kOwn * 32 * kW : 0);
}

template <int R, bool PSF, bool ATT, bool ADJ, bool PTAB, class V, int L>
__device__ __forceinline__ void spread_pair_body(const YgArgs& a, int u0, const float* ptab) {
  using TS = TileShape<R, L>;
  constexpr bool KAHAN = StorageTraits<V>::kKahan;
  constexpr int NB = kSingleTile<R, ADJ, V> ? 1 : 2;  // tile buffers
  constexpr int NS = TS::NS;
  constexpr int K = 2 * R + 1;
  const V* __restrict__ mu = reinterpret_cast<const V*>(a.mu) + a.row0;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* sb = reinterpret_cast<float4*>(smem);                              // [NB stages][2][NS][L]
  Tap* taps = reinterpret_cast<Tap*>(smem + NB * TS::kSbBytes);               // [2][kTapSlots]
  float4* scomp = reinterpret_cast<float4*>(smem + NB * TS::kSbBytes + TS::kTapBytes);  // [kOwn][256] (KAHAN)
  float* s_psf = reinterpret_cast<float*>(smem + spread_pair_fixed_smem<R, L, ADJ, V>());  // [zper][2K], mate's next

  const int grp = threadIdx.x / L, lane = threadIdx.x % L;
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const int nsl = a.bslabs, slots = nsl + 1;
  const int slab = blockIdx.x % nsl;
  const int item = blockIdx.x / nsl;
  const int g = item / ntile;
  const int unit = u0 + g;
  const int2 uc = a.units[unit];
  const int cam = uc.x, mate = uc.y;
  const bool paired = mate >= 0;  // uniform over the CTA
  const int x0 = (item % ntile) * kTX<L>;
  const int yb = lane * 4;
  const bool yok = lane_rows_ok(a, yb);
  const int zper = (a.nz + nsl - 1) / nsl;
  const int zbeg = slab * zper, zend = min(a.nz, zbeg + zper);
  if (zbeg >= zend) return;  // uniform over the CTA
  float* s_psf_m = s_psf + zper * 2 * K;
  if (PSF && !PTAB) {
    // reversed index of a row (j < K) or column (j >= K) kernel entry
    auto rev = [&](int j) { return j < K ? K - 1 - j : 3 * K - 1 - j; };
    for (int i = threadIdx.x; i < (zend - zbeg) * 2 * K; i += blockDim.x) {
      const int z = zbeg + i / (2 * K), j = i % (2 * K);
      s_psf[i] = __ldg(a.psf + z * 2 * K + (ADJ ? rev(j) : j));
      if (paired) {  // mate: reference row reversed; transpose column reversed
        const int jm = (j < K) != ADJ ? rev(j) : j;
        s_psf_m[i] = __ldg(a.psf + (a.nz - 1 - z) * 2 * K + jm);
      }
    }
  }
  const CamRows cr = cam_rows(a.geom[cam].fwd);
  const size_t vol = static_cast<size_t>(a.nz) * a.nx * a.cs;  // one scratch volume
  const bool scatter = ADJ && !a.det;  // uniform over the launch
  float* __restrict__ tmp = scatter ? a.out + a.row0 : a.temp + vol * g;
  const float* __restrict__ srow = a.sino + static_cast<size_t>(cam) * a.nx * a.cy + a.row0;
  const float* __restrict__ mrow = a.sino + static_cast<size_t>(paired ? mate : cam) * a.nx * a.cy + a.row0;

  // transmissions per sampled column: forward (from the slab carry) and, for
  // the mate, from the far end (column total minus the carry; with KAHAN Tr
  // holds the column total)
  float4 Tc[TS::kOwn], Tr[TS::kOwn];
#pragma unroll
  for (int k = 0; k < TS::kOwn; ++k) {
    Tc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    Tr[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (KAHAN) scomp[k * 32 * kW + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int xp = x0 - R + grp + TS::G * k;
    if (ATT && grp + TS::G * k < NS && xp >= 0 && xp < a.nx && yok) {
      const float* cp = a.slab_T + ((static_cast<size_t>(cam) * slots + slab) * a.nx + xp) * a.cy + a.row0 + yb;
      Tc[k] = ldg4(cp);
      if (paired) {
        const float4 tot = ldg4(cp + static_cast<size_t>(nsl - slab) * a.nx * a.cy);
        Tr[k] = KAHAN ? tot : make_float4(tot.x - Tc[k].x, tot.y - Tc[k].y, tot.z - Tc[k].z, tot.w - Tc[k].w);
      }
    }
  }
  ybuf_zero_pads<L>();
  __syncthreads();

  for (int z = zbeg; z < zend; ++z) {
    const int b = z & 1;
    float4* sc = sb + (NB == 2 ? b : 0) * 2 * NS * L;
    float4* sm = sc + NS * L;
    Tap* tb = taps + b * TS::kTapSlots;
    if ((ATT || ADJ) && lane < TS::kOwn) {
      const int c = grp + TS::G * lane;
      if (c < NS) {
        const int xp = x0 - R + c;
        tb[tap_slot<R, L>(c)] = make_tap(xp, z, cr.m00, cr.m02, cr.m03, cr.m20, cr.m22, cr.m23, a.nx, a.nz, a.cy,
                                      xp >= 0 && xp < a.nx);
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < TS::kOwn; ++k) {
      const int c = grp + TS::G * k;
      if (c < NS) {
        const int xp = x0 - R + c;
        const bool ok = xp >= 0 && xp < a.nx && yok;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f), q = s;
        if (ok) s = ldg4(srow + static_cast<size_t>(xp) * a.cy + yb);
        if (paired && ok) q = ldg4(mrow + static_cast<size_t>(a.nx - 1 - xp) * a.cy + yb);
        if (ATT) {
          // the branch: the predicated form leaves too few registers beside the
          // two transmissions (128^3 x 120: 0.298 ms a launch, predicated 0.349)
          const float4 m = sample4_branch(mu, tb[tap_slot<R, L>(c)], yb, yok);
          if constexpr (KAHAN) {
            float4 cc = scomp[k * 32 * kW + threadIdx.x];
            kahan_add4p(Tc[k], cc, m);
            scomp[k * 32 * kW + threadIdx.x] = cc;
            const float4 tv = kahan_value4p(Tc[k], cc);
            s = mul4p(s, exp_neg4(tv));
            if (paired) {  // sum from the far end, inclusive: total - forward sum + this plane
              const Pair4 tot = pair4(Tr[k]), v = pair4(tv), mm = pair4(m);
              q = mul4p(q, exp_neg4(unpair4({add2(sub2(tot.lo, v.lo), mm.lo), add2(sub2(tot.hi, v.hi), mm.hi)})));
            }
          } else {
            add4p(Tc[k], m);
            s = mul4p(s, exp_neg4(Tc[k]));
            if (paired) {
              q = mul4p(q, exp_neg4(Tr[k]));
              const Pair4 tr = pair4(Tr[k]), mm = pair4(m);
              Tr[k] = unpair4({sub2(tr.lo, mm.lo), sub2(tr.hi, mm.hi)});
            }
          }
        }
        sc[c * L + lane] = s;
        if (paired) sm[c * L + lane] = q;
      }
    }
    __syncthreads();
    auto write = [&](int i, const float4& v) {
      const int x = x0 + grp * kTXW + i;
      if (x >= a.nx || !yok) return;
      if (scatter) {
        // halo rows lack part of their PSF support: their owner window adds them
        if (lane_writes(a, yb)) scatter4(tmp, tb[tap_slot<R, L>(grp * kTXW + i + R)], yb, v);
      } else {
        *reinterpret_cast<float4*>(tmp + (static_cast<size_t>(z) * a.nx + x) * a.cs + yb) = v;
      }
    };
    float4 pend;  // the mate's term of the output being written
    auto keep = [&](int i, const float4& v) { pend = v; };
    auto write_sum = [&](int i, float4 v) {
      add4p(v, pend);
      write(i, v);
    };
    if (PSF) {
      const float* kr = PTAB ? ptab + z * 2 * K : s_psf + (z - zbeg) * 2 * K;
      if (paired) {  // both row passes in one sweep over the two tiles
        if constexpr (PTAB && ADJ) {
          const float* km = ptab + (a.nz - 1 - z) * 2 * K;
          rowpass2_from_tiles<R, L, L>(sc, sm, grp * kTXW, write_sum, Reversed<R>{kr}, Reversed<R>{kr + K}, keep, km,
                                 Reversed<R>{km + K}, lane, a.ny);
        } else if constexpr (PTAB) {
          const float* km = ptab + (a.nz - 1 - z) * 2 * K;
          rowpass2_from_tiles<R, L, L>(sc, sm, grp * kTXW, write_sum, kr, kr + K, keep, Reversed<R>{km}, km + K, lane,
                                 a.ny);
        } else {
          const float* km = s_psf_m + (z - zbeg) * 2 * K;
          rowpass2_from_tiles<R, L, L>(sc, sm, grp * kTXW, write_sum, kr, kr + K, keep, km, km + K, lane, a.ny);
        }
      } else if constexpr (PTAB && ADJ) {
        rowpass_from_tile<R, L, L>(sc, grp * kTXW, write, Reversed<R>{kr}, Reversed<R>{kr + K}, lane, a.ny);
      } else {
        rowpass_from_tile<R, L, L>(sc, grp * kTXW, write, kr, kr + K, lane, a.ny);
      }
    } else {
#pragma unroll
      for (int i = 0; i < kTXW; ++i) {
        float4 v = sc[(grp * kTXW + i) * L + lane];
        if (paired) add4(v, sm[(grp * kTXW + i) * L + lane]);
        write(i, v);
      }
    }
    if (NB == 1) __syncthreads();  // the single tile buffer is rewritten next plane
  }
}

template <int R, bool PSF, bool ATT, bool ADJ, class V, int L>
__global__ void __launch_bounds__(32 * kW, 2) k_spread_pair_yg(const YgArgs a, int u0) {
  spread_pair_body<R, PSF, ATT, ADJ, false, V, L>(a, u0, nullptr);
}

template <int R, bool ATT, bool ADJ, class V, int L>
__global__ void __launch_bounds__(32 * kW, 2)
    k_spread_pair_ptab_yg(const YgArgs a, int u0, const __grid_constant__ PsfTable t) {
  spread_pair_body<R, true, ATT, ADJ, true, V, L>(a, u0, t.c);
}

// The separated PSF of a.nz planes as a kernel-parameter table, or null when
// it is not available on the host or does not fit.
template <int R>
const PsfTable* psf_table(const YgArgs& a) {
  if (!psf_in_parameters<R>(a)) return nullptr;
  static thread_local PsfTable table;
  std::memcpy(table.c, a.psf_host, sizeof(float) * a.nz * 2 * (2 * R + 1));
  return &table;
}

template <int R, bool ADJ, int L>
int launch_spread_lanes(const YgArgs& a, int c0, int gcount, cudaStream_t st) {
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const dim3 grid(gcount * ntile * a.bslabs), block(32 * kW);
  const bool psf = a.psf != nullptr;
  const PsfTable* tab = psf_table<R>(a);
  const size_t smem = tile_smem_bytes<R, L>(psf && !tab ? a.nz : 0);
  auto go = [&](auto k) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE(ADJ ? "k_adjoint_yg" : "k_spread_yg", st);
    k<<<grid, block, smem, st>>>(a, c0);
  };
  auto go_tab = [&](auto k) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE(ADJ ? "k_adjoint_yg" : "k_spread_yg", st);
    k<<<grid, block, smem, st>>>(a, c0, *tab);
  };
  // only mu is sampled from storage here (the sinogram is float32)
  const bool bf16 = a.storage == kStorageBF16;
  const bool three = 3 * (smem + kYBufBytes<L> + 1024) <= 228 * 1024;
  if (psf && tab) {
    if (a.mu && bf16) {
      go_tab(k_spread_ptab_yg<R, true, ADJ, __nv_bfloat16, 2, L>);
    } else if (a.mu) {
      if constexpr (!ADJ) {
        if (three)
          go_tab(k_spread_ptab_yg<R, true, false, float, 3, L>);
        else
          go_tab(k_spread_ptab_yg<R, true, false, float, 2, L>);
      } else {
        go_tab(k_spread_ptab_yg<R, true, true, float, 2, L>);
      }
    } else {
      go_tab(k_spread_ptab_yg<R, false, ADJ, float, 2, L>);
    }
  } else if (psf) {
    if constexpr (L == 32) {
      if (a.mu && bf16) {
        go(k_spread_yg<R, true, true, ADJ, __nv_bfloat16, 2, L>);
      } else if (a.mu) {
        if constexpr (!ADJ) {
          if (three)
            go(k_spread_yg<R, true, true, false, float, 3, L>);
          else
            go(k_spread_yg<R, true, true, false, float, 2, L>);
        } else {
          go(k_spread_yg<R, true, true, true, float, 2, L>);
        }
      } else {
        go(k_spread_yg<R, true, false, ADJ, float, 2, L>);
      }
    }
  } else if constexpr (R == 0) {
    if (a.mu && bf16) go(k_spread_yg<0, false, true, ADJ, __nv_bfloat16, 2, L>);
    else if (a.mu) go(k_spread_yg<0, false, true, ADJ, float, 2, L>);
    else go(k_spread_yg<0, false, false, ADJ, float, 2, L>);
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}

template <int R, bool ADJ, int L>
int launch_spread_pair_lanes(const YgArgs& a, int u0, int gcount, cudaStream_t st) {
  const int ntile = (a.nx + kTX<L> - 1) / kTX<L>;
  const dim3 grid(gcount * ntile * a.bslabs), block(32 * kW);
  const bool psf = a.psf != nullptr;
  const int zper = (a.nz + a.bslabs - 1) / a.bslabs;
  const PsfTable* tab = psf_table<R>(a);
  // bfloat16 mu: the Kahan form (reference mode only)
  const bool bf16 = a.storage == kStorageBF16 && a.mu && !ADJ;
  const size_t smem = (bf16 ? spread_pair_fixed_smem<R, L, ADJ, __nv_bfloat16>() : spread_pair_fixed_smem<R, L, ADJ, float>()) +
                      (psf && !tab ? sizeof(float) * 2 * zper * 2 * (2 * R + 1) : 0);
  auto go = [&](auto k) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE(ADJ ? "k_adjoint_pair_yg" : "k_spread_pair_yg", st);
    k<<<grid, block, smem, st>>>(a, u0);
  };
  auto go_tab = [&](auto k) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    NRGB_LAUNCH_SCOPE(ADJ ? "k_adjoint_pair_yg" : "k_spread_pair_yg", st);
    k<<<grid, block, smem, st>>>(a, u0, *tab);
  };
  if constexpr (!ADJ) {
    if (bf16) {
      if (psf && tab) go_tab(k_spread_pair_ptab_yg<R, true, false, __nv_bfloat16, L>);
      else if (psf) { if constexpr (L == 32) go(k_spread_pair_yg<R, true, true, false, __nv_bfloat16, L>); }
      else if constexpr (R == 0) go(k_spread_pair_yg<0, false, true, false, __nv_bfloat16, L>);
      return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
    }
  }
  if (psf && tab) {
    if (a.mu) go_tab(k_spread_pair_ptab_yg<R, true, ADJ, float, L>);
    else go_tab(k_spread_pair_ptab_yg<R, false, ADJ, float, L>);
  } else if (psf) {
    if constexpr (L == 32) {
      if (a.mu) go(k_spread_pair_yg<R, true, true, ADJ, float, L>);
      else go(k_spread_pair_yg<R, true, false, ADJ, float, L>);
    }
  } else if constexpr (R == 0) {
    if (a.mu) go(k_spread_pair_yg<0, false, true, ADJ, float, L>);
    else go(k_spread_pair_yg<0, false, false, ADJ, float, L>);
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrKernel;
}


}  // namespace

// Launch the spread of units (or cameras) [c0, c0 + gcount) for one row window
// with its lane count (narrow windows: no PSF, or the PSF in the kernel
// parameters); explicitly instantiated in et_yg_spread_r*.cu.
template <int R, bool ADJ>
int launch_spread_R(const YgArgs& a, int c0, int gcount, cudaStream_t st) {
  if (!a.psf || psf_in_parameters<R>(a)) {
    if (a.lanes == 8) return launch_spread_lanes<R, ADJ, 8>(a, c0, gcount, st);
    if (a.lanes == 16) return launch_spread_lanes<R, ADJ, 16>(a, c0, gcount, st);
  }
  return launch_spread_lanes<R, ADJ, 32>(a, c0, gcount, st);
}

template <int R, bool ADJ>
int launch_spread_pair_R(const YgArgs& a, int u0, int gcount, cudaStream_t st) {
  if (!a.psf || psf_in_parameters<R>(a)) {
    if (a.lanes == 8) return launch_spread_pair_lanes<R, ADJ, 8>(a, u0, gcount, st);
    if (a.lanes == 16) return launch_spread_pair_lanes<R, ADJ, 16>(a, u0, gcount, st);
  }
  return launch_spread_pair_lanes<R, ADJ, 32>(a, u0, gcount, st);
}

}  // namespace nrgb
