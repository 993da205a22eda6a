// Forcing and leapfrog step of the turbulent kinetic energy for sm_100a
// (tubopt=2, isoopt=1, flat terrain, no surface flux): s_forcetke
// (SrcOrig/forcetke.f90:269-354) and the TKE part of s_steps, with the
// terms added in the reference's order, each to FP32 rounding
//   tkefrc = advs of the present TKE             (advs.f90:205-370)
//          + jcb rkv ssq                         (sheartke.f90:112-120)
//          + smoo4s of rbr*tkep                  (smoo4s.f90:184-296)
//          - dissipation                         (disptke.f90:181-195)
//          + div(2 K grad tkep), K = rkv/jcb     (eddyvisj.f90:121-134,
//                                                 tkeflx.f90:251-462, turbtke.f90:203-237)
//          - vsps0 of tkep when vspvar(10:10)='o' (vsps0.f90:114-124)
//          - (b(k) + b(k+1)), b(k) = jcb8w N^2(k) (r8s(k-1) + r8s(k)),
//            r8s = 0.5 jcb 1/Pr rkv/jcb         (eddydif.f90:333-359, buoytke.f90:124-151)
//   tkef   = max(0, tkep + tkefrc 2dtb/rst)      (steps.f90:999-1014), then vbcs.
// The shear and dissipation terms, N^2 and the scalar diffusivity come
// per point from k_turb_visc (rks, nsq, shr, dsp); they are read on the
// thread's own columns one level ahead of their use, N^2 and the
// diffusivity of levels k-1 .. k+1 carried in registers as the march goes
// up.
//
// Design (2.5-D), as the moist scalar kernel: a block owns a 32 x 8 tile
// of columns and marches k upward; one elected thread issues TMA boxes of
// the TKE at t and t-dt (two rows of y halo), u, v, w and the eddy
// viscosity (one row of y halo) of every level 1..nk-1 into an S-stage
// shared-memory ring guarded by bounded mbarrier waits, so every neighbour
// of the advection, smoothing and transport stencils is a shared-memory
// read.  Each thread owns a pair of x-neighbouring columns and computes
// both with packed FP32x2 arithmetic (f2.cuh).
//
// What bounds it: instruction issue.  The terms are sums with the per-level
// constants factored out, and the launch bounds name the four blocks per SM
// the ring leaves room for (99 registers, no spills): 270 -> 219 us at
// 512 x 512 x 64.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "common.cuh"
#include "f2.cuh"
#include "forcing.cuh"
#include "hevi.cuh"
#include "stencil.cuh"
#include "tke.cuh"
#include "tma.cuh"

namespace cress {
namespace {

__host__ __device__ constexpr int r128f(int n) { return (n + 31) / 32 * 32; }  // floats -> multiple of 128 B

constexpr int kTkePairs = kHeviTX / 2;

template <int S>
struct TkeLayout {
  using R = TkeRows;
  static constexpr int BX = kHeviBoxX;
  static constexpr int oS = 0;                              // TKE at t, rows j0-2 ..
  static constexpr int oSP = oS + r128f(BX * R::s);         // TKE at t-dt, rows j0-2 ..
  static constexpr int oU = oSP + r128f(BX * R::s);         // rows j0 ..
  static constexpr int oV = oU + r128f(BX * R::u);          // rows j0-1 ..
  static constexpr int oW = oV + r128f(BX * R::v);          // rows j0 ..
  static constexpr int oR = oW + r128f(BX * R::w);          // eddy viscosity, rows j0-1 ..
  static constexpr int stage = oR + r128f(BX * R::r);       // floats per ring stage
  static constexpr uint32_t tx_bytes = 4u * BX * (2 * R::s + R::u + R::v + R::w + R::r);
  static constexpr int NF = kLevelStride;
  __host__ __device__ static size_t bytes() { return 4 * (size_t)S * stage + 8 * (size_t)S; }
};

template <int S>
__global__ void __launch_bounds__(kTkePairs * kScalarTY, 4) k_tke(const __grid_constant__ TkeMaps m, const TkeArgs a) {
  static_assert(S >= 6, "ring too shallow for the k-2..k+2 window");
  using L = TkeLayout<S>;
  constexpr int TY = kScalarTY, BX = kHeviBoxX;
  const Grid g = a.g;
  const int ni = g.ni, nj = g.nj, nk = g.nk;
  const int i0 = 2 + blockIdx.x * kHeviTX, j0 = 2 + blockIdx.y * TY;
  const int xb = i0 - 2;   // box x origin (multiple of 32)
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTkePairs + tx;
  const int i = i0 + 2 * tx, j = j0 + ty;
  // ownB implies ownA (i+1 <= ni-2 gives i <= ni-2)
  const bool ownA = (i <= ni - 2) && (j <= nj - 2), ownB = (i + 1 <= ni - 2) && (j <= nj - 2);

  extern __shared__ __align__(1024) float smem[];
  float* ring = smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + S * L::stage);
  if (tid == 0) {
    for (int s = 0; s < S; ++s) mbar_init(&bars[s], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // this block's levels kA..kB of 2..nk-2 (blockIdx.z), and the levels it
  // stages, two more at either end; level lv lives in slot (lv-lv0) % S
  const int kA = 2 + blockIdx.z * a.kchunk, kB = min(kA + a.kchunk - 1, nk - 2);
  const int lv0 = max(kA - 2, 1), lmax = min(nk - 1, kB + 2);
  int issued = 0;   // highest level thread 0 has issued
  auto issue = [&](int lv) {
    issued = lv;
    const int s = (lv - lv0) % S;
    float* st = ring + s * L::stage;
    uint64_t* bar = &bars[s];
    const int z = lv - 1;
    mbar_arrive_expect_tx(bar, L::tx_bytes);
    tma_load_3d(st + L::oS, &m.s, xb, j0 - 2, z, bar);
    tma_load_3d(st + L::oSP, &m.sp, xb, j0 - 2, z, bar);
    tma_load_3d(st + L::oU, &m.u, xb, j0, z, bar);
    tma_load_3d(st + L::oV, &m.v, xb, j0 - 1, z, bar);
    tma_load_3d(st + L::oW, &m.w, xb, j0, z, bar);
    tma_load_3d(st + L::oR, &m.rkv, xb, j0 - 1, z, bar);
  };
  if (tid == 0)
    for (int lv = lv0; lv <= min(lv0 + S - 1, lmax); ++lv) issue(lv);

  bool fail = false;
  auto wait_level = [&](int lv) {
    if (!fail && lv <= lmax) fail = !mbar_wait(&bars[(lv - lv0) % S], ((lv - lv0) / S) & 1);
  };
  for (int lv = lv0; lv <= kA + 1; ++lv) wait_level(lv);

  const float oned24 = 1.f / 24.f, fourd3 = 4.f / 3.f;
  const float dxv24 = oned24 * a.dxiv, dyv24 = oned24 * a.dyiv;
  const float dxv05n = -.5f * a.dxiv, dyv05n = -.5f * a.dyiv, dzv05n = -.5f * a.dziv;
  const float dxv5 = .5f * a.dxiv, dyv5 = .5f * a.dyiv, dzv5 = .5f * a.dziv;          // tkeflx.f90:192-194
  const float dxiv2 = 2.f * a.dxiv, dyiv2 = 2.f * a.dyiv, dziv2 = 2.f * a.dziv;      // turbtke.f90:193-195
  const bool smooth = (a.smtopt % 10 == 2) || (a.smtopt % 10 == 3);
  const bool vsp = a.vspopt >= 1 && a.vsp_tke;
  // own pair in the boxes (x offset even, so every pair load is 8-byte
  // aligned): TKE rows from j0-2, u and w rows from j0, v and viscosity
  // rows from j0-1
  const int ox = 2 * tx + 2, oU = ty * BX + ox, oV = (ty + 1) * BX + ox;
  const int oS = (ty + 2) * BX + ox, oR = (ty + 1) * BX + ox;
  const long long plane = g.plane;
  long long id = g.at(i, j, kA);
  // per-point fields of levels k-1 .. k+1 on the own columns (registers),
  // each loaded one level ahead of its use
  F2 r8m = f2(0.f), r80 = f2(0.f), nq0 = f2(0.f);
  F2 shr_n = f2(0.f), dsp_n = f2(0.f), r8p_n = f2(0.f), nq1_n = f2(0.f);
  if (ownA) {
    r8m = gld2(a.rks + id - plane);
    r80 = gld2(a.rks + id);
    nq0 = gld2(a.nsq + id);
    shr_n = gld2(a.shr + id);
    dsp_n = gld2(a.dsp + id);
    r8p_n = gld2(a.rks + id + plane);
    nq1_n = gld2(a.nsq + id + plane);
  }
  auto slot_ptr = [&](int lv) { return ring + ((lv - lv0 + S) % S) * L::stage; };
  const float* stp[5] = {slot_ptr(kA - 2), slot_ptr(kA - 1), slot_ptr(kA), slot_ptr(kA + 1), slot_ptr(kA + 2)};

  for (int k = kA; k <= kB; ++k, id += plane) {
    wait_level(k + 2);
    // Every thread has finished level k-1, so the slot of level k-3 (last
    // read as k'-2 at k' = k-1) may be refilled with level k+S-3.
    __syncthreads();
    if (tid == 0 && !fail && k - 3 >= lv0 && k + S - 3 <= lmax) {   // refill only after its copy was seen to land
      fence_proxy_async_smem();
      issue(k + S - 3);
    }
    if (ownA && !fail) {
      const float* ck = a.lvl + k * L::NF;
      auto C = [&](int f, int kk) { return __ldg(ck + (kk - k) * L::NF + f); };
      auto st = [&](int d) { return stp[d + 2]; };
      const float* st0 = st(0);
      const float* S0 = st0 + L::oS + oS;
      const float* SP0 = st0 + L::oSP + oS;
      const float* U = st0 + L::oU + oU;
      const float* V = st0 + L::oV + oV;
      const F2 shr = shr_n, dsp = dsp_n, r8p = r8p_n, nq1 = nq1_n;
      if (k + 1 <= nk - 2) {   // the next level's
        shr_n = gld2(a.shr + id + plane);
        dsp_n = gld2(a.dsp + id + plane);
        r8p_n = gld2(a.rks + id + 2 * plane);
        nq1_n = gld2(a.nsq + id + 2 * plane);
      }

      // advs.f90:205-370 with the fluxes of rstuvwc.f90:172-210, as sums of
      // (wind sum) x (difference) times one per-level constant
      const float r8u = C(C_RST8U, k), r8v = C(C_RST8V, k);
      auto rw = [&](int z) { return a.sthopt ? C(C_RST8W, k + z) * C(C_IJCB8W, k + z) : C(C_RST8W, k + z); };
      auto Wc = [&](int z) { return ld2(st(z) + L::oW + oU); };
      auto Sz = [&](int z) { return ld2(st(z) + L::oS + oS); };
      const F2 u0 = ld2(U), u1 = pair_at(U, 1), v0 = ld2(V), v1 = ld2(V + BX);
      const F2 s0 = ld2(S0);
      F2 f = f2(fourd3 * dxv05n * r8u) * (u0 * (s0 - pair_at(S0, -1)) + u1 * (pair_at(S0, 1) - s0));
      f = fma2(f2(fourd3 * dyv05n * r8v), v0 * (s0 - ld2(S0 - BX)) + v1 * (ld2(S0 + BX) - s0), f);
      f = fma2(f2(dxv24 * r8u),
               (pair_at(U, -1) + u0) * (s0 - ld2(S0 - 2)) + (u1 + ld2(U + 2)) * (ld2(S0 + 2) - s0), f);
      f = fma2(f2(dyv24 * r8v),
               (ld2(V - BX) + v0) * (s0 - ld2(S0 - 2 * BX)) + (v1 + ld2(V + 2 * BX)) * (ld2(S0 + 2 * BX) - s0), f);
      const F2 w0 = rw(0) * Wc(0), w1 = rw(1) * Wc(1);
      const F2 z2 = w0 * (s0 - Sz(-1)) + w1 * (Sz(1) - s0);
      if (a.advopt == 3 && k >= 3 && k <= nk - 3) {   // advs.f90:372-416: 4th order in z
        f = fma2(f2(fourd3 * dzv05n), z2, f);
        f = fma2(f2(oned24 * a.dziv),
                 (rw(-1) * Wc(-1) + w0) * (s0 - Sz(-2)) + (w1 + rw(2) * Wc(2)) * (Sz(2) - s0), f);
      } else {
        f = fma2(f2(dzv05n), z2, f);
      }

      f = f + shr;   // sheartke

      // the TKE at t-dt at an offset (horizontal ones on level k only)
      auto SPo = [&](int dx, int dy, int dz) {
        return dz == 0 ? pair_at(SP0 + dy * BX, dx) : ld2(st(dz) + L::oSP + oS);
      };
      if (smooth) {
        auto H = [&](int dx, int dy) { return SPo(dx, dy, 0); };
        auto A = [&](int dz) { return C(C_RBR, k + dz) * SPo(0, 0, dz); };
        f = smooth_sum(f, a.smtopt, a.smhcoe * C(C_RBR, k), a.smvcoe, k, 2, nk - 2, H, A);
      }

      f = f - dsp;   // disptke

      // eddyvisj + tkeflx + turbtke: K = rkv/jcb, fluxes of jcb*tkep along x
      // and y (where jcb and 1/jcb are per-level constants) and of tkep along z
      const F2 e0 = ld2(SP0);
      const float* R0 = st0 + L::oR + oR;
      const F2 r0 = ld2(R0);
      const F2 mx = (r0 + pair_at(R0, 1)) * (SPo(1, 0, 0) - e0) - (pair_at(R0, -1) + r0) * (e0 - SPo(-1, 0, 0));
      const F2 my = (r0 + ld2(R0 + BX)) * (SPo(0, 1, 0) - e0) - (ld2(R0 - BX) + r0) * (e0 - SPo(0, -1, 0));
      auto Kz = [&](int z) { return C(C_IJCB, k + z) * ld2(st(z) + L::oR + oR); };
      const F2 k0 = C(C_IJCB, k) * r0;
      const F2 mz = (k0 + Kz(1)) * (SPo(0, 0, 1) - e0) - (Kz(-1) + k0) * (e0 - SPo(0, 0, -1));
      const float jk = C(C_JCB, k) * C(C_IJCB, k);
      f = fma2(f2(dzv5 * dziv2), mz, f);
      f = fma2(f2(dxv5 * dxiv2 * (jk * C(C_JCB8U, k))), mx, f);
      f = fma2(f2(dyv5 * dyiv2 * (jk * C(C_JCB8V, k))), my, f);

      if (vsp && k >= a.ksp0 - 1) f = f - (.5f * (C(C_RBCT, k) + C(C_RBCT, k + 1))) * C(C_RST, k) * e0;

      // buoytke with the half diffusivities 0.5 jcb rks of eddydif
      const F2 q0 = C(C_JCB, k) * r80;
      const F2 b0 = nq0 * fma2(f2(C(C_JCB, k - 1)), r8m, q0), b1 = nq1 * fma2(f2(C(C_JCB, k + 1)), r8p, q0);
      f = f - fma2(f2(.5f * C(C_JCB8W, k)), b0, .5f * C(C_JCB8W, k + 1) * b1);

      const F2 sf = fmax2(fma2(f2(C(D_DTDRST, k)), f, e0), 0.f);
      auto put = [&](long long at) {
        if (ownB) st2(a.tkef + at, sf);
        else a.tkef[at] = sf.x();
      };
      put(id);
      if (k == 2) put(id - plane);        // vbcs.f90:118
      if (k == nk - 2) put(id + plane);   // vbcs.f90:132
      r8m = r80;
      r80 = r8p;
      nq0 = nq1;
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) stp[d] = stp[d + 1];
    stp[4] = slot_ptr(k + 3);
  }

  if (__syncthreads_or(fail)) {
    // A bounded wait gave up: record it and let the copies still in flight
    // land (bounded again) so no TMA write outlives the block.
    if (tid == 0) {
      if (a.err) atomicExch(a.err, 1);
      for (int s = 0; s < S; ++s) {
        int kl = -1;
        for (int lv = lv0; lv <= issued; ++lv)
          if ((lv - lv0) % S == s) kl = lv;
        if (kl >= 0) mbar_wait(&bars[s], ((kl - lv0) / S) & 1);
      }
    }
  }
}

}  // namespace

int launch_tke(const TkeArgs& a, const TkeMaps& maps, cudaStream_t st) {
  constexpr int S = 6;
  using L = TkeLayout<S>;
  const Grid& g = a.g;
  if (g.nk < 5) return CRESS_E_UNSUPPORTED;
  const size_t bytes = L::bytes();
  if (cudaFuncSetAttribute(k_tke<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return CRESS_E_CUDA;
  const int nx = g.ni - 3, ny = g.nj - 3;
  dim3 block(kTkePairs, kScalarTY, 1);
  dim3 grid((nx + kHeviTX - 1) / kHeviTX, (ny + kScalarTY - 1) / kScalarTY);
  const int n = g.nk - 3;   // levels 2..nk-2
  TkeArgs b = a;
  b.kchunk = level_chunk(n, (long long)grid.x * grid.y, resident_blocks(k_tke<S>, kTkePairs * kScalarTY, bytes));
  grid.z = (n + b.kchunk - 1) / b.kchunk;
  k_tke<S><<<grid, block, bytes, st>>>(maps, b);
  return cudaGetLastError() == cudaSuccess ? 0 : CRESS_E_CUDA;
}

}  // namespace cress
