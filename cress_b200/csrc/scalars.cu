// Forcing and leapfrog step of the nine moist scalars for sm_100a
// (s_forceqv, s_forceq and their s_steps, cphopt=3):
//   sfrc = advs (advs.f90:205-416, 4th-order horizontal, 2nd- or 4th-order vertical)
//        + smoo4qv / smoo4s of rbr*(qvp-qvbr) or rbr*sp (smoo4s.f90:184-296)
//        + turbs of sp with the eddy diffusivity (forceqv.f90:331-345,
//          forceq.f90:438-452; tubopt 1 and 2)
//        + vspqv / vsps / vsps0 (vspqv.f90:181-198, vsps.f90:181-198, vsps0.f90:114-124)
//   sf   = sp + sfrc*2dtb/rst, clipped at 0 for the mixing ratios
//          (steps.f90:590-764), then vbcs at k = 1, nk-1 (vbcs.f90:116-132).
//
// Design (2.5-D).  A block owns a 32 x 8 tile of columns of THREE species and
// marches its levels upward; a thread owns a pair of x-neighbouring columns
// of all three and computes both with packed FP32x2 arithmetic (f2.cuh).
// For every level one elected thread issues TMA box loads of the species at
// t and t-dt (two rows of y halo), u, v, w (and the eddy viscosity) into a
// 4-stage shared-memory ring guarded by mbarriers: the level being formed, the
// two above it whose own columns it needs, one in flight.
//
// What bounds it: instruction issue.  With one species per thread and the
// terms in the reference's parenthesisation it took about 410 warp
// instructions per pair and species.  Three things cut that: the face
// coefficients (winds times constants, and the mixing's diffusivities) are
// formed once for the three species; the fourth difference of the smoothing
// is one weighted sum per direction, -(s(2) + s(-2)) + 4 (s(1) + s(-1)) - 6 s(0);
// and along z every face product and second difference is formed at one
// level and kept in registers for the next.  The sums are the reference's in
// another order: they differ by FP32 rounding.  At 512 x 512 x 64 1190 -> 665 us, with the
// eddy mixing 1517 -> 747 (the bytes of the nine species at three levels
// and the winds take 310 us at the measured copy bandwidth).
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "common.cuh"
#include "forcing.cuh"
#include "hevi.cuh"
#include "f2.cuh"
#include "tma.cuh"

namespace cress {
namespace {

__host__ __device__ constexpr int r128f(int n) { return (n + 31) / 32 * 32; }  // floats -> multiple of 128 B

constexpr int kScGroup = 3;          // species per block
static_assert(kMoistN % kScGroup == 0, "species groups must tile the nine species");
constexpr int kScPairs = kHeviTX / 2;
constexpr int kScThreads = kScPairs * kScalarTY;
constexpr int kScStages = 4;

// Per-level constants, each twice (one operand pair): advection at a face in
// x (2nd- and 4th-order part), y, z; rbr, -rbr qvbr, the horizontal
// smoothing's rbr smhcoe, 2dtb/rst, the sponge's coefficient, qvbr, and the
// mixing's coefficients in x, y and the diffusivity's factor.
enum ScConst { K_AX, K_BX, K_AY, K_BY, K_W, K_RBR, K_NRQ, K_SMH, K_STEP, K_VSP, K_QV, K_TX, K_TY, K_KR, K_N };

template <bool TURB>
struct ScLayout {
  using R = ScalarRows;
  static constexpr int BX = kHeviBoxX;
  static constexpr int sbox = r128f(BX * R::s);
  // species q of the group at q * 2 * sbox (t), + sbox (t-dt)
  static constexpr int oU = kScGroup * 2 * sbox;
  static constexpr int oV = oU + r128f(BX * R::u);
  static constexpr int oW = oV + r128f(BX * R::v);
  static constexpr int oR = oW + r128f(BX * R::w);
  static constexpr int stage = oR + (TURB ? r128f(BX * R::r) : 0);   // floats per ring stage
  static constexpr uint32_t tx_bytes =
      4u * BX * (kScGroup * 2 * R::s + R::u + R::v + R::w + (TURB ? R::r : 0));
  // ring, mbarriers, then the constants of levels kA-2 .. kB+2
  static constexpr size_t tab = 4 * (size_t)kScStages * stage + 8 * (size_t)kScStages;
  __host__ __device__ static size_t bytes(int levels) { return tab + 8 * (size_t)K_N * (levels + 4); }
};

template <bool TURB, bool ADV3>
__global__ void __launch_bounds__(kScThreads, 3)
k_scalars(const __grid_constant__ MoistMaps m, const __grid_constant__ MoistScalarArgs a) {
  using L = ScLayout<TURB>;
  constexpr int TY = kScalarTY, BX = kHeviBoxX, S = kScStages, NQ = kScGroup;
  const Grid& g = a.g;
  const int ni = g.ni, nj = g.nj, nk = g.nk;
  constexpr int NG = kMoistN / kScGroup;               // species groups
  const int grp = blockIdx.x % NG;                     // the groups of a tile are neighbours
  const int i0 = 2 + (blockIdx.x / NG) * kHeviTX, j0 = 2 + blockIdx.y * TY;
  const int xb = i0 - 2;                              // box x origin (multiple of 32)
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kScPairs + tx;
  const int i = i0 + 2 * tx, j = j0 + ty;
  const bool ownA = (i <= ni - 2) && (j <= nj - 2), ownB = (i + 1 <= ni - 2) && (j <= nj - 2);
  // open x: the points in the columns next to the boundaries (i = 2, ni-2)
  const int edge = g.openx ? ((i == 2 || i == ni - 2) ? 1 : 0) | ((i + 1 == 2 || i + 1 == ni - 2) ? 2 : 0) : 0;
  // this block's levels kA..kB of 2..nk-2 (blockIdx.z) and the last one it
  // stages; level lv lives in slot (lv-kA) % S
  const int kA = 2 + blockIdx.z * a.kchunk, kB = min(kA + a.kchunk - 1, nk - 2);
  const int lmax = min(nk - 1, kB + 2);

  extern __shared__ __align__(1024) float smem[];
  float* ring = smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + S * L::stage);
  float* tab = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(smem) + L::tab);   // [level - (kA-2)][K_N] pairs

  int issued = kA - 1;   // highest level thread 0 has issued
  auto issue = [&](int lv) {
    issued = lv;
    const int s = (lv - kA) % S;
    float* st = ring + s * L::stage;
    uint64_t* bar = &bars[s];
    const int z = lv - 1;
    mbar_arrive_expect_tx(bar, L::tx_bytes);
    for (int p = 0; p < NQ; ++p) {
      tma_load_3d(st + p * 2 * L::sbox, &m.s[grp * NQ + p], xb, j0 - 2, z, bar);
      tma_load_3d(st + (p * 2 + 1) * L::sbox, &m.sp[grp * NQ + p], xb, j0 - 2, z, bar);
    }
    tma_load_3d(st + L::oU, &m.u, xb, j0, z, bar);
    tma_load_3d(st + L::oV, &m.v, xb, j0 - 1, z, bar);
    tma_load_3d(st + L::oW, &m.w, xb, j0, z, bar);
    if constexpr (TURB) tma_load_3d(st + L::oR, &m.rkv, xb, j0 - 2, z, bar);
  };
  if (tid == 0) {
    for (int s = 0; s < S; ++s) mbar_init(&bars[s], 1);
    fence_mbar_init();
    for (int lv = kA; lv <= min(kA + S - 1, lmax); ++lv) issue(lv);
  }
  const float oned24 = 1.f / 24.f;
  for (int n = tid; n < kB - kA + 5; n += kScThreads) {
    const int k = kA - 2 + n;
    if (k < 1 || k > nk) continue;
    const float* c = a.lvl + k * kLevelStride;
    auto C = [&](int f) { return __ldg(c + f); };
    const float rbr = C(C_RBR), qv = C(C_QVBR), jc = C(C_JCB);
    const float kr = a.kdiv ? 1.f : a.cpriv * C(C_IJCB);
    const float rb2 = k < nk ? C(C_RBCT) + __ldg(c + kLevelStride + C_RBCT) : 0.f;
    float v[K_N];
    v[K_AX] = 4.f / 3.f * -.5f * a.dxiv * C(C_RST8U);
    v[K_BX] = oned24 * a.dxiv * C(C_RST8U);
    v[K_AY] = 4.f / 3.f * -.5f * a.dyiv * C(C_RST8V);
    v[K_BY] = oned24 * a.dyiv * C(C_RST8V);
    v[K_W] = -.5f * a.dziv * C(C_RST8W) * (a.sthopt ? C(C_IJCB8W) : 1.f);
    v[K_RBR] = rbr;
    v[K_NRQ] = -rbr * qv;
    v[K_SMH] = a.smhcoe * rbr;
    v[K_STEP] = C(D_DTDRST);
    v[K_VSP] = k >= a.ksp0 - 1 ? .5f * rb2 * C(C_RST) : 0.f;
    v[K_QV] = qv;
    v[K_TX] = .5f * a.dxiv * a.dxiv * jc * C(C_JCB8U) * kr;
    v[K_TY] = .5f * a.dyiv * a.dyiv * jc * C(C_JCB8V) * kr;
    v[K_KR] = kr;
    float2* d = reinterpret_cast<float2*>(tab) + (size_t)n * K_N;
#pragma unroll
    for (int q = 0; q < K_N; ++q) d[q] = make_float2(v[q], v[q]);
  }
  __syncthreads();

  bool fail = false;
  auto wait_level = [&](int lv) {
    if (!fail && lv <= lmax) fail = !mbar_wait(&bars[(lv - kA) % S], ((lv - kA) / S) & 1);
  };
  wait_level(kA);
  wait_level(kA + 1);

  const bool smooth = (a.smtopt % 10 == 2) || (a.smtopt % 10 == 3), smz4 = a.smtopt % 10 == 3;
  const bool qvgrp = grp == 0;   // this block's first species is qv
  const bool vsp0 = a.vspopt >= 1 && (qvgrp ? a.vsp_qv : a.vsp_q), vsp1 = a.vspopt >= 1 && a.vsp_q;
  const F2 zero{0}, four = f2(4.f, 4.f), m12 = f2(-12.f, -12.f), m2 = f2(-2.f, -2.f), smv = f2(a.smvcoe, a.smvcoe);
  // own pair in the boxes (x offset even, so every pair load is 8-byte
  // aligned): species/viscosity rows from j0-2, u and w rows from j0, v
  // rows from j0-1
  const int ox = 2 * tx + 2, oU = L::oU + ty * BX + ox, oV = L::oV + (ty + 1) * BX + ox, oW = L::oW + ty * BX + ox;
  const int oS = (ty + 2) * BX + ox;
  const size_t plane = (size_t)g.plane;
  // non-owned threads read inside the array (their values go nowhere)
  size_t id = (size_t)g.at(min(i, g.px - 2), min(j, nj), kA);
  auto K = [&](int d, int n) { return F2{reinterpret_cast<const uint64_t*>(tab)[(size_t)(d + 2) * K_N + n]}; };
  const float* t_ = tab;   // advanced with k
  auto stage_of = [&](int lv) { return ring + ((lv - kA) % S) * L::stage; };

  // Along z, per species: s at k; sp at k, k+1; the smoothed quantity A =
  // rbr (sp - base) at k, k+1 and its second difference at k-1, k; the
  // advective and the turbulent flux product at the face below level k.
  F2 s0[NQ], sp0[NQ], sp1[NQ], A0[NQ], A1[NQ], d2m[NQ], d20[NQ], tz[NQ], tk[NQ], sm2[NQ], sm1[NQ];
  F2 gm = zero, g0, kz0 = zero;   // w flux at the faces k-1, k (times its constant); diffusivity at k
  {
    const float* st0 = stage_of(kA);
    const float* st1 = stage_of(min(kA + 1, lmax));
    g0 = K(0, K_W) * ld2(st0 + oW);
    const size_t lo1 = id - plane, lo2 = kA > 2 ? id - 2 * plane : lo1;
    if constexpr (TURB) {
      kz0 = K(0, K_KR) * ld2(st0 + L::oR + oS);
    }
    if constexpr (ADV3) gm = K(-1, K_W) * gld2(a.w + lo1);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int n = grp * NQ + q;
      const F2 base0 = q == 0 && qvgrp ? K(0, K_NRQ) : zero, base1 = q == 0 && qvgrp ? K(1, K_NRQ) : zero;
      const F2 basem = q == 0 && qvgrp ? K(-1, K_NRQ) : zero, basem2 = q == 0 && qvgrp && kA > 2 ? K(-2, K_NRQ) : zero;
      s0[q] = ld2(st0 + q * 2 * L::sbox + oS);
      sp0[q] = ld2(st0 + (q * 2 + 1) * L::sbox + oS);
      sp1[q] = ld2(st1 + (q * 2 + 1) * L::sbox + oS);
      const F2 sm = gld2(a.s[n] + lo1), spm = gld2(a.sp[n] + lo1), spm2 = gld2(a.sp[n] + lo2);
      A0[q] = fma2(K(0, K_RBR), sp0[q], base0);
      A1[q] = fma2(K(1, K_RBR), sp1[q], base1);
      const F2 Am = fma2(K(-1, K_RBR), spm, basem);
      const F2 Am2 = kA > 2 ? fma2(K(-2, K_RBR), spm2, basem2) : Am;
      d20[q] = fma2(m2, A0[q], A1[q] + Am);
      d2m[q] = kA > 2 ? fma2(m2, Am, A0[q] + Am2) : d20[q];   // tmp3(kmin-1) = tmp3(kmin)
      tz[q] = g0 * (s0[q] - sm);
      if constexpr (ADV3) {
        sm1[q] = sm;
        sm2[q] = gld2(a.s[n] + lo2);
      }
      if constexpr (TURB) tk[q] = (kz0 + K(-1, K_KR) * gld2(a.rkv + lo1)) * (sp0[q] - spm);
    }
  }
  const F2 tzc = f2(.5f * a.dziv * a.dziv, .5f * a.dziv * a.dziv), z24 = f2(-1.f / 12.f, -1.f / 12.f);
  const F2 f43 = f2(4.f / 3.f, 4.f / 3.f);

  for (int k = kA; k <= kB; ++k, id += plane) {
    wait_level(k + 2);
    // Every thread has finished level k-1: its slot takes level k+S-1.
    __syncthreads();
    if (tid == 0 && !fail && k > kA && k + S - 1 <= lmax) {   // refill only after its copy was seen to land
      fence_proxy_async_smem();
      issue(k + S - 1);
    }
    if (ownA && !fail) {
      tab = const_cast<float*>(t_) + (size_t)(k - kA) * 2 * K_N;
      const float* st0 = stage_of(k);
      const float* st1 = stage_of(k + 1);
      const float* st2 = stage_of(k + 2);
      // face coefficients of the three species (rstuvwc.f90:172-210)
      F2 ax0, ax1, bx0, bx1, ay0, ay1, by0, by1;
      {
        const F2 um = ld2(st0 + oU - 2), u0 = ld2(st0 + oU), u2 = ld2(st0 + oU + 2);
        const F2 uw = mid2(um, u0), u1 = mid2(u0, u2);   // columns -1 and 1
        ax0 = K(0, K_AX) * u0;
        ax1 = K(0, K_AX) * u1;
        bx0 = K(0, K_BX) * (uw + u0);
        bx1 = K(0, K_BX) * (u1 + u2);
        const F2 vm = ld2(st0 + oV - BX), v0 = ld2(st0 + oV), v1 = ld2(st0 + oV + BX), v2 = ld2(st0 + oV + 2 * BX);
        ay0 = K(0, K_AY) * v0;
        ay1 = K(0, K_AY) * v1;
        by0 = K(0, K_BY) * (vm + v0);
        by1 = K(0, K_BY) * (v1 + v2);
      }
      const F2 g1 = K(1, K_W) * ld2(st1 + oW);
      F2 tx0 = zero, tx1 = zero, ty0 = zero, ty1 = zero, kz1 = zero, tks = zero;
      if constexpr (TURB) {   // s_eddydif / s_kh8uv / s_turbs: diffusivity sums at the faces
        const float* r = st0 + L::oR + oS;
        const F2 rm = ld2(r - 2), r0 = ld2(r), r2 = ld2(r + 2);
        tx0 = K(0, K_TX) * (mid2(rm, r0) + r0);
        tx1 = K(0, K_TX) * (r0 + mid2(r0, r2));
        ty0 = K(0, K_TY) * (ld2(r - BX) + r0);
        ty1 = K(0, K_TY) * (r0 + ld2(r + BX));
        kz1 = K(1, K_KR) * ld2(st1 + L::oR + oS);
        tks = kz0 + kz1;
        kz0 = kz1;
      }
      F2 c4m = zero, c4p = zero;
      const bool z4 = ADV3 && k >= 3 && k <= nk - 3;   // advs.f90:372-416: 4th order in z
      if constexpr (ADV3) {
        c4m = z24 * (gm + g0);
        if (z4) c4p = z24 * (g1 + K(2, K_W) * ld2(st2 + oW));
        gm = g0;
      }
      g0 = g1;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const float* ps = st0 + q * 2 * L::sbox + oS;
        const float* pp = ps + L::sbox;
        const F2 c0 = s0[q];
        const F2 sw2 = ld2(ps - 2), se2 = ld2(ps + 2), sw = mid2(sw2, c0), se = mid2(c0, se2);
        const F2 dw = c0 - sw, de = se - c0, ds = c0 - ld2(ps - BX), dn = ld2(ps + BX) - c0;
        // advs.f90:205-370
        F2 f = ax0 * dw;
        f = fma2(ax1, de, f);
        F2 f4 = bx0 * (c0 - sw2);
        f4 = fma2(bx1, se2 - c0, f4);
        f = fma2(ay0, ds, f);
        f = fma2(ay1, dn, f);
        f4 = fma2(by0, c0 - ld2(ps - 2 * BX), f4);
        f4 = fma2(by1, ld2(ps + 2 * BX) - c0, f4);
        F2 h = f + f4;
        const F2 e0 = sp0[q];
        const F2 ew2 = ld2(pp - 2), ee2 = ld2(pp + 2), ew = mid2(ew2, e0), ee = mid2(e0, ee2);
        const F2 es = ld2(pp - BX), en = ld2(pp + BX);
        const F2 n1 = (ew + ee) + (es + en);
        F2 sm4 = zero;
        if (smooth) {   // the horizontal part of smooth_sum
          const F2 n2 = (ew2 + ee2) + (ld2(pp - 2 * BX) + ld2(pp + 2 * BX));
          sm4 = fma2(m12, e0, fma2(four, n1, zero - n2));
        }
        if (edge) {   // open x: 2nd order in the boundary columns (advs.f90:312-350, smoo4s.f90:216-226)
          const F2 h2 = f2(.75f, .75f) * f, s2 = fma2(f2(-4.f, -4.f), e0, n1);
          h = f2((edge & 1) ? h2.x() : h.x(), (edge & 2) ? h2.y() : h.y());
          if (smooth) sm4 = f2((edge & 1) ? s2.x() : sm4.x(), (edge & 2) ? s2.y() : sm4.y());
        }
        // along z
        const F2 c1 = ld2(st1 + q * 2 * L::sbox + oS);
        const F2 tz1 = g1 * (c1 - c0);
        F2 vadv = tz[q] + tz1;
        tz[q] = tz1;
        if constexpr (ADV3) {
          if (z4) {
            const F2 c2 = ld2(st2 + q * 2 * L::sbox + oS);
            vadv = fma2(f43, vadv, fma2(c4m, c0 - sm2[q], c4p * (c2 - c0)));
          }
          sm2[q] = sm1[q];
          sm1[q] = c0;
        }
        h = h + vadv;
        s0[q] = c1;
        const F2 e1 = sp1[q];
        F2 e2 = e1;
        if (smooth) {
          if (k < nk - 2) e2 = ld2(st2 + (q * 2 + 1) * L::sbox + oS);
          const F2 A2 = fma2(K(2, K_RBR), e2, q == 0 && qvgrp ? K(2, K_NRQ) : zero);
          const F2 d2p = k < nk - 2 ? fma2(m2, A1[q], A2 + A0[q]) : d20[q];   // tmp3(kmax+1) = tmp3(kmax)
          h = fma2(K(0, K_SMH), sm4, h);
          F2 v = d20[q];
          // open x: the 4th-order increment skips the boundary columns
          if (smz4) {
            const F2 v4 = (v + v) - (d2p + d2m[q]);
            v = edge ? f2((edge & 1) ? v.x() : v4.x(), (edge & 2) ? v.y() : v4.y()) : v4;
          }
          h = fma2(smv, v, h);
          A0[q] = A1[q];
          A1[q] = A2;
          d2m[q] = d20[q];
          d20[q] = d2p;
        } else if (k < nk - 2) {
          e2 = ld2(st2 + (q * 2 + 1) * L::sbox + oS);
        }
        if constexpr (TURB) {   // turbflx.f90:236-352, turbs.f90:189-232
          F2 t = tx1 * (ee - e0);
          t = fma2(ty1, en - e0, t);
          F2 u = tx0 * (e0 - ew);
          u = fma2(ty0, e0 - es, u);
          const F2 tk1 = tks * (e1 - e0);
          h = h + fma2(tzc, tk1 - tk[q], t - u);
          tk[q] = tk1;
        }
        if (q == 0 ? vsp0 : vsp1) h = h - K(0, K_VSP) * (q == 0 && qvgrp ? e0 - K(0, K_QV) : e0);
        F2 sf = fma2(h, K(0, K_STEP), e0);
        sp0[q] = e1;
        sp1[q] = e2;
        if (grp * NQ + q < 6) sf = f2(fmaxf(sf.x(), 0.f), fmaxf(sf.y(), 0.f));
        // the pair's first index is even, so the pair store is 8-byte aligned
        float* out = a.sf[grp * NQ + q];
        auto put = [&](size_t at) {
          if (ownB) *reinterpret_cast<uint64_t*>(out + at) = sf.b;
          else out[at] = sf.x();
        };
        put(id);
        if (k == 2) put(id - plane);        // vbcs.f90:118
        if (k == nk - 2) put(id + plane);   // vbcs.f90:132
      }
    }
  }

  if (__syncthreads_or(fail)) {
    // A bounded wait gave up: record it and let the copies still in flight
    // land (bounded again) so no TMA write outlives the block.
    if (tid == 0) {
      if (a.err) atomicExch(a.err, 1);
      for (int s = 0; s < S; ++s) {
        int kl = -1;
        for (int lv = kA; lv <= issued; ++lv)
          if ((lv - kA) % S == s) kl = lv;
        if (kl >= 0) mbar_wait(&bars[s], ((kl - kA) / S) & 1);
      }
    }
  }
}

template <bool TURB, bool ADV3>
int launch_sc(const MoistScalarArgs& a, const MoistMaps& maps, cudaStream_t st) {
  using L = ScLayout<TURB>;
  const Grid& g = a.g;
  auto kern = k_scalars<TURB, ADV3>;
  const int n = g.nk - 3;   // levels 2..nk-2
  const size_t most = L::bytes(n);
  if (most > 227 * 1024) return CRESS_E_UNSUPPORTED;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess)
    return CRESS_E_CUDA;
  const int nx = g.ni - 3, ny = g.nj - 3;
  dim3 block(kScPairs, kScalarTY);
  dim3 grid((nx + kHeviTX - 1) / kHeviTX * (kMoistN / kScGroup), (ny + kScalarTY - 1) / kScalarTY);
  MoistScalarArgs b = a;
  b.kchunk = level_chunk(n, (long long)grid.x * grid.y, resident_blocks(kern, kScThreads, most));
  grid.z = (n + b.kchunk - 1) / b.kchunk;
  kern<<<grid, block, L::bytes(b.kchunk), st>>>(maps, b);
  return cudaGetLastError() == cudaSuccess ? 0 : CRESS_E_CUDA;
}

}  // namespace

int launch_moist_scalars(const MoistScalarArgs& a, const MoistMaps& maps, cudaStream_t st) {
  if (a.g.nk < 5) return CRESS_E_UNSUPPORTED;
  if (a.advopt == 3) return a.rkv ? launch_sc<true, true>(a, maps, st) : launch_sc<false, true>(a, maps, st);
  return a.rkv ? launch_sc<true, false>(a, maps, st) : launch_sc<false, false>(a, maps, st);
}

}  // namespace cress
