// HE-VI acoustic substep marching rows (s_hevi, SrcOrig/hevi.f90:339-426,
// impopt=1, flat terrain, periodic lateral or open x boundaries, rigid
// lid): the same operators and boundary rules as k_hevi2.
//
// Layout.  A block owns a strip of 60 columns in x and `rows` rows in y
// over the whole height, and marches j.  Warp c holds the levels
// k = 2 + c L .. 2 + c L + L - 1 of the column (its chunk, at most 16 chunks);
// lane t holds the column pair i0 - 2 + 2t, i0 - 1 + 2t, so lanes 1..30 own 60
// columns and lanes 0 and 31 recompute the neighbouring tiles' edge columns:
// every x neighbour is a shuffle and no lane takes a special path.  Marching
// j, the y neighbours are the thread's own previous row, kept in registers.
// Both columns of the pair go through packed FP32x2 instructions.  Each warp
// stages its own row of the eight input fields with TMA (boxes of 64 columns x
// 1 row x L levels, one mbarrier per warp): the next row's copy starts as soon
// as the warp has read this one and lands while it works on the solve.
//
// The FP64 solve.  The matrix depends on k only, so the elimination
// f(k) = a(k) r(k) + b(k) f(k-1) and the back substitution
// w(k) = f(k) - cp(k) w(k+1) are linear recurrences with fixed factors.
// Each warp runs its chunk from a zero entry value, the chunks' end values
// go through shared memory, every warp folds the chunks below (above) it
// into its own entry value, and the chunk is corrected with the known
// products of its factors: two block barriers per row, and the column stays in
// FP64 registers from the right-hand side to w.
//
// The periodic images in x are stored with the points; the y ghosts and the
// levels 1, nk-1 and nk are not read by the next substep (it reads the rows
// the ghosts repeat, HeviRowArgs::wrap) and are written once after the last
// one (k_hevi_row_ends).
//
// Why this shape, and what it measured (us per substep; marching k with a
// ring of xy tiles before, tile 0 / tile 13 -> this kernel):
//   64 x 64 x 40    85 -> 10    (16 tiles on 148 SMs, 64 levels in a row)
//   203 x 131 x 54  125 -> 27
//   512 x 512 x 64  321 / 289 -> 175: 4.6 TB/s of its 48 bytes per cell, 0.70 of
//                   the measured copy bandwidth, 54.3 bytes per cell of DRAM traffic
// Marching k, all levels of a column wait for one another and a grid of few
// tiles leaves SMs idle; a substep also spent about 270 warp instructions per 32
// cells, half of them on ring, address and halo bookkeeping.  Here the levels
// of a row run at once, the strip length adapts to the grid, and it is about
// 155 per 32 cells.  It is bound by the latency of its 16 warps per SM: 128 registers each
// (which is why a row's p' tendency and w right-hand side wait in
// shared memory, and why the row's addresses, the stage's place and the number of
// own levels are formed again each row: 195 -> 175 us at 512 x 512 x 64), two
// barriers per row.  Tried and slower: direct global loads instead of TMA (406 us at
// 512 x 512 x 64: the row's loads are not in flight during the solve),
// prefetching a second row into L2 by TMA (235 us), both rows' values in
// registers (265 us: spills).
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include "common.cuh"
#include "f2.cuh"
#include "hevi_row.cuh"
#include "status.h"
#include "tma.cuh"

namespace cress {
namespace {

constexpr int kHrCols = 60;       // columns a tile owns (64 held)
constexpr int kHrMaxWarps = 16;

// (second column, first of the next lane): the pair one column to the east
__device__ __forceinline__ F2 east(F2 a) { return f2(a.y(), __shfl_down_sync(0xffffffffu, a.x(), 1)); }
// (second of the previous lane, first column): the pair one column to the west
__device__ __forceinline__ F2 west(F2 a) { return f2(__shfl_up_sync(0xffffffffu, a.y(), 1), a.x()); }

// The row of the old level that holds row r's values: itself, or with the
// wrap (the y ghosts not written) its periodic image (SrcOrig/bcycle.f90).
__device__ __forceinline__ int wrap_row(const HeviRowArgs& a, bool vrow, int r) {
  if (a.wrap) {
    if (r == 1) return a.g.nj - 2;
    if (vrow ? r == a.g.nj : r == a.g.nj - 1) return vrow ? 3 : 2;
  }
  return r;
}

// Programmatic dependent launch: the next substep's blocks are scheduled once
// every block of this one is in its last row, as they leave their SMs, and set up
// (barriers, tables) while the rest finish; grid_dependency_wait then waits
// for all of it, with its stores visible.  Plain launches / triggered at
// the block's start / in the last row, us per substep: 64 x 64 x 40 14.3 / 11.0 /
// 10.4, 203 x 131 x 54 31.2 / 29.3 / 28.0, 512 x 512 x 64 196.8 / 202.8 / 196.0 (blocks that wait
// on a free SM while others work cost more than they save).
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
int launch_dependent(dim3 grid, int threads, size_t bytes, cudaStream_t st, void (*kernel)(P...), const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...) == cudaSuccess ? 0 : CRESS_E_CUDA;
}

// What only lanes at the domain's x edges store besides their pair, as one
// word (0: nothing): bit 0: the first column alone (the pair's second is not
// the tile's), bits 2 and up: byte offset to the periodic image (0: none) of the
// second (bit 1) or the first column.  n0, n1: whether the pair's columns
// are the tile's.
__device__ __forceinline__ int edge_code(const Grid& g, bool ustag, int i, bool n0, bool n1) {
  int e = n0 && !n1 ? 1 : 0;
  if (g.openx) return e;
  if (n0 && i == g.ni - 2) return e | 4 * (4 * (1 - i));
  if (n1 && i + 1 == g.ni - 2) return e | 2 | 4 * (4 * (1 - i));   // from the pair's place to column 1
  if (n0 && i == 2) return ustag ? e | 2 | 4 * (4 * (g.ni - 2)) : e | 4 * (4 * (g.ni - 3));   // u: column 3 to ni
  return e;
}
__device__ __forceinline__ void put_edge(char* p, F2 x, int e) {
  if (e & 1) *reinterpret_cast<float*>(p) = x.x();
  if (e >> 2) *reinterpret_cast<float*>(p + (e >> 2)) = (e & 2) ? x.y() : x.x();
}

// Shared memory (bytes), at offsets known to the compiler; only the stages,
// which come last, depend on the number of warps.
template <int L>
struct HrLayout {
  static constexpr int W = kHrMaxWarps;
  static constexpr int oE = 0, oW = oE + 16 * W * 32;             // exchange buffers [chunk][lane]: double2
  static constexpr int oM = oW + 16 * W * 32;                     // two fold matrices [chunk][16]: double
  static constexpr int oD = oM + 2 * 8 * W * W;                   // per level (a, b, cp, P): 2 double2
  static constexpr int oN = oD + 32 * W * L;                      // per chunk (bn, an): double2
  static constexpr int oT = oN + 16 * W;                          // level table: kHrVec float4 per level
  static constexpr int oB = oT + 16 * kHrVec * W * L;             // barriers
  static constexpr int oS = (oB + 8 * W + 127) / 128 * 128;       // stages
  // a warp's stage: row pieces (64 floats) of L levels of u, v, p and the
  // forcings, L + 1 levels of w
  static constexpr int row = 256;
  static constexpr int sU = 0, sV = row * L, sP = 2 * row * L, sUF = 3 * row * L, sVF = 4 * row * L,
                       sWF = 5 * row * L, sPF = 6 * row * L, sW = 7 * row * L, stage = row * (8 * L + 1);
  // row r-1's wr and Bs wait in shared memory where they fit beside the
  // stages (Bs with up to four levels per chunk): with them in registers the
  // row loop spills (five levels with wr in registers too: 86.4 us per
  // substep at 512 x 128 x 80, with it here 80.9)
  static constexpr bool park = L <= 4;   // Bs too
  static constexpr int parked = (park ? 2 : 1) * row * L;
  __host__ __device__ static size_t bytes(int nC) { return oS + (size_t)nC * (stage + parked); }
};

// EDGE: the tile holds columns whose values have images in x (the others
// carry no code for them).  BATCH: the block has the warps of the launch's
// tallest grid; those beyond this one's chunks leave, and the barriers count
// the others.
template <int L, bool EDGE, bool BATCH>
__device__ __forceinline__ void hevi_row_strip(const HeviRowMaps& m, const HeviRowArgs& a, unsigned char* smem, int bx,
                                               int by) {
  using Y = HrLayout<L>;
  const Grid& g = a.g;
  const int nk = g.nk, ni = g.ni, nj = g.nj;
  const int lane0 = threadIdx.x & 31, c0 = threadIdx.x >> 5;
  const int nC = BATCH ? (nk - 4 + L) / L : blockDim.x >> 5;   // levels 2..nk-2
  const int k0 = 2 + c0 * L;

  auto stage_of = [&](int c) { return smem + Y::oS + c * (Y::stage + Y::parked); };
  auto bar_of = [&](int c) { return reinterpret_cast<uint64_t*>(smem + Y::oB) + c; };
  const int i0 = 2 + bx * kHrCols, i = i0 - 2 + 2 * lane0;
  const int j0 = 2 + by * a.rows, j1 = min(j0 + a.rows - 1, nj - 2);

  // Lane 0: stage row r (v one row further north) of the warp's levels.
  auto issue = [&](int r, int c) {
    unsigned char* stage = stage_of(c);
    uint64_t* bar = bar_of(c);
    mbar_arrive_expect_tx(bar, Y::stage);
    const int x = i0 - 2, z = 1 + c * L;   // x = 60 bx: a multiple of 4 floats
    const int rs = wrap_row(a, false, r);
    tma_load_3d(stage + Y::sU, &m.u, x, rs, z, bar);
    tma_load_3d(stage + Y::sV, &m.v, x, wrap_row(a, true, r + 1), z, bar);
    tma_load_3d(stage + Y::sP, &m.p, x, rs, z, bar);
    tma_load_3d(stage + Y::sW, &m.w, x, rs, z, bar);
    tma_load_3d(stage + Y::sUF, &m.uf, x, r, z, bar);
    tma_load_3d(stage + Y::sVF, &m.vf, x, r, z, bar);
    tma_load_3d(stage + Y::sWF, &m.wf, x, r, z, bar);
    tma_load_3d(stage + Y::sPF, &m.pf, x, r, z, bar);
  };
  if (lane0 == 0) {
    mbar_init(bar_of(c0), 1);
    fence_mbar_init();
  }
  // Up to here and through the tables below nothing a running kernel writes
  // is read.
  {
    auto fill = [&](int o, const void* src, int n16) {
      for (int n = threadIdx.x; n < n16; n += blockDim.x)
        reinterpret_cast<uint4*>(smem + o)[n] = __ldg(reinterpret_cast<const uint4*>(src) + n);
    };
    fill(Y::oT, a.tab.lev, nC * L * kHrVec);
    fill(Y::oD, a.tab.dbl, 2 * nC * L);
    fill(Y::oN, a.tab.dbl + 2 * nC * L, nC);
    fill(Y::oM, a.tab.dbl + (2 * L + 1) * nC, kHrMaxWarps * kHrMaxWarps);
    // hand-overs of chunks beyond nC: the folds run in steps of four, and of the
    // top chunk, which hands nothing on (its levels above nk-2 may hold
    // NaN)
    for (int n = (nC - 1) * 32 + threadIdx.x; n < kHrMaxWarps * 32; n += blockDim.x)
      reinterpret_cast<uint4*>(smem + Y::oE)[n] = reinterpret_cast<uint4*>(smem + Y::oW)[n] = make_uint4(0, 0, 0, 0);
  }
  grid_dependency_wait();
  if (lane0 == 0 && (!BATCH || c0 < nC)) issue(j0 - 1, c0);
  __syncthreads();
  if (BATCH && c0 >= nC) return;
  auto block_sync = [&]() {
    if constexpr (BATCH) asm volatile("bar.sync 1, %0;" ::"r"(32 * nC) : "memory");
    else __syncthreads();
  };

  const int ilast = min(i0 + kHrCols - 1, ni - 2);
  const bool o0 = i >= i0 && i <= ilast, o1 = i + 1 >= i0 && i + 1 <= ilast;
  // the u face at ni-1 belongs to the tile that owns column ni-2
  const bool uf = ilast == ni - 2, u0 = o0 || (uf && i == ni - 1), u1 = o1 || (uf && i + 1 == ni - 1);
  const uint32_t px4 = 4u * (uint32_t)g.px, plane4 = 4u * (uint32_t)g.plane;
  const size_t at0 = 4 * ((size_t)(k0 - 1) * g.plane + (size_t)(j0 - 2) * g.px + i);   // (i, j0-2, k0)
  size_t at_r = at0;   // row r of the new u and v; row r-1 of the new w and p' is px4 below
  auto lo2 = [](ulonglong2 q) { return F2{q.x}; };
  auto hi2 = [](ulonglong2 q) { return F2{q.y}; };

  const int es = EDGE ? edge_code(a.g, false, i, o0, o1) : 0, eu = EDGE ? edge_code(a.g, true, i, u0, u1) : 0;
  const bool edge = es | eu;
  const F2 zero{0}, dxiv{a.dxiv2}, dyiv{a.dyiv2}, dziv{a.dziv2};
  F2 tc[L], vc[L], vsp[L];                     // row r-1: damped pressure, new v; row r: v
  F2 pk[L];                                    // row r-1: p'
  F2 held[Y::park ? 1 : L];                    // row r-1: explicit p' tendency but the v part (w right-hand side: parked)
  F2 wf0 = zero, t30 = zero, t3l = zero;       // row r-1: what the chunk's first and last level hand on
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const int k = min(k0 + l, nk), ic = min(i, g.px - 2);
    const size_t at = (size_t)(k - 1) * g.plane + (size_t)wrap_row(a, true, j0 - 1) * g.px + ic;
    vc[l] = ld2(a.v + at);   // not a read-only load: it must stay below the dependency wait
    tc[l] = vsp[l] = pk[l] = zero;
    uint64_t* h = reinterpret_cast<uint64_t*>(stage_of(c0) + Y::stage + Y::row * l + 8 * lane0);
    h[0] = 0;
    if constexpr (Y::park) h[Y::row / 8 * L] = 0;
    else held[l] = zero;
  }
  bool fail = false;
  uint32_t par = 0;

  // row j0-1 gives the damped pressure only, row j1+1 that and the v face
  // north of the strip
  for (int r = j0 - 1; r <= j1 + 1; ++r) {
    at_r += px4;
    // opaque to the compiler, so that what is derived from them is formed
    // where it is used instead of being held in registers across the loop
    int lane = lane0, c = c0;
    uint32_t pl4 = plane4;
    size_t at = at_r;
    asm volatile("" : "+r"(lane), "+r"(c), "+r"(pl4), "+l"(at));
    char* const pu = reinterpret_cast<char*>(a.un) + at;
    char* const pv = reinterpret_cast<char*>(a.vn) + at;
    char* const pw = reinterpret_cast<char*>(a.wn) + at - px4;
    char* const pp = reinterpret_cast<char*>(a.pn) + at - px4;
    const int nlev = min(L, nk - 3 - c * L);      // own levels k0 .. k0 + nlev - 1 <= nk-2
    const bool top = c * L + nlev == nk - 3;
    const unsigned char* sp = smem + Y::oS + c * (Y::stage + Y::parked) + 8 * lane;
    const unsigned char* ct = smem + Y::oT + c * (16 * kHrVec * L);
    const unsigned char* dt = smem + Y::oD + c * (32 * L);
    auto T = [&](int l, int n) { return *reinterpret_cast<const ulonglong2*>(ct + 16 * (kHrVec * l + n)); };
    auto D = [&](int l, int n) { return *reinterpret_cast<const double2*>(dt + 16 * (2 * l + n)); };
    auto S = [&](int o, int l) { return F2{*reinterpret_cast<const uint64_t*>(sp + o + Y::row * l)}; };
    auto get = [&](int n) {
      if (n & 1) return S(Y::stage, n >> 1);
      if constexpr (Y::park) return S(Y::stage, L + (n >> 1));
      else return held[n >> 1];
    };
    auto set = [&](int n, F2 x) {
      auto put = [&](int m) {
        *reinterpret_cast<uint64_t*>(const_cast<unsigned char*>(sp) + Y::stage + Y::row * m) = x.b;
      };
      if (n & 1) put(n >> 1);
      else if constexpr (Y::park) put(L + (n >> 1));
      else held[n >> 1] = x;
    };
    // level l's pair into a new field, and what an edge lane adds
    auto emit = [&](char* p, int l, F2 x, bool on) {
      if (on) *reinterpret_cast<uint64_t*>(p + (uint64_t)pl4 * l) = x.b;
    };
    auto extra = [&](char* p, int l, F2 x, int e) {
      if (e) put_edge(p + (uint64_t)pl4 * l, x, e);
    };
    if (!fail) {   // a warp whose wait gave up stages nothing more and goes on with the barriers
      fail = !__all_sync(0xffffffffu, mbar_wait(bar_of(c), par, a.spin));
      if (L <= 4 && !fail) par ^= 1u;
    }
    // Level by level: row r's divergence and faces, then what row r-1 still
    // needed of them (its v part: row r-1 is complete from here on), then the
    // explicit part of row r.  Rows j0-1 and j1+1 go through the same
    // arithmetic; only the results that belong to the strip are stored.
    const bool su = r >= j0 && r <= j1, sv = r >= j0 && (r <= j1 || r == nj - 1);   // row nj-1: the last v face
    const bool fu = su && u1, fv = sv && o1;
    F2 q[L];
    double fa[L], fb[L];
    {
      F2 Gpp = zero, t3p = zero, w = S(Y::sW, 0), W0 = hi2(T(0, 3)) * w;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        const ulonglong2 q0 = T(l, 0), q1 = T(l, 1), q2 = T(l, 2), q3 = T(l, 3);
        const F2 u = S(Y::sU, l), vN = S(Y::sV, l), p = S(Y::sP, l), w1 = S(Y::sW, l + 1), wf = S(Y::sWF, l);
        // diver3d.f90:318 with phy2cnt.f90:219
        const F2 W1 = lo2(q1) * w1;
        F2 div = fma2(lo2(q0), u - east(u), W0 - W1);
        div = fma2(hi2(q0), vc[l] - vN, div);
        // pgrad.f90:341,363 and :300
        const F2 t = fma2(lo2(q2), div, hi2(q1) * p), t3 = fma2(hi2(q2), div, p);
        // stepuv.f90:304 with pgrad.f90:389: the south v face
        const F2 vs = fma2(lo2(q3), fma2(tc[l] - t, dyiv, S(Y::sVF, l)), vc[l]);
        vc[l] = vN;
        tc[l] = t;
        {   // row r-1
          const ulonglong2 q4 = T(l, 4), q5 = T(l, 5), q6 = T(l, 6);
          const F2 fp = fma2(lo2(q4), vsp[l] - vs, get(2 * l));            // advbspi.f90:158 with diver2d.f90:288
          q[l] = fma2(hi2(q4), fp, pk[l]);                              // steppi.f90:217, explicit part
          const F2 gd = lo2(q5) * fp;                                   // pgradiv.f90:149,163
          const F2 wb = fma2(lo2(q6), fp, hi2(q5) * pk[l]);             // buoywsi.f90:171
          const F2 Gp = gd + wb, Gm = gd - wb;
          const double2 ab = D(l, 0);
          const F2 wp = get(2 * l + 1);
          if (l == 0) {   // the level below belongs to the chunk below: its part enters with the chunk's entry value
            const double cw = (double)(hi2(q6)).x(), dz = (double)dziv.x();
            fa[0] = __dmul_rn(ab.x, __fma_rn(cw, __fma_rn(-dz, (double)t30.x(), (double)wf0.x()) - (double)Gm.x(), (double)wp.x()));
            fb[0] = __dmul_rn(ab.x, __fma_rn(cw, __fma_rn(-dz, (double)t30.y(), (double)wf0.y()) - (double)Gm.y(), (double)wp.y()));
            // w of level 2 is zero whatever its forcing, which is not the
            // operator's to read, holds (a factor of zero would pass NaN on)
            if (c == 0) fa[0] = fb[0] = 0.0;
          } else {        // stepwi.f90:325, gaussel.f90:189-240
            const F2 rw = fma2(hi2(q6), Gpp - Gm, wp);
            fa[l] = __fma_rn(ab.y, fa[l - 1], __dmul_rn(ab.x, (double)rw.x()));
            fb[l] = __fma_rn(ab.y, fb[l - 1], __dmul_rn(ab.x, (double)rw.y()));
          }
          Gpp = Gp;
          if (l == L - 1) {   // what this chunk hands to the one above
            const double dz = (double)dziv.x();
            const double2 e = *reinterpret_cast<const double2*>(smem + Y::oN + 16 * c);   // bn, an
            if (!top)
              *reinterpret_cast<double2*>(smem + Y::oE + 16 * (c * 32 + lane)) =
                  make_double2(__fma_rn(e.x, fa[l], __dmul_rn(e.y, __fma_rn((double)t3l.x(), dz, (double)Gpp.x()))),
                               __fma_rn(e.x, fb[l], __dmul_rn(e.y, __fma_rn((double)t3l.y(), dz, (double)Gpp.y()))));
          }
          vsp[l] = vs;
        }
        // stepuv.f90:294 with pgrad.f90:379: the west u face
        const ulonglong2 q7 = T(l, 7), q8 = T(l, 8);
        const F2 un = fma2(lo2(q7), fma2(west(t) - t, dxiv, S(Y::sUF, l)), u);
        if (l < nlev) {
          emit(pv, l, vs, fv);
          emit(pu, l, un, fu);
          if constexpr (EDGE) {
            if (edge) {
              if (sv) extra(pv, l, vs, es);
              if (su) extra(pu, l, un, eu);
            }
          }
        }
        // advbspi.f90:158 without the v part of diver2d.f90:288
        const F2 B = fma2(lo2(q8), w + w1, fma2(hi2(q7), un - east(un), S(Y::sPF, l)));
        set(2 * l, fma2(hi2(q8), w - w1, B));
        pk[l] = p;
        if (l == 0) { set(1, w); wf0 = wf; t30 = t3; }
        else set(2 * l + 1, fma2(hi2(T(l, 6)), fma2(t3p - t3, dziv, wf), w));   // pgrad.f90:320, stepwi.f90:325
        if (l == L - 1) t3l = t3;
        t3p = t3;
        w = w1;
        W0 = W1;
      }
    }
    __syncwarp();   // every lane has read the stage
    if (lane == 0 && !fail && r <= j1) {
      fence_proxy_async_smem();
      issue(r + 1, c);
    }
    // Where the parity is turned decides what the compiler spills: here for
    // five levels (75 us per substep at 512 x 128 x 80, 81 above), above for
    // four (178.8 at 512 x 512 x 64, 191.5 here).
    if (L > 4 && !fail) par ^= 1u;
    if (r <= j0) continue;
    if (r == j1 + 1) grid_launch_dependents();   // the strip's last solve
    if (nlev < L) {   // levels above nk-2: nothing they hold may enter the sums
#pragma unroll
      for (int l = 1; l < L; ++l)
        if (l >= nlev) fa[l] = fb[l] = 0.0;
    }
    block_sync();
    double xa = 0.0, xb = 0.0;
    for (int n = 0; n < c; n += 4) {   // the entry value from the chunks below
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double2 h = *reinterpret_cast<const double2*>(smem + Y::oE + 16 * ((n + e) * 32 + lane));
        const double m = *reinterpret_cast<const double*>(smem + Y::oM + 8 * (c * Y::W + n + e));
        xa = __fma_rn(m, h.x, xa);
        xb = __fma_rn(m, h.y, xb);
      }
    }
    double ya = 0.0, yb = 0.0;
#pragma unroll
    for (int l = L - 1; l >= 0; --l) {
      const double2 cp = D(l, 1);   // cp, P
      fa[l] = __fma_rn(cp.y, xa, fa[l]);
      fb[l] = __fma_rn(cp.y, xb, fb[l]);
      ya = __fma_rn(-cp.x, ya, fa[l]);
      yb = __fma_rn(-cp.x, yb, fb[l]);
    }
    *reinterpret_cast<double2*>(smem + Y::oW + 16 * (c * 32 + lane)) = make_double2(ya, yb);
    block_sync();
    ya = yb = 0.0;
    for (int n = (c + 1) & ~3; n < nC; n += 4) {   // w of the level above, from the chunks above
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double2 h = *reinterpret_cast<const double2*>(smem + Y::oW + 16 * ((n + e) * 32 + lane));
        const double m = *reinterpret_cast<const double*>(smem + Y::oM + 8 * ((Y::W + c) * Y::W + n + e));
        ya = __fma_rn(m, h.x, ya);
        yb = __fma_rn(m, h.y, yb);
      }
    }
    // back substitution (gaussel.f90:254) and the p' update (steppi.f90:217,
    // diverpiv.f90:124, advbspi.f90:175)
    F2 wup = f2((float)ya, (float)yb);
#pragma unroll
    for (int l = L - 1; l >= 0; --l) {
      const ulonglong2 q9 = T(l, 9);
      const double cp = D(l, 1).x;
      ya = __fma_rn(-cp, ya, fa[l]);
      yb = __fma_rn(-cp, yb, fb[l]);
      const F2 wn = f2((float)ya, (float)yb);
      const F2 pn = fma2(hi2(q9), wn - wup, fma2(lo2(q9), wn + wup, q[l]));
      if (l < nlev) {
        emit(pw, l, wn, o1);
        emit(pp, l, pn, o1);
        if constexpr (EDGE) {
          if (edge) {
            extra(pw, l, wn, es);
            extra(pp, l, pn, es);
          }
        }
      }
      wup = wn;
    }
    if (top) {   // w(nk-1) = 0 (vbcw.f90:481): the next substep reads it
      emit(pw, nlev, zero, o1);
      if constexpr (EDGE) extra(pw, nlev, zero, es);
    }
  }

  if (fail && lane0 == 0) {   // the copy in flight lands before the block leaves
    atomicExch(a.err, 1);
    mbar_wait(bar_of(c0), par);
  }
}

template <int L>
__global__ void __launch_bounds__(32 * kHrMaxWarps, 1)
k_hevi_row(const __grid_constant__ HeviRowMaps m, const __grid_constant__ HeviRowArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  if (blockIdx.x == 0 || blockIdx.x + 1 == a.tiles_x) hevi_row_strip<L, true, false>(m, a, smem, blockIdx.x, blockIdx.y);
  else hevi_row_strip<L, false, false>(m, a, smem, blockIdx.x, blockIdx.y);
}

// Every member of an ensemble in one launch: block b belongs to the member
// whose first_block is the largest not above b.
template <int L>
__global__ void __launch_bounds__(32 * kHrMaxWarps, 1) k_hevi_row_batch(const HeviRowJob* __restrict__ jobs, int njobs) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int b = blockIdx.x;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].first_block <= b) lo = mid;
    else hi = mid - 1;
  }
  const HeviRowJob& job = jobs[lo];
  if ((threadIdx.x & 31) == 0) {
    // the maps were copied into global memory by the host: make that copy
    // visible to the tensor-map proxy before this thread's loads read them
    const CUtensorMap* mp = &job.maps.u;
    for (int q = 0; q < 8; ++q)
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(mp + q) : "memory");
  }
  // the member's arguments in shared memory, where the kernel's stores do
  // not alias them
  __shared__ alignas(16) uint32_t words[sizeof(HeviRowArgs) / 4];
  static_assert(sizeof(HeviRowArgs) % 4 == 0, "HeviRowArgs is copied as words");
  for (int w = threadIdx.x; w < (int)(sizeof(HeviRowArgs) / 4); w += blockDim.x)
    words[w] = reinterpret_cast<const uint32_t*>(&job.args)[w];
  __syncthreads();
  const HeviRowArgs& a = *reinterpret_cast<const HeviRowArgs*>(words);
  const int t = b - job.first_block, bx = t % a.tiles_x;
  if (bx == 0 || bx + 1 == a.tiles_x) hevi_row_strip<L, true, true>(job.maps, a, smem, bx, t / a.tiles_x);
  else hevi_row_strip<L, false, true>(job.maps, a, smem, bx, t / a.tiles_x);
}

// The boundary levels and the y ghosts the row kernel leaves out, once after
// the last substep.  blockIdx.z = 0: one thread per column writes levels 1,
// nk-1 and nk (vbcu.f90:120,134, vbcw.f90:285,317,471,481, vbcp.f90:126-160,
// level nk of u, v, p' carried over); blockIdx.z = 1..4: one field's y ghost
// rows, levels blockIdx.y + 2.
__global__ void __launch_bounds__(256) k_hevi_row_ends(const HeviRowArgs a) {
  const Grid g = a.g;
  const int ni = g.ni, nj = g.nj, nk = g.nk;
  const int i = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.z == 0) {
    for (int j = 2 + blockIdx.y; j <= nj - 1; j += gridDim.y) {
      const bool ins = i <= ni - 2 && j <= nj - 2;
      if (i <= ni - 1 && j <= nj - 2) {
        store_periodic(a.un, g, STAG_U, i, j, 1, a.un[g.at(i, j, 2)]);
        store_periodic(a.un, g, STAG_U, i, j, nk - 1, a.un[g.at(i, j, nk - 2)]);
        store_periodic(a.un, g, STAG_U, i, j, nk, __ldg(a.u + g.at(i, j, nk)));
      }
      if (i <= ni - 2) {
        store_periodic(a.vn, g, STAG_V, i, j, 1, a.vn[g.at(i, j, 2)]);
        store_periodic(a.vn, g, STAG_V, i, j, nk - 1, a.vn[g.at(i, j, nk - 2)]);
        store_periodic(a.vn, g, STAG_V, i, j, nk, __ldg(a.v + g.at(i, j, nk)));
      }
      if (!ins) continue;
      const float w3 = a.wn[g.at(i, j, 3)], wt = a.wn[g.at(i, j, nk - 2)];
      const float wc3 = a.sth ? w3 / a.jw3 : w3, wct = a.sth ? wt / a.jwt : wt;   // wc = w / jcb8w when stretched
      store_periodic(a.wn, g, STAG_S, i, j, 1, -a.jw3 * wc3 - 0.f);
      store_periodic(a.wn, g, STAG_S, i, j, nk - 1, 0.f);
      store_periodic(a.wn, g, STAG_S, i, j, nk, -a.jwt * wct - 0.f);
      const float p2 = a.pn[g.at(i, j, 2)];
      store_periodic(a.pn, g, STAG_S, i, j, 1, a.bbc == 2 ? 2.f * p2 - a.pn[g.at(i, j, 3)] : p2);
      store_periodic(a.pn, g, STAG_S, i, j, nk - 1, a.pn[g.at(i, j, nk - 2)]);
      store_periodic(a.pn, g, STAG_S, i, j, nk, __ldg(a.p + g.at(i, j, nk)));
    }
    return;
  }
  if (g.slaby) return;   // the neighbours' rows fill them (slab.h)
  const int f = blockIdx.z - 1;
  const bool us = f == 0, vs = f == 1;
  float* x = f == 0 ? a.un : f == 1 ? a.vn : f == 2 ? a.wn : a.pn;
  if (i > (us ? ni - 1 : ni - 2)) return;
  for (int k = 2 + blockIdx.y; k <= nk - 2; k += gridDim.y) {
    store_periodic(x, g, us ? STAG_U : vs ? STAG_V : STAG_S, i, nj - 2, k, x[g.at(i, nj - 2, k)]);
    const int jn = vs ? 3 : 2;
    if (jn != nj - 2) store_periodic(x, g, us ? STAG_U : vs ? STAG_V : STAG_S, i, jn, k, x[g.at(i, jn, k)]);
  }
}

int chunks(int nk, int L) { return (nk - 3 + L - 1) / L; }

template <int L>
int launch(const HeviRowMaps& m, const HeviRowArgs& a, cudaStream_t st) {
  const Grid& g = a.g;
  const int nC = chunks(g.nk, L);
  const size_t bytes = HrLayout<L>::bytes(nC);
  if (cudaFuncSetAttribute(k_hevi_row<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return CRESS_E_CUDA;
  const dim3 grid((unsigned)a.tiles_x, (unsigned)((g.nj - 3 + a.rows - 1) / a.rows));
  return launch_dependent(grid, 32 * nC, bytes, st, k_hevi_row<L>, m, a);
}

}  // namespace

bool hevi_row_supported(const Grid& g) {
  // a plane's bytes and the levels of a chunk are 32-bit offsets; the wrapped rows and columns are distinct
  return hevi_row_chunk(g.nk) && g.nk >= 8 && g.ni >= 8 && g.nj >= 8 && g.count() < (1LL << 31);
}

int hevi_row_tiles_x(const Grid& g) { return (g.ni - 3 + kHrCols - 1) / kHrCols; }

// Blocks of a column of nk levels an SM holds: 4096 registers (128 per
// thread) and a stage of shared memory per warp.  Two from 8 chunks down (nk = 19),
// five at the fewest; one for tall columns.
static int blocks_per_sm(int nk) {
  const int L = hevi_row_chunk(nk), nC = chunks(nk, L);
  const size_t bytes = L == 2 ? HrLayout<2>::bytes(nC) : L == 3 ? HrLayout<3>::bytes(nC)
                     : L == 4 ? HrLayout<4>::bytes(nC) : HrLayout<5>::bytes(nC);
  const int by_smem = (int)(228 * 1024 / (bytes + 1024 + sizeof(HeviRowArgs)));
  return std::max(1, std::min(kHrMaxWarps / nC, by_smem));
}

// Rows per strip: a block costs its rows plus about 1.3 for the row it
// recomputes and its start, and the blocks run in waves of what the SMs hold; the
// shortest total wins.  (Waves of one per SM whatever the height: 512 x 512 x 5
// 65 us per substep, this 25; the level march before it 42.)
int hevi_row_rows(const Grid* const* g, int n) {
  const int nsm = sm_count();
  std::vector<int> per(n);
  int best = 1, ny_max = 1;
  for (int m = 0; m < n; ++m) {
    ny_max = std::max(ny_max, g[m]->nj - 3);
    per[m] = blocks_per_sm(g[m]->nk);
  }
  double cost = 1e30;
  for (int r = 1; r <= ny_max; ++r) {
    double t = 0.0;   // SMs' worth of blocks
    for (int m = 0; m < n; ++m)
      t += (double)hevi_row_tiles_x(*g[m]) * ((g[m]->nj - 3 + r - 1) / r) / per[m];
    const double c = std::ceil(t / nsm - 1e-9) * (r + 1.3);
    if (c < cost - 1e-9) { cost = c; best = r; }
  }
  return best;
}

void hevi_row_table(const float* col, int nk, const float* rr, const double* aa, const double* cp, const HeviArgs& a,
                    std::vector<float>* lev, std::vector<double>* dbl) {
  const int L = hevi_row_chunk(nk), nC = chunks(nk, L), n = nC * L;
  auto C = [&](int f, int k) { return (double)col[(size_t)f * (nk + 1) + std::min(k, nk)]; };
  lev->assign((size_t)n * kHrVec * 4, 0.f);
  dbl->assign((size_t)n * 4 + (size_t)nC * 2 + 2 * kHrMaxWarps * kHrMaxWarps, 0.0);
  const bool sth = a.sthopt != 0, buy = a.buyopt == 1;
  const double dts = a.dts, dxiv = a.dxiv, dyiv = a.dyiv, dziv = a.dziv, wei = a.weicoe, wei1 = (double)(1.f - a.weicoe);
  std::vector<double> A(n, 0.0), B(n, 0.0), K(n, 0.0), CW(n + 1, 0.0);
  for (int m = 0; m < n; ++m) {
    const int k = 2 + m;
    if (k > nk - 2) break;
    const double ij = C(C_IJCB, k), jcb = C(C_JCB, k), rcsq = C(C_RCSQ, k), rst = C(C_RST, k);
    auto aw = [&](int kk) { return C(C_RST8W, kk) * (sth ? C(C_IJCB8W, kk) : 1.0) * dziv; };
    const double cv = a.divopt >= 1 ? (double)a.divcv * jcb : 0.0;
    const double ch = a.divopt == 2 ? (double)a.divch : a.divopt == 1 ? jcb * cv : 0.0;
    const double cw = dts * C(C_IRST8W, k);
    const double vals[2 * kHrVec] = {
        C(C_RST8U, k) * dxiv, C(C_RST8V, k) * dyiv,                       // 0: divergence, u and v
        aw(k + 1), jcb,                                                   // 1: w face above; jcb
        ch, cv,                                                           // 2: damping, horizontal and vertical
        dts * C(C_IRST8V, k), aw(k),                                      // 3: v step; w face below
        rcsq * C(C_JCB8V, k) * dyiv, dts * ij,                            // 4: v part of the p' tendency; p' step
        ij * (double)a.dtdzw, buy ? rst * C(C_IRCSQ, k) * (double)a.g05n : 0.0,         // 5: pgradiv; buoyancy of p'
        buy ? C(C_RBR, k) * (double)a.dtw * C(C_IRCSQ, k) * (double)a.g05n : 0.0, cw,   // 6: of the tendency; w step
        dts * C(C_IRST8U, k), rcsq * C(C_JCB8U, k) * dxiv,                // 7: u step; u part of the p' tendency
        wei1 * (double)a.g05 * rst, wei1 * rcsq * dziv,                   // 8: explicit w part: sum, difference
        dts * ij * wei * (double)a.g05 * rst, dts * ij * wei * rcsq * dziv};            // 9: implicit w part
    for (int v = 0; v < 2 * kHrVec; ++v)
      (*lev)[(size_t)m * kHrVec * 4 + 2 * v] = (*lev)[(size_t)m * kHrVec * 4 + 2 * v + 1] = (float)vals[v];
    CW[m] = (double)(float)cw;
    if (k >= 3) {
      A[m] = aa[k];
      B[m] = k == 3 ? 0.0 : -(double)rr[k] * aa[k];
      K[m] = cp[k];
    }
  }
  std::vector<double> Q(nC), H(nC);   // products of a chunk's factors: entry to entry, top to bottom
  for (int c = 0; c < nC; ++c) {
    double P = 1.0;
    H[c] = 1.0;
    for (int l = 0; l < L; ++l) {
      const int m = c * L + l;
      P = l == 0 ? 1.0 : P * B[m];
      H[c] *= -K[m];
      double* d = dbl->data() + 4 * (size_t)m;
      d[0] = A[m]; d[1] = B[m]; d[2] = K[m]; d[3] = P;
    }
    const int mn = (c + 1) * L;
    const double bn = mn < n ? B[mn] : 0.0, an = mn < n ? A[mn] * CW[mn] : 0.0;
    Q[c] = bn * P;
    double* d = dbl->data() + 4 * (size_t)n + 2 * (size_t)c;
    d[0] = bn; d[1] = an;
  }
  // chunk c's entry values from the others' hand-overs: from below, from above
  double* M = dbl->data() + 4 * (size_t)n + 2 * (size_t)nC;
  for (int c = 0; c < nC; ++c) {
    double f = 1.0;
    for (int q = c - 1; q >= 0; --q) { M[c * kHrMaxWarps + q] = f; f *= Q[q]; }
    f = 1.0;
    for (int q = c + 1; q < nC; ++q) { M[(kHrMaxWarps + c) * kHrMaxWarps + q] = f; f *= H[q]; }
  }
}

template <int L>
static int launch_batch(const HeviRowJob* jobs_d, int njobs, int nblocks, int nC, cudaStream_t st) {
  const size_t bytes = HrLayout<L>::bytes(nC);
  if (cudaFuncSetAttribute(k_hevi_row_batch<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return CRESS_E_CUDA;
  return launch_dependent(dim3(nblocks), 32 * nC, bytes, st, k_hevi_row_batch<L>, jobs_d, njobs);
}

int launch_hevi_row_batch(const HeviRowJob* jobs_d, int njobs, int nblocks, int nk, cudaStream_t st) {
  const int L = hevi_row_chunk(nk), nC = L ? chunks(nk, L) : 0;
  switch (L) {
    case 2: return launch_batch<2>(jobs_d, njobs, nblocks, nC, st);
    case 3: return launch_batch<3>(jobs_d, njobs, nblocks, nC, st);
    case 4: return launch_batch<4>(jobs_d, njobs, nblocks, nC, st);
    case 5: return launch_batch<5>(jobs_d, njobs, nblocks, nC, st);
  }
  return CRESS_E_UNSUPPORTED;
}

int launch_hevi_row_ends(const HeviRowArgs& a, cudaStream_t st) {
  const Grid& g = a.g;
  const dim3 grid((unsigned)((g.ni - 2 + 255) / 256), (unsigned)std::min(std::max(g.nj - 2, g.nk - 3), 65535), 5);
  k_hevi_row_ends<<<grid, 256, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : CRESS_E_CUDA;
}

int launch_hevi_row(const HeviRowMaps& m, const HeviRowArgs& a, cudaStream_t st) {
  switch (hevi_row_chunk(a.g.nk)) {
    case 2: return launch<2>(m, a, st);
    case 3: return launch<3>(m, a, st);
    case 4: return launch<4>(m, a, st);
    case 5: return launch<5>(m, a, st);
  }
  return CRESS_E_UNSUPPORTED;
}

}  // namespace cress
