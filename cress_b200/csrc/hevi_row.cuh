// HE-VI substep that marches rows (internal): interface of hevi_row.cu.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <vector>
#include "common.cuh"
#include "hevi.cuh"

namespace cress {

// Levels a warp of the row kernel carries (its chunk of the column) for a
// grid of nk levels: the fewest that keep the block at 16 warps.  0: the
// grid has more levels than the kernel's largest chunk covers.
inline int hevi_row_chunk(int nk) {
  const int n = nk - 3;   // levels 2..nk-2
  const int sizes[] = {2, 3, 4, 5};
  for (int L : sizes)
    if (n <= 16 * L) return L;
  return 0;
}

// Level table: kHrVec float4 per level k = 2, 3, ... (whole chunks, rows
// beyond nk-2 zero), every constant stored twice so that a 16-byte load
// yields two operand pairs of the packed FP32x2 arithmetic; then four
// doubles per level (a, b, cp, P), two per chunk (bn, an) and the two fold
// matrices (16 x 16).
constexpr int kHrVec = 10;
struct HeviRowTable {
  const float4* lev = nullptr;
  const double2* dbl = nullptr;
};

// Tensor maps (3-D, x = i, y = j, z = k-1): boxes of 64 columns, one row and
// a chunk's levels (w: one level more).
struct HeviRowMaps {
  CUtensorMap u, v, w, p, uf, vf, wf, pf;
};

struct HeviRowArgs {
  Grid g;
  const float *u, *v, *p;            // the old level (ends: the level the loop started from)
  float *un, *vn, *wn, *pn;          // the new level
  HeviRowTable tab;
  uint64_t dxiv2, dyiv2, dziv2;      // each float twice
  float jw3, jwt;                    // jcb8w at levels 3 and nk-2
  int sth, bbc;
  int wrap;                          // 1: the old level's y ghosts are not written, read their images
  int rows;                          // rows of a block's strip
  int tiles_x;
  int* err;                          // device error word (nonzero: a bounded wait gave up)
  uint32_t spin;                     // probes of each wait before it gives up
};

// Host form of the table for one dts: lev (kHrVec * 4 floats per level) and
// dbl (4 doubles per level, 2 per chunk, the folds).
void hevi_row_table(const float* col, int nk, const float* rr, const double* aa, const double* cp, const HeviArgs& a,
                    std::vector<float>* lev, std::vector<double>* dbl);
// One member's substep in an ensemble launch, in block order.
struct alignas(64) HeviRowJob {
  HeviRowMaps maps;
  HeviRowArgs args;
  int first_block;
};
// Rows of a block's strip when n grids share a launch, and a grid's tiles in x.
int hevi_row_rows(const Grid* const* g, int n);
int hevi_row_tiles_x(const Grid& g);
bool hevi_row_supported(const Grid& g);
// One substep: the new level's points of levels 2..nk-2 (w to nk-1) and their
// x ghosts; the boundary levels and the y ghosts are left to
// launch_hevi_row_ends.
int launch_hevi_row(const HeviRowMaps& m, const HeviRowArgs& a, cudaStream_t st);
// The same for njobs members with equal chunk lengths (jobs in device memory,
// nblocks blocks in all), the tallest of nk_max levels.
int launch_hevi_row_batch(const HeviRowJob* jobs_d, int njobs, int nblocks, int nk_max, cudaStream_t st);
// The boundary levels and y ghosts, once after the last substep of a loop
// (a.u, a.v, a.p: the level the loop started from).
int launch_hevi_row_ends(const HeviRowArgs& a, cudaStream_t st);

}  // namespace cress
