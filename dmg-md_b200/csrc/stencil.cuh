// stencil.cuh -- the candidates of one center from a cell grid, by one warp.
//
// Cells are at least half the search radius thick, so a 5x5x5 stencil covers
// it.  The stencil is taken as its 25 rows of cells along x (fewer on narrow
// grids): a row's cells are consecutive in the cell order, so its atoms are one
// contiguous run of the cell-ordered arrays, two where the row wraps around the
// box.  In an orthogonal box each row is trimmed to the cells that can hold a
// neighbour: a row whose y-z distance from the center exceeds the radius is
// dropped, and the x extent keeps the offsets whose distance along x fits in what
// is left (exact geometric distances to the cells; the caller widens the radius
// by 1e-5 relative so that no pair the float predicate accepts is ever cut).
// Lane r takes row r, a warp prefix sum of the runs flattens them into one range,
// and the warp sweeps it 32 candidates at a time.
#pragma once

#include "common.cuh"

namespace nepx {

struct CellGrid {
  int nc[3];      // cells per direction
  double w[3];    // their widths (orthogonal boxes)
  int base;       // first cell of this grid in the cell arrays
};

struct Stencil {
  int incl, cnt, st1, n1, st2;   // this lane's row: inclusive sum, atoms, runs
  int total;                     // candidates of the center

  // cell: the center's cell within the grid; (xi, yi, zi) its position; r2 the
  // squared trimming radius.
  __device__ __forceinline__ Stencil(const Box& b, const CellGrid& g, int cell, double xi,
                                     double yi, double zi, double r2, const int* cell_start,
                                     const int* cell_count, int lane)
  {
    const int nc0 = g.nc[0], nc1 = g.nc[1], nc2 = g.nc[2];
    const int span0 = (b.pbc[0] && nc0 >= 5) ? 5 : nc0;
    const int span1 = (b.pbc[1] && nc1 >= 5) ? 5 : nc1;
    const int span2 = (b.pbc[2] && nc2 >= 5) ? 5 : nc2;
    const int nrows = span1 * span2;   // at most 25
    const bool prune = b.ortho != 0;
    const int cx = cell % nc0, cy = (cell / nc0) % nc1, cz = cell / (nc0 * nc1);
    st1 = n1 = st2 = 0;
    int n2 = 0;
    if (lane < nrows) {
      const int q1 = lane % span1, q2 = lane / span1;
      // the center's position inside its cell, in cell widths (the fractional
      // coordinates that assigned the cells)
      auto frac = [&](int d, int c, int nc) {
        double sd = b.hinv[3 * d] * xi + b.hinv[3 * d + 1] * yi + b.hinv[3 * d + 2] * zi;
        sd -= floor(sd);
        return fmin(fmax(sd * nc - c, 0.0), 1.0);
      };
      // distance from the center to the cells k rows away along a direction
      auto gap = [](int k, double u, double w) {
        return k > 0 ? (k - u) * w : (k < 0 ? (u - k - 1) * w : 0.0);
      };
      double dyz2 = 0.0;
      double ux = 0.0;
      if (prune) {
        if (span1 == 5) {
          const double d = gap(q1 - 2, frac(1, cy, nc1), g.w[1]);
          dyz2 += d * d;
        }
        if (span2 == 5) {
          const double d = gap(q2 - 2, frac(2, cz, nc2), g.w[2]);
          dyz2 += d * d;
        }
        if (span0 == 5) ux = frac(0, cx, nc0);
      }
      if (dyz2 < r2) {
        int gy = span1 == 5 ? cy + q1 - 2 : q1;
        int gz = span2 == 5 ? cz + q2 - 2 : q2;
        if (gy < 0) gy += nc1; else if (gy >= nc1) gy -= nc1;
        if (gz < 0) gz += nc2; else if (gz >= nc2) gz -= nc2;
        const int row = g.base + (gz * nc1 + gy) * nc0;
        // atoms of the row's cells c0..c1 (consecutive)
        auto run = [&](int c0, int c1, int& st, int& n) {
          st = cell_start[row + c0];
          n = cell_start[row + c1] + cell_count[row + c1] - st;
        };
        if (span0 < 5) {
          run(0, nc0 - 1, st1, n1);
        } else {
          int klo = -2, khi = 2;
          if (prune) {
            const double rx2 = r2 - dyz2;
            auto within = [&](int k) {
              const double d = gap(k, ux, g.w[0]);
              return d * d < rx2;
            };
            klo = within(-1) ? (within(-2) ? -2 : -1) : 0;
            khi = within(1) ? (within(2) ? 2 : 1) : 0;
          }
          const int g0 = cx + klo, g1 = cx + khi;
          if (g0 < 0) {
            run(g0 + nc0, nc0 - 1, st1, n1);
            run(0, g1, st2, n2);
          } else if (g1 >= nc0) {
            run(g0, nc0 - 1, st1, n1);
            run(0, g1 - nc0, st2, n2);
          } else {
            run(g0, g1, st1, n1);
          }
        }
      }
    }
    cnt = n1 + n2;
    incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    total = __shfl_sync(0xffffffffu, incl, 31);
  }

  // Place of candidate k (whole warp; k < total where the result is used) in the
  // cell-ordered arrays: its row is the first lane whose inclusive sum exceeds k.
  __device__ __forceinline__ int place(int k) const
  {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const int v = __shfl_sync(0xffffffffu, incl, lo + step - 1);
      if (v <= k) lo += step;
    }
    const int r_incl = __shfl_sync(0xffffffffu, incl, lo);
    const int r_cnt = __shfl_sync(0xffffffffu, cnt, lo);
    const int r_st1 = __shfl_sync(0xffffffffu, st1, lo);
    const int r_n1 = __shfl_sync(0xffffffffu, n1, lo);
    const int r_st2 = __shfl_sync(0xffffffffu, st2, lo);
    const int local = k - (r_incl - r_cnt);
    return local < r_n1 ? r_st1 + local : r_st2 + (local - r_n1);
  }
};

}  // namespace nepx
