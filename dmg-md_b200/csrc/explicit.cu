// explicit.cu -- neighbour rows with explicit displacements: the small-box
// path and the batched path.
//
// Reference small-box path (src/gpumd_compat/nep_small_box.cuh:56-120,
// find_neighbor_list_small_box; nep.cu:1900-2000, compute_small_box): when a
// periodic direction is thinner than 2.5 (rc + 1) every center scans every
// atom of its system and every image of the expanded box, keeping the pairs
// inside the typewise radial / angular cutoffs together with the float
// displacement r12 of that image.  Rows follow (j ascending, then images
// ia, ib, ic) and are rebuilt at every force call.
//
// Here one warp owns a center and its lanes take consecutive candidates
// (j, image) in the reference's order, compacted by ballot (ImageWalk).  The same
// kernel serves any number of structures packed into one atom range (the batched
// path): a center finds its structure among the structure offsets.  Structures
// that are not small use the large-box arithmetic (double difference rounded
// to float, float minimum image, reference nep.cu:503-561); their candidates
// come from a cell grid of their own (stencil.cuh; cells at least rc/2 thick, a
// counting sort per batch scanned per structure), and each row is sorted
// (warp-shuffle bitonic network up to 64 entries, shared memory above), which
// yields the large-box path's typewise rows exactly.  Those structures' rows
// hold each neighbour once, so a batch marks their centers (large[]) for the
// directed-f12 scheme of the large-box path.
//
// Row entry: float4 (x12, y12, z12, bits of j | type(j) << 28), row-major
// [center][slot]; radial and angular rows are separate.
#include <algorithm>
#include <climits>
#include <cmath>
#include <string>

#include "engine.h"
#include "stencil.cuh"
#include "xbox.h"

namespace nepx {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// The first kernel of an explicit-row evaluation: the site records, and for a
// single system its StructInfo -- from the host when the call brings the box
// (si_mode 2: host_si, whose box also goes to the device copy; the FP64 chain on
// the device takes 5 us), or from the device box (1).
__global__ void k_xr_begin(int N, const double* __restrict__ pos, const int* __restrict__ type,
                           Site* __restrict__ sites, NeighborState* st, int si_mode,
                           const StructInfo host_si, Box* box, double rc, StructInfo* si,
                           int* soff)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N)
    sites[i] = Site{pos[i], pos[N + i], pos[2 * N + i], static_cast<long long>(type[i])};
  if (i != 0) return;
  st->call_nn[0] = 0;   // the row maxima of this evaluation start here
  st->call_nn[1] = 0;
  if (si_mode == 0) return;
  StructInfo s;
  if (si_mode == 2) {
    s = host_si;
    *box = host_si.box;
  } else if (expanded_box(*box, rc, s)) {
    st->box_error = 1;
  }
  s.off = 0;
  s.n = N;
  *si = s;
  soff[0] = 0;
  soff[1] = N;
}

// What the small-box arithmetic reads of a structure, in registers (read through
// the structure's pointer, every candidate loaded it again after the row writes).
struct ImageBox {
  float fh[9], e[18];
  int pbc[3];
  __device__ __forceinline__ explicit ImageBox(const StructInfo& s)
  {
#pragma unroll
    for (int k = 0; k < 9; ++k) fh[k] = s.box.fh[k];
#pragma unroll
    for (int k = 0; k < 18; ++k) e[k] = s.eh[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) pbc[k] = s.box.pbc[k];
  }
};

// Displacement from a center (float position) to atom j (double position) at
// image (ia, ib, ic) of the expanded box: the reference's small-box
// arithmetic (nep_small_box.cuh:134-143) with its minimum image in the expanded
// box (:39-54).  Shared by the row builder and the Verlet-candidate filter, so
// both produce the same float values.
__device__ __forceinline__ void small_box_delta(const ImageBox& s, float x1, float y1, float z1,
                                                double xj, double yj, double zj, int ia, int ib,
                                                int ic, float& x12, float& y12, float& z12)
{
  const float* fh = s.fh;
  const float* e = s.e;
  const float d0 = fh[0] * ia + fh[1] * ib + fh[2] * ic;
  const float d1 = fh[3] * ia + fh[4] * ib + fh[5] * ic;
  const float d2 = fh[6] * ia + fh[7] * ib + fh[8] * ic;
  x12 = xj + d0 - x1;
  y12 = yj + d1 - y1;
  z12 = zj + d2 - z1;
  float sx12 = e[9] * x12 + e[10] * y12 + e[11] * z12;
  float sy12 = e[12] * x12 + e[13] * y12 + e[14] * z12;
  float sz12 = e[15] * x12 + e[16] * y12 + e[17] * z12;
  if (s.pbc[0] == 1) sx12 -= nearbyintf(sx12);
  if (s.pbc[1] == 1) sy12 -= nearbyintf(sy12);
  if (s.pbc[2] == 1) sz12 -= nearbyintf(sz12);
  x12 = e[0] * sx12 + e[1] * sy12 + e[2] * sz12;
  y12 = e[3] * sx12 + e[4] * sy12 + e[5] * sz12;
  z12 = e[6] * sx12 + e[7] * sy12 + e[8] * sz12;
}

// The structure of center i, the last s with soff[s] <= i, by one warp: 32
// probes per round (two rounds up to 1,024 structures).
__device__ __forceinline__ int warp_find_struct(const int* __restrict__ soff, int S, int i,
                                                int lane)
{
  int lo = 0, n = S;
  while (n > 1) {
    const int step = (n + 31) >> 5;
    const int k = lane * step;
    const unsigned m = __ballot_sync(kFull, k < n && __ldg(soff + lo + k) <= i);
    const int q = 31 - __clz(m);   // lane 0 always holds
    lo += q * step;
    n = min(step, n - q * step);
  }
  return lo;
}

// The candidates of a small-box center, (j, image) with j ascending and then the
// images, taken 32 at a time: lane l starts at candidate l and steps by 32 in
// the mixed radix (j, ia, ib, ic), so the hits of a ballot are in row order and
// one sweep suffices (a lane per j counted its images' hits, scanned and swept
// them again to write).
struct ImageWalk {
  int j, ia, ib, ic;          // this lane's candidate (j local to the structure)
  int dj, da, db, dc;         // 32 candidates further
  int nb, nc, na;
  __device__ __forceinline__ ImageWalk(const StructInfo& s, int lane)
  {
    na = s.ncell[0];
    nb = s.ncell[1];
    nc = s.ncell[2];
    auto split = [&](int c, int& q, int& a, int& b, int& d) {
      d = c % nc;
      c /= nc;
      b = c % nb;
      c /= nb;
      a = c % na;
      q = c / na;
    };
    split(lane, j, ia, ib, ic);
    split(32, dj, da, db, dc);
  }
  __device__ __forceinline__ void next()
  {
    ic += dc;
    ib += db;
    ia += da;
    j += dj;
    if (ic >= nc) {
      ic -= nc;
      ++ib;
    }
    if (ib >= nb) {
      ib -= nb;
      ++ia;
    }
    if (ia >= na) {
      ia -= na;
      ++j;
    }
  }
};

__device__ __forceinline__ float4 row_entry(float x, float y, float z, int j, int t)
{
  return make_float4(x, y, z, __int_as_float(j | (t << kRowTypeShift)));
}

// The angular neighbours of large structures by index, as the Verlet path's rows
// hold them, with the length and every eighth in a row of heads: the gather's
// reverse slots.
struct RowHeads {
  int* nl;
  int* heads;
  int st_a, st_h;
  __device__ __forceinline__ void put(int i, int at, int j) const
  {
    nl[static_cast<size_t>(i) * st_a + at] = j;
    if (at % 8 == 0) heads[static_cast<size_t>(i) * st_h + 1 + at / 8] = j;
  }
  __device__ __forceinline__ void length(int i, int n) const
  {
    heads[static_cast<size_t>(i) * st_h] = n;
  }
};

// Rows of the centers of small structures (SMALL: images), or of the others. One
// kernel for both took 97 registers, two CTAs per SM, and issued on 46 % of its
// cycles; apart, and held to three and four CTAs, they took the batch call of 188
// structures from 2.54 to 2.21 ms.
template <bool SMALL>
__global__ void __launch_bounds__(256, SMALL ? 3 : 4)
k_rows_explicit(const ModelParams p, int total, const StructInfo* __restrict__ si,
                const int* __restrict__ soff, int S, const double* __restrict__ pos,
                const int* __restrict__ type, int* __restrict__ nn_r, float4* __restrict__ er,
                int mn_r, int* __restrict__ nn_a, float4* __restrict__ ea, int mn_a,
                const RowHeads rh, const int* __restrict__ cell_count, const int* __restrict__ cell_start,
                const int* __restrict__ cell_atoms, const int* __restrict__ cell_of,
                const Site* __restrict__ cell_sites, float rc_max, int p2r,
                const Site* __restrict__ sites, unsigned char* __restrict__ large, int mark_large,
                const BatchVerlet bv, NeighborState* st)
{
  extern __shared__ int s_rows[];   // per warp: p2r row slots + a counter
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  for (int i = blockIdx.x * wpb + (threadIdx.x >> 5); i < total; i += gridDim.x * wpb) {
    const int lo = warp_find_struct(soff, S, i, lane);
    const StructInfo& s = si[lo];
    if ((s.small != 0) != SMALL) continue;
    const int off = s.off, n = s.n;
    const int t1 = type[i];
    const float rr1 = p.rc_r[t1], ra1 = p.rc_a[t1];
    // a structure that keeps Verlet candidates: (re)build them here when it is
    // new or has moved more than skin / 2 since the build; its rows come from
    // them in k_rows_verlet
    const int sf = bv.sflag ? bv.sflag[lo] : 0;
    const bool keep = (sf & 2) != 0;
    if (keep && !(sf & 4) && bv.dmax2[lo] <= bv.half_skin2) continue;
    auto cand_cut = [&](int tj) {
      return fmaxf((rr1 + p.rc_r[tj]) * 0.5f, (ra1 + p.rc_a[tj]) * 0.5f) + bv.skin;
    };
    float4* rrow = er + static_cast<size_t>(i) * mn_r;
    float4* arow = ea + static_cast<size_t>(i) * mn_a;
    int cr = 0, ca = 0;
    if constexpr (!SMALL) {
      const double xi = pos[i], yi = pos[total + i], zi = pos[2 * total + i];
      const MinImage mic(s.box);
      int* buf = s_rows + (threadIdx.x >> 5) * (p2r + 1);
      int found = 0;
      auto consider = [&](bool valid, int j, const double2& sa, const double2& sc) {
        bool hit = false;
        if (valid) {
          float x12, y12, z12;
          int tj;
          site_delta(mic, sa, sc, xi, yi, zi, x12, y12, z12, tj);
          const float d12_square = x12 * x12 + y12 * y12 + z12 * z12;
          const float rcut = keep ? cand_cut(tj) : (rr1 + p.rc_r[tj]) * 0.5f;
          hit = j != i && d12_square < rcut * rcut;
        }
        const unsigned m = __ballot_sync(kFull, hit);
        if (hit) {
          const int slot = found + __popc(m & below);
          if (slot < p2r) buf[slot] = j;
        }
        found += __popc(m);
      };
      if (s.nc[0] > 0) {
        // no pair cutoff of this center is above (its own + the largest) / 2, nor a
        // candidate cutoff above the largest cutoff plus the skin
        const double rmax = (keep ? static_cast<double>(rc_max) + bv.skin
                                  : static_cast<double>(rr1 + rc_max) * 0.5) * (1.0 + 1e-5) + 1e-5;
        const CellGrid grid{{s.nc[0], s.nc[1], s.nc[2]},
                            {s.cell_w[0], s.cell_w[1], s.cell_w[2]}, s.cell_base};
        const Stencil cand(s.box, grid, cell_of[i] - s.cell_base, xi, yi, zi, rmax * rmax, cell_start,
                           cell_count, lane);
        for (int base = 0; base < cand.total; base += 32) {
          const int at = cand.place(base + lane);
          const bool valid = base + lane < cand.total;
          double2 sa = make_double2(0.0, 0.0), sc = sa;
          int j = 0;
          if (valid) {
            j = cell_atoms[at];
            site_load(cell_sites, at, sa, sc);
          }
          consider(valid, j, sa, sc);
        }
      } else {
        for (int base = 0; base < n; base += 32) {
          const int j = off + base + lane;
          const bool valid = base + lane < n;
          double2 sa = make_double2(0.0, 0.0), sc = sa;
          if (valid) site_load(sites, j, sa, sc);
          consider(valid, j, sa, sc);
        }
      }
      __syncwarp();
      const int used = min(found, p2r);
      int p2 = 1;
      while (p2 < used) p2 <<= 1;
      if (p2 <= 64) {
        // bitonic sort in registers: element e = lane in a, e = lane + 32 in
        // c; partners e ^ jj exchange by shuffle (jj < 32) or inside the lane
        // (jj = 32); e keeps the smaller value when (e < partner) matches the
        // ascending direction (e & k) == 0 of its block
        int a = lane < used ? buf[lane] : INT_MAX;
        int c = lane + 32 < used ? buf[lane + 32] : INT_MAX;
        const bool two = p2 > 32;   // warp-uniform
        for (int k = 2; k <= p2; k <<= 1) {
          for (int jj = k >> 1; jj > 0; jj >>= 1) {
            if (jj == 32) {
              const int lo_v = min(a, c);
              c = max(a, c);
              a = lo_v;
            } else {
              const bool lower = (lane & jj) == 0;
              const int pa = __shfl_xor_sync(kFull, a, jj);
              a = (lower == ((lane & k) == 0)) ? min(a, pa) : max(a, pa);
              if (two) {
                const int pc = __shfl_xor_sync(kFull, c, jj);
                c = (lower == (((lane + 32) & k) == 0)) ? min(c, pc) : max(c, pc);
              }
            }
          }
        }
        __syncwarp();   // every lane has read buf before it is overwritten
        if (lane < used) buf[lane] = a;
        if (lane + 32 < used) buf[lane + 32] = c;
        __syncwarp();
      } else {
        for (int k = used + lane; k < p2; k += 32) buf[k] = INT_MAX;
        __syncwarp();
        for (int k = 2; k <= p2; k <<= 1) {   // bitonic sort, one pair per lane and pass
          for (int jj = k >> 1; jj > 0; jj >>= 1) {
            for (int q = lane; q < (p2 >> 1); q += 32) {
              const int t = ((q & ~(jj - 1)) << 1) | (q & (jj - 1));
              const int u = t | jj;
              const int a = buf[t], c = buf[u];
              if ((a > c) == ((t & k) == 0)) {
                buf[t] = c;
                buf[u] = a;
              }
            }
            __syncwarp();
          }
        }
      }
      if (keep) {
        // ascending candidates, structure-local
        int* vr = bv.vrow + static_cast<size_t>(i) * bv.mn;
        for (int k = lane; k < used && k < bv.mn; k += 32) vr[k] = buf[k] - off;
        if (lane == 0) {
          bv.vcnt[i] = min(found, bv.mn);
          if (found > bv.mn || found > p2r) atomicOr(&st->overflow, 1);
          bv.x0[i] = xi;
          bv.x0[total + i] = yi;
          bv.x0[2 * total + i] = zi;
          atomicAdd(&st->xr_builds, 1u);
        }
        __syncwarp();   // the buffer is reused by this warp's next center
        continue;
      }
      // ascending radial row; the angular row is its subset inside the angular cutoff
      for (int k0 = 0; k0 < used; k0 += 32) {
        const int k = k0 + lane;
        bool in_a = false;
        float4 entry = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k < used) {
          const int j = buf[k];
          float x12, y12, z12;
          int t2;
          double2 sa, sc;
          site_load(sites, j, sa, sc);
          site_delta(mic, sa, sc, xi, yi, zi, x12, y12, z12, t2);
          const float d12_square = x12 * x12 + y12 * y12 + z12 * z12;
          const float rc_angular = (ra1 + p.rc_a[t2]) * 0.5f;
          in_a = d12_square < rc_angular * rc_angular;
          entry = row_entry(x12, y12, z12, j, t2);
          if (k < mn_r) rrow[k] = entry;
        }
        const unsigned ma = __ballot_sync(kFull, in_a);
        if (in_a) {
          const int at = ca + __popc(ma & below);
          if (at < mn_a) {
            arow[at] = entry;
            rh.put(i, at, __float_as_int(entry.w) & kRowIndexMask);
          }
        }
        ca += __popc(ma);
      }
      cr = found;
      __syncwarp();   // the buffer is reused by this warp's next center
    } else if (keep) {
      // candidates (j, image) within the cutoff plus the skin, in row order
      const float x1 = pos[i], y1 = pos[total + i], z1 = pos[2 * total + i];
      int* vr = bv.vrow + static_cast<size_t>(i) * bv.mn;
      const long long total_c =
        static_cast<long long>(n) * (s.ncell[0] * s.ncell[1] * s.ncell[2]);
      ImageWalk w(s, lane);
      const ImageBox ib(s);
      int cv = 0;
#pragma unroll 2
      for (long long base = 0; base < total_c; base += 32) {
        bool hit = false;
        unsigned code = 0u;
        if (w.j < n) {
          const int j = off + w.j;
          const float rcut = cand_cut(type[j]);
          float x12, y12, z12;
          double2 sa, sc;
          site_load(sites, j, sa, sc);
          small_box_delta(ib, x1, y1, z1, sa.x, sa.y, sc.x, w.ia, w.ib, w.ic, x12, y12, z12);
          const bool self = j == i && w.ia == 0 && w.ib == 0 && w.ic == 0;
          hit = !self && x12 * x12 + y12 * y12 + z12 * z12 < rcut * rcut;
          code = static_cast<unsigned>(w.j) | (static_cast<unsigned>(w.ia) << kCandIndexBits) |
                 (static_cast<unsigned>(w.ib) << (kCandIndexBits + 4)) |
                 (static_cast<unsigned>(w.ic) << (kCandIndexBits + 8));
        }
        const unsigned m = __ballot_sync(kFull, hit);
        const int at = cv + __popc(m & below);
        if (hit && at < bv.mn) vr[at] = static_cast<int>(code);
        cv += __popc(m);
        w.next();
      }
      if (lane == 0) {
        bv.vcnt[i] = min(cv, bv.mn);
        if (cv > bv.mn) atomicOr(&st->overflow, 1);
        bv.x0[i] = pos[i];
        bv.x0[total + i] = pos[total + i];
        bv.x0[2 * total + i] = pos[2 * total + i];
        atomicAdd(&st->xr_builds, 1u);
      }
      continue;
    } else {
      // the small-box arithmetic: float center, double image position
      const float x1 = pos[i], y1 = pos[total + i], z1 = pos[2 * total + i];
      const long long total_c =
        static_cast<long long>(n) * (s.ncell[0] * s.ncell[1] * s.ncell[2]);
      ImageWalk w(s, lane);
      const ImageBox ib(s);
#pragma unroll 2
      for (long long base = 0; base < total_c; base += 32) {
        bool in_r = false, in_a = false;
        float4 entry = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (w.j < n) {
          const int j = off + w.j;
          const int t2 = type[j];
          const float rc_radial = (rr1 + p.rc_r[t2]) * 0.5f;
          const float rc_angular = (ra1 + p.rc_a[t2]) * 0.5f;
          float x12, y12, z12;
          double2 sa, sc;
          site_load(sites, j, sa, sc);
          small_box_delta(ib, x1, y1, z1, sa.x, sa.y, sc.x, w.ia, w.ib, w.ic, x12, y12, z12);
          const float d12_square = x12 * x12 + y12 * y12 + z12 * z12;
          const bool self = j == i && w.ia == 0 && w.ib == 0 && w.ic == 0;
          in_r = !self && d12_square < rc_radial * rc_radial;
          in_a = !self && d12_square < rc_angular * rc_angular;
          entry = row_entry(x12, y12, z12, j, t2);
        }
        const unsigned mr = __ballot_sync(kFull, in_r);
        const unsigned ma = __ballot_sync(kFull, in_a);
        const int at_r = cr + __popc(mr & below), at_a = ca + __popc(ma & below);
        if (in_r && at_r < mn_r) rrow[at_r] = entry;
        if (in_a && at_a < mn_a) arow[at_a] = entry;
        cr += __popc(mr);
        ca += __popc(ma);
        w.next();
      }
    }
    if (lane == 0) {
      nn_r[i] = min(cr, mn_r);
      nn_a[i] = min(ca, mn_a);
      if constexpr (!SMALL) rh.length(i, min(ca, mn_a));
      large[i] = mark_large && !SMALL ? 1 : 0;
      if (cr > mn_r) atomicOr(&st->overflow, 2);
      if (ca > mn_a) atomicOr(&st->overflow, 4);
      atomicMax(&st->max_nn[1], cr);
      atomicMax(&st->max_nn[2], ca);
      atomicMax(&st->call_nn[0], cr);
      atomicMax(&st->call_nn[1], ca);
    }
  }
}

// Rows of the centers whose structure keeps Verlet candidates: one warp per
// center filters its candidates (in row order) with the predicates and the
// arithmetic of k_rows_explicit, so the rows equal a fresh build's bit for
// bit while no atom of the structure has moved more than skin / 2 since the
// candidates were built.  Radial and angular rows are written in order by
// warp ballot + popcount.
__global__ void __launch_bounds__(256, 3)
k_rows_verlet(const ModelParams p, int total, const StructInfo* __restrict__ si,
              const int* __restrict__ soff, int S, const double* __restrict__ pos,
              const int* __restrict__ type, int* __restrict__ nn_r, float4* __restrict__ er,
              int mn_r, int* __restrict__ nn_a, float4* __restrict__ ea, int mn_a,
              const RowHeads rh, const Site* __restrict__ sites, unsigned char* __restrict__ large,
              const BatchVerlet bv, NeighborState* st)
{
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  for (int i = blockIdx.x * wpb + (threadIdx.x >> 5); i < total; i += gridDim.x * wpb) {
    const int lo = warp_find_struct(soff, S, i, lane);
    if (!(bv.sflag[lo] & 2)) continue;
    const StructInfo& s = si[lo];
    const int off = s.off;
    const int t1 = type[i];
    const float rr1 = p.rc_r[t1], ra1 = p.rc_a[t1];
    float4* rrow = er + static_cast<size_t>(i) * mn_r;
    float4* arow = ea + static_cast<size_t>(i) * mn_a;
    const int* vr = bv.vrow + static_cast<size_t>(i) * bv.mn;
    const int nv = bv.vcnt[i];
    int cr = 0, ca = 0;
    const double xi = pos[i], yi = pos[total + i], zi = pos[2 * total + i];
    const float x1 = static_cast<float>(xi), y1 = static_cast<float>(yi),
                z1 = static_cast<float>(zi);
    const MinImage mic(s.box);
    const ImageBox ib(s);
    for (int k0 = 0; k0 < nv; k0 += 32) {
      const int k = k0 + lane;
      bool in_r = false, in_a = false;
      float4 entry = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (k < nv) {
        const unsigned code = static_cast<unsigned>(vr[k]);
        int j, t2;
        float x12, y12, z12;
        if (!s.small) {
          j = off + static_cast<int>(code);
          double2 sa, sc;
          site_load(sites, j, sa, sc);
          site_delta(mic, sa, sc, xi, yi, zi, x12, y12, z12, t2);
        } else {
          j = off + static_cast<int>(code & ((1u << kCandIndexBits) - 1u));
          const int ia = static_cast<int>((code >> kCandIndexBits) & 15u);
          const int jb = static_cast<int>((code >> (kCandIndexBits + 4)) & 15u);
          const int ic = static_cast<int>(code >> (kCandIndexBits + 8));
          t2 = type[j];
          small_box_delta(ib, x1, y1, z1, pos[j], pos[total + j], pos[2 * total + j], ia, jb, ic,
                          x12, y12, z12);
        }
        const float d12_square = x12 * x12 + y12 * y12 + z12 * z12;
        const float rc_radial = (rr1 + p.rc_r[t2]) * 0.5f;
        const float rc_angular = (ra1 + p.rc_a[t2]) * 0.5f;
        in_r = d12_square < rc_radial * rc_radial;
        // large structures: the angular row is the radial row's subset (as
        // k_rows_explicit builds it); small boxes test both cutoffs apart
        in_a = (s.small || in_r) && d12_square < rc_angular * rc_angular;
        entry = row_entry(x12, y12, z12, j, t2);
      }
      const unsigned mr = __ballot_sync(kFull, in_r);
      const unsigned ma = __ballot_sync(kFull, in_a);
      if (in_r) {
        const int at = cr + __popc(mr & below);
        if (at < mn_r) rrow[at] = entry;
      }
      if (in_a) {
        const int at = ca + __popc(ma & below);
        if (at < mn_a) {
          arow[at] = entry;
          if (!s.small) rh.put(i, at, __float_as_int(entry.w) & kRowIndexMask);
        }
      }
      cr += __popc(mr);
      ca += __popc(ma);
    }
    if (lane == 0) {
      nn_r[i] = min(cr, mn_r);
      nn_a[i] = min(ca, mn_a);
      if (!s.small) rh.length(i, min(ca, mn_a));
      large[i] = s.small ? 0 : 1;
      if (cr > mn_r) atomicOr(&st->overflow, 2);
      if (ca > mn_a) atomicOr(&st->overflow, 4);
      atomicMax(&st->max_nn[1], cr);
      atomicMax(&st->max_nn[2], ca);
      atomicMax(&st->call_nn[0], cr);
      atomicMax(&st->call_nn[1], ca);
    }
  }
}

// Cell of every atom of a large structure (fractional coordinates, wrapped
// where periodic, one cell where not), counted per cell.
__global__ void k_xcell_assign(int total, const StructInfo* __restrict__ si,
                               const int* __restrict__ soff, int S, const double* __restrict__ pos,
                               int* cell_count, int* cell_of)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  int lo = 0, hi = S - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (soff[mid] <= i) lo = mid; else hi = mid - 1;
  }
  const StructInfo& s = si[lo];
  if (s.small || s.nc[0] == 0) {
    cell_of[i] = -1;
    return;
  }
  const double r[3] = {pos[i], pos[total + i], pos[2 * total + i]};
  int c[3];
  for (int d = 0; d < 3; ++d) {
    double f = s.box.hinv[3 * d] * r[0] + s.box.hinv[3 * d + 1] * r[1] + s.box.hinv[3 * d + 2] * r[2];
    f -= floor(f);
    int k = static_cast<int>(f * s.nc[d]);
    c[d] = k < 0 ? 0 : (k >= s.nc[d] ? s.nc[d] - 1 : k);
  }
  const int cell = s.cell_base + (c[2] * s.nc[1] + c[1]) * s.nc[0] + c[0];
  cell_of[i] = cell;
  atomicAdd(cell_count + cell, 1);
}

// Exclusive scan of the cell counts, one block per structure: a structure's
// cells are contiguous and its atoms fill [off, off + n) of cell_atoms, so
// its cells start at off plus the scan of its own counts (coalesced chunks
// of blockDim.x cells with a running carry).  Counts reset as fill cursors.
__global__ void k_xcell_scan(const StructInfo* __restrict__ si, int* cell_count, int* cell_start)
{
  __shared__ int warp_sum[32];
  __shared__ int carry_s;
  const StructInfo& s = si[blockIdx.x];
  if (s.nc[0] == 0) return;   // block-uniform: the structure scans all its atoms
  const int ncs = s.nc[0] * s.nc[1] * s.nc[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int carry = s.off;
  for (int c0 = 0; c0 < ncs; c0 += blockDim.x) {
    const int c = c0 + threadIdx.x;
    const int v = c < ncs ? cell_count[s.cell_base + c] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nw ? warp_sum[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFull, w, o);
        if (lane >= o) w += u;
      }
      if (lane < nw) warp_sum[lane] = w;   // inclusive over warps
      if (lane == 31) carry_s = w;         // chunk total
    }
    __syncthreads();
    const int before = (warp > 0 ? warp_sum[warp - 1] : 0) + incl - v;
    if (c < ncs) {
      cell_start[s.cell_base + c] = carry + before;
      cell_count[s.cell_base + c] = 0;
    }
    carry += carry_s;
    __syncthreads();   // warp_sum and carry_s are rewritten by the next chunk
  }
}

// The atoms (index and site record) into their cells.
__global__ void k_xcell_fill(int total, const int* __restrict__ cell_of, int* cell_count,
                             const int* __restrict__ cell_start, const Site* __restrict__ sites,
                             int* cell_atoms, Site* cell_sites)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int c = cell_of[i];
  if (c < 0) return;
  const int at = cell_start[c] + atomicAdd(cell_count + c, 1);
  cell_atoms[at] = i;
  cell_sites[at] = sites[i];
}

__global__ void k_row_indices(int n, const int* __restrict__ cnt, const float4* __restrict__ rows,
                              int src_mn, int* nn, int* nl, int mn)
{
  const int i = blockIdx.x;
  if (i >= n) return;
  const int c = cnt[i];
  if (threadIdx.x == 0) nn[i] = c;
  for (int k = threadIdx.x; k < c; k += blockDim.x)
    nl[static_cast<size_t>(i) * mn + k] =
      __float_as_int(rows[static_cast<size_t>(i) * src_mn + k].w) & kRowIndexMask;
}

template <typename T>
cudaError_t dalloc(T*& ptr, size_t count)
{
  return cudaMalloc(reinterpret_cast<void**>(&ptr), std::max<size_t>(count, 1) * sizeof(T));
}

}  // namespace

int structure_cells(const Engine& e, const StructInfo& s, int* nc_out)
{
  if (s.small) return 0;
  // cells at least half the candidate radius: the cutoff, plus the skin for
  // a structure that keeps Verlet candidates
  const double rc = s.keep ? e.model.rc_max + e.skin : e.model.rc_radial_max;
  int nc[3], cells = 1;
  for (int d = 0; d < 3; ++d) {
    const double* r = s.box.hinv + 3 * d;
    const double thick = 1.0 / std::sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    nc[d] = s.box.pbc[d] ? std::max(1, static_cast<int>(thick / (0.5 * rc))) : 1;
    cells *= nc[d];
  }
  // a 5x5x5 stencil of cells at least rc/2 wide covers the cutoff; grids of
  // fewer than 125 cells scan all the structure's atoms instead
  if (cells < 125) return 0;
  if (nc_out)
    for (int d = 0; d < 3; ++d) nc_out[d] = nc[d];
  return cells;
}

int assign_cells(Engine& e, StructInfo* si, int n)
{
  int used = 0;
  e.xr.kinds = 0;
  for (int k = 0; k < n; ++k) {
    StructInfo& s = si[k];
    e.xr.kinds |= s.small ? kSmallRows : kLargeRows;
    s.nc[0] = s.nc[1] = s.nc[2] = 0;
    s.cell_base = 0;
    int nc[3];
    const int cells = structure_cells(e, s, nc);
    if (cells == 0 || used + cells > e.xr.cell_cap) continue;
    for (int d = 0; d < 3; ++d) {
      s.nc[d] = nc[d];
      s.cell_w[d] = s.box.h[4 * d] / nc[d];
    }
    s.cell_base = used;
    used += cells;
  }
  return used;
}

int box_kind(const Engine& e, const Box& b)
{
  StructInfo s;
  if (expanded_box(b, e.model.rc_radial_max, s)) return -1;
  return s.small;
}

std::string engine_enable_xr(Engine& e, int max_struct)
{
  ExplicitRows& x = e.xr;
  if (x.er && x.max_struct >= max_struct) return "";
  const size_t N = e.capacity;
  if (N > static_cast<size_t>(kRowIndexMask))
    return "explicit neighbour rows address at most 2^28 atoms";
  if (!x.er) {
    x.cell_cap = static_cast<int>(std::max<size_t>(N, 4096));
    bool ok = dalloc(x.er, N * e.nbr.mn_r) == cudaSuccess;
    ok &= dalloc(x.ea, N * e.nbr.mn_a) == cudaSuccess;
    ok &= dalloc(x.cell_count, x.cell_cap) == cudaSuccess;
    ok &= dalloc(x.cell_start, x.cell_cap) == cudaSuccess;
    ok &= dalloc(x.cell_atoms, N) == cudaSuccess;
    ok &= dalloc(x.cell_of, N) == cudaSuccess;
    ok &= dalloc(x.large, N) == cudaSuccess;
    if (!ok) return "cudaMalloc failed (explicit neighbour rows)";
  }
  if (x.max_struct < max_struct) {
    if (x.d_si) cudaFree(x.d_si);
    if (x.d_soff) cudaFree(x.d_soff);
    x.d_si = nullptr;
    x.d_soff = nullptr;
    bool ok = dalloc(x.d_si, max_struct) == cudaSuccess;
    ok &= dalloc(x.d_soff, max_struct + 1) == cudaSuccess;
    if (!ok) return "cudaMalloc failed (structure table)";
    x.max_struct = max_struct;
  }
  return "";
}

void launch_explicit_rows(Engine& e, int N, const double* pos, const int* type,
                          cudaStream_t stream)
{
  ExplicitRows& x = e.xr;
  const int threads = 256;
  const int si_mode = !x.from_box ? 0 : e.staged_box ? 2 : 1;
  StructInfo host_si{};
  if (si_mode == 2) expanded_box(*e.staged_box, e.model.rc_radial_max, host_si);
  k_xr_begin<<<(N + threads - 1) / threads, threads, 0, stream>>>(
    N, pos, type, e.scratch.sites, e.d_nstate, si_mode, host_si, e.d_box, e.model.rc_radial_max,
    x.d_si, x.d_soff);
  if (x.from_box) {
    x.n_struct = 1;
    // the box's kind where the host knows it (MD under a barostat does not)
    x.kinds = si_mode != 2 ? kSmallRows | kLargeRows : host_si.small ? kSmallRows : kLargeRows;
  }
  if (!x.from_box && x.n_cells > 0) {
    cudaMemsetAsync(x.cell_count, 0, sizeof(int) * x.n_cells, stream);
    k_xcell_assign<<<(N + threads - 1) / threads, threads, 0, stream>>>(
      N, x.d_si, x.d_soff, x.n_struct, pos, x.cell_count, x.cell_of);
    k_xcell_scan<<<x.n_struct, 1024, 0, stream>>>(x.d_si, x.cell_count, x.cell_start);
    k_xcell_fill<<<(N + threads - 1) / threads, threads, 0, stream>>>(
      N, x.cell_of, x.cell_count, x.cell_start, e.scratch.sites, x.cell_atoms,
      e.nbr.cell_sites);
  }
  const bool verlet = !x.from_box && x.bv.sflag != nullptr;
  int p2r = 1;
  while (p2r < std::max(e.nbr.mn_r, verlet ? x.bv.mn : 0)) p2r <<= 1;
  const int warps = threads / 32;
  const int blocks = std::min((N + warps - 1) / warps, 148 * 8);
  const size_t smem = sizeof(int) * warps * (p2r + 1);
  BatchVerlet bv = x.bv;
  const RowHeads rh{e.nbr.nl_a, e.nbr.heads, e.nbr.st_a, e.nbr.st_h};
  if (!verlet) bv.sflag = nullptr;
  auto rows = [&](auto kernel, size_t bytes) {
    if (bytes > 48 * 1024)
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(bytes));
    kernel<<<blocks, threads, bytes, stream>>>(
      e.params, N, x.d_si, x.d_soff, x.n_struct, pos, type, e.nbr.nn_r, x.er, e.nbr.mn_r,
      e.nbr.nn_a, x.ea, e.nbr.mn_a, rh, x.cell_count, x.cell_start, x.cell_atoms, x.cell_of,
      e.nbr.cell_sites, e.model.rc_max, p2r, e.scratch.sites, x.large, x.from_box ? 0 : 1, bv,
      e.d_nstate);
  };
  if (x.kinds & kSmallRows) rows(k_rows_explicit<true>, 0);
  if (x.kinds & kLargeRows) rows(k_rows_explicit<false>, smem);
  if (verlet)
    k_rows_verlet<<<blocks, threads, 0, stream>>>(
      e.params, N, x.d_si, x.d_soff, x.n_struct, pos, type, e.nbr.nn_r, x.er, e.nbr.mn_r,
      e.nbr.nn_a, x.ea, e.nbr.mn_a, rh, e.scratch.sites, x.large, bv, e.d_nstate);
}

bool verlet_encodable(const StructInfo& s, double skin)
{
  for (int d = 0; d < 3; ++d) {
    const double* r = s.box.hinv + 3 * d;
    const double thick = 1.0 / std::sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    if (s.box.pbc[d] && thick < 4.0 * skin) return false;
  }
  if (!s.small) return true;
  return s.n <= (1 << kCandIndexBits) && s.ncell[0] <= kCandMaxImages &&
         s.ncell[1] <= kCandMaxImages && s.ncell[2] <= kCandMaxImages;
}

void launch_explicit_row_indices(const Engine& e, int which, int n, int* nn, int* nl, int mn,
                                 cudaStream_t stream)
{
  const int src_mn = which == 0 ? e.nbr.mn_r : e.nbr.mn_a;
  k_row_indices<<<n, 64, 0, stream>>>(n, which == 0 ? e.nbr.nn_r : e.nbr.nn_a,
                                      which == 0 ? e.xr.er : e.xr.ea, src_mn, nn, nl, mn);
}

}  // namespace nepx
